"""The shared-memory arithmetic of the stream kernel's plan (no GPU needed):
over footprints, plane counts, polarizations and passes, a slice that the plan
sends through the ring fits the ring, and the ring the CTA's shared memory."""
import ctypes

import numpy as np
import pytest

from hpg_b200 import abi

SMEM = 227 * 1024  # what a CTA can have
DEGRID = abi.DO_DEGRID
GRID = abi.DO_GRID


def plan(npol, mueller, taps, nvis, flags, precision, tiled):
    m = np.asarray(mueller, np.int32)
    t = np.asarray(taps, np.int32).reshape(-1, 2)
    out = abi.StreamPlan()
    abi.check(abi.load().hpgb_debug_stream_plan(
        npol, len(m), abi.ptr(m), abi.ptr(t), len(t), nvis, flags, 1,
        precision, int(tiled), ctypes.byref(out)))
    return out


def tables():
    """npol x npol tables with their first k elements active."""
    for npol in (2, 3, 4):
        for k in range(1, npol * npol + 1):
            m = np.arange(npol * npol).reshape(npol, npol)
            yield npol, np.where(m < k, m, -1)


def check(p):
    if not p.accepted:
        return False
    assert p.ring_offset + p.ring_bytes <= p.smem_bytes <= SMEM
    if p.ring:
        assert p.slice_bytes <= p.ring_bytes
    return bool(p.ring)


@pytest.mark.parametrize("npol,mueller", list(tables()),
                         ids=lambda v: str(v) if isinstance(v, int)
                         else f"{int((v >= 0).sum())}planes")
def test_slices_fit_the_ring(device_lib, npol, mueller):
    taps = list(range(1, 128, 2))
    most = 0
    for i, tx in enumerate(taps):
        for ty in taps[i:]:
            # more than the ring's shared memory: only the refusal is checked
            if (tx * ty + 1) * 8 * int((mueller >= 0).sum()) > 300 * 1024:
                break
            for flags, prec in ((DEGRID | GRID, abi.PRECISION_FP64),
                                (DEGRID, abi.PRECISION_MIXED)):
                p = plan(npol, mueller, [(tx, ty)], 2500, flags, prec, True)
                if check(p):
                    most = max(most, p.slice_bytes)
    if (mueller >= 0).sum() > npol:  # several planes in some row
        assert most > 190 * 1024  # the ring's end was reached


@pytest.mark.parametrize("npol,planes,taps", [(4, 16, (41, 41)),
                                              (4, 16, (33, 51)),
                                              (4, 6, (55, 81)),
                                              (3, 9, (35, 85)),
                                              (3, 5, (73, 73))])
@pytest.mark.parametrize("tiled", [False, True])
def test_slices_near_the_rings_end(device_lib, npol, planes, taps, tiled):
    """Slices that exceed the ring by less than its rounding."""
    m = np.arange(npol * npol).reshape(npol, npol)
    m = np.where(m < planes, m, -1)
    for prec in (abi.PRECISION_FP64, abi.PRECISION_MIXED):
        for flags in (DEGRID, GRID, DEGRID | GRID):
            for nvis in (1, 2500, 6000):
                check(plan(npol, m, [taps], nvis, flags, prec, tiled))
