"""CF ingestion from the logical order (one pass, cf_runs_kernel) against the
reference's device layout version "0-Cuda" of the same values (the other
layouts' kernel): runs of 1 to 40 values per position, several cubes, odd and
even oversampling, unequal sides, more rows than one step turns.  The same
slices give the same products in another order of FP64 additions (1e-13), and
the slices' sums the grid weights (1e-13)."""
import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, abi, workloads

pytestmark = pytest.mark.gpu


def cuda_v0(v, os_):
    """Logical (x, y, mueller, cube) values in the layout "0-Cuda"."""
    nx, ny, nm, nc = v.shape
    xm, ym = -(-nx // os_), -(-ny // os_)
    out = np.zeros((os_, os_, nc, nm, ym, xm), np.complex64)
    for xi in range(os_):
        for yi in range(os_):
            part = v[xi::os_, yi::os_]
            out[yi, xi, :, :, :part.shape[1], :part.shape[0]] = \
                part.transpose(3, 2, 1, 0)
    return out.reshape(-1)


@pytest.mark.parametrize("planes,ncube,os_,sx,sy,npol,mi", [
    (1, 1, 1, 3, 4, 1, [[0]]),
    (1, 3, 7, 9, 6, 1, [[0]]),
    (2, 1, 20, 7, 7, 2, [[0, -1], [-1, 1]]),
    (5, 1, 8, 11, 3, 1, [[3]]),
    (16, 1, 6, 40, 33, 4,
     [[r * 4 + c for c in range(4)] for r in range(4)]),
    (16, 2, 5, 8, 10, 4,
     [[r * 4 + c for c in range(4)] for r in range(4)]),
    (40, 1, 4, 6, 9, 1, [[37]]),
])
def test_logical_order_equals_device_layout(gpu, planes, ncube, os_, sx, sy,
                                            npol, mi):
    rng = np.random.default_rng(planes + os_)
    ext = ((sx + 4) * os_, (sy + 4) * os_, planes, ncube)
    v = (rng.standard_normal(ext) + 1j * rng.standard_normal(ext)).astype(
        np.complex64)
    gs = (120, 110, npol, 1)
    vis = workloads.visibilities(4000, npol, gs, (0.05, 0.05), 1.4e9, rng,
                                 disk=0.25, w_frac=0.2, ncube_cf=ncube)
    got = []
    for cf in (CFArray(os_, [ext], [v]),
               CFArray(os_, [ext], [cuda_v0(v, os_)], layout="0-Cuda")):
        g = Gridder.create(0, 0, len(vis), None, gs, (0.05, 0.05), mi, mi)
        g.set_convolution_function(cf)
        g.grid_visibilities(vis)
        g.fence()
        got.append((g.grid_values(), g.grid_weights()))
        g.close()
    (ga, wa), (gb, wb) = got
    assert np.linalg.norm(gb) > 0
    assert np.linalg.norm(ga - gb) <= 1e-13 * np.linalg.norm(gb)
    np.testing.assert_allclose(wa, wb, rtol=1e-13)
