"""Device records under the automatic choice, which reads them where they lie
when it can: results beside them, in their place or nowhere, records that only
a copy can take, and a captured call, against the same call on host records."""
import ctypes

import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, abi, workloads
from test_gpu_stream import dense, diag, rel_norm

pytestmark = pytest.mark.gpu

# polarizations, Mueller table, CF supports, visibilities
CASES = {"diag": (2, diag(2), (6, 11), 1501),
         "ring": (4, dense(4), (8, 14), 901),
         "tiled": (4, dense(4), (30,), 7001)}
PREDICT = abi.DO_DEGRID | abi.RETURN_VISIBILITIES
GRID = abi.DO_GRID | abi.UPDATE_GRID_WEIGHTS
RESIDUAL = abi.DO_DEGRID | abi.RETURN_VISIBILITIES | GRID


def make(case, with_model=True):
    npol, mi, supports, n = CASES[case]
    rng = np.random.default_rng(12)
    gs = (140, 150, npol, 1)
    planes = max(max(r) for r in mi) + 1
    ext, vals = workloads.separable_cf(
        supports, 6, rng.standard_normal(planes) +
        1j * rng.standard_normal(planes))
    vis = workloads.visibilities(n, npol, gs, (0.05, -0.07), 1.2e9, rng,
                                 w_frac=0.2, ngroups=len(supports), grad=0.2)
    vis["uvw"][::17, 0] *= 1.3  # some footprints off the grid
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), mi, mi)
    g.set_convolution_function(CFArray(6, ext, vals))
    if with_model:
        g.set_model(rng.standard_normal((1, npol, 150, 140)) +
                    1j * rng.standard_normal((1, npol, 150, 140)))
    return g, vis


def on_device(vis, pad=0):
    """The records' bytes on the device, `pad` bytes into an allocation."""
    import torch
    t = torch.zeros(pad + vis.nbytes, dtype=torch.uint8, device="cuda:0")
    t[pad:] = torch.from_numpy(np.frombuffer(vis.tobytes(), np.uint8).copy())
    torch.cuda.synchronize()
    return t[pad:]


def call(g, n, flags, vis, returned):
    abi.check(abi.load().hpgb_grid_visibilities(
        g._h, ctypes.c_void_p(vis), n, g.npol, flags, 1,
        ctypes.c_void_p(returned)))
    g.fence()


def on_host(case, flags, with_model=True):
    """Returned records (or the batch's own), grid and weights."""
    g, vis = make(case, with_model)
    out = g.raw_grid_visibilities(vis, flags)
    g.fence()
    r = (vis if out is None else out, g.grid_values(), g.grid_weights())
    g.close()
    return r


def same(g, case, flags, expected, records, with_model=True):
    if flags & abi.DO_GRID:
        assert rel_norm(g.grid_values(), expected[1]) <= 1e-12
    np.testing.assert_allclose(g.grid_weights(), expected[2], rtol=1e-12)
    if records is not None:
        got = records.cpu().numpy().view(abi.visdata_dtype(g.npol))
        assert np.array_equal(got, expected[0])


@pytest.mark.parametrize("flags", [PREDICT, GRID, RESIDUAL,
                                   GRID | abi.RETURN_VISIBILITIES],
                         ids=["predict", "grid", "residual", "grid-returned"])
@pytest.mark.parametrize("where", ["same", "beside", "unaligned",
                                   "unaligned-out", "overlapping", "pinned"])
@pytest.mark.parametrize("case", list(CASES))
def test_results_as_with_host_records(gpu, case, where, flags):
    import torch
    expected = on_host(case, flags)
    g, vis = make(case)
    rec = vis.dtype.itemsize
    if where == "overlapping":  # results from the third record on
        keep = torch.cat([on_device(vis), on_device(vis[:3])])
        src, dst = keep[:vis.nbytes], keep[3 * rec:]
    elif where == "pinned":
        src = torch.from_numpy(
            np.frombuffer(vis.tobytes(), np.uint8).copy()).pin_memory()
        dst = src
    else:
        src = on_device(vis, 4 if where == "unaligned" else 0)
        dst = src if where == "same" else on_device(
            vis, 4 if where == "unaligned-out" else 0).zero_()
    torch.cuda.synchronize()
    back = flags & abi.RETURN_VISIBILITIES
    call(g, len(vis), flags, src.data_ptr(), dst.data_ptr() if back else None)
    same(g, case, flags, expected, dst if back else None)
    if not back or where in ("beside", "unaligned", "unaligned-out"):
        assert src.cpu().numpy().tobytes() == vis.tobytes()  # untouched
    g.close()


@pytest.mark.parametrize("case", list(CASES))
def test_no_results_leave_the_records_alone(gpu, case):
    flags = abi.DO_DEGRID | GRID
    expected = on_host(case, flags)
    g, vis = make(case)
    src = on_device(vis)
    call(g, len(vis), flags, src.data_ptr(), None)
    same(g, case, flags, expected, None)
    assert src.cpu().numpy().tobytes() == vis.tobytes()
    g.close()


@pytest.mark.parametrize("with_model", [True, False], ids=["model", "no-model"])
@pytest.mark.parametrize("case", list(CASES))
def test_captured_call(gpu, case, with_model):
    """Residuals of records in place, captured and replayed on new values."""
    import torch
    g, vis = make(case, with_model)
    src = on_device(vis)
    g.degrid_grid_get_residual_visibilities(src, on_device=True)  # buffers
    g.fence()
    g.reset_grid()
    with g.capture() as graph:
        g.degrid_grid_get_residual_visibilities(src, on_device=True)
    for seed in (1, 2):
        new = vis.copy()
        new["vis"] *= np.float32(seed)
        src.copy_(torch.from_numpy(np.frombuffer(new.tobytes(), np.uint8).copy()))
        torch.cuda.synchronize()
        g.reset_grid()
        graph.launch()
        g.fence()
        h, _ = make(case, with_model)
        out = h.raw_grid_visibilities(new, RESIDUAL)
        h.fence()
        same(g, case, RESIDUAL, (out, h.grid_values(), h.grid_weights()), src)
        h.close()
    graph.close()
    g.close()


def in_place(device, vis, nbytes, returned=None):
    r = ctypes.c_int(-1)
    abi.check(abi.load().hpgb_debug_records_in_place(
        device, ctypes.c_void_p(vis), nbytes, ctypes.c_void_p(returned),
        ctypes.byref(r)))
    return r.value


def test_which_records_are_read_in_place(gpu):
    import torch
    t = torch.zeros(4096, dtype=torch.uint8, device="cuda:0")
    host = torch.zeros(1024, dtype=torch.uint8)
    pinned = host.pin_memory()
    p = t.data_ptr()
    for returned, yes in ((None, 1), (p, 1), (p + 1024, 1), (p + 1016, 0),
                          (p + 1028, 0), (pinned.data_ptr(), 0)):
        assert in_place(0, p, 1024, returned) == yes, returned
    assert in_place(0, p + 2048, 1024, p + 1024) == 1
    assert in_place(0, p + 2048, 1024, p + 1032) == 0
    assert in_place(0, p + 4, 1024) == 0
    assert in_place(0, pinned.data_ptr(), 1024) == 0
    assert in_place(0, host.data_ptr(), 1024) == 0
    # a gridder of another device than the records'
    assert in_place(1, p, 1024) == 0
