"""Batches that the stream kernel puts into tile order (grids above 64 MB that
the footprints cover several times over): several cubes, odd sides, footprints
off the grid and records with bad indexes, against the per-visibility kernels.
Tolerances as in test_gpu_stream.py."""
import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, HpgError, abi, workloads
from test_gpu_stream import dense, diag, linear_ops, rel_norm

pytestmark = pytest.mark.gpu

# polarizations, Mueller table, grid side (y, one more), CF supports,
# visibilities: the grid's cells, footprints' cells and so on past the lines
CASES = {
    "one-polarization": (1, diag(1), 1499, (19, 24), 45001),
    "two-polarizations": (2, diag(2), 1101, (24,), 30011),
    "ring": (4, dense(4), 1031, (12,), 60007),
}


def make(case, prec, kind):
    npol, mi, side, supports, n = CASES[case]
    rng = np.random.default_rng(21)
    # (the mixed form's FP32 model wants an even width)
    gs = (side + (prec == abi.PRECISION_MIXED), side + 1, npol, 2)
    planes = max(max(r) for r in mi) + 1
    ext, vals = workloads.separable_cf(
        supports, 2, rng.standard_normal(planes) +
        1j * rng.standard_normal(planes))
    vis = workloads.visibilities(n, npol, gs, (0.05, -0.07), 1.2e9, rng,
                                 w_frac=0.2, ngroups=len(supports))
    vis["grid_cube"] = rng.integers(0, 2, n)
    vis["uvw"][::17, 0] *= 1.3  # some footprints off the grid
    vis["grid_cube"][::1009] = 2  # and some records with bad indexes
    vis["cf_index"][::997, 1] = len(supports)
    model = (rng.standard_normal((2, npol, side + 1, side)) +
             1j * rng.standard_normal((2, npol, side + 1, side)))
    if gs[0] > side:
        model = np.pad(model, ((0, 0), (0, 0), (0, 0), (0, 1)))
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), mi, mi)
    g.set_precision(prec)
    g.set_gridding_kernel(kind)
    g.set_convolution_function(CFArray(2, ext, vals))
    return g, vis, model


def run(case, prec, kind, what):
    import torch
    g, vis, model = make(case, prec, kind)
    if what != "grid":
        g.set_model(model)
    t = torch.from_numpy(np.frombuffer(vis.tobytes(), np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    before = g.kernel_launches()
    if what == "grid":
        g.grid_visibilities(t, on_device=True)
    elif what == "predict":
        g.degrid_get_predicted_visibilities(t, on_device=True)
    else:
        g.degrid_grid_get_residual_visibilities(t, on_device=True)
    with pytest.raises(HpgError) as e:
        g.fence()
    assert e.value.type == "OutOfBoundsCFIndex"
    if kind == abi.KERNEL_AUTO:
        assert g.last_kernel_streamed()
        # sort keys, descriptors, the kernel (and the FP32 model)
        assert g.kernel_launches() - before == 3 + (
            prec == abi.PRECISION_MIXED and what != "grid")
    r = (t.cpu().numpy().view(abi.visdata_dtype(g.npol)), g.grid_values(),
         g.grid_weights())
    g.close()
    return r


@pytest.mark.parametrize("what", ["grid", "predict", "residual"])
@pytest.mark.parametrize("prec", [abi.PRECISION_FP64, abi.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("case", list(CASES))
def test_against_per_visibility_kernels(gpu, case, prec, what):
    a = run(case, prec, abi.KERNEL_AUTO, what)
    b = run(case, prec, abi.KERNEL_DIRECT, what)
    fp64 = prec == abi.PRECISION_FP64
    va, vb = a[0]["vis"], b[0]["vis"]
    if what == "grid":
        assert a[0].tobytes() == b[0].tobytes()
    elif what == "predict" and fp64:
        mag = np.maximum(np.abs(vb.real), np.abs(vb.imag))
        assert (np.abs(va - vb) <=
                4 * np.spacing(mag.astype(np.float32))).all()
    else:
        assert rel_norm(va, vb) <= 1e-6
    if what != "predict":
        assert rel_norm(a[1], b[1]) <= (
            1e-12 if fp64 and what == "grid" else 1e-6)
        np.testing.assert_allclose(a[2], b[2], rtol=1e-12)


@pytest.mark.parametrize("case", list(CASES))
def test_linear_operators(gpu, case):
    """(Wide footprints in full tiles may be the tile operators'.)"""
    npol, _, side, _, n = CASES[case]
    out = []
    for kind in (abi.KERNEL_AUTO, abi.KERNEL_DIRECT):
        g, vis, _ = make(case, abi.PRECISION_FP64, kind)
        vis["grid_cube"] %= 2
        vis["cf_index"][:, 1] = 0
        out.append(linear_ops(g, vis, n, npol, (2, npol, side + 1, side), kind))
        g.close()
    for a, b in zip(*out):
        assert rel_norm(a, b) <= 1e-12
