"""Arithmetic of the mixed form's automatic choice: as exact as the tiled
kernel's where that takes the batch, FP64 where only the per-visibility
kernels (an FP64 form) do."""
import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, HpgError, abi, workloads
from test_gpu_stream import dense, diag, rel_norm

pytestmark = pytest.mark.gpu


def results(npol, mi, supports, n, what, prec, kind, comp=0):
    """Predictions (or None) and grid of one seeded batch."""
    rng = np.random.default_rng(7)
    gs = (400, 400, npol, 1)
    planes = max(max(r) for r in mi) + 1
    ext, vals = workloads.separable_cf(
        supports, 2, rng.standard_normal(planes) +
        1j * rng.standard_normal(planes), w_phases=[0.01] * len(supports))
    vis = workloads.visibilities(n, npol, gs, (0.05, -0.07), 1.2e9, rng,
                                 disk=0.3, w_frac=0.2, ngroups=len(supports))
    model = (rng.standard_normal((1, npol, 400, 400)) +
             1j * rng.standard_normal((1, npol, 400, 400)))
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), mi, mi)
    g.set_precision(prec)
    g.set_gridding_kernel(kind)
    if comp:
        g.set_tiled_plan(compensated=comp)
    g.set_convolution_function(CFArray(2, ext, vals))
    g.set_model(model)
    out = None
    if what == "predict":
        f = g.degrid_get_predicted_visibilities(vis)
        g.fence()
        out = f.get()["vis"]
    else:
        g.grid_visibilities(vis)
        g.fence()
    r = (out, g.grid_values())
    g.close()
    return r


# polarizations, table, supports, visibilities, compensated tiles, calls
# that the tiled kernel refuses (its tiles are those of the call's passes)
REFUSED = {
    "wide-among-narrow": (1, diag(1), (8, 8, 8, 100), 6001, 0,
                          ("grid", "predict")),
    "two-polarizations": (2, diag(2), (100,), 907, 0, ("grid", "predict")),
    "sixteen-warps": (4, dense(4), (52,), 203, 0, ("grid",)),
    "sixteen-warps-predict": (4, dense(4), (64,), 203, 0, ("predict",)),
    "compensated": (2, dense(2), (60,), 1103, abi.COMPENSATED_ON, ("grid",)),
}


@pytest.mark.parametrize("case,what", [(c, w) for c in REFUSED
                                       for w in REFUSED[c][-1]])
def test_fp64_where_the_tiled_kernel_refuses(gpu, case, what):
    npol, mi, supports, n, comp = REFUSED[case][:-1]
    with pytest.raises(HpgError):
        results(npol, mi, supports, n, what, abi.PRECISION_MIXED,
                abi.KERNEL_TILED, comp)
    a = results(npol, mi, supports, n, what, abi.PRECISION_MIXED,
                abi.KERNEL_AUTO, comp)
    b = results(npol, mi, supports, n, what, abi.PRECISION_FP64,
                abi.KERNEL_DIRECT)
    if what == "predict":
        mag = np.maximum(np.abs(b[0].real), np.abs(b[0].imag))
        assert (np.abs(a[0] - b[0]) <=
                4 * np.spacing(mag.astype(np.float32))).all()
    else:
        assert rel_norm(a[1], b[1]) <= 1e-12


# polarizations, table, supports, visibilities
TAKEN = {
    "diag-1": (1, diag(1), (31,), 8000),
    "diag-2": (2, diag(2), (64,), 5000),
    "diag-2-few": (2, diag(2), (64,), 1500),
    "diag-4": (4, diag(4), (30,), 5000),
    "dense-global-2": (2, dense(2), (14,), 8000),
    "dense-global-4": (4, dense(4), (7,), 8000),
    "ring-two-warps-2": (2, dense(2), (30,), 8000),
    "ring-two-warps-3": (3, dense(3), (20,), 6000),
    "ring-two-warps-4": (4, dense(4), (16,), 8000),
    "ring-seven-warps-2": (2, dense(2), (60,), 2500),
    "ring-seven-warps-4": (4, dense(4), (32,), 2500),
    "ring-seven-warps-4-wide": (4, dense(4), (36,), 2500),
}


@pytest.mark.parametrize("case", list(TAKEN))
def test_predictions_as_exact_as_the_tiled_kernels(gpu, case):
    """The mixed form's sums against the FP64 form, in the variants that take
    batches from the tiled kernel: no further off than its sums are."""
    npol, mi, supports, n = TAKEN[case]
    ref, auto, tiled = (
        results(npol, mi, supports, n, "predict", prec, kind)[0]
        .astype(np.complex128) for prec, kind in (
            (abi.PRECISION_FP64, abi.KERNEL_DIRECT),
            (abi.PRECISION_MIXED, abi.KERNEL_AUTO),
            (abi.PRECISION_MIXED, abi.KERNEL_TILED)))
    err = rel_norm(auto, ref), rel_norm(tiled, ref)
    print("%s: %.3e, tiled kernel %.3e" % ((case,) + err))
    assert err[0] <= err[1]
