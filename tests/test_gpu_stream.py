"""The automatic choice's one-visibility-per-group kernel (stream_kernel.cuh)
against the per-visibility kernels (HPGB_KERNEL_DIRECT), which the parity
tests pin to the oracle, at the edges of its variants: one to sixteen warps
per visibility, CF slices from global memory and through the ring (which wraps
and holds a single part), partial Mueller rows, several cubes, footprints off
the grid, batches that end inside a CTA's block.

Tolerances: the FP64 form's products are the same FP32 products, summed in
FP64 in another order (1e-12 of the grid's norm for gridding; predictions are
rounded once to complex<float>, 4 ulps); the mixed form's FP32 sums are held
to its 1e-6.
"""
import ctypes

import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, abi, workloads

pytestmark = pytest.mark.gpu


def rel_norm(a, b):
    return np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel())


def diag(n):
    return [[r if c == r else -1 for c in range(n)] for r in range(n)]


def dense(n):
    return [[r * n + c for c in range(n)] for r in range(n)]


# polarizations, Mueller table, its transpose as the conjugate's?, CF supports,
# visibilities, phase screens
CASES = {
    "one-warp-1": (1, dense(1), False, (3,), 1, None),
    "one-warp": (1, dense(1), False, (4, 7, 10), 2371, 0.3),
    "two-warps": (2, diag(2), False, (40, 48), 5003, None),
    "four-warps": (2, diag(2), False, (24, 31), 333, 0.2),
    "diag-4": (4, diag(4), False, (5, 12, 20), 1777, 0.2),
    "dense-global": (4, dense(4), False, (4, 5), 2999, 0.3),
    "dense-transposed": (2, dense(2), True, (5, 9), 1501, 0.3),
    "partial": (4, [[0, -1, 1, -1], [-1, 2, -1, -1], [3, 4, 5, -1],
                    [-1, -1, -1, -1]], False, (4, 8), 1203, 0.2),
    "ring-two-warps": (4, dense(4), False, (8, 12, 16), 1999, 0.2),
    "ring-seven-warps": (4, dense(4), False, (8, 24, 36), 1013, None),
    "sixteen-warps": (4, dense(4), False, (9, 52), 207, 0.2),
}


def make(case, prec, kind, seed=5):
    npol, mi, transposed, supports, n, grad = CASES[case]
    rng = np.random.default_rng(seed)
    planes = max(max(r) for r in mi) + 1
    ci = [list(r) for r in np.array(mi).T] if transposed else mi
    gs = (131, 150, npol, 2)
    ext, vals = workloads.separable_cf(
        supports, 6, rng.standard_normal(planes) +
        1j * rng.standard_normal(planes), ncube=2)
    vis = workloads.visibilities(n, npol, gs, (0.05, -0.07), 1.2e9, rng,
                                 w_frac=0.2, ngroups=len(supports), grad=grad,
                                 ncube_cf=2)
    vis["phase"] = rng.uniform(-3, 3, n)
    vis["grid_cube"] = rng.integers(0, 2, n)
    vis["uvw"][::17, 0] *= 1.3  # some footprints off the grid
    model = (rng.standard_normal((2, npol, 150, 131)) +
             1j * rng.standard_normal((2, npol, 150, 131)))
    if prec == abi.PRECISION_MIXED:  # its FP32 model wants an even width
        gs = (132, 150, npol, 2)
        model = np.pad(model, ((0, 0), (0, 0), (0, 0), (0, 1)))
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), mi, ci)
    g.set_precision(prec)
    g.set_gridding_kernel(kind)
    g.set_convolution_function(CFArray(6, ext, vals))
    g.set_model(model)
    return g, vis


def run(case, prec, kind, what):
    g, vis = make(case, prec, kind)
    out = None
    if what == "grid":
        g.grid_visibilities(vis)
        g.fence()
    else:
        f = (g.degrid_get_predicted_visibilities(vis) if what == "predict"
             else g.degrid_grid_get_residual_visibilities(vis))
        g.fence()
        out = f.get()["vis"]
    r = (out, g.grid_values(), g.grid_weights())
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
    if a[0] is not None:
        if fp64:
            mag = np.maximum(np.abs(b[0].real), np.abs(b[0].imag))
            assert (np.abs(a[0] - b[0]) <=
                    4 * np.spacing(mag.astype(np.float32))).all()
        else:
            assert rel_norm(a[0], b[0]) <= 1e-6
    if what != "predict":
        assert rel_norm(a[1], b[1]) <= (
            1e-12 if fp64 and what == "grid" else 1e-6)
        np.testing.assert_allclose(a[2], b[2], rtol=1e-12, atol=1e-12)
    else:
        assert not a[1].any()


def linear_ops(g, vis, n, npol, shape, kind, seed=3):
    """D, D^H, G and G^H of one batch, each on the same random input."""
    import torch
    gen = torch.Generator(device="cuda:0").manual_seed(seed)
    dvis = torch.from_numpy(
        np.frombuffer(vis.tobytes(), np.uint8).copy()).to("cuda:0")
    crandn = lambda s: torch.randn(s, generator=gen, dtype=torch.complex128,
                                   device="cuda:0")
    grid, vals = crandn(shape), crandn((n, npol))
    g.set_gridding_kernel(kind)
    lib, out = abi.load(), []
    for f, a, to_vals in ((lib.hpgb_degrid_linear, grid, True),
                          (lib.hpgb_degrid_adjoint, vals, False),
                          (lib.hpgb_grid_linear, vals, False),
                          (lib.hpgb_grid_adjoint, grid, True)):
        b = torch.zeros((n, npol) if to_vals else shape,
                        dtype=torch.complex128, device="cuda:0")
        torch.cuda.synchronize()
        abi.check(f(g._h, ctypes.c_void_p(dvis.data_ptr()), n, npol,
                    ctypes.c_void_p(a.data_ptr()),
                    ctypes.c_void_p(b.data_ptr())))
        g.fence()
        out.append(b.cpu().numpy())
    return out


def assert_linear_ops_agree(g, vis, n, npol, shape):
    auto = linear_ops(g, vis, n, npol, shape, abi.KERNEL_AUTO)
    direct = linear_ops(g, vis, n, npol, shape, abi.KERNEL_DIRECT)
    for a, b in zip(auto, direct):
        assert rel_norm(a, b) <= 1e-12


@pytest.mark.parametrize("case", list(CASES))
def test_linear_operators(gpu, case):
    g, vis = make(case, abi.PRECISION_FP64, abi.KERNEL_AUTO)
    npol, n = CASES[case][0], CASES[case][4]
    assert_linear_ops_agree(g, vis, n, npol, (2, npol, 150, 131))
    g.close()


@pytest.mark.parametrize("n", [5000, 40000, 160000])
def test_linear_operators_tile_line(gpu, n):
    """Batches on both sides of the rule that leaves wide footprints in full
    tiles to the tile kernels: 27 x 27 tiles of 7, 55 and 220 visibilities
    (the adjoints' line is near 25, the forward operators' near 130)."""
    rng = np.random.default_rng(9)
    gs = (1100, 1111, 2, 1)
    ext, vals = workloads.separable_cf(
        (40,), 2, rng.standard_normal(2) + 1j * rng.standard_normal(2), ncube=1)
    vis = workloads.visibilities(n, 2, gs, (0.05, -0.07), 1.2e9, rng,
                                 w_frac=0.2, ngroups=1, grad=None, ncube_cf=1)
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), diag(2), diag(2))
    g.set_convolution_function(CFArray(2, ext, vals))
    assert_linear_ops_agree(g, vis, n, 2, (1, 2, 1111, 1100))
    g.close()


def test_wait_limit_and_status(gpu):
    """The ring variant under the shortest wait limit: nothing waits long."""
    g, vis = make("ring-two-warps", abi.PRECISION_FP64, abi.KERNEL_AUTO)
    g.set_wait_limit(0.01)
    for _ in range(3):
        g.grid_visibilities(vis)
    g.fence()
    g.close()
