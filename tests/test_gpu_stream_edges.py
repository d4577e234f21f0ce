"""CF slices near the end of the stream kernel's shared-memory ring, through
every call that plans with it, against the per-visibility kernels.  Cases and
tolerances as in test_gpu_stream.py."""
import numpy as np
import pytest

import hpg_b200
import test_gpu_stream as stream
from hpg_b200 import CFArray, Gridder, abi, workloads
from test_gpu_stream import dense, rel_norm

pytestmark = pytest.mark.gpu

FORMS = [abi.PRECISION_FP64, abi.PRECISION_MIXED]
FORM_IDS = ["fp64", "mixed"]


def first(n, k):
    """n x n table with its first k elements active."""
    return [[r * n + c if r * n + c < k else -1 for c in range(n)]
            for r in range(n)]


# the widest slice that fits (one visibility at a time in the ring), the first
# that exceeds the ring by less than its rounding, and shapes beside them
EDGES = {
    "ring-one-slice": (4, dense(4), False, (6, 38), 907, 0.2),
    "ring-just-beyond": (4, dense(4), False, (6, 40), 1201, 0.2),
    "ring-3pol-beyond": (3, first(3, 5), False, (9, 72), 401, None),
    "ring-2pol": (2, dense(2), False, (12, 60), 1103, 0.2),
}


@pytest.fixture(autouse=True)
def edges(monkeypatch):
    for name, case in EDGES.items():
        monkeypatch.setitem(stream.CASES, name, case)


@pytest.mark.parametrize("what", ["grid", "predict", "residual"])
@pytest.mark.parametrize("prec", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("case", list(EDGES))
def test_single_calls(gpu, case, prec, what):
    stream.test_against_per_visibility_kernels(gpu, case, prec, what)


@pytest.mark.parametrize("case", list(EDGES))
def test_linear_operators(gpu, case):
    stream.test_linear_operators(gpu, case)


# supports of the gridders of one launch and visibilities of each: slices
# that share the ring, and the widest that it holds
BATCHES = {"two-warps": ((8, 12), (16,), (9, 10, 11), 701),
           "seven-warps": ((8, 24), (38,), (20, 32), 211),
           "just-beyond": ((8, 24), (40,), (20, 32), 211)}


@pytest.mark.parametrize("what", ["grid", "residual"])
@pytest.mark.parametrize("prec", FORMS, ids=FORM_IDS)
@pytest.mark.parametrize("batch", list(BATCHES))
def test_ring_across_the_gridders_of_a_batch(gpu, batch, prec, what):
    *sets, n = BATCHES[batch]
    rng = np.random.default_rng(11)
    jobs = []
    for k, supports in enumerate(sets):
        gs = (160 + 8 * k, 170 - 10 * k, 4, 1)
        ext, vals = workloads.separable_cf(
            supports, 6, rng.standard_normal(16) + 1j * rng.standard_normal(16))
        vis = workloads.visibilities(n + 37 * k, 4, gs, (0.05, -0.07), 1.2e9,
                                     rng, disk=0.35, w_frac=0.2,
                                     ngroups=len(supports), grad=0.2)
        vis["uvw"][::17, 0] *= 2.0  # some footprints off the grid
        model = (rng.standard_normal((1, 4) + gs[1::-1]) +
                 1j * rng.standard_normal((1, 4) + gs[1::-1]))
        jobs.append((gs, CFArray(6, ext, vals), vis, model))

    def gridders(precision, kind):
        out = []
        for gs, cf, vis, model in jobs:
            g = Gridder.create(0, 0, len(vis), None, gs, (0.05, -0.07),
                               dense(4), dense(4))
            g.set_precision(precision)
            g.set_gridding_kernel(kind)
            g.set_convolution_function(cf)
            if what == "residual":
                g.set_model(model)
            out.append(g)
        return out

    batched = gridders(prec, abi.KERNEL_AUTO)
    futs = hpg_b200.grid_visibilities_batch(
        batched, [j[2] for j in jobs], do_degrid=what == "residual",
        return_visibilities=True)
    batched[0].fence()
    single = gridders(abi.PRECISION_FP64, abi.KERNEL_DIRECT)
    for a, b, job, fut in zip(batched, single, jobs, futs):
        if what == "residual":
            f = b.degrid_grid_get_residual_visibilities(job[2])
            b.fence()
            assert rel_norm(fut.get()["vis"], f.get()["vis"]) <= 1e-6
        else:
            b.grid_visibilities(job[2])
        assert rel_norm(a.grid_values(), b.grid_values()) <= (
            1e-12 if prec == abi.PRECISION_FP64 and what == "grid" else 1e-6)
        np.testing.assert_allclose(a.grid_weights(), b.grid_weights(),
                                   rtol=1e-12)
    for g in batched + single:
        g.close()
