"""Which kernel the automatic choice takes, told by hpgb_last_kernel_streamed,
and the tiled kernels where the automatic choice has left them: batched
launches and the linear operators at wide supports, through the same checks
as the automatic choice."""
import numpy as np
import pytest

import hpg_b200
import test_adjoint
import test_gpu_batch
import test_gpu_stream as stream
from hpg_b200 import CFArray, Gridder, abi, workloads
from test_gpu_stream import dense, diag, rel_norm

pytestmark = pytest.mark.gpu


def gridder(npol, mi, supports, n, kind=abi.KERNEL_AUTO, side=160, seed=8):
    rng = np.random.default_rng(seed)
    gs = (side, side, npol, 1)
    planes = max(max(r) for r in mi) + 1
    ext, vals = workloads.separable_cf(
        supports, 4, rng.standard_normal(planes) +
        1j * rng.standard_normal(planes))
    vis = workloads.visibilities(n, npol, gs, (0.05, -0.07), 1.2e9, rng,
                                 disk=0.3, w_frac=0.2, ngroups=len(supports))
    g = Gridder.create(0, 0, n, None, gs, (0.05, -0.07), mi, mi)
    g.set_gridding_kernel(kind)
    g.set_convolution_function(CFArray(4, ext, vals))
    return g, vis


@pytest.mark.parametrize("npol,mi,supports,n,kind,plan,streamed", [
    (1, diag(1), (7,), 1000, abi.KERNEL_AUTO, 0, True),
    (1, diag(1), (7,), 1000, abi.KERNEL_TILED, 0, False),
    (1, diag(1), (7,), 1000, abi.KERNEL_DIRECT, 0, False),
    (1, diag(1), (7,), 1000, abi.KERNEL_AUTO, 4, False),  # a plan by hand
    (2, diag(2), (20, 30), 500, abi.KERNEL_AUTO, 0, True),
    (4, dense(4), (8, 12), 500, abi.KERNEL_AUTO, 0, True),
    (4, dense(4), (30,), 500, abi.KERNEL_AUTO, 0, True),
    (4, dense(4), (30,), 7000, abi.KERNEL_AUTO, 0, False),
    (4, dense(4), (40,), 500, abi.KERNEL_AUTO, 0, False),
    (4, dense(4), (52,), 100, abi.KERNEL_AUTO, 0, True),
])
def test_kernel_of_single_calls(gpu, npol, mi, supports, n, kind, plan,
                                streamed):
    g, vis = gridder(npol, mi, supports, n, kind)
    g.set_tiled_plan(ring_parts=plan)
    assert not g.last_kernel_streamed()
    g.grid_visibilities(vis)
    g.fence()
    assert g.last_kernel_streamed() is streamed
    g.set_gridding_kernel(abi.KERNEL_DIRECT)
    g.grid_visibilities(vis[:0])  # an empty batch says nothing
    assert g.last_kernel_streamed() is streamed
    g.grid_visibilities(vis)
    g.fence()
    assert not g.last_kernel_streamed()
    g.close()


@pytest.mark.parametrize("kind,streamed", [(abi.KERNEL_AUTO, True),
                                           (abi.KERNEL_TILED, False),
                                           (abi.KERNEL_DIRECT, False)])
def test_kernel_of_linear_operators(gpu, kind, streamed):
    g, vis = gridder(2, diag(2), (8, 14), 700)
    stream.linear_ops(g, vis, len(vis), 2, (1, 2, 160, 160), kind)
    assert g.last_kernel_streamed() is streamed
    g.close()


def of_kind(kind, made):
    """test_gpu_batch.gridders_for with the kernel selected; the gridders go
    into `made`."""
    plain = test_gpu_batch.gridders_for

    def gridders(*args):
        gs = plain(*args)
        for g in gs:
            g.set_gridding_kernel(kind)
        made.append([(g, g.close) for g in gs])
        for g in gs:
            g.close = lambda: None  # looked at after the test
        return gs
    return gridders


@pytest.mark.parametrize("kind", [abi.KERNEL_AUTO, abi.KERNEL_TILED],
                         ids=["auto", "tiled"])
@pytest.mark.parametrize("degrid", [False, True], ids=["grid", "degrid+grid"])
@pytest.mark.parametrize("precision,comp", test_gpu_batch.FORMS,
                         ids=test_gpu_batch.FORM_IDS)
def test_batches(gpu, oracle_lib, monkeypatch, precision, comp, degrid, kind):
    made = []
    monkeypatch.setattr(test_gpu_batch, "gridders_for", of_kind(kind, made))
    test_gpu_batch.test_batch_matches_oracle(gpu, oracle_lib, precision, comp,
                                             degrid)
    for j, (g, close) in enumerate(made[0]):
        # (job 7 is empty)
        assert g.last_kernel_streamed() is (kind == abi.KERNEL_AUTO and j != 7)
        close()


@pytest.mark.parametrize("kind", [abi.KERNEL_AUTO, abi.KERNEL_TILED],
                         ids=["auto", "tiled"])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
def test_batches_of_wide_supports(gpu, oracle_lib, monkeypatch, precision,
                                  kind):
    made = []
    monkeypatch.setattr(test_gpu_batch, "gridders_for", of_kind(kind, made))
    test_gpu_batch.test_batch_wide_supports(gpu, oracle_lib, precision)
    for g, close in made[0]:
        assert g.last_kernel_streamed() is (kind == abi.KERNEL_AUTO)
        close()


def test_batch_split_between_kernels(gpu, oracle_lib, monkeypatch):
    made = []
    monkeypatch.setattr(test_gpu_batch, "gridders_for",
                        of_kind(abi.KERNEL_AUTO, made))
    test_gpu_batch.test_batch_split_between_kernels(gpu, oracle_lib)
    kinds = [g.last_kernel_streamed() for g, _ in made[0]]
    assert any(kinds) and not all(kinds)
    for _, close in made[0]:
        close()


def test_dense_batch_through_the_tiled_kernel(gpu):
    """Dense 4x4 slices beyond what the stream kernel takes: the automatic
    choice's batched launch, against one per-visibility call a gridder."""
    sets = [((16, 30), 4000), ((30,), 3500)]
    made = [gridder(4, dense(4), s, n, side=180 + 20 * k, seed=k)
            for k, (s, n) in enumerate(sets)]
    hpg_b200.grid_visibilities_batch([g for g, _ in made],
                                     [v for _, v in made])
    made[0][0].fence()
    for k, (g, vis) in enumerate(made):
        assert not g.last_kernel_streamed()
        d, _ = gridder(4, dense(4), *sets[k], kind=abi.KERNEL_DIRECT,
                       side=180 + 20 * k, seed=k)
        d.grid_visibilities(vis)
        d.fence()
        assert rel_norm(g.grid_values(), d.grid_values()) <= 1e-12
        np.testing.assert_allclose(g.grid_weights(), d.grid_weights(),
                                   rtol=1e-12)
        d.close()
        g.close()


@pytest.mark.parametrize("grad", [0.2, None], ids=["screen", "no-screen"])
@pytest.mark.parametrize("npol", [1, 2])
def test_tiled_operators_at_wide_supports(gpu, monkeypatch, npol, grad):
    # (the test selects the kernel by this name)
    monkeypatch.setattr(abi, "KERNEL_AUTO", abi.KERNEL_TILED)
    test_adjoint.test_wide_support_dot_products(gpu, npol, abi.KERNEL_TILED,
                                                grad)


def test_autotuner_keeps_the_automatic_choice_where_it_is_faster(gpu):
    """Small footprints: several times faster through the stream kernel, which
    a tiled plan would switch off; the tuned call is that one.  The same batch
    under KERNEL_TILED, and a batch that the stream kernel does not take, get
    a plan."""
    g, vis = gridder(2, diag(2), (5, 7, 11, 15), 20000)
    before = (g.grid_values(), g.grid_weights())
    assert g.autotune_tiled(vis, abi.DO_GRID) == (0, 0)
    assert g.autotune_tiled(vis, abi.DO_GRID) == (0, 0)  # from the cache
    assert g.tiled_plan()["ring_parts"] == 0
    assert g.last_gridding_kernel() == abi.KERNEL_AUTO  # no batch yet
    assert not g.last_kernel_streamed()
    assert np.array_equal(g.grid_values(), before[0])
    assert np.array_equal(g.grid_weights(), before[1])
    g.grid_visibilities(vis)
    g.fence()
    assert g.last_kernel_streamed()
    g.close()
    for args in ((2, diag(2), (5, 7, 11, 15), 20000, abi.KERNEL_TILED),
                 (4, dense(4), (30,), 7000, abi.KERNEL_AUTO)):
        g, vis = gridder(*args)
        ring, _ = g.autotune_tiled(vis, abi.DO_GRID)
        assert 2 <= ring <= 8 and g.tiled_plan()["ring_parts"] == ring
        g.grid_visibilities(vis)
        g.fence()
        assert not g.last_kernel_streamed()
        g.close()


@pytest.mark.parametrize("kind", [abi.KERNEL_AUTO, abi.KERNEL_TILED],
                         ids=["auto", "tiled"])
def test_profiled_launches_are_gridding_launches(gpu, kind):
    g, vis = gridder(2, diag(2), (8, 14), 700, kind)
    g.profile_tiled_kernel(True)
    stream.linear_ops(g, vis, len(vis), 2, (1, 2, 160, 160), kind)
    assert g.tiled_kernel_time()[1] == 0
    for _ in range(3):
        g.grid_visibilities(vis)
    ms, n = g.tiled_kernel_time()
    assert n == 3 and ms > 0
    g.close()
