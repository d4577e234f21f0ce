"""Bounded waits under the automatic choice: with a copy withheld (a flag that
nothing sets), the wait for it runs out, the next fence reports it, and the
gridder stays usable.  The stream kernel's ring withholds it itself; batches
that it takes without a ring, and batched launches, go to the tiled kernel."""
import time

import numpy as np
import pytest

import hpg_b200
import test_gpu_stream as stream
from hpg_b200 import HpgError, abi
from test_gpu_stream import rel_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("position", [0, 5, 700])
@pytest.mark.parametrize("prec", [abi.PRECISION_FP64, abi.PRECISION_MIXED],
                         ids=["fp64", "mixed"])
@pytest.mark.parametrize("case", ["ring-two-warps", "ring-seven-warps",
                                  "two-warps", "diag-4"])
def test_withheld_copy_is_reported(gpu, case, prec, position):
    g, vis = stream.make(case, prec, abi.KERNEL_AUTO)
    g.set_wait_limit(0.02)
    g.debug_withhold_copy(position)
    t0 = time.perf_counter()
    g.degrid_grid_visibilities(vis)
    with pytest.raises(HpgError) as e:
        g.fence()
    assert e.value.type == "Other" and "wait" in str(e.value)
    assert time.perf_counter() - t0 < 10.0
    g.fence()  # reported once and cleared
    g.debug_withhold_copy(-1)
    g.set_wait_limit(0.5)
    g.reset_grid()
    g.degrid_grid_visibilities(vis)
    g.fence()
    h, _ = stream.make(case, prec, abi.KERNEL_DIRECT)
    h.degrid_grid_visibilities(vis)
    h.fence()
    assert rel_norm(g.grid_values(), h.grid_values()) <= 1e-6
    np.testing.assert_allclose(g.grid_weights(), h.grid_weights(), rtol=1e-12)
    g.close()
    h.close()


def test_withheld_copy_of_a_batch(gpu):
    g, vis = stream.make("ring-two-warps", abi.PRECISION_FP64, abi.KERNEL_AUTO)
    h, _ = stream.make("ring-two-warps", abi.PRECISION_FP64, abi.KERNEL_AUTO)
    g.set_wait_limit(0.02)
    g.debug_withhold_copy(3)
    hpg_b200.grid_visibilities_batch([g, h], [vis, vis])
    with pytest.raises(HpgError) as e:
        g.fence()
    assert "wait" in str(e.value)
    g.debug_withhold_copy(-1)
    g.reset_grid()
    hpg_b200.grid_visibilities_batch([g, h], [vis, vis])
    g.fence()
    d, _ = stream.make("ring-two-warps", abi.PRECISION_FP64, abi.KERNEL_DIRECT)
    d.grid_visibilities(vis)
    d.fence()
    assert rel_norm(g.grid_values(), d.grid_values()) <= 1e-12
    for x in (g, h, d):
        x.close()
