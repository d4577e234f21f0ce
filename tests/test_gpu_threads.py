"""Gridders in threads of their own, whose launches of the same kernels want
different amounts of shared memory."""
import threading

import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, abi, workloads
from test_gpu_stream import dense, diag

pytestmark = pytest.mark.gpu

# polarizations, table, kernel, CF supports of each thread's gridder
CASES = {
    "stream": (1, diag(1), abi.KERNEL_AUTO, ((3,), (10,), (6,))),
    "stream-ring": (2, dense(2), abi.KERNEL_AUTO, ((18,), (24,), (18, 24))),
    "tiled": (2, diag(2), abi.KERNEL_TILED, ((4,), (30,), (12,))),
}


@pytest.mark.parametrize("case", list(CASES))
def test_launches_from_several_threads(gpu, case):
    npol, mi, kind, sets = CASES[case]
    rng = np.random.default_rng(3)
    planes = max(max(r) for r in mi) + 1
    jobs = []
    for supports in sets:
        ext, vals = workloads.separable_cf(supports, 2, np.ones(planes))
        vis = workloads.visibilities(8, npol, (128, 128, npol, 1),
                                     (0.05, -0.07), 1.2e9, rng, disk=0.3,
                                     ngroups=len(supports))
        g = Gridder.create(0, 0, len(vis), None, (128, 128, npol, 1),
                           (0.05, -0.07), mi, mi)
        g.set_gridding_kernel(kind)
        g.set_convolution_function(CFArray(2, ext, vals))
        g.grid_visibilities(vis)
        g.fence()
        jobs.append((g, vis, g.grid_values()))
        g.reset_grid()
    errors, calls = [], 400

    def work(g, vis):
        try:
            for _ in range(calls):
                g.grid_visibilities(vis)
            g.fence()
        except Exception as e:  # told to the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=j[:2]) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, _, once in jobs:
        grid = g.grid_values()
        assert (np.linalg.norm(grid - calls * once) <=
                1e-12 * np.linalg.norm(calls * once))
        g.close()


def test_convolution_functions_from_several_threads(gpu):
    """CF ingestion likewise: supports whose turned rows exceed 48 KB."""
    import torch
    jobs = []
    for support in (210, 300):
        ext, vals = workloads.separable_cf_torch((support,), 1, np.ones(32),
                                                 "cuda:0")
        g = Gridder.create(0, 0, 1, None, (320, 320, 4, 1), (0.05, -0.07),
                           dense(4), dense(4))
        jobs.append((g, CFArray(1, ext, vals)))
    torch.cuda.synchronize()
    errors = []

    def work(g, cf):
        try:
            for _ in range(300):
                g.set_convolution_function(cf, on_device=True)
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, _ in jobs:
        g.close()
