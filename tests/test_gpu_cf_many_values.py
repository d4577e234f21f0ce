"""CF sets with more values at a position (Mueller elements times cubes) than
the one-pass ingestion's blocks take, and the most that they take."""
import numpy as np
import pytest

from hpg_b200 import CFArray, Gridder, abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncube", [131070, 131071, 131072, 140001])
def test_cubes_beyond_a_launchs_blocks(gpu, ncube):
    """One cell of support: a visibility's grid increment is its cube's CF
    value times its own."""
    import torch
    gen = torch.Generator(device="cuda:0").manual_seed(ncube)
    v = torch.randn((4, 4, 16, ncube), generator=gen, dtype=torch.complex64,
                    device="cuda:0")
    torch.cuda.synchronize()
    g = Gridder.create(0, 0, 3, None, (16, 16, 1, 1), (0.05, 0.05), [[13]],
                       [[13]])
    g.set_convolution_function(CFArray(1, [tuple(v.shape)], [v]),
                               on_device=True)
    vis = np.zeros(3, abi.visdata_dtype(1))
    vis["vis"] = [[1], [2], [4]]
    vis["weights"] = 1
    vis["freq"] = 1e9
    vis["cf_index"][:, 0] = [0, ncube // 2, ncube - 1]
    g.grid_visibilities(vis)
    g.fence()
    cf = v[2, 2, 13].cpu().numpy()[vis["cf_index"][:, 0]].astype(np.complex128)
    grid = g.grid_values().ravel()
    total = (np.conj(cf) * vis["vis"][:, 0]).sum()
    assert np.count_nonzero(grid) == 1
    # (either sign of the CF's imaginary part, by the sign of w)
    got = grid[np.nonzero(grid)][0]
    assert min(abs(got - total), abs(got - (cf * vis["vis"][:, 0]).sum())) <= (
        1e-6 * abs(total))
    g.close()
