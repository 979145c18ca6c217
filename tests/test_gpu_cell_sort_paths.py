"""The cell sort's two routes (ranking within small cells, radix sort) and their changeover, at the sizes
where tiles, warps and the routes meet, against a host stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# n, cells, keys crowded into one cell: below / at / past the small-cell limit (256), few and many keys a
# cell on average (64), tile edges (2048), more than 4096 scan tiles, one cell
CASES = [(1, 1, 0), (2047, 900, 0), (2048, 900, 255), (2049, 900, 256), (2049, 900, 257), (2049, 900, 258),
         (64 * 500 + 63, 500, 0), (64 * 501, 500, 0), (100003, 50021, 5000), (3001, 9_000_000, 300), (70001, 1, 0)]


@pytest.mark.parametrize("n,ncells,crowd", CASES)
@pytest.mark.parametrize("static", [False, True])
def test_cell_sort_routes(cuda_lib, n, ncells, crowd, static):
    import torch
    from deorbit_gb300 import sph
    rng = np.random.default_rng(n + ncells + crowd)
    keys = rng.integers(0, ncells, size=n).astype(np.uint32)
    if crowd:
        keys[keys == ncells // 3] = 0
        keys[rng.choice(n, crowd, replace=False)] = ncells // 3
    dk = torch.from_numpy(keys.view(np.int32)).cuda()
    perm = torch.full((n,), -7, dtype=torch.int32, device="cuda")
    start = torch.full((ncells + 1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    fn = sph.lib().sph_cell_sort_static if static else sph.lib().sph_cell_sort
    sph.check(fn(dk.data_ptr(), n, ncells, perm.data_ptr(), start.data_ptr(), None))
    assert np.array_equal(perm.cpu().numpy(), np.argsort(keys, kind="stable"))
    assert np.array_equal(start.cpu().numpy(), np.r_[0, np.cumsum(np.bincount(keys, minlength=ncells))])
