"""A point without a usable position (a NaN or infinite coordinate, its grid cell
known) neither answers nor disturbs the other queries of its work item: their
rows equal those of the same call without the point, bit for bit."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1, 2)])
@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("cut", [math.inf, 0.01])
@pytest.mark.parametrize("n,k,side", [(6000, 8, 3), (6000, 16, 3), (6000, 16, 12),
                                      (100000, 16, 9), (100000, 16, 28)])
def test_bad_point_leaves_the_others_alone(n, k, side, cut, bad, axes):
    """side: parent cells per axis, for groups of a few candidates (packed items)
    up to thousands (chunked items of 4 up to 32 queries); with a cut radius
    the bad query's own bound is finite too."""
    import flashknn_exprepo_b200 as fk
    gen = torch.Generator(device=DEV)
    gen.manual_seed(side)
    xyz = torch.rand((n, 3), generator=gen, device=DEV)
    xyz[-1] = 0.5
    grid = torch.floor(xyz * (4 * side)).long()
    want_idx, want_dist = fk.ops.knn_grid(xyz[:-1].contiguous(), grid[:-1].contiguous(), None, k,
                                          2, cut_r2=cut, idx_dtype=torch.int32, validate=True)
    xyz[-1, list(axes)] = bad
    idx, dist = fk.ops.knn_grid(xyz, grid, None, k, 2, cut_r2=cut, idx_dtype=torch.int32,
                                validate=True)
    assert torch.equal(idx[:-1], want_idx) and torch.equal(dist[:-1], want_dist)
    assert bool((idx[-1] == n - 1).all()) and bool(torch.isinf(dist[-1]).all())
