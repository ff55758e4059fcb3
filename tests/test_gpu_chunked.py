"""Chunked items (groups with more candidates than a tile) at the edges of the
tile and of the 32-record steps in which the sphere filter compacts it:
bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _check(xyz, k, voxel):
    import flashknn_exprepo_b200 as fk
    offs = np.array([len(xyz)])
    oi, od = O.knn_offsets(xyz, offs, k, voxel, 2)
    gi, gd = fk.ops.knn_offsets(torch.from_numpy(xyz).to(DEV), torch.from_numpy(offs).to(DEV), k,
                                voxel, 2, validate=True)
    assert np.array_equal(gi.cpu().numpy(), oi)
    assert np.array_equal(gd.cpu().numpy().view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("spread", [0.02, 0.45])  # the filter keeps most records / few
@pytest.mark.parametrize("extra", [1, 31, 32, 33, 447, 448, 449, 480, 1000])
@pytest.mark.parametrize("k", [4, 16])
def test_filter_steps(k, extra, spread):
    """One cell of 3k points and a neighbour with the rest of 448 + extra: the
    first run ends the scan's first phase, the second goes through the filter."""
    rng = np.random.default_rng(extra)
    own = rng.random((3 * k, 3)) * spread + 0.5
    rest = rng.random((448 + extra - 3 * k, 3)) * spread + np.array([1.0, 0.5, 0.5])
    xyz = np.ascontiguousarray(np.concatenate([own, rest]), dtype=np.float32)
    rng.shuffle(xyz)
    _check(xyz, k, 0.25)


@pytest.mark.parametrize("dense,side", [(0.0, 7), (0.5, 24), (0.05, 30)])
def test_item_sizes_in_large_problems(dense, side):
    """From a full item's worth of queries per resident warp up, items shrink
    by the group's share of the whole work: points of one density, half of them
    in a dense ball, a few dense cells.  Self, general and selected queries."""
    import flashknn_exprepo_b200 as fk
    rng = np.random.default_rng(side)
    n, k, voxel = 100003, 8, 0.25 / side
    xyz = rng.random((n, 3), dtype=np.float32)
    if dense:
        hot = rng.choice(n, int(dense * n), replace=False)
        xyz[hot] = np.float32(0.4) + xyz[hot] * np.float32(2.4 / side)
    offs = np.array([n])
    oi, od = O.knn_offsets(xyz, offs, k, voxel, 2)
    x, o = torch.from_numpy(xyz).to(DEV), torch.from_numpy(offs).to(DEV)
    gi, gd = fk.ops.knn_offsets(x, o, k, voxel, 2, validate=True)
    assert np.array_equal(gi.cpu().numpy(), oi)
    assert np.array_equal(gd.cpu().numpy().view(np.uint32), od.view(np.uint32))
    order = torch.from_numpy(rng.permutation(n)).to(DEV)
    qi, qd = fk.ops.knn_offsets(x, o, k, voxel, 2, x[order].contiguous(), o, validate=True)
    inv = float(np.float32(1.0) / np.float32(voxel))
    grid = torch.floor(x * inv).long()
    si, sd = fk.ops.knn_grid(x, grid, None, k, 2, query_indices=order, idx_dtype=torch.int32,
                             validate=True)
    found = torch.isfinite(gd[order])
    assert torch.equal(qd, gd[order]) and torch.equal(sd, gd[order])
    assert torch.equal(si, gi[order]) and torch.equal(qi[found], gi[order][found])
