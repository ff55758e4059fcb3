"""The packed scan's 32-bit block selection where it can go wrong: distances
that differ only in the bits its keys drop, exact ties at the K-th place,
candidate counts around the block size, K below the list's capacity, both
position widths -- bit-exact against the oracle."""
import math

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _check(xyz, k, voxel, config=None, cut_r2=math.inf):
    import flashknn_exprepo_b200 as fk
    offs = np.array([len(xyz)])
    oi, od = O.knn_offsets(xyz, offs, k, voxel, 2, cut_r2=np.float32(cut_r2))
    gi, gd = fk.ops.knn_offsets(torch.from_numpy(xyz).to(DEV), torch.from_numpy(offs).to(DEV), k,
                                voxel, 2, cut_r2=cut_r2, config=config, validate=True)
    assert np.array_equal(gi.cpu().numpy(), oi)
    assert np.array_equal(gd.cpu().numpy().view(np.uint32), od.view(np.uint32))


def _lattice(side, jitter):
    """A shuffled unit lattice, every coordinate moved by up to `jitter`: the
    neighbours' distances fall into a few classes, equal (jitter 0) or apart
    by less than the keys resolve."""
    rng = np.random.default_rng(side)
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xyz = g.astype(np.float32) + np.float32(0.5)
    xyz = xyz + (rng.random(xyz.shape, dtype=np.float32) - np.float32(0.5)) * np.float32(2 * jitter)
    rng.shuffle(xyz)
    return np.ascontiguousarray(xyz, dtype=np.float32)


@pytest.mark.parametrize("jitter", [0.0, 2e-6, 2e-5, 1e-3])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 16, 17, 24, 32, 33, 64])
def test_distance_classes(k, jitter):
    _check(_lattice(17, jitter), k, 0.5)


@pytest.mark.parametrize("k", [8, 16, 32])
def test_wide_tile_positions(k):
    from flashknn_exprepo_b200 import _lib
    xyz = _lattice(17, 2e-5)
    for voxel in (0.5, 0.7):  # 216 and up to 729 candidates per cell neighbourhood
        _check(xyz, k, voxel, _lib.FknnConfig(2, 1024, 8, 0, 1))
        _check(xyz, k, voxel, _lib.FknnConfig(2, 512, 8, 0, 2))


@pytest.mark.parametrize("k", [1, 3, 5, 8, 16, 24])
def test_candidate_counts_around_a_block(k):
    """Cells far apart, each its own neighbourhood of 1..70 points, some of
    them duplicates."""
    rng = np.random.default_rng(k)
    parts = [rng.random((n, 3), dtype=np.float32) * np.float32(0.3) + np.float32(4 * n)
             for n in range(1, 71)]
    xyz = np.concatenate(parts)
    dup = rng.integers(0, len(xyz), len(xyz) // 4)
    xyz = np.ascontiguousarray(np.concatenate([xyz, xyz[dup]]))
    _check(xyz, k, 0.1)
    _check(xyz, k, 0.1, cut_r2=0.01)


@pytest.mark.parametrize("radius", [0.25, 99999.0, 100001.0, 4e5])
def test_ball_padding_on_both_sides_of_its_radius_rule(radius):
    import flashknn_exprepo_b200 as fk
    rng = np.random.default_rng(7)
    xyz = torch.from_numpy((rng.random((300, 3)) * 4 * radius).astype(np.float32)).to(DEV)
    offs = torch.tensor([300], device=DEV)
    idx, dist = fk.ball_query(24, radius, 0.0, xyz, offs)
    want_idx, d2 = fk.ops.ball_query_offsets(xyz, offs, 24, radius, radius / 4, 2, None, None)
    assert torch.equal(idx, want_idx) and bool((idx < 0).any()) and bool((idx >= 0).any())
    assert torch.equal(dist, torch.where(idx < 0, torch.full_like(d2, 1e5), torch.sqrt(d2)))


@pytest.mark.parametrize("copies", [31, 33, 70])
@pytest.mark.parametrize("k", [1, 5, 8, 16, 17, 32, 50, 64])
def test_many_equal_points(k, copies):
    """Points repeated more often than a test step holds positions: a class of
    equal distances spans several steps, some lanes' classes more than others'."""
    rng = np.random.default_rng(copies)
    base = np.stack(np.meshgrid(np.arange(9), np.arange(9), [0.0], indexing="ij"), -1)
    xyz = np.repeat((base.reshape(-1, 3) * 3.0 + 0.5).astype(np.float32), copies, 0)
    xyz[::7] += np.float32(1e-6)
    rng.shuffle(xyz)
    _check(np.ascontiguousarray(xyz), k, 0.5)
    _check(np.ascontiguousarray(xyz), k, 0.8)
