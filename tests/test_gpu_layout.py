"""Cells laid out by one atomic per CTA and items placed by another, where the
pieces meet: cell counts around a CTA's share, runs of items that must not
span a gap between two CTAs' records, many clouds (the key layout read by
every CTA up to 1,024 of them, by one kernel beyond) -- bit-exact against the
oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _points(rng, cells):
    """One to three points in each of `cells` voxels of 1 in a slab."""
    w = int(np.ceil(np.sqrt(cells)))
    at = np.stack(np.meshgrid(np.arange(w), np.arange(w), indexing="ij"), -1).reshape(-1, 2)[:cells]
    reps = rng.integers(1, 4, cells)
    xy = np.repeat(at, reps, 0) + rng.random((reps.sum(), 2))
    xyz = np.concatenate([xy, rng.random((len(xy), 1))], 1).astype(np.float32)
    rng.shuffle(xyz)
    return np.ascontiguousarray(xyz)


def _check(xyz, offs, k, new=None, new_offs=None):
    import flashknn_exprepo_b200 as fk
    oi, od = O.knn_offsets(xyz, offs, k, 0.25, 2, new, new_offs)
    to = lambda a: None if a is None else torch.from_numpy(a).to(DEV)
    gi, gd = fk.ops.knn_offsets(to(xyz), to(offs), k, 0.25, 2, to(new), to(new_offs),
                                validate=True)
    assert np.array_equal(gi.cpu().numpy(), oi)
    assert np.array_equal(gd.cpu().numpy().view(np.uint32), od.view(np.uint32))


@pytest.mark.parametrize("cells", [1, 255, 256, 257, 1023, 2049, 40000])
def test_cell_counts_around_a_share(cells):
    rng = np.random.default_rng(cells)
    xyz = _points(rng, cells)
    new = _points(rng, max(1, cells // 2))
    _check(xyz, np.array([len(xyz)]), 8)
    _check(xyz, np.array([len(xyz)]), 3, new, np.array([len(new)]))


@pytest.mark.parametrize("clouds", [1023, 1024, 1025, 3000])
def test_many_clouds(clouds):
    rng = np.random.default_rng(clouds)
    counts = rng.integers(1, 20, clouds)
    xyz = (rng.random((counts.sum(), 3)) * rng.choice([1, 1, 1, 9], counts.sum())[:, None])
    _check(np.ascontiguousarray(xyz, dtype=np.float32), np.cumsum(counts).astype(np.int64), 4)


@pytest.mark.parametrize("queries", [1, 63, 64, 65, 95, 96, 2000, 12001, 50000])
def test_groups_of_many_queries(queries):
    """A query cell that fills several items by itself, beside cells that share
    items: the line at two items, remainders, item sizes from 4 to 32."""
    rng = np.random.default_rng(queries)
    xyz = _points(rng, 60)
    many = np.concatenate([rng.random((queries, 3)), _points(rng, 30)]).astype(np.float32)
    rng.shuffle(many)
    _check(xyz, np.array([len(xyz)]), 5, np.ascontiguousarray(many), np.array([len(many)]))


@pytest.mark.parametrize("n", [1, 31, 300, 5000])
def test_few_points_with_ids_up_to_their_bound(n):
    """Cloud ids that come with the points are bounded by 32,768 however few
    the points: every box is emptied, also after a call that filled them."""
    import flashknn_exprepo_b200 as fk
    rng = np.random.default_rng(n)
    for ids in (np.arange(32768), rng.choice([0, 1, 1023, 1024, 20000, 32767], n)):
        m = len(ids)
        grid = rng.integers(-40, 40, (m, 3)).astype(np.int64)
        xyz = (grid + rng.random((m, 3))).astype(np.float32)
        order = np.argsort(ids, kind="stable")
        clouds = np.cumsum(np.bincount(ids, minlength=32768)).astype(np.int64)
        oi, od = O.knn_offsets(xyz[order], clouds, 4, 1.0, 3)
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
        gi, gd = fk.ops.knn_grid(to(xyz), to(np.floor(xyz).astype(np.int64)),
                                 to(ids.astype(np.int64)), 4, 3, validate=True)
        dist = gd.cpu().numpy()[order]
        assert np.array_equal(dist.view(np.uint32), od.view(np.uint32))
        rank = np.empty(m, np.int64)
        rank[order] = np.arange(m)
        assert np.array_equal(rank[gi.cpu().numpy()[order]], oi)
