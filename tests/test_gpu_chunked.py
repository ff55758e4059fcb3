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
