"""Caller tables whose candidate counts overflow 32 bits: each run is a valid
range of the support, their sum is not.  Reported through the status word; the
context stays usable."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.mark.parametrize("n", [80_000_000, 160_000_000])
def test_candidate_sum_beyond_int32(n):
    """27 runs of the whole support: the sum wraps to a negative or a small
    positive number."""
    import flashknn_exprepo_b200 as fk
    xyz = torch.zeros((n, 3), device=DEV)
    queries = torch.zeros((64, 3), device=DEV)
    to = lambda a: torch.from_numpy(a).to(DEV)
    steps = to(np.array([0, n], np.int32))
    steps_query = to(np.array([0, 64], np.int32))
    neigh = torch.zeros((1, 27), dtype=torch.int32, device=DEV)
    cnt = to((np.arange(28, dtype=np.int64) * n).astype(np.uint32).view(np.int32)[None].copy())
    with pytest.raises(fk.FknnError, match="table"):
        fk.ops.general_query_tables(xyz, queries, steps, steps_query, neigh, cnt, 4, validate=True)
    small = torch.rand((100, 3), device=DEV)
    ends = torch.tensor([100], device=DEV)
    idx, _ = fk.ops.knn_offsets(small, ends, 1, 0.5, 2, validate=True)
    assert torch.equal(idx[:, 0], torch.arange(100, device=DEV, dtype=torch.int32))
