"""GPU parity of neighbour grouping (grouping / knn_query_and_group).

Forward: the gathered rows equal Pointcept's own grouping output exactly
(it is a copy plus one FP32 subtraction).  Backward: the hand-written
deterministic gradients equal torch autograd's (Pointcept fixtures) and an
FP64 restatement within 1e-5 relative, and are bitwise identical run to run.
"""
import os

import numpy as np
import pytest
import torch

from tests.conftest import GOLDEN
from tests.test_oracle_golden import grouping_cases, grouping_f64

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def fk():
    import flashknn_exprepo_b200 as fk
    from flashknn_exprepo_b200.build import build
    build()
    return fk


def T(a, grad=False):
    t = torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    return t.requires_grad_(True) if grad else t


def rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-30)


def run_case(fk, z):
    with_xyz, separate = bool(z["with_xyz"]), bool(z["separate"])
    feat, xyz = T(z["feat"], True), T(z["xyz"], with_xyz)
    new = T(z["new_xyz"], True) if separate else None
    out = fk.grouping(T(z["idx"]), feat, xyz, new, with_xyz=with_xyz)
    (out * T(z["grad_out"])).sum().backward()
    grads = {"feat": feat.grad.cpu().numpy()}
    if with_xyz:
        grads["xyz"] = xyz.grad.cpu().numpy()
        if separate:
            grads["new_xyz"] = new.grad.cpu().numpy()
    return out.detach().cpu().numpy(), grads


@pytest.mark.parametrize("case", grouping_cases())
def test_grouping_matches_pointcept(fk, case):
    z = np.load(os.path.join(GOLDEN, f"grouping_{case}.npz"))
    out, grads = run_case(fk, z)
    assert np.array_equal(out, z["ref_out"])
    _, want = grouping_f64(z)
    assert rel(grads["feat"], z["ref_grad_feat"]) <= 1e-5
    assert rel(grads["feat"], want["feat"]) <= 1e-5
    for key in ("xyz", "new_xyz"):
        if key in grads:
            assert rel(grads[key], want[key]) <= 1e-5
            assert rel(grads[key], z[f"ref_grad_{key}"]) <= 1e-5
    out2, grads2 = run_case(fk, z)                   # bitwise reproducible
    for key in grads:
        assert np.array_equal(grads[key].view(np.uint32), grads2[key].view(np.uint32))


def test_hub_points_long_segments(fk):
    rng = np.random.default_rng(9)
    n, m, k, c = 500, 400, 16, 20
    idx = rng.integers(0, n, (m, k)).astype(np.int32)
    idx[:, 0] = 7                                    # point 7: 400 entries
    idx[::2, 1] = 11                                 # point 11: 200 entries
    z = {"idx": idx, "feat": rng.standard_normal((n, c)).astype(np.float32),
         "xyz": rng.random((n, 3), dtype=np.float32),
         "new_xyz": rng.random((m, 3), dtype=np.float32),
         "grad_out": rng.standard_normal((m, k, c + 3)).astype(np.float32),
         "with_xyz": np.bool_(True), "separate": np.bool_(True)}
    out, grads = run_case(fk, z)
    ref_out, want = grouping_f64(z)
    assert np.array_equal(out, ref_out.astype(np.float32))
    for key in ("feat", "xyz", "new_xyz"):
        assert rel(grads[key], want[key]) <= 1e-5


def test_knn_query_and_group_full_size(fk):
    from flashknn_exprepo_b200 import synthetic as S
    b = S.first_clouds(S.uneven_batch(), 6)
    xyz, offs = T(b.xyz), T(b.offsets)
    feat = torch.randn((len(b.xyz), 64), device=DEV)
    grouped, idx = fk.knn_query_and_group(feat, xyz, offs, nsample=16, with_xyz=True,
                                          voxel_size=S.C4_VOXEL)
    il = idx.long()
    want = torch.cat([xyz[il] - xyz[:, None, :], feat[il]], -1)
    assert torch.equal(grouped, want)
    plain, idx2 = fk.knn_query_and_group(feat, xyz, offs, idx=idx, with_xyz=False)
    assert torch.equal(plain, feat[il]) and idx2 is idx


@pytest.mark.parametrize("with_xyz", [False, True])
@pytest.mark.parametrize("m,k,c,shift", [
    (1, 1, 1, 0), (3, 5, 3, 0), (37, 16, 4, 0), (37, 16, 4, 1), (61, 33, 29, 0), (41, 7, 64, 0),
    (41, 7, 64, 1), (50, 8, 67, 0), (33, 3, 96, 0), (33, 3, 128, 0), (29, 9, 157, 0),
    (29, 9, 160, 0), (13, 5, 381, 0), (13, 5, 384, 0), (13, 5, 388, 0)])
def test_row_widths_and_alignments(fk, m, k, c, shift, with_xyz):
    """Every gather path (float4 rows, staged runs, row by row) at the edges
    of its widths, with feature rows off the 16-byte alignment (shift) and
    padding entries; gradients against FP64 sums of at most m*k FP32 terms."""
    rng = np.random.default_rng(m * 1000 + c)
    n = 53
    idx = rng.integers(-1, n, (m, k)).astype(np.int32)
    z = {"idx": idx, "feat": rng.standard_normal((n, c)).astype(np.float32),
         "xyz": rng.random((n, 3), dtype=np.float32),
         "new_xyz": rng.random((m, 3), dtype=np.float32),
         "grad_out": rng.standard_normal((m, k, c + 3 * with_xyz)).astype(np.float32),
         "with_xyz": np.bool_(with_xyz), "separate": np.bool_(True)}
    flat = torch.empty(n * c + shift, device=DEV)
    feat = flat[shift:].view(n, c)
    feat.copy_(T(z["feat"]))
    feat.requires_grad_(True)
    xyz, new = T(z["xyz"], True), T(z["new_xyz"], True)
    out = fk.grouping(T(idx), feat, xyz, new, with_xyz=with_xyz)
    want_out, want = grouping_f64(z)
    assert np.array_equal(out.detach().cpu().numpy(), want_out.astype(np.float32))
    out.backward(T(z["grad_out"]))
    got = {"feat": feat.grad, "xyz": xyz.grad, "new_xyz": new.grad}
    for key in ("feat",) + (("xyz", "new_xyz") if with_xyz else ()):
        assert rel(got[key].cpu().numpy(), want[key]) <= 1e-5


@pytest.mark.parametrize("with_xyz", [False, True])
@pytest.mark.parametrize("m,k", [(1365, 3), (256, 16), (8192, 8), (65535, 1)])
@pytest.mark.parametrize("c,shift", [(12, 0), (16, 0), (16, 1), (56, 0), (57, 0), (57, 1), (157, 0),
                                     (160, 0), (381, 0), (384, 0), (385, 0)])
def test_gather_paths_by_width_and_rows(fk, m, k, c, shift, with_xyz):
    """The gather's paths on both sides of their lines (16 channels and 4,096
    rows, 57 channels and 65,536 rows, runs of 8 and 4 rows, none)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(c + m)
    n = 1000
    idx = torch.randint(-1, n, (m, k), generator=gen, device=DEV, dtype=torch.int32)
    feat = torch.randn(n * c + shift, generator=gen, device=DEV)[shift:].view(n, c)
    xyz = torch.rand((n, 3), generator=gen, device=DEV)
    new = torch.rand((m, 3), generator=gen, device=DEV)
    il = idx.long()
    want = feat[il]
    if with_xyz:
        want = torch.cat([xyz[il] - new[:, None, :], want], -1)
    want = torch.where((il >= 0)[..., None], want, torch.zeros_like(want))
    got = fk.ops.group_features(feat, idx, xyz, new, with_xyz=with_xyz, validate=True)
    assert torch.equal(got, want)


def test_gather_of_more_than_2_31_words(fk):
    """Narrow rows are gathered in slabs of fewer than 2^31 words: the rows
    around the line between two slabs, inside one query's run, and the last."""
    m, k, c, n = 14_000_001, 3, 50, 997
    gen = torch.Generator(device=DEV)
    gen.manual_seed(3)
    idx = torch.randint(-1, n, (m, k), generator=gen, device=DEV, dtype=torch.int32)
    feat = torch.randn((n, c), generator=gen, device=DEV)
    xyz = torch.rand((n, 3), generator=gen, device=DEV)
    new = torch.rand((m, 3), generator=gen, device=DEV)
    out = fk.ops.group_features(feat, idx, xyz, new, with_xyz=True, validate=True)
    line = (2 ** 31 - 1) // (c + 3) // k
    for q in (slice(0, 1000), slice(line - 1000, line + 1000), slice(m - 1000, m)):
        il = idx[q].long()
        want = torch.cat([xyz[il] - new[q, None, :], feat[il]], -1)
        assert torch.equal(out[q], torch.where((il >= 0)[..., None], want, torch.zeros_like(want)))


@pytest.mark.parametrize("c,with_xyz", [(3, False), (16, False), (29, True), (64, False),
                                        (61, True), (100, False), (93, True), (131, False)])
def test_backward_adds_rows_in_entry_order(fk, c, with_xyz):
    """Segment lengths on both sides of a warp's 32 entries and of the long
    segments' passes (two entries each, 256 loaded at a time), odd and even,
    every column split: the FP32 sums in ascending entry order, bit for bit."""
    lens = [0, 1, 3, 4, 5, 7, 8, 9, 31, 32, 33, 34, 63, 64, 65, 224, 225, 255, 256, 257, 300, 513]
    rng = np.random.default_rng(c)
    idx = np.concatenate([np.full(q, t, np.int32) for t, q in enumerate(lens)] +
                         [np.full(40, -1, np.int32)])
    rng.shuffle(idx)
    off = 3 if with_xyz else 0
    grad = rng.standard_normal((len(idx), 1, c + off)).astype(np.float32)
    want = np.zeros((len(lens), c + off), np.float32)
    for e, t in enumerate(idx):
        if t >= 0:
            want[t] += grad[e, 0]
    n = len(lens)
    feat = torch.empty((n, c), device=DEV)
    xyz = torch.empty((n, 3), device=DEV) if with_xyz else None
    fk.ops.group_backward(T(grad), T(idx[:, None]), n, c, with_xyz, feat, xyz)
    assert np.array_equal(feat.cpu().numpy(), want[:, off:])
    if with_xyz:
        assert np.array_equal(xyz.cpu().numpy(), want[:, :3])
