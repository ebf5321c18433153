"""The pruned k-means against the direct nearest-centroid kernel (bit-exact assignments) and a
float64 mean of the assigned points, at tile edges, with ties, and for data of any scale."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(n, kind):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 4)).astype(np.float32) * 0.25
    if kind == "ties":                                 # a coarse grid: many points exactly between centroids
        x = np.round(x * 8) / 8
    if kind == "large":
        x *= 3000.0
    if kind == "equal":
        x[:] = x[0]
    if kind == "narrow":                               # everything within a hundredth of the bound
        x *= 0.01
        x[0] = 1.0
    return torch.from_numpy(x.astype(np.float32)).cuda()


@pytest.mark.parametrize("n,kind", [(256, "plain"), (257, "ties"), (383, "plain"), (20000, "ties"), (300001, "plain"),
                                    (300001, "large"), (1100001, "equal"), (64, "plain"), (1, "plain"), (100003, "narrow"), (6000000, "plain")])
def test_kmeans_iterations(n, kind):
    from shard_b200 import ops
    x = _data(n, kind)
    cent = x[torch.arange(256, device="cuda") * n // 256].clone()
    if kind == "ties":
        cent[100:110] = cent[5:15]                     # duplicates: the first of equals wins
    for its in (1, 3):
        before = cent.clone()
        if its > 1:
            ops.kmeans_lloyd(x, before, its - 1)
        c = cent.clone()
        idx = ops.kmeans_lloyd(x, c, its)
        want, _ = ops.vq_assign(x, before, want_i64=False)
        assert torch.equal(idx, want)
        xi, ii = x.double().cpu().numpy(), idx.long().cpu().numpy()
        counts = np.bincount(ii, minlength=256)
        mean = np.stack([np.bincount(ii, xi[:, k], 256) for k in range(4)], 1) / np.maximum(counts, 1)[:, None]
        mean[counts == 0] = before.double().cpu().numpy()[counts == 0]
        assert np.abs(c.double().cpu().numpy() - mean).max() <= 2e-7 * float(x.abs().max())
        c2 = cent.clone()
        assert torch.equal(ops.kmeans_lloyd(x, c2, its), idx) and torch.equal(c2, c)


def test_kmeans_stops_when_settled():
    from shard_b200 import ops
    x = _data(256, "plain").repeat(8, 1)
    c = x[:256].clone()
    idx = ops.kmeans_lloyd(x, c, 30)
    assert (c - x[:256]).abs().max() < 2e-9 and torch.equal(idx, ops.vq_assign(x, c, want_i64=False)[0])


def test_kmeans_sets_side_by_side():
    from shard_b200 import ops
    x = torch.stack([_data(70001, k) for k in ("plain", "narrow", "ties")]) * torch.tensor([1.0, 0.5, 0.25], device="cuda").view(3, 1, 1)
    cent = x[:, 1000:1256].contiguous()
    together = cent.clone()
    idx = ops.kmeans_lloyd(x, together, 8, 4.0)
    for i in range(3):
        alone = cent[i].clone()
        assert torch.equal(idx[i], ops.kmeans_lloyd(x[i], alone, 8, 4.0)) and torch.equal(alone, together[i])


@pytest.mark.parametrize("max_abs", [0.0, 4.0])
@pytest.mark.parametrize("odd", [{7: float("inf")}, {7: float("nan"), 9000: float("-inf")}, {0: float("inf"), 63: float("-inf"), 64: float("nan")}])
def test_kmeans_of_points_that_are_not_finite(odd, max_abs):
    """They go to centroid 0 and take it with them, channel by channel; the others are clustered as ever."""
    from shard_b200 import ops
    x = _data(20000, "plain")
    for j, (i, v) in enumerate(odd.items()):
        x[i, (j + 1) % 4] = v
        x[i, (j + 3) % 4] *= 0.5
    cent = x[torch.arange(256, device="cuda") * 78 + 1].clone()
    cent[0] = 0.01
    c = cent.clone()
    idx = ops.kmeans_lloyd(x, c, 9, max_abs)
    want, u8 = cent.clone(), None
    for it in range(9):
        u8, _ = ops.vq_assign(x, want, want_i64=False)
        counts = torch.bincount(u8.long(), minlength=256)
        sums = torch.zeros(256, 4, dtype=torch.float64, device="cuda").index_add_(0, u8.long(), x.double())
        want = torch.where(counts[:, None] > 0, sums / counts[:, None], want.double()).float()
    assert torch.equal(idx, u8) and all(int(idx[i]) == 0 for i in odd)
    assert torch.equal(torch.isfinite(c), torch.isfinite(want)) and not torch.isfinite(c[0]).all()
    assert torch.allclose(c, want, rtol=0, atol=2e-6, equal_nan=True)
