"""The eigensolver of the PCA fit against float64 `torch.linalg.eigh`."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(p, kind, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "rank192":                              # keys of the configurations: 192 strong directions, the rest noise
        x = torch.randn(2000, 192, generator=g, device="cuda") @ torch.randn(192, p, generator=g, device="cuda") / 14
        x += 0.01 * torch.randn(2000, p, generator=g, device="cuda")
    elif kind == "decay":                              # a spectrum without a gap
        x = torch.randn(3000, p, generator=g, device="cuda") * torch.exp(-0.02 * torch.arange(p, device="cuda"))
        x = x @ torch.linalg.qr(torch.randn(p, p, generator=g, device="cuda"))[0]
    else:                                              # fewer samples than dimensions
        x = torch.randn(150, p, generator=g, device="cuda")
    return (x.T @ x).contiguous()


@pytest.mark.parametrize("p,rank,kind,count", [(128, 128, "decay", 1), (256, 192, "rank192", 3), (384, 100, "decay", 2),
                                               (512, 192, "rank192", 2), (640, 192, "decay", 1), (768, 7, "rank192", 1),
                                               (896, 192, "decay", 1), (1024, 192, "rank192", 10), (1024, 192, "decay", 2),
                                               (1024, 149, "few", 1), (1024, 1, "decay", 1)])
def test_eigh_top(p, rank, kind, count):
    from shard_b200 import ops
    a = torch.stack([_matrix(p, kind, s) for s in range(count)])
    basis, eig, flag = ops.eigh_top(a, rank)
    assert int(flag.sum()) == 0
    want = torch.linalg.eigvalsh(a.double()).flip(-1)[:, :rank]
    top = want[:, :1]
    assert ((eig.double() - want).abs() / top).max() < 2e-6
    b = basis.double()
    assert (b.transpose(1, 2) @ b - torch.eye(rank, device="cuda")).abs().max() < 2e-5
    res = a.double() @ b - b * eig.double().unsqueeze(1)
    assert (res.norm(dim=1) / top).max() < 3e-6


def test_eigh_top_reports_what_it_cannot_do():
    from shard_b200 import ops
    a = torch.eye(256, device="cuda").unsqueeze(0).repeat(2, 1, 1)       # all eigenvalues equal
    a[1] = _matrix(256, "decay", 1)
    a[0, 3, 3] = float("nan")
    _, _, flag = ops.eigh_top(a, 64)
    assert flag.tolist() == [1, 0]


@pytest.mark.parametrize("sizes", [((128, 9), (256, 9)), ((384, 8), (640, 8)), ((1024, 7), (128, 12))])
def test_launches_on_two_streams(sizes):
    """More clusters than fit the GPU, of two sizes at once (smaller matrices need fewer registers: without the
    reserved shared memory their CTAs could share SMs): every result is the one of a launch alone."""
    from shard_b200 import ops
    a = [torch.stack([_matrix(p, "decay", s) for s in range(count)]) for p, count in sizes]
    want = [ops.eigh_top(m, 64) for m in a]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in a]
    for _ in range(3):
        got = []
        for m, st in zip(a, streams):
            with torch.cuda.stream(st):
                got.append(ops.eigh_top(m, 64))
        torch.cuda.synchronize()
        for w, g in zip(want, got):
            assert int(g[2].sum()) == 0 and all(torch.equal(x, y) for x, y in zip(w, g))
