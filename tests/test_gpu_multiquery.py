"""Attention of several new tokens over a compressed layer (one launch for all of them) against float64
attention over the layer's read-back, at the edges of query and key tiles, in both append modes."""
import pytest
import torch

from gpu_helpers import random_gc
from test_gpu_readback import _cache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_comp,rank,nkv,before,s,streaming", [
    (1, 32, 1, 0, 3, True), (128, 192, 8, 2, 4, False), (129, 150, 2, 70, 31, True), (700, 192, 8, 5, 32, True),
    (2000, 192, 4, 60, 33, False), (5000, 192, 8, 0, 200, True), (300, 64, 8, 1, 256, False), (9001, 192, 8, 9, 7, True)])
def test_multiquery(n_comp, rank, nkv, before, s, streaming):
    from shard_b200 import fused_attention_compressed
    gc_np = random_gc(n_comp, rank=rank, nkv=nkv, seed=s)
    cache, layer = _cache(gc_np, nkv, streaming, capacity=before + s)
    g = torch.Generator(device="cuda").manual_seed(s)
    k, v = (torch.randn(1, before + s, nkv, 128, generator=g, device="cuda").half().transpose(1, 2) for _ in range(2))
    q = torch.randn(1, s, 4 * nkv, 128, generator=g, device="cuda").half().transpose(1, 2)
    cache._fused_decode_update = True
    if before:
        layer.update(k[:, :, :before], v[:, :, :before])
    layer.update(k[:, :, before:], v[:, :, before:])
    cache._fused_decode_update = False
    out = fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq)
    cache.check()
    assert out.shape == (1, 4 * nkv, s, 128)
    layer._needs_decompress = True
    keys, values = layer.keys[0].double(), layer.values[0].double()
    n = keys.shape[1]
    sc = torch.einsum("hqd,hnd->hqn", q[0].double(), keys.repeat_interleave(4, 0)) / 128 ** 0.5
    # rows: sink, middle, window, then the tokens in order: the last s are the queries' own
    hidden = torch.arange(n, device="cuda")[None, :] > n - s + torch.arange(s, device="cuda")[:, None]
    want = torch.softmax(sc.masked_fill(hidden, float("-inf")), -1) @ values.repeat_interleave(4, 0)
    err = (out[0].double() - want).abs()
    assert (err <= 1.5e-3 + 5e-3 * want.abs()).all(), err.max()
    again = fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq, out=torch.empty_like(out).contiguous())
    assert torch.equal(again, out)


@pytest.mark.parametrize("s", [1, 2, 3, 40])
def test_queries_of_two_sequences_are_refused(s):
    from shard_b200 import fused_attention_compressed
    cache, layer = _cache(random_gc(200, nkv=2, seed=s), 2, True)
    cache._fused_decode_update = True
    new = torch.randn(1, 2, s, 128, device="cuda").half()
    layer.update(new, new)
    q = torch.randn(2, 8, s, 128, device="cuda").half()
    with pytest.raises(NotImplementedError):
        fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq)


@pytest.mark.parametrize("nkv,last", [(8, 25000), (4, 50000), (2, 90000), (1, 90000)])
@pytest.mark.parametrize("over", [0, 1])
def test_three_tokens_either_side_of_the_rule(nkv, last, over, monkeypatch):
    """The longest middle that is read back once, and one token more, which takes decode launches."""
    from shard_b200 import attention
    assert last == min(attention.THREE_TOKENS_MAX_MIDDLE, attention.THREE_TOKENS_MAX_PAIRS // nkv)
    real, calls = attention.ops.multiquery_attn, []
    monkeypatch.setattr(attention.ops, "multiquery_attn", lambda *a: (calls.append(1), real(*a))[1])
    test_multiquery(last + over, 192, nkv, 3, 3, True)
    assert len(calls) == (0 if over else 2)            # (the test attends twice)


@pytest.mark.parametrize("nkv,rows,s", [(4, 1400, 20), (8, 300, 3), (1, 77, 33)])
def test_rows_outside_the_middle_are_weighed_in_full(nkv, rows, s):
    """Where the decoded tokens carry the attention the output is float64's, rounded to fp16: their weights
    have 22 bits, so nothing but the rounding of the output (and a tenth of it) is left."""
    from shard_b200 import fused_attention_compressed
    gc_np = random_gc(1, nkv=nkv, seed=s)
    cache, layer = _cache(gc_np, nkv, False, capacity=rows + s)
    g = torch.Generator(device="cuda").manual_seed(s)
    k, v = (torch.randn(1, nkv, rows + s, 128, generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn(1, 4 * nkv, s, 128, generator=g, device="cuda").half()
    cache._fused_decode_update = True
    layer.update(k, v)
    out = fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq)[0].double()
    layer._needs_decompress = True
    keys, values = layer.keys[0].double(), layer.values[0].double()
    n = keys.shape[1]
    sc = torch.einsum("hqd,hnd->hqn", q[0].double(), keys.repeat_interleave(4, 0)) / 128 ** 0.5
    hidden = torch.arange(n, device="cuda")[None, :] > n - s + torch.arange(s, device="cuda")[:, None]
    want = torch.softmax(sc.masked_fill(hidden, float("-inf")), -1) @ values.repeat_interleave(4, 0)
    assert (out - want).norm() <= 1.1 * (want.half().double() - want).norm()
