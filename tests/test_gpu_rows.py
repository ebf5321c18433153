"""Decode attention with few and with many rows outside the compressed middle (fp16 or streamed): pairs and
odd rows, all warps on the rows, more row CTAs than tiles, many partial results to merge, against float64 attention over the read-back."""
import pytest
import torch

from gpu_helpers import random_gc
from test_gpu_readback import _cache, middle_float64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_comp,nkv,rows,streaming", [
    (700, 8, 1, True), (700, 8, 2, False), (130, 8, 75, True), (130, 8, 76, False), (1, 2, 700, False), (1, 8, 901, True),
    (2560, 8, 1153, True), (2560, 8, 1100, False), (5000, 8, 3001, True), (300, 1, 4001, True),
    (4096, 1, 2, True), (4097, 1, 3, False), (18900, 1, 2, True), (8300, 2, 5, False)])   # 32, 33, 148 and 65 partial results to merge
def test_decode_rows(n_comp, nkv, rows, streaming):
    from shard_b200 import fused_attention_compressed
    cache, layer = _cache(random_gc(n_comp, nkv=nkv, seed=rows), nkv, streaming, capacity=rows + 4)
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda").half() for _ in range(2))
    cache._fused_decode_update = True
    if rows > 1:
        layer.update(k[:, :, :-1], v[:, :, :-1])
    for step in range(2):
        if step == 0:
            layer.update(k[:, :, -1:], v[:, :, -1:])       # the newest row is written by the decode launch
        q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
        out = fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq)
        cache.check()
        layer._needs_decompress = True
        keys, values = layer.keys[0].double(), layer.values[0].double()
        sc = torch.einsum("hqd,hnd->hqn", q[0].double(), keys.repeat_interleave(4, 0)) / 128 ** 0.5
        want = torch.softmax(sc, -1) @ values.repeat_interleave(4, 0)
        err = (out[0].double() - want).abs()
        assert (err <= 1.5e-3 + 5e-3 * want.abs()).all(), err.max()


@pytest.mark.parametrize("n_comp,nkv,rows,streaming,scale", [
    (300, 8, 15, True, 1.0), (300, 8, 16, True, 300.0), (300, 2, 17, True, 2e-3), (1, 1, 33, True, 300.0), (1500, 8, 1200, True, 300.0),
    (2304, 8, 4000, True, 1.0),    # all warps on the rows, behind a tile or two of their own
    (300, 8, 28, False, 300.0), (300, 2, 29, False, 2e-3), (1, 1, 13, False, 1.0), (1500, 8, 1200, False, 300.0)])
def test_row_blocks(n_comp, nkv, rows, streaming, scale):
    """The ends of the blocks of sixteen rows, in one block, several blocks of a warp and all warps, with values far from one (a streamed row's
    norm goes into its weight).  Bound: that of the other rows (fp16 rounding of values, weights and output), in units of the values;
    what the weights keep is measured by the tests of the launch's fp32 sums above."""
    from shard_b200 import fused_attention_compressed
    gc_np = random_gc(n_comp, nkv=nkv, seed=rows)
    cache, layer = _cache(gc_np, nkv, streaming, capacity=rows + 4)
    gc = layer._gpu_compressed
    for name in ("sink_v", "win_v", "v_ch_f16"):           # everything that is summed, on the rows' scale
        gc[name].mul_(scale if scale < 1 else 1.0)
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda") for _ in range(2))
    v *= scale * torch.exp2(torch.randint(-6, 1, (1, nkv, rows, 1), generator=g, device="cuda").float())
    cache._fused_decode_update = True
    layer.update(k.half(), v.half())
    q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
    out = fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq)
    cache.check()
    layer._needs_decompress = True
    keys, values = layer.keys[0].double(), layer.values[0].double()
    sc = torch.einsum("hqd,hnd->hqn", q[0].double(), keys.repeat_interleave(4, 0)) / 128 ** 0.5
    want = torch.softmax(sc, -1) @ values.repeat_interleave(4, 0)
    err = (out[0].double() - want).abs()
    assert (err <= 1.5e-3 * scale + 5e-3 * want.abs()).all(), (err / scale).max()


def rows_float64(layer, nkv):
    """Keys and values (nkv, rows, 128) of everything outside the middle, float64, streamed rows from their codes."""
    from shard_b200.streaming import get_codebook
    gc = layer._gpu_compressed
    keys, values = ([gc[s + x][0].double() for s in ("sink_", "win_")] for x in "kv")
    if "decode_k" in gc:
        keys.append(gc["decode_k"][0].double())
        values.append(gc["decode_v"][0].double())
    m = gc.get("stream_n", 0)
    if m:
        had = torch.ones(1, 1, dtype=torch.float64, device="cuda")
        for _ in range(7):
            had = torch.cat([torch.cat([had, had], 1), torch.cat([had, -had], 1)], 0)
        codebook = get_codebook(128, 8, torch.device("cuda", 0)).double()
        for x, out in (("k", keys), ("v", values)):
            e = codebook[gc[x + "_idx_buf"][:m].long()].view(m, nkv, 128) @ had / 128 ** 0.5
            out.append((e * gc["signs"].double() * gc[x + "_norm_buf"][:m].view(m, nkv, 1).double()).transpose(0, 1))
    return torch.cat(keys, 1), torch.cat(values, 1)


def attend_float64(q, keys, values):
    sc = torch.einsum("hgd,hnd->hgn", q.double().view(keys.shape[0], 4, 128), keys) / 128 ** 0.5
    return (torch.softmax(sc, -1) @ values).view(-1, 128)


def rows_layer(nkv, streaming, k, v, seed):
    """A layer whose middle is one token without a value, and its keys and values in float64 (the token's key in fp16 terms: its weight
    is that of one row, in the sum of the weights alone)."""
    gc_np = random_gc(1, nkv=nkv, seed=seed)
    cache, layer = _cache(gc_np, nkv, streaming, capacity=k.shape[2] + 4)
    layer._gpu_compressed["v_ch_f16"].zero_()
    cache._fused_decode_update = True
    layer.update(k, v)
    middle = torch.from_numpy(middle_float64(gc_np, nkv)[0]).cuda()
    keys, values = rows_float64(layer, nkv)
    return cache, layer, torch.cat([middle, keys], 1), torch.cat([0 * middle, values], 1)


def partial_attention(cache, layer, q):
    """The launch's fp32 sums, divided: what it has before it rounds to fp16."""
    from shard_b200.attention import decode_layer
    rec = decode_layer(q, layer, layer.get_seq_length() - 1, partial_out=True)
    cache.check()
    return rec[:, 4:].double() / rec[:, 1:2].double()


@pytest.mark.parametrize("streaming", [True, False])
def test_queries_beyond_the_range_of_fp16_in_code_space(streaming):
    """A query whose coordinate in the stream's code space is 67 882 (128 channels of 6000 with the transform's signs), one of 1e-3 and an
    all-zero one beside it: every coordinate is finite, and so is the attention."""
    nkv, rows = 2, 40
    g = torch.Generator(device="cuda").manual_seed(1)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda").half() * s for s in (0.01, 1.0))
    from shard_b200.streaming import stream_signs
    signs = stream_signs(0, 128, torch.device("cuda")).half()
    k[:, :, 7] = 0.5 * signs
    cache, layer, keys, values = rows_layer(nkv, streaming, k, v, 1)
    q = torch.stack([6000 * signs, 1e-3 * signs, 0 * signs, signs] * nkv).view(1, 4 * nkv, 1, 128)
    got = partial_attention(cache, layer, q)
    want = attend_float64(q, keys, values)
    # bound: the weights' (two roundings to 2**-22, scores of up to 30 in fp32) and the fp32 sums'; the token's key is an fp16 product
    assert ((got - want).norm(dim=1) <= 2e-5 * want.norm(dim=1)).all(), ((got - want).norm(dim=1) / want.norm(dim=1)).max()


# What 32-bit arithmetic leaves: a score of up to 24 in the log2 domain with three roundings at its full size (3 . 24 . 2**-24 . ln 2 = 3e-6 of
# a weight), ex2 and the fp32 sums; the middle's token, whose key is an fp16 product, has 1e-3 of its weight in 85 (8, 16) to 4069 rows'.
# A part dropped anywhere leaves 11 bits, 2e-4; second parts in fp16's subnormals 2e-5 and more where small weights carry the result.
ROWS_REL = 4e-6


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("nkv,rows", [(8, 16), (2, 333), (8, 1200), (1, 4000)])
def test_rows_are_weighed_in_full(nkv, rows, streaming):
    """Even attention over the rows: the launch's fp32 sums are float64's to the precision of 32-bit arithmetic."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda").half() for _ in range(2))
    cache, layer, keys, values = rows_layer(nkv, streaming, k, v, rows)
    q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
    got, want = partial_attention(cache, layer, q), attend_float64(q, keys, values)
    err = (got - want).norm() / want.norm()
    assert err <= ROWS_REL, err


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("nkv,rows,power", [(8, 40, 12), (2, 333, 20), (8, 1200, 16), (1, 4000, 24)])
def test_rows_of_small_weight_and_large_values(nkv, rows, power, streaming):
    """One row has nearly all of the attention and a value of nearly nothing; the result is made of the others, whose weights are about
    2**-power of its."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    base = torch.randn(nkv, 1, 128, generator=g, device="cuda")
    base *= 128 ** 0.5 / base.norm(dim=-1, keepdim=True)
    q = (base + 0.05 * torch.randn(nkv, 4, 128, generator=g, device="cuda")).half().view(1, 4 * nkv, 1, 128)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda") for _ in range(2))
    v *= 2.0 ** min(power - 8, 8)
    k[:, :, rows // 3] = base[:, 0] * (power * 0.6931 / 128 ** 0.5)
    v[:, :, rows // 3] = 2.0 ** -12
    cache, layer, keys, values = rows_layer(nkv, streaming, k.half(), v.half(), rows)
    got, want = partial_attention(cache, layer, q), attend_float64(q, keys, values)
    small = values.clone()
    small[:, 69 + rows // 3] = 0
    assert attend_float64(q, keys, small).norm() > 0.9 * want.norm()
    err = (got - want).norm() / want.norm()
    assert err <= ROWS_REL, err


@pytest.mark.parametrize("n_comp,rows", [(1, 901), (130, 75), (2304, 300), (4608, 40), (9000, 700), (11520, 2000)])   # 0 to 5 tiles a CTA
def test_codes_are_looked_up_in_this_launch_s_codebook(n_comp, rows):
    """Plain launches out of a cold L2, each behind one that left another codebook's tables in the same shared memory: a look-up that
    does not wait for the tables finds entries of the wrong sign."""
    from shard_b200 import ops
    from shard_b200.attention import decode_layer
    from shard_b200.streaming import get_codebook
    nkv = 8
    cache, layer = _cache(random_gc(n_comp, nkv=nkv, seed=rows), nkv, True, capacity=rows)
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn(1, nkv, rows, 128, generator=g, device="cuda").half() for _ in range(2))
    cache._fused_decode_update = True
    layer.update(k, v)
    q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
    first = decode_layer(q, layer, layer.get_seq_length() - 1).clone()
    layer._needs_decompress = True
    keys, values = layer.keys[0].double(), layer.values[0].double()
    sc = torch.einsum("hqd,hnd->hqn", q[0].double(), keys.repeat_interleave(4, 0)) / 128 ** 0.5
    want = (torch.softmax(sc, -1) @ values.repeat_interleave(4, 0))[:, 0]
    assert ((first - want).abs() <= 1.5e-3 + 5e-3 * want.abs()).all()
    ls, out, other = layer._gpu_compressed["_launch"], torch.empty_like(first), torch.empty_like(first)
    right = get_codebook(128, 8, torch.device("cuda", 0))
    wrong, flush = -right, torch.empty(1 << 26, device="cuda")
    ls.shape.no_overlap = 1
    for _ in range(10):
        for codebook, dst in ((wrong, other), (right, out)):
            flush.zero_()
            ls.seq.out = dst.data_ptr()
            ops.decode_attn(ls.seq, 1, ls.shape, ls.inv_ptr, codebook, cache._decode_ws)
        assert torch.equal(out, first) and not torch.equal(other, first)
    cache.check()


@pytest.mark.parametrize("n_comp", [300, 9000])
def test_channel_scales_from_the_launch_in_front(n_comp):
    """The channel scales may be written by a launch that lets its successors start early (here a decode launch's output): they are not
    among the tensors that are read ahead of it."""
    from shard_b200 import ops
    from shard_b200.attention import decode_layer
    nkv = 8
    layers = [_cache(random_gc(n, nkv=nkv, seed=n), nkv, False) for n in (20000, n_comp)]
    g = torch.Generator(device="cuda").manual_seed(n_comp)
    q = [torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half() for _ in range(5)]
    scales = torch.empty(4 * nkv, 128, dtype=torch.float16, device="cuda")
    (front_cache, front), (cache, layer) = layers
    decode_layer(q[0], front, 30000, out=scales)
    decode_layer(q[0], layer, 30000)
    ls = layer._gpu_compressed["_launch"]
    ls.seq.v_ch, ls.seq.q, ls.shape.no_overlap = scales.data_ptr(), q[0].data_ptr(), 0

    def launch():
        out = torch.empty(4 * nkv, 128, dtype=torch.float16, device="cuda")
        ls.seq.out = out.data_ptr()
        ops.decode_attn(ls.seq, 1, ls.shape, ls.inv_ptr, None, cache._decode_ws)
        return out

    for x in q:
        scales.fill_(7.0)
        decode_layer(x, front, 30000, out=scales)
        got = launch()
        torch.cuda.synchronize()
        assert torch.equal(got, launch())
    cache.check()
    front_cache.check()


@pytest.mark.parametrize("streaming", [True, False])
def test_rows_between_16_byte_boundaries(streaming):
    """Rows that start 8 bytes (fp16) or 4 bytes (codes) behind a 16-byte boundary are read in pieces: the same result to the bit."""
    from shard_b200 import fused_attention_compressed

    def shifted(x, by):
        room = torch.zeros(x.numel() + 64, dtype=x.dtype, device=x.device)
        y = room[by:by + x.numel()].view(x.shape)
        y.copy_(x)
        return y

    outs = []
    g = torch.Generator(device="cuda").manual_seed(3)
    k, v, q = (torch.randn(1, h, n, 128, generator=g, device="cuda").half() for h, n in ((2, 45), (2, 45), (8, 1)))
    for shift in (False, True):
        cache, layer = _cache(random_gc(300, nkv=2, seed=9), 2, streaming, capacity=64)
        gc = layer._gpu_compressed
        cache._fused_decode_update = True
        layer.update(k, v)
        if shift:
            for name in ("sink_k", "sink_v", "win_k", "win_v"):
                gc[name] = shifted(gc[name], 4)
            for name in ("k_idx_buf", "v_idx_buf") if streaming else ():
                gc[name] = shifted(gc[name], 4)
            gc.pop("_launch", None)
            gc.pop("_native", None)
        outs.append(fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq))
        cache.check()
        if shift:
            assert gc["sink_k"].data_ptr() % 16 == 8 and (not streaming or gc["k_idx_buf"].data_ptr() % 16 == 4)
    assert torch.equal(*outs)


@pytest.mark.parametrize("n_comp,nkv", [(700, 8), (0, 2)])
def test_decode_launch_writes_the_newest_fp16_row(n_comp, nkv):
    """`append = 2` of the C entry point: the launch copies new_k / new_v into the last row, then attends."""
    from shard_b200 import ops
    from shard_b200.attention import decode_layer
    cache, layer = _cache(random_gc(max(n_comp, 1), nkv=nkv, seed=5), nkv, False, capacity=16)
    g = torch.Generator(device="cuda").manual_seed(5)
    k, v = (torch.randn(1, nkv, 9, 128, generator=g, device="cuda").half() for _ in range(2))
    layer._fp16_append(k, v)
    q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
    tok = (0, n_comp)
    want = decode_layer(q, layer, 800, tok_range=tok).clone()
    gc, out = layer._gpu_compressed, torch.empty(4 * nkv, 128, dtype=torch.float16, device="cuda")
    for name in ("decode_k", "decode_v"):
        gc[name][:, :, -1:].zero_()
    last = [x[0, :, -1].contiguous() for x in (k, v)]
    ls = gc["_launch"]
    ls.seq.new_k, ls.seq.new_v, ls.seq.out, ls.shape.append = last[0].data_ptr(), last[1].data_ptr(), out.data_ptr(), 2
    ops.decode_attn(ls.seq, 1, ls.shape, ls.inv_ptr, None, cache._decode_ws)
    assert torch.equal(out, want) and torch.equal(gc["decode_k"], k) and torch.equal(gc["decode_v"], v)


@pytest.mark.parametrize("n", [65535, 65536, 70001])
def test_many_tokens_in_one_append(n):
    """A turn of more tokens than a grid has rows: the codes are those of the same tokens appended in parts."""
    cache, layer = _cache(random_gc(1, nkv=2, seed=5), 2, True, capacity=16)
    other, ref = _cache(random_gc(1, nkv=2, seed=5), 2, True, capacity=n)
    g = torch.Generator(device="cuda").manual_seed(n)
    k, v = (torch.randn(1, 2, n, 128, generator=g, device="cuda").half() for _ in range(2))
    cache._fused_decode_update = other._fused_decode_update = True
    layer.update(k, v)
    for i in range(0, n, 9000):
        ref.update(k[:, :, i:i + 9000], v[:, :, i:i + 9000])
    assert layer.get_seq_length() == ref.get_seq_length()
    for name in ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf"):
        assert torch.equal(layer._gpu_compressed[name][:n], ref._gpu_compressed[name][:n])
