"""The work a user of this package has it do, as cases that can be timed.

A model's decoder calls the cache layer by layer: `update` with the layer's new keys and values, then
either the fused attention (`fused_attention_compressed`, what the Llama hook does) or stock attention
over the keys and values that `update` returned (any other model).  The cases are passes of exactly
those calls over the layers of one cache, plus `BatchedDecoder.step` for many sequences and the prefill
compression.  Geometry: head_dim 128 and 4 query heads per KV head; 8 KV heads are a whole model, 4 and
2 a tensor-parallel share of one.

A pass over a decode state generates the next token of a reply: after `WINDOW` tokens the reply starts
over from the same prefix, as when several replies to one prompt are drawn.  So every pass has its own
query position and its own row of the stream, and the amount of work stays the case's.
"""
import math

import torch

from shard_b200 import Cache, fused_attention_compressed
from shard_b200.cache import attach_kernel_format
from shard_b200.parallel import BatchedDecoder

HD = 128
GQA = 4
SINK, WINDOW_TOKENS = 4, 64          # fp16 tokens the cache keeps at both ends of the prompt (its defaults)
WINDOW = 16                          # tokens of a reply before it starts over
MAX_OUTPUTS = 60


def _case(kind, ctx, layers, *, name=None, nkv=8, rank=192, mode="stream", decoded=1, new=1, seqs=1):
    c = {"kind": kind, "ctx": ctx, "layers": layers, "nkv": nkv, "rank": rank, "mode": mode, "decoded": decoded,
         "new": new, "seqs": seqs}
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # one layer of a 2048-token prompt, start of the reply: the smallest call there is, launch and
        # host latency count
        _case("decode", 2048, 1, name="decode_2k_one_layer", decoded=3),
        # the everyday request: an 8K prompt, a hundred-odd tokens into the reply, 8-bit stream
        _case("decode", 8192, 12, name="decode_8k", decoded=120),
        # the headline: 32K tokens of context
        _case("decode", 32768, 12, name="decode_32k", decoded=24),
        # the longest single sequence
        _case("decode", 131072, 4, name="decode_131k", decoded=24),
        # a long reply (thousands of streamed tokens) to a ragged prompt
        _case("decode", 5003, 8, name="decode_5k_long_reply", decoded=3001),
        # the cache's default mode: decoded tokens stay fp16; the kept rank is whatever the bit
        # allocation left (not a multiple of 32), on a tensor-parallel share of the heads
        _case("decode", 12345, 8, name="decode_12k_fp16_rows", mode="default", decoded=333, nkv=4, rank=150),
        # the next user turn of a chat: 48 new tokens in one forward after compression
        _case("turn", 8192, 2, name="turn_48_tokens_8k", decoded=200, new=48),
        # a server decoding 64 sequences of 8192 tokens in lock step
        _case("batch", 8192, 2, name="batch_64x8k", decoded=100, seqs=64),
        # a model without the hook: every step reads the cache back as fp16 keys and values
        _case("read", 8190, 3, name="read_back_8k", decoded=77),
        # prompts being compressed, up to and including the first decode step: short, hooked and
        # ordinary, long
        _case("prefill", 1100, 4, name="prefill_1k", mode="stream"),
        _case("prefill", 8191, 2, name="prefill_8k_hooked", mode="hooked"),
        _case("prefill", 32768, 2, name="prefill_32k", mode="default"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "turn", "batch", "read", "prefill", "prefill"))
    nkv = rng.choice((8, 8, 8, 4, 2))
    rank = rng.choice((192, 192, 192, 160, 150, 128, 90))
    mode = rng.choice(("stream", "stream", "default"))
    if kind == "decode":
        ctx = _log(rng, 150, 131072)
        return _case(kind, ctx, rng.randint(1, max(1, min(12, 400000 // ctx))), nkv=nkv, rank=rank, mode=mode,
                     decoded=_log(rng, 1, 4000))
    if kind == "turn":
        ctx = _log(rng, 300, 20000)
        return _case(kind, ctx, rng.randint(1, 2), nkv=nkv, rank=rank, mode=mode, decoded=_log(rng, 1, 1500),
                     new=_log(rng, 2, 256))
    if kind == "batch":
        seqs = _log(rng, 2, 64)
        ctx = _log(rng, 500, 16384)
        return _case(kind, ctx, rng.randint(1, 2), nkv=nkv, rank=rank, decoded=_log(rng, 1, 400), seqs=seqs)
    if kind == "read":
        return _case(kind, _log(rng, 200, 32768), rng.randint(1, 4), nkv=nkv, rank=rank, mode=mode,
                     decoded=_log(rng, 1, 1000))
    ctx = _log(rng, 900, 32768)
    return _case(kind, ctx, rng.randint(1, max(1, min(4, 65536 // ctx))), nkv=max(nkv, 4),
                 mode=rng.choice(("stream", "default", "hooked")))


# ---- inputs --------------------------------------------------------------------------------------
def _inv_freq():
    return 1.0 / (500000.0 ** (torch.arange(0, HD, 2, dtype=torch.float32) / HD))


def _rotate(x, positions):
    ph = positions.to(torch.float32)[:, None] * _inv_freq().to(x.device)[None, :]
    cos, sin = torch.cat([ph, ph], -1).cos(), torch.cat([ph, ph], -1).sin()
    return x * cos + torch.cat([-x[..., HD // 2:], x[..., :HD // 2]], -1) * sin


def _values(g, nkv, n, dev):
    """Values with four outlier channels per head, fp16 (1, nkv, n, HD)."""
    v = torch.randn(1, nkv, n, HD, generator=g, device=dev)
    v[..., 5::32] *= 20.0
    return v.half()


def _prompt(g, nkv, ctx, dev):
    """Keys (rank 192 plus a little noise before RoPE) and values of a prompt."""
    p = nkv * HD
    k = torch.randn(ctx, 192, generator=g, device=dev) @ (torch.randn(192, p, generator=g, device=dev) / math.sqrt(192))
    k += 0.01 * torch.randn(ctx, p, generator=g, device=dev)
    k = _rotate(k.view(ctx, nkv, HD).transpose(0, 1), torch.arange(ctx, device=dev))
    return k.unsqueeze(0).half().contiguous(), _values(g, nkv, ctx, dev)


def _compressed_layer(g, case, dev):
    """The tensor dictionary a compressed layer has, with coefficients, codes and scales of the sizes
    and spreads that compressing such a prompt gives."""
    nkv, rank, n = case["nkv"], case["rank"], case["ctx"] - SINK - WINDOW_TOKENS
    p = nkv * HD
    q = (torch.randn(n, rank, generator=g, device=dev, dtype=torch.float16) * 1.75).round_().clamp_(-7, 7).add_(8).to(torch.uint8)
    basis_q = (torch.randn(p, rank, generator=g, device=dev) * 36).round().clamp(-127, 127).to(torch.int8)
    basis_scale = (torch.rand(rank, generator=g, device=dev) * 2e-4 + 8e-4).half()
    mean = (torch.randn(p, generator=g, device=dev) * 0.02).half()
    idx = torch.randint(0, 256, (nkv, n, HD // 4), generator=g, device=dev, dtype=torch.uint8)
    gc = {
        "k_coeffs": (q[:, 0::2] | (q[:, 1::2] << 4)).contiguous().view(-1),
        "k_coeff_scale": (1.3 * math.sqrt(p / 1024 * 192 / rank) * torch.exp(-0.002 * torch.arange(rank, device=dev))).half(),
        "k_coeffs_shape": (n, rank),
        "k_basis_q": basis_q, "k_basis_scale": basis_scale,
        "k_basis_f16": (basis_q.half() * basis_scale).contiguous(),
        "k_mean": mean, "k_mean_f16": mean,
        "v_packed": idx.view(-1), "v_indices_u8": idx,
        "v_centroids_f16": (torch.randn(256, 4, generator=g, device=dev) * 0.25).half(),
        "v_ch_f16": (torch.rand(nkv, HD, generator=g, device=dev) * 4 + 14).half(),
        "sink_k": torch.randn(1, nkv, SINK, HD, generator=g, device=dev).half(), "sink_v": _values(g, nkv, SINK, dev),
        "win_k": torch.randn(1, nkv, WINDOW_TOKENS, HD, generator=g, device=dev).half(),
        "win_v": _values(g, nkv, WINDOW_TOKENS, dev),
        "n_compress": n, "batch": 1, "compress_start": SINK,
    }
    return attach_kernel_format(gc, nkv)


def _compressed_cache(g, case, dev, decoded):
    """A cache as it stands `decoded` tokens into a reply."""
    nkv, layers = case["nkv"], case["layers"]
    cache = Cache(num_layers=layers, n_kv_heads=nkv, rope_inv_freq=_inv_freq(), device=str(dev),
                  decode_capacity=decoded + WINDOW * case["new"])
    cache._streaming = case["mode"] == "stream"
    cache._compressed = True
    for layer in cache.layers:
        layer._gpu_compressed = _compressed_layer(g, case, dev)
        layer._prefilled = layer._needs_decompress = True
        layer._seq_len = case["ctx"]
    if decoded:
        cache._fused_decode_update = True
        k, v = torch.randn(1, nkv, decoded, HD, generator=g, device=dev).half(), _values(g, nkv, decoded, dev)
        for layer in cache.layers:
            layer.update(k, v)
        cache._fused_decode_update = False
    return cache


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    kind, nkv, layers, new = case["kind"], case["nkv"], case["layers"], case["new"]
    st = {"case": case, "pass": 0}

    def tokens(*lead):
        """q, k and v of new tokens, as a model's projections hand them over."""
        return (torch.randn(*lead, GQA * nkv, new, HD, generator=g, device=dev).half(),
                torch.randn(*lead, nkv, new, HD, generator=g, device=dev).half(),
                torch.randn(*lead, nkv, new, HD, generator=g, device=dev).half())

    if kind == "prefill":
        st["kv"] = [_prompt(g, nkv, case["ctx"], dev) for _ in range(layers)]
        st["q"], st["k"], st["v"] = tokens(layers, 1)
    elif kind == "batch":
        caches = [_compressed_cache(g, case, dev, 0) for _ in range(case["seqs"])]
        st["decoder"] = dec = BatchedDecoder(caches, stream_capacity=case["decoded"] + WINDOW)
        dec.q.normal_(generator=g)
        # the prefix of the reply: one token per step, as the decoder takes them
        for t in range(case["decoded"]):
            dec.new_k.normal_(generator=g)
            dec.new_v.normal_(generator=g)
            dec.step(case["ctx"] + t)
    else:
        st["cache"] = cache = _compressed_cache(g, case, dev, case["decoded"])
        st["tokens"] = [tokens(layers, 1) for _ in range(WINDOW)]
        st["rows"] = [(layer._gpu_compressed.get("decode_k"), layer._gpu_compressed.get("decode_v")) for layer in cache.layers]
    return st


# ---- passes --------------------------------------------------------------------------------------
def _restart_reply(st, w):
    """Before the first token of a reply, drop the rows of the reply before it."""
    if w == 0:
        for layer, (dk, dv) in zip(st["cache"].layers, st["rows"]):
            if dk is None:
                layer._gpu_compressed["stream_n"] = st["case"]["decoded"]
            else:
                layer._gpu_compressed["decode_k"], layer._gpu_compressed["decode_v"] = dk, dv


def _rows(gc):
    """The rows of decoded tokens a layer holds: what `update` changes."""
    return [gc[k] for k in ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf", "decode_k", "decode_v") if k in gc]


def _prefill(st):
    """A whole prompt: the prefill's `update` of every layer, then the first decode step, which
    compresses the cache."""
    case = st["case"]
    cache = Cache(num_layers=case["layers"], n_kv_heads=case["nkv"], rope_inv_freq=_inv_freq())
    cache._streaming = case["mode"] != "default"
    for li, (k, v) in enumerate(st["kv"]):
        cache.update(k, v, li)
    out = []
    if case["mode"] != "hooked":
        for li in range(case["layers"]):
            out += cache.update(st["k"][li], st["v"][li], li)
        return out
    cache.compress()
    cache._fused_decode_update = True
    for li, layer in enumerate(cache.layers):
        layer.update(st["k"][li], st["v"][li])
        gc = layer._gpu_compressed
        out += [fused_attention_compressed(st["q"][li], layer, case["ctx"], cache._rope_inv_freq), gc["v_indices_u8"],
                gc["v_centroids_f16"], gc["v_ch_f16"], gc["k_mean_f16"], gc["k_coeff_scale"], gc["k_basis_scale"]]
    return out


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "prefill":
        return _prefill(st)
    w = st["pass"] % WINDOW
    st["pass"] += 1
    if kind == "batch":
        dec = st["decoder"]
        dec.n_stream = case["decoded"] + w
        return dec.step(case["ctx"] + dec.n_stream)
    _restart_reply(st, w)
    cache = st["cache"]
    q, k, v = st["tokens"][w]
    if kind == "read":
        out = []
        for li, layer in enumerate(cache.layers):
            out += layer.update(k[li], v[li])
        return out
    # a hooked model: decode step (one new token) or the next turn (several)
    pos = case["ctx"] + case["decoded"] + (w + 1) * case["new"] - 1
    cache._fused_decode_update = True
    out = []
    for li, layer in enumerate(cache.layers):
        layer.update(k[li], v[li])
        out.append(fused_attention_compressed(q[li], layer, pos, cache._rope_inv_freq))
    cache._fused_decode_update = False
    if len(out) * 5 <= MAX_OUTPUTS:
        for layer in cache.layers:
            out += _rows(layer._gpu_compressed)
    return out


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    nkv, rank, new, layers = case["nkv"], case["rank"], case["new"], case["layers"]
    p, n = nkv * HD, case["ctx"] - SINK - WINDOW_TOKENS
    half = 2
    if case["kind"] == "prefill":
        # prompt in, compressed layer out (hooked) or fp16 keys and values out; the Gram matrix (half of
        # it), the projection, and 30 passes of k-means, each point against 256 centroids of 4 channels
        rank = min(192, p)
        b = 2 * case["ctx"] * p * half
        b += n * (rank // 2 + p // 4) if case["mode"] == "hooked" else b
        f = n * p * p + 2 * n * p * rank + 30 * (n * p // 4) * 256 * 8
        return {"bytes": layers * b, "flops": layers * f}
    # the compressed layer and its fp16 tokens, once
    b = n * (rank // 2 + p // 4) + p * rank + 2 * (SINK + WINDOW_TOKENS) * p * half
    rows = case["decoded"] + WINDOW // 2 * new
    b += 2 * rows * (p + half * nkv if case["mode"] == "stream" else p * half)
    if case["kind"] == "read":
        b += 2 * (case["ctx"] + rows) * p * half
        return {"bytes": layers * b, "flops": layers * 2 * n * p * rank}
    b += 2 * new * GQA * p * half
    # keys from their coefficients once; scores and weighted sum for every query
    f = 2 * n * p * rank + new * 4 * GQA * p * (case["ctx"] + rows)
    return {"bytes": layers * b * case["seqs"], "flops": layers * f * case["seqs"]}


def tolerance(case):
    # fp16 outputs of sums whose terms (rotated keys, weights) are fp16; stream codes are the same for
    # the same tokens
    if case["kind"] in ("decode", "turn", "batch"):
        return {"rel": 5e-3}
    # fp16 keys and values, the products behind them in fp16 or fp32
    if case["kind"] == "read":
        return {"rel": 2e-3}
    # k-means stops after 30 passes, well before it has settled: sums in another order move centroids in
    # the last digits, a point between two centroids falls on the other side, and the small clusters
    # drift apart from there (two runs of one program differ by 0.5 to 2 percent in the values, more in
    # short prompts; the keys agree)
    return {"rel": 3e-2, "max": 0.99, "differ": 1e-2}
