"""The compressor's fused entry points against their parts and float64, at tile edges and with strided views."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _keys(nkv, n, seed, scale=1.0, offset=0.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.randn(n + 3, nkv, 128, generator=g, device="cuda") * scale + offset
    return k.half().transpose(0, 1)[:, 2:n + 2, :]         # token-major storage, a view of it


def _inv_freq():
    return 1.0 / (500000.0 ** (torch.arange(0, 128, 2, dtype=torch.float32, device="cuda") / 128))


@pytest.mark.parametrize("nkv,n,scale,offset", [(1, 1, 1.0, 0.0), (1, 65, 1.0, 3.0), (2, 63, 1e-3, 0.0), (8, 200, 100.0, 0.0),
                                                (4, 1985, 1.0, 0.5), (8, 9000, 1.0, 0.0), (16, 700, 1.0, 0.0)])
def test_k_covariance(nkv, n, scale, offset):
    from shard_b200 import ops
    k, p = _keys(nkv, n, n, scale, offset), nkv * 128
    flat = torch.empty(n, p, device="cuda")
    mean, mean16, gram = torch.empty(p, device="cuda"), torch.empty(p, dtype=torch.float16, device="cuda"), torch.empty(p, p, device="cuda")
    ws = ops.k_covariance(k, 7, _inv_freq(), flat, mean, mean16, gram)
    assert int(ws[4:8].view(torch.int32)) == 0
    assert torch.equal(flat, ops.undo_rope(k, 7, _inv_freq()))
    want = flat.double().mean(0)
    assert (mean.double() - want).abs().max() <= 1e-6 * flat.abs().max() and torch.equal(mean16, mean.half())
    xc = flat.double() - mean.double()
    g64 = xc.T @ xc
    # relative to the columns' lengths: two fp16 parts per value, promoted sums
    norm = xc.norm(dim=0).clamp(min=1e-30)
    assert ((gram.double() - g64).abs() / (norm[:, None] * norm[None, :])).max() < (1e-6 if n > 1 else float("inf"))
    assert torch.equal(gram, gram.T.contiguous())


@pytest.mark.parametrize("nkv,n,keep", [(2, 129, 64), (8, 1000, 192), (4, 333, 150), (8, 77, 2)])
def test_k_encode_equals_its_parts(nkv, n, keep):
    from shard_b200 import ops
    p = nkv * 128
    g = torch.Generator(device="cuda").manual_seed(n)
    flat = torch.randn(n, p, generator=g, device="cuda")
    mean = flat.mean(0)
    basis = torch.linalg.qr(torch.randn(p, 192, generator=g, device="cuda"))[0].contiguous()
    alloc = [(8, 6, 4, 2)[j * 4 // keep] for j in range(keep)]
    q, scale, b16, packed, cs, wprep, _ = ops.k_encode(flat, mean, mean.half(), basis[:, :keep], alloc)
    b = basis[:, :keep].contiguous()
    s = b.abs().max(dim=0).values.clamp(min=1e-6) / 127.0
    bq = (b / s).round().clamp(-127, 127).to(torch.int8)
    assert torch.equal(q, bq) and torch.equal(scale, s.half()) and torch.equal(b16, bq.half() * s.half())
    proj = ops.k_project(flat, mean, (bq.float() * s).contiguous())
    pk, c32 = ops.k_quantize_pack(proj, alloc)
    assert torch.equal(packed, pk) and torch.equal(cs, c32.half())
    if keep % 32:
        assert wprep is None
    else:
        assert torch.equal(wprep, ops.decode_prepare(b16, cs, mean.half(), nkv, keep))


@pytest.mark.parametrize("n_sink,n_win,n", [(4, 64, 200), (0, 3, 9), (5, 0, 5)])
def test_kv_ends(n_sink, n_win, n):
    from shard_b200 import ops
    k, v = _keys(8, n, 1), _keys(8, n, 2).contiguous()
    sk, sv, wk, wv = ops.kv_ends(k, v, n_sink, n_win, n - n_win)
    assert torch.equal(sk[0], k[:, :n_sink]) and torch.equal(sv[0], v[:, :n_sink])
    assert torch.equal(wk[0], k[:, n - n_win:]) and torch.equal(wv[0], v[:, n - n_win:])


@pytest.mark.parametrize("nkv,n", [(1, 1), (3, 31), (8, 33), (8, 5001)])
def test_v_hadamard_normalise_views(nkv, n):
    from shard_b200 import ops
    v = _keys(nkv, n, n)
    x, ch = ops.v_hadamard_normalise(v)
    y = v.double()
    h = 1
    while h < 128:
        y = y.reshape(nkv, n, -1, 2, h)
        y = torch.cat([y[..., :1, :] + y[..., 1:, :], y[..., :1, :] - y[..., 1:, :]], -2).reshape(nkv, n, 128)
        h *= 2
    y = y / 128 ** 0.5
    m = y.abs().amax(dim=1)
    assert ((ch.double() - m).abs() <= 1e-6 * m).all()
    assert (x.double() - y / m[:, None, :]).abs().max() < 1e-5


@pytest.mark.parametrize("where,nkv", [("k_covariance", 8), ("k_encode", 8), ("k_encode", 2)])
def test_a_wait_that_gave_up_is_reported(where, nkv, monkeypatch):
    """The status words of the compressor's kernels end as an error of `compress`, whichever layer raised them."""
    from shard_b200 import Cache, ops
    from shard_b200._lib import ShardError
    real, calls = getattr(ops, where), []
    word = ops.covariance_status if where == "k_covariance" else ops.encode_status

    def once(*a):
        r = real(*a)
        calls.append(1)
        if len(calls) == 2:                                # the second layer of nine, in the first of two groups
            word(r if where == "k_covariance" else r[-1]).fill_(1)
        return r

    monkeypatch.setattr(ops, where, once)
    cache = Cache(num_layers=9, n_kv_heads=nkv, rope_inv_freq=_inv_freq().cpu())
    for li in range(9):
        cache.update(_keys(nkv, 400, li).unsqueeze(0), _keys(nkv, 400, 50 + li).unsqueeze(0), li)
    with pytest.raises(ShardError, match="gave up"):
        cache.compress()
    assert not cache._compressed
    if where == "k_covariance":                            # nothing was built on that matrix
        assert all(layer._gpu_compressed is None and layer._keys is not None for layer in cache.layers)


def test_status_words_stay_set():
    """A later call does not clear what an earlier one reported."""
    from shard_b200 import ops
    k, p = _keys(8, 300, 1), 1024
    flat, mean, gram = torch.empty(300, p, device="cuda"), torch.empty(p, device="cuda"), torch.empty(p, p, device="cuda")
    mean16 = torch.empty(p, dtype=torch.float16, device="cuda")
    basis = torch.linalg.qr(torch.randn(p, 64, device="cuda"))[0].contiguous()
    cov = ops.k_covariance(k, 7, _inv_freq(), flat, mean, mean16, gram)
    enc = ops.k_encode(flat, mean, mean16, basis, [4] * 64)[-1]
    assert int(ops.covariance_status(cov)) == 0 and int(ops.encode_status(enc)) == 0
    ops.covariance_status(cov).fill_(1)
    ops.encode_status(enc).fill_(1)
    ops.k_covariance(k, 7, _inv_freq(), flat, mean, mean16, gram, cov)
    ops.k_encode(flat, mean, mean16, basis, [4] * 64, enc)
    assert int(ops.covariance_status(cov)) == 1 and int(ops.encode_status(enc)) == 1


@pytest.mark.parametrize("kind,ratio", [("element", 256.0), ("element", 4096.0), ("channel", 1024.0), ("token", 1024.0), ("small", 1e-4)])
def test_k_covariance_of_uneven_keys(kind, ratio):
    """One large element, channel or token beside ordinary ones, or channels far below the others: the matrix
    stays within a fp32 product's error of float64, relative to each pair of columns."""
    from shard_b200 import ops
    n, p = 8192, 1024
    g = torch.Generator(device="cuda").manual_seed(int(ratio) + len(kind))
    k = torch.randn(8, n, 128, generator=g, device="cuda")
    if kind == "element":
        k[3, 77, 5] = 4 * ratio
    elif kind == "channel":
        k[3, :, 5] *= ratio
    elif kind == "token":
        k[:, 77] *= ratio
    else:
        k[4:, :, ::3] *= ratio
    k = k.half()
    flat, mean, gram = torch.empty(n, p, device="cuda"), torch.empty(p, device="cuda"), torch.empty(p, p, device="cuda")
    # no rotation: the channels stay as uneven as they are
    ops.k_covariance(k, 0, torch.zeros(64, device="cuda"), flat, mean, torch.empty(p, dtype=torch.float16, device="cuda"), gram)
    xc = flat.double() - mean.double()
    norm = xc.norm(dim=0)
    err = (gram.double() - xc.T @ xc).abs() / (norm[:, None] * norm[None, :])
    # the tensor core truncates: 12 additions (4 k-steps of 3 products) to one accumulator at 2^-23 of it, all at
    # the size of the result where one token dominates; the split drops 2^-22 of either factor
    assert err.max() < 12 * 2.0 ** -23 + 2 * 2.0 ** -22


@pytest.mark.parametrize("nkv", [8, 4])
def test_memory_of_compressing_many_layers(nkv):
    """Peak memory: k-means over as many points as run side by side (fp32 points, their sorted copy, numbers and
    codes: 40 bytes each), the fp32 rows that may be kept, a few copies of ONE layer's, and the result."""
    from shard_b200 import Cache
    from shard_b200.cache import KMEANS_POINTS, ROWS_BYTES
    layers, n, p = 14, 320000 // nkv, nkv * 128
    cache = Cache(num_layers=layers, n_kv_heads=nkv, rope_inv_freq=_inv_freq().cpu())
    for li in range(layers):
        cache.update(_keys(nkv, n, li).unsqueeze(0), _keys(nkv, n, 50 + li).unsqueeze(0), li)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    cache.compress()
    extra = torch.cuda.max_memory_allocated() - before
    result = layers * n * (p // 4 + 192 // 2) + layers * 4 * p * p          # codes; weights and the like
    assert extra < max(KMEANS_POINTS, n * p // 4) * 40 + ROWS_BYTES + 4 * n * p * 4 + result + (64 << 20)


@pytest.mark.parametrize("nkv,layers", [(8, 1), (8, 8), (4, 3), (8, 17)])
def test_rows_made_twice_give_the_same_cache(nkv, layers, monkeypatch):
    """The keys' codes do not depend on whether the un-rotated rows were kept or made again."""
    from shard_b200 import Cache
    from shard_b200 import cache as mod
    made = []
    for budget in (1 << 40, 0):
        monkeypatch.setattr(mod, "ROWS_BYTES", budget)
        cache = Cache(num_layers=layers, n_kv_heads=nkv, rope_inv_freq=_inv_freq().cpu())
        for li in range(layers):
            cache.update(_keys(nkv, 300, li).unsqueeze(0), _keys(nkv, 300, 50 + li).unsqueeze(0), li)
        cache.compress()
        made.append([layer._gpu_compressed for layer in cache.layers])
    for a, b in zip(*made):
        for name in ("k_coeffs", "k_coeff_scale", "k_basis_q", "k_basis_scale", "k_mean", "k_wprep"):
            assert torch.equal(a[name], b[name]), name


@pytest.mark.parametrize("nkv", [8, 4])
def test_threads_compress_side_by_side(nkv):
    """Caches compressed at the same time by threads with streams of their own come out as one after the other."""
    import threading
    from shard_b200 import Cache
    names = ("k_coeffs", "k_coeff_scale", "k_basis_q", "k_basis_scale", "k_mean", "k_wprep", "v_indices_u8", "v_centroids_f16", "sink_k", "win_v")
    prompts = [[(_keys(nkv, 600 + 128 * c, 10 * c + li).unsqueeze(0), _keys(nkv, 600 + 128 * c, 50 + 10 * c + li).unsqueeze(0))
                for li in range(9)] for c in range(4)]
    torch.cuda.synchronize()

    def compressed(c):
        cache = Cache(num_layers=9, n_kv_heads=nkv, rope_inv_freq=_inv_freq().cpu())
        for li, (k, v) in enumerate(prompts[c]):
            cache.update(k, v, li)
        cache.compress()
        return [{n: layer._gpu_compressed[n].clone() for n in names} for layer in cache.layers]

    want = [compressed(c) for c in range(4)]
    got, errors = [None] * 4, []

    def work(c):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(4):
                    got[c] = compressed(c)
                torch.cuda.current_stream().synchronize()
        except Exception as e:                             # (raised in the test's own thread below)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(want, got):
        for x, y in zip(a, b):
            for n in names:
                assert torch.equal(x[n], y[n]), n


@pytest.mark.parametrize("nkv", [8, 4])
@pytest.mark.parametrize("streaming", [True, False])
def test_prompt_and_reply_under_inference_mode(nkv, streaming):
    """torch.inference_mode around everything: the same cache and the same attention as under no_grad."""
    from shard_b200 import Cache, fused_attention_compressed
    res = []
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            cache = Cache(num_layers=2, n_kv_heads=nkv, rope_inv_freq=_inv_freq().cpu())
            cache._streaming = streaming
            for li in range(2):
                cache.update(_keys(nkv, 400, li).unsqueeze(0), _keys(nkv, 400, 50 + li).unsqueeze(0), li)
            cache.compress()
            out = []
            for t in range(3):
                for fused in (True, False):
                    cache._fused_decode_update = fused
                    for li, layer in enumerate(cache.layers):
                        k, v = (_keys(nkv, 1, 100 + 10 * t + li + s).unsqueeze(0) for s in (0, 500))
                        r = layer.update(k, v)
                        q = _keys(4 * nkv, 1, 900 + t).unsqueeze(0)
                        out += [fused_attention_compressed(q, layer, layer.get_seq_length() - 1).clone()] if fused else list(r)
            out += [layer._gpu_compressed[n] for layer in cache.layers for n in ("k_coeffs", "k_basis_q", "v_indices_u8")]
            res.append([o.clone() for o in out])
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("n", [31, 33, 16383, 16384, 16449])
def test_k_quantize_pack_either_side_of_the_row_rule(n):
    """Codes and scales are the oracle's with 32 and with 64 rows per block, also where the last block is short."""
    import numpy as np
    from oracle import shard_oracle as O
    from shard_b200 import ops
    rng = np.random.default_rng(n)
    proj = (rng.standard_normal((n, 6)) * [10, 3, 1, 0.3, 0.1, 1e-4]).astype(np.float32)
    proj[-1] *= 4                                          # the extremes lie in the last block
    alloc = [8, 6, 4, 2, 2, 0]
    packed, scale = ops.k_quantize_pack(torch.from_numpy(proj).cuda(), alloc)
    q, want, _ = O.k_int4_codes(proj, alloc)
    assert np.array_equal(scale.cpu().numpy(), want) and np.array_equal(packed.cpu().numpy(), O.int4_pack(q))


@pytest.mark.parametrize("nkv,n", [(8, 32768), (8, 1100), (5, 4096)])
def test_reconstruction_with_either_solver(nkv, n, monkeypatch):
    """Another eigensolver flips codes at rounding boundaries; what counts is the distance of the keys from the
    uncompressed prompt's, which is the library solver's to a thousandth (a code in a hundred flipped by half a
    step at random moves it by less)."""
    import synth
    from shard_b200 import Cache
    from shard_b200 import cache as mod
    k, v, _ = synth.make_kvq(n, 3, device="cuda", nkv=nkv)
    errs = []
    for limit in (mod.TORCH_EIGH_MAX, 1 << 20):
        monkeypatch.setattr(mod, "TORCH_EIGH_MAX", limit)
        cache = Cache(num_layers=1, n_kv_heads=nkv, rope_inv_freq=synth.rope_inv_freq())
        cache.update(k, v, 0)
        cache.compress()
        layer = cache.layers[0]
        errs.append([float((a[:, :, 4:n - 64].double() - b[:, :, 4:n - 64].double()).norm() / b[:, :, 4:n - 64].double().norm())
                     for a, b in ((layer.keys, k), (layer.values, v))])
        del cache, layer
    assert abs(errs[0][0] / errs[1][0] - 1) < 1e-3 and abs(errs[0][1] / errs[1][1] - 1) < 1e-3, errs
