"""Read-back of a compressed layer (`layer.keys` / `layer.values`) against a float64 evaluation of the
same tensor dictionary, at tile edges, padded ranks and every kind of row."""
import numpy as np
import pytest
import torch

from gpu_helpers import random_gc

pytestmark = pytest.mark.gpu


def _cache(gc_np, nkv, streaming, capacity=64):
    from gpu_helpers import gc_to_device
    from oracle import shard_oracle as O
    from shard_b200 import Cache
    cache = Cache(num_layers=1, n_kv_heads=nkv, rope_inv_freq=torch.from_numpy(O.default_inv_freq()), decode_capacity=capacity)
    cache._streaming, cache._compressed = streaming, True
    layer = cache.layers[0]
    layer._gpu_compressed = gc_to_device(gc_np, nkv=nkv)
    layer._prefilled = layer._needs_decompress = True
    layer._seq_len = gc_np["n_compress"] + gc_np["sink_k"].shape[1] + gc_np["win_k"].shape[1]
    return cache, layer


def middle_float64(gc_np, nkv):
    """(nkv, n, 128) keys (with RoPE) and values of the middle segment, float64."""
    from oracle import shard_oracle as O
    n, rank = gc_np["k_coeffs_shape"]
    packed = gc_np["k_coeffs"]
    q = np.stack([packed & 15, packed >> 4], 1).reshape(-1)[: n * rank].reshape(n, rank).astype(np.float64) - 8
    k = (q * gc_np["k_coeff_scale"].astype(np.float64)) @ gc_np["k_basis_f16"].astype(np.float64).T + gc_np["k_mean"].astype(np.float64)
    k = k.reshape(n, nkv, 128).transpose(1, 0, 2)
    pos = (gc_np["compress_start"] + np.arange(n)).astype(np.float32)
    ph = (pos[:, None] * O.default_inv_freq().astype(np.float32)[None, :]).astype(np.float64)
    c, d = k[..., :64], k[..., 64:]
    k = np.concatenate([c * np.cos(ph) - d * np.sin(ph), d * np.cos(ph) + c * np.sin(ph)], -1)
    v = gc_np["v_centroids_f16"].astype(np.float64)[gc_np["v_indices_u8"]].reshape(nkv, n, 128) * gc_np["v_ch_f16"].astype(np.float64)[:, None, :]
    h = 1
    while h < 128:
        v = v.reshape(nkv, n, -1, 2, h)
        v = np.concatenate([v[..., :1, :] + v[..., 1:, :], v[..., :1, :] - v[..., 1:, :]], -2).reshape(nkv, n, 128)
        h *= 2
    return k, v / np.sqrt(128.0)


@pytest.mark.parametrize("n_comp,rank,nkv,n_new,streaming", [
    (1, 192, 8, 0, True), (127, 32, 2, 1, True), (128, 64, 1, 2, False), (129, 150, 8, 5, True), (700, 192, 8, 40, False),
    (1500, 160, 4, 3, True), (20000, 128, 8, 70, True)])
def test_read_back(n_comp, rank, nkv, n_new, streaming):
    from shard_b200 import ops
    from shard_b200.streaming import get_codebook
    gc_np = random_gc(n_comp, rank=rank, nkv=nkv, seed=n_comp)
    cache, layer = _cache(gc_np, nkv, streaming)
    gc = layer._gpu_compressed
    g = torch.Generator(device="cuda").manual_seed(3)
    new_k = torch.randn(1, nkv, n_new + 1, 128, generator=g, device="cuda").half()
    new_v = torch.randn(1, nkv, n_new + 1, 128, generator=g, device="cuda").half()
    if n_new:
        cache._fused_decode_update = True
        layer.update(new_k[:, :, :n_new], new_v[:, :, :n_new])       # several tokens: one launch
        cache._fused_decode_update = False
    keys, values = layer.update(new_k[:, :, n_new:], new_v[:, :, n_new:])   # the last: inside the read-back
    cache.check()
    if streaming:
        # the appended rows equal the single-token quantizer's, and read back as the dequantizer gives them
        cb = get_codebook(128, 8, torch.device("cuda", 0))
        bufs = [torch.zeros_like(gc[k][: n_new + 1]) for k in ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf")]
        for t in range(n_new + 1):
            ops.stream_quantize(new_k[0, :, t].contiguous(), new_v[0, :, t].contiguous(), gc["signs"], cb, *bufs, t)
        for b, k in zip(bufs, ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf")):
            assert torch.equal(b, gc[k][: n_new + 1])
        tail_k = ops.stream_dequant(bufs[0], bufs[2], gc["signs"], cb)
        tail_v = ops.stream_dequant(bufs[1], bufs[3], gc["signs"], cb)
    else:
        tail_k, tail_v = new_k[0], new_v[0]
    ns, nw = gc["sink_k"].shape[2], gc["win_k"].shape[2]
    assert keys.shape == values.shape == (1, nkv, ns + n_comp + nw + n_new + 1, 128)
    for got, sink, win, tail in ((keys, gc["sink_k"], gc["win_k"], tail_k), (values, gc["sink_v"], gc["win_v"], tail_v)):
        assert torch.equal(got[0, :, :ns], sink[0])
        assert torch.equal(got[0, :, ns + n_comp:ns + n_comp + nw], win[0])
        assert torch.equal(got[0, :, ns + n_comp + nw:], tail)
    k64, v64 = middle_float64(gc_np, nkv)
    gk = keys[0, :, ns:ns + n_comp].double().cpu().numpy()
    gv = values[0, :, ns:ns + n_comp].double().cpu().numpy()
    # fp16 output, weights rounded to fp16 once
    assert np.abs(gk - k64).max() <= 2e-3 * np.abs(k64).max() and np.linalg.norm(gk - k64) <= 6e-4 * np.linalg.norm(k64)
    assert (np.abs(gv - v64) <= 1e-5 + 6e-4 * np.abs(v64)).all()


def test_read_back_of_tokens_in_another_dtype():
    """A reply whose tokens are not fp16 (the model's type changed after compression): they are kept and read
    back as they are, behind the layer's own."""
    cache, layer = _cache(random_gc(300, nkv=2, seed=1), 2, False)
    want = layer.keys.clone(), layer.values.clone()
    k, v = (torch.randn(1, 2, 3, 128, device="cuda") for _ in range(2))
    layer.update(k[:, :, :2], v[:, :, :2])
    keys, values = layer.update(k[:, :, 2:], v[:, :, 2:])
    for got, old, new in ((keys, want[0], k), (values, want[1], v)):
        assert got.dtype == torch.float32 and torch.equal(got, torch.cat([old, new], 2))


def test_read_back_of_a_dictionary_without_kernel_tensors():
    """The reference's tensors are enough to read a layer back."""
    cache, layer = _cache(random_gc(300, rank=150, nkv=2, seed=1), 2, True)
    gc = layer._gpu_compressed
    want = layer.keys.clone(), layer.values.clone()
    for name in ("k_wprep", "k_coeffs_kernel", "k_coeffs_padded", "k_rank_kernel", "_fresh", "_seq"):
        gc.pop(name, None)
    layer._needs_decompress = True
    assert torch.equal(layer.keys, want[0]) and torch.equal(layer.values, want[1])


@pytest.mark.parametrize("streaming", [True, False])
def test_a_token_survives_a_read_back_that_failed(streaming, monkeypatch):
    """The newest token is not lost when the launch that would have written it cannot be made."""
    from shard_b200 import ops
    from shard_b200._lib import ShardError
    caches = [_cache(random_gc(300, nkv=2, seed=1), 2, streaming) for _ in range(2)]
    k, v = (torch.randn(1, 2, 3, 128, device="cuda").half() for _ in range(2))

    def fail(*a):
        raise ShardError("no")

    for i, (cache, layer) in enumerate(caches):
        layer.update(k[:, :, :1], v[:, :, :1])
        if i == 0:
            with monkeypatch.context() as m:
                m.setattr(ops, "read_back", fail)
                with pytest.raises(ShardError):
                    layer.update(k[:, :, 1:2], v[:, :, 1:2])
        else:
            layer.update(k[:, :, 1:2], v[:, :, 1:2])
    (_, a), (_, b) = caches
    assert torch.equal(a.keys, b.keys) and torch.equal(a.values, b.values)


@pytest.mark.parametrize("streaming", [True, False])
def test_fused_steps_do_not_hold_read_back_layers(streaming):
    """A reply that goes on with the fused kernel keeps no fp16 copy of a layer from an earlier read-back."""
    from gpu_helpers import gc_to_device
    from shard_b200 import Cache
    cache = Cache(num_layers=3, n_kv_heads=2, rope_inv_freq=torch.ones(64))
    cache._streaming, cache._compressed = streaming, True
    k, v = (torch.randn(1, 2, 1, 128, device="cuda").half() for _ in range(2))
    for layer in cache.layers:
        layer._gpu_compressed = gc_to_device(random_gc(300, nkv=2, seed=1), nkv=2)
        layer._prefilled = layer._needs_decompress = True
        layer._seq_len = 368
    for fused in (False, True):
        cache._fused_decode_update = fused
        for layer in cache.layers:
            layer.update(k, v)
    assert all(layer._keys is None and layer._values is None for layer in cache.layers)
    assert cache.layers[2].keys.shape[2] == 370
