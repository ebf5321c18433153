"""The native host half of a decode step: same rows and same outputs as the Python path, in both append
modes, over buffer growth and a restarted reply."""
import gc

import pytest
import torch

from gpu_helpers import random_gc
from test_gpu_readback import _cache

pytestmark = pytest.mark.gpu


class _Counting:
    """The native module, counting the steps it took."""

    def __init__(self, real):
        self.real, self.taken = real, 0

    def __getattr__(self, name):
        return getattr(self.real, name)

    def attend(self, *a):
        r = self.real.attend(*a)
        self.taken += r is not None
        return r


@pytest.mark.parametrize("streaming,nkv,n_comp", [(True, 8, 700), (False, 8, 700), (False, 1, 130), (True, 2, 1)])
def test_native_steps(streaming, nkv, n_comp, monkeypatch):
    from shard_b200 import _lib, fused_attention_compressed
    from shard_b200.attention import decode_layer
    counting = _Counting(_lib.host())
    monkeypatch.setattr(_lib, "_host", counting)
    cache, layer = _cache(random_gc(n_comp, nkv=nkv, seed=1), nkv, streaming, capacity=16)
    other, ref = _cache(random_gc(n_comp, nkv=nkv, seed=1), nkv, streaming, capacity=16)
    cache._fused_decode_update = other._fused_decode_update = True
    g = torch.Generator(device="cuda").manual_seed(2)
    gc, rgc = layer._gpu_compressed, ref._gpu_compressed

    def token():
        return [torch.randn(1, nkv, 1, 128, generator=g, device="cuda").half() for _ in range(2)]

    def append_ref(k, v):                                   # the same rows, written the general way
        if streaming:
            ref._stream_append(k, v, 0)
        else:
            ref._fp16_append(k, v)

    for step in range(20):                                  # the buffers (16 rows) grow on the way
        k, v = token()
        q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
        layer.update(k, v)
        out = fused_attention_compressed(q, layer, 5000 + step, cache._rope_inv_freq)
        append_ref(k, v)
        assert torch.equal(out.view(-1, 128), decode_layer(q, ref, 5000 + step))
        if step == 10:                                      # the reply starts over: rows are dropped
            if streaming:
                gc["stream_n"] = rgc["stream_n"] = 3
            else:
                for d in (gc, rgc):
                    d["decode_k"], d["decode_v"] = d["decode_k"][:, :, :3], d["decode_v"][:, :, :3]
    assert counting.taken >= 17
    n = gc["stream_n"] if streaming else None
    for name in ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf") if streaming else ("decode_k", "decode_v"):
        assert torch.equal(gc[name][:n], rgc[name][:n])
    # a token whose append never met a launch is written by the next one that reads the rows
    k, v = token()
    for _ in range(2):
        layer.update(k, v)
        append_ref(k, v)
    assert torch.equal(layer.keys, ref.keys) and torch.equal(layer.values, ref.values)


def test_stream_buffers_that_moved_behind_the_same_object():
    """A step takes the stream buffers' memory from the tensors as they are, also where a tensor object of the
    same identity holds other memory (as when a freed object's address is used again)."""
    from shard_b200 import fused_attention_compressed
    from shard_b200.attention import decode_layer
    cache, layer = _cache(random_gc(300, nkv=2, seed=1), 2, True, capacity=16)
    other, ref = _cache(random_gc(300, nkv=2, seed=1), 2, True, capacity=16)
    cache._fused_decode_update = True
    g = torch.Generator(device="cuda").manual_seed(3)
    gc, names = layer._gpu_compressed, ("k_idx_buf", "v_idx_buf", "k_norm_buf", "v_norm_buf")
    before = None
    for t in range(8):
        k, v = (torch.randn(1, 2, 1, 128, generator=g, device="cuda").half() for _ in range(2))
        q = torch.randn(1, 8, 1, 128, generator=g, device="cuda").half()
        if t in (4, 6):
            before = [gc[n].data for n in names]            # (stays allocated)
            for n in names:
                gc[n].data = gc[n].data.clone()
            copies = [b.clone() for b in before]
        layer.update(k, v)
        out = (fused_attention_compressed(q, layer, 400 + t, cache._rope_inv_freq) if t != 6
               else decode_layer(q, layer, 400 + t))        # (the general path as well)
        ref._stream_append(k, v, 0)
        assert torch.equal(out.view(-1, 128), decode_layer(q, ref, 400 + t))
        if before is not None:
            assert all(torch.equal(b, c) for b, c in zip(before, copies))
    for n in names:
        assert torch.equal(gc[n][:8], ref._gpu_compressed[n][:8])


def test_a_failed_allocation_is_a_python_exception():
    """The native step's output does not fit: the error torch raises, not the end of the process."""
    from shard_b200 import fused_attention_compressed
    cache, layer = _cache(random_gc(300, nkv=8, seed=1), 8, True, capacity=16)
    cache._fused_decode_update = True
    g = torch.Generator(device="cuda").manual_seed(3)

    def step(t):
        k, v = (torch.randn(1, 8, 1, 128, generator=g, device="cuda").half() for _ in range(2))
        layer.update(k, v)
        return k, v, torch.randn(1, 32, 1, 128, generator=g, device="cuda").half()

    for t in range(3):
        _, _, q = step(t)
        want = fused_attention_compressed(q, layer, 400 + t, cache._rope_inv_freq)
    _, _, q = step(3)
    gc.collect()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
    held = []
    try:
        for size in (1 << 20, 32 * 128, 32 * 128):         # (until nothing is left, whatever earlier work had cached)
            while len(held) < 200000:
                try:
                    held.append(torch.empty(size, dtype=torch.float16, device="cuda"))
                except torch.cuda.OutOfMemoryError:
                    break
        with pytest.raises(torch.cuda.OutOfMemoryError):
            fused_attention_compressed(q, layer, 403, cache._rope_inv_freq)
    finally:
        held.clear()
        torch.cuda.set_per_process_memory_fraction(1.0)
    out = fused_attention_compressed(q, layer, 403, cache._rope_inv_freq)      # the token is still to be appended
    cache.check()
    assert out.shape == want.shape and "_pending" not in layer._gpu_compressed


@pytest.mark.parametrize("nkv,n_comp", [(8, 300), (1, 1)])
def test_fp16_rows_are_the_caches_own(nkv, n_comp):
    """A cache that keeps tokens as they are has copied them when `update` returns: the caller's tensors may
    change before it attends, and the rows are there for whoever reads `decode_k` / `decode_v`."""
    from shard_b200 import fused_attention_compressed
    from shard_b200.attention import decode_layer
    cache, layer = _cache(random_gc(n_comp, nkv=nkv, seed=1), nkv, False, capacity=16)
    other, ref = _cache(random_gc(n_comp, nkv=nkv, seed=1), nkv, False, capacity=16)
    cache._fused_decode_update = True
    g = torch.Generator(device="cuda").manual_seed(3)
    k, v = (torch.empty(1, nkv, 1, 128, dtype=torch.float16, device="cuda") for _ in range(2))
    gc, rows = layer._gpu_compressed, []
    for t in range(24):                                    # the same two tensors for every token, over a growth of the buffers
        k.normal_(generator=g)
        v.normal_(generator=g)
        rows.append((k.clone(), v.clone()))
        ref._fp16_append(*rows[-1])
        q = torch.randn(1, 4 * nkv, 1, 128, generator=g, device="cuda").half()
        layer.update(k, v)
        k.zero_()
        v.fill_(float("nan"))
        for name, i in (("decode_k", 0), ("decode_v", 1)):
            assert torch.equal(gc[name], torch.cat([r[i] for r in rows], 2))
        out = fused_attention_compressed(q, layer, 400 + t, cache._rope_inv_freq)
        assert torch.equal(out.view(-1, 128), decode_layer(q, ref, 400 + t))
    cache._fused_decode_update = False
    k.normal_(generator=g)
    v.normal_(generator=g)
    rows.append((k.clone(), v.clone()))
    keys, values = layer.update(k, v)                      # written by the read-back
    k.zero_()
    v.zero_()
    for got, name, i in ((keys, "decode_k", 0), (values, "decode_v", 1)):
        want = torch.cat([r[i] for r in rows], 2)
        assert torch.equal(gc[name], want) and torch.equal(got[:, :, -len(rows):], want)


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("s", [1, 3])
def test_tokens_that_do_not_fit_the_cache_are_refused(streaming, s):
    """Tokens of two sequences, of other heads, or (stream) with options the kernels do not have: refused
    also when the buffers have room, and the cache is as it was."""
    from shard_b200._lib import ShardError
    cache, layer = _cache(random_gc(200, nkv=2, seed=1), 2, streaming, capacity=64)
    g = torch.Generator(device="cuda").manual_seed(3)

    def new(*shape):
        return torch.randn(*shape, 128, generator=g, device="cuda").half()

    keys, _ = layer.update(new(1, 2, 2), new(1, 2, 2))
    n, want = layer.get_seq_length(), keys.clone()
    for fused in (True, False):
        cache._fused_decode_update = fused
        for shape, err in (((2, 2, s), NotImplementedError), ((1, 1, s), ShardError), ((1, 4, s), ShardError)):
            with pytest.raises(err):
                layer.update(new(*shape), new(*shape))
        with pytest.raises(ShardError):
            layer.update(new(1, 2, s), new(1, 2, s + 1))
        if streaming:
            for flag, value in (("_stream_qjl", True), ("_stream_bits", 4)):
                was = getattr(cache, flag)
                setattr(cache, flag, value)
                with pytest.raises(NotImplementedError):
                    layer.update(new(1, 2, s), new(1, 2, s))
                setattr(cache, flag, was)
    assert layer.get_seq_length() == n
    layer._needs_decompress = True
    assert torch.equal(layer.keys, want)


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("s", [1, 2, 5])
def test_tensors_that_start_between_8_byte_boundaries(streaming, s):
    """Views that start one element into a buffer: same rows, same attention."""
    from shard_b200 import fused_attention_compressed
    caches = [_cache(random_gc(300, nkv=2, seed=1), 2, streaming, capacity=16) for _ in range(2)]
    g = torch.Generator(device="cuda").manual_seed(3)

    def shifted(t):
        buf = torch.empty(t.numel() + 1, dtype=t.dtype, device="cuda")
        buf[1:].copy_(t.reshape(-1))
        return buf[1:].view(t.shape)

    for step in range(3):
        k, v = (torch.randn(1, 2, s, 128, generator=g, device="cuda").half() for _ in range(2))
        q = torch.randn(1, 8, s, 128, generator=g, device="cuda").half()
        outs = []
        for (cache, layer), f in zip(caches, (lambda t: t, shifted)):
            cache._fused_decode_update = True
            layer.update(f(k), f(v))
            outs.append(fused_attention_compressed(f(q), layer, layer.get_seq_length() - 1, cache._rope_inv_freq))
            cache._fused_decode_update = False
            if step == 2:
                outs.append(layer.update(f(k), f(v))[0])
        assert all(torch.equal(a, b) for a, b in zip(outs[:len(outs) // 2], outs[len(outs) // 2:]))


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("fused", [True, False])
def test_a_cache_can_be_copied_between_steps(streaming, fused):
    """copy.deepcopy in the middle of a reply (a prompt's cache drawn from twice): both go on by themselves."""
    import copy

    from shard_b200 import fused_attention_compressed
    cache, layer = _cache(random_gc(300, nkv=2, seed=1), 2, streaming, capacity=16)
    g = torch.Generator(device="cuda").manual_seed(3)

    def token():
        return [torch.randn(1, n, 1, 128, generator=g, device="cuda").half() for n in (2, 2, 8)]

    def step(cache, k, v, q):
        layer = cache.layers[0]
        cache._fused_decode_update = fused
        r = layer.update(k, v)
        if not fused:
            return [x.clone() for x in r]
        return [fused_attention_compressed(q, layer, layer.get_seq_length() - 1, cache._rope_inv_freq).clone()]

    for _ in range(4):
        step(cache, *token())
    other = copy.deepcopy(cache)
    first, second = token(), token()
    a = step(cache, *first)                                # the original goes one way ...
    b = step(other, *second)                               # ... the copy another ...
    again = copy.deepcopy(other)
    assert all(not torch.equal(x, y) for x, y in zip(a, b))
    third = token()
    assert all(torch.equal(x, y) for x, y in zip(step(other, *third), step(again, *third)))


def test_a_layer_moved_to_another_cache():
    """The dictionary of a layer that has taken native steps serves a cache with other RoPE frequencies."""
    from shard_b200 import fused_attention_compressed
    from shard_b200.attention import decode_layer
    cache, layer = _cache(random_gc(300, nkv=2, seed=1), 2, True, capacity=16)
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(1, 8, 1, 128, generator=g, device="cuda").half()
    for t in range(3):
        fused_attention_compressed(q, layer, 400 + t, cache._rope_inv_freq)
    others = [_cache(random_gc(300, nkv=2, seed=1), 2, True, capacity=16) for _ in range(2)]
    for c, _ in others:
        c._rope_inv_freq = c._rope_inv_freq * 0.5
    (_, moved), (_, ref) = others
    moved._gpu_compressed = layer._gpu_compressed
    for t in range(3):
        out = fused_attention_compressed(q, moved, 400 + t)
        assert torch.equal(out.view(-1, 128), decode_layer(q, ref, 400 + t))
    assert not torch.equal(out, fused_attention_compressed(q, layer, 402))


@pytest.mark.parametrize("streaming", [True, False])
@pytest.mark.parametrize("fused", [True, False])
def test_an_update_without_tokens(streaming, fused):
    """Nothing is appended, with and without rows already there."""
    cache, layer = _cache(random_gc(300, nkv=2, seed=1), 2, streaming, capacity=16)
    none = torch.empty(1, 2, 0, 128, dtype=torch.float16, device="cuda")
    k = torch.randn(1, 2, 3, 128, device="cuda").half()
    want = layer.keys.clone()
    cache._fused_decode_update = fused
    layer.update(none, none)
    assert layer.get_seq_length() == 368 and torch.equal(layer.keys, want)
    layer.update(k, k)
    want = layer.keys.clone()
    layer.update(none, none)
    assert layer.get_seq_length() == 371 and torch.equal(layer.keys, want) and want.shape[2] == 371
