"""`Cache`: the reference's drop-in Hugging Face KV cache, backed by sm_100a kernels.

Same constructor, flags, state machine and per-layer tensor dictionary as the
reference's src/shard/cache.py (prefill keeps raw K/V; the first decode step
compresses every layer; later steps append to an 8-bit stream or an fp16
buffer), but every array-sized computation runs in libshard_b200.so:

* K: RoPE removal -> covariance -> eigensolver kernels -> host bit allocation -> int8 basis
  -> projection kernel -> two-stage int4 quantiser + nibble packing;
* V: Hadamard + per-channel normalisation kernel -> k-means kernels;
* decode append: the Lloyd-Max stream quantizer kernel.

There is no CPU path: tensors must live on a CUDA device.
"""
from __future__ import annotations

import math
import threading
from concurrent.futures import ThreadPoolExecutor

import torch
from transformers.cache_utils import Cache as HFCache, CacheLayerMixin

from . import _lib, ops
from ._lib import ShardError
from .rope import dp_bit_allocation, get_rope_inv_freq
from .streaming import get_codebook, layer_signs

KERNEL_HEAD_DIM = 128
KERNEL_RANK_STEP = 32
KERNEL_MAX_RANK = 192


# matrices whose eigensolver launches run side by side: each takes a cluster of 16 SMs, and seven such
# clusters fit a B200 (its GPCs are a little short of 148 SMs' worth of them)
EIGH_GROUP = 7


# sub-vectors whose k-means run side by side: layers of up to 8K tokens share launches, which a single
# short layer leaves mostly empty
KMEANS_POINTS = 16 << 20


# Bytes of un-rotated fp32 keys (twice the size of a layer's prompt keys) that compression holds from the
# covariance to the projection, over the two groups of layers in flight.  Where they would be more (7.5 GB for a
# prompt of 131K tokens) they exist for one layer at a time and are made a second time for its projection: 40 us for
# a layer of 32K tokens, under 1 % of its compression.
ROWS_BYTES = 512 << 20


def gram_matrix(flat, mean):
    """(flat - mean)^T (flat - mean) of the rows of `flat` (n, p), fp32."""
    xc = flat - mean
    # full-precision fp32 products whatever the global TF32 switch says: the trailing
    # eigenvalues are 1e-4 of the leading ones and decide the bit allocation
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        return xc.T @ xc
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev


# Matrices of up to this many rows go to torch.linalg.eigh, which has a Jacobi solver for them.  Its
# vectors are a few 1e-6 of the largest eigenvalue off, and at the 2 bits per coefficient that so few
# heads get, that decides about one code in a hundred: with a more exact solver the reconstructed keys
# move by 4 percent.  Caches of such models have to come out as they always did, so solver, covariance
# and mean stay PyTorch's there; what can be done is to solve the layers side by side (8 matrices of 512
# rows: 170 ms one after the other, 26 ms in eight threads).
TORCH_EIGH_MAX = 512


class TorchEigenpairs:
    """`LeadingEigenpairs` by torch.linalg.eigh, one thread and stream per matrix."""
    _threads, _lock = None, threading.Lock()

    def __init__(self, gram, rank):
        count, p, _ = gram.shape
        self.rank = rank
        self.basis = torch.empty(count, p, rank, dtype=torch.float32, device=gram.device)
        self.host = torch.empty(count, rank, dtype=torch.float32)
        self.inference = torch.is_inference_mode_enabled()     # (the mode is a thread's own, and the result is of this one)
        done = torch.cuda.current_stream().record_event()
        with TorchEigenpairs._lock:
            if TorchEigenpairs._threads is None:
                torch.linalg.eigh(torch.eye(2, device=gram.device))    # PyTorch loads its solver in one thread
                TorchEigenpairs._threads = ThreadPoolExecutor(EIGH_GROUP, thread_name_prefix="shard_b200_eigh")
        self.jobs = [TorchEigenpairs._threads.submit(self._solve, gram[i], i, done) for i in range(count)]

    def _solve(self, gram, i, done):
        stream = _stream_of_thread(gram.device)
        with torch.inference_mode(self.inference), torch.no_grad(), torch.cuda.device(gram.device), torch.cuda.stream(stream):
            stream.wait_event(done)
            w, v = torch.linalg.eigh(gram)
            self.basis[i].copy_(v.flip(-1)[:, :self.rank])
            self.host[i] = w.flip(-1)[:self.rank].cpu()
            stream.synchronize()

    def result(self):
        for job in self.jobs:
            job.result()
        return self.basis, self.host


_thread_local = threading.local()


def _stream_of_thread(device):
    streams = _thread_local.__dict__.setdefault("streams", {})
    if device not in streams:
        streams[device] = torch.cuda.Stream(device)
    return streams[device]


class LeadingEigenpairs:
    """The `rank` largest eigenpairs of each (p, p) matrix of `gram` (count, p, p): launched on the current
    stream when made, waited for by `result` (on the same stream).  `status`: the status word of the kernels
    that made `gram`, looked at then."""

    def __init__(self, gram, rank, status=None):
        self.gram, self.rank = gram, rank
        self.status = None if status is None else word_on_host(status)
        self.basis, self.eigvals, self.flag = ops.eigh_top(gram, rank)

    def result(self):
        """basis (count, p, rank), eigenvectors in the columns, largest first; eigenvalues (count, rank)
        on the host.  Matrices the package's solver reports as too close to degenerate go to
        torch.linalg.eigh."""
        rank = self.rank
        host = torch.cat([self.eigvals, self.flag.unsqueeze(1).float()], dim=1).cpu()
        if self.status is not None and int(self.status):
            raise ShardError("the covariance of the keys is undefined: a wait inside its kernel gave up")
        for i in torch.nonzero(host[:, rank]).flatten().tolist():
            w, v = torch.linalg.eigh(self.gram[i])
            self.basis[i] = v.flip(-1)[:, :rank]
            host[i, :rank] = w.flip(-1)[:rank].cpu()
        return self.basis, host[:, :rank]


def leading_eigenpairs(gram, rank, status=None):
    return TorchEigenpairs(gram, rank) if gram.shape[1] <= TORCH_EIGH_MAX else LeadingEigenpairs(gram, rank, status)


def word_on_host(word):
    """Pinned copy of a device word, valid once the current stream has reached this point."""
    return torch.empty(1, dtype=word.dtype, pin_memory=True).copy_(word, non_blocking=True)


def check_encoded(word):
    """Raise if a wait inside a `k_encode` call gave up (`word`: its scratch's `encode_status`, on the host)."""
    if int(word):
        raise ShardError("the key codes are undefined: a wait inside the projection gave up")


def pca_fit(flat, mean, rank):
    """Top-`rank` principal directions of the rows of `flat` (n, p) around `mean`: the
    eigenvectors of the p x p covariance, largest eigenvalue first, and those eigenvalues.

    Replaces the reference's randomised `torch.svd_lowrank(flat - mean, q=rank, niter=24)`
    (src/shard/cache.py:376: 48 passes over the n x p matrix) by one pass -- the Gram matrix
    (flat - mean)^T (flat - mean), a p x p x n contraction in fp32 -- and a symmetric
    eigensolver on the small p x p matrix (`leading_eigenpairs`).  The subspace is the exact optimum the
    randomised method approximates, so it captures at least as much variance; individual vectors differ
    in sign and, within near-equal eigenvalues, by rotations, which the rest of the path is
    indifferent to (the basis is an input of everything downstream).
    """
    basis, eigvals = leading_eigenpairs(gram_matrix(flat, mean).unsqueeze(0), rank).result()
    return basis[0], (eigvals[0].clamp(min=0) / flat.shape[0]).to(flat.device)


def hadamard(x):
    """Normalised Walsh-Hadamard transform on the last dim (self-inverse).

    Torch expression (the reference's src/shard/cache.py:10-19) for callers; the paths of
    this package run the butterfly inside the kernels.
    """
    d = x.shape[-1]
    h = 1
    while h < d:
        y = x.unflatten(-1, (-1, 2 * h))
        lo, hi = y[..., :h], y[..., h:]
        x = torch.cat([lo + hi, lo - hi], dim=-1).flatten(-2)
        h *= 2
    return x / math.sqrt(d)


def initial_rows(n, k, device, seed=42):
    """The rows `kmeans` starts from: the first k of a seeded permutation of n (src/shard/cache.py:24-25)."""
    g = torch.Generator(device=device).manual_seed(seed)
    return torch.randperm(n, generator=g, device=device)[:k]


def kmeans(data, k, n_iter=30, seed=42, init=None, max_abs=0.0):
    """Lloyd's algorithm as the reference runs it (src/shard/cache.py:21-39), all iterations and the
    stopping rule on the GPU (`ops.kmeans_lloyd`).  Returns the updated centroids and the assignment
    made against the previous ones.  `init` overrides the seeded random initial centroids, `max_abs`
    is a bound on |data| if the caller knows one.
    """
    if init is None:
        init = data[initial_rows(data.shape[0], k, data.device, seed)]
    centroids = init.to(data.device, data.dtype).clone()
    if n_iter < 1:
        return centroids, None
    idx_u8 = ops.kmeans_lloyd(data, centroids, n_iter, max_abs)
    return centroids, idx_u8


_second_streams = {}


def _second_stream(device):
    """The stream compression uses beside the current one, one per device: what is allocated on it comes
    from the allocator's pool of that stream call after call.  High priority: the eigensolver's few CTAs
    are placed before k-means' many."""
    if device not in _second_streams:
        _second_streams[device] = torch.cuda.Stream(device, priority=-1)
    return _second_streams[device]


class CacheLayer(CacheLayerMixin):
    """One layer's K/V: raw after prefill, compressed (`_gpu_compressed`) afterwards."""

    def __init__(self, layer_idx):
        self.layer_idx = layer_idx
        self._keys = None
        self._values = None
        self._prefilled = False
        self._seq_len = 0
        self._cache_ref = None
        self._needs_decompress = False
        self._gpu_compressed = None
        self.is_initialized = False

    def __getstate__(self):
        """For copies of a cache (`copy.deepcopy`, pickle): everything but the launch records, which hold
        addresses; they are made again at the copy's first launch."""
        state = self.__dict__.copy()
        gc = state["_gpu_compressed"]
        if gc is not None:
            state["_gpu_compressed"] = {k: v for k, v in gc.items() if k not in ("_seq", "_launch", "_native")}
        return state

    def __copy__(self):
        new = type(self).__new__(type(self))               # (a shallow copy shares the dictionary itself)
        new.__dict__.update(self.__dict__)
        return new

    # -- lazy materialisation (non-fused reads) -------------------------------
    def _lazy_evict(self):
        c = self._cache_ref
        if c is None or not c._lazy_per_layer:
            return
        last = c._last_accessed_layer
        if last != -1 and last != self.layer_idx:
            prev = c.layers[last]
            if prev._gpu_compressed is not None:
                prev._keys = None
                prev._values = None
                prev._needs_decompress = True
        c._last_accessed_layer = self.layer_idx

    def _ensure_dequant(self, new=None):
        """Full fp16 K/V as [sink | middle | window | stream | fp16 decode buffer]
        (reference: src/shard/cache.py:87-124), one launch: what models without the fused
        hook attend to at every step.  `new`: keys and values of the newest fp16 row, which is still to be
        written."""
        if not self._needs_decompress:
            return
        gc = self._gpu_compressed
        if gc is None:
            return
        from .attention import layer_record, status_word
        c = self._cache_ref
        nkv, hd = c._n_kv_heads, c.head_dim
        dev = gc["k_coeffs"].device
        if dev.type == "cuda" and dev.index != torch.cuda.current_device():
            with torch.cuda.device(dev):
                return self._ensure_dequant(new)
        _lib.require_cuda(gc["k_coeffs"])
        if "k_wprep" not in gc:                            # a dictionary in the reference's form
            attach_kernel_format(gc, nkv)
        pend = gc.get("_pending")
        if pend is not None and pend[2] != gc.get("stream_n", 0) - 1:
            self._flush_pending()
            pend = None
        # decoded tokens of another dtype are not the kernel's: they are appended to what it returns
        other = "decode_k" in gc and not (gc["decode_k"].dtype == gc["decode_v"].dtype == torch.float16)
        seq, shape, rows = layer_record(gc, nkv, hd, dev, with_rows=not other)
        if pend is not None or new is not None:
            shape.append = 1 if pend is not None else 2
            new = pend if pend is not None else new
            seq.new_k, seq.new_v = new[0].data_ptr(), new[1].data_ptr()
        keys = torch.empty(1, nkv, rows, hd, dtype=torch.float16, device=dev)
        values = torch.empty_like(keys)
        # (no RoPE is a rotation by nothing)
        inv_freq = c._inv_freq(dev) if c._rope_inv_freq is not None else torch.zeros(hd // 2, device=dev)
        ops.read_back(seq, shape, inv_freq, get_codebook(hd, 8, dev) if shape.n_stream else None,
                      gc["compress_start"], keys, values, status_word(c, dev))
        gc.pop("_pending", None)                           # (only now: the launch has it)
        if other:
            keys, values = torch.cat([keys, gc["decode_k"]], dim=2), torch.cat([values, gc["decode_v"]], dim=2)
        self._keys, self._values = keys, values
        self._needs_decompress = False

    @property
    def keys(self):
        self._lazy_evict()
        self._ensure_dequant()
        return self._keys

    @keys.setter
    def keys(self, v):
        self._keys = v

    @property
    def values(self):
        self._lazy_evict()
        self._ensure_dequant()
        return self._values

    @values.setter
    def values(self, v):
        self._values = v

    # -- HF entry point --------------------------------------------------------
    def update(self, key_states, value_states, *args, **kwargs):
        """Prefill stores raw K/V; the first decode step compresses; later steps append
        (reference: src/shard/cache.py:138-191)."""
        seq_new = key_states.shape[2]
        c = self._cache_ref
        if seq_new > 1 and not self._prefilled:
            self._prefilled = True
            self.is_initialized = True
            self._seq_len = seq_new
            self._keys = key_states
            self._values = value_states
            return key_states, value_states

        if self._gpu_compressed is None and self.layer_idx == 0 and c is not None and not c._compressed:
            c.compress()

        gc = self._gpu_compressed
        if gc is not None:
            fused = bool(getattr(c, "_fused_decode_update", False))
            if not fused:
                self._lazy_evict()
            streaming = bool(c._streaming)
            # One token of the stream is handed to the launch that reads it next (fused decode or read-back),
            # which quantises it into its row: nothing is launched here, and until then the tensors are the
            # caller's own.  A fp16 row is written before `update` returns: the buffer is public, and the
            # caller may use its tensors for other things before it attends.
            new = None
            native = seq_new == 1 and not (streaming and (c._stream_qjl or c._stream_bits != 8))
            if not (native and _lib.host().append(gc, key_states, value_states, streaming, fused)):
                if streaming:
                    self._stream_append(key_states, value_states, self._seq_len, defer=seq_new == 1)
                else:
                    self._fp16_append(key_states, value_states)
            elif not (streaming or fused):
                new = key_states, value_states             # (the read-back below writes it)
            self._seq_len += seq_new
            self._needs_decompress = True
            if fused:
                if self._keys is not None:                 # an earlier read-back, out of date by now: a layer's fp16
                    self._keys = self._values = None       # keys and values need not be held through the reply
                c._last_accessed_layer = self.layer_idx
                return key_states, value_states
            try:
                self._ensure_dequant(new)
            except BaseException:
                if new is not None:                        # its row has been given out
                    gc["decode_k"][:, :, -1:].copy_(new[0])
                    gc["decode_v"][:, :, -1:].copy_(new[1])
                raise
            return self._keys, self._values

        self._lazy_evict()
        self._ensure_dequant()
        self._seq_len += seq_new
        if self._keys is not None:
            self._keys = torch.cat([self._keys, key_states], dim=2)
            self._values = torch.cat([self._values, value_states], dim=2)
        else:
            self._keys = key_states
            self._values = value_states
        return self._keys, self._values

    def _check_tokens(self, k, v):
        """New tokens of the one sequence, with the cache's heads (the kernels take as many as the cache has)."""
        c = self._cache_ref
        if k.shape[0] != 1:
            raise NotImplementedError("one sequence per Cache (use one Cache per sequence)")
        if k.shape != v.shape or k.shape[1] != c._n_kv_heads or k.shape[3] != c.head_dim:
            raise ShardError(f"expected keys and values (1, {c._n_kv_heads}, s, {c.head_dim}), got {tuple(k.shape)} and {tuple(v.shape)}")

    # -- fp16 decode buffer ------------------------------------------------------
    def _fp16_append(self, k, v):
        """Append (1, nkv, s, hd) new tokens as they are, in place, to a buffer allocated ahead (doubling
        when full); gc["decode_k"] / ["decode_v"] are views of the rows in use."""
        self._check_tokens(k, v)
        self._flush_pending()
        gc, c = self._gpu_compressed, self._cache_ref
        new = k.shape[2]
        n = gc["decode_k"].shape[2] if "decode_k" in gc else 0
        buf_k = gc.get("_dec_buf_k")
        if buf_k is None or n + new > buf_k.shape[2] or buf_k.dtype != k.dtype:
            cap = max(c._decode_capacity, 2 * (n + new))
            B, nkv, _, hd = k.shape
            new_k = torch.empty(B, nkv, cap, hd, dtype=k.dtype, device=k.device)
            new_v = torch.empty(B, nkv, cap, hd, dtype=v.dtype, device=v.device)
            if n:
                new_k[:, :, :n].copy_(gc["decode_k"])
                new_v[:, :, :n].copy_(gc["decode_v"])
            buf_k, gc["_dec_buf_k"], gc["_dec_buf_v"] = new_k, new_k, new_v
        buf_v = gc["_dec_buf_v"]
        buf_k[:, :, n:n + new].copy_(k)
        buf_v[:, :, n:n + new].copy_(v)
        gc["decode_k"] = buf_k[:, :, :n + new]
        gc["decode_v"] = buf_v[:, :, :n + new]

    # -- 8-bit stream -----------------------------------------------------------
    def _flush_pending(self):
        """Write the row of a token whose append was left to the next launch and never got one."""
        gc = self._gpu_compressed
        pend = gc.pop("_pending", None) if gc is not None else None
        if pend is not None:
            k2, v2, slot = pend
            k2 = k2.reshape(-1, k2.shape[-1]).contiguous()       # (nkv, hd)
            v2 = v2.reshape(-1, v2.shape[-1]).contiguous()
            ops.stream_quantize(k2, v2, gc["signs"], get_codebook(k2.shape[-1], 8, k2.device),
                                gc["k_idx_buf"], gc["v_idx_buf"], gc["k_norm_buf"], gc["v_norm_buf"], slot)

    def _grow_stream(self, gc, k, need):
        """(Re)allocate the stream buffers for at least `need` rows: the cache's decode capacity at
        first, doubling afterwards (reference: src/shard/cache.py:220-230, which starts at 16 rows)."""
        c = self._cache_ref
        B, heads, _, hd = k.shape
        dev = k.device
        if "signs" not in gc:
            gc["signs"] = layer_signs(self.layer_idx, hd, dev)
        cap = gc["k_idx_buf"].shape[0] if "k_idx_buf" in gc else 0
        if need <= cap:
            return
        new_cap = max(need, c._decode_capacity if cap == 0 else cap * 2)
        # one allocation: codes of K and V, then their norms
        n_idx, n_norm = new_cap * heads * hd, new_cap * heads
        raw = torch.zeros(2 * n_idx + 4 * n_norm, device=dev, dtype=torch.uint8)
        k_idx, v_idx, norms = raw.split([n_idx, n_idx, 4 * n_norm])
        k_norm, v_norm = norms.view(torch.float16).view(2, new_cap, B, heads).unbind(0)
        for key, new in (("k_idx_buf", k_idx.view(new_cap, B, heads, hd)), ("v_idx_buf", v_idx.view(new_cap, B, heads, hd)),
                         ("k_norm_buf", k_norm), ("v_norm_buf", v_norm)):
            if key in gc:
                new[: cap].copy_(gc[key])
            gc[key] = new

    def _stream_append(self, k, v, position, defer=False):
        """Quantise (1, nkv, s, hd) new tokens into the stream buffers
        (reference: src/shard/cache.py:193-241).  With `defer` the row is reserved and the one
        token is handed to the next launch that reads the stream, whose kernel quantises it."""
        c = self._cache_ref
        if c._stream_qjl:
            raise NotImplementedError("the QJL residual is not part of the CUDA stream path")
        if c._stream_bits != 8:
            raise NotImplementedError("the CUDA stream quantizer emits 8-bit codes only")
        self._check_tokens(k, v)
        if k.dtype != torch.float16 or v.dtype != torch.float16:
            raise NotImplementedError("fp16 models only")
        self._flush_pending()
        gc = self._gpu_compressed
        new = k.shape[2]
        if new == 0:
            return
        s = gc.get("stream_n", 0)
        if "signs" not in gc or s + new > gc["k_idx_buf"].shape[0]:
            self._grow_stream(gc, k, s + new)
        if defer:
            gc["_pending"] = (ops.packed_token(k), ops.packed_token(v), s)
        else:
            ops.stream_quantize_rows(k[0], v[0], gc["signs"], get_codebook(k.shape[3], 8, k.device),
                                     gc["k_idx_buf"], gc["v_idx_buf"], gc["k_norm_buf"], gc["v_norm_buf"], s)
        gc["stream_n"] = s + new

    # -- HF glue -----------------------------------------------------------------
    def get_seq_length(self, *args, **kwargs):
        return self._seq_len

    def get_max_cache_shape(self):
        return None

    def get_mask_sizes(self, query_length, *args, **kwargs):
        if not isinstance(query_length, int):
            query_length = int(query_length.shape[0])
        return self._seq_len + query_length, 0

    def lazy_initialization(self, *args, **kwargs):
        pass

    def reorder_cache(self, beam_idx):
        if self._needs_decompress:
            _ = self.keys
        if self._keys is not None:
            self._keys = self._keys.index_select(0, beam_idx.to(self._keys.device))
        if self._values is not None:
            self._values = self._values.index_select(0, beam_idx.to(self._values.device))


class Cache(HFCache):
    """Compressed KV cache with the reference's constructor and flags
    (src/shard/cache.py:295-336)."""

    def __init__(self, head_dim=128, num_layers=32, n_kv_heads=8, device="cuda",
                 k_target_cr=20.0, max_rank_k=192,
                 v_vq_group_size=4, v_vq_codebook_size=256,
                 sink_tokens=4, residual_window=64, rope_inv_freq=None, decode_capacity=256):
        self.head_dim = head_dim
        # rows the per-layer buffers of decoded tokens (8-bit stream, fp16 decode buffer) are
        # allocated for when the cache is compressed; they double when they run full
        self._decode_capacity = max(16, int(decode_capacity))
        self._num_layers = num_layers
        self._n_kv_heads = n_kv_heads
        self._per_layer_dim = n_kv_heads * head_dim
        self._k_target_cr = k_target_cr
        self._max_rank_k = max_rank_k
        self._v_vq_group_size = v_vq_group_size
        self._v_vq_codebook_size = v_vq_codebook_size
        self._sink_tokens = sink_tokens
        self._residual_window = residual_window
        self._rope_inv_freq = rope_inv_freq
        self._streaming = False
        self._stream_bits = 8
        self._stream_qjl = False
        self._lazy_per_layer = True
        self._full_fused = False
        # how the PCA basis of the keys is fitted: "eigh" (covariance + symmetric eigensolver on the
        # GPU) or "svd_lowrank" (the reference's randomised call)
        self._k_pca = "eigh"
        self._last_accessed_layer = -1
        self._compressed = False
        self._device = device
        self._decode_ws = None
        self._phase = None
        self._phase_key = None
        self._inv_freq_dev = None
        self.compress_seconds = None
        try:
            _lib.host()                                    # loaded here and not inside the first decode step (1.2 ms)
        except (ShardError, OSError):
            pass                                           # (the first call that needs it says what is missing)
        super().__init__(layers=[CacheLayer(i) for i in range(num_layers)])
        for layer in self.layers:
            layer._cache_ref = self

    @classmethod
    def from_model(cls, model, k_target_cr=16.0, **kwargs):
        cfg = model.config
        hd = getattr(cfg, "head_dim", None) or cfg.hidden_size // cfg.num_attention_heads
        return cls(head_dim=hd, num_layers=cfg.num_hidden_layers,
                   n_kv_heads=getattr(cfg, "num_key_value_heads", cfg.num_attention_heads),
                   device=str(next(model.parameters()).device),
                   k_target_cr=k_target_cr,
                   rope_inv_freq=get_rope_inv_freq(model), **kwargs)

    # -- compression ------------------------------------------------------------
    def _check_supported(self, k0):
        if not k0.is_cuda:
            raise ShardError("shard_b200.Cache compresses on a CUDA device; there is no CPU fallback")
        if self.head_dim != KERNEL_HEAD_DIM:
            raise NotImplementedError("kernels are built for head_dim 128")
        if self._v_vq_group_size != 4 or self._v_vq_codebook_size != 256:
            raise NotImplementedError("kernels are built for 256-entry codebooks of 4-channel sub-vectors")
        if k0.dtype != torch.float16:
            raise NotImplementedError("fp16 models only")
        if k0.shape[0] != 1:
            raise NotImplementedError("one sequence per Cache; batch by holding one Cache per sequence")
        if self._rope_inv_freq is None:
            raise NotImplementedError("rope_inv_freq is required by the compressed-score identity")

    def compress(self):
        """Compress every layer's prefill K/V (reference: src/shard/cache.py:338-366)."""
        if self._compressed:
            return
        k0 = self.layers[0]._keys
        if k0 is None:
            return
        B, _, seq, _ = k0.shape
        sink, win = self._sink_tokens, self._residual_window
        if seq <= sink + win + 4:
            return
        self._check_supported(k0)
        start, end = sink, seq - win
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record()
        if self._k_pca == "svd_lowrank":
            for li in range(self._num_layers):
                torch.manual_seed(42 + li)
                k_full, v_full = self.layers[li]._keys, self.layers[li]._values
                kpart = self._compress_k(k_full[0, :, start:end, :], start)
                vpart = self._compress_v(v_full[0, :, start:end, :])
                self._finish_layer(li, kpart, vpart, self._ends(li, end), start, end)
            encoded = None
        else:
            try:
                encoded = self._compress_side_by_side(start, end)
            except BaseException:
                _second_stream(k0.device).wait_stream(torch.cuda.current_stream())   # (as at its end)
                raise
        ev1.record()
        ev1.synchronize()
        if encoded is not None:
            check_encoded(encoded)
        self.compress_seconds = ev0.elapsed_time(ev1) / 1e3
        self._compressed = True

    def _compress_side_by_side(self, start, end):
        """Layers in groups.  The eigensolver of a group's key covariances is a long chain of small steps
        on a few SMs: it runs on a second stream beside the group's value path (k-means) and the next
        group's covariances; the host waits only for the eigenvalues, which decide the bit widths."""
        n_layers = self._num_layers
        main = torch.cuda.current_stream()
        side = _second_stream(main.device)
        n_groups = -(-n_layers // EIGH_GROUP)
        bounds = [n_layers * g // n_groups for g in range(n_groups + 1)]

        n, p = end - start, self._per_layer_dim
        rank = min(self._max_rank_k, p, n - 1)
        side.wait_stream(main)
        dev = main.device
        inv_freq = self._inv_freq(dev)
        cov_ws = enc_ws = None
        bases = []
        in_flight = max(hi - lo for lo, hi in zip(bounds[:-2] or bounds, bounds[2:] or bounds[1:]))
        keep_rows = 4 * n * p * in_flight <= ROWS_BYTES

        def keys(li):
            return self.layers[li]._keys[0, :, start:end, :]

        def covariances(g):
            nonlocal cov_ws
            count = bounds[g + 1] - bounds[g]
            flat = torch.empty(count if keep_rows else 1, n, p, dtype=torch.float32, device=dev)
            mean = torch.empty(count, p, dtype=torch.float32, device=dev)
            mean_f16 = torch.empty(count, p, dtype=torch.float16, device=dev)
            gram = torch.empty(count, p, p, dtype=torch.float32, device=dev)
            rows = list(zip(flat.expand(count, n, p).unbind(0), mean.unbind(0), mean_f16.unbind(0)))
            for li, (f, m, m16), gr in zip(range(bounds[g], bounds[g + 1]), rows, gram.unbind(0)):
                if p <= TORCH_EIGH_MAX:
                    ops.undo_rope(keys(li), start, inv_freq, out=f)
                    torch.mean(f, dim=0, out=m)
                    m16.copy_(m)
                    gr.copy_(gram_matrix(f, m))
                else:
                    cov_ws = ops.k_covariance(keys(li), start, inv_freq, f, m, m16, gr, cov_ws)
            return rows, gram, main.record_event()

        # The covariances first, with the eigensolver right behind them: they are the long chain.
        ready = covariances(0)
        with torch.cuda.stream(side):
            # every layer's k-means starts from the same rows (same seed, same number of sub-vectors)
            init_rows = initial_rows(n * p // self._v_vq_group_size, self._v_vq_codebook_size, main.device)
            drawn = side.record_event()
        for g in range(n_groups):
            rows, gram, done = ready
            side.wait_event(done)
            with torch.cuda.stream(side):
                solved = leading_eigenpairs(gram, rank, None if cov_ws is None else ops.covariance_status(cov_ws))
            if g == 0:
                main.wait_event(drawn)
                # (the state the global generator is left in: the reference seeds it for every layer's randomised SVD)
                torch.manual_seed(42 + n_layers - 1)
            vparts = self._compress_v_layers([self.layers[li]._values[0, :, start:end, :]
                                              for li in range(bounds[g], bounds[g + 1])], init_rows=init_rows)
            ends = [self._ends(li, end) for li in range(bounds[g], bounds[g + 1])]
            if g + 1 < n_groups:
                ready = covariances(g + 1)
            with torch.cuda.stream(side):
                basis, eig_host = solved.result()
                fin = side.record_event()
            main.wait_event(fin)
            bases.append(basis)
            for i, li in enumerate(range(bounds[g], bounds[g + 1])):
                if not keep_rows:
                    ops.undo_rope(keys(li), start, inv_freq, out=rows[i][0])
                kpart, enc_ws = self._quantise_k(*rows[i], basis[i], eig_host[i].clamp(min=0) / n, enc_ws)
                self._finish_layer(li, kpart, vparts[i], ends[i], start, end)
        # What was made on the second stream and read on this one (the bases, the rows drawn) goes back to the
        # allocator behind everything enqueued here: other threads of the device share the second stream, and
        # their allocations there come after this wait.
        side.wait_stream(main)
        return word_on_host(ops.encode_status(enc_ws))

    def _ends(self, li, end):
        layer = self.layers[li]
        return ops.kv_ends(layer._keys[0], layer._values[0], self._sink_tokens, self._residual_window, end)

    def _finish_layer(self, li, kpart, vpart, ends, start, end):
        sink_k, sink_v, win_k, win_v = ends
        self._build_gpu_format(self.layers[li], kpart, vpart, sink_k=sink_k, sink_v=sink_v, win_k=win_k, win_v=win_v,
                               n_comp=end - start, batch=1, start=start)

    def _compress_k(self, k_mid, pos_start, basis=None):
        """Un-rotate, fit a joint PCA over all KV heads, quantise basis to int8 and
        coefficients to int4 (reference: src/shard/cache.py:368-396, 416-420).

        k_mid: (nkv, n, hd) fp16 view.  `basis` (dim, rank) overrides the SVD (used by
        the parity tests, which take the basis as given).
        """
        dev = k_mid.device
        inv_freq = self._inv_freq(dev)
        flat = ops.undo_rope(k_mid, pos_start, inv_freq)
        n, p = flat.shape
        mean = flat.mean(dim=0)
        rank = min(self._max_rank_k, p, n - 1)
        if basis is None and self._k_pca == "svd_lowrank":
            # the reference's own call (src/shard/cache.py:376): randomised, 24 power iterations
            _, S, V = torch.svd_lowrank(flat - mean, q=rank, niter=24)
            basis = V[:, :rank]
            eigvals = (S[:rank].float() ** 2) / n
        elif basis is None:
            basis, eigvals = pca_fit(flat, mean, rank)
        else:
            basis = basis.to(dev, torch.float32)[:, :rank]
            eigvals = ((flat - mean) @ basis).pow(2).sum(dim=0) / n
        kpart, workspace = self._quantise_k(flat, mean, mean.half(), basis, eigvals)
        check_encoded(ops.encode_status(workspace).cpu())
        return kpart

    def _quantise_k(self, flat, mean, mean_f16, basis, eigvals, workspace=None):
        """Bit allocation, int8 basis, projection and int4 codes of un-rotated keys `flat` (n, dim)."""
        n = flat.shape[0]
        budget = max(64, int(self._per_layer_dim * 16 / self._k_target_cr))
        alloc = dp_bit_allocation(eigvals, budget)
        keep = sum(1 for b in alloc if b > 0)
        keep -= keep & 1
        if keep <= 0:
            raise ShardError("bit allocation kept no PCA component")
        alloc = alloc[:keep]
        basis = basis[:, :keep]
        basis_q, scale, basis_f16, packed, coeff_scale, wprep, workspace = ops.k_encode(
            flat, mean, mean_f16, basis if basis.stride(1) == 1 else basis.contiguous(), alloc, workspace)
        return {"k_basis_q": basis_q, "k_scale": scale, "k_basis_f16": basis_f16, "k_mean": mean_f16, "k_alloc": alloc,
                "k_coeffs": packed, "k_coeff_scale": coeff_scale, "k_wprep": wprep, "k_n_total": n}, workspace

    def _compress_v(self, v_mid, init_centroids=None, init_rows=None):
        """Hadamard-rotate, normalise per channel and vector-quantise 4-channel groups
        (reference: src/shard/cache.py:398-404, 41-52).  v_mid: (nkv, n, hd) fp16 view; `init_rows` are the
        sub-vectors to start from if the caller has drawn them (`initial_rows`)."""
        return self._compress_v_layers([v_mid], init_centroids, init_rows)[0]

    def _compress_v_layers(self, v_mids, init_centroids=None, init_rows=None):
        """`_compress_v` of several layers; short prompts' layers go through k-means side by side."""
        nkv, n, hd = v_mids[0].shape
        gs = self._v_vq_group_size
        n_sub = nkv * n * (hd // gs)
        side_by_side = max(1, min(len(v_mids), KMEANS_POINTS // n_sub))
        parts = []
        for i in range(0, len(v_mids), side_by_side):
            vs = v_mids[i:i + side_by_side]
            x = torch.empty(len(vs), n_sub, gs, dtype=torch.float32, device=vs[0].device)
            ch_max = [ops.v_hadamard_normalise(v, out=x[j])[1].half() for j, v in enumerate(vs)]
            if init_centroids is not None:
                centroids = init_centroids.to(x.device, torch.float32).clone().unsqueeze(0)
            else:
                if init_rows is None:
                    init_rows = initial_rows(n_sub, self._v_vq_codebook_size, x.device)
                centroids = x[:, init_rows].contiguous()
            # the data is normalised by the channels' largest magnitudes
            idx = ops.kmeans_lloyd(x, centroids, 30, 1.0)
            parts += [{"centroids": centroids[j].half(), "packed": idx[j], "ch_maxabs": ch_max[j], "shape": (nkv, n, hd),
                       "group_size": gs, "bits": 8, "n_orig": n_sub} for j in range(len(vs))]
        return parts

    def _build_gpu_format(self, layer, k, v, sink_k, sink_v, win_k, win_v, n_comp, batch, start):
        """Assemble the per-layer tensor dictionary (reference: src/shard/cache.py:406-460)
        and the kernel-side prepared weights."""
        nkv, hd = self._n_kv_heads, self.head_dim
        keep = len(k["k_alloc"])
        ng = hd // v["group_size"]
        basis_f16 = k["k_basis_f16"]
        coeff_scale_f16 = k["k_coeff_scale"]
        gc = {
            "k_coeffs": k["k_coeffs"],
            "k_coeff_scale": coeff_scale_f16,
            "k_coeffs_shape": (k["k_n_total"], keep),
            "k_basis_q": k["k_basis_q"],
            "k_basis_scale": k["k_scale"],
            "k_basis_f16": basis_f16,
            "k_mean": k["k_mean"],
            "k_mean_f16": k["k_mean"],
            "k_alloc": k["k_alloc"],
            "v_qdata": v,
            "v_packed": v["packed"],
            "v_indices_u8": v["packed"].view(nkv, n_comp, ng),
            "v_centroids_f16": v["centroids"].contiguous(),
            "v_ch_f16": v["ch_maxabs"].view(nkv, hd).contiguous(),
            "sink_k": sink_k, "sink_v": sink_v, "win_k": win_k, "win_v": win_v,
            "n_compress": n_comp, "batch": batch, "compress_start": start,
        }
        attach_kernel_format(gc, nkv, k["k_wprep"])
        layer._gpu_compressed = gc
        layer._keys = None
        layer._values = None
        layer._needs_decompress = True

    def check(self):
        """Raise `ShardError` if a decode launch on this cache gave up on one of its bounded
        in-kernel waits since the last check (its output is then undefined).  Waits for the
        current stream; call it once per step or per request, not per layer."""
        if self._decode_ws is not None:
            ops.decode_status_check(self._decode_ws)

    def _inv_freq(self, dev):
        if self._inv_freq_dev is None or self._inv_freq_dev.device != torch.device(dev):
            self._inv_freq_dev = self._rope_inv_freq.to(dev, torch.float32).contiguous()
        return self._inv_freq_dev

    # -- accounting (reference: src/shard/cache.py:462-539) -------------------------
    @staticmethod
    def _nb(t):
        return t.nelement() * t.element_size()

    _STORAGE_KEYS = ("k_coeffs", "k_coeff_scale", "k_basis_q", "k_basis_scale", "k_mean", "v_packed",
                     "sink_k", "sink_v", "win_k", "win_v")

    def clean_memory_bytes(self):
        """Storage-only size of the compressed cache (no decode-time scratch)."""
        total, has = 0, False
        for layer in self.layers:
            gc = layer._gpu_compressed
            if gc is None:
                continue
            has = True
            total += sum(self._nb(gc[k]) for k in self._STORAGE_KEYS)
            total += self._nb(gc["v_qdata"]["ch_maxabs"]) + self._nb(gc["v_qdata"]["centroids"])
        if has:
            return total
        return sum(self._nb(l._keys) + self._nb(l._values) for l in self.layers if l._keys is not None)

    def memory_bytes(self):
        """Everything resident for the cache: storage, the decode-time copies this
        implementation keeps (fp16 basis, fragment-ordered weights) and the stream."""
        total, has = 0, False
        for layer in self.layers:
            gc = layer._gpu_compressed
            if gc is None:
                continue
            has = True
            total += sum(self._nb(gc[k]) for k in self._STORAGE_KEYS)
            total += self._nb(gc["v_qdata"]["ch_maxabs"]) + self._nb(gc["v_qdata"]["centroids"])
            for k in ("k_basis_f16", "k_mean_f16", "v_centroids_f16", "v_ch_f16", "k_wprep"):
                if k in gc:
                    total += self._nb(gc[k])
            if "k_coeffs_padded" in gc:
                total += self._nb(gc["k_coeffs_padded"])
            if "k_idx_buf" in gc:
                s = gc.get("stream_n", 0)
                bpv = self._stream_bits / 8.0
                for k in ("k_idx_buf", "v_idx_buf"):
                    total += int(gc[k][:s].nelement() * bpv)
                for k in ("k_norm_buf", "v_norm_buf"):
                    total += self._nb(gc[k][:s])
            if "decode_k" in gc:
                total += self._nb(gc["decode_k"]) + self._nb(gc["decode_v"])
        if has:
            return total
        return sum(self._nb(l._keys) + self._nb(l._values) for l in self.layers if l._keys is not None)

    def fp16_equivalent_bytes(self):
        gc = self.layers[0]._gpu_compressed
        if gc is not None:
            seq = gc["n_compress"] + self._sink_tokens + self._residual_window + gc.get("stream_n", 0)
        elif self.layers[0]._keys is not None:
            seq = self.layers[0]._keys.shape[2]
        else:
            return 0
        return seq * self._n_kv_heads * self.head_dim * 4 * self._num_layers

    def compress_ratio(self):
        return self.fp16_equivalent_bytes() / max(self.memory_bytes(), 1)

    def clean_compress_ratio(self):
        gc = self.layers[0]._gpu_compressed
        if gc is not None:
            seq = gc["n_compress"] + self._sink_tokens + self._residual_window
            fp16_bytes = seq * self._n_kv_heads * self.head_dim * 4 * self._num_layers
            return fp16_bytes / max(self.clean_memory_bytes(), 1)
        return self.compress_ratio()


def attach_kernel_format(gc, nkv, wprep=None):
    """Add what the decode kernel needs beyond the reference's dictionary: the
    fragment-ordered weights, and (only when the kept rank is not a multiple of 32) a
    copy of the coefficients padded with zero nibbles to the next multiple.  `wprep`: those weights
    if the caller has them already."""
    n_total, keep = gc["k_coeffs_shape"]
    basis = gc["k_basis_f16"]
    cscale = gc["k_coeff_scale"].to(torch.float16).contiguous()
    rank_k = ((keep + KERNEL_RANK_STEP - 1) // KERNEL_RANK_STEP) * KERNEL_RANK_STEP
    if rank_k > KERNEL_MAX_RANK:
        raise NotImplementedError("kernels support PCA ranks up to 192")
    coeffs = gc["k_coeffs"]
    if rank_k != keep:
        pad = rank_k - keep
        basis = torch.cat([basis, basis.new_zeros(basis.shape[0], pad)], dim=1).contiguous()
        cscale = torch.cat([cscale, cscale.new_zeros(pad)]).contiguous()
        rows = coeffs.view(n_total, keep // 2)
        coeffs = torch.cat([rows, rows.new_full((n_total, pad // 2), 0x88)], dim=1).contiguous().view(-1)
        gc["k_coeffs_padded"] = coeffs
    gc["k_rank_kernel"] = rank_k
    gc["k_coeffs_kernel"] = coeffs
    gc["k_wprep"] = wprep if wprep is not None else ops.decode_prepare(basis, cscale, gc["k_mean_f16"], nkv, rank_k)
    gc["_fresh"] = True      # the next decode launch follows the kernels that wrote these tensors
    return gc
