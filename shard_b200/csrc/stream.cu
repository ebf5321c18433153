// 8-bit Lloyd-Max quantiser for tokens appended during decode, and its inverse; the append of tokens kept as
// they are.
//
// One warp handles one (tensor, KV head) vector of 128 channels; lane l owns
// channels 4l..4l+3.  Every arithmetic step that decides a code is a single
// correctly rounded fp32 operation in a fixed order, so codes are reproducible
// bit for bit from the same fp16 input:
//   n   = fp32(sqrt(sum of squares in fp64))      (exact sum: fp16 squares fit)
//   u   = x / n                                   (IEEE division)
//   rot = H128(u * signs) / fp32(sqrt(128))       (butterfly order h = 1..64)
//   idx = nearest codebook entry, ties to the right neighbour
#include "tcgen05.cuh"

namespace shard {

struct StreamParams {
  ShardSeq one;
  const ShardSeq* table;
  const float* codebook;
  int nkv;
  int slot;
};

__global__ void __launch_bounds__(128) stream_quantize_kernel(const __grid_constant__ StreamParams p) {
  __shared__ float cb[256];
  const ShardSeq& s = p.table ? p.table[blockIdx.y] : p.one;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) cb[i] = p.codebook[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int vec = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // 0 .. 2*nkv-1
  if (vec >= 2 * p.nkv) return;
  const bool is_v = vec >= p.nkv;
  const int kv = is_v ? vec - p.nkv : vec;
  const __half* src = reinterpret_cast<const __half*>(is_v ? s.new_v : s.new_k) + kv * HD;
  uint8_t* idx_out = (is_v ? s.st_v_idx : s.st_k_idx) + ((size_t)p.slot * p.nkv + kv) * HD;
  __half* norm_out = reinterpret_cast<__half*>(is_v ? s.st_v_norm : s.st_k_norm) + (size_t)p.slot * p.nkv + kv;
  quantize_vec_warp(src, s.signs, cb, idx_out, norm_out, lane);
}

// Several new tokens at once (a forward over more than one token): token t of `k` / `v` (element strides per
// KV head and token, channels contiguous) goes to row slot + t; a warp per vector.
struct StreamRowsParams {
  const __half *k, *v;
  int64_t k_head, k_tok, v_head, v_tok;
  const float *signs, *codebook;
  uint8_t *k_idx, *v_idx;
  __half *k_norm, *v_norm;
  int nkv, slot, n_tok;
};

__global__ void __launch_bounds__(128) stream_quantize_rows_kernel(const __grid_constant__ StreamRowsParams p) {
  __shared__ float cb[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) cb[i] = p.codebook[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const long long n_vec = 2ll * p.nkv * p.n_tok;
  for (long long u = (long long)blockIdx.x * 4 + (threadIdx.x >> 5); u < n_vec; u += (long long)gridDim.x * 4) {
    const long long t = u / (2 * p.nkv);
    const int vec = (int)(u - t * (2 * p.nkv));
    const bool is_v = vec >= p.nkv;
    const int kv = is_v ? vec - p.nkv : vec;
    const __half* src = is_v ? p.v + kv * p.v_head + t * p.v_tok : p.k + kv * p.k_head + t * p.k_tok;
    const size_t row = (size_t)(p.slot + t) * p.nkv + kv;
    quantize_vec_warp(src, p.signs, cb, (is_v ? p.v_idx : p.k_idx) + row * HD, (is_v ? p.v_norm : p.k_norm) + row, lane);
  }
}

// New tokens of a cache that keeps them as they are: keys and values to rows row .. row + n_tok - 1 of the
// fp16 decode buffers [nkv][cap][128], a warp per vector.  One launch instead of two strided copies, and it
// lets the decode launch behind it place its CTAs meanwhile.  Bound: one launch's latency, 1.7 us a layer (12K tokens
// of context, 4 KV heads, 8 layers: 142 us a step; 129 us with the row written by the decode launch, which is
// sound only as long as the caller leaves its tensors alone until then).
struct AppendRowsParams {
  const __half *k, *v;
  int64_t k_head, k_tok, v_head, v_tok;
  __half *dst_k, *dst_v;
  int64_t cap, row;
  int nkv, n_tok;
};

__global__ void __launch_bounds__(256) append_rows_kernel(const __grid_constant__ AppendRowsParams p) {
  griddep_launch();
  griddep_wait();                                        // the tokens may come from the kernel in front
  const int lane = threadIdx.x & 31;
  const long long half_units = (long long)p.nkv * p.n_tok;
  for (long long u = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); u < 2 * half_units; u += (long long)gridDim.x * 8) {
    const bool is_v = u >= half_units;
    const long long w = is_v ? u - half_units : u;
    const long long kv = w / p.n_tok, t = w - kv * p.n_tok;
    const __half* src = is_v ? p.v + kv * p.v_head + t * p.v_tok : p.k + kv * p.k_head + t * p.k_tok;
    __half* dst = (is_v ? p.dst_v : p.dst_k) + (kv * p.cap + p.row + t) * HD;
    reinterpret_cast<uint2*>(dst)[lane] = reinterpret_cast<const uint2*>(src)[lane];
  }
}

// out[kv][t][:] = fp16( fp32(fp16(H128(cb[idx]) / sqrt(128) * signs)) * fp32(norm) )
__global__ void __launch_bounds__(128) stream_dequant_kernel(const uint8_t* __restrict__ idx,
                                                             const __half* __restrict__ norm,
                                                             const float* __restrict__ signs,
                                                             const float* __restrict__ codebook,
                                                             int n_stream, int nkv, __half* __restrict__ out) {
  __shared__ float cb[256];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) cb[i] = codebook[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int vec = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // t * nkv + kv
  if (vec >= n_stream * nkv) return;
  const int t = vec / nkv, kv = vec - t * nkv;
  const uint32_t codes = *reinterpret_cast<const uint32_t*>(idx + (size_t)vec * HD + 4 * lane);
  float x[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) x[i] = cb[(codes >> (8 * i)) & 0xff];
  fwht128_lane4(x, lane);
  const float4 sg = *reinterpret_cast<const float4*>(signs + 4 * lane);
  const float sgn[4] = {sg.x, sg.y, sg.z, sg.w};
  const float nrm = __half2float(norm[vec]);
  __half o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half unit = __float2half_rn(__fmul_rn(__fdiv_rn(x[i], SQRT_HD), sgn[i]));
    o[i] = __float2half_rn(__fmul_rn(__half2float(unit), nrm));
  }
  uint2 w;
  w.x = (uint32_t)__half_as_ushort(o[0]) | ((uint32_t)__half_as_ushort(o[1]) << 16);
  w.y = (uint32_t)__half_as_ushort(o[2]) | ((uint32_t)__half_as_ushort(o[3]) << 16);
  *reinterpret_cast<uint2*>(out + ((size_t)kv * n_stream + t) * HD + 4 * lane) = w;
}

}  // namespace shard

extern "C" int shard_b200_stream_quantize(const ShardSeq* seqs, int32_t batch, int32_t nkv, int32_t slot,
                                          const float* codebook, void* stream) {
  if (!seqs || !codebook || batch < 1 || nkv < 1 || slot < 0) return SHARD_E_ARG;
  shard::StreamParams p{};
  if (batch == 1) {
    p.one = *seqs;
    p.table = nullptr;
    if (!p.one.new_k || !p.one.new_v || !p.one.st_k_idx || !p.one.st_v_idx || !p.one.st_k_norm ||
        !p.one.st_v_norm || !p.one.signs)
      return SHARD_E_ARG;
  } else {
    p.table = seqs;
  }
  p.codebook = codebook;
  p.nkv = nkv;
  p.slot = slot;
  dim3 grid((2 * nkv + 3) / 4, batch);
  shard::stream_quantize_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(p);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_stream_quantize_rows(const void* k_f16, const void* v_f16, int64_t k_head_stride,
                                               int64_t k_tok_stride, int64_t v_head_stride, int64_t v_tok_stride,
                                               int32_t n_tok, int32_t nkv, const float* signs, const float* codebook,
                                               uint8_t* k_idx, uint8_t* v_idx, void* k_norm, void* v_norm, int32_t slot,
                                               void* stream) {
  if (!k_f16 || !v_f16 || !signs || !codebook || !k_idx || !v_idx || !k_norm || !v_norm || n_tok < 0 || nkv < 1 || slot < 0 ||
      n_tok > INT32_MAX - slot)
    return SHARD_E_ARG;
  if (((uintptr_t)k_f16 & 7) || ((uintptr_t)v_f16 & 7) || (k_head_stride & 3) || (k_tok_stride & 3) || (v_head_stride & 3) ||
      (v_tok_stride & 3) || ((uintptr_t)k_idx & 3) || ((uintptr_t)v_idx & 3) || ((uintptr_t)signs & 15))
    return SHARD_E_ALIGN;
  if (n_tok == 0) return SHARD_OK;
  shard::StreamRowsParams p{(const __half*)k_f16, (const __half*)v_f16, k_head_stride, k_tok_stride, v_head_stride, v_tok_stride,
                            signs, codebook, k_idx, v_idx, (__half*)k_norm, (__half*)v_norm, nkv, slot, n_tok};
  shard::stream_quantize_rows_kernel<<<shard::capped_blocks((2ll * nkv * n_tok + 3) / 4, 16), 128, 0, (cudaStream_t)stream>>>(p);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_append_rows(const void* k_f16, const void* v_f16, int64_t k_head_stride, int64_t k_tok_stride,
                                      int64_t v_head_stride, int64_t v_tok_stride, int32_t n_tok, int32_t nkv, void* dec_k_f16,
                                      void* dec_v_f16, int64_t dec_cap, int64_t row, void* stream) {
  if (!k_f16 || !v_f16 || !dec_k_f16 || !dec_v_f16 || n_tok < 0 || nkv < 1 || row < 0 || row + n_tok > dec_cap) return SHARD_E_ARG;
  if ((((uintptr_t)k_f16 | (uintptr_t)v_f16 | (uintptr_t)dec_k_f16 | (uintptr_t)dec_v_f16) & 7) ||
      ((k_head_stride | k_tok_stride | v_head_stride | v_tok_stride) & 3))
    return SHARD_E_ALIGN;
  if (n_tok == 0) return SHARD_OK;
  shard::AppendRowsParams p{(const __half*)k_f16, (const __half*)v_f16, k_head_stride, k_tok_stride, v_head_stride, v_tok_stride,
                            (__half*)dec_k_f16, (__half*)dec_v_f16, dec_cap, row, nkv, n_tok};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(shard::capped_blocks((2ll * nkv * n_tok + 7) / 8, 8));
  cfg.blockDim = dim3(256);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, shard::append_rows_kernel, p);
  return e == cudaSuccess ? SHARD_OK : (int)e;
}

extern "C" int shard_b200_stream_dequant(const uint8_t* idx, const void* norm_f16, const float* signs,
                                         const float* codebook, int32_t n_stream, int32_t nkv,
                                         void* out_f16, void* stream) {
  if (!idx || !norm_f16 || !signs || !codebook || !out_f16 || nkv < 1 || n_stream < 0) return SHARD_E_ARG;
  if (n_stream == 0) return SHARD_OK;
  const int vecs = n_stream * nkv;
  shard::stream_dequant_kernel<<<(vecs + 3) / 4, 128, 0, (cudaStream_t)stream>>>(
      idx, (const __half*)norm_f16, signs, codebook, n_stream, nkv, (__half*)out_f16);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}
