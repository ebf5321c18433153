// Prefill compressor kernels: the two-stage int4
// quantiser with nibble packing, Hadamard + per-channel normalisation of V and
// nearest-centroid VQ assignment.
//
// Every stage that ends in an integer code uses explicitly rounded fp32
// operations (__fmul_rn/__fadd_rn/__fdiv_rn, rintf) in the order the reference's
// PyTorch code performs them, so that the codes are bit-identical for identical
// fp32 inputs.  Reductions that decide codes (min, max, max-abs) are
// order-independent.
#include <new>
#include <vector>

#include "common.cuh"

namespace shard {

// ---------------------------------------------------------------------------
// K quantiser
// ---------------------------------------------------------------------------
// Monotone map float -> uint32 so that unsigned atomicMin/atomicMax order floats.
__device__ __forceinline__ uint32_t f2ord(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// ws layout (uint32): [0,keep) ordered min, [keep,2keep) ordered max, [2keep,3keep) max|xhat| bits
__global__ void kq_init_kernel(uint32_t* ws, int keep) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < keep) { ws[j] = 0xffffffffu; ws[keep + j] = 0u; ws[2 * keep + j] = 0u; }
}

// the same, and the bit widths handed over as a kernel argument; passes the projection's status word on
struct KqBits { uint8_t b[256]; };
__global__ void kq_init_bits_kernel(uint32_t* ws, int keep, const __grid_constant__ KqBits bits, int32_t* __restrict__ alloc,
                                    const int* __restrict__ gave_up, int* __restrict__ status) {
  const int j = threadIdx.x;
  if (j == 0 && *gave_up) *status = 1;
  if (j < keep) { ws[j] = 0xffffffffu; ws[keep + j] = 0u; ws[2 * keep + j] = 0u; alloc[j] = bits.b[j]; }
}

// Rows per block: a short prompt needs the blocks (1K tokens: 62 us with 32 rows, 63 with 64 and without the eight
// loads in flight per thread), a long one more rows per atomic (32K: 80 us with 64, 84 with 32; 131K: 231, 238).
static inline int kq_rows(int n) { return n >= 16384 ? 64 : 32; }

__global__ void __launch_bounds__(256) kq_minmax_kernel(const float* __restrict__ proj, int n, int keep, int rows,
                                                        uint32_t* __restrict__ ws) {
  const int r0 = blockIdx.x * rows;
  for (int j = threadIdx.x; j < keep; j += blockDim.x) {
    float lo = __int_as_float(0x7f800000), hi = neg_inf();
    const int r1 = min(r0 + rows, n);
#pragma unroll 8
    for (int r = r0; r < r1; ++r) {
      const float v = proj[(size_t)r * keep + j];
      lo = fminf(lo, v); hi = fmaxf(hi, v);
    }
    atomicMin(ws + j, f2ord(lo));
    atomicMax(ws + keep + j, f2ord(hi));
  }
}

__device__ __forceinline__ float kq_xhat(float x, float lo, float rng, float levels) {
  float unit = __fdiv_rn(__fsub_rn(x, lo), rng);
  unit = fminf(fmaxf(unit, 0.f), 1.f);
  float code = rintf(__fmul_rn(unit, levels));
  code = fminf(fmaxf(code, 0.f), levels);
  return __fadd_rn(__fmul_rn(__fdiv_rn(code, levels), rng), lo);
}

__global__ void __launch_bounds__(256) kq_absmax_kernel(const float* __restrict__ proj,
                                                        const int32_t* __restrict__ alloc, int n, int keep, int rows,
                                                        uint32_t* __restrict__ ws) {
  const int r0 = blockIdx.x * rows;
  for (int j = threadIdx.x; j < keep; j += blockDim.x) {
    const int bits = alloc[j];
    if (bits == 0) continue;
    const float lo = ord2f(ws[j]);
    const float rng = fmaxf(__fsub_rn(ord2f(ws[keep + j]), lo), 1e-6f);
    const float levels = (float)((1 << bits) - 1);
    float am = 0.f;
    const int r1 = min(r0 + rows, n);
#pragma unroll 8
    for (int r = r0; r < r1; ++r) am = fmaxf(am, fabsf(kq_xhat(proj[(size_t)r * keep + j], lo, rng, levels)));
    atomicMax(ws + 2 * keep + j, __float_as_uint(am));  // non-negative floats order as integers
  }
}

__global__ void kq_scale_kernel(const uint32_t* __restrict__ ws, int keep, float* __restrict__ coeff_scale,
                                __half* __restrict__ scale_f16) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= keep) return;
  const float s = __fdiv_rn(fmaxf(__uint_as_float(ws[2 * keep + j]), 1e-6f), 7.0f);
  coeff_scale[j] = s;
  if (scale_f16) scale_f16[j] = __float2half_rn(s);
}

__global__ void __launch_bounds__(256) kq_pack_kernel(const float* __restrict__ proj,
                                                      const int32_t* __restrict__ alloc, int n, int keep,
                                                      const uint32_t* __restrict__ ws,
                                                      const float* __restrict__ coeff_scale,
                                                      uint8_t* __restrict__ packed) {
  const int half = keep >> 1;
  const size_t total = (size_t)n * half;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t r = i / half;
    const int j = (int)(i - r * half) * 2;
    const float2 x = *reinterpret_cast<const float2*>(proj + r * keep + j);
    int q[2];
    const float xv[2] = {x.x, x.y};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int bits = alloc[j + e];
      float xh = 0.f;
      if (bits) {
        const float lo = ord2f(ws[j + e]);
        const float rng = fmaxf(__fsub_rn(ord2f(ws[keep + j + e]), lo), 1e-6f);
        xh = kq_xhat(xv[e], lo, rng, (float)((1 << bits) - 1));
      }
      float v = rintf(__fdiv_rn(xh, coeff_scale[j + e]));
      v = fminf(fmaxf(v, -7.f), 7.f);
      q[e] = (int)v;
    }
    packed[i] = (uint8_t)(((q[0] + 8) & 15) | (((q[1] + 8) & 15) << 4));
  }
}

// int8 basis: per column scale = max(max|b|, 1e-6) / 127, code = clamp(rint(b / scale), +-127); and what
// the projection and the decode kernels take: w = code * scale (fp32) and fp16(code) * fp16(scale).
// A block takes 16 columns, 64 rows at a time.
__global__ void __launch_bounds__(1024) k_basis_quantise_kernel(const float* __restrict__ basis, int64_t stride, int dim, int keep,
                                                                int8_t* __restrict__ basis_q, __half* __restrict__ scale_f16,
                                                                float* __restrict__ w, __half* __restrict__ basis_f16) {
  constexpr int KEPT = 16;                     // rows a thread keeps in registers between the passes (dim <= 1024)
  __shared__ float mx[64][17];
  const int cl = threadIdx.x & 15, c = blockIdx.x * 16 + cl, r0 = threadIdx.x >> 4;
  const bool live = c < keep;
  float v[KEPT], m = 0.f;
#pragma unroll
  for (int i = 0; i < KEPT; ++i) {
    const int r = r0 + 64 * i;
    v[i] = live && r < dim ? basis[(size_t)r * stride + c] : 0.f;
    m = fmaxf(m, fabsf(v[i]));
  }
  if (live)
    for (int r = r0 + 64 * KEPT; r < dim; r += 64) m = fmaxf(m, fabsf(basis[(size_t)r * stride + c]));
  mx[r0][cl] = m;
  __syncthreads();
  for (int h = 32; h > 0; h >>= 1) {
    if (r0 < h) mx[r0][cl] = fmaxf(mx[r0][cl], mx[r0 + h][cl]);
    __syncthreads();
  }
  m = mx[0][cl];
  if (!live) return;
  const float scale = __fdiv_rn(fmaxf(m, 1e-6f), 127.0f);
  const __half s16 = __float2half_rn(scale);
  if (r0 == 0) scale_f16[c] = s16;
  auto put = [&](int r, float x) {
    float q = rintf(__fdiv_rn(x, scale));
    q = fminf(fmaxf(q, -127.f), 127.f);
    const size_t o = (size_t)r * keep + c;
    basis_q[o] = (int8_t)(int)q;
    w[o] = __fmul_rn(q, scale);
    basis_f16[o] = __hmul(__float2half_rn(q), s16);
  };
#pragma unroll
  for (int i = 0; i < KEPT; ++i)
    if (r0 + 64 * i < dim) put(r0 + 64 * i, v[i]);
  for (int r = r0 + 64 * KEPT; r < dim; r += 64) put(r, basis[(size_t)r * stride + c]);
}

__global__ void int4_pack_kernel(const int8_t* __restrict__ q, int64_t n_values, uint8_t* __restrict__ packed) {
  const int64_t n_bytes = (n_values + 1) >> 1;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_bytes;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int lo = q[2 * i];
    const int hi = (2 * i + 1 < n_values) ? q[2 * i + 1] : 0;
    packed[i] = (uint8_t)(((lo + 8) & 15) | (((hi + 8) & 15) << 4));
  }
}

// ---------------------------------------------------------------------------
// V: Hadamard + per-channel max-abs normalisation
// ---------------------------------------------------------------------------
// Bound: memory traffic.  The rotated values are computed twice -- pass 1 reads the fp16 values and keeps
// only the channels' maxima, pass 2 reads them again and writes the normalised fp32 result -- because
// writing them out and reading them back costs more than the butterfly.  A row is held by 8 lanes, 16
// channels each: stages 1..8 of the butterfly inside a lane, 16..64 by shuffle (12 shuffles a row; with
// 4 channels a lane it was 20, and the pass was bound by them).
// 32K tokens x 8 heads: 106 us for both passes (67 MB read twice, 134 MB written), 295 us with the rotated
// values written by pass 1 and 4-channel lanes.
//
// H128(v) / sqrt(128) of the lane's 16 channels of one row (bit-identical to the stage-by-stage form)
__device__ __forceinline__ void v_rotate16(const __half* __restrict__ row, int sub, float (&y)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint2 raw = reinterpret_cast<const uint2*>(row + 16 * sub)[i];
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
    y[4 * i] = a.x; y[4 * i + 1] = a.y; y[4 * i + 2] = b.x; y[4 * i + 3] = b.y;
  }
#pragma unroll
  for (int h = 1; h < 16; h <<= 1) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (!(i & h)) { const float a = y[i], b = y[i + h]; y[i] = __fadd_rn(a, b); y[i + h] = __fsub_rn(a, b); }
    }
  }
#pragma unroll
  for (int bit = 1; bit < 8; bit <<= 1) {
    const bool upper = (sub & bit) != 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, y[i], bit);
      y[i] = upper ? __fsub_rn(other, y[i]) : __fadd_rn(y[i], other);
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) y[i] = __fdiv_rn(y[i], SQRT_HD);
}

// pass 1: ch_max = max_t |x|   (uint atomicMax on non-negative floats, one per block and channel)
__global__ void __launch_bounds__(256) v_channel_max_kernel(const __half* __restrict__ v, int64_t head_stride,
                                                            int64_t tok_stride, int n, uint32_t* __restrict__ ch_max) {
  __shared__ uint32_t m_s[HD];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, kv = blockIdx.y;
  if (threadIdx.x < HD) m_s[threadIdx.x] = 0u;
  __syncthreads();
  float am[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) am[i] = 0.f;
  // (every lane takes part in the shuffles: rows behind the last one repeat it)
  for (int t0 = (blockIdx.x * 8 + warp) * 4; t0 < n; t0 += gridDim.x * 32) {
    const int t = min(t0 + (lane >> 3), n - 1);
    float y[16];
    v_rotate16(v + kv * head_stride + (int64_t)t * tok_stride, sub, y);
#pragma unroll
    for (int i = 0; i < 16; ++i) am[i] = fmaxf(am[i], fabsf(y[i]));
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    am[i] = fmaxf(am[i], __shfl_xor_sync(0xffffffffu, am[i], 8));
    am[i] = fmaxf(am[i], __shfl_xor_sync(0xffffffffu, am[i], 16));
    if (lane < 8) atomicMax(&m_s[16 * sub + i], __float_as_uint(am[i]));
  }
  __syncthreads();
  if (threadIdx.x < HD) atomicMax(ch_max + kv * HD + threadIdx.x, m_s[threadIdx.x]);
}

__global__ void v_clamp_kernel(float* ch_max, int count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) ch_max[i] = fmaxf(ch_max[i], 1e-8f);
}

// pass 2: x = H128(v) / sqrt(128) / ch_max
__global__ void __launch_bounds__(256) v_normalise_kernel(const __half* __restrict__ v, int64_t head_stride,
                                                          int64_t tok_stride, int n, const float* __restrict__ ch_max,
                                                          float* __restrict__ x) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 7, kv = blockIdx.y;
  float c[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) c[i] = ch_max[kv * HD + 16 * sub + i];
  for (int t0 = (blockIdx.x * 8 + warp) * 4; t0 < n; t0 += gridDim.x * 32) {
    const int t = min(t0 + (lane >> 3), n - 1);
    float y[16];
    v_rotate16(v + kv * head_stride + (int64_t)t * tok_stride, sub, y);
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = __fdiv_rn(y[i], c[i]);
    if (t0 + (lane >> 3) < n) {
      float4* o = reinterpret_cast<float4*>(x + ((size_t)kv * n + t) * HD + 16 * sub);
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = make_float4(y[4 * i], y[4 * i + 1], y[4 * i + 2], y[4 * i + 3]);
    }
  }
}

// ---------------------------------------------------------------------------
// VQ assign: argmin_k ((x0-c0)^2 + (x1-c1)^2) + (x2-c2)^2) + (x3-c3)^2, first minimum
// ---------------------------------------------------------------------------
// With ACCUMULATE the kernel also does the k-means statistics of the same pass: per-centroid sums
// and counts are collected in shared memory (atomics) and added to `sums` / `counts` once per CTA,
// replacing two index_add_ passes over all points.  The order of those additions is not fixed,
// exactly as with index_add_ on a GPU.
template <bool ACCUMULATE>
__global__ void __launch_bounds__(256) vq_assign_kernel(const float4* __restrict__ x,
                                                        const float4* __restrict__ centroids, int64_t n,
                                                        uint8_t* __restrict__ idx_u8, int64_t* __restrict__ idx_i64,
                                                        float* __restrict__ sums, float* __restrict__ counts) {
  __shared__ float4 cb[256];
  __shared__ float acc_s[ACCUMULATE ? 256 * 5 : 1];
  cb[threadIdx.x] = centroids[threadIdx.x];
  if (ACCUMULATE)
    for (int i = threadIdx.x; i < 256 * 5; i += 256) acc_s[i] = 0.f;
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 p = x[i];
    float best = __int_as_float(0x7f800000);
    int arg = 0;
#pragma unroll 8
    for (int k = 0; k < 256; ++k) {
      const float4 c = cb[k];
      const float d0 = __fsub_rn(p.x, c.x), d1 = __fsub_rn(p.y, c.y);
      const float d2 = __fsub_rn(p.z, c.z), d3 = __fsub_rn(p.w, c.w);
      float dist = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
      dist = __fadd_rn(dist, __fmul_rn(d2, d2));
      dist = __fadd_rn(dist, __fmul_rn(d3, d3));
      if (dist < best) { best = dist; arg = k; }
    }
    idx_u8[i] = (uint8_t)arg;
    if (idx_i64) idx_i64[i] = arg;
    if (ACCUMULATE) {
      atomicAdd(&acc_s[arg * 5 + 0], p.x);
      atomicAdd(&acc_s[arg * 5 + 1], p.y);
      atomicAdd(&acc_s[arg * 5 + 2], p.z);
      atomicAdd(&acc_s[arg * 5 + 3], p.w);
      atomicAdd(&acc_s[arg * 5 + 4], 1.f);
    }
  }
  if (ACCUMULATE) {
    __syncthreads();
    const int k = threadIdx.x;
    if (acc_s[k * 5 + 4] > 0.f) {
#pragma unroll
      for (int c = 0; c < 4; ++c) atomicAdd(&sums[k * 4 + c], acc_s[k * 5 + c]);
      atomicAdd(&counts[k], acc_s[k * 5 + 4]);
    }
  }
}

}  // namespace shard

using namespace shard;

extern "C" size_t shard_b200_k_quantize_workspace_bytes(int32_t n, int32_t keep) {
  (void)n;
  return (size_t)3 * (keep > 0 ? keep : 0) * sizeof(uint32_t);
}

// (the counters and bit widths are in place)
static void launch_kq(const float* proj, const int32_t* alloc, int n, int keep, uint32_t* ws, float* coeff_scale, __half* scale_f16,
                      uint8_t* packed, cudaStream_t st) {
  const int rows = kq_rows(n), row_blocks = (n + rows - 1) / rows;
  kq_minmax_kernel<<<row_blocks, 256, 0, st>>>(proj, n, keep, rows, ws);
  kq_absmax_kernel<<<row_blocks, 256, 0, st>>>(proj, alloc, n, keep, rows, ws);
  kq_scale_kernel<<<(keep + 255) / 256, 256, 0, st>>>(ws, keep, coeff_scale, scale_f16);
  const size_t total = (size_t)n * (keep / 2);
  kq_pack_kernel<<<capped_blocks((long long)((total + 255) / 256), 16), 256, 0, st>>>(proj, alloc, n, keep, ws, coeff_scale, packed);
}

extern "C" int shard_b200_k_quantize_pack(const float* proj, const int32_t* alloc_bits, int32_t n, int32_t keep,
                                          float* coeff_scale_out, uint8_t* packed_out, void* workspace,
                                          size_t workspace_bytes, void* stream) {
  if (!proj || !alloc_bits || !coeff_scale_out || !packed_out || !workspace || n < 1 || keep < 2 || (keep & 1))
    return SHARD_E_ARG;
  if (workspace_bytes < shard_b200_k_quantize_workspace_bytes(n, keep)) return SHARD_E_WORKSPACE;
  if ((uintptr_t)proj & 7) return SHARD_E_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  uint32_t* ws = (uint32_t*)workspace;
  kq_init_kernel<<<(keep + 255) / 256, 256, 0, st>>>(ws, keep);
  launch_kq(proj, alloc_bits, n, keep, ws, coeff_scale_out, nullptr, packed_out, st);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

// workspace of shard_b200_k_encode: status word | w | projection | bit widths, counters, scales | projection's own
struct KEncodeLayout { size_t w, proj, small, project, bytes; };
static KEncodeLayout k_encode_layout(int nkv, int n, int keep) {
  KEncodeLayout l;
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  l.w = 256;
  l.proj = l.w + up((size_t)nkv * HD * keep * 4);
  l.small = l.proj + up((size_t)n * keep * 4);
  l.project = l.small + up((size_t)5 * keep * 4);
  l.bytes = l.project + shard_b200_k_project_workspace_bytes(nkv * HD, keep);
  return l;
}

extern "C" size_t shard_b200_k_encode_workspace_bytes(int32_t nkv, int32_t n, int32_t keep) {
  if (nkv < 1 || n < 1 || shard_b200_k_project_workspace_bytes(nkv * HD, keep) == 0) return 0;
  return k_encode_layout(nkv, n, keep).bytes;
}

extern "C" int shard_b200_k_encode(const float* flat, const float* mean, const void* mean_f16, const float* basis,
                                   int64_t basis_row_stride, const int32_t* alloc_bits_host, int32_t n, int32_t nkv, int32_t keep,
                                   int8_t* basis_q_out, void* scale_f16_out, void* basis_f16_out, uint8_t* packed_out,
                                   void* coeff_scale_f16_out, void* wprep_out, void* workspace, size_t workspace_bytes, void* stream) {
  if (!flat || !mean || !mean_f16 || !basis || !alloc_bits_host || !basis_q_out || !scale_f16_out || !basis_f16_out || !packed_out ||
      !coeff_scale_f16_out || !workspace)
    return SHARD_E_ARG;
  const size_t need = shard_b200_k_encode_workspace_bytes(nkv, n, keep);
  if (need == 0) return SHARD_E_ARG;
  if (workspace_bytes < need) return SHARD_E_WORKSPACE;
  KqBits bits{};
  for (int j = 0; j < keep; ++j) {
    if (alloc_bits_host[j] < 0 || alloc_bits_host[j] > 8) return SHARD_E_ARG;
    bits.b[j] = (uint8_t)alloc_bits_host[j];
  }
  const KEncodeLayout l = k_encode_layout(nkv, n, keep);
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = (unsigned char*)workspace;
  float* w = (float*)(ws + l.w);
  float* proj = (float*)(ws + l.proj);
  int32_t* alloc = (int32_t*)(ws + l.small);
  uint32_t* counters = (uint32_t*)alloc + keep;
  float* coeff_scale = (float*)(counters + 3 * keep);
  int rc = shard_b200_k_basis_quantise(basis, basis_row_stride, nkv * HD, keep, basis_q_out, scale_f16_out, w, basis_f16_out, stream);
  if (rc) return rc;
  rc = shard_b200_k_project(flat, mean, w, n, nkv * HD, keep, proj, ws + l.project, l.bytes - l.project, stream);
  if (rc) return rc;
  kq_init_bits_kernel<<<1, 256, 0, st>>>(counters, keep, bits, alloc, (const int*)(ws + l.project), (int*)ws);
  launch_kq(proj, alloc, n, keep, counters, coeff_scale, (__half*)coeff_scale_f16_out, packed_out, st);
  if (wprep_out) return shard_b200_decode_prepare(basis_f16_out, coeff_scale_f16_out, mean_f16, nkv, keep, wprep_out, stream);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_k_basis_quantise(const float* basis, int64_t row_stride, int32_t dim, int32_t keep, int8_t* basis_q_out,
                                           void* scale_f16_out, float* w_out, void* basis_f16_out, void* stream) {
  if (!basis || !basis_q_out || !scale_f16_out || !w_out || !basis_f16_out || dim < 1 || keep < 1 || row_stride < keep) return SHARD_E_ARG;
  k_basis_quantise_kernel<<<(keep + 15) / 16, 1024, 0, (cudaStream_t)stream>>>(basis, row_stride, dim, keep, basis_q_out,
                                                                              (__half*)scale_f16_out, w_out, (__half*)basis_f16_out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

// Host: the dynamic programme of dp_bit_allocation in double precision, first minimum wins.
extern "C" int shard_b200_dp_bit_allocation(const double* group_var_host, const int32_t* group_size_host, int32_t n_groups,
                                            int32_t total_budget, int32_t* group_bits_host) {
  constexpr int UNIT = 16;
  static const int choices[5] = {0, 2, 4, 6, 8};
  if (!group_var_host || !group_size_host || !group_bits_host || n_groups < 1 || total_budget < -UNIT) return SHARD_E_ARG;
  // (a budget beyond what eight bits for everything cost changes nothing, but would be a table of that length)
  long long most = 0;
  for (int g = 0; g < n_groups; ++g) most += ((long long)group_size_host[g] * 8 + UNIT - 1) / UNIT;
  const long long asked = (total_budget < 0 ? -1 : total_budget / UNIT) + 1;
  const int cap = (int)(asked < most ? asked : most);
  const double inf = 1.0 / 0.0;
  std::vector<double> best;
  std::vector<int> pick;
  try {
    best.assign((size_t)(n_groups + 1) * (cap + 1), inf);
    pick.assign((size_t)(n_groups + 1) * (cap + 1), 0);
  } catch (const std::bad_alloc&) {
    return SHARD_E_TOO_LARGE;
  }
  for (int b = 0; b <= cap; ++b) best[b] = 0.0;
  auto cost_of = [&](int g, int bits) { return bits == 0 ? 0 : (group_size_host[g] * bits + UNIT - 1) / UNIT; };
  for (int g = 0; g < n_groups; ++g) {
    const double* from = best.data() + (size_t)g * (cap + 1);
    double* to = best.data() + (size_t)(g + 1) * (cap + 1);
    int* pk = pick.data() + (size_t)(g + 1) * (cap + 1);
    for (int c = 0; c < 5; ++c) {                       // (choices outside: the order in which a minimum is first met is the same)
      const int bits = choices[c], cost = cost_of(g, bits);
      const double err = bits == 0 ? group_var_host[g] * 4.0 : group_var_host[g] / (3.0 * (double)(1 << (2 * bits)));
      for (int b = cost; b <= cap; ++b) {
        const double total = from[b - cost] + err;
        if (total < to[b]) { to[b] = total; pk[b] = bits; }
      }
    }
  }
  int b = 0;
  const double* last = best.data() + (size_t)n_groups * (cap + 1);
  for (int i = 1; i <= cap; ++i)
    if (last[i] < last[b]) b = i;
  for (int g = n_groups - 1; g >= 0; --g) {
    const int bits = pick[(size_t)(g + 1) * (cap + 1) + b];
    group_bits_host[g] = bits;
    b -= cost_of(g, bits);
  }
  return SHARD_OK;
}

// Sink and window rows of a layer's prompt, four contiguous tensors: out = [sink K | sink V | window K | window V],
// each [nkv][rows][128].  A warp per row.
__global__ void __launch_bounds__(256) kv_ends_kernel(const __half* __restrict__ k, const __half* __restrict__ v, int64_t k_head,
                                                      int64_t k_tok, int64_t v_head, int64_t v_tok, int nkv, int n_sink, int n_win,
                                                      int win_start, __half* __restrict__ out) {
  const int lane = threadIdx.x & 31, rows = n_sink + n_win;
  const int u = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (u >= 2 * rows * nkv) return;
  const int r = u % rows, kv = (u / rows) % nkv, is_v = u / (rows * nkv);
  const int t = r < n_sink ? r : win_start + r - n_sink;
  const __half* src = (is_v ? v + kv * v_head + (int64_t)t * v_tok : k + kv * k_head + (int64_t)t * k_tok) + 4 * lane;
  __half* dst = r < n_sink ? out + (((size_t)is_v * nkv + kv) * n_sink + r) * HD
                           : out + (size_t)2 * nkv * n_sink * HD + (((size_t)is_v * nkv + kv) * n_win + r - n_sink) * HD;
#pragma unroll
  for (int i = 0; i < 4; ++i) dst[4 * lane + i] = src[i];
}

extern "C" int shard_b200_kv_ends(const void* k_f16, const void* v_f16, int64_t k_head_stride, int64_t k_tok_stride,
                                  int64_t v_head_stride, int64_t v_tok_stride, int32_t nkv, int32_t n_sink, int32_t n_win,
                                  int32_t win_start, void* out_f16, void* stream) {
  if (!k_f16 || !v_f16 || !out_f16 || nkv < 1 || n_sink < 0 || n_win < 0) return SHARD_E_ARG;
  const long long warps = 2ll * (n_sink + n_win) * nkv;
  if (warps == 0) return SHARD_OK;
  kv_ends_kernel<<<(unsigned int)((warps + 7) / 8), 256, 0, (cudaStream_t)stream>>>(
      (const __half*)k_f16, (const __half*)v_f16, k_head_stride, k_tok_stride, v_head_stride, v_tok_stride, nkv, n_sink, n_win, win_start,
      (__half*)out_f16);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_int4_pack(const int8_t* q, int64_t n_values, uint8_t* packed_out, void* stream) {
  if (!q || !packed_out || n_values < 0) return SHARD_E_ARG;
  if (n_values == 0) return SHARD_OK;
  const int64_t n_bytes = (n_values + 1) / 2;
  const int blocks = capped_blocks((n_bytes + 255) / 256, 16);
  int4_pack_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(q, n_values, packed_out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_v_hadamard_normalise(const void* v_f16, int64_t head_stride, int64_t tok_stride,
                                               int32_t nkv, int32_t n, float* x_out, float* ch_max_out,
                                               void* stream) {
  if (!v_f16 || !x_out || !ch_max_out || nkv < 1 || n < 1) return SHARD_E_ARG;
  if (((uintptr_t)v_f16 & 7) || (head_stride & 3) || (tok_stride & 3) || ((uintptr_t)x_out & 15))
    return SHARD_E_ALIGN;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(ch_max_out, 0, (size_t)nkv * HD * sizeof(float), st);
  if (e != cudaSuccess) return (int)e;
  const int per_head = capped_blocks((long long)nkv * ((n + 31) / 32), 8) / nkv;   // blocks of 32 rows, eight per SM at most
  const dim3 grid(per_head > 0 ? per_head : 1, nkv);
  v_channel_max_kernel<<<grid, 256, 0, st>>>((const __half*)v_f16, head_stride, tok_stride, n, (uint32_t*)ch_max_out);
  v_clamp_kernel<<<(nkv * HD + 255) / 256, 256, 0, st>>>(ch_max_out, nkv * HD);
  v_normalise_kernel<<<grid, 256, 0, st>>>((const __half*)v_f16, head_stride, tok_stride, n, ch_max_out, x_out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_vq_assign(const float* x, const float* centroids, int64_t n, uint8_t* idx_u8,
                                    int64_t* idx_i64, void* stream) {
  if (!x || !centroids || !idx_u8 || n < 0) return SHARD_E_ARG;
  if (((uintptr_t)x | (uintptr_t)centroids) & 15) return SHARD_E_ALIGN;
  if (n == 0) return SHARD_OK;
  const int64_t want = (n + 255) / 256;
  const int blocks = capped_blocks(want, 8);
  vq_assign_kernel<false><<<blocks, 256, 0, (cudaStream_t)stream>>>((const float4*)x, (const float4*)centroids, n,
                                                                     idx_u8, idx_i64, nullptr, nullptr);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" int shard_b200_vq_assign_accumulate(const float* x, const float* centroids, int64_t n, uint8_t* idx_u8,
                                               float* sums, float* counts, void* stream) {
  if (!x || !centroids || !idx_u8 || !sums || !counts || n < 0) return SHARD_E_ARG;
  if (((uintptr_t)x | (uintptr_t)centroids) & 15) return SHARD_E_ALIGN;
  if (n == 0) return SHARD_OK;
  const int64_t want = (n + 255) / 256;
  const int blocks = capped_blocks(want, 8);
  vq_assign_kernel<true><<<blocks, 256, 0, (cudaStream_t)stream>>>((const float4*)x, (const float4*)centroids, n,
                                                                    idx_u8, nullptr, sums, counts);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}
