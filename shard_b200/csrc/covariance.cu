// Keys of a prompt -> un-rotated fp32 rows, their mean, and the Gram matrix of the centred rows: the
// inputs of the PCA fit and of the projection.
//
//   flat[t][kv*128+d] = undo RoPE(k)      mean = column means      G = (flat - mean)^T (flat - mean)
//
// G is the largest dense contraction of the compressor (2 n p^2: 69 GFLOP for a 32K layer; a library
// fp32 GEMM takes 1.25 ms).  It runs on the tensor cores at fp32 accuracy: the centred values, scaled to
// the top of fp16's range, are split into two fp16 parts (22 bits for every value within 2^17 of the largest; a
// scale to [0, 1] would leave the parts of a value 2^10 below it 12 bits), three products -- head.head, head.tail, tail.head -- go into
// one fp32 accumulator, and because the tensor core adds with truncation the accumulator is added to
// fp32 registers (round to nearest) every 64 tokens.  Rows are tokens, so both operands are
// MN-major: a token's 64 dimensions are one 128-byte row of the swizzled operand, no transposition.
//
// A CTA computes one 128 x 128 tile of the upper triangle over a share of the tokens (the shares fill
// the machine); gram_sum_kernel adds the shares in order and mirrors the tile.
//
//   warps 0-7   load fp32 rows (the next 64 tokens in flight), subtract the mean, split, store
//   warps 8-11  accumulator -> registers
//   warp 12     issues the MMAs
//
// Bound: the conversion work of the producers and the L2 reads (each of the tile's blocks is converted
// by every CTA that needs it), about as long as the tensor work beside it.  p = 1024: 230 us for 32K
// tokens (1 250 us as a library fp32 GEMM), 62 us for 8K.
#include <atomic>

#include "tcgen05.cuh"

namespace shard {

// ---------------------------------------------------------------------------
// undo RoPE: flat[t][kv*128+d] = k*cos - rotate_half(k)*sin, fp32
// ---------------------------------------------------------------------------
__device__ __forceinline__ void undo_rope_pair(const __half* __restrict__ row, float* __restrict__ o, int i, float cs, float sn,
                                               float& a, float& b) {
  const float lo = __half2float(row[i]), hi = __half2float(row[i + 64]);
  // d < 64: k[d]*cos - (-k[d+64])*sin ; d >= 64: k[d]*cos - k[d-64]*sin
  a = __fadd_rn(__fmul_rn(lo, cs), __fmul_rn(hi, sn));
  b = __fsub_rn(__fmul_rn(hi, cs), __fmul_rn(lo, sn));
  o[i] = a;
  o[i + 64] = b;
}

// A block per token: as many of them in flight as the loads and stores need (32K tokens x 8 heads, 201 MB: 51 us;
// with the loop over tokens of the kernel below 95 us).
__global__ void __launch_bounds__(128) undo_rope_kernel(const __half* __restrict__ k, int64_t head_stride, int64_t tok_stride, int nkv,
                                                        int pos_start, const float* __restrict__ inv_freq, float* __restrict__ flat) {
  const int t = blockIdx.x, i = threadIdx.x & 63;
  float sn, cs, a, b;
  sincosf(__fmul_rn((float)(pos_start + t), inv_freq[i]), &sn, &cs);
  for (int kv = threadIdx.x >> 6; kv < nkv; kv += 2)
    undo_rope_pair(k + kv * head_stride + (int64_t)t * tok_stride, flat + (size_t)t * nkv * HD + kv * HD, i, cs, sn, a, b);
}

// The same with the columns' sums and the largest magnitude.
constexpr int UR_MAX_HEADS_PER_THREAD = 8;   // column sums are kept for up to 32 KV heads

// Block: tokens blockIdx.x * per_block ...; thread: pair i = tid & 63 of heads tid / 64, + 4, ...
__global__ void __launch_bounds__(256) undo_rope_stats_kernel(const __half* __restrict__ k, int64_t head_stride, int64_t tok_stride,
                                                        int nkv, int n, int per_block, int pos_start,
                                                        const float* __restrict__ inv_freq, float* __restrict__ flat,
                                                        float* __restrict__ part_sums, unsigned int* __restrict__ max_bits) {
  const int i = threadIdx.x & 63, h0 = threadIdx.x >> 6;
  const float freq = inv_freq[i];
  const int t0 = blockIdx.x * per_block, t1 = min(t0 + per_block, n);
  float s_lo[UR_MAX_HEADS_PER_THREAD], s_hi[UR_MAX_HEADS_PER_THREAD], mx = 0.f;
#pragma unroll
  for (int j = 0; j < UR_MAX_HEADS_PER_THREAD; ++j) s_lo[j] = s_hi[j] = 0.f;
  for (int t = t0; t < t1; ++t) {
    const float phase = __fmul_rn((float)(pos_start + t), freq);
    float sn, cs;
    sincosf(phase, &sn, &cs);
#pragma unroll
    for (int j = 0; j < UR_MAX_HEADS_PER_THREAD; ++j) {
      const int kv = h0 + 4 * j;
      if (kv < nkv) {
        float a, b;
        undo_rope_pair(k + kv * head_stride + (int64_t)t * tok_stride, flat + (size_t)t * nkv * HD + kv * HD, i, cs, sn, a, b);
        s_lo[j] += a;
        s_hi[j] += b;
        mx = fmaxf(mx, fmaxf(fabsf(a), fabsf(b)));
      }
    }
  }
  float* o = part_sums + (size_t)blockIdx.x * nkv * HD;
#pragma unroll
  for (int j = 0; j < UR_MAX_HEADS_PER_THREAD; ++j)
    if (h0 + 4 * j < nkv) { o[(h0 + 4 * j) * HD + i] = s_lo[j]; o[(h0 + 4 * j) * HD + 64 + i] = s_hi[j]; }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) atomicMax(max_bits, __float_as_uint(mx));
}

// mean of 32 columns per block: 8 rows of partial sums at a time
__global__ void __launch_bounds__(256) column_mean_kernel(const float* __restrict__ part_sums, int parts, int p, int n,
                                                          float* __restrict__ mean, __half* __restrict__ mean_f16) {
  __shared__ float s_s[8][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), r0 = threadIdx.x >> 5;
  float s = 0.f;
#pragma unroll 4
  for (int r = r0; r < parts; r += 8) s += part_sums[(size_t)r * p + c];
  s_s[r0][threadIdx.x & 31] = s;
  __syncthreads();
  if (r0 == 0) {
    for (int i = 1; i < 8; ++i) s += s_s[i][threadIdx.x];
    const float m = s / (float)n;
    mean[c] = m;
    if (mean_f16) mean_f16[c] = __float2half_rn(m);
  }
}

// ---------------------------------------------------------------------------
// Gram matrix
// ---------------------------------------------------------------------------
constexpr int GR_CHUNK = 64;                       // tokens per stage
constexpr int GR_STAGES = 3;
constexpr int GR_OP_BYTES = 128 * GR_CHUNK * 2;    // one operand part of a stage: [2 x 64 dims][64 tokens][128 bytes]
constexpr int GR_STAGE_BYTES = 4 * GR_OP_BYTES;    // A head, A tail, B head, B tail
constexpr int GR_PRODUCERS = 256;
constexpr int GR_THREADS = 13 * 32;
constexpr int GR_GROUP = 1;                        // chunks accumulated in tensor memory between two promotions
constexpr int GR_SMEM_BYTES = 1024 + GR_STAGES * GR_STAGE_BYTES + 256;

struct GramParams {
  const float* flat;
  const float* mean;
  int n, p;
  int chunks_per_share;
  float* part;              // [shares][tiles][128][128]
  const unsigned int* max_bits;
  int* status;
};

// scale that brings |x - mean| (at most twice the largest |x|) below 2^15: a tail then has its full precision
// unless its value is 2^17 times smaller (fp16's smallest step is 2^-24), and squares stay far from fp32's limit
__device__ __forceinline__ float gram_scale(const unsigned int* max_bits) {
  const float m = 2.f * __uint_as_float(__ldcg(max_bits));
  if (!(m > 0.f) || isinf(m)) return 1.f;
  int e;
  frexpf(m, &e);
  return ldexpf(1.f, 15 - e);
}
// tile number -> blocks (i, j), i <= j, of the upper triangle
__device__ __forceinline__ void gram_tile(int t, int blocks, int& i, int& j) {
  i = 0;
  while (t >= blocks - i) { t -= blocks - i; ++i; }
  j = i + t;
}

__global__ void __launch_bounds__(GR_THREADS, 1) gram_kernel(const __grid_constant__ GramParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GR_STAGES * GR_STAGE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * GR_STAGES + 4);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto FULL = [&](int s) { return bar0 + 8u * (uint32_t)s; };                       // operands of the stage written
  auto EMPTY = [&](int s) { return bar0 + 8u * (uint32_t)(GR_STAGES + s); };        // the stage's MMAs have run
  auto ACC_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(2 * GR_STAGES + b); };
  auto ACC_FREE = [&](int b) { return bar0 + 8u * (uint32_t)(2 * GR_STAGES + 2 + b); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blocks = p.p / 128;
  int bi, bj;
  gram_tile(blockIdx.x, blocks, bi, bj);
  const bool diag = bi == bj;
  const int c_lo = blockIdx.y * p.chunks_per_share;
  const int n_chunks = min((p.n + GR_CHUNK - 1) / GR_CHUNK - c_lo, p.chunks_per_share);   // (at least one)
  const int n_groups = (n_chunks + GR_GROUP - 1) / GR_GROUP;

  if (warp == 12) {
    tmem_alloc(smem_u32(tmem_slot), 256);
    tmem_relinquish();
    if (lane == 0) {
      for (int s = 0; s < GR_STAGES; ++s) { mbar_init(FULL(s), GR_PRODUCERS / 32); mbar_init(EMPTY(s), 1); }
      for (int b = 0; b < 2; ++b) { mbar_init(ACC_FULL(b), 1); mbar_init(ACC_FREE(b), 4); }
      *abort_s = 0;
      fence_mbar_init();
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < 8) {
    // ---- producers: thread = 8 dimensions (tid % 16) of tokens tid / 16, + 16, ... of both blocks ------
    const float scale = gram_scale(p.max_bits);
    const int c16 = tid & 15, r0 = tid >> 4;
    float mu[2][8];
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int e = 0; e < 8; ++e) mu[o][e] = p.mean[(o ? bj : bi) * 128 + 8 * c16 + e];
    float4 x[2][4][2];
    auto load = [&](int c) {
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        if (o && diag) break;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int t = (c_lo + c) * GR_CHUNK + r0 + 16 * u;
          const float4* src = reinterpret_cast<const float4*>(p.flat + (size_t)min(t, p.n - 1) * p.p + (o ? bj : bi) * 128 + 8 * c16);
          x[o][u][0] = src[0];
          x[o][u][1] = src[1];
        }
      }
    };
    load(0);
    bool bad = false;
    for (int c = 0; c < n_chunks; ++c) {
      const int s = c % GR_STAGES;
      if (c >= GR_STAGES) bad = !mbar_wait(EMPTY(s), (uint32_t)((c / GR_STAGES - 1) & 1), abort_s);
      bad = __any_sync(0xffffffffu, bad || *abort_s);
      if (bad) break;
      unsigned char* st = smem + s * GR_STAGE_BYTES;
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        if (o && diag) break;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const bool live = (c_lo + c) * GR_CHUNK + r0 + 16 * u < p.n;
          const float v[8] = {x[o][u][0].x, x[o][u][0].y, x[o][u][0].z, x[o][u][0].w, x[o][u][1].x, x[o][u][1].y, x[o][u][1].z, x[o][u][1].w};
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float a = live ? (v[2 * e] - mu[o][2 * e]) * scale : 0.f, b = live ? (v[2 * e + 1] - mu[o][2 * e + 1]) * scale : 0.f;
            const __half2 h = __floats2half2_rn(a, b);
            const float2 f = __half22float2(h);
            hi[e] = as_u32(h);
            lo[e] = pack_half2(a - f.x, b - f.y);
          }
          unsigned char* dst = st + 2 * o * GR_OP_BYTES + (c16 >> 3) * (GR_OP_BYTES / 2) + sw128_off(r0 + 16 * u, c16 & 7);
          *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(dst + GR_OP_BYTES) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      if (c + 1 < n_chunks) load(c + 1);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(FULL(s));
    }
  } else if (warp == 12) {
    // ---- MMAs ---------------------------------------------------------------------------------------
    if (lane == 0) {
      constexpr uint32_t IDESC = umma_idesc(128, 128, true, true);
      bool ok = true;
      for (int c = 0; c < n_chunks && ok; ++c) {
        const int s = c % GR_STAGES, grp = c / GR_GROUP, b = grp & 1;
        const bool first = c % GR_GROUP == 0;
        if (first && grp >= 2) ok = mbar_wait(ACC_FREE(b), (uint32_t)(((grp >> 1) - 1) & 1), abort_s);
        ok = ok && mbar_wait(FULL(s), (uint32_t)((c / GR_STAGES) & 1), abort_s);
        if (!ok) break;
        tc_fence_after();
        const uint32_t base = smem_u32(smem + s * GR_STAGE_BYTES), bbase = diag ? base : base + 2 * GR_OP_BYTES;
        const uint64_t ah = smem_desc_sw128(base, GR_OP_BYTES / 2, 1024), al = smem_desc_sw128(base + GR_OP_BYTES, GR_OP_BYTES / 2, 1024);
        const uint64_t bh = smem_desc_sw128(bbase, GR_OP_BYTES / 2, 1024), bl = smem_desc_sw128(bbase + GR_OP_BYTES, GR_OP_BYTES / 2, 1024);
        const uint32_t acc = tmem_base + (uint32_t)(128 * b);
#pragma unroll
        for (int ks = 0; ks < GR_CHUNK / 16; ++ks) {
          const uint64_t adv = (uint64_t)((ks * 2048) >> 4);
          umma_ss(acc, al + adv, bh + adv, IDESC, (!first || ks > 0) ? 1u : 0u, 1u);   // the small terms first
          umma_ss(acc, ah + adv, bl + adv, IDESC, 1u, 1u);
          umma_ss(acc, ah + adv, bh + adv, IDESC, 1u, 1u);
        }
        umma_commit(EMPTY(s), 1u);
        if (c % GR_GROUP == GR_GROUP - 1 || c == n_chunks - 1) umma_commit(ACC_FULL(b), 1u);
      }
      if (!ok) *abort_s = 1;
    }
    __syncwarp();
  } else {
    // ---- promotion: thread = row of the tile -----------------------------------------------------------
    const int quad = warp & 3;
    const uint32_t lane_off = (uint32_t)(quad * 32) << 16;
    float sum[128];
#pragma unroll
    for (int j = 0; j < 128; ++j) sum[j] = 0.f;
    bool bad = false;
    for (int grp = 0; grp < n_groups; ++grp) {
      const int b = grp & 1;
      bad = !mbar_wait(ACC_FULL(b), (uint32_t)((grp >> 1) & 1), abort_s);
      bad = __any_sync(0xffffffffu, bad || *abort_s);
      if (bad) break;
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t o[16];
        tmem_ld_x16(tmem_base + (uint32_t)(128 * b + 16 * q) + lane_off, o);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[16 * q + j] = __fadd_rn(sum[16 * q + j], __uint_as_float(o[j]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ACC_FREE(b));
    }
    if (!bad) {
      float* dst = p.part + (((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 128 + quad * 32 + lane) * 128;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        reinterpret_cast<float4*>(dst)[j] = make_float4(sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
    }
  }
  if (tid == 0 && *abort_s) atomicExch(p.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem_base, 256);
}

// Shares added in order, unscaled, written to both triangles; a block takes 16 rows of a tile.
__global__ void __launch_bounds__(256) gram_sum_kernel(const float* __restrict__ part, int shares, int tiles, int p,
                                                       const unsigned int* __restrict__ max_bits, float* __restrict__ g) {
  __shared__ float t_s[16][129];
  int bi, bj;
  gram_tile(blockIdx.x, p / 128, bi, bj);
  const float s = gram_scale(max_bits), inv = 1.f / (s * s);
  const int r0 = blockIdx.y * 16;
  for (int u = threadIdx.x; u < 16 * 128; u += 256) {
    const int r = u >> 7, c = u & 127;
    // a tile on the diagonal is symmetric up to the order of its products: its upper half counts
    const bool low = bi == bj && r0 + r > c;
    const size_t at = low ? (size_t)c * 128 + r0 + r : (size_t)(r0 + r) * 128 + c;
    float v = 0.f;
#pragma unroll 4
    for (int h = 0; h < shares; ++h) v += part[((size_t)h * tiles + blockIdx.x) * 128 * 128 + at];
    v *= inv;
    g[(size_t)(bi * 128 + r0 + r) * p + bj * 128 + c] = v;
    t_s[r][c] = v;
  }
  if (bi == bj) return;
  __syncthreads();
  for (int u = threadIdx.x; u < 16 * 128; u += 256) {
    const int r = u & 15, c = u >> 4;
    g[(size_t)(bj * 128 + c) * p + bi * 128 + r0 + r] = t_s[r][c];
  }
}

struct CovLayout { size_t head, sums, part, bytes; int rope_blocks, per_block, tiles, shares, chunks_per_share; };
static CovLayout cov_layout(int nkv, int n) {
  CovLayout l;
  const int sms = sm_count() > 0 ? sm_count() : 148, p = nkv * HD;
  l.per_block = (n + 4 * sms - 1) / (4 * sms);                 // four blocks per SM
  l.rope_blocks = (n + l.per_block - 1) / l.per_block;
  const int blocks = p / 128, chunks = (n + GR_CHUNK - 1) / GR_CHUNK;
  l.tiles = blocks * (blocks + 1) / 2;
  // shares of the tokens: one CTA per SM in all, but no share shorter than two chunks
  l.shares = sms / l.tiles;
  if (l.shares > (chunks + 1) / 2) l.shares = (chunks + 1) / 2;
  if (l.shares < 1) l.shares = 1;
  l.chunks_per_share = (chunks + l.shares - 1) / l.shares;
  l.shares = (chunks + l.chunks_per_share - 1) / l.chunks_per_share;
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  l.head = 0;                                                  // max bits, status
  l.sums = 256;
  l.part = l.sums + up((size_t)l.rope_blocks * p * 4);
  l.bytes = l.part + (size_t)l.shares * l.tiles * 128 * 128 * 4;
  return l;
}

}  // namespace shard

using namespace shard;

extern "C" int shard_b200_undo_rope(const void* k_f16, int64_t head_stride, int64_t tok_stride, int32_t nkv,
                                    int32_t n, int32_t pos_start, const float* inv_freq, float* flat_out,
                                    void* stream) {
  if (!k_f16 || !inv_freq || !flat_out || nkv < 1 || n < 0) return SHARD_E_ARG;
  if (n == 0) return SHARD_OK;
  undo_rope_kernel<<<n, 128, 0, (cudaStream_t)stream>>>((const __half*)k_f16, head_stride, tok_stride, nkv, pos_start, inv_freq, flat_out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}

extern "C" size_t shard_b200_k_covariance_workspace_bytes(int32_t nkv, int32_t n) {
  if (nkv < 1 || nkv > 4 * UR_MAX_HEADS_PER_THREAD || n < 1) return 0;
  return cov_layout(nkv, n).bytes;
}

extern "C" int shard_b200_k_covariance(const void* k_f16, int64_t head_stride, int64_t tok_stride, int32_t nkv, int32_t n,
                                       int32_t pos_start, const float* inv_freq, float* flat_out, float* mean_out,
                                       void* mean_f16_out, float* gram_out, void* workspace, size_t workspace_bytes, void* stream) {
  if (!k_f16 || !inv_freq || !flat_out || !mean_out || !gram_out || !workspace) return SHARD_E_ARG;
  const size_t need = shard_b200_k_covariance_workspace_bytes(nkv, n);
  if (need == 0) return SHARD_E_ARG;
  if (workspace_bytes < need) return SHARD_E_WORKSPACE;
  if (((uintptr_t)flat_out | (uintptr_t)workspace) & 15) return SHARD_E_ALIGN;
  static std::atomic<bool> configured[MAX_DEVICES];
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= MAX_DEVICES) return SHARD_E_ARG;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(gram_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured[dev].store(true, std::memory_order_release);
  }
  const CovLayout l = cov_layout(nkv, n);
  const int p = nkv * HD;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = (unsigned char*)workspace;
  unsigned int* max_bits = (unsigned int*)ws;
  int* status = (int*)(ws + 4);
  float* sums = (float*)(ws + l.sums);
  float* part = (float*)(ws + l.part);
  e = cudaMemsetAsync(max_bits, 0, sizeof(*max_bits), st);      // (the status word stays as it is: the caller's to zero)
  if (e != cudaSuccess) return (int)e;
  undo_rope_stats_kernel<<<l.rope_blocks, 256, 0, st>>>((const __half*)k_f16, head_stride, tok_stride, nkv, n, l.per_block, pos_start,
                                                        inv_freq, flat_out, sums, max_bits);
  column_mean_kernel<<<p / 32, 256, 0, st>>>(sums, l.rope_blocks, p, n, mean_out, (__half*)mean_f16_out);
  GramParams g{flat_out, mean_out, n, p, l.chunks_per_share, part, max_bits, status};
  gram_kernel<<<dim3(l.tiles, l.shares), GR_THREADS, GR_SMEM_BYTES, st>>>(g);
  gram_sum_kernel<<<dim3(l.tiles, 8), 256, 0, st>>>(part, l.shares, l.tiles, p, max_bits, gram_out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}
