// Attention of several new query tokens over a compressed layer (the next user turn of a chat, a
// speculative batch): causal among the new tokens, everything before them visible to all.
//
// The layer is read back once as fp16 keys and values -- written as tile images in the tensor-core
// operand layout (read_back_kernel) -- and all queries attend to it: one KV head's 4 s query rows are
// the M dimension of dense products, instead of one reconstruction of all keys per query token.
//
//   CTA = (share of the tiles, 128 query rows, KV head), 5 warps:
//     warps 0-3   thread = query row: scores (tensor memory) -> online softmax -> weights, written over the
//                 scores as two fp16 parts (22 bits); the accumulator is rescaled only when a row's
//                 reference point moves by more than 2^8
//     warp 4      bulk copies of the tile images (two stages each) and all MMAs: S = Q K^T for the next
//                 tile while the softmax works on this one, then O += P V with P's parts from tensor memory
//
// Weights of 11 bits would leave the output further from float64 than the decode launch's, which weighs
// the rows outside the middle with 22 bits and has exact fp16 values in the middle: up to 25 % where decoded tokens carry
// the attention (2-norm 2.9e-4 against 2.3e-4; 2.2e-4 with both parts), 5 % with two KV heads.
//
// Shares are merged by multiquery_merge_kernel (their partial rows are fp32; a single share writes the
// result itself).
//
// Bound: the exponentials (16 per SM and cycle: 1 K cycles a tile) and the tensor work (1 K cycles a
// tile) are about equal and overlap only partly, one softmax group per CTA; the images' 64 KB per tile
// and KV head come from L2.  48 new tokens over 8K, 8 KV heads: 30 us a layer (26 with weights of 11 bits), and
// 26 us for the read-back in front of it (one decode launch per query token: 1 600 us a layer).
#include <atomic>

#include "decode_common.cuh"
#include "tcgen05.cuh"

namespace shard {

// implemented in readback.cu
int launch_read_back_any(const ShardSeq& seq, const ShardDecodeShape& sh, const float* inv_freq, const float* codebook,
                         int compress_start, void* k_out, void* v_out, bool image, int* status, cudaStream_t st);

constexpr int MQ_THREADS = 160;
constexpr int MQ_TILE_BYTES = 32768;
constexpr int MQ_SMEM_BYTES = 1024 + 5 * MQ_TILE_BYTES + 256;   // Q, two stages of K and of V
constexpr int MQ_COL_O = 256;                                    // two score stages of 128 columns, then the accumulator
constexpr float MQ_LAZY_LOG2 = 8.f;

struct MultiQueryParams {
  const __half* q;          // query token j of head h: q + h * q_head + j * q_tok
  int64_t q_head, q_tok;
  __half* out;              // [s][n_q][128]
  const unsigned char* k_img;   // [nkv][tiles][32 KB]
  const unsigned char* v_img;
  float* part;              // [shares][nkv][m_tiles * 128][132]
  int* status;
  int s, nkv;
  int n_mid_tiles, n_comp;  // the middle's tiles come first; its last one may be short
  int n_rows;               // other rows, in tiles behind the middle; the s new tokens are the last of them
  int n_tiles;
  int shares;
};

__global__ void __launch_bounds__(MQ_THREADS, 1) multiquery_kernel(const __grid_constant__ MultiQueryParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* q_s = smem;
  unsigned char* k_s = q_s + MQ_TILE_BYTES;
  unsigned char* v_s = k_s + 2 * MQ_TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + 2 * MQ_TILE_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 12);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t bar0 = smem_u32(bars);
  auto K_FULL = [&](int b) { return bar0 + 8u * (uint32_t)b; };
  auto V_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(2 + b); };
  auto S_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(4 + b); };     // scores of the stage are complete
  auto P_READY = [&](int b) { return bar0 + 8u * (uint32_t)(6 + b); };    // weights written, accumulator rescaled
  auto O_DONE = [&](int b) { return bar0 + 8u * (uint32_t)(8 + b); };     // the stage's P V product has run
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int share = blockIdx.x, mt = blockIdx.y, kv = blockIdx.z;
  const int base = p.n_tiles / p.shares, rem = p.n_tiles % p.shares;
  const int t0 = share * base + min(share, rem), nt = base + (share < rem ? 1 : 0);   // (nt >= 1)

  if (warp == 4) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
    if (lane == 0) {
      for (int b = 0; b < 2; ++b) {
        mbar_init(K_FULL(b), 1); mbar_init(V_FULL(b), 1); mbar_init(S_FULL(b), 1); mbar_init(P_READY(b), 4); mbar_init(O_DONE(b), 1);
      }
      *abort_s = 0;
      fence_mbar_init();
    }
  } else {
    // query rows -> operand: row r = query token (128 mt + r) / 4, head r % 4; rows behind the last are zero
    for (int u = tid; u < 128 * 16; u += 128) {
      const int r = u >> 4, c = u & 15, row = 128 * mt + r, j = row >> 2, h = kv * GQA + (row & 3);
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (j < p.s) {
        const uint2* src = reinterpret_cast<const uint2*>(p.q + h * p.q_head + j * p.q_tok + 8 * c);
        const uint2 a = src[0], b = src[1];
        v = make_uint4(a.x, a.y, b.x, b.y);
      }
      *reinterpret_cast<uint4*>(q_s + (c >> 3) * 16384 + sw128_off(r, c & 7)) = v;
    }
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 4) {
    if (lane == 0) {
      const size_t img0 = ((size_t)kv * p.n_tiles + t0) * MQ_TILE_BYTES;
      auto load = [&](bool is_v, int t) {
        const int b = t & 1;
        const uint32_t bar = is_v ? V_FULL(b) : K_FULL(b);
        mbar_expect_tx(bar, MQ_TILE_BYTES);
        bulk_g2s(smem_u32((is_v ? v_s : k_s) + b * MQ_TILE_BYTES), (is_v ? p.v_img : p.k_img) + img0 + (size_t)t * MQ_TILE_BYTES,
                 MQ_TILE_BYTES, bar);
      };
      constexpr uint32_t IDESC_S = umma_idesc(128, 128, false, false), IDESC_O = umma_idesc(128, 128, false, true);
      const uint64_t qd = smem_desc_sw128(smem_u32(q_s), 16, 1024);
      auto scores = [&](int t) -> bool {
        const int b = t & 1;
        if (!mbar_wait(K_FULL(b), (uint32_t)((t >> 1) & 1), abort_s)) return false;
        tc_fence_after();
        const uint64_t kd = smem_desc_sw128(smem_u32(k_s + b * MQ_TILE_BYTES), 16, 1024);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const uint64_t adv = (uint64_t)(((ks >> 2) * 16384 + (ks & 3) * 32) >> 4);
          umma_ss(tmem_base + 128 * b, qd + adv, kd + adv, IDESC_S, ks > 0 ? 1u : 0u, 1u);
        }
        umma_commit(S_FULL(b), 1u);
        return true;
      };
      load(false, 0);
      load(true, 0);
      if (nt > 1) { load(false, 1); load(true, 1); }
      bool ok = scores(0);
      int k_asked = min(nt, 2), v_asked = k_asked;
      for (int t = 0; t < nt && ok; ++t) {
        const int b = t & 1;
        if (t + 1 < nt) {
          // the other score stage holds the weights of tile t - 1 until their product has run
          if (t > 0) {
            ok = mbar_wait(O_DONE(b ^ 1), (uint32_t)(((t - 1) >> 1) & 1), abort_s);
            if (!ok) break;
            load(true, t + 1);                                   // (its V stage is free with it)
            v_asked = t + 2;
          }
          ok = scores(t + 1);
          if (!ok) break;
        }
        // K of tile t has been read once its scores are complete: the weights below depend on them
        ok = mbar_wait(P_READY(b), (uint32_t)((t >> 1) & 1), abort_s) && mbar_wait(V_FULL(b), (uint32_t)((t >> 1) & 1), abort_s);
        if (!ok) break;
        if (t + 2 < nt) { load(false, t + 2); k_asked = t + 3; }
        tc_fence_after();
        const uint64_t vd = smem_desc_sw128(smem_u32(v_s + b * MQ_TILE_BYTES), 16384, 1024);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          umma_ts(tmem_base + MQ_COL_O, tmem_base + 128 * b + 8 * ks, vd + (uint64_t)((ks * 2048) >> 4), IDESC_O, (t > 0 || ks > 0) ? 1u : 0u, 1u);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)                          // the weights' tails
          umma_ts(tmem_base + MQ_COL_O, tmem_base + 128 * b + 64 + 8 * ks, vd + (uint64_t)((ks * 2048) >> 4), IDESC_O, 1u, 1u);
        umma_commit(O_DONE(b), 1u);
      }
      if (!ok) {
        // gave up: do not leave while a copy is still landing in this CTA's shared memory
        *abort_s = 1;
        for (int t = max(0, k_asked - 2); t < k_asked; ++t) mbar_wait(K_FULL(t & 1), (uint32_t)((t >> 1) & 1), abort_s);
        for (int t = max(0, v_asked - 2); t < v_asked; ++t) mbar_wait(V_FULL(t & 1), (uint32_t)((t >> 1) & 1), abort_s);
      }
    }
    __syncwarp();
  } else {
    const int row = 128 * mt + tid, j = row >> 2;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    // other rows query token j sees: all but the new tokens behind it
    const int vis = p.n_rows - p.s + min(j, p.s - 1) + 1;
    float m = neg_inf(), l = 0.f;                                // reference point (log2 domain) and sum of weights
    bool bad = false;
    for (int t = 0; t < nt; ++t) {
      const int b = t & 1, tile = t0 + t;
      bad = !mbar_wait(S_FULL(b), (uint32_t)((t >> 1) & 1), abort_s);
      bad = __any_sync(0xffffffffu, bad || *abort_s);
      if (bad) break;
      tc_fence_after();
      const uint32_t S = tmem_base + 128 * b + lane_off;
      uint32_t sc[128];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_x32(S + 32 * c, *reinterpret_cast<uint32_t(*)[32]>(&sc[32 * c]));
      tmem_wait_ld();
      const int limit = tile < p.n_mid_tiles ? p.n_comp - 128 * tile : vis - 128 * (tile - p.n_mid_tiles);
      if (__any_sync(0xffffffffu, limit < 128)) {
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (c >= limit) sc[c] = 0xff800000u;
      }
      float mx[4] = {neg_inf(), neg_inf(), neg_inf(), neg_inf()};
#pragma unroll
      for (int c = 0; c < 128; ++c) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(sc[c]));
      constexpr float K = INV_SQRT_HD * LOG2E;
      const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * K;
      float alpha = 1.f;
      if (top > m + MQ_LAZY_LOG2 || m == neg_inf()) {
        alpha = m == neg_inf() ? 0.f : exp2f(m - top);
        m = top;
      }
      const float ref = m == neg_inf() ? 0.f : m;                // (nothing visible yet: weights are exp2(-inf) = 0)
      float sum[2] = {0.f, 0.f};
      // (in registers since tmem_wait_ld: the stage's columns may be overwritten, heads 0..63, tails 64..127)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float a = exp2f(fmaf(__uint_as_float(sc[32 * q + 2 * e]), K, -ref)), d = exp2f(fmaf(__uint_as_float(sc[32 * q + 2 * e + 1]), K, -ref));
          sum[0] += a;
          sum[1] += d;
          const __half2 h = __floats2half2_rn(a, d);
          const float2 f = __half22float2(h);
          hi[e] = as_u32(h);
          lo[e] = pack_half2(a - f.x, d - f.y);
        }
        tmem_st_x16(S + 16 * q, hi);
        tmem_st_x16(S + 64 + 16 * q, lo);
      }
      l = l * alpha + (sum[0] + sum[1]);
      if (t > 0) {
        // the accumulator may be touched once the product of the tile before has run
        if (__any_sync(0xffffffffu, alpha != 1.f)) {
          bad = !mbar_wait(O_DONE(b ^ 1), (uint32_t)(((t - 1) >> 1) & 1), abort_s);
          bad = __any_sync(0xffffffffu, bad);
          if (bad) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t o[16];
            tmem_ld_x16(tmem_base + MQ_COL_O + 16 * c + lane_off, o);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st_x16(tmem_base + MQ_COL_O + 16 * c + lane_off, o);
          }
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(P_READY(b));
    }
    if (!bad) {
      bad = !mbar_wait(O_DONE((nt - 1) & 1), (uint32_t)(((nt - 1) >> 1) & 1), abort_s);
      bad = __any_sync(0xffffffffu, bad);
    }
    if (!bad) {
      tc_fence_after();
      const int h = kv * GQA + (row & 3);
      float* rec = p.part + (((size_t)share * p.nkv + kv) * (gridDim.y * 128) + row) * PART;
      const float inv = 1.f / l;
      if (p.shares > 1) *reinterpret_cast<float4*>(rec) = make_float4(m, l, 0.f, 0.f);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint32_t o[16];
        tmem_ld_x16(tmem_base + MQ_COL_O + 16 * c + lane_off, o);
        tmem_wait_ld();
        if (j >= p.s) {
          // a row behind the last query token
        } else if (p.shares > 1) {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<float4*>(rec + 4 + 16 * c + 4 * e) =
                make_float4(__uint_as_float(o[4 * e]), __uint_as_float(o[4 * e + 1]), __uint_as_float(o[4 * e + 2]), __uint_as_float(o[4 * e + 3]));
        } else {
          uint32_t w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) w[e] = pack_half2(__uint_as_float(o[2 * e]) * inv, __uint_as_float(o[2 * e + 1]) * inv);
          uint4* dst = reinterpret_cast<uint4*>(p.out + ((size_t)j * p.nkv * GQA + h) * HD + 16 * c);
          dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
          dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
        __syncwarp();
      }
    }
  }
  if (tid == 0 && *abort_s && p.status) atomicExch(p.status, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem_base, 512);
}

// one warp per (query token, head): lane owns channels 4 lane .. + 3
__global__ void __launch_bounds__(256) multiquery_merge_kernel(const float* __restrict__ part, int shares, int nkv, int rows_pad, int s,
                                                               __half* __restrict__ out) {
  const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, n_q = nkv * GQA;
  if (w >= s * n_q) return;
  const int j = w / n_q, h = w - j * n_q, kv = h / GQA, row = 4 * j + (h % GQA);
  const float* rec = part + ((size_t)kv * rows_pad + row) * PART;
  const size_t stride = (size_t)nkv * rows_pad * PART;
  float M = neg_inf();
  for (int i = lane; i < shares; i += 32) M = fmaxf(M, rec[i * stride]);
  M = warp_max(M);
  float L = 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
  for (int i = 0; i < shares; ++i) {
    const float* r = rec + i * stride;
    const float m = r[0], wt = m == neg_inf() ? 0.f : exp2f(m - M);
    const float4 x = *reinterpret_cast<const float4*>(r + 4 + 4 * lane);
    L = fmaf(wt, r[1], L);
    a.x = fmaf(wt, x.x, a.x); a.y = fmaf(wt, x.y, a.y); a.z = fmaf(wt, x.z, a.z); a.w = fmaf(wt, x.w, a.w);
  }
  const float inv = 1.f / L;
  *reinterpret_cast<uint2*>(out + ((size_t)j * n_q + h) * HD + 4 * lane) = make_uint2(pack_half2(a.x * inv, a.y * inv), pack_half2(a.z * inv, a.w * inv));
}

struct MqLayout { size_t k, v, part, bytes; int n_mid_tiles, n_tiles, m_tiles, shares; };
static MqLayout mq_layout(const ShardDecodeShape& sh, int s) {
  MqLayout l;
  const int n_rows = sh.n_sink + sh.n_win + sh.n_stream + sh.n_dec;
  l.n_mid_tiles = (sh.n_comp + 127) / 128;
  l.n_tiles = l.n_mid_tiles + (n_rows + 127) / 128;
  l.m_tiles = (4 * s + 127) / 128;
  // shares of the tiles: one CTA per SM in all, at least two tiles each
  const int sms = sm_count() > 0 ? sm_count() : 148;
  l.shares = sms / (l.m_tiles * sh.nkv);
  if (l.shares > l.n_tiles / 2) l.shares = l.n_tiles / 2;
  if (l.shares < 1) l.shares = 1;
  const size_t img = (size_t)sh.nkv * l.n_tiles * MQ_TILE_BYTES;
  l.k = 0;
  l.v = img;
  l.part = 2 * img;
  l.bytes = l.part + (l.shares > 1 ? (size_t)l.shares * sh.nkv * l.m_tiles * 128 * PART * 4 : 0);
  return l;
}

}  // namespace shard

using namespace shard;

// implemented in readback.cu
int shard_b200_check_read_back(const ShardSeq* seq_host, const ShardDecodeShape* shape_host, const float* codebook);

static int mq_check(const ShardDecodeShape* sh, int s) {
  if (!sh || s < 1 || s > 65536 || sh->nkv < 1 || sh->n_q != sh->nkv * GQA || sh->rank < 32 || sh->rank > 192 || (sh->rank % 32) ||
      sh->n_comp < 0 || sh->n_sink < 0 || sh->n_win < 0 || sh->n_stream < 0 || sh->n_dec < 0 || (sh->dec_cap != 0 && sh->dec_cap < sh->n_dec))
    return SHARD_E_ARG;
  // the new tokens are the last rows of the stream, or of the fp16 decode buffer
  if (sh->n_dec > 0 ? s > sh->n_dec || sh->n_stream > 0 : s > sh->n_stream) return SHARD_E_ARG;
  return SHARD_OK;
}

extern "C" size_t shard_b200_multiquery_workspace_bytes(const ShardDecodeShape* shape_host, int32_t n_tok) {
  if (mq_check(shape_host, n_tok) != SHARD_OK) return 0;
  return mq_layout(*shape_host, n_tok).bytes;
}

extern "C" int shard_b200_multiquery_attn(const ShardSeq* seq_host, const ShardDecodeShape* shape_host, const void* q_f16,
                                          int64_t q_head_stride, int64_t q_tok_stride, int32_t n_tok, const float* inv_freq,
                                          const float* codebook, int32_t compress_start, void* out_f16, void* workspace,
                                          size_t workspace_bytes, int* status_dev, void* stream) {
  if (!seq_host || !q_f16 || !inv_freq || !out_f16 || !workspace) return SHARD_E_ARG;
  int rc = mq_check(shape_host, n_tok);
  if (rc != SHARD_OK) return rc;
  const ShardDecodeShape& sh = *shape_host;
  const MqLayout l = mq_layout(sh, n_tok);
  if (workspace_bytes < l.bytes) return SHARD_E_WORKSPACE;
  if (((uintptr_t)workspace & 127) || ((uintptr_t)q_f16 & 7) || (q_head_stride & 3) || (q_tok_stride & 3) || ((uintptr_t)out_f16 & 15))
    return SHARD_E_ALIGN;
  static std::atomic<bool> configured[MAX_DEVICES];
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= MAX_DEVICES) return SHARD_E_ARG;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(multiquery_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MQ_SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured[dev].store(true, std::memory_order_release);
  }
  unsigned char* ws = (unsigned char*)workspace;
  cudaStream_t st = (cudaStream_t)stream;
  rc = shard_b200_check_read_back(seq_host, shape_host, codebook);
  if (rc != SHARD_OK) return rc;
  rc = launch_read_back_any(*seq_host, sh, inv_freq, codebook, compress_start, ws + l.k, ws + l.v, true, status_dev, st);
  if (rc) return rc;
  MultiQueryParams p{};
  p.q = (const __half*)q_f16;
  p.q_head = q_head_stride;
  p.q_tok = q_tok_stride;
  p.out = (__half*)out_f16;
  p.k_img = ws + l.k;
  p.v_img = ws + l.v;
  p.part = (float*)(ws + l.part);
  p.status = status_dev;
  p.s = n_tok;
  p.nkv = sh.nkv;
  p.n_mid_tiles = l.n_mid_tiles;
  p.n_comp = sh.n_comp;
  p.n_rows = sh.n_sink + sh.n_win + sh.n_stream + sh.n_dec;
  p.n_tiles = l.n_tiles;
  p.shares = l.shares;
  multiquery_kernel<<<dim3(l.shares, l.m_tiles, sh.nkv), MQ_THREADS, MQ_SMEM_BYTES, st>>>(p);
  if (l.shares > 1)
    multiquery_merge_kernel<<<(n_tok * sh.n_q + 7) / 8, 256, 0, st>>>(p.part, l.shares, sh.nkv, l.m_tiles * 128, n_tok, p.out);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}
