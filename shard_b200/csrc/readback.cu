// Compressed layer -> fp16 keys and values: [sink | middle | window | stream | fp16 decode buffer],
// the whole `layer.keys` / `layer.values` of the non-fused read path in one launch.
//
//   K[t] = RoPE_{pos_t}( coef_t . W + mean )      V[t] = H128( codebook[idx_t] * ch ) / sqrt(128)
//
// Two output forms: row-major [nkv][rows][128] (what a model's stock attention reads), and tile
// images -- 128-row tiles in the 128-byte-swizzled operand layout of tcgen05.mma, row pieces padded to
// whole tiles -- which the multi-query attention kernel fetches with plain bulk copies.
//
// Bound: the fp16 output (134 MB for one 32K layer, 21 us at the measured copy rate; the compressed
// input is a tenth of it).  One CTA per SM takes a 128-token tile and a run of KV heads: the tile's
// int4 coefficients become the tensor-memory A operand once, the weights of the next head land by bulk
// copy while the current head is worked on, and the rotation's cos / sin (one sincosf per token and
// pair, the expensive part of the epilogue) are computed once per tile and kept in tensor memory for
// all heads.  Warps 0-3 turn accumulators into keys; warps 4-7 do the values meanwhile, one thread per
// (token, head) vector with the whole 128-point butterfly in registers (no shuffles).  Both write
// through a swizzled shared-memory tile so that global stores are full lines.
// Measured (8 KV heads, 192 components): 22 us for a layer of 8K tokens (34 MB written: 1.5 TB/s), 70 us for
// one of 32K (1.9 TB/s); three 8K layers with their host work 71 us, 5 477 us as PyTorch operations.
#include <atomic>

#include "decode_common.cuh"
#include "tcgen05.cuh"

namespace shard {

constexpr int RB_THREADS = 256;
constexpr int RB_TILE_BYTES = 32768;      // 128 rows x 128 fp16, two 64-channel halves of 16 KB
constexpr int RB_CB_COPIES = 4;
__host__ __device__ constexpr int rb_w_bytes(int nw) { return ((32 * nw + 16 + 63) / 64) * 16384; }
__host__ __device__ constexpr int rb_smem_bytes(int nw) {
  return 1024 + 2 * rb_w_bytes(nw) + 2 * RB_TILE_BYTES + 2048 * RB_CB_COPIES + 1024 /* codebook of streamed rows */ + 256;
}
// tensor memory columns: two accumulator stages, A operand, cos / sin of the tile's tokens
constexpr int RB_COL_A = 256, RB_COL_CS = 384;

struct ReadBackParams {
  ShardSeq seq;
  ShardDecodeShape sh;
  const float* inv_freq;
  const float* codebook;
  int compress_start;
  int n_tiles;            // 128-token tiles of the middle
  int heads_per_cta;      // KV heads of one CTA
  int n_mid_ctas;         // CTAs on the middle; the ones behind it take the other rows
  int rows_per_head;      // output rows per KV head: all rows, or (image form) 128 * tiles
  __half* k_out;
  __half* v_out;
  int* status;
};

// byte offset of 16-byte chunk c (0..15) of row r (0..127) inside a tile image
__device__ __forceinline__ uint32_t rb_img(int r, int c) { return (uint32_t)((c >> 3) * 16384) + sw128_off(r, c & 7); }

// One row (row `r` of the output, channels 4*lane..+3 of KV head `kv`) outside the middle.
template <bool IMAGE>
__device__ __forceinline__ void rb_store4(__half* out, int rows_per_head, int kv, int r, int lane, uint2 v) {
  if (IMAGE) {
    unsigned char* tile = reinterpret_cast<unsigned char*>(out) + ((size_t)kv * (rows_per_head >> 7) + (r >> 7)) * RB_TILE_BYTES;
    *reinterpret_cast<uint2*>(tile + rb_img(r & 127, lane >> 1) + (lane & 1) * 8) = v;
  } else {
    *reinterpret_cast<uint2*>(out + ((size_t)kv * rows_per_head + r) * HD + 4 * lane) = v;
  }
}

// Rows outside the middle, a warp per (row, KV head): fp16 rows are copied, streamed rows dequantised
// exactly as stream_dequant_kernel does; the newest streamed row is quantised first if it is pending.
template <bool IMAGE>
__device__ __forceinline__ void rb_rows(const ReadBackParams& p, int cta, int n_ctas, float* cbs, int tid) {
  const ShardSeq& sq = p.seq;
  const ShardDecodeShape& sh = p.sh;
  const int warp = tid >> 5, lane = tid & 31;
  const int n_fp = sh.n_sink + sh.n_win, n_rows = n_fp + sh.n_stream + sh.n_dec;
  // image form: the rows follow the middle's tiles, and the last tile is filled up with zeros
  const int n_img = IMAGE ? ((n_rows + 127) & ~127) : n_rows;
  if (sh.n_stream > 0) {
    for (int i = tid; i < 256; i += RB_THREADS) cbs[i] = p.codebook[i];
    __syncthreads();
  }
  const float4 sg = sh.n_stream > 0 ? *reinterpret_cast<const float4*>(sq.signs + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
  const float sgn[4] = {sg.x, sg.y, sg.z, sg.w};
  for (int w = cta * (RB_THREADS / 32) + warp; w < n_img * sh.nkv; w += n_ctas * (RB_THREADS / 32)) {
    const int u = w / sh.nkv, kv = w - u * sh.nkv;
    uint2 k = make_uint2(0u, 0u), v = make_uint2(0u, 0u);
    if (u < n_rows) {
      const bool streamed = u >= n_fp && u < n_fp + sh.n_stream;
      if (!streamed) {
        const bool in_sink = u < sh.n_sink, in_dec = u >= n_fp;
        const int r = in_sink ? u : (in_dec ? u - n_fp - sh.n_stream : u - sh.n_sink);
        const int rows = in_sink ? sh.n_sink : (in_dec ? (sh.dec_cap > 0 ? sh.dec_cap : sh.n_dec) : sh.n_win);
        const __half* kb = reinterpret_cast<const __half*>(in_sink ? sq.sink_k : (in_dec ? sq.dec_k : sq.win_k));
        const __half* vb = reinterpret_cast<const __half*>(in_sink ? sq.sink_v : (in_dec ? sq.dec_v : sq.win_v));
        const size_t off = ((size_t)kv * rows + r) * HD + 4 * lane;
        if (sh.append == 2 && u == n_rows - 1) {                 // the newest fp16 row is still to be written
          k = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(sq.new_k) + kv * HD + 4 * lane);
          v = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(sq.new_v) + kv * HD + 4 * lane);
          *reinterpret_cast<uint2*>(const_cast<__half*>(kb) + off) = k;
          *reinterpret_cast<uint2*>(const_cast<__half*>(vb) + off) = v;
        } else {
          k = *reinterpret_cast<const uint2*>(kb + off);
          v = *reinterpret_cast<const uint2*>(vb + off);
        }
      } else {
        if (sh.append == 1 && u == n_fp + sh.n_stream - 1) {
          append_new_token(sq, sh, kv, cbs, false, lane);
          append_new_token(sq, sh, kv, cbs, true, lane);
          __syncwarp();
        }
        const size_t row = (size_t)(u - n_fp) * sh.nkv + kv;
        const uint32_t kc = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_k_idx + row * HD + 4 * lane));
        const uint32_t vc = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_v_idx + row * HD + 4 * lane));
        const float kn = __half2float(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(sq.st_k_norm) + row)));
        const float vn = __half2float(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(sq.st_v_norm) + row)));
        float xk[4], xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { xk[i] = cbs[(kc >> (8 * i)) & 0xff]; xv[i] = cbs[(vc >> (8 * i)) & 0xff]; }
        fwht128_lane4(xk, lane);
        fwht128_lane4(xv, lane);
        __half ko[4], vo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __half ku = __float2half_rn(__fmul_rn(__fdiv_rn(xk[i], SQRT_HD), sgn[i]));
          const __half vu = __float2half_rn(__fmul_rn(__fdiv_rn(xv[i], SQRT_HD), sgn[i]));
          ko[i] = __float2half_rn(__fmul_rn(__half2float(ku), kn));
          vo[i] = __float2half_rn(__fmul_rn(__half2float(vu), vn));
        }
        k = make_uint2((uint32_t)__half_as_ushort(ko[0]) | ((uint32_t)__half_as_ushort(ko[1]) << 16),
                       (uint32_t)__half_as_ushort(ko[2]) | ((uint32_t)__half_as_ushort(ko[3]) << 16));
        v = make_uint2((uint32_t)__half_as_ushort(vo[0]) | ((uint32_t)__half_as_ushort(vo[1]) << 16),
                       (uint32_t)__half_as_ushort(vo[2]) | ((uint32_t)__half_as_ushort(vo[3]) << 16));
      }
    }
    const int n_mid = sh.n_comp;
    const int r = IMAGE ? p.n_tiles * 128 + u : (u < sh.n_sink ? u : u + n_mid);
    rb_store4<IMAGE>(p.k_out, p.rows_per_head, kv, r, lane, k);
    rb_store4<IMAGE>(p.v_out, p.rows_per_head, kv, r, lane, v);
  }
}

// A warp's 32 rows of a finished tile image in shared memory -> row-major global rows: sixteen lanes
// write one 256-byte row, two rows per instruction.
__device__ __forceinline__ void rb_flush_rows(const unsigned char* img, __half* dst_row0, int row0, int n_valid, int lane) {
  const int c = lane & 15;
#pragma unroll 4
  for (int i = 0; i < 16; ++i) {
    const int r = row0 + 2 * i + (lane >> 4);
    const uint4 v = *reinterpret_cast<const uint4*>(img + rb_img(r, c));
    if (r < n_valid) *reinterpret_cast<uint4*>(dst_row0 + (size_t)r * HD + 8 * c) = v;
  }
}
// The same rows -> the tile image in global memory, as it lies in shared memory (rows behind n_valid
// are zero in both): lanes copy consecutive 16-byte pieces.
__device__ __forceinline__ void rb_flush_image(const unsigned char* img, unsigned char* dst, int row0, int lane) {
#pragma unroll 4
  for (int i = 0; i < 16; ++i) {
    const uint32_t off = (uint32_t)((i >> 3) * 16384 + row0 * 128 + (i & 7) * 512 + lane * 16);
    *reinterpret_cast<uint4*>(dst + off) = *reinterpret_cast<const uint4*>(img + off);
  }
}

template <int NW, bool IMAGE>
__global__ void __launch_bounds__(RB_THREADS, 1) read_back_kernel(const __grid_constant__ ReadBackParams p) {
  constexpr int R = NW * 32, KSTEPS = R / 16 + 1, W_BYTES = rb_w_bytes(NW);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  unsigned char* w_s = smem;                                   // [2] weights of a head
  unsigned char* k_img = w_s + 2 * W_BYTES;                    // keys of a (tile, head)
  unsigned char* v_img = k_img + RB_TILE_BYTES;                // values
  uint2* cbv = reinterpret_cast<uint2*>(v_img + RB_TILE_BYTES);   // V codebook, four interleaved copies
  float* cbs = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(cbv) + 2048 * RB_CB_COPIES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(cbs + 256);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  volatile int* abort_s = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const ShardSeq& sq = p.seq;
  const ShardDecodeShape& sh = p.sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((int)blockIdx.x >= p.n_mid_ctas) {                       // (uniform over the CTA: no tensor memory, no barriers)
    rb_rows<IMAGE>(p, blockIdx.x - p.n_mid_ctas, gridDim.x - p.n_mid_ctas, cbs, tid);
    return;
  }
  const int groups = sh.nkv / p.heads_per_cta;
  const int tile = blockIdx.x / groups, kv0 = (blockIdx.x - tile * groups) * p.heads_per_cta, nh = p.heads_per_cta;
  const int t0 = tile * 128, n_valid = min(128, sh.n_comp - t0);

  const uint32_t bar0 = smem_u32(bars);
  auto W_FULL = [&](int b) { return bar0 + 8u * (uint32_t)b; };
  auto D_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(2 + b); };
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
    if (lane == 0) {
      for (int b = 0; b < 2; ++b) { mbar_init(W_FULL(b), 1); mbar_init(D_FULL(b), 1); }
      *abort_s = 0;
      fence_mbar_init();
    }
  }
  {
    const uint2 e = reinterpret_cast<const uint2*>(sq.v_centroids)[tid];
#pragma unroll
    for (int c = 0; c < RB_CB_COPIES; ++c) cbv[RB_CB_COPIES * tid + c] = e;
  }
  auto issue_w = [&](int h) {
    mbar_expect_tx(W_FULL(h & 1), (uint32_t)W_BYTES);
    for (int a = 0; a < W_BYTES / 16384; ++a)
      bulk_g2s(smem_u32(w_s + (h & 1) * W_BYTES + a * 16384),
               reinterpret_cast<const unsigned char*>(sq.k_wprep) + (size_t)(kv0 + h) * W_BYTES + a * 16384, 16384u, W_FULL(h & 1));
  };
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (tid == 0) {
    issue_w(0);
    if (nh > 1) issue_w(1);
  }
  bool bad = false;
  if (warp < 4) {
    // ---- keys: thread = token ------------------------------------------------------------------
    const int m = warp * 32 + lane;
    const uint32_t lane_off = (uint32_t)(warp * 32) << 16;
    {
      // coefficients -> A operand (position R is 1: it multiplies the mean slice of the weights)
      const uint32_t lane_A = tmem_base + RB_COL_A + lane_off;
      const uint4* row = reinterpret_cast<const uint4*>(sq.k_coeffs + (size_t)(t0 + min(m, n_valid - 1)) * (R / 2));
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const uint4 xi = row[i];
        const uint32_t wv[4] = {xi.x, xi.y, xi.z, xi.w};
        uint32_t o[16];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t hi = wv[e] >> 8;
          o[4 * e + 0] = nib2half2_tc(wv[e]);
          o[4 * e + 1] = nib2half2_hi(wv[e]);
          o[4 * e + 2] = nib2half2_tc(hi);
          o[4 * e + 3] = nib2half2_hi(hi);
        }
        tmem_st_x16(lane_A + 16 * i, o);
      }
      const uint32_t ones[8] = {0x00003C00u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      tmem_st_x8(lane_A + R / 2, ones);
      tmem_wait_st();
      tc_fence_before();
    }
    auto issue_mma = [&](int h) -> bool {
      if (!mbar_wait(W_FULL(h & 1), (uint32_t)((h >> 1) & 1), abort_s)) return false;
      tc_fence_after();
      const uint64_t wdesc = smem_desc_sw128(smem_u32(w_s + (h & 1) * W_BYTES), 16, 1024);
      constexpr uint32_t IDESC = umma_idesc(128, 128, false, false);
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ++ks)
        umma_ts(tmem_base + 128 * (h & 1), tmem_base + RB_COL_A + 8 * ks, wdesc + (uint64_t)(((ks >> 2) * 16384 + (ks & 3) * 32) >> 4),
                IDESC, ks > 0 ? 1u : 0u, 1u);
      umma_commit(D_FULL(h & 1), 1u);
      return true;
    };
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (tid == 0) {
      tc_fence_after();
      bad |= !issue_mma(0);
    }
    __syncwarp();
    {
      // cos / sin of the token's 64 pairs, fp32, eight pairs a column block (16 columns)
      const float pos = (float)(p.compress_start + t0 + m);
#pragma unroll 1
      for (int ch = 0; ch < 8; ++ch) {
        uint32_t cs[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float sn, co;
          sincosf(__fmul_rn(pos, __ldg(p.inv_freq + 8 * ch + j)), &sn, &co);
          cs[j] = __float_as_uint(co);
          cs[8 + j] = __float_as_uint(sn);
        }
        tmem_st_x16(tmem_base + RB_COL_CS + 16 * ch + lane_off, cs);
      }
      tmem_wait_st();
    }
    for (int h = 0; h < nh; ++h) {
      if (tid == 0 && h + 1 < nh) bad |= !issue_mma(h + 1);    // stage (h+1)&1 was read by all four warps before the barrier below
      __syncwarp();
      bad |= !mbar_wait(D_FULL(h & 1), (uint32_t)((h >> 1) & 1), abort_s);
      tc_fence_after();
      const uint32_t D = tmem_base + 128 * (h & 1) + lane_off, CS = tmem_base + RB_COL_CS + lane_off;
#pragma unroll 2
      for (int ch = 0; ch < 8; ++ch) {
        uint32_t cr[8], dr[8], cs[16];
        tmem_ld_x8(D + 8 * ch, cr);
        tmem_ld_x8(D + 64 + 8 * ch, dr);
        tmem_ld_x16(CS + 16 * ch, cs);
        tmem_wait_ld();
        uint32_t oc[4], od[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float c[2], d[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = __uint_as_float(cr[2 * j + e]), y = __uint_as_float(dr[2 * j + e]);
            const float co = __uint_as_float(cs[2 * j + e]), sn = __uint_as_float(cs[8 + 2 * j + e]);
            c[e] = fmaf(x, co, -__fmul_rn(y, sn));
            d[e] = fmaf(y, co, __fmul_rn(x, sn));
          }
          oc[j] = pack_half2(c[0], c[1]);
          od[j] = pack_half2(d[0], d[1]);
        }
        const bool live = m < n_valid;
        *reinterpret_cast<uint4*>(k_img + rb_img(m, ch)) = live ? make_uint4(oc[0], oc[1], oc[2], oc[3]) : make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(k_img + rb_img(m, 8 + ch)) = live ? make_uint4(od[0], od[1], od[2], od[3]) : make_uint4(0u, 0u, 0u, 0u);
      }
      tc_fence_before();
      asm volatile("bar.sync 1, 128;" ::: "memory");           // the stage and its weights are free
      if (tid == 0 && h + 2 < nh) issue_w(h + 2);
      if (IMAGE)
        rb_flush_image(k_img, reinterpret_cast<unsigned char*>(p.k_out) + ((size_t)(kv0 + h) * (p.rows_per_head >> 7) + tile) * RB_TILE_BYTES, warp * 32, lane);
      else
        rb_flush_rows(k_img, p.k_out + ((size_t)(kv0 + h) * p.rows_per_head + sh.n_sink + t0) * HD, warp * 32, n_valid, lane);
      __syncwarp();
    }
  } else {
    // ---- values: thread = (token, head) vector --------------------------------------------------
    const int row0 = (warp - 4) * 32, m = row0 + lane;
    const uint2* cb = cbv + (lane & (RB_CB_COPIES - 1));
    for (int h = 0; h < nh; ++h) {
      const int kv = kv0 + h;
      const uint4* codes = reinterpret_cast<const uint4*>(sq.v_indices + ((size_t)kv * sh.n_comp + t0 + min(m, n_valid - 1)) * VQ_GROUPS);
      const uint4 c0 = codes[0], c1 = codes[1];
      const uint32_t cw[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
      const uint2* chp = reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(sq.v_ch) + (size_t)kv * HD);
      float x[HD];
#pragma unroll
      for (int g = 0; g < VQ_GROUPS; ++g) {
        const uint2 e = cb[RB_CB_COPIES * ((cw[g >> 2] >> (8 * (g & 3))) & 0xff)];
        const uint2 s = __ldg(chp + g);
        const float2 e0 = __half22float2(as_half2(e.x)), e1 = __half22float2(as_half2(e.y));
        const float2 s0 = __half22float2(as_half2(s.x)), s1 = __half22float2(as_half2(s.y));
        // the group's first two butterfly stages on the way in
        const float a0 = __fmul_rn(e0.x, s0.x), a1 = __fmul_rn(e0.y, s0.y), a2 = __fmul_rn(e1.x, s1.x), a3 = __fmul_rn(e1.y, s1.y);
        const float b0 = a0 + a1, b1 = a0 - a1, b2 = a2 + a3, b3 = a2 - a3;
        x[4 * g] = b0 + b2; x[4 * g + 1] = b1 + b3; x[4 * g + 2] = b0 - b2; x[4 * g + 3] = b1 - b3;
      }
#pragma unroll
      for (int hh = 4; hh < HD; hh <<= 1) {
#pragma unroll
        for (int i = 0; i < HD; ++i) {
          if (!(i & hh)) { const float a = x[i], b = x[i + hh]; x[i] = a + b; x[i + hh] = a - b; }
        }
      }
      const float scale = m < n_valid ? INV_SQRT_HD : 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c)
        *reinterpret_cast<uint4*>(v_img + rb_img(m, c)) =
            make_uint4(pack_half2(x[8 * c] * scale, x[8 * c + 1] * scale), pack_half2(x[8 * c + 2] * scale, x[8 * c + 3] * scale),
                       pack_half2(x[8 * c + 4] * scale, x[8 * c + 5] * scale), pack_half2(x[8 * c + 6] * scale, x[8 * c + 7] * scale));
      __syncwarp();
      if (IMAGE)
        rb_flush_image(v_img, reinterpret_cast<unsigned char*>(p.v_out) + ((size_t)kv * (p.rows_per_head >> 7) + tile) * RB_TILE_BYTES, row0, lane);
      else
        rb_flush_rows(v_img, p.v_out + ((size_t)kv * p.rows_per_head + sh.n_sink + t0) * HD, row0, n_valid, lane);
      __syncwarp();
    }
  }
  if (bad && p.status) atomicExch(p.status, 1);
  if (tid == 0 && *abort_s) {
    // gave up: weights may still be landing in this CTA's shared memory
    for (int h = max(0, nh - 2); h < nh; ++h) mbar_wait(W_FULL(h & 1), (uint32_t)((h >> 1) & 1), abort_s);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, 512);
}

template <int NW, bool IMAGE>
static int launch_read_back(const ReadBackParams& p, int grid, cudaStream_t st) {
  constexpr int SMEM = rb_smem_bytes(NW);
  static std::atomic<bool> configured[MAX_DEVICES];
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= MAX_DEVICES) return SHARD_E_ARG;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(read_back_kernel<NW, IMAGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev].store(true, std::memory_order_release);
  }
  read_back_kernel<NW, IMAGE><<<grid, RB_THREADS, SMEM, st>>>(p);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// Row-major (image = 0) or tile-image (image = 1) read-back of one layer; shared by the C entry point
// and the multi-query attention.
int launch_read_back_any(const ShardSeq& seq, const ShardDecodeShape& sh, const float* inv_freq, const float* codebook,
                         int compress_start, void* k_out, void* v_out, bool image, int* status, cudaStream_t st) {
  ReadBackParams p{};
  p.status = status;
  p.seq = seq;
  p.sh = sh;
  p.inv_freq = inv_freq;
  p.codebook = codebook;
  p.compress_start = compress_start;
  p.n_tiles = (sh.n_comp + 127) / 128;
  const int n_rows = sh.n_sink + sh.n_win + sh.n_stream + sh.n_dec;
  p.rows_per_head = image ? 128 * (p.n_tiles + (n_rows + 127) / 128) : sh.n_comp + n_rows;
  p.k_out = (__half*)k_out;
  p.v_out = (__half*)v_out;
  // Heads per CTA: a wave costs its heads plus about two heads' worth of set-up (A operand, cos / sin,
  // first weights); take the split whose waves cost least.  Few tiles: heads go to CTAs of their own;
  // many: all heads of a tile share its set-up.
  const int sms = sm_count() > 0 ? sm_count() : 1;
  long long best = -1;
  for (int hpc = 1; hpc <= sh.nkv; ++hpc) {
    if (sh.nkv % hpc) continue;
    const long long ctas = (long long)p.n_tiles * (sh.nkv / hpc);
    const long long cost = (ctas + sms - 1) / sms * (hpc + 2);
    if (best < 0 || cost < best) { best = cost; p.heads_per_cta = hpc; }
  }
  p.n_mid_ctas = p.n_tiles * (sh.nkv / (p.heads_per_cta > 0 ? p.heads_per_cta : 1));
  const int row_units = (image ? ((n_rows + 127) & ~127) : n_rows) * sh.nkv;
  int row_ctas = (row_units + 31) / 32;                 // four rows a warp
  if (row_ctas > 2 * sms) row_ctas = 2 * sms;
  const int grid = p.n_mid_ctas + row_ctas;
  if (grid == 0) return 0;
#define SHARD_RB(NW) (image ? launch_read_back<NW, true>(p, grid, st) : launch_read_back<NW, false>(p, grid, st))
  switch (sh.rank / 32) {
    case 1: return SHARD_RB(1);
    case 2: return SHARD_RB(2);
    case 3: return SHARD_RB(3);
    case 4: return SHARD_RB(4);
    case 5: return SHARD_RB(5);
    default: return SHARD_RB(6);
  }
#undef SHARD_RB
}

}  // namespace shard

using namespace shard;

// Pointers and sizes of a read-back (also of the multi-query attention, which starts with one).
int shard_b200_check_read_back(const ShardSeq* seq_host, const ShardDecodeShape* shape_host, const float* codebook) {
  if (!seq_host || !shape_host) return SHARD_E_ARG;
  const ShardSeq& s = *seq_host;
  const ShardDecodeShape& sh = *shape_host;
  if (sh.nkv < 1 || sh.rank < 32 || sh.rank > 192 || (sh.rank % 32) || sh.n_comp < 0 || sh.n_sink < 0 || sh.n_win < 0 ||
      sh.n_stream < 0 || sh.n_dec < 0 || (sh.dec_cap != 0 && sh.dec_cap < sh.n_dec))
    return SHARD_E_ARG;
  if (sh.n_comp > 0 && (!s.k_coeffs || !s.k_wprep || !s.v_indices || !s.v_centroids || !s.v_ch)) return SHARD_E_ARG;
  if (sh.n_sink > 0 && (!s.sink_k || !s.sink_v)) return SHARD_E_ARG;
  if (sh.n_win > 0 && (!s.win_k || !s.win_v)) return SHARD_E_ARG;
  if (sh.n_dec > 0 && (!s.dec_k || !s.dec_v)) return SHARD_E_ARG;
  if (sh.n_stream > 0 && (!codebook || !s.st_k_idx || !s.st_v_idx || !s.st_k_norm || !s.st_v_norm || !s.signs)) return SHARD_E_ARG;
  if (sh.append < 0 || sh.append > 2 || (sh.append && (!s.new_k || !s.new_v)) || (sh.append == 1 && sh.n_stream < 1) ||
      (sh.append == 2 && sh.n_dec < 1))
    return SHARD_E_ARG;
  if (((uintptr_t)s.k_coeffs & 15) || ((uintptr_t)s.k_wprep & 15) || ((uintptr_t)s.v_indices & 15) || ((uintptr_t)s.v_centroids & 7) ||
      ((uintptr_t)s.v_ch & 7) || ((uintptr_t)s.sink_k & 7) || ((uintptr_t)s.sink_v & 7) || ((uintptr_t)s.win_k & 7) ||
      ((uintptr_t)s.win_v & 7) || ((uintptr_t)s.dec_k & 7) || ((uintptr_t)s.dec_v & 7) || ((uintptr_t)s.st_k_idx & 3) ||
      ((uintptr_t)s.st_v_idx & 3) || ((uintptr_t)s.signs & 15) || ((uintptr_t)s.new_k & 7) || ((uintptr_t)s.new_v & 7))
    return SHARD_E_ALIGN;
  return SHARD_OK;
}

extern "C" int shard_b200_read_back(const ShardSeq* seq_host, const ShardDecodeShape* shape_host, const float* inv_freq,
                                    const float* codebook, int32_t compress_start, void* k_out_f16, void* v_out_f16,
                                    int* status_dev, void* stream) {
  if (!inv_freq || !k_out_f16 || !v_out_f16) return SHARD_E_ARG;
  const int rc = shard_b200_check_read_back(seq_host, shape_host, codebook);
  if (rc != SHARD_OK) return rc;
  const ShardSeq& s = *seq_host;
  const ShardDecodeShape& sh = *shape_host;
  if (((uintptr_t)k_out_f16 | (uintptr_t)v_out_f16) & 15) return SHARD_E_ALIGN;
  return launch_read_back_any(s, sh, inv_freq, codebook, compress_start, k_out_f16, v_out_f16, false, status_dev, (cudaStream_t)stream);
}
