// One decode step of one layer in one launch: split-KV pass over the compressed middle
// (tcgen05 + tensor memory + bulk copy engine for the reconstruction of the keys, mma.sync fragments for the
// narrow products), the fp16 / streamed rows, the stream append and the combine.
//
// One CTA per SM (16 warps) owns one KV head and a run of 128-token tiles of the middle segment.  Two pipelines take the
// tiles in turn; each has an A slot and a key stage in tensor memory, an issuing thread and a group of four consumer warps.
//
//   copying warps (2)   one thread each: bulk copies of the weights W once, the packed int4 coefficient rows of a tile, its V
//                       codes.  No load instruction touches the cache data.  When the launch before has finished, the two warps
//                       stage the query and, in the CTA that owns the newest streamed row, quantise the new token into it
//   unpack warps (4)    coefficient rows -> fp16 A operand in tensor memory; then this CTA's share of the fp16 sink / window /
//                       decode rows and the streamed rows, sixteen at a time
//   issuing threads (2) MMA1  K_n[128 tok x 128] = A . W^T   (A from tensor memory, W in shared memory; the last k-step adds the
//                       mean).  Two threads, because a hand-over takes a few hundred cycles, during which the tensor core
//                       would stand still: 368 us for four layers of 131K tokens, 393 with one
//   consumer warps (8)  K_n -> half2 -> rotated by the relative phase, in the registers' layout of an mma.sync fragment, so that
//                       S[token][query] = K~ . Q^T needs no trip back through memory; per-warp online softmax with a lazily moving
//                       reference point; the weights transposed in registers (movmatrix) and
//                       O[pair of channels][(query, parity)] += V[pair][(token, parity')] . P -- contracted over (token, parity), a
//                       codebook entry of four channels IS the A fragment: the codes are looked up straight into it and no V tile is ever
//                       written.  All sums of a warp stay in 16 registers
//   epilogue            the 12 warps' states merge into ONE record per CTA and query head
//   combine             per query head: the last warp to write a record merges all of them
//
// A 16-column product on tcgen05 costs as much as one of 128 columns (59 cycles against 67 for a k-step), so scores and P.V took
// 0.94 of a tile's 1.8 K cycles on the tensor core; as mma.sync they take 32 instructions of 8 cycles a warp.  What they cost
// instead: a stream of tcgen05.mma keeps mma.sync waiting, so the consumers' products run between the reconstruction
// products of two tiles.  That, with the latency of a consumer's chain (tensor memory, rotation, scores, softmax, look-ups, P.V: about
// 3 K cycles), bounds a tile: 2.4 to 2.7 K cycles.  Against the kernel with all products on tcgen05, shared-memory V tiles and three groups
// (us a pass): 8K x 12 layers 198 -> 162, 32K x 12 383 -> 324, 131K x 4 408 -> 354, 64 sequences of 8K x 2 923 -> 738.
// Measured and not kept: eight warps to a tile (80 registers: 8K 197, 131K 377), one paced issuing thread, the stage
// handed back before the scores product, polling instead of suspended waits (131K 396).
//
// Launched with programmatic stream serialization: the set-up, the first tiles' unpack and reconstruction products and the rotation of
// each group's first keys (which wait for the query in registers: 32K x 12 345 -> 324 us, 131K x 4 360 -> 354) use only tensors that no
// decode call writes and run before griddepcontrol.wait.
//
// Tensor memory: two key stages of 128 columns, two A slots of R/2 + 8 columns from column 256 on.
// Every hand-over is an mbarrier whose waiters see each of its phases; every wait is bounded and
// raises the CTA's abort flag when it gives up, after which all roles drain, bulk copies and tensor-core work in flight
// are waited for, tensor memory is freed and the status word is set.
#include <atomic>
#include <cstdlib>

#include "decode_common.cuh"
#include "tcgen05.cuh"

namespace shard {

constexpr int PP_ST = 2;                            // pipelines: each an A slot, a key stage, an issuing thread and a consumer group; tile t is pipeline t % 2's
constexpr int PP_CONS_WARPS = 4 * PP_ST;
constexpr int PP_UNPACK_WARP0 = PP_CONS_WARPS;
constexpr int PP_MMA_WARP = PP_CONS_WARPS + 4;
constexpr int PP_ROW_WARPS = PP_CONS_WARPS + 4;     // warps that can attend to rows
constexpr int PP_MEET = HD + 4;                     // floats of a warp's sum in the epilogue
constexpr int PP_SUB = PP_ROW_WARPS / GQA;          // warps per query head in the epilogue and the combine
constexpr int PP_COEF_WARP = PP_MMA_WARP + PP_ST, PP_VCODE_WARP = PP_COEF_WARP + 1;   // one copying thread each
constexpr int PP_THREADS = (PP_VCODE_WARP + 1) * 32;
constexpr int PP_TMEM_COLS = 512;
constexpr int PP_COL_A = 128 * PP_ST;               // the A operand slots: R/2 coefficient columns + 8 constant columns 1, 0, ... each
__host__ __device__ constexpr int pp_a_cols(int nw) { return 16 * nw + 8; }
constexpr int PP_STATE = GQA * HD + 2 * GQA;        // a warp's state, floats: acc[4][128], max[4], sum-exp[4]
constexpr int PP_W_LOG2 = 14;                       // weights of rows' values, at most 2^0.5, times 2^14 in fp16
constexpr float PP_LAZY_LOG2 = 8.f;                 // a softmax reference point moves only when exceeded by more than 2^8
constexpr int PP_C_BUFS = 4;                        // coefficient tiles in shared memory
constexpr int PP_V_BUFS = 6;                        // V code tiles (4 KB) in shared memory
constexpr int PP_SPLIT_COPIES = 16;                 // copies of the stream codebook as two fp16 parts, entry e of copy c at 16 e + c: at most two look-ups of a warp meet in a bank
constexpr int PP_SPLIT_BYTES = 256 * 4 * PP_SPLIT_COPIES;
constexpr int PP_CB_COPIES = 16;                    // copies of the V codebook, entry e of copy c at 16 e + c: a half-warp's look-ups never meet in a bank

// W holds R + 16 contraction positions (the last 16 carry the mean), in 64-position atoms of 16 KB
__host__ __device__ constexpr int pp_w_bytes(int nw) { return ((32 * nw + 16 + 63) / 64) * 16384; }
__host__ __device__ constexpr int pp_c_bytes(int nw) { return nw < 2 ? 2560 : 128 * 16 * nw; }    // (all of them hold the epilogue's sums)
// Shared memory, by address within the CTA's window.  The codebook sits on a multiple of 32 KB, so that a
// look-up's address is (code's bits | this lane's base): one shift and one three-input logic operation.
constexpr int PP_OFF_MISC = 0;                                        // barriers, flags
constexpr int PP_OFF_QUP = 384;                                       // the powers of two by which the queries in code space are scaled, inverse, fp32 [4]
constexpr int PP_OFF_CH = 640;                                        // the head's channel scales, fp16 [128]
constexpr int PP_OFF_QG = 1024;                                       // queries as given, fp16 [4][128]
constexpr int PP_OFF_QS = PP_OFF_QG + GQA * HD * 2;                   // queries in the stream's code space, two fp16 parts [4][2][128]
constexpr int PP_OFF_QF = PP_OFF_QS + GQA * HD * 4;                   // un-rotated queries as matrix fragments [8 k-steps][4 q x 4][2 x half2]
constexpr int PP_OFF_CBS = PP_OFF_QF + 1024;                          // stream codebook, fp32 [256]
constexpr int PP_OFF_V = PP_OFF_CBS + 1024;                           // V codes [buffer][128 tokens][32]
constexpr int PP_HEAD_BYTES = PP_OFF_V + PP_V_BUFS * 4096;
constexpr int PP_CB_ALIGN = 256 * 8 * PP_CB_COPIES;
static_assert(PP_CB_ALIGN % PP_SPLIT_BYTES == 0, "both tables are looked up by (bits of the code | base of the lane)");
static_assert(PP_C_BUFS * 2560 >= GQA * PP_SUB * PP_MEET * 4, "the epilogue's sums fit the coefficients' place");
static_assert(PP_HEAD_BYTES <= PP_CB_ALIGN - 2048, "the head of the layout ends before the first multiple of 32 KB");
__host__ __device__ constexpr int pp_smem_bytes(int nw) {             // from the end of the 1 KB the system keeps
  return 2 * PP_CB_ALIGN + PP_SPLIT_BYTES - 1024 + pp_w_bytes(nw) + PP_C_BUFS * pp_c_bytes(nw) + PP_ROW_WARPS * PP_STATE * 4;
}
// The dynamic part starts behind what the system keeps and the kernel's static variables, on a multiple of 1 KB; the codebook is on the first
// multiple of 32 KB only if the head of the layout ends before it.  The host asks for both sizes before the first launch on a device.
constexpr bool pp_layout_fits(size_t system_bytes, size_t static_bytes) {
  return ((system_bytes + static_bytes + 1023) & ~(size_t)1023) + PP_HEAD_BYTES <= PP_CB_ALIGN;
}
static_assert(pp_layout_fits(1024, 1024) && pp_layout_fits(1024, 0) && !pp_layout_fits(1024, 1025) && !pp_layout_fits(2048, 1024) && !pp_layout_fits(4096, 0),
              "what is there today fits, a static variable beyond the first KB or a larger share of the system's does not");

// single-thread forms (the caller is one elected thread)
__device__ __forceinline__ void umma_ts_1t(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void umma_commit_1t(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Legacy tensor path for the narrow products: D[16 x 8] += A[16 x 16] . B[16 x 8], fp16 with fp32 accumulation.
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16 lanes (rows) x 16 columns of tensor memory, in the register layout of an mma.sync accumulator: r[4 i + 0, 1] are columns
// 8 i + 2 (lane % 4) + 0, 1 of row lane / 4, r[4 i + 2, 3] those of row lane / 4 + 8
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
// wait for the loads above, naming their registers so that no use moves in front of the wait
__device__ __forceinline__ void tmem_wait_frags(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
// transpose of an 8 x 8 matrix of 16-bit values spread over the warp, two per lane
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t x) {
  uint32_t r;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}
__device__ __forceinline__ uint2 lds_u2(uint32_t addr) {
  uint2 r;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(addr));
  return r;
}
__device__ __forceinline__ uint32_t lds_u1(uint32_t addr) {
  uint32_t r;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r) : "r"(addr));
  return r;
}
// ---- rows outside the middle, sixteen at a time on the tensor core -----------------------------------------------------------
// A block of rows has the form of the middle's products: keys are A fragments (a row's 128 channels in any order, as long as the
// query's are in the same), the scores come out with row lane / 4 (+ 8) and query head lane % 4 in a lane, and the values
// are contracted over (row, parity of the channel).  What was 32-bit arithmetic when a warp took two rows at a time (and is in a launch
// without a middle) keeps 22 bits: the weights, the codebook and the queries in code space are two fp16 parts each, the second scaled by 2^11 with
// sums of its own; queries and keys of fp16 rows are exact, and all sums are fp32, rounded to nearest between products.  (A second part
// that is not scaled falls into fp16's subnormals: a weight of 2^-16 kept 9 bits.  A product accumulates with truncation, which a chain of
// them over all channels or blocks adds up.  Values take three of the four products of two parts: the fourth is 2^-22 of the first.)
// The weights of the values, p times the norm of a streamed row, are split as w . 2^14 for w <= 2^0.5, w = p norm over a power
// of two that follows the largest: 22 bits from 1 down to 2^-28, and an error of 2^-50 below.
// Relative error of the sums against float64, fp16 rows / streamed ones: with even weights over 333 rows 6.8e-7 / 7.1e-7 (in 32-bit
// arithmetic 7.0e-7 / 6.4e-7), where rows of weight 2^-20 carry the result 9.4e-7 / 9.4e-7 (8.5e-7 / 8.2e-7; 1.7e-3 and 6.3e-6 with unscaled
// second parts and the products chained).  Against that cheaper form: 8K x 12 layers 160.8 -> 161.7 us, 8 layers with 3001 streamed rows
// 133.7 -> 133.5, one layer of 2K tokens 15.9 -> 16.3 (with what the rounded quotient of the output costs).
// Bound: latency of one block (loads, a chain of products, a softmax over 16 rows) -- some 200 instructions for 16 fp16 rows and
// 700 for streamed ones, whose codes are looked up one by one; two rows at a time, with a reduction over the lanes for each, took
// 1 K cycles a pair.
//
// A streamed row is never rotated back: its key is norm / sqrt(128) . signs o H(codebook[code]), so the QUERY is taken to the
// code space (H(signs o q) / sqrt(128)) and the score is norm . (query . codebook[code]); streamed values are summed in code space
// and the SUM is rotated back, once per warp.  Streamed rows come first, so that one set of accumulators serves both kinds.
struct RowState {
  float m, l;         // of query head lane % 4: reference (log2 domain) and sum of the weights
  int j;              // o is in units of 2^(m + j - PP_W_LOG2)
  float o[4][4];      // channels 16 (lane / 4) + 4 i + j of that head
};
__device__ __forceinline__ void row_state_init(RowState& st) {
  st.m = neg_inf(); st.l = 0.f; st.j = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) st.o[i >> 2][i & 3] = 0.f;
}
// x = a + b / 2^11 with two fp16 values, a in the lower half: 22 bits of x where |x| >= 2^-14, an error of 2^-36 below
constexpr float PP_LO_UP = 2048.f, PP_LO_DOWN = 1.f / PP_LO_UP;
__device__ __forceinline__ uint32_t split_half2(float x) {
  const __half hi = __float2half_rn(x), lo = __float2half_rn((x - __half2float(hi)) * PP_LO_UP);
  return (uint32_t)__half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16);
}
// 16 bytes, L2-coherent, in pieces of PIECE bytes where the address is no multiple of 16
template <int PIECE>
__device__ __forceinline__ uint4 row_load16(const void* at, bool aligned) {
  if (aligned) return __ldcg(reinterpret_cast<const uint4*>(at));
  if (PIECE == 8) {
    const uint2 a = __ldcg(reinterpret_cast<const uint2*>(at)), b = __ldcg(reinterpret_cast<const uint2*>(at) + 1);
    return make_uint4(a.x, a.y, b.x, b.y);
  }
  const unsigned int* w = reinterpret_cast<const unsigned int*>(at);
  return make_uint4(__ldcg(w), __ldcg(w + 1), __ldcg(w + 2), __ldcg(w + 3));
}
// one query head as given -> the code space, fp16 parts out[0..127] and out[128..255] of the query times a power of two that takes
// it into fp16's range (a coordinate is at most 128 / sqrt(128) < 2^3.6 of the largest channel, which the scaling takes to 2^10 .. 2^11);
// returns the power's inverse.  One warp, `sg` its lanes' four signs
__device__ __forceinline__ float stream_query(const float4 sg, const __half* q, __half* out, int lane) {
  const uint2 raw = *reinterpret_cast<const uint2*>(q + 4 * lane);
  const uint32_t mags = __vmaxu2(raw.x & 0x7FFF7FFFu, raw.y & 0x7FFF7FFFu);
  const uint32_t e = __reduce_max_sync(0xffffffffu, max(mags & 0xFFFFu, mags >> 16)) >> 10;   // biased by 15; 0: below 2^-14
  const float2 a = __half22float2(as_half2(raw.x)), c = __half22float2(as_half2(raw.y));
  float x[4] = {a.x * sg.x, a.y * sg.y, c.x * sg.z, c.y * sg.w};
  fwht128_lane4(x, lane);
  const float up = __uint_as_float((127u + 25u - e) << 23);
  uint32_t sp[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) sp[j] = split_half2(x[j] * INV_SQRT_HD * up);
  *reinterpret_cast<uint2*>(out + 4 * lane) = make_uint2(__byte_perm(sp[0], sp[1], 0x5410), __byte_perm(sp[2], sp[3], 0x5410));
  *reinterpret_cast<uint2*>(out + HD + 4 * lane) = make_uint2(__byte_perm(sp[0], sp[1], 0x7632), __byte_perm(sp[2], sp[3], 0x7632));
  return __uint_as_float((127u - 25u + e) << 23);
}
// 2^n, n within -126 .. 127
__device__ __forceinline__ float pow2_whole(int n) { return __int_as_float((n + 127) << 23); }
// weights of a block's rows: this lane has the scores sc[r] of rows lane / 4 + 8 r (log2 domain, -inf: no such row) and the norms vn[r] of
// their values; gives the value weights as B fragments, w[part][m][slot] for rows 8 m + 2 (lane % 4) + slot
__device__ __forceinline__ void block_weights(RowState& st, const float (&sc)[2], const float (&vn)[2], uint32_t (&w)[2][2][2], int lane) {
  // (the logarithms choose the reference and nothing else: the weight is p times the norm)
  float tm = fmaxf(sc[0], sc[1]), tu = fmaxf(sc[0] + __log2f(vn[0]), sc[1] + __log2f(vn[1]));
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) {
    tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, off));
    tu = fmaxf(tu, __shfl_xor_sync(0xffffffffu, tu, off));
  }
  const float m = fmaxf(st.m, tm), m0 = m == neg_inf() ? 0.f : m, u = fmaxf(st.m + (float)st.j, tu);
  // (adding 1.5 . 2^23 rounds to a whole number in the low bits: the weights are at most 2^0.5)
  const int j = u == neg_inf() ? st.j : __float_as_int(fminf(fmaxf(u - m0, -100.f), 100.f) + 12582912.f) - 0x4B400000;
  const float pr[2] = {ex2(sc[0] - m0), ex2(sc[1] - m0)}, al = ex2(st.m - m0);
  st.l = fmaf(st.l, al, pr[0] + pr[1]);
  const float al_o = al * pow2_whole(min(max(st.j - j, -126), 126)), up = pow2_whole(PP_W_LOG2 - j);
  st.m = m; st.j = j;
#pragma unroll
  for (int i = 0; i < 16; ++i) st.o[i >> 2][i & 3] *= al_o;
  const uint32_t odd = (lane >> 2) & 1, sel0 = odd ? 0x1044u : 0x4410u, sel1 = odd ? 0x3244u : 0x4432u;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const uint32_t sp = split_half2(pr[r] * vn[r] * up);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const uint32_t x = transpose_8x8(__byte_perm(sp, 0u, part ? 0x3232 : 0x1010));
      w[part][r][0] = __byte_perm(x, 0u, sel0);
      w[part][r][1] = __byte_perm(x, 0u, sel1);
    }
  }
}
// fp16 rows u0 .. u0 + 15 (sink rows first, then window, then the fp16 decode buffer)
__device__ __forceinline__ void fp16_block(RowState& st, const ShardSeq& sq, const ShardDecodeShape& sh, int kv, int u0, const __half* qg_s, int lane) {
  const int g8 = lane >> 2, t4 = lane & 3, last = sh.n_sink + sh.n_win + sh.n_dec - 1;
  // keys: channels 32 j + 8 t4 .. + 7 of rows g8 and g8 + 8; values: channels 16 g8 .. + 15 of rows 2 t4, 2 t4 + 1, and 8 further
  // (the rows may start between 16-byte boundaries; L2-coherent: the newest row may be this CTA's.  A row behind the last repeats it
  // and gets no weight.)
  uint4 k[2][4], v[4][2];
  const __half *kp, *vp;
  const bool aligned = (((uintptr_t)sq.sink_k | (uintptr_t)sq.sink_v | (uintptr_t)sq.win_k | (uintptr_t)sq.win_v | (uintptr_t)sq.dec_k | (uintptr_t)sq.dec_v) & 15) == 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    fp16_row(sq, sh, kv, min(u0 + g8 + 8 * r, last), kp, vp);
#pragma unroll
    for (int j = 0; j < 4; ++j) k[r][j] = row_load16<8>(kp + 32 * j + 8 * t4, aligned);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    fp16_row(sq, sh, kv, min(u0 + 8 * (r >> 1) + 2 * t4 + (r & 1), last), kp, vp);
#pragma unroll
    for (int i = 0; i < 2; ++i) v[r][i] = row_load16<8>(vp + 16 * g8 + 8 * i, aligned);
  }
  float dot[2][4];                                    // (summed pairwise, rounded to nearest: a chain of products truncates)
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 q = *reinterpret_cast<const uint4*>(qg_s + (g8 >> 1) * HD + 32 * j + 8 * t4);
    float s[2][4] = {};
    mma_16816(s[0], k[0][j].x, k[1][j].x, k[0][j].y, k[1][j].y, q.x, q.y);
    mma_16816(s[1], k[0][j].z, k[1][j].z, k[0][j].w, k[1][j].w, q.z, q.w);
#pragma unroll
    for (int r = 0; r < 2; ++r) dot[r][j] = s[0][2 * r] + s[1][2 * r];
  }
  float sc[2];
  const float vn[2] = {1.f, 1.f};
#pragma unroll
  for (int r = 0; r < 2; ++r) sc[r] = u0 + g8 + 8 * r <= last ? ((dot[r][0] + dot[r][1]) + (dot[r][2] + dot[r][3])) * (INV_SQRT_HD * LOG2E) : neg_inf();
  uint32_t w[2][2][2];
  block_weights(st, sc, vn, w, lane);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float o[2][4] = {};
#pragma unroll
    for (int part = 0; part < 2; ++part)
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const uint4 a = v[2 * m][i >> 1], b = v[2 * m + 1][i >> 1];
        if (i & 1) mma_16816(o[part], a.z, a.w, b.z, b.w, w[part][m][0], w[part][m][1]);
        else mma_16816(o[part], a.x, a.y, b.x, b.y, w[part][m][0], w[part][m][1]);
      }
#pragma unroll
    for (int c = 0; c < 4; ++c) st.o[i][c] += fmaf(o[1][c], PP_LO_DOWN, o[0][c]);
  }
}
// four codes -> the two fp16 parts of their codebook entries, part p of entries (0, 1) in x[p][0] and of (2, 3) in x[p][1]
__device__ __forceinline__ void split_values(uint32_t codes, uint32_t split, uint32_t (&x)[2][2]) {
  uint32_t e[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) e[j] = lds_u1(((j == 0 ? codes << 6 : codes >> (8 * j - 6)) & 0x3FC0u) | split);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    x[0][j] = __byte_perm(e[2 * j], e[2 * j + 1], 0x5410);
    x[1][j] = __byte_perm(e[2 * j], e[2 * j + 1], 0x7632);
  }
}
// streamed rows u0 .. u0 + 15; `unit`: what a score of query head lane % 4 counts, in the log2 domain; `split`: address of this lane's copy of
// the split codebook
__device__ __forceinline__ void stream_block(RowState& st, const ShardSeq& sq, const ShardDecodeShape& sh, int kv, int u0, const __half* qs_s,
                                             float unit, uint32_t split, int lane) {
  const int g8 = lane >> 2, t4 = lane & 3, last = sh.n_stream - 1;
  // keys: channels 32 t4 .. + 31 of rows g8 and g8 + 8; values: channels 16 g8 .. + 15 of rows 2 t4, 2 t4 + 1, and 8 further.  All loads
  // before the first use of one, and 16 bytes wide: with the norms converted where they were read, the block began with three round
  // trips to L2 instead of one, and 32 loads of 4 bytes, eight rows each, kept the L1 busy: 2.8 K of a block's 8 K cycles.
  uint4 k[2][2], v[4];
  unsigned short kn[2], vn[2];
  const bool aligned = (((uintptr_t)sq.st_k_idx | (uintptr_t)sq.st_v_idx) & 15) == 0;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const size_t row = (size_t)min(u0 + g8 + 8 * r, last) * sh.nkv + kv;
    kn[r] = __ldcg(reinterpret_cast<const unsigned short*>(sq.st_k_norm) + row);
    vn[r] = __ldcg(reinterpret_cast<const unsigned short*>(sq.st_v_norm) + row);
#pragma unroll
    for (int j = 0; j < 2; ++j) k[r][j] = row_load16<4>(sq.st_k_idx + row * HD + 32 * t4 + 16 * j, aligned);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const size_t row = (size_t)min(u0 + 8 * (r >> 1) + 2 * t4 + (r & 1), last) * sh.nkv + kv;
    v[r] = row_load16<4>(sq.st_v_idx + row * HD + 16 * g8, aligned);
  }
  auto word = [](const uint4& x, int i) { return i == 0 ? x.x : i == 1 ? x.y : i == 2 ? x.z : x.w; };
  // columns 2 h and 2 h + 1 are the two parts of query head h
  float lo[4] = {}, dot[2][4], cross[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint4 q = *reinterpret_cast<const uint4*>(qs_s + g8 * HD + 32 * t4 + 8 * j);
    float hi[2][4] = {};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t x0[2][2], x1[2][2];
      split_values(word(k[0][j >> 1], 2 * (j & 1) + h), split, x0);
      split_values(word(k[1][j >> 1], 2 * (j & 1) + h), split, x1);
      mma_16816(hi[h], x0[0][0], x1[0][0], x0[0][1], x1[0][1], h ? q.z : q.x, h ? q.w : q.y);
      mma_16816(lo, x0[1][0], x1[1][0], x0[1][1], x1[1][1], h ? q.z : q.x, h ? q.w : q.y);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) { dot[r][j] = hi[0][2 * r] + hi[1][2 * r]; cross[r] += hi[0][2 * r + 1] + hi[1][2 * r + 1]; }
  }
  float sc[2], nv[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    nv[r] = __half2float(__ushort_as_half(vn[r]));
    const float x = fmaf(fmaf(lo[2 * r + 1], PP_LO_DOWN, lo[2 * r] + cross[r]), PP_LO_DOWN, (dot[r][0] + dot[r][1]) + (dot[r][2] + dot[r][3]));
    sc[r] = u0 + g8 + 8 * r <= last ? x * (__half2float(__ushort_as_half(kn[r])) * unit) : neg_inf();
  }
  uint32_t w[2][2][2];
  block_weights(st, sc, nv, w, lane);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t x[2][2][2][2];                           // [m][row][part][pair of codes]
#pragma unroll
    for (int r = 0; r < 4; ++r) split_values(word(v[r], i), split, x[r >> 1][r & 1]);
    float cross[4] = {}, hi[4] = {};
    auto products = [&](float(&o)[4], int vp, int wp) {
#pragma unroll
      for (int m = 0; m < 2; ++m) mma_16816(o, x[m][0][vp][0], x[m][0][vp][1], x[m][1][vp][0], x[m][1][vp][1], w[wp][m][0], w[wp][m][1]);
    };
    products(cross, 0, 1);
    products(cross, 1, 0);
    products(hi, 0, 0);
#pragma unroll
    for (int c = 0; c < 4; ++c) st.o[i][c] += fmaf(cross[c], PP_LO_DOWN, hi[c]);
  }
}
// normalised 128-point Hadamard transform of every query head's sums (channel 16 (lane / 4) + 4 i + j in o[i][j])
__device__ __forceinline__ void row_sums_fwht(RowState& st, int lane) {
#pragma unroll
  for (int h = 1; h < 16; h <<= 1)
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (!(i & h)) {
        const float a = st.o[i >> 2][i & 3], b = st.o[(i | h) >> 2][(i | h) & 3];
        st.o[i >> 2][i & 3] = a + b;
        st.o[(i | h) >> 2][(i | h) & 3] = a - b;
      }
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) {
    const float sgn = (lane & off) ? -1.f : 1.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float& x = st.o[i >> 2][i & 3];
      x = fmaf(sgn, x, __shfl_xor_sync(0xffffffffu, x, off));
    }
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) st.o[i >> 2][i & 3] *= INV_SQRT_HD;
}
// the streamed sums out of the code space
__device__ __forceinline__ void stream_sums_back(RowState& st, const float* __restrict__ signs, int lane) {
  float4 sg[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) sg[i] = __ldg(reinterpret_cast<const float4*>(signs + 16 * (lane >> 2) + 4 * i));
  row_sums_fwht(st, lane);
#pragma unroll
  for (int i = 0; i < 4; ++i) { st.o[i][0] *= sg[i].x; st.o[i][1] *= sg[i].y; st.o[i][2] *= sg[i].z; st.o[i][3] *= sg[i].w; }
}
// into the rotated space, and out to the epilogue as a warp's state (acc[4][128], max[4], sum-exp[4]); `merge`: joined with the state
// that the warp has there from its tiles
__device__ __forceinline__ void row_state_store(RowState& st, float* out, bool merge, int lane) {
  const int g8 = lane >> 2, t4 = lane & 3;
  row_sums_fwht(st, lane);
  float l = st.l;
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
  float m = st.m, f0 = 0.f;
  if (merge) {
    __syncwarp();                                     // (the maxima and sums are other lanes' stores)
    const float m_mid = out[GQA * HD + t4], l_mid = out[GQA * HD + GQA + t4];
    m = fmaxf(m, m_mid);
    const float ref = m == neg_inf() ? 0.f : m;
    f0 = ex2(m_mid - ref);
    l = fmaf(l, ex2(st.m - ref), l_mid * f0);
  }
  const float f = st.m == neg_inf() ? 0.f : ex2(st.m - m) * pow2_whole(st.j - PP_W_LOG2);
  __syncwarp();
  if (g8 == 0) { out[GQA * HD + t4] = m; out[GQA * HD + GQA + t4] = l; }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float4* at = reinterpret_cast<float4*>(out + t4 * HD + 16 * g8 + 4 * i);
    float4 x = make_float4(st.o[i][0] * f, st.o[i][1] * f, st.o[i][2] * f, st.o[i][3] * f);
    if (merge) {
      const float4 mid = *at;
      x.x = fmaf(mid.x, f0, x.x); x.y = fmaf(mid.y, f0, x.y); x.z = fmaf(mid.z, f0, x.z); x.w = fmaf(mid.w, f0, x.w);
    }
    *at = x;
  }
}

// A launch without a middle segment (a cache that holds fp16 and streamed rows only): every CTA
// attends to its share of the rows (pair b belongs to CTA b % gridDim.x), the CTA
// that owns the newest streamed row quantises it first, the last CTA of a KV head combines.
constexpr int ROWS_THREADS = 512;
constexpr int ROWS_SMEM_BYTES = (2 * GQA * HD + 256 + (ROWS_THREADS / 32) * GQA * 130) * 4;
__global__ void __launch_bounds__(ROWS_THREADS, 1) decode_rows_only_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(128) unsigned char smem_rows[];
  const ShardSeq& sq = p.table ? p.table[blockIdx.z] : p.one;
  const ShardDecodeShape& sh = p.sh;
  const int kv = blockIdx.y, part = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool append_here = sh.append && p.n_row_parts > 0 && (row_pairs(sh) - 1) % p.n_row_parts == part;
  float* rec_rows = p.ws + (((size_t)blockIdx.z * p.n_parts + part) * sh.n_q + (size_t)kv * GQA) * PART;
  griddep_launch();
  griddep_wait();
  float* qn = reinterpret_cast<float*>(smem_rows);
  float* qr = qn + GQA * HD;
  float* cbs = qr + GQA * HD;
  float* scratch = cbs + 256;
  if (sh.n_stream > 0) for (int i = tid; i < 256; i += ROWS_THREADS) cbs[i] = p.codebook[i];
  if (tid < HD) stage_query(sq, kv, sh.pos_q, p.inv_freq, tid, qn, qr);
  __syncthreads();
  if (append_here) {
    if (warp < 2) append_new_token(sq, sh, kv, cbs, warp == 1, lane);
    __syncthreads();
  }
  SoftmaxState st;
  softmax_init(st);
  process_rows(st, sq, sh, kv, part + p.n_row_parts * warp, p.n_row_parts * (ROWS_THREADS / 32), qr, cbs, lane);
  partial_store<ROWS_THREADS / 32>(st, scratch, warp, lane);
  __syncthreads();
  if (warp < GQA) partial_merge<ROWS_THREADS / 32>(scratch, rec_rows, warp, lane);
  ticket_combine<ROWS_THREADS, 4>(p, sq, kv, blockIdx.z, scratch, tid);
}

template <int NW>  // rank / 32
__global__ void __launch_bounds__(PP_THREADS, 1) decode_partial_pipe_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int R = NW * 32;
  constexpr int KSTEPS = R / 16 + 1;   // + one step whose A columns are (1, 0, ...) and whose W slice is the mean
  constexpr int W_BYTES = pp_w_bytes(NW);
  constexpr int W_ATOMS = W_BYTES / 16384;
  constexpr int A_COLS = pp_a_cols(NW);

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t raw_u = smem_u32(smem_raw);
  const uint32_t cb_u = (raw_u + PP_HEAD_BYTES + PP_CB_ALIGN - 1) & ~(uint32_t)(PP_CB_ALIGN - 1);
  if (cb_u != PP_CB_ALIGN) {                                       // (the host has refused such a launch already: pp_layout_fits)
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1);
    return;
  }
  unsigned char* cbv = smem_raw + (cb_u - raw_u);                  // V codebook, 16 copies
  uint4* split_s = reinterpret_cast<uint4*>(cbv + PP_CB_ALIGN);    // split stream codebook
  unsigned char* w_s = cbv + PP_CB_ALIGN + PP_SPLIT_BYTES;                      // weights (1 KB aligned)
  unsigned char* c_s = w_s + W_BYTES;                              // coefficient tiles
  float* state_s = reinterpret_cast<float*>(c_s + PP_C_BUFS * pp_c_bytes(NW));   // states: consumer warps, unpack warps
  __half* qg_s = reinterpret_cast<__half*>(smem_raw + PP_OFF_QG);
  __half* qs_s = reinterpret_cast<__half*>(smem_raw + PP_OFF_QS);
  float* cbs_s = reinterpret_cast<float*>(smem_raw + PP_OFF_CBS);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + PP_OFF_MISC);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_raw + PP_OFF_MISC + 960);
  volatile int* abort_s = reinterpret_cast<volatile int*>(smem_raw + PP_OFF_MISC + 964);

  const ShardSeq& sq = p.table ? p.table[blockIdx.z] : p.one;
  const ShardDecodeShape& sh = p.sh;
  const int kv = blockIdx.y;
  const int part = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* rec_base = p.ws + (((size_t)blockIdx.z * p.n_parts + part) * sh.n_q + (size_t)kv * GQA) * PART;

  // The rows outside the middle go in blocks of 16 of a kind, the streamed ones' first; block b is CTA b % n_row_parts's.  They
  // are the unpack warps' while those have about a block to every two tiles; beyond that all warps but the issuing and copying ones
  // take a share when their tiles are done.
  const int blocks_s = (sh.n_stream + 15) >> 4, n_fp16 = sh.n_sink + sh.n_win + sh.n_dec, blocks = blocks_s + ((n_fp16 + 15) >> 4);
  // the CTA that owns the newest row writes it before anybody reads it
  const bool append_here = sh.append && p.n_row_parts > 0 && ((sh.append == 1 ? blocks_s : blocks) - 1) % p.n_row_parts == part;
  const bool wide_rows = p.n_row_parts > 0 && blocks > 4 * p.n_row_parts * max(1, (p.tiles_per_chunk + 1) >> 1);
  const int n_row_warps = wide_rows ? PP_ROW_WARPS : 4;

  griddep_launch();

  const uint32_t bar0 = smem_u32(bars);
  auto KN_FULL = [&](int s) { return bar0 + 8u * (uint32_t)s; };           // MMA1 of pipeline s done: keys in its stage, its A slot free
  auto KN_EMPTY = [&](int s) { return bar0 + 8u * (uint32_t)(2 + s); };    // the group's four warps have read the stage
  auto A_FULL = [&](int s) { return bar0 + 8u * (uint32_t)(4 + s); };      // the A operand is in its slot
  auto MMA_DONE = [&](int s) { return bar0 + 8u * (uint32_t)(6 + s); };    // an issuing thread's work has completed (after giving up)
  auto W_FULL = [&](int a) { return bar0 + 8u * (uint32_t)(8 + a); };      // atom a (64 contraction positions) of the weights has landed
  auto C_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(12 + b); };     // coefficient tile has landed
  auto C_EMPTY = [&](int b) { return bar0 + 8u * (uint32_t)(16 + b); };    // the unpack warps have read it
  auto V_FULL = [&](int b) { return bar0 + 8u * (uint32_t)(20 + b); };     // V code tile has landed
  auto V_EMPTY = [&](int b) { return bar0 + 8u * (uint32_t)(28 + b); };    // its group has read it
  const uint32_t CB_READY = bar0 + 8u * 36u;                               // the codebooks are in shared memory (whoever looks codes up waits for it)
  const uint32_t Q_READY = bar0 + 8u * 37u;                                // the query fragments, the queries as given and the channel scales are staged
  const uint32_t QS_READY = bar0 + 8u * 39u;                               // the queries in code space are there
  const uint32_t APPEND_DONE = bar0 + 8u * 38u;                            // the newest streamed row has been written

  // tiles of this chunk: evenly spread, the first `tiles_rem` chunks get one more
  const int tile_lo = part * p.tiles_per_chunk + min(part, p.tiles_rem);
  const int n_my = p.tiles_per_chunk + (part < p.tiles_rem ? 1 : 0);
  const int tok_lo = sh.tok_begin + tile_lo * 128;
  // Bulk copy of the packed coefficient rows of tile `it` into its buffer.  The last tile of the segment may be
  // short; the rows behind it keep whatever the buffer held (any byte pattern decodes to finite values, and
  // those rows get zero weight).
  auto issue_coef = [&](int it) {
    const int t0 = tok_lo + it * 128, b = it % PP_C_BUFS;
    const uint32_t bytes = (uint32_t)min(128, sh.tok_end - t0) * (uint32_t)(R / 2);
    mbar_expect_tx(C_FULL(b), bytes);
    bulk_g2s(smem_u32(c_s + b * pp_c_bytes(NW)), sq.k_coeffs + (size_t)t0 * (R / 2), bytes, C_FULL(b));
  };

  auto issue_vcodes = [&](int it) {
    const int t0 = tok_lo + it * 128, b = it % PP_V_BUFS;
    const uint32_t bytes = (uint32_t)min(128, sh.tok_end - t0) * (uint32_t)VQ_GROUPS;
    mbar_expect_tx(V_FULL(b), bytes);
    bulk_g2s(smem_u32(smem_raw + PP_OFF_V) + (uint32_t)b * 4096u, sq.v_indices + ((size_t)kv * sh.n_comp + t0) * VQ_GROUPS, bytes, V_FULL(b));
  };

  // ---- one-time set-up ----------------------------------------------------------------------------
  if (warp == PP_UNPACK_WARP0) {
    tmem_alloc(smem_u32(tmem_slot), PP_TMEM_COLS);
    tmem_relinquish();
  }
  if (tid == PP_COEF_WARP * 32) {
    // first the barriers of the bulk copies, so that the copy engine starts as early as possible
    for (int b = 0; b < PP_C_BUFS; ++b) { mbar_init(C_FULL(b), 1); mbar_init(C_EMPTY(b), 4); }
    for (int a = 0; a < W_ATOMS; ++a) mbar_init(W_FULL(a), 1);
    fence_mbar_init();
    if (n_my > 0) issue_coef(0);
    for (int a = 0; a < W_ATOMS && n_my > 0; ++a) {        // (a CTA for rows alone needs no weights)
      mbar_expect_tx(W_FULL(a), 16384u);
      bulk_g2s(smem_u32(w_s + a * 16384), reinterpret_cast<const unsigned char*>(sq.k_wprep) + (size_t)kv * W_BYTES + a * 16384,
               16384u, W_FULL(a));
    }
    for (int it = 1; it < min(PP_C_BUFS, n_my); ++it) issue_coef(it);
  } else if (tid == PP_VCODE_WARP * 32) {
    for (int b = 0; b < PP_V_BUFS; ++b) { mbar_init(V_FULL(b), 1); mbar_init(V_EMPTY(b), 4); }
    fence_mbar_init();
    for (int it = 0; it < min(PP_V_BUFS, n_my); ++it) issue_vcodes(it);
  } else if (tid == PP_MMA_WARP * 32) {
    for (int s = 0; s < PP_ST; ++s) { mbar_init(KN_FULL(s), 1); mbar_init(KN_EMPTY(s), 4); mbar_init(A_FULL(s), 4); mbar_init(MMA_DONE(s), 1); }
    mbar_init(CB_READY, PP_CONS_WARPS);
    mbar_init(Q_READY, 2);
    mbar_init(APPEND_DONE, 2);
    mbar_init(QS_READY, 4);
    *abort_s = 0;
    fence_mbar_init();
  }
  const int quad = warp & 3, grp = warp >> 2;
  const int n_use = warp < PP_CONS_WARPS && n_my > grp ? (n_my - grp + PP_ST - 1) / PP_ST : 0;   // tiles of this warp's group
  // (one CTA barrier for what everybody needs: tensor memory, the mbarriers, the copies in flight)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  int asked = min(warp == PP_COEF_WARP ? PP_C_BUFS : PP_V_BUFS, n_my);   // tiles a copying thread has asked for

  if (warp < PP_CONS_WARPS) {
    // =============================== consumer groups ======================================
    const int g8 = lane >> 2, t4 = lane & 3;          // the lane's row and column pair in a matrix fragment
    // the codebooks into shared memory, by the consumer warps alone: the others are already at work
    {
      const uint2 e = reinterpret_cast<const uint2*>(sq.v_centroids)[tid & 255];
      if (tid < 256) {
#pragma unroll
        for (int c = 0; c < PP_CB_COPIES / 2; ++c)
          *reinterpret_cast<uint4*>(cbv + tid * (8 * PP_CB_COPIES) + (((c + lane) & (PP_CB_COPIES / 2 - 1)) << 4)) = make_uint4(e.x, e.y, e.x, e.y);
      }
      if (sh.n_stream > 0 && tid < 256) {
        const float c = p.codebook[tid];
        cbs_s[tid] = c;
        const uint32_t sp = split_half2(c);
#pragma unroll
        for (int j = 0; j < PP_SPLIT_COPIES / 4; ++j) split_s[PP_SPLIT_COPIES / 4 * tid + ((j + (lane >> 1)) & (PP_SPLIT_COPIES / 4 - 1))] = make_uint4(sp, sp, sp, sp);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(CB_READY);
    }
    // cos / sin of the rows, laid out as the fragments want them (phase_table_kernel); step i of a tile takes pairs
    // 16 (i / 2) .. + 15 of rows 16 (i % 2) .. + 15; loaded four steps ahead (131K x 4 layers: 355 us; two ahead 393, three 378, six 375)
    const uint4* phase_tab = reinterpret_cast<const uint4*>(sq.phase) + lane;
    const int last_blk = (sh.tok_end - sh.tok_begin - 1) >> 5;
    auto phase_of = [&](int it) { return phase_tab + (size_t)min((tile_lo + it) * 4 + quad, last_blk) * 512; };
    uint4 ph[8][2];
    const uint4* prow = phase_of(min(grp, max(n_my - 1, 0)));
    auto load_phase = [&](int i, const uint4* pr) {
      ph[i][0] = pr[((2 * (i & 1)) * 4 + (i >> 1)) * 32];
      ph[i][1] = pr[((2 * (i & 1) + 1) * 4 + (i >> 1)) * 32];
    };
    const uint32_t kn = tmem_base + (uint32_t)(128 * grp) + ((uint32_t)(32 * quad) << 16);       // the warp's rows of its key stage
    auto load_keys = [&](int i, uint32_t* r) {        // columns of step i: 16 of the first half of the channels, the same 16 of the second
      const uint32_t at = kn + ((uint32_t)(16 * (i & 1)) << 16) + 16 * (i >> 1);
      tmem_ld_frag(at, r);
      tmem_ld_frag(at + 64, r + 8);
    };
    // keys of step i, half k, rotated by the relative phase: an A fragment of the scores product
    auto rotate = [&](const uint32_t* r, int i, int k, uint32_t (&a)[4]) {
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {                // rows g8, g8 + 8
        const __half2 c2 = __floats2half2_rn(__uint_as_float(r[4 * k + 2 * rr]), __uint_as_float(r[4 * k + 2 * rr + 1]));
        const __half2 d2 = __floats2half2_rn(__uint_as_float(r[8 + 4 * k + 2 * rr]), __uint_as_float(r[8 + 4 * k + 2 * rr + 1]));
        const __half2 cs = as_half2(k ? ph[i][rr].z : ph[i][rr].x), sn = as_half2(k ? ph[i][rr].w : ph[i][rr].y);
        a[rr] = as_u32(__hfma2(c2, cs, __hneg2(__hmul2(d2, sn))));           // c cos - d sin
        a[2 + rr] = as_u32(__hfma2(d2, cs, __hmul2(c2, sn)));                // d cos + c sin
      }
    };
    // the group's first tile: its keys are rotated here and wait in registers for the query
    uint32_t first[8][2][4];
    if (n_use > 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) load_phase(i, prow);
      const uint4* pnext = phase_of(min(grp + PP_ST, n_my - 1));
      ok = __all_sync(0xffffffffu, mbar_wait_soon(KN_FULL(grp), 0u, abort_s));
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t r[16];
        load_keys(i, r);
        tmem_wait_frags(r);
        rotate(r, i, 0, first[i][0]);
        rotate(r, i, 1, first[i][1]);
        load_phase((i + 4) & 7, i < 4 ? prow : pnext);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(KN_EMPTY(grp));
      prow = pnext;
    }
    // Up to here only tensors that no decode call ever writes were touched (weights, coefficients, V codes,
    // codebooks) and the phase table, complete before any CTA of this launch starts: the kernel that writes it never
    // releases its dependents early.  All this, the first tiles' unpack and reconstruction products among it, runs
    // while the launch before this one is still finishing.  The query, the new token, the stream rows, the scratch
    // and the output may come from, or still be in use by, that launch: every role waits before it touches them.
    // (The copying warps stage the query: these may still be at their first tile when the launch before has finished.)
    griddep_wait();
    ok = __all_sync(0xffffffffu, ok && mbar_wait(CB_READY, 0u, abort_s) && mbar_wait(Q_READY, 0u, abort_s));
    const uint2* qf_s = reinterpret_cast<const uint2*>(smem_raw + PP_OFF_QF) + (g8 >> 1) * 4 + t4;
    const uint32_t v_u = smem_u32(smem_raw + PP_OFF_V);
    const uint32_t cb_lane = cb_u + (uint32_t)(lane & (PP_CB_COPIES - 1)) * 8u;
    const uint32_t sel0 = (g8 & 1) ? 0x1044u : 0x4410u, sel1 = (g8 & 1) ? 0x3244u : 0x4432u;
    float run_m = neg_inf(), run_l = 0.f;             // of query head t4; log2 domain
    float o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] = 0.f;

    float sc[2][2][4];                                // scores: two sums of each, so that one product does not wait for the last
    auto clear_scores = [&]() {
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int j = 0; j < 4; ++j) sc[b >> 1][b & 1][j] = 0.f;
    };
    clear_scores();
    if (n_use > 0 && ok) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint2 qf = qf_s[16 * (2 * (i >> 1) + k)];
          mma_16816(sc[i & 1][k], first[i][k][0], first[i][k][1], first[i][k][2], first[i][k][3], qf.x, qf.y);
        }
    }
#pragma unroll 1
    for (int use = 0; use < n_use && ok; ) {
      const int it = grp + use * PP_ST;
      // ---- V codes of the tile: row 8 m + 2 t4 (+ 1), codes 4 g8 .. + 3 ----------------------------------------
      const int vb = it % PP_V_BUFS;
      ok = __all_sync(0xffffffffu, mbar_wait_soon(V_FULL(vb), (uint32_t)((it / PP_V_BUFS) & 1), abort_s));
      if (!ok) break;
      uint32_t vc[4][2];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t at = v_u + (uint32_t)vb * 4096u + (uint32_t)((32 * quad + 8 * m + 2 * t4) * VQ_GROUPS + 4 * g8);
        vc[m][0] = lds_u1(at);
        vc[m][1] = lds_u1(at + VQ_GROUPS);
      }
      // ---- softmax: this lane has rows g8 + 8 m of query head t4 (columns 2 t4 and 2 t4 + 1 are the same head) ------
      const int left = sh.tok_end - (tok_lo + it * 128 + 32 * quad + g8);
      float pr[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) pr[m] = 8 * m < left ? (sc[m >> 1][0][2 * (m & 1)] + sc[m >> 1][1][2 * (m & 1)]) * (INV_SQRT_HD * LOG2E) : neg_inf();
      const float top = fmaxf(fmaxf(pr[0], pr[1]), fmaxf(pr[2], pr[3]));
      if (__any_sync(0xffffffffu, top > run_m + PP_LAZY_LOG2)) {
        // The reference point of a (warp, head) only moves when the tile's maximum exceeds it by more than
        // 2^PP_LAZY_LOG2 (weights then stay below that factor, far inside fp16 range).
        float tm = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
        tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 8));
        tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 16));
        if (tm > run_m + PP_LAZY_LOG2) {
          const float al = ex2(run_m - tm);           // (0 at the first valid token)
          run_m = tm;
          run_l *= al;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) o[i][j] *= al;
        }
      }
      const float ref = run_m == neg_inf() ? 0.f : run_m;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        pr[m] = ex2(pr[m] - ref);
        run_l += pr[m];
      }
      // ---- P.V: contraction over (token, parity of the channel), so that a codebook entry is a fragment as it is:
      // O[pair of channels][(head, parity)] += V[pair][(token, parity')] . (P[token][head] if the parities agree) ---------
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t x = transpose_8x8(pack_half2(pr[m], pr[m]));          // weights of rows 8 m + 2 t4, + 1 for head g8 / 2
        const uint32_t b0 = __byte_perm(x, 0u, sel0), b1 = __byte_perm(x, 0u, sel1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const uint2 e0 = lds_u2((((i == 0 ? vc[m][0] << 7 : vc[m][0] >> (8 * i - 7))) & 0x7F80u) | cb_lane);
          const uint2 e1 = lds_u2((((i == 0 ? vc[m][1] << 7 : vc[m][1] >> (8 * i - 7))) & 0x7F80u) | cb_lane);
          mma_16816(o[i], e0.x, e0.y, e1.x, e1.y, b0, b1);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(V_EMPTY(vb));
      if (++use == n_use) break;
      // ---- keys of the next tile: rotated straight into the A fragments of its scores product -------------------
      const uint4* pnext = phase_of(min(it + 2 * PP_ST, n_my - 1));
      ok = __all_sync(0xffffffffu, mbar_wait_soon(KN_FULL(grp), (uint32_t)(use & 1), abort_s));
      if (!ok) break;
      tc_fence_after();
      clear_scores();
      uint2 qf[2];
      uint32_t kr[2][16];
      load_keys(0, kr[0]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint32_t* r = kr[i & 1];
        tmem_wait_frags(r);
        if (i < 7) {
          load_keys(i + 1, kr[(i + 1) & 1]);
        } else {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(KN_EMPTY(grp));
        }
        load_phase((i + 4) & 7, i < 4 ? prow : pnext);
        if ((i & 1) == 0) { qf[0] = qf_s[16 * i]; qf[1] = qf_s[16 * i + 16]; }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          uint32_t a[4];
          rotate(r, i, k, a);
          mma_16816(sc[i & 1][k], a[0], a[1], a[2], a[3], qf[k].x, qf[k].y);
        }
      }
      prow = pnext;
    }
    // the warp's state: this lane has channels 16 g8 .. + 15 of query head t4, in units of the channels' scales
    {
      float* st = state_s + warp * PP_STATE;
      float l = run_l + __shfl_xor_sync(0xffffffffu, run_l, 4);
      l += __shfl_xor_sync(0xffffffffu, l, 8);
      l += __shfl_xor_sync(0xffffffffu, l, 16);
      if (g8 == 0) { st[GQA * HD + t4] = run_m; st[GQA * HD + GQA + t4] = l; }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint2 cw = *reinterpret_cast<const uint2*>(smem_raw + PP_OFF_CH + 2 * (16 * g8 + 4 * i));
        const float2 ca = __half22float2(as_half2(cw.x)), cb = __half22float2(as_half2(cw.y));
        *reinterpret_cast<float4*>(st + t4 * HD + 16 * g8 + 4 * i) = make_float4(o[i][0] * ca.x, o[i][1] * ca.y, o[i][2] * cb.x, o[i][3] * cb.y);
      }
    }
  } else if (warp < PP_MMA_WARP) {
    // =============================== unpack warps =========================================
    const int m = quad * 32 + lane;
    const uint32_t lane_A = tmem_base + PP_COL_A + ((uint32_t)(quad * 32) << 16);
#pragma unroll
    for (int s = 0; s < PP_ST; ++s) {
      // constant part of the A operand: position R is 1.0 (it multiplies the mean slice of W)
      const uint32_t ones[8] = {0x00003C00u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
      tmem_st_x8(lane_A + s * A_COLS + R / 2, ones);
    }
#pragma unroll 1
    for (int it = 0; it < n_my; ++it) {
      const int cb = it % PP_C_BUFS, s = it % PP_ST;
      ok = __all_sync(0xffffffffu, mbar_wait_soon(C_FULL(cb), (uint32_t)((it / PP_C_BUFS) & 1), abort_s));
      if (!ok) break;                                     // uniform over the warp
      const uint4* row = reinterpret_cast<const uint4*>(c_s + cb * pp_c_bytes(NW) + m * (R / 2));
      uint4 x[NW];
#pragma unroll
      for (int i = 0; i < NW; ++i) x[i] = row[i];
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        uint32_t ov[16];
        const uint32_t wv[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t hi = wv[e] >> 8;
          ov[4 * e + 0] = nib2half2_tc(wv[e]);            // ranks 8c+0, 8c+4 of word c = 4i+e
          ov[4 * e + 1] = nib2half2_hi(wv[e]);            //       8c+1, 8c+5
          ov[4 * e + 2] = nib2half2_tc(hi);               //       8c+2, 8c+6
          ov[4 * e + 3] = nib2half2_hi(hi);               //       8c+3, 8c+7
        }
        // the slot is free once the MMA1 two tiles back has completed
        if (i == 0 && it >= PP_ST) {
          ok = __all_sync(0xffffffffu, mbar_wait_soon(KN_FULL(s), (uint32_t)((it / PP_ST - 1) & 1), abort_s));
          if (!ok) break;
          tc_fence_after();
        }
        tmem_st_x16(lane_A + s * A_COLS + 16 * i, ov);
      }
      if (!ok) break;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(A_FULL(s)); mbar_arrive(C_EMPTY(cb)); }
    }
    griddep_wait();
  } else if (warp < PP_COEF_WARP) {
    // =============================== issuing warp =========================================
    // One thread each: MMA1 of every second tile, K_n[128 tok x 128] = A . W^T into the pipeline's key stage.  Two of them, because
    // the tensor core would stand still during the waits of one (a hand-over takes a few hundred cycles).
    if (lane == 0) {
      constexpr uint32_t IDESC1 = umma_idesc(128, 128, false, false);
      const uint64_t wdesc = smem_desc_sw128(smem_u32(w_s), 16, 1024);
      const int s = warp - PP_MMA_WARP;
      const uint32_t T_t = tmem_base + (uint32_t)(128 * s), A_t = tmem_base + PP_COL_A + (uint32_t)(s * A_COLS);
#pragma unroll 1
      for (int it = s; it < n_my && ok; it += PP_ST) {
        ok = mbar_wait_soon(A_FULL(s), (uint32_t)((it / PP_ST) & 1), abort_s);
        if (ok && it >= PP_ST) ok = mbar_wait_soon(KN_EMPTY(s), (uint32_t)((it / PP_ST - 1) & 1), abort_s);
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          if ((ks & 3) == 0) {
            if (it == s) ok = ok && mbar_wait(W_FULL(ks >> 2), 0u, abort_s);    // only a thread's first MMA1 can be ahead of the weights
            if (!ok) break;
            if (ks == 0 || it == s) tc_fence_after();
          }
          umma_ts_1t(T_t, A_t + 8 * ks, wdesc + (uint64_t)(((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), IDESC1, ks > 0 ? 1u : 0u);
        }
        if (ok) umma_commit_1t(KN_FULL(s));
      }
    }
    __syncwarp();
    griddep_wait();
  } else {
    // =============================== copying warps ========================================
    // First the query, and in the CTA that owns the newest streamed row the new token, quantised into it (bit-identical to
    // stream_quantize_kernel); the copies asked for so far last meanwhile.
    {
      // un-rotated queries (fp16 arithmetic as the reference): thread = pair i of all heads
      const int i = (warp - PP_COEF_WARP) * 32 + lane;
      float sn, cs;
      sincosf(__fmul_rn((float)sh.pos_q, p.inv_freq[i]), &sn, &cs);
      const __half c16 = __float2half_rn(cs), s16 = __float2half_rn(sn);
      const __half* qg = reinterpret_cast<const __half*>(sq.q) + (size_t)kv * GQA * HD;
      __half x_lo[GQA], x_hi[GQA];
      griddep_wait();
#pragma unroll
      for (int h = 0; h < GQA; ++h) { x_lo[h] = qg[h * HD + i]; x_hi[h] = qg[h * HD + i + 64]; }
      // (the channel scales with the query: the kernel in front may be the one that writes them, and they cost no trip of their own here)
      const uint32_t scales = reinterpret_cast<const uint32_t*>(reinterpret_cast<const __half*>(sq.v_ch) + kv * HD)[i];
#pragma unroll
      for (int h = 0; h < GQA; ++h) {
        __half* f = reinterpret_cast<__half*>(smem_raw + PP_OFF_QF) + ((i >> 3) * 16 + 4 * h + ((i & 7) >> 1)) * 4 + (i & 1);
        f[0] = __hsub(__hmul(x_lo[h], c16), __hmul(__hneg(x_hi[h]), s16));
        f[2] = __hsub(__hmul(x_hi[h], c16), __hmul(x_lo[h], s16));
        qg_s[h * HD + i] = x_lo[h];
        qg_s[h * HD + i + 64] = x_hi[h];
      }
      *reinterpret_cast<uint32_t*>(smem_raw + PP_OFF_CH + 4 * i) = scales;
      __syncwarp();
      if (lane == 0) mbar_arrive(Q_READY);
    }
    if (append_here) {
      ok = __all_sync(0xffffffffu, mbar_wait(CB_READY, 0u, abort_s));
      if (ok) append_new_token(sq, sh, kv, cbs_s, warp == PP_VCODE_WARP, lane);
      __syncwarp();
      if (lane == 0) mbar_arrive(APPEND_DONE);
    }
    if (lane == 0 && warp == PP_COEF_WARP) {
      for (int it = PP_C_BUFS; it < n_my && ok; ++it) {
        ok = mbar_wait(C_EMPTY(it % PP_C_BUFS), (uint32_t)((it / PP_C_BUFS - 1) & 1), abort_s);
        if (ok) { issue_coef(it); asked = it + 1; }
      }
    } else if (lane == 0) {
      for (int it = PP_V_BUFS; it < n_my && ok; ++it) {
        ok = mbar_wait(V_EMPTY(it % PP_V_BUFS), (uint32_t)((it / PP_V_BUFS - 1) & 1), abort_s);
        if (ok) { issue_vcodes(it); asked = it + 1; }
      }
    }
    __syncwarp();
  }

  // ---- rows: this warp's share of the blocks, taken to the rotated space of the middle's accumulator.  (Some rows behind every tile
  // instead of all behind the last: the unpack is on the tile loop's critical path, slower.) --------------------------------------
  if (wide_rows ? warp < PP_MMA_WARP : warp >= PP_UNPACK_WARP0 && warp < PP_MMA_WARP) {
    const int row_w = warp >= PP_UNPACK_WARP0 ? warp - PP_UNPACK_WARP0 : warp + 4;        // unpack warps first
    RowState st;
    row_state_init(st);
    if (ok && p.n_row_parts > 0) {
      float4 sg = make_float4(0.f, 0.f, 0.f, 0.f);
      if (blocks_s > 0 && row_w < 4) sg = *reinterpret_cast<const float4*>(sq.signs + 4 * lane);
      ok = __all_sync(0xffffffffu, mbar_wait(Q_READY, 0u, abort_s));
      if (ok && blocks_s > 0) {
        // the unpack warps take a query head each to the code space; the others wait for them
        if (row_w < 4) {
          const float inv = stream_query(sg, qg_s + row_w * HD, qs_s + row_w * 2 * HD, lane);
          if (lane == 0) reinterpret_cast<float*>(smem_raw + PP_OFF_QUP)[row_w] = inv;
          __syncwarp();
          if (lane == 0) mbar_arrive(QS_READY);
        }
        // (the split codebook too: the consumer warps write it behind the CTA's only barrier, and in a CTA of a few tiles, or none,
        // nothing else here comes after that)
        ok = __all_sync(0xffffffffu, mbar_wait(QS_READY, 0u, abort_s) && mbar_wait(CB_READY, 0u, abort_s));
      }
      if (ok && append_here) ok = __all_sync(0xffffffffu, mbar_wait(APPEND_DONE, 0u, abort_s));
      if (ok) {
        int b = part + p.n_row_parts * row_w;
        const int step = p.n_row_parts * n_row_warps;
        if (b < blocks_s) {
          const float unit = reinterpret_cast<const float*>(smem_raw + PP_OFF_QUP)[lane & 3] * (INV_SQRT_HD * LOG2E);
#pragma unroll 1
          for (; b < blocks_s; b += step) stream_block(st, sq, sh, kv, 16 * b, qs_s, unit, cb_u + PP_CB_ALIGN + 4u * (uint32_t)(lane & (PP_SPLIT_COPIES - 1)), lane);
          stream_sums_back(st, sq.signs, lane);
        }
#pragma unroll 1
        for (; b < blocks; b += step) fp16_block(st, sq, sh, kv, 16 * (b - blocks_s), qg_s, lane);
      }
    }
    row_state_store(st, state_s + warp * PP_STATE, warp < PP_CONS_WARPS, lane);
  }

  // ---- epilogue: merge the warps' states per head and emit the record -----------------------------------
  tc_fence_before();
  __syncthreads();
  if (__builtin_expect(*abort_s, 0)) {
    // gave up somewhere, whichever role it was (nobody changes the flag any more): nobody leaves, and tensor memory is not freed, while the
    // tensor core may still be at work in it or a bulk copy may still be landing in this CTA's memory
    if (tid == 0 && p.status) atomicExch(p.status, 1);
    if (warp >= PP_MMA_WARP && warp < PP_COEF_WARP && lane == 0) {
      umma_commit_1t(MMA_DONE(warp - PP_MMA_WARP));
      mbar_wait(MMA_DONE(warp - PP_MMA_WARP), 0u, abort_s);
    } else if (tid == PP_COEF_WARP * 32) {
      for (int a = 0; a < W_ATOMS && n_my > 0; ++a) mbar_wait(W_FULL(a), 0u, abort_s);
      for (int c = max(0, asked - PP_C_BUFS); c < asked; ++c) mbar_wait(C_FULL(c % PP_C_BUFS), (uint32_t)((c / PP_C_BUFS) & 1), abort_s);
    } else if (tid == PP_VCODE_WARP * 32) {
      for (int c = max(0, asked - PP_V_BUFS); c < asked; ++c) mbar_wait(V_FULL(c % PP_V_BUFS), (uint32_t)((c / PP_V_BUFS) & 1), abort_s);
    }
    __syncthreads();
  }
  if (warp == PP_UNPACK_WARP0) tmem_dealloc(tmem_base, PP_TMEM_COLS);
  if (warp < PP_MMA_WARP) {
    // Warp = (query head, one of three), lane = four channels; maxima are in the log2 domain, the record carries the natural
    // logarithm's.  Each merges every third state, the head's first warp the three sums.
    const int hq = warp & 3, sub = warp >> 2;
    float M = neg_inf(), L = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
    auto add = [&](float m, float l, const float4& x) {
      const float top = fmaxf(M, m), ref = top == neg_inf() ? 0.f : top, w0 = ex2(M - ref), w1 = ex2(m - ref);
      M = top;
      L = fmaf(w1, l, L * w0);
      a[0] = fmaf(w1, x.x, a[0] * w0); a[1] = fmaf(w1, x.y, a[1] * w0); a[2] = fmaf(w1, x.z, a[2] * w0); a[3] = fmaf(w1, x.w, a[3] * w0);
    };
#pragma unroll
    for (int e = sub; e < PP_ROW_WARPS; e += PP_SUB) {
      const float* st = state_s + e * PP_STATE;
      add(st[GQA * HD + hq], st[GQA * HD + GQA + hq], *reinterpret_cast<const float4*>(st + hq * HD + 4 * lane));
    }
    float* meet = reinterpret_cast<float*>(c_s) + hq * (PP_SUB * PP_MEET);        // (the coefficients have all been read)
    if (sub > 0) {
      *reinterpret_cast<float4*>(meet + sub * PP_MEET + 4 * lane) = make_float4(a[0], a[1], a[2], a[3]);
      if (lane == 0) { meet[sub * PP_MEET + HD] = M; meet[sub * PP_MEET + HD + 1] = L; }
    }
    asm volatile("bar.sync %0, %1;" ::"r"(8 + hq), "n"(PP_SUB * 32) : "memory");
    if (sub == 0) {
#pragma unroll
      for (int e = 1; e < PP_SUB; ++e) add(meet[e * PP_MEET + HD], meet[e * PP_MEET + HD + 1], *reinterpret_cast<const float4*>(meet + e * PP_MEET + 4 * lane));
      float* rec = rec_base + hq * PART;
      if (lane == 0) *reinterpret_cast<float4*>(rec) = make_float4(M * LN2, L, 0.f, 0.f);
      *reinterpret_cast<float4*>(rec + 4 + 4 * lane) = make_float4(a[0], a[1], a[2], a[3]);
    }
    if (p.push.world == 0) {
      head_combine<PP_SUB>(p, sq, kv, blockIdx.z, hq, sub, lane, meet);
      return;
    }
  }
  if (p.push.world > 0) ticket_combine<PP_THREADS, PP_SUB>(p, sq, kv, blockIdx.z, reinterpret_cast<float*>(state_s), tid);
}

// Prepared weights: per KV head, W = basis * coefficient scale as fp16 in the K-major, 128-byte
// swizzled operand layout (atoms of 64 contraction positions x 128 rows).  Position kk = 8c + p
// holds rank 8c + perm[p] (the order in which the unpack step emits the nibbles of word c);
// position R holds the mean, positions R+1 .. R+15 are zero.
__global__ void __launch_bounds__(256) decode_prepare_pipe_kernel(const __half* __restrict__ basis,
                                                                  const __half* __restrict__ cscale,
                                                                  const __half* __restrict__ mean, int nkv, int rank,
                                                                  unsigned char* __restrict__ out) {
  const int kpos = rank + 16;
  const int w_bytes = ((kpos + 63) / 64) * 16384;
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= nkv * HD * kpos) return;
  const int kk = idx % kpos;
  const int j = (idx / kpos) % HD;
  const int kv = idx / (kpos * HD);
  const int c = kk >> 3, pp = kk & 7;
  __half v = __float2half(0.f);
  if (kk < rank) {
    const int perm = ((pp & 1) << 2) | (pp >> 1);                // 0,4,1,5,2,6,3,7
    const int r = 8 * c + perm;
    v = __hmul(basis[(size_t)(kv * HD + j) * rank + r], cscale[r]);
  } else if (kk == rank) {
    v = mean[kv * HD + j];
  }
  *reinterpret_cast<__half*>(out + (size_t)kv * w_bytes + (c >> 3) * 16384 + (j >> 3) * 1024 + (j & 7) * 128 +
                             (((c & 7) ^ (j & 7)) << 4) + pp * 2) = v;
}

size_t pipe_wprep_bytes(int nkv, int rank) { return (size_t)nkv * (((rank + 16 + 63) / 64) * 16384); }

int launch_prepare_pipe(const void* basis, const void* cscale, const void* mean, int nkv, int rank, void* out,
                        cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(out, 0, pipe_wprep_bytes(nkv, rank), st);   // unused tail of the last atom
  if (e != cudaSuccess) return (int)e;
  const int total = nkv * HD * (rank + 16);
  decode_prepare_pipe_kernel<<<(total + 255) / 256, 256, 0, st>>>((const __half*)basis, (const __half*)cscale,
                                                                   (const __half*)mean, nkv, rank, (unsigned char*)out);
  return 0;
}

template <int NW>
static int launch_pipe_one(const DecodeParams& p, dim3 grid, cudaStream_t st) {
  constexpr int SMEM = pp_smem_bytes(NW);
  // the opt-in to more than 48 KB of dynamic shared memory is a per-device attribute of the kernel
  static std::atomic<bool> configured[MAX_DEVICES];
  int dev = -1;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess) return (int)de;
  if (dev < 0 || dev >= MAX_DEVICES) return SHARD_E_ARG;
  if (!configured[dev].load(std::memory_order_acquire)) {
    cudaFuncAttributes attrs;
    int reserved = 0;
    cudaError_t e = cudaFuncGetAttributes(&attrs, decode_partial_pipe_kernel<NW>);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    if (e != cudaSuccess) return (int)e;
    if (!pp_layout_fits((size_t)reserved, attrs.sharedSizeBytes)) return (int)cudaErrorInvalidConfiguration;
    e = cudaFuncSetAttribute(decode_partial_pipe_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev].store(true, std::memory_order_release);
  }
  // Programmatic dependent launch: this launch's CTAs may move onto SMs and run their set-up
  // (barriers, first bulk copies of tensors that no decode call writes) while the kernel in front
  // of it in the stream is still finishing; griddep_wait in the kernel keeps the order of
  // everything else.  Off for a call with shape.no_overlap, or for all calls with
  // SHARD_B200_PDL=0 in the environment.
  static int use_pdl_env = -1;
  if (use_pdl_env < 0) {
    const char* e = getenv("SHARD_B200_PDL");
    use_pdl_env = (e && e[0] == '0') ? 0 : 1;
  }
  const int use_pdl = use_pdl_env && !p.sh.no_overlap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(PP_THREADS);
  cfg.dynamicSmemBytes = SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = use_pdl ? 1 : 0;
  cudaError_t e = cudaLaunchKernelEx(&cfg, decode_partial_pipe_kernel<NW>, p);
  return e == cudaSuccess ? 0 : (int)e;
}

static int launch_rows_only(const DecodeParams& p, dim3 grid, cudaStream_t st) {
  // (38 KB of dynamic shared memory: no opt-in needed)
  static_assert(ROWS_SMEM_BYTES <= 48 * 1024, "fits the default dynamic shared memory");
  decode_rows_only_kernel<<<grid, ROWS_THREADS, ROWS_SMEM_BYTES, st>>>(p);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

int launch_partial_pipe(const DecodeParams& p, dim3 grid, cudaStream_t st) {
  if (p.n_chunks == 0) return launch_rows_only(p, grid, st);
  switch (p.sh.rank / 32) {
    case 1: return launch_pipe_one<1>(p, grid, st);
    case 2: return launch_pipe_one<2>(p, grid, st);
    case 3: return launch_pipe_one<3>(p, grid, st);
    case 4: return launch_pipe_one<4>(p, grid, st);
    case 5: return launch_pipe_one<5>(p, grid, st);
    default: return launch_pipe_one<6>(p, grid, st);
  }
}

}  // namespace shard
