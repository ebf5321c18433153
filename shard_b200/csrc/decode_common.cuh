// Pieces shared by the decode kernels: launch parameters, per-CTA query staging, the rows of launches
// without a middle segment, and the merges into one (max, sum-exp, acc[128]) record per query head.
#pragma once

#include "common.cuh"
#include "peer_layout.cuh"

namespace shard {

constexpr int ROWS_PER_CTA = 32;        // rows per CTA when a launch has no middle segment
constexpr int MAX_ROW_CTAS = 18;
constexpr int HEAD_PARTS = 8;           // records of a query head that one warp loads at a time
constexpr int MAX_PARTS = 160;          // records of a (sequence, KV head) that the fused combine merges

// Sequence-split decode: where the launch's result goes when it is delivered straight into the
// exchange buffers of all ranks (layout in peer_layout.cuh).  world == 0: no delivery.
struct PeerPush {
  unsigned char* bufs[PEER_MAX_WORLD];
  int rank, world;
  unsigned int epoch;
  void* merged_out;              // fp16 [n_q][128]: if set, the delivering CTA also waits for all ranks' records and merges
  int* status;                   // set to 1 when that wait gives up (may be null)
  unsigned long long wait_ns;    // its bound
};

struct DecodeParams {
  ShardSeq one;
  const ShardSeq* table;
  ShardDecodeShape sh;
  const float* inv_freq;
  const float* codebook;
  float* ws;
  int* status;          // device word set non-zero when a bounded wait gave up
  int* tickets;         // [batch][nkv] arrival counters of the fused combine (zero between calls)
  int n_chunks;         // CTAs (per KV head) that walk the compressed middle (0: there is no middle)
  int tiles_per_chunk;
  int tiles_rem;        // the first tiles_rem chunks walk one tile more
  int n_row_parts;      // CTAs (per KV head) that share the fp16 / streamed rows: the chunk CTAs
                        // themselves when there is a middle, else CTAs of their own; 0: no rows
  int n_parts;          // records per (sequence, query head): n_chunks in rotated space, or without a middle n_row_parts in standard space
  int n_ctas;           // CTAs per (sequence, KV head) = gridDim.x
  PeerPush push;        // sequence-split: deliver the combined record to every rank's exchange buffer
};

// add that releases what this thread's warp has written and acquires what the others had written before theirs (lighter than
// sequentially consistent fences around a plain one)
__device__ __forceinline__ unsigned int atomic_add_acq_rel(unsigned int* at, unsigned int v) {
  unsigned int old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(at), "r"(v) : "memory");
  return old;
}

struct SoftmaxState {
  float m[GQA];
  float l[GQA];       // lane-local partial sums (see call sites)
  float acc[GQA][4];  // lane owns channels 4*lane .. 4*lane+3
};

__device__ __forceinline__ void softmax_init(SoftmaxState& st) {
#pragma unroll
  for (int h = 0; h < GQA; ++h) {
    st.m[h] = neg_inf();
    st.l[h] = 0.f;
#pragma unroll
    for (int c = 0; c < 4; ++c) st.acc[h][c] = 0.f;
  }
}

// Un-rotated query (fp16 arithmetic, as the reference does it) and the query as given,
// for the 4 heads of KV group `kv`; thread d < 128 handles channel d.
__device__ __forceinline__ void stage_query(const ShardSeq& sq, int kv, int pos_q, const float* __restrict__ inv_freq,
                                            int d, float* __restrict__ qn, float* __restrict__ qr) {
  const int i = d & 63;
  const float phase = __fmul_rn((float)pos_q, inv_freq[i]);
  float sn, cs;
  sincosf(phase, &sn, &cs);
  const __half c16 = __float2half_rn(cs), s16 = __float2half_rn(sn);
  const __half* qg = reinterpret_cast<const __half*>(sq.q) + (size_t)kv * GQA * HD;
#pragma unroll
  for (int h = 0; h < GQA; ++h) {
    const __half x = qg[h * HD + d];
    const __half other = qg[h * HD + (d ^ 64)];
    const __half rot = (d < 64) ? __hneg(other) : other;
    const __half un = __hsub(__hmul(x, c16), __hmul(rot, s16));
    qn[h * HD + d] = __half2float(un);
    qr[h * HD + d] = __half2float(x);
  }
}

// Fused append: the CTA that owns the newest row first puts the step's new K/V vector of its KV head
// into it (one warp each for K and V): quantised into streamed row n_stream-1 (append = 1), or copied
// into row n_dec-1 of the fp16 decode buffer (append = 2).  The caller synchronises the CTA afterwards;
// the rows are then read back with L2-coherent loads.
__device__ __forceinline__ void append_new_token(const ShardSeq& sq, const ShardDecodeShape& sh, int kv,
                                                 const float* __restrict__ cbs, bool is_v, int lane) {
  const __half* src = reinterpret_cast<const __half*>(is_v ? sq.new_v : sq.new_k) + kv * HD;
  if (sh.append == 2) {
    __half* dst = reinterpret_cast<__half*>(const_cast<void*>(is_v ? sq.dec_v : sq.dec_k)) +
                  ((size_t)kv * (sh.dec_cap > 0 ? sh.dec_cap : sh.n_dec) + sh.n_dec - 1) * HD;
    reinterpret_cast<uint2*>(dst)[lane] = reinterpret_cast<const uint2*>(src)[lane];
    return;
  }
  const size_t row = (size_t)(sh.n_stream - 1) * sh.nkv + kv;
  uint8_t* idx_out = (is_v ? sq.st_v_idx : sq.st_k_idx) + row * HD;
  __half* norm_out = reinterpret_cast<__half*>(is_v ? sq.st_v_norm : sq.st_k_norm) + row;
  quantize_vec_warp(src, sq.signs, cbs, idx_out, norm_out, lane);
}

// Rows of a launch without a middle segment (with one: decode_pipe.cu's blocks of sixteen), in one index space: u < n_sink + n_win + n_dec is an fp16 row
// (sink rows first, then window, then the fp16 decode buffer), the rest are streamed rows.  They are dealt
// out in pairs of a kind, the fp16 rows' pairs first: a warp takes pairs b_first, b_first + b_step, ....
// Lane owns channels 4*lane..+3 of both rows; the eight dot products (row, head) are summed over the lanes by
// halving (9 shuffles, which leave product lane / 4 in the lane), so a lane weighs one (row, head) alone,
// and the weights go round by shuffle.
//
// A streamed row is never rotated back: its key is norm / sqrt(128) . signs o H(codebook[code]), so the
// QUERY is taken to the code space (H(signs o q) / sqrt(128)) and the score is
// norm . (query . codebook[code]); streamed values are summed in code space (weight . norm .
// codebook[code]) and the SUM is rotated back, once per warp.  Streamed rows come first, so that one set of
// accumulators serves both kinds.
//
// Bound: a warp's chain of dependent instructions and loads, so the code is kept short, and small in registers.  A
// streamed row with two butterflies and four full reductions of its own took 3 K cycles, a pair here about 1 K.
// `qr` is the query as given (fp32 copy in shared memory), `cbs` the stream codebook in shared memory
// (needed for streamed rows only).
__device__ __forceinline__ void fp16_row(const ShardSeq& sq, const ShardDecodeShape& sh, int kv, int u, const __half*& k, const __half*& v) {
  const int n_sw = sh.n_sink + sh.n_win;
  const bool in_sink = u < sh.n_sink, in_dec = u >= n_sw;
  const int r = in_sink ? u : (in_dec ? u - n_sw : u - sh.n_sink);
  const int rows = in_sink ? sh.n_sink : (in_dec ? (sh.dec_cap > 0 ? sh.dec_cap : sh.n_dec) : sh.n_win);
  const size_t off = ((size_t)kv * rows + r) * HD;
  k = reinterpret_cast<const __half*>(in_sink ? sq.sink_k : (in_dec ? sq.dec_k : sq.win_k)) + off;
  v = reinterpret_cast<const __half*>(in_sink ? sq.sink_v : (in_dec ? sq.dec_v : sq.win_v)) + off;
}
// pairs of fp16 rows, and of all rows (the newest row is in the last)
__host__ __device__ inline int row_pairs_fp16(const ShardDecodeShape& sh) { return (sh.n_sink + sh.n_win + sh.n_dec + 1) >> 1; }
__host__ __device__ inline int row_pairs(const ShardDecodeShape& sh) { return row_pairs_fp16(sh) + ((sh.n_stream + 1) >> 1); }

__device__ __forceinline__ float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// st.m in the log2 domain
__device__ __forceinline__ void process_rows(SoftmaxState& st, const ShardSeq& sq, const ShardDecodeShape& sh,
                                             int kv, int b_first, int b_step,
                                             const float* __restrict__ qr, const float* __restrict__ cbs, int lane) {
  const int fp_pairs = row_pairs_fp16(sh), pairs = row_pairs(sh);
  if (b_first >= pairs) return;
  const int own = lane >> 4;                             // the (row of a pair, head lane / 4 % 4) this lane weighs
  float m_own = neg_inf(), l_own = 0.f;                  // of that head; log2 domain
  uint2 kr[2], vr[2];                                    // the next pair: four codes (x), or four fp16 values
  unsigned short kn16 = 0, vn16 = 0;                     // norms of row `own`
  // (L2-coherent loads: the newest row may have been written by this CTA a moment ago; a row behind the
  // last repeats it and gets no weight)
  auto load = [&](int b) {
    if (b >= fp_pairs) {
      const int u = 2 * (b - fp_pairs), more = u + 1 < sh.n_stream ? 1 : 0;
      const size_t row = (size_t)u * sh.nkv + kv, at = row * HD + 4 * lane, next = (size_t)(more * sh.nkv) * HD;
      kr[0].x = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_k_idx + at));
      kr[1].x = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_k_idx + at + next));
      vr[0].x = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_v_idx + at));
      vr[1].x = __ldcg(reinterpret_cast<const unsigned int*>(sq.st_v_idx + at + next));
      kn16 = __ldcg(reinterpret_cast<const unsigned short*>(sq.st_k_norm) + row + own * more * sh.nkv);
      vn16 = __ldcg(reinterpret_cast<const unsigned short*>(sq.st_v_norm) + row + own * more * sh.nkv);
    } else {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const __half *k, *v;
        fp16_row(sq, sh, kv, min(2 * b + r, sh.n_sink + sh.n_win + sh.n_dec - 1), k, v);
        kr[r] = __ldcg(reinterpret_cast<const uint2*>(k) + lane);
        vr[r] = __ldcg(reinterpret_cast<const uint2*>(v) + lane);
      }
    }
  };
  int b = b_first;
  if (b < fp_pairs) b += (fp_pairs - b_first + b_step - 1) / b_step * b_step;
  bool stream = b < pairs;
  if (!stream) b = b_first;
  load(b);
  float4 q[GQA];
#pragma unroll
  for (int h = 0; h < GQA; ++h) q[h] = *reinterpret_cast<const float4*>(qr + h * HD + 4 * lane);
  if (stream) {
    const float4 sg = *reinterpret_cast<const float4*>(sq.signs + 4 * lane);
#pragma unroll
    for (int h = 0; h < GQA; ++h) {
      float x[4] = {q[h].x * sg.x, q[h].y * sg.y, q[h].z * sg.z, q[h].w * sg.w};
      fwht128_lane4(x, lane);
      q[h] = make_float4(x[0] * INV_SQRT_HD, x[1] * INV_SQRT_HD, x[2] * INV_SQRT_HD, x[3] * INV_SQRT_HD);
    }
  }
  auto values = [&](uint2 raw, float (&x)[4]) {
    if (stream) {
      x[0] = cbs[raw.x & 0xff]; x[1] = cbs[(raw.x >> 8) & 0xff]; x[2] = cbs[(raw.x >> 16) & 0xff]; x[3] = cbs[raw.x >> 24];
    } else {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), c = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
      x[0] = a.x; x[1] = a.y; x[2] = c.x; x[3] = c.y;
    }
  };
#pragma unroll 1
  while (true) {
    // ---- scores --------------------------------------------------------------------------------------
    float s[8], x0[4], x1[4];
    values(kr[0], x0);
    values(kr[1], x1);
#pragma unroll
    for (int h = 0; h < GQA; ++h) {
      s[h] = fmaf(q[h].x, x0[0], fmaf(q[h].y, x0[1], fmaf(q[h].z, x0[2], q[h].w * x0[3])));
      s[4 + h] = fmaf(q[h].x, x1[0], fmaf(q[h].y, x1[1], fmaf(q[h].z, x1[2], q[h].w * x1[3])));
    }
    values(vr[0], x0);                                   // (the value rows' look-ups overlap the reduction)
    values(vr[1], x1);
    const float kn = stream ? __half2float(__ushort_as_half(kn16)) : 1.f, vn = stream ? __half2float(__ushort_as_half(vn16)) : 1.f;
    const bool live = stream ? 2 * (b - fp_pairs) + own < sh.n_stream : 2 * b + own < sh.n_sink + sh.n_win + sh.n_dec;
    b += b_step;
    const bool more = b < (stream ? pairs : fp_pairs), turn = !more && stream && b_first < fp_pairs;
    if (turn) b = b_first;
    if (more || turn) load(b);                           // the next pair on its way
#pragma unroll
    for (int half = 4, off = 16; half >= 1; half >>= 1, off >>= 1) {
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float keep = up ? s[i + half] : s[i], give = up ? s[i] : s[i + half];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
      }
    }
    float sc = s[0] + __shfl_xor_sync(0xffffffffu, s[0], 2);
    sc += __shfl_xor_sync(0xffffffffu, sc, 1);           // product lane / 4 = (own, head)
    sc = live ? sc * kn * (INV_SQRT_HD * LOG2E) : neg_inf();
    const float mn = fmaxf(m_own, fmaxf(sc, __shfl_xor_sync(0xffffffffu, sc, 16)));   // (at least one row is live)
    const float al = ex2(m_own - mn), pr = ex2(sc - mn), pv = pr * vn;
    m_own = mn;
    l_own = fmaf(l_own, al, pr);
    // ---- values ---------------------------------------------------------------------------------------
#pragma unroll
    for (int h = 0; h < GQA; ++h) {
      const float a = __shfl_sync(0xffffffffu, al, 4 * h), p0 = __shfl_sync(0xffffffffu, pv, 4 * h), p1 = __shfl_sync(0xffffffffu, pv, 16 + 4 * h);
#pragma unroll
      for (int c = 0; c < 4; ++c) st.acc[h][c] = fmaf(p1, x1[c], fmaf(p0, x0[c], st.acc[h][c] * a));
    }
    if (more) continue;
    if (!stream) break;
    // ---- the streamed sums back from the code space, the fp16 rows next ---------------------------------
    const float4 sg = *reinterpret_cast<const float4*>(sq.signs + 4 * lane);
#pragma unroll
    for (int h = 0; h < GQA; ++h) {
      fwht128_lane4(st.acc[h], lane);
      st.acc[h][0] *= sg.x * INV_SQRT_HD; st.acc[h][1] *= sg.y * INV_SQRT_HD;
      st.acc[h][2] *= sg.z * INV_SQRT_HD; st.acc[h][3] *= sg.w * INV_SQRT_HD;
    }
    if (!turn) break;
#pragma unroll
    for (int h = 0; h < GQA; ++h) q[h] = *reinterpret_cast<const float4*>(qr + h * HD + 4 * lane);
    stream = false;
  }
  // state per head, the same in every lane: lanes 4 h + 16 r hold head h's sums of row r
  l_own += __shfl_xor_sync(0xffffffffu, l_own, 16);
#pragma unroll
  for (int h = 0; h < GQA; ++h) {
    st.m[h] = __shfl_sync(0xffffffffu, m_own, 4 * h);
    st.l[h] = __shfl_sync(0xffffffffu, l_own, 4 * h);
  }
}

// Merge of per-warp softmax states (lane owns channels 4*lane..+3, m/l are warp-uniform, m in the log2
// domain) into one
// record per head, in two steps with a barrier of the caller's choice in between:
// partial_store by every one of the NWARPS warps (index `w`), then partial_merge by four warps.  `scratch` needs NWARPS*4*130 floats.
template <int NWARPS>
__device__ __forceinline__ void partial_store(const SoftmaxState& st, float* __restrict__ scratch, int w, int lane) {
  float* mw = scratch;
  float* lw = mw + NWARPS * GQA;
  float* aw = lw + NWARPS * GQA;
  if (lane == 0) {
#pragma unroll
    for (int h = 0; h < GQA; ++h) { mw[w * GQA + h] = st.m[h]; lw[w * GQA + h] = st.l[h]; }
  }
#pragma unroll
  for (int h = 0; h < GQA; ++h)
    *reinterpret_cast<float4*>(aw + (w * GQA + h) * HD + 4 * lane) =
        make_float4(st.acc[h][0], st.acc[h][1], st.acc[h][2], st.acc[h][3]);
}

// Warp `h` < 4 merges query head h.
template <int NWARPS>
__device__ __forceinline__ void partial_merge(const float* scratch, float* __restrict__ rec_base, int h, int lane) {
  const float* mw = scratch;
  const float* lw = mw + NWARPS * GQA;
  const float* aw = lw + NWARPS * GQA;
  float M = neg_inf();
#pragma unroll
  for (int w = 0; w < NWARPS; ++w) M = fmaxf(M, mw[w * GQA + h]);
  float L = 0.f, a[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int w = 0; w < NWARPS; ++w) {
    const float mwv = mw[w * GQA + h];
    const float wt = (mwv == neg_inf()) ? 0.f : ex2(mwv - M);
    const float4 v = *reinterpret_cast<const float4*>(aw + (w * GQA + h) * HD + 4 * lane);
    L = fmaf(wt, lw[w * GQA + h], L);
    a[0] = fmaf(wt, v.x, a[0]); a[1] = fmaf(wt, v.y, a[1]); a[2] = fmaf(wt, v.z, a[2]); a[3] = fmaf(wt, v.w, a[3]);
  }
  float* rec = rec_base + h * PART;
  if (lane == 0) *reinterpret_cast<float4*>(rec) = make_float4(M * LN2, L, 0.f, 0.f);    // (the record carries the natural-log maximum)
  *reinterpret_cast<float4*>(rec + 4 + 4 * lane) = make_float4(a[0], a[1], a[2], a[3]);
}

// Merge of all records of a query head, by the NSUB warps (w = 0 .. NSUB - 1) that a CTA gives it.  Few records: warp 0 merges
// them; more: each warp takes every NSUB-th and the sums meet in `sm_head` (NSUB * 128 floats, the head's own, 16-byte aligned).
// True in the warp that has the result: maximum, sum-exp (the same in every lane) and channels 4 lane .. + 3, back from the rotated
// space.  The order of the sums depends on the number of parts alone, not on which CTA merges.  The merging CTA is the
// critical path of its launch and runs this code once, out of a cold instruction cache: it is kept short, and all loads of KB
// parts are in flight together.  Lane j also fetches (max, sum-exp) of parts j, j + 32, ..., from which the warp derives the weights and
// hands them round by shuffle.
template <int NSUB>
__device__ __forceinline__ bool head_merge(const DecodeParams& p, int b, int h, int hq, int w, int lane, float* sm_head, float& M, float& L, float (&o4)[4]) {
  constexpr int KB = HEAD_PARTS;
  const int n_parts = p.n_parts, n_q = p.sh.n_q;
  const bool split = n_parts > KB;
  if (w > 0 && !split) return false;
  const float* rec0 = p.ws + ((size_t)b * n_parts * n_q + h) * PART;
  const size_t pstride = (size_t)n_q * PART;
  const int step = split ? NSUB : 1;
  float4 a[KB];
  auto load = [&](int p0) {
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      const int pi = p0 + w + step * k;
      a[k] = pi < n_parts ? __ldcg(reinterpret_cast<const float4*>(rec0 + pi * pstride + 4) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  load(0);
  float mj[MAX_PARTS / 32], lj[MAX_PARTS / 32];
  M = neg_inf(); L = 0.f;
#pragma unroll
  for (int k = 0; k < MAX_PARTS / 32; ++k) {
    const int pj = lane + 32 * k;
    mj[k] = neg_inf();
    lj[k] = 0.f;
    if (pj < n_parts) {
      const float2 ml = __ldcg(reinterpret_cast<const float2*>(rec0 + pj * pstride));
      mj[k] = ml.x;
      lj[k] = ml.y;
    }
    M = fmaxf(M, mj[k]);
  }
  M = warp_max(M);
  const float Ms = M == neg_inf() ? 0.f : M;             // (nothing attended to: all weights 0)
#pragma unroll
  for (int k = 0; k < MAX_PARTS / 32; ++k) {
    mj[k] = ex2((mj[k] - Ms) * LOG2E);                   // now the weights; 0 behind the last part
    L = fmaf(mj[k], lj[k], L);
  }
  L = warp_sum(L);
#pragma unroll
  for (int c = 0; c < 4; ++c) o4[c] = 0.f;
#pragma unroll 1
  for (int p0 = 0; p0 < n_parts; p0 += KB * step) {
    if (p0 > 0) load(p0);
#pragma unroll
    for (int k = 0; k < KB; ++k) {
      const int pi = p0 + w + step * k;
      float wj = mj[0];
      if (split) {
#pragma unroll
        for (int j = 1; j < MAX_PARTS / 32; ++j) wj = (pi >> 5) == j ? mj[j] : wj;
      }
      const float wt = __shfl_sync(0xffffffffu, wj, pi & 31);
      o4[0] = fmaf(wt, a[k].x, o4[0]); o4[1] = fmaf(wt, a[k].y, o4[1]);
      o4[2] = fmaf(wt, a[k].z, o4[2]); o4[3] = fmaf(wt, a[k].w, o4[3]);
    }
  }
  if (split) {
    float4* sums = reinterpret_cast<float4*>(sm_head) + lane;
    if (w > 0) sums[w * 32] = make_float4(o4[0], o4[1], o4[2], o4[3]);
    asm volatile("bar.sync %0, %1;" ::"r"(8 + hq), "r"(NSUB * 32) : "memory");
    if (w > 0) return false;
#pragma unroll
    for (int j = 1; j < NSUB; ++j) {
      const float4 r = sums[j * 32];
      o4[0] += r.x; o4[1] += r.y; o4[2] += r.z; o4[3] += r.w;
    }
  }
  // (the records of a launch are all of a kind: in rotated space, or, without a middle segment, standard)
  if (p.n_chunks > 0) {
    // inverse (= forward) normalised Hadamard over the 128 channels
    fwht128_lane4(o4, lane);
#pragma unroll
    for (int c = 0; c < 4; ++c) o4[c] = o4[c] * INV_SQRT_HD;
  }
  return true;
}

// the launch's output for one query head, by the warp that has its merged record
__device__ __forceinline__ void head_output(const DecodeParams& p, const ShardSeq& sq, int h, int lane, float M, float L, const float (&o4)[4]) {
  if (p.sh.partial_out) {
    float4* rec = reinterpret_cast<float4*>(reinterpret_cast<float*>(sq.out) + (size_t)h * PART);
    if (lane == 0) rec[0] = make_float4(M, L, 0.f, 0.f);
    rec[1 + lane] = make_float4(o4[0], o4[1], o4[2], o4[3]);
  } else {
    // o / L as the other merges round it, the reciprocal shared by the four: with inv and q = o . inv rounded to nearest, q + (o - q L) inv
    // is the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34, 1990); a q that is exact, or infinite, stays
    // (8K x 12 layers: four divisions 162.8 us, this 162.0)
    const float inv = 1.f / L;
    float x[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float q = o4[c] * inv, r = fmaf(-q, L, o4[c]);
      x[c] = fabsf(r) > 0.f ? fmaf(r, inv, q) : q;
    }
    const __half2 lo = __floats2half2_rn(x[0], x[1]), hi = __floats2half2_rn(x[2], x[3]);
    uint2 pk;
    pk.x = *reinterpret_cast<const uint32_t*>(&lo);
    pk.y = *reinterpret_cast<const uint32_t*>(&hi);
    reinterpret_cast<uint2*>(reinterpret_cast<__half*>(sq.out) + (size_t)h * HD)[lane] = pk;
  }
}

// Fused combine, head by head.  The warp that has written a query head's record (w = 0 of the head's NSUB) takes a ticket for it; the
// warp that draws the last one sees all records of that head and merges them.  No CTA barrier: heads finish on their own.
// The four heads' counts share the KV head's word, a byte each (at most MAX_PARTS = 160 arrivals); each is back at zero for the
// next call.
template <int NSUB>
__device__ __forceinline__ void head_combine(const DecodeParams& p, const ShardSeq& sq, int kv, int b, int hq, int w, int lane, float* sm_head) {
  __shared__ int last_of[GQA];
  int last = 0;
  if (w == 0) {
    __syncwarp();
    if (lane == 0) {
      unsigned int* ctr = reinterpret_cast<unsigned int*>(p.tickets) + b * p.sh.nkv + kv;
      last = ((atomic_add_acq_rel(ctr, 1u << (8 * hq)) >> (8 * hq)) & 255u) == (unsigned int)(p.n_ctas - 1);
      if (last) atomicSub(ctr, (unsigned int)p.n_ctas << (8 * hq));   // (nobody looks at it before the next launch)
      last_of[hq] = last;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();                                        // (the records that lane 0 has acquired are read by all)
  }
  if (p.n_parts > HEAD_PARTS) {                          // (the head's other warps are needed)
    asm volatile("bar.sync %0, %1;" ::"r"(8 + hq), "r"(NSUB * 32) : "memory");
    last = last_of[hq];
  }
  if (!last) return;
  float M, L, o4[4];
  if (head_merge<NSUB>(p, b, kv * GQA + hq, hq, w, lane, sm_head, M, L, o4)) head_output(p, sq, kv * GQA + hq, lane, M, L, o4);
}

// Fused combine, all four heads by the CTA that draws the KV head's last ticket: for launches that deliver to the exchange buffers, where
// one flag stands for the KV head, and for launches without a middle segment.  Every CTA of one (sequence, KV head) calls this after
// its record is written.  (The ticket's thread releases the CTA's writes, which the barrier has ordered before it, and
// acquires the others'.)  Warp h + 4 w is the w-th of query head h's NSUB.
template <int NTHREADS, int NSUB>
__device__ __forceinline__ void ticket_combine(const DecodeParams& p, const ShardSeq& sq, int kv, int b, float* sm_raw, int tid) {
  static_assert(NTHREADS >= NSUB * GQA * 32, "the merging warps");
  __shared__ int last_s;
  __syncthreads();
  if (tid == 0) {
    int* ctr = p.tickets + b * p.sh.nkv + kv;
    __threadfence();
    const int last = atomicAdd(ctr, 1) == p.n_ctas - 1;
    if (last) {
      __threadfence();
      *reinterpret_cast<volatile int*>(ctr) = 0;         // (nobody looks at it before the next launch)
    }
    last_s = last;
  }
  __syncthreads();
  if (!last_s) return;
  const int n_q = p.sh.n_q, lane = tid & 31, w = tid >> 5;
  const int h = kv * GQA + (w & 3);                      // query head of the warp
  float M, L, o4[4];
  const bool fin = w < NSUB * GQA && head_merge<NSUB>(p, b, h, w & 3, w >> 2, lane, sm_raw + (w & 3) * (NSUB * HD), M, L, o4);
  if (p.push.world > 0) {
    // Sequence-split decode: this CTA holds the rank's final record of four query heads.  It goes
    // straight into slot epoch % 2 of EVERY rank's exchange buffer (plain peer stores over
    // NVLink), then -- after a system-scope fence by every storing thread -- the epoch number is
    // published in every rank's flag word for (this rank, this KV head).  The merge kernel of
    // each rank waits for those flags.
    const int slot = (int)(p.push.epoch & 1u);
    const size_t flag_bytes = peer_flag_bytes(p.push.world, p.sh.nkv);
    const size_t slot_floats = peer_slot_floats(p.push.world, p.sh.nkv);
    if (fin) {
      for (int r = 0; r < p.push.world; ++r) {
        float4* rec = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.push.bufs[r] + flag_bytes) + slot * slot_floats +
                                                ((size_t)p.push.rank * n_q + h) * PART);
        if (lane == 0) rec[0] = make_float4(M, L, 0.f, 0.f);
        rec[1 + lane] = make_float4(o4[0], o4[1], o4[2], o4[3]);
      }
    }
    __threadfence_system();
    __syncthreads();
    if (tid < p.push.world) {
      volatile unsigned int* flag = reinterpret_cast<volatile unsigned int*>(p.push.bufs[tid]) +
                                    ((size_t)slot * p.push.world + p.push.rank) * p.sh.nkv + kv;
      *flag = p.push.epoch;
    }
    if (p.push.merged_out) {
      // ... and finishes the step itself: wait -- bounded by the global timer -- for every rank's
      // records of this KV head in the own buffer, merge them in rank order, write the attention
      // output.  (Eight CTAs of the launch do this, one per KV head, while the others have retired.)
      if (tid == 0) last_s = 0;                        // reused as "gave up"
      __syncthreads();
      if (tid < p.push.world) {
        volatile unsigned int* flag = reinterpret_cast<volatile unsigned int*>(p.push.bufs[p.push.rank]) +
                                      ((size_t)slot * p.push.world + tid) * p.sh.nkv + kv;
        if (!wait_epoch(flag, p.push.epoch, p.push.wait_ns)) last_s = 1;
        __threadfence_system();
      }
      __syncthreads();
      if (last_s) {
        if (tid == 0 && p.push.status) atomicExch(p.push.status, 1);
      } else {
        for (int i = tid; i < GQA * HD; i += NTHREADS) {
          const int hq = kv * GQA + (i >> 7), d = i & (HD - 1);
          reinterpret_cast<__half*>(p.push.merged_out)[(size_t)hq * HD + d] =
              merge_rank_records(p.push.bufs[p.push.rank], p.push.world, p.sh.nkv, slot, hq, d);
        }
      }
    }
    if (!sq.out) return;
  }
  if (fin) head_output(p, sq, h, lane, M, L, o4);
}

}  // namespace shard
