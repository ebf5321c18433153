// Leading eigenpairs of small symmetric matrices (the p x p Gram matrices of the PCA fit, p = 128 ..
// 1024), several matrices side by side.
//
//   1. tridiag_kernel      Householder reduction to tridiagonal form, one cluster of 16 CTAs per matrix.
//                          The whole matrix stays on chip: row r lives in CTA r % 16, in TENSOR MEMORY
//                          (64 rows x 1024 columns of fp32 are exactly its 256 KB), which its warps
//                          read and write as a register file: thread = 8 matrix columns, for which the
//                          three vectors of a step stay in registers.  One exchange per step: every CTA
//                          sends its rows of A v and of the next column to all others with st.async
//                          (distributed shared memory, completion counted on the receivers' mbarriers);
//                          everything else of a step is recomputed by every CTA from the same numbers.
//   2. tridiag_values_kernel   eigenvalues by 129-section on Sturm counts, a CTA per eigenvalue, fp64;
//                          division-free recurrence (one multiply-add of latency per row).
//   3. tridiag_vectors_kernel  eigenvectors of the tridiagonal matrix by twisted factorisation, fp64,
//                          thread = vector, one warp from either end.
//   4. eig_products_kernel, eig_back_kernel    the reflectors applied to the vectors, eight per pass to the four vectors of a CTA.
//   5. eig_check_kernel    neighbouring vectors must be orthogonal; a matrix with eigenvalues too close
//                          for step 3 is reported to the caller.
//
// Bound: the latency chain of step 1 (p steps of exchange, two reductions and one pass over the matrix).
// p = 1024, rank 192, one matrix / four side by side: step 1 2.1 ms (4.5 ms before its column phases and packed multiply-adds),
// step 2 0.11 / 0.26 ms, step 3 0.08 ms (0.26 ms before its loads went ahead of its stores), step 4 0.19 / 0.27 ms (0.33 / 0.35),
// step 5 0.02 ms; torch.linalg.eigh takes 8 to 12 ms a matrix.
#include <atomic>
#include <type_traits>

#include "tcgen05.cuh"

namespace shard {

constexpr int EG_CL = 16;                  // CTAs of a cluster
constexpr int EG_THREADS = 256;
constexpr int EG_MAX_P = 1024;

struct EighParams {
  const float* a;         // [L][p][p]
  int p, rank;
  float* refl;            // [L][p][p] reflector k in row k (zeros up to k, one at k + 1; the last row is zero)
  float* tau;             // [L][p]
  float* d;               // [L][p]
  float* e;               // [L][p]
  double* lam;            // [L][rank] eigenvalues, descending
  double* dplus;          // [L][blocks of 32 vectors][p][32]
  double* dminus;
  float* z;               // [L][blocks][p][32] vectors of the tridiagonal matrix
  float* products;        // [L][p / 8][8][8] of the reflectors of a group
  float* basis;           // [L][p][rank]
  float* eigvals;         // [L][rank]
  int* flag;              // [L] 1: vectors not orthogonal, or a wait gave up
};

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(cta));
  return r;
}
__device__ __forceinline__ void st_async_f4(uint32_t addr, float a, float b, float c, float d, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async_f1(uint32_t addr, float a, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];"
               ::"r"(addr), "f"(a), "r"(bar) : "memory");
}

// A row's columns of this thread, tensor memory <-> registers.
template <int W, int O = 0, int M>
__device__ __forceinline__ void eg_ld(uint32_t t, uint32_t (&u)[M]) {
  if constexpr (W - O >= 8)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[O]), "=r"(u[O + 1]), "=r"(u[O + 2]), "=r"(u[O + 3]), "=r"(u[O + 4]), "=r"(u[O + 5]), "=r"(u[O + 6]), "=r"(u[O + 7]) : "r"(t + O));
  else if constexpr (W - O >= 4) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(u[O]), "=r"(u[O + 1]), "=r"(u[O + 2]), "=r"(u[O + 3]) : "r"(t + O));
    eg_ld<W, O + 4>(t, u);
  } else if constexpr (W - O >= 2) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(u[O]), "=r"(u[O + 1]) : "r"(t + O));
    eg_ld<W, O + 2>(t, u);
  } else if constexpr (W - O == 1)
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(u[O]) : "r"(t + O));
}
template <int W, int O = 0, int M>
__device__ __forceinline__ void eg_st(uint32_t t, const uint32_t (&u)[M]) {
  if constexpr (W - O >= 8)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(t + O), "r"(u[O]), "r"(u[O + 1]),
                 "r"(u[O + 2]), "r"(u[O + 3]), "r"(u[O + 4]), "r"(u[O + 5]), "r"(u[O + 6]), "r"(u[O + 7]) : "memory");
  else if constexpr (W - O >= 4) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(t + O), "r"(u[O]), "r"(u[O + 1]), "r"(u[O + 2]), "r"(u[O + 3]) : "memory");
    eg_st<W, O + 4>(t, u);
  } else if constexpr (W - O >= 2) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(t + O), "r"(u[O]), "r"(u[O + 1]) : "memory");
    eg_st<W, O + 2>(t, u);
  } else if constexpr (W - O == 1)
    asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(t + O), "r"(u[O]) : "memory");
}
// barrier of the CTA, ORing a flag over it
__device__ __forceinline__ bool eg_bar_or(int id, bool flag) {
  uint32_t out;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %2, 0;\n\tbar.red.or.pred p, %1, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(out) : "r"(id), "r"((uint32_t)flag) : "memory");
  return out != 0;
}

// Packed pairs of fp32: one instruction does both multiply-adds.
__device__ __forceinline__ unsigned long long f2_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// CB = p / 128 columns per thread; a CTA has RL = p / 16 rows, worked on in chunks of RC rows of 4-row
// loads (p = 128: one chunk of 8).  Eight warps: a step's scalar work is a chain that more warps would only repeat.
//
// One CTA per SM, whatever the registers would allow: a CTA takes all of the SM's tensor memory and then waits for
// its cluster, so two clusters that shared two SMs, each holding the tensor memory of one, would wait for each other
// for good.  The launch asks for more shared memory than half an SM has, which keeps every two of these CTAs apart,
// also those of launches on different streams; CTAs of other kernels wait for tensor memory but nobody waits for them.
constexpr int EG_RESERVED_SMEM = 116 << 10;
static_assert(2 * EG_RESERVED_SMEM > (228 << 10), "two CTAs do not fit one SM");
constexpr int EG_MAIL = 66;                 // float2 per sender in the mailbox: 64 rows + padding against bank conflicts

template <int CB>
__global__ void __launch_bounds__(EG_THREADS, 1) tridiag_kernel(const __grid_constant__ EighParams p) {
  constexpr int N = CB * 128, RL = CB * 8, RC = RL % 16 ? 8 : 16, LOG = RC == 16 ? 4 : 3;
  __shared__ __align__(16) float2 mail[2][EG_CL * EG_MAIL];   // (A v, next column) of every row, by sender
  __shared__ __align__(16) float mail_g[2][EG_CL];         // parts of tau / 2 v . p
  __shared__ __align__(16) float part[4][RL];   // A v of the own rows, quarter of the columns
  __shared__ __align__(16) float acol[RL];   // next column, own rows
  __shared__ __align__(16) float vrow[2][RL];   // v of the own rows (this step's and the last one's)
  __shared__ __align__(16) float4 vw[RL];    // (-v, -v, -w, -w) of the own rows
  __shared__ float red[12];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_w;
  volatile int* abort_s = &abort_w;
  // warps q and q + 4 hold the same columns (and repeat each other's scalar work); the rows' chunks are split
  const int tid = threadIdx.x & 127, rg = threadIdx.x >> 7, q = tid >> 5, lane = tid & 31;
  const int m = blockIdx.x / EG_CL;
  const int rank = (int)cluster_rank();
  const float* A = p.a + (size_t)m * N * N;

  if (threadIdx.x < 32) {
    tmem_alloc(smem_u32(&tmem_slot), 512);
    tmem_relinquish();
    if (lane == 0) {
      mbar_init(smem_u32(&bars[0]), 1);
      mbar_init(smem_u32(&bars[1]), 1);
      *abort_s = 0;
      fence_mbar_init();
    }
  }
  constexpr uint32_t TX = N * 8 + EG_CL * 4; // bytes a CTA receives per step
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0) { mbar_expect_tx(smem_u32(&bars[0]), TX); mbar_expect_tx(smem_u32(&bars[1]), TX); }
  const uint32_t T = tmem_slot + ((uint32_t)(q * 32) << 16);
  const int c0 = tid;                        // own columns c0 + 128 j
  // local row i is matrix row 16 i + rank, at tensor-memory columns CB * i
#pragma unroll 4
  for (int i = rg; i < RL; i += 2) {
    const float* row = A + (size_t)(16 * i + rank) * N + c0;
    uint32_t v[CB];
#pragma unroll
    for (int j = 0; j < CB; ++j) v[j] = __float_as_uint(row[128 * j]);
    eg_st<CB>(T + CB * i, v);
    if (c0 == 0) acol[i] = __uint_as_float(v[0]);               // column 0
  }
  tmem_wait_st();
  if (tid < RL) {
    vrow[0][tid] = vrow[1][tid] = 0.f;
    part[0][tid] = part[1][tid] = part[2][tid] = part[3][tid] = 0.f;
  }
  __syncthreads();
  cluster_sync();                            // every CTA's barriers are armed
  // Warp w delivers to CTAs 2 w and 2 w + 1: lane = row pair, both (A v, next column) pairs in one 16-byte store.
  uint32_t far[2];
#pragma unroll
  for (int d = 0; d < 2; ++d) far[d] = map_to_cta(smem_u32(&mail[0][0]), 2 * (q + 4 * rg) + d);
  const uint32_t bar_off = smem_u32(&bars[0]) - smem_u32(&mail[0][0]), g_off = smem_u32(&mail_g[0][0]) - smem_u32(&mail[0][0]);
  auto send_rows = [&](int b, float p0, float a0, float p1, float a1) {
    if (2 * lane < RL) {
#pragma unroll
      for (int d = 0; d < 2; ++d)
        st_async_f4(far[d] + (uint32_t)((b * EG_CL + rank) * EG_MAIL + 2 * lane) * 8u, p0, a0, p1, a1, far[d] + bar_off + 8u * (uint32_t)b);
    }
  };
  auto send_gamma = [&](int b, float g) {
    if (lane == 0) {
#pragma unroll
      for (int d = 0; d < 2; ++d)
        st_async_f1(far[d] + g_off + 4u * (uint32_t)(b * EG_CL + rank), g, far[d] + bar_off + 8u * (uint32_t)b);
    }
  };
  const int pair = min(2 * lane, RL - 2);    // own rows of this lane in the delivery
  send_rows(0, 0.f, acol[pair], 0.f, acol[pair + 1]);
  send_gamma(0, 0.f);

  float v[CB];                               // the last reflector (columns from block J0 on)
#pragma unroll
  for (int j = 0; j < CB; ++j) v[j] = 0.f;
  // gamma = tau / 2 v . p with p = tau A v: the same sum, in the same order, everywhere
  auto gamma = [&](int b) {
    const float4* g4 = reinterpret_cast<const float4*>(mail_g[b]);
    float4 s4 = g4[0];
#pragma unroll
    for (int i = 1; i < EG_CL / 4; ++i) { const float4 t = g4[i]; s4.x += t.x; s4.y += t.y; s4.z += t.z; s4.w += t.w; }
    return (s4.x + s4.y) + (s4.z + s4.w);
  };
  // Columns k with (k + 1) / 128 == J0: the blocks of 128 columns before J0 have retired, and the next
  // column lies in block J0.  Column k: its reflector; then one pass over the own rows still active:
  // A -= v w' + w v' with the last reflector, A times the new one, the next column.
  auto phase = [&](auto j0c) -> bool {
    constexpr int J0 = decltype(j0c)::value, W = CB - J0, P = W / 2;
#pragma unroll 1
    for (int k = J0 ? 128 * J0 - 1 : 0; k < 128 * J0 + 127; ++k) {
      const int b = k & 1;
      mbar_wait(smem_u32(&bars[b]), (uint32_t)((k >> 1) & 1), abort_s);
      if (threadIdx.x == 0) mbar_expect_tx(smem_u32(&bars[b]), TX);
      const float gam = gamma(b);
      const float2 mk = mail[b][(k & 15) * EG_MAIL + (k >> 4)];
      const float w1 = mk.x - gam;                              // w[k]; v[k] = 1 (no v yet at k = 0: all zero)
      float x[W], w[W], ss = 0.f;
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const float2 pa = mail[b][(c0 & 15) * EG_MAIL + (c0 >> 4) + 8 * (J0 + j)];
        w[j] = fmaf(-gam, v[J0 + j], pa.x);
        x[j] = pa.y - fmaf(v[J0 + j], w1, w[j]);
      }
      const int cj = c0 + 128 * J0;                             // only block J0 has columns up to k + 1
      if (cj <= k) x[0] = 0.f;
      if (cj == k + 1) red[4] = x[0];                           // (both of its threads, the same value)
      else ss = x[0] * x[0];
#pragma unroll
      for (int j = 1; j < W; ++j) ss = fmaf(x[j], x[j], ss);
      if (tid < RL) {                                           // row scalars of the update
        const float vr = vrow[b ^ 1][tid];
        const float wr = fmaf(-gam, vr, mail[b][rank * EG_MAIL + tid].x);
        vw[tid] = make_float4(-vr, -vr, -wr, -wr);
      }
      ss = warp_sum(ss);
      if (lane == 0) red[q] = ss;
      __syncthreads();
      const float x0 = red[4];
      ss = (red[0] + red[1]) + (red[2] + red[3]);
      float beta = x0, tau = 0.f, scale = 0.f;
      if (ss > 0.f) {
        beta = -copysignf(sqrtf(fmaf(x0, x0, ss)), x0);
        tau = (beta - x0) / beta;
        scale = 1.f / (x0 - beta);
      }
      float vn[W];
#pragma unroll
      for (int j = 0; j < W; ++j) vn[j] = x[j] * scale;         // (x is zero up to row k)
      if (cj == k + 1) vn[0] = 1.f;
      if ((tid & 15) == rank) {
#pragma unroll
        for (int j = 0; j < W; ++j) vrow[b][(c0 >> 4) + 8 * (J0 + j)] = vn[j];   // own columns that are own rows too
      }
      unsigned long long v2[P + 1], w2[P + 1], n2[P + 1];
#pragma unroll
      for (int j = 0; j < P; ++j) {
        v2[j] = f2_pack(v[J0 + 2 * j], v[J0 + 2 * j + 1]);
        w2[j] = f2_pack(w[2 * j], w[2 * j + 1]);
        n2[j] = f2_pack(vn[2 * j], vn[2 * j + 1]);
      }
      const bool has_col = cj == k + 1;                         // this thread holds the next column
#pragma unroll 1
      for (int ch = rg; ch < RL / RC; ch += 2) {
        if (16 * (RC * ch + RC - 1) + rank <= k) continue;      // (uniform) all of the chunk's rows have retired
        float dot[RC];
        uint32_t u[2][4][W];
        const uint32_t Tc = T + CB * RC * ch + J0;
#pragma unroll
        for (int r = 0; r < 4; ++r) eg_ld<W>(Tc + CB * r, u[0][r]);
#pragma unroll
        for (int b4 = 0; b4 < RC / 4; ++b4) {
          ulonglong2 rw[4];                                     // (fetched and stored four rows at a time: the rows' chains overlap)
#pragma unroll
          for (int r = 0; r < 4; ++r) rw[r] = *reinterpret_cast<const ulonglong2*>(&vw[RC * ch + 4 * b4 + r]);
          tmem_wait_ld();
          if (b4 + 1 < RC / 4) {                                // the next four rows come in while these are worked on
#pragma unroll
            for (int r = 0; r < 4; ++r) eg_ld<W>(Tc + CB * (4 * (b4 + 1) + r), u[(b4 + 1) & 1][r]);
          }
          unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
          for (int j = 0; j < P; ++j) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              uint32_t(&y)[W] = u[b4 & 1][r];
              unsigned long long a = f2_pack(__uint_as_float(y[2 * j]), __uint_as_float(y[2 * j + 1]));
              a = f2_fma(rw[r].y, v2[j], f2_fma(rw[r].x, w2[j], a));
              acc[r] = f2_fma(a, n2[j], acc[r]);
              const float2 f = f2_unpack(a);
              y[2 * j] = __float_as_uint(f.x);
              y[2 * j + 1] = __float_as_uint(f.y);
            }
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            uint32_t(&y)[W] = u[b4 & 1][r];
            const float2 f = f2_unpack(acc[r]);
            float sum = f.x + f.y;
            if (W & 1) {
              const float2 rv = f2_unpack(rw[r].x), rz = f2_unpack(rw[r].y);
              const float a = fmaf(rz.x, v[CB - 1], fmaf(rv.x, w[W - 1], __uint_as_float(y[W - 1])));
              sum = fmaf(a, vn[W - 1], sum);
              y[W - 1] = __float_as_uint(a);
            }
            dot[4 * b4 + r] = sum;
          }
#pragma unroll
          for (int r = 0; r < 4; ++r) eg_st<W>(Tc + CB * (4 * b4 + r), u[b4 & 1][r]);
          if (has_col) {
#pragma unroll
            for (int r = 0; r < 4; ++r) acol[RC * ch + 4 * b4 + r] = __uint_as_float(u[b4 & 1][r][0]);
          }
        }
        // sums over the lanes, all rows of the chunk at once: halve the rows a lane carries, fold the lanes
        int off = 16;
#pragma unroll
        for (int h = RC / 2; h >= 1; h >>= 1) {
          const bool up = (lane & off) != 0;
#pragma unroll
          for (int r = 0; r < h; ++r) {
            const float keep = up ? dot[r + h] : dot[r], give = up ? dot[r] : dot[r + h];
            dot[r] = keep + __shfl_xor_sync(0xffffffffu, give, off);
          }
          off >>= 1;
        }
        for (; off >= 1; off >>= 1) dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], off);
        // lane bits from the top select the row
        if ((lane & ((32 >> LOG) - 1)) == 0) part[q][RC * ch + (lane >> (5 - LOG))] = dot[0];
      }
      tmem_wait_st();
      if (eg_bar_or(1, *abort_s != 0)) return false;            // (uniform over the CTA)
      {
        float2 s0 = *reinterpret_cast<const float2*>(&part[0][pair]), s1 = *reinterpret_cast<const float2*>(&part[1][pair]);
        const float2 s2 = *reinterpret_cast<const float2*>(&part[2][pair]), s3 = *reinterpret_cast<const float2*>(&part[3][pair]);
        const float2 ac = *reinterpret_cast<const float2*>(&acol[pair]), vr = *reinterpret_cast<const float2*>(&vrow[b][pair]);
        const float p0 = 16 * pair + rank > k ? tau * ((s0.x + s1.x) + (s2.x + s3.x)) : 0.f;
        const float p1 = 16 * (pair + 1) + rank > k ? tau * ((s0.y + s1.y) + (s2.y + s3.y)) : 0.f;
        send_rows(b ^ 1, p0, ac.x, p1, ac.y);
        const float g = 2 * lane < RL ? fmaf(vr.x, p0, vr.y * p1) : 0.f;
        send_gamma(b ^ 1, 0.5f * tau * warp_sum(g));
      }
      if ((k & 15) == rank && rg == 0) {                        // the record of the step, off the critical path
        float* o = p.refl + ((size_t)m * N + k) * N + c0 + 128 * J0;   // (retired columns stay zero)
#pragma unroll
        for (int j = 0; j < W; ++j) o[128 * j] = vn[j];
        if (tid == 0) {
          p.d[m * N + k] = mk.y - 2.f * w1;
          p.e[m * N + k] = beta;
          p.tau[m * N + k] = tau;
        }
      }
#pragma unroll
      for (int j = 0; j < W; ++j) v[J0 + j] = vn[j];
    }
    return true;
  };
  bool ok = phase(std::integral_constant<int, 0>());
  if constexpr (CB > 1) ok = ok && phase(std::integral_constant<int, (CB > 1 ? 1 : 0)>());
  if constexpr (CB > 2) ok = ok && phase(std::integral_constant<int, (CB > 2 ? 2 : 0)>());
  if constexpr (CB > 3) ok = ok && phase(std::integral_constant<int, (CB > 3 ? 3 : 0)>());
  if constexpr (CB > 4) ok = ok && phase(std::integral_constant<int, (CB > 4 ? 4 : 0)>());
  if constexpr (CB > 5) ok = ok && phase(std::integral_constant<int, (CB > 5 ? 5 : 0)>());
  if constexpr (CB > 6) ok = ok && phase(std::integral_constant<int, (CB > 6 ? 6 : 0)>());
  if constexpr (CB > 7) ok = ok && phase(std::integral_constant<int, (CB > 7 ? 7 : 0)>());
  if (ok) {                                  // the last column: only its diagonal entry
    constexpr int k = N - 1, b = k & 1;
    mbar_wait(smem_u32(&bars[b]), (uint32_t)((k >> 1) & 1), abort_s);
    const float2 mk = mail[b][(k & 15) * EG_MAIL + (k >> 4)];
    if ((k & 15) == rank && threadIdx.x == 0) {
      p.d[m * N + k] = mk.y - 2.f * (mk.x - gamma(b));
      p.e[m * N + k] = p.tau[m * N + k] = 0.f;
    }
  }
  if (threadIdx.x == 0 && *abort_s) atomicExch(p.flag + m, 1);
  tc_fence_before();
  cluster_sync();                            // nobody is still sending to a CTA that leaves
  if (*abort_s) {
    // gave up: what the others had sent by then was not waited for and may still be on its way into this CTA's
    // shared memory (a microsecond)
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (threadIdx.x < 32) tmem_dealloc(tmem_slot, 512);
}

// ---------------------------------------------------------------------------
// eigenvalues of the tridiagonal matrix
// ---------------------------------------------------------------------------
// The matrix in fp64, scaled to eigenvalues within [-1, 1] (Gershgorin): td[i] = (d_i, e_i^2).
// Returns the scale.
__device__ __forceinline__ double eg_load(const EighParams& p, int m, double2* td, int tid, int threads) {
  __shared__ float mx[32];
  const int n = p.p;
  const float *d = p.d + (size_t)m * n, *e = p.e + (size_t)m * n;
  float g = 0.f;
  for (int i = tid; i < n; i += threads)
    g = fmaxf(g, fabsf(d[i]) + (i ? fabsf(e[i - 1]) : 0.f) + (i + 1 < n ? fabsf(e[i]) : 0.f));
  g = warp_max(g);
  if ((tid & 31) == 0) mx[tid >> 5] = g;
  __syncthreads();
  for (int i = 0; i < threads / 32; ++i) g = fmaxf(g, mx[i]);
  const double s = g > 0.f ? 1.0 / (1.0001 * (double)g) : 1.0;
  for (int i = tid; i < n; i += threads) {
    const double ei = i + 1 < n ? (double)e[i] * s : 0.0;
    td[i] = make_double2((double)d[i] * s, ei * ei > 1e-40 ? ei * ei : 1e-40);   // (never zero: the recurrence goes on)
  }
  __syncthreads();
  return 1.0 / s;
}
// keeps (a, b), consecutive terms of the recurrence, away from overflow and underflow
__device__ __forceinline__ void eg_rescale(double& a, double& b) {
  const int ex = max(__double2hiint(a) & 0x7ff00000, __double2hiint(b) & 0x7ff00000);
  const double f = __hiloint2double(0x7fe00000 - max(ex, 0x00100000), 0);
  a *= f;
  b *= f;
}

// CTA = eigenvalue number w (descending); 128 trial points, two per thread (they share the reads of the
// matrix), split its interval into 129 per round.  A step of the recurrence is the latency of one
// multiply-add; more points per round would save rounds, but four matrices fill the fp64 pipes already.
constexpr int EG_PTS = 128;
__global__ void __launch_bounds__(EG_PTS / 2) tridiag_values_kernel(const __grid_constant__ EighParams p) {
  __shared__ double2 td[EG_MAX_P];
  __shared__ int left[2][EG_PTS / 64];
  const int m = blockIdx.y, n = p.p, w = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double unscale = eg_load(p, m, td, threadIdx.x, EG_PTS / 2);
  double lo = -1.0, width = 2.0;
  for (int round = 0; round < 7; ++round) {             // 129^-7 = 2^-49 of the interval
    const double step = width / 129.0, x0 = lo + step * (double)(threadIdx.x + 1), x1 = lo + step * (double)(threadIdx.x + 1 + EG_PTS / 2);
    double b0 = 1.0, a0 = td[0].x - x0, b1 = 1.0, a1 = td[0].x - x1;   // p_{i-1}, p_i at both points
    int neg0 = __double2hiint(a0) < 0, neg1 = __double2hiint(a1) < 0;
    double e2 = td[0].y;
    auto row = [&](int i) {
      const double2 t = td[i];
      const double c0 = fma(t.x - x0, a0, -e2 * b0), c1 = fma(t.x - x1, a1, -e2 * b1);
      neg0 += (unsigned)(__double2hiint(c0) ^ __double2hiint(a0)) >> 31;
      neg1 += (unsigned)(__double2hiint(c1) ^ __double2hiint(a1)) >> 31;
      b0 = a0; a0 = c0; b1 = a1; a1 = c1;
      e2 = t.y;
    };
    int i = 1;
    for (; i + 8 <= n; i += 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) row(i + j);
      eg_rescale(a0, b0);
      eg_rescale(a1, b1);
    }
    for (; i < n; ++i) row(i);
    // neg eigenvalues lie below a point; the one sought has n - 1 - w below it, so it lies right of the
    // first k points
    const int both = __popc(__ballot_sync(0xffffffffu, neg0 <= n - 1 - w)) + __popc(__ballot_sync(0xffffffffu, neg1 <= n - 1 - w));
    if (lane == 0) left[round & 1][warp] = both;
    __syncthreads();
    int k = 0;
#pragma unroll
    for (int t = 0; t < EG_PTS / 64; ++t) k += left[round & 1][t];
    lo += step * k;
    width = step;
  }
  if (threadIdx.x == 0) {
    const double l = lo + 0.5 * width;
    p.lam[(size_t)m * p.rank + w] = l;                  // of the scaled matrix
    p.eigvals[(size_t)m * p.rank + w] = (float)(l * unscale);
  }
}

// ---------------------------------------------------------------------------
// eigenvectors of the tridiagonal matrix: T - lambda = L D+ L' = U D- U'; the vector is built from the
// row where the two factorisations meet best, z_r = 1, z_i = -(e_i / D+_i) z_{i+1} above it and
// z_i = -(e_{i-1} / D-_i) z_{i-1} below
// ---------------------------------------------------------------------------
// 1 / b to fp64 accuracy: two Newton steps on the hardware's 20-bit estimate
__device__ __forceinline__ double eg_recip(double b) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
  r = fma(r, fma(-b, r, 1.0), r);
  return fma(r, fma(-b, r, 1.0), r);
}

__global__ void __launch_bounds__(64) tridiag_vectors_kernel(const __grid_constant__ EighParams p) {
  __shared__ double2 td[EG_MAX_P];
  __shared__ double off_s[EG_MAX_P];                    // e_i, scaled like td
  __shared__ double gmin[2][32];
  __shared__ int gat[2][32];
  const int m = blockIdx.y, n = p.p, lane = threadIdx.x & 31, side = threadIdx.x >> 5;
  eg_load(p, m, td, threadIdx.x, 64);
  for (int i = threadIdx.x; i < n; i += 64) off_s[i] = copysign(sqrt(td[i].y), (double)p.e[(size_t)m * n + i]);
  const int w = blockIdx.x * 32 + lane;
  const double lam = p.lam[(size_t)m * p.rank + min(w, p.rank - 1)];
  const size_t base = ((size_t)m * gridDim.x + blockIdx.x) * n * 32 + lane;
  double* dp = p.dplus + base;
  double* dm = p.dminus + base;
  {
    // D_i = p_i / p_{i-1}: the recurrence carries the numerators, the divisions hang off it
    double* out = side ? dm : dp;
    double b = 1.0, a = 0.0;
    int i = 0;
    auto step = [&](int r) {                            // r: row, from this side
      const int row = side ? n - 1 - r : r;
      const double off = r ? (side ? td[row].y : td[row - 1].y) : 0.0;
      const double c = r ? fma(td[row].x - lam, a, -off * b) : td[row].x - lam;
      if (r) b = a;
      a = c;
      double q = a * eg_recip(b);
      if (fabs(q) < 1e-30) q = 1e-30;
      out[(size_t)row * 32] = q;
    };
    for (; i + 8 <= n; i += 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) step(i + j);
      eg_rescale(a, b);
    }
    for (; i < n; ++i) step(i);
  }
  __syncthreads();
  {
    double best = 1e300;
    int at = 0;
    const int lo = side ? n / 2 : 0, hi = side ? n : n / 2;
    // (n / 2 is a multiple of 64: sixteen rows' loads in flight)
#pragma unroll 1
    for (int i = lo; i < hi; i += 16) {
      double a[16], b[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) { a[j] = dp[(size_t)(i + j) * 32]; b[j] = dm[(size_t)(i + j) * 32]; }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const double g = fabs(a[j] + b[j] - (td[i + j].x - lam));
        if (g < best) { best = g; at = i + j; }
      }
    }
    gmin[side][lane] = best;
    gat[side][lane] = at;
  }
  __syncthreads();
  const int r = gmin[1][lane] < gmin[0][lane] ? gat[1][lane] : gat[0][lane];
  // outwards from row r, sixteen rows at a time: the next sixteen quotients are on their way, and the reciprocals hang off the chain of
  // products (read one by one they waited for the store of the row before: 200 cycles a row)
  float* z = p.z + base;
  const double* quot = side ? dm : dp;
  auto row_of = [&](int j) { return side ? j : n - 1 - j; };         // j = 1 .. n - 1 counts from this side's far end
  if (side == 0) z[(size_t)r * 32] = 1.f;
  double v = 1.0, q[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) q[j] = quot[(size_t)row_of(j) * 32];
#pragma unroll 1
  for (int j0 = 0; j0 < n; j0 += 16) {
    double f[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = row_of(j0 + j);
      f[j] = j0 + j ? -off_s[side ? i - 1 : i] * eg_recip(q[j]) : 0.0;
    }
    if (j0 + 16 < n) {
#pragma unroll
      for (int j = 0; j < 16; ++j) q[j] = quot[(size_t)row_of(j0 + 16 + j) * 32];
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int i = row_of(j0 + j);
      if (side ? i > r : i < r) { v *= f[j]; z[(size_t)i * 32] = (float)v; }
    }
  }
}

// ---------------------------------------------------------------------------
// back to the matrix's own coordinates: x = H_0 H_1 ... H_{n-3} z, four vectors per CTA
// ---------------------------------------------------------------------------
// Eight reflectors per pass, k = 8 g + 7 - i for i = 0 .. 7: with y_i = v_i . x and the products G of the group's reflectors among
// themselves, s_i = tau_i (y_i - sum over m < i of s_m G_im) and x -= sum of s_i v_i.  Element j of a thread is row 256 j + thread
// of all four vectors; a reflector is read once for the four (a warp per vector read all of them for each: 768 warps x 2 MB,
// 1.5 GB through L2, took 332 us for one 1024 x 1024 matrix and 352 us for four).  Pairs of vectors share packed multiply-adds.
// 189 us for one matrix, 271 us for four (192 CTAs on 148 SMs).  Bound by a pass's chain: 32 sums over the lanes, two CTA
// barriers, the eight-step substitution.  Eight vectors a CTA: 299 and 315 us; a thread of 128 with twice the rows: 386 us.
constexpr int EB_V = 4, EB_G = 8;          // vectors of a CTA, reflectors of a group
constexpr int EB_THREADS = 256;
// products of a group's reflectors among themselves, G[m][group][i][l] = v_i . v_l for l < i; a warp per reflector
template <int CB>
__global__ void __launch_bounds__(32 * EB_G) eig_products_kernel(const __grid_constant__ EighParams p) {
  constexpr int N = CB * 128;
  const int g = blockIdx.x, m = blockIdx.y, i = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* refl = p.refl + (size_t)m * N * N;
  float v[4 * CB];
#pragma unroll
  for (int j = 0; j < 4 * CB; ++j) v[j] = __ldg(refl + (size_t)(EB_G * g + EB_G - 1 - i) * N + 32 * j + lane);
#pragma unroll 1
  for (int l = 0; l < i; ++l) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 4 * CB; ++j) s = fmaf(v[j], __ldg(refl + (size_t)(EB_G * g + EB_G - 1 - l) * N + 32 * j + lane), s);
    s = warp_sum(s);
    if (lane == 0) p.products[(((size_t)m * (N / EB_G) + g) * EB_G + i) * EB_G + l] = s;
  }
}
template <int CB>
__global__ void __launch_bounds__(EB_THREADS) eig_back_kernel(const __grid_constant__ EighParams p) {
  constexpr int N = CB * 128, NG = N / EB_G, EL = (N + EB_THREADS - 1) / EB_THREADS, NW = EB_THREADS / 32, Q = EB_V / 2;
  __shared__ float y_s[NW][EB_G * EB_V];   // sums of a warp's rows, [reflector][vector]
  __shared__ __align__(16) float s_s[EB_G * EB_V];
  __shared__ float g_s[2][EB_G * EB_G], tau_s[2][EB_G];
  const int m = blockIdx.y, t = threadIdx.x, warp = t >> 5, lane = t & 31, w0 = blockIdx.x * EB_V;
  const int n_blocks = (p.rank + 31) / 32;
  const float* z = p.z + ((size_t)m * n_blocks + (w0 >> 5)) * N * 32 + (w0 & 31);
  const float* refl = p.refl + (size_t)m * N * N;
  const float* tau = p.tau + (size_t)m * N;
  const float* products = p.products + (size_t)m * NG * EB_G * EB_G;
  // 32 sums over the lanes: halve the values a lane carries; lane l ends up with value l
  auto sums = [&](float (&a)[EB_G * EB_V], float* out) {
    int off = 16;
#pragma unroll
    for (int h = EB_G * EB_V / 2; h >= 1; h >>= 1) {
      const bool up = (lane & off) != 0;
#pragma unroll
      for (int r = 0; r < h; ++r) {
        const float keep = up ? a[r + h] : a[r], give = up ? a[r] : a[r + h];
        a[r] = keep + __shfl_xor_sync(0xffffffffu, give, off);
      }
      off >>= 1;
    }
    out[lane] = a[0];
  };
  auto total = [&](int i) {                // of value i, over the warps
    float y = y_s[0][i];
#pragma unroll
    for (int w = 1; w < NW; ++w) y += y_s[w][i];
    return y;
  };
  auto load_group = [&](int g, float (&v)[EB_G][EL]) {
    const float* rows = refl + (size_t)(EB_G * g) * N + t;
#pragma unroll
    for (int i = 0; i < EB_G; ++i)
#pragma unroll
      for (int j = 0; j < EL; ++j)         // (an odd number of blocks: the upper half of the last 256 rows does not exist)
        v[i][j] = (CB % 2 == 0 || j < EL - 1 || t < 128) ? __ldg(rows + (EB_G - 1 - i) * N + EB_THREADS * j) : 0.f;
  };
  unsigned long long x[EL][Q];             // pairs of vectors
#pragma unroll
  for (int j = 0; j < EL; ++j) {
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (2 * j + (t >> 7) < CB) f = *reinterpret_cast<const float4*>(z + (size_t)(EB_THREADS * j + t) * 32);
    x[j][0] = f2_pack(f.x, f.y); x[j][1] = f2_pack(f.z, f.w);
  }
  {                                        // to length one
    float a[EB_G * EB_V];
#pragma unroll
    for (int q = 0; q < EB_G * EB_V; ++q) a[q] = 0.f;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      unsigned long long s = 0ull;
#pragma unroll
      for (int j = 0; j < EL; ++j) s = f2_fma(x[j][q], x[j][q], s);
      const float2 f = f2_unpack(s);
      a[2 * q] = f.x;
      a[2 * q + 1] = f.y;
    }
    sums(a, y_s[warp]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const unsigned long long inv = f2_pack(rsqrtf(total(2 * q)), rsqrtf(total(2 * q + 1)));
#pragma unroll
      for (int j = 0; j < EL; ++j) x[j][q] = f2_fma(x[j][q], inv, 0ull);
    }
    __syncthreads();
  }
  // the next group's reflectors are on their way while one is applied
  float v[EB_G][EL];
  load_group(NG - 1, v);
#pragma unroll 1
  for (int g = NG - 1; g >= 0; --g) {
    const int j0 = g >> 5;                 // first 256 rows with a non-zero element
    if (t < EB_G * EB_G) g_s[g & 1][t] = products[(size_t)g * EB_G * EB_G + t];
    else if (t < EB_G * EB_G + EB_G) tau_s[g & 1][t - EB_G * EB_G] = tau[EB_G * g + EB_G - 1 - (t - EB_G * EB_G)];
    float next[EB_G][EL];
    load_group(max(g - 1, 0), next);
    {
      unsigned long long acc[EB_G][Q];
#pragma unroll
      for (int i = 0; i < EB_G * Q; ++i) acc[i / Q][i % Q] = 0ull;
#pragma unroll
      for (int j = 0; j < EL; ++j)
        if (j >= j0) {
#pragma unroll
          for (int i = 0; i < EB_G; ++i) {
            const unsigned long long vv = f2_pack(v[i][j], v[i][j]);
#pragma unroll
            for (int q = 0; q < Q; ++q) acc[i][q] = f2_fma(vv, x[j][q], acc[i][q]);
          }
        }
      float a[EB_G * EB_V];
#pragma unroll
      for (int i = 0; i < EB_G * Q; ++i) {
        const float2 f = f2_unpack(acc[i / Q][i % Q]);
        a[2 * i] = f.x;
        a[2 * i + 1] = f.y;
      }
      sums(a, y_s[warp]);
    }
    __syncthreads();
    if (t < EB_V) {                        // vector t
      float y[EB_G];
#pragma unroll
      for (int i = 0; i < EB_G; ++i) y[i] = total(EB_V * i + t);
#pragma unroll
      for (int i = 0; i < EB_G; ++i) {
        const float s = tau_s[g & 1][i] * y[i];
        s_s[EB_V * i + t] = -s;
#pragma unroll
        for (int l = i + 1; l < EB_G; ++l) y[l] = fmaf(-s, g_s[g & 1][EB_G * l + i], y[l]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < EB_G; ++i) {
      const ulonglong2 s2 = *reinterpret_cast<const ulonglong2*>(&s_s[EB_V * i]);
      const unsigned long long s[Q] = {s2.x, s2.y};
#pragma unroll
      for (int j = 0; j < EL; ++j)
        if (j >= j0) {
          const unsigned long long vv = f2_pack(v[i][j], v[i][j]);
#pragma unroll
          for (int q = 0; q < Q; ++q) x[j][q] = f2_fma(vv, s[q], x[j][q]);
        }
    }
#pragma unroll
    for (int i = 0; i < EB_G * EL; ++i) v[i / EL][i % EL] = next[i / EL][i % EL];
  }
  float* out = p.basis + (size_t)m * N * p.rank;
#pragma unroll
  for (int j = 0; j < EL; ++j)
    if (2 * j + (t >> 7) < CB) {
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float2 f = f2_unpack(x[j][q]);
        float* at = out + (size_t)(EB_THREADS * j + t) * p.rank + w0 + 2 * q;
        if (w0 + 2 * q < p.rank) at[0] = f.x;
        if (w0 + 2 * q + 1 < p.rank) at[1] = f.y;
      }
    }
}

// Vectors of close eigenvalues that step 3 could not tell apart: the next two neighbours of every vector
// must be orthogonal to it, and its length one.
// CTA = 32 vectors, lane = vector, warp = every 32nd row.
constexpr int EC_WARPS = 32;
__global__ void __launch_bounds__(32 * EC_WARPS) eig_check_kernel(const __grid_constant__ EighParams p) {
  __shared__ float sum[EC_WARPS][3][32];
  const int m = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = blockIdx.x * 32 + lane;
  const float* v = p.basis + (size_t)m * p.p * p.rank;
  const int w0 = min(w, p.rank - 1), w1 = min(w + 1, p.rank - 1), w2 = min(w + 2, p.rank - 1);
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll 8
  for (int i = warp; i < p.p; i += EC_WARPS) {
    const float* row = v + (size_t)i * p.rank;
    const float a = row[w0];
    s0 = fmaf(a, a, s0);
    s1 = fmaf(a, row[w1], s1);
    s2 = fmaf(a, row[w2], s2);
  }
  sum[warp][0][lane] = s0; sum[warp][1][lane] = s1; sum[warp][2][lane] = s2;
  __syncthreads();
  if (warp > 0 || w >= p.rank) return;
#pragma unroll
  for (int i = 1; i < EC_WARPS; ++i) { s0 += sum[i][0][lane]; s1 += sum[i][1][lane]; s2 += sum[i][2][lane]; }
  if (w + 1 >= p.rank) s1 = 0.f;
  if (w + 2 >= p.rank) s2 = 0.f;
  if (!(fabsf(s0 - 1.f) < 1e-3f && fabsf(s1) < 1e-3f && fabsf(s2) < 1e-3f)) p.flag[m] = 1;   // (NaN: flagged)
}

template <int CB>
static int launch_eigh(const EighParams& p, int count, cudaStream_t st) {
  static std::atomic<bool> configured[MAX_DEVICES];
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= MAX_DEVICES) return SHARD_E_ARG;
  if (!configured[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(tridiag_kernel<CB>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return (int)e;
    e = cudaFuncSetAttribute(tridiag_kernel<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, EG_RESERVED_SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev].store(true, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(EG_CL * count);
  cfg.blockDim = dim3(EG_THREADS);
  cfg.dynamicSmemBytes = EG_RESERVED_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = EG_CL;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, tridiag_kernel<CB>, p);
  if (e != cudaSuccess) return (int)e;
  tridiag_values_kernel<<<dim3(p.rank, count), EG_PTS / 2, 0, st>>>(p);
  tridiag_vectors_kernel<<<dim3((p.rank + 31) / 32, count), 64, 0, st>>>(p);
  eig_products_kernel<CB><<<dim3(CB * 128 / EB_G, count), 32 * EB_G, 0, st>>>(p);
  eig_back_kernel<CB><<<dim3((p.rank + EB_V - 1) / EB_V, count), EB_THREADS, 0, st>>>(p);
  eig_check_kernel<<<dim3((p.rank + 31) / 32, count), 32 * EC_WARPS, 0, st>>>(p);
  e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

struct EighLayout { size_t refl, tau, d, e, lam, dplus, dminus, z, products, bytes; };
static EighLayout eg_layout(size_t L, size_t p, size_t rank) {
  EighLayout l;
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t nb = (rank + 31) / 32 * 32;
  l.refl = 0;
  l.tau = l.refl + up(L * p * p * 4);
  l.d = l.tau + up(L * p * 4);
  l.e = l.d + up(L * p * 4);
  l.lam = l.e + up(L * p * 4);
  l.dplus = l.lam + up(L * rank * 8);
  l.dminus = l.dplus + up(L * nb * p * 8);
  l.z = l.dminus + up(L * nb * p * 8);
  l.products = l.dplus;                    // (the factorisations have been used by then)
  l.bytes = l.z + up(L * nb * p * 4);
  return l;
}

}  // namespace shard

using namespace shard;

extern "C" size_t shard_b200_eigh_workspace_bytes(int32_t count, int32_t p, int32_t rank) {
  if (count < 1 || p < 128 || p > EG_MAX_P || (p % 128) || rank < 1 || rank > p) return 0;
  return eg_layout(count, p, rank).bytes;
}

extern "C" int shard_b200_eigh(const float* a, int32_t count, int32_t p, int32_t rank, float* basis_out, float* eigvals_out,
                               int32_t* flag_out, void* workspace, size_t workspace_bytes, void* stream) {
  if (!a || !basis_out || !eigvals_out || !flag_out || !workspace) return SHARD_E_ARG;
  const size_t need = shard_b200_eigh_workspace_bytes(count, p, rank);
  if (need == 0) return SHARD_E_ARG;
  if (workspace_bytes < need) return SHARD_E_WORKSPACE;
  if (((uintptr_t)a | (uintptr_t)workspace) & 15) return SHARD_E_ALIGN;
  const EighLayout l = eg_layout(count, p, rank);
  unsigned char* ws = (unsigned char*)workspace;
  EighParams q{};
  q.a = a;
  q.p = p;
  q.rank = rank;
  q.refl = (float*)(ws + l.refl);
  q.tau = (float*)(ws + l.tau);
  q.d = (float*)(ws + l.d);
  q.e = (float*)(ws + l.e);
  q.lam = (double*)(ws + l.lam);
  q.dplus = (double*)(ws + l.dplus);
  q.dminus = (double*)(ws + l.dminus);
  q.z = (float*)(ws + l.z);
  q.products = (float*)(ws + l.products);
  q.basis = basis_out;
  q.eigvals = eigvals_out;
  q.flag = flag_out;
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(flag_out, 0, (size_t)count * 4, st);
  // (a step leaves the blocks of columns that have retired alone, and the back-transformation reads whole rows)
  if (e == cudaSuccess) e = cudaMemsetAsync(q.refl, 0, (size_t)count * p * p * 4, st);
  if (e != cudaSuccess) return (int)e;
  switch (p / 128) {
    case 1: return launch_eigh<1>(q, count, st);
    case 2: return launch_eigh<2>(q, count, st);
    case 3: return launch_eigh<3>(q, count, st);
    case 4: return launch_eigh<4>(q, count, st);
    case 5: return launch_eigh<5>(q, count, st);
    case 6: return launch_eigh<6>(q, count, st);
    case 7: return launch_eigh<7>(q, count, st);
    default: return launch_eigh<8>(q, count, st);
  }
}
