// Lloyd's algorithm over 4-channel sub-vectors with a 256-entry codebook, the training of the V
// quantiser: no host round trips, one launch per iteration.
//
// An iteration assigns every point to its nearest centroid -- fp32 differences, squares and sums rounded
// one by one, first minimum wins, bit for bit as vq_assign_kernel -- and moves the centroids.  The
// points are first sorted along a Morton curve (a counting sort of 16- or 20-bit cell numbers), so that
// 64 consecutive points lie in a small box; then an iteration looks at few centroids instead of 256:
//
//   a warp takes a run of 64-point tiles.  Of all 256 centroids, spread over the lanes, it finds the one
//   nearest to the middle of the run's box, c', and drops every c that is farther than c' from each
//   point of the box: dist(p, c) - dist(p, c') is linear in p, so its minimum over the box is
//   dist(mid, c) - dist(mid, c') - 2 sum |c - c'| half-width.  The survivors (about 15 at 8.4 M points,
//   30 at 2 M) go through the same test with each tile's own box, and the few left (5, 10) are evaluated
//   for the points.
//
// A point that is not finite is at no distance below infinity from anything, so it belongs to centroid 0 like a
// first minimum: its infinities and NaN go into that centroid beside the fixed-point sums (`odd`).
//
// A centroid is dropped only if it is farther by more than the rounding of both sides can hide
// (KM_SLACK), so the assignment is the exact one.
//
// Centroid sums are fixed-point integers (2^-30 of the data's range): they do not depend on the order of
// additions -- two runs give the same bits -- and an iteration only books the points that changed
// sides.  The last CTA to finish divides, tests for convergence and leaves a flag that turns the
// remaining launches into empty ones.
//
// Bound: instruction issue (about 250 instructions per 32 points and iteration; the direct search needs
// 3 500, a tensor-core search with exact re-check of the close calls measured 370 us per iteration at
// 8.4 M points) and 20 us per launch at either end; the points' 134 MB at 8.4 M are 21 us at the measured
// copy rate.  8.4 M points, 30 iterations: 40 ms for the direct search with host round trips, 4.1 ms with
// every move booked where it is found, 3.7 ms with moves collected until they fill a warp (600 -> 500
// instructions per 64 points) and every warp's first run dealt out without asking.  Distances in packed
// fp32 pairs (2 instructions fewer in 3) measured 3 % more: the pairs cost registers.  Keeping each tile's
// distance to its nearest boundary to skip tiles the centroids' moves cannot have touched would skip one
// tile in ten by the last iteration.
#include "tcgen05.cuh"

namespace shard {

constexpr int KM_THREADS = 512, KM_WARPS = KM_THREADS / 32;
constexpr int KM_TILE = 64;                   // points per box: two per lane
constexpr int KM_MAX_RUN = 8;                 // tiles per run
constexpr int KM_QUEUE = 64;                  // points a warp may have waiting to be booked (see `flush`)
constexpr int KM_CTA_POINTS = 60000;          // points a CTA books at most: its partial sums stay within int32

struct KmeansHeader {      // head of the workspace; zero when the first iteration starts
  int done;                // converged: the launches behind it do nothing
  int ticket;              // CTAs that have finished the current iteration
  unsigned int max_bits;   // max |x| (as float bits) if the caller did not name a bound
  unsigned int next_run;   // runs handed out in the current iteration
  unsigned int odd;        // three bits per channel: some point has +inf, -inf, NaN there
  long long sums[256 * 4]; // fixed point
  int counts[256];
};

// workspace: header | cell counters [cells] | totals of 1024-cell blocks | sorted points | their original
// numbers | boxes (low corner, high corner) | assignment of the sorted points
struct KmeansLayout {
  size_t cells, totals, xs, perm, boxes, idx, bytes;
  int bits;                // per channel
};
__host__ inline KmeansLayout km_layout(long long n) {
  KmeansLayout l;
  l.bits = n >= (1 << 20) ? 5 : 4;            // cells of about eight points or more at either size
  const size_t n_cells = (size_t)1 << (4 * l.bits);
  const size_t n_pad = ((size_t)n + KM_TILE - 1) / KM_TILE * KM_TILE;
  auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
  l.cells = up(sizeof(KmeansHeader));
  l.totals = l.cells + up(n_cells * 4);
  l.xs = l.totals + up(1024 * 4);
  l.perm = l.xs + n_pad * 16;
  l.boxes = l.perm + up(n_pad * 4);
  l.idx = l.boxes + up(n_pad / KM_TILE * 32);
  l.bytes = l.idx + up(n_pad);
  return l;
}

struct KmeansParams {
  const float4* x;         // points as given
  long long n;
  float4* centroids;
  uint8_t* idx;            // result, in the order of x
  KmeansHeader* h;
  unsigned int *cells, *totals;
  float4* xs;
  unsigned int* perm;
  float4* boxes;
  uint8_t* idx_s;
  float max_abs;           // bound on |x|, or 0: take h->max_bits
  int bits;
  int run;                 // tiles per run
  int warp_runs;           // runs a warp takes at most
  int it;
  size_t ws_stride;        // bytes from one problem's workspace to the next one's (problem = blockIdx.y)
};
// the parameters of problem number b of a batch
__device__ __forceinline__ KmeansParams km_problem(KmeansParams p, int b) {
  const size_t o = (size_t)b * p.ws_stride;
  auto at = [&](auto* ptr) { return reinterpret_cast<decltype(ptr)>(reinterpret_cast<unsigned char*>(ptr) + o); };
  p.x += (size_t)b * p.n;
  p.centroids += (size_t)b * 256;
  p.idx += (size_t)b * p.n;
  p.h = at(p.h);
  p.cells = at(p.cells);
  p.totals = at(p.totals);
  p.xs = at(p.xs);
  p.perm = at(p.perm);
  p.boxes = at(p.boxes);
  p.idx_s = at(p.idx_s);
  return p;
}

// Middle and half-widths of a box (the half-widths rounded up), and their squared length.
struct KmBox { float4 mid, h; float hh; };
__device__ __forceinline__ KmBox km_box(float4 lo, float4 hi) {
  KmBox b;
  const float up = 1.f + 1e-6f;
  b.mid = make_float4(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z), 0.5f * (lo.w + hi.w));
  b.h = make_float4(fmaxf(hi.x - b.mid.x, b.mid.x - lo.x) * up, fmaxf(hi.y - b.mid.y, b.mid.y - lo.y) * up,
                    fmaxf(hi.z - b.mid.z, b.mid.z - lo.z) * up, fmaxf(hi.w - b.mid.w, b.mid.w - lo.w) * up);
  b.hh = b.h.x * b.h.x + b.h.y * b.h.y + b.h.z * b.h.z + b.h.w * b.h.w;
  return b;
}
__device__ __forceinline__ float km_mid_dist(const KmBox& b, float4 c) {
  const float d0 = b.mid.x - c.x, d1 = b.mid.y - c.y, d2 = b.mid.z - c.z, d3 = b.mid.w - c.w;
  return fmaf(d0, d0, fmaf(d1, d1, fmaf(d2, d2, d3 * d3)));
}
// May c (at distance d from the middle) be as near as c' (at distance d_near) to some point of the box?
// All of it -- d, d_near, the half-width term, and the two distances whose order is at stake, at most
// 2 d + 2 hh each -- is rounded to a few 2^-24 of itself; the sum of that stays below KM_SLACK (d + hh).
constexpr float KM_SLACK = 4e-6f;
__device__ __forceinline__ bool km_may_win(const KmBox& b, float4 c, float d, float4 near, float d_near) {
  const float reach = fmaf(fabsf(c.x - near.x), b.h.x, fmaf(fabsf(c.y - near.y), b.h.y,
                      fmaf(fabsf(c.z - near.z), b.h.z, fabsf(c.w - near.w) * b.h.w)));
  return !(d - d_near - 2.f * reach > KM_SLACK * (d + b.hh));   // (true for NaN)
}
// distance exactly as the nearest-centroid rule defines it
__device__ __forceinline__ float km_dist(float4 p, float4 c) {
  const float d0 = __fsub_rn(p.x, c.x), d1 = __fsub_rn(p.y, c.y), d2 = __fsub_rn(p.z, c.z), d3 = __fsub_rn(p.w, c.w);
  float dist = __fadd_rn(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
  dist = __fadd_rn(dist, __fmul_rn(d2, d2));
  return __fadd_rn(dist, __fmul_rn(d3, d3));
}
// minimum over the warp of a non-negative float (or +inf)
__device__ __forceinline__ float warp_min_nonneg(float v) {
  return __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(v)));
}
// power of two s with max_abs * s in (1/2, 1]
__device__ __forceinline__ float km_scale(float max_abs) {
  int e;
  if (!(max_abs > 0.f) || isinf(max_abs)) return 1.f;
  const float f = frexpf(max_abs, &e);          // max_abs = f * 2^e, f in [1/2, 1)
  if (f == 0.5f) e -= 1;
  return ldexpf(1.f, -e);
}
__device__ __forceinline__ float km_scale(const KmeansParams& p) {
  return km_scale(p.max_abs > 0.f ? p.max_abs : __uint_as_float(__ldcg(&p.h->max_bits)));
}
// Cell number: per channel 2^bits cells, finer towards zero (square-root spacing: the data is dense
// there), the channels' bits interleaved.
__device__ __forceinline__ unsigned int km_cell(float4 v, float scale, int bits) {
  const float f[4] = {v.x * scale, v.y * scale, v.z * scale, v.w * scale};
  const int half = 1 << (bits - 1);
  unsigned int q[4], key = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s = min((int)(sqrtf(fabsf(f[j])) * (float)half), half - 1);
    q[j] = (unsigned int)(f[j] < 0.f ? half - 1 - s : half + s);
  }
  for (int b = bits - 1; b >= 0; --b)
#pragma unroll
    for (int j = 0; j < 4; ++j) key = (key << 1) | ((q[j] >> b) & 1u);
  return key;
}

__global__ void __launch_bounds__(256) kmeans_max_abs_kernel(const __grid_constant__ KmeansParams pp) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  float m = 0.f;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += (long long)gridDim.x * blockDim.x) {
    const float4 v = p.x[i];
    const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (isfinite(f[j])) m = fmaxf(m, fabsf(f[j]));
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomicMax(&p.h->max_bits, __float_as_uint(m));
}

// Points per cell, then (SCATTER) the points to their places.  Lanes whose points all fall into one
// cell count together: constant data would otherwise queue up at one counter.
template <bool SCATTER>
__global__ void __launch_bounds__(256) kmeans_sort_kernel(const __grid_constant__ KmeansParams pp) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  const float scale = km_scale(p);
  const int lane = threadIdx.x & 31;
  const long long n_up = (p.n + 31) & ~31ll;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_up; i += (long long)gridDim.x * blockDim.x) {
    const bool live = i < p.n;
    const float4 v = live ? p.x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    const unsigned int key = live ? km_cell(v, scale, p.bits) : 0xffffffffu;
    if (!SCATTER && live && !isfinite((v.x - v.x) + (v.y - v.y) + (v.z - v.z) + (v.w - v.w))) {
      const float f[4] = {v.x, v.y, v.z, v.w};
      unsigned int bits = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) bits |= (isnan(f[j]) ? 4u : isinf(f[j]) ? (f[j] > 0.f ? 1u : 2u) : 0u) << (3 * j);
      atomicOr(&p.h->odd, bits);
    }
    const bool one = __all_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 0));
    unsigned int pos = 0;
    if (one) {
      if (lane == 0) pos = atomicAdd(p.cells + key, 32u);
      pos = __shfl_sync(0xffffffffu, pos, 0) + lane;
    } else if (live) {
      pos = atomicAdd(p.cells + key, 1u);
    }
    if (SCATTER && live) {
      pos += p.totals[key >> 10];
      p.xs[pos] = v;
      p.perm[pos] = (unsigned int)i;
    }
  }
}
// counters -> places within a block of 1024 cells; the blocks' totals
__global__ void __launch_bounds__(1024) kmeans_scan_kernel(const __grid_constant__ KmeansParams pp, bool of_totals) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  unsigned int* cells = of_totals ? p.totals : p.cells;
  unsigned int* totals = of_totals ? nullptr : p.totals;
  __shared__ unsigned int ws[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned int* c = cells + (size_t)blockIdx.x * 1024 + tid;
  const unsigned int v = *c;
  unsigned int s = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const unsigned int t = __shfl_up_sync(0xffffffffu, s, o); if (lane >= o) s += t; }
  if (lane == 31) ws[warp] = s;
  __syncthreads();
  if (warp == 0) {
    unsigned int w = ws[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const unsigned int t = __shfl_up_sync(0xffffffffu, w, o); if (lane >= o) w += t; }
    ws[lane] = w;
  }
  __syncthreads();
  s += warp ? ws[warp - 1] : 0u;
  *c = s - v;
  if (tid == 1023 && totals) totals[blockIdx.x] = s;
}

// boxes of the sorted points; the last tile is filled up with its last point
__global__ void __launch_bounds__(256) kmeans_boxes_kernel(const __grid_constant__ KmeansParams pp) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  const int lane = threadIdx.x & 31;
  const long long n_tiles = (p.n + KM_TILE - 1) / KM_TILE;
  for (long long t = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); t < n_tiles; t += (long long)gridDim.x * 8) {
    const long long i0 = t * KM_TILE + lane, i1 = i0 + 32;
    const float4 a = p.xs[min(i0, p.n - 1)], b = p.xs[min(i1, p.n - 1)];
    float lo[4] = {fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), fminf(a.w, b.w)};
    float hi[4] = {fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), fmaxf(a.w, b.w)};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo[j] = fminf(lo[j], __shfl_xor_sync(0xffffffffu, lo[j], o));
        hi[j] = fmaxf(hi[j], __shfl_xor_sync(0xffffffffu, hi[j], o));
      }
    }
    if (lane == 0) p.boxes[2 * t] = make_float4(lo[0], lo[1], lo[2], lo[3]);
    if (lane == 1) p.boxes[2 * t + 1] = make_float4(hi[0], hi[1], hi[2], hi[3]);
  }
}

__global__ void __launch_bounds__(256) kmeans_unsort_kernel(const __grid_constant__ KmeansParams pp) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += (long long)gridDim.x * blockDim.x)
    p.idx[p.perm[i]] = p.idx_s[i];
}

__global__ void __launch_bounds__(KM_THREADS, 2) kmeans_iteration_kernel(const __grid_constant__ KmeansParams pp) {
  const KmeansParams p = km_problem(pp, blockIdx.y);
  __shared__ float4 c_s[256];
  __shared__ int acc_s[256 * 9];                               // high and low halves of the sums' changes, count's change
  __shared__ float4 wait_s[KM_WARPS][KM_QUEUE];                // points that changed sides, not booked yet
  __shared__ uint16_t sides_s[KM_WARPS][KM_QUEUE];             // ... their centroids: new, old << 8
  __shared__ uint8_t run_s[KM_WARPS][256];                     // survivors of the run test, ascending
  __shared__ __align__(2) uint8_t few_s[KM_WARPS][258];        // survivors of the tile test
  __shared__ int last_s;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < 256 * 9; i += KM_THREADS) acc_s[i] = 0;
  griddep_launch();
  griddep_wait();                                              // the centroids of the iteration before
  if (__ldcg(&p.h->done)) return;                              // (uniform over the grid: set by an earlier launch)
  const float qscale = km_scale(p) * 1073741824.f;             // fixed point: 2^30 per unit of scaled data
  if (tid < 256) c_s[tid] = __ldcg(p.centroids + tid);
  __syncthreads();

  auto fixed = [&](float v, int& hi, int& lo) {
    const int fx = __float2int_rn(v * qscale);                 // |.| <= 2^30
    hi = fx >> 15;
    lo = fx & 32767;
  };
  // Books the lanes' points with `go` under centroid k, summed per centroid first (sorted points: a warp
  // knows two or three).
  auto book = [&](float4 pt, int k, bool go) {
    unsigned int todo = __ballot_sync(0xffffffffu, go);
    int hi[4], lo[4];
    fixed(pt.x, hi[0], lo[0]); fixed(pt.y, hi[1], lo[1]); fixed(pt.z, hi[2], lo[2]); fixed(pt.w, hi[3], lo[3]);
    while (todo) {
      const int kk = __shfl_sync(0xffffffffu, k, __ffs(todo) - 1);
      const bool mine = go && k == kk;
      const unsigned int who = __ballot_sync(0xffffffffu, mine);
      int s = __popc(who);                                     // lane c < 8 ends up with sum c, the others with the count
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int a = __reduce_add_sync(0xffffffffu, mine ? hi[c] : 0), b = __reduce_add_sync(0xffffffffu, mine ? lo[c] : 0);
        if (lane == c) s = a;
        if (lane == 4 + c) s = b;
      }
      if (lane < 9) atomicAdd(&acc_s[kk * 9 + lane], s);
      todo &= ~who;
    }
  };
  // Later iterations move one point in a hundred.  Booking those where they are found would run mostly
  // empty warps through it (a third of the kernel's instructions); they wait in shared memory until
  // there is one for every lane.
  int waiting = 0;
  auto flush = [&](int first) {
    __syncwarp();
    if (first + lane < waiting) {
      const float4 pt = wait_s[warp][first + lane];
      const int sides = sides_s[warp][first + lane];
      int *on = acc_s + (sides & 255) * 9, *off = acc_s + (sides >> 8) * 9;
      const float pv[4] = {pt.x, pt.y, pt.z, pt.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        int hi, lo;
        fixed(pv[c], hi, lo);
        atomicAdd(on + c, hi);
        atomicAdd(on + 4 + c, lo);
        atomicAdd(off + c, -hi);
        atomicAdd(off + 4 + c, -lo);
      }
      atomicAdd(on + 8, 1);
      atomicAdd(off + 8, -1);
    }
    waiting = first;
    __syncwarp();
  };

  const long long n_tiles = (p.n + KM_TILE - 1) / KM_TILE;
  const long long n_runs = (n_tiles + p.run - 1) / p.run;
  const float inf = __int_as_float(0x7f800000);
  // Runs are handed out one at a time (their work differs, and some SMs may be busy with another
  // stream's kernels); the next one is asked for while the current one is worked on.
  auto ask = [&]() {
    unsigned int v = 0;
    if (lane == 0) v = gridDim.x * KM_WARPS + atomicAdd(&p.h->next_run, 1u);
    return v;
  };
  unsigned int asked = blockIdx.x * KM_WARPS + warp;           // (the first without asking: they would queue up at the counter)
  for (int quota = p.warp_runs; quota > 0; --quota) {
    const long long run = __shfl_sync(0xffffffffu, asked, 0);
    if (run >= n_runs) break;
    if (quota > 1) asked = ask();
    const long long t_lo = run * p.run;
    const int nt = (int)min((long long)p.run, n_tiles - t_lo);
    {
      // ---- the run's box against all centroids ---------------------------------------------------
      const float4* bx = p.boxes + 2 * t_lo;
      const float4 my_lo = bx[2 * min(lane, nt - 1)], my_hi = bx[2 * min(lane, nt - 1) + 1];   // lane j < nt: box of tile j
      const KmBox mine = km_box(my_lo, my_hi);
      float4 lo = my_lo, hi = my_hi;
      for (int o = 1; o < p.run; o <<= 1) {                    // (lanes 0..run-1 hold every box: run is a power of two)
        lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o)); hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
        lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o)); hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
        lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o)); hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
        lo.w = fminf(lo.w, __shfl_xor_sync(0xffffffffu, lo.w, o)); hi.w = fmaxf(hi.w, __shfl_xor_sync(0xffffffffu, hi.w, o));
      }
      lo.x = __shfl_sync(0xffffffffu, lo.x, 0); lo.y = __shfl_sync(0xffffffffu, lo.y, 0);
      lo.z = __shfl_sync(0xffffffffu, lo.z, 0); lo.w = __shfl_sync(0xffffffffu, lo.w, 0);
      hi.x = __shfl_sync(0xffffffffu, hi.x, 0); hi.y = __shfl_sync(0xffffffffu, hi.y, 0);
      hi.z = __shfl_sync(0xffffffffu, hi.z, 0); hi.w = __shfl_sync(0xffffffffu, hi.w, 0);
      const KmBox rb = km_box(lo, hi);
      float d[8], dn = inf;
      int kn = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        d[j] = km_mid_dist(rb, c_s[32 * j + lane]);
        if (d[j] < dn) { dn = d[j]; kn = 32 * j + lane; }
      }
      float dmin = warp_min_nonneg(dn);
      kn = __shfl_sync(0xffffffffu, kn, (__ffs(__ballot_sync(0xffffffffu, dn == dmin)) - 1) & 31);
      float4 near = c_s[kn];
      int len = 0;
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool in = km_may_win(rb, c_s[32 * j + lane], d[j], near, dmin);
        const unsigned int bal = __ballot_sync(0xffffffffu, in);
        if (in) run_s[warp][len + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)(32 * j + lane);
        len += __popc(bal);
      }
      __syncwarp();
      // ---- tile by tile -----------------------------------------------------------------------------
      float4 n0 = make_float4(0.f, 0.f, 0.f, 0.f), n1 = n0;
      int o0 = 0, o1 = 0;
      const unsigned int at = (unsigned int)t_lo * KM_TILE + lane, end = (unsigned int)p.n;
      auto fetch = [&](int q) {
        const unsigned int i0 = min(at + q * KM_TILE, end - 1), i1 = min(at + q * KM_TILE + 32, end - 1);
        n0 = p.xs[i0];
        n1 = p.xs[i1];
        if (p.it > 0) { o0 = __ldcg(p.idx_s + i0); o1 = __ldcg(p.idx_s + i1); }
      };
      fetch(0);
      for (int q = 0; q < nt; ++q) {
        const float4 p0 = n0, p1 = n1;
        const int old0 = o0, old1 = o1;
        if (q + 1 < nt) fetch(q + 1);
        KmBox tb;
        tb.mid.x = __shfl_sync(0xffffffffu, mine.mid.x, q); tb.mid.y = __shfl_sync(0xffffffffu, mine.mid.y, q);
        tb.mid.z = __shfl_sync(0xffffffffu, mine.mid.z, q); tb.mid.w = __shfl_sync(0xffffffffu, mine.mid.w, q);
        tb.h.x = __shfl_sync(0xffffffffu, mine.h.x, q); tb.h.y = __shfl_sync(0xffffffffu, mine.h.y, q);
        tb.h.z = __shfl_sync(0xffffffffu, mine.h.z, q); tb.h.w = __shfl_sync(0xffffffffu, mine.h.w, q);
        tb.hh = __shfl_sync(0xffffffffu, mine.hh, q);
        int cnt = 0;
        auto keep = [&](bool in, int k) {
          const unsigned int bal = __ballot_sync(0xffffffffu, in);
          if (in) few_s[warp][cnt + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)k;
          cnt += __popc(bal);
        };
        if (len <= 32) {                                       // (nearly always)
          const int k = run_s[warp][min(lane, len - 1)];
          const float4 c = c_s[k];
          const float dk = km_mid_dist(tb, c);
          dmin = warp_min_nonneg(dk);
          near = c_s[__shfl_sync(0xffffffffu, k, (__ffs(__ballot_sync(0xffffffffu, dk == dmin)) - 1) & 31)];
          keep(lane < len && km_may_win(tb, c, dk, near, dmin), k);
        } else {
          dn = inf;
          kn = 0;
          for (int j = lane; j < len; j += 32) {
            const int k = run_s[warp][j];
            const float dk = km_mid_dist(tb, c_s[k]);
            if (dk < dn) { dn = dk; kn = k; }
          }
          dmin = warp_min_nonneg(dn);
          near = c_s[__shfl_sync(0xffffffffu, kn, (__ffs(__ballot_sync(0xffffffffu, dn == dmin)) - 1) & 31)];
          for (int j0 = 0; j0 < len; j0 += 32) {
            const int k = run_s[warp][min(j0 + lane, len - 1)];
            const float4 c = c_s[k];
            keep(j0 + lane < len && km_may_win(tb, c, km_mid_dist(tb, c), near, dmin), k);
          }
        }
        __syncwarp();
        // the few left, two at a time; an odd last one twice (a tie changes nothing)
        float best0 = inf, best1 = inf;
        int arg0 = 0, arg1 = 0;
        for (int j = 0; j < cnt; j += 2) {
          const unsigned int ks = *reinterpret_cast<const uint16_t*>(&few_s[warp][j]);
          const int ka = ks & 255, kb = j + 1 < cnt ? ks >> 8 : ka;
          float a0, a1, b0, b1;
          const float4 ca = c_s[ka], cb = c_s[kb];
          a0 = km_dist(p0, ca); a1 = km_dist(p1, ca);
          b0 = km_dist(p0, cb); b1 = km_dist(p1, cb);
          if (a0 < best0) { best0 = a0; arg0 = ka; }
          if (a1 < best1) { best1 = a1; arg1 = ka; }
          if (b0 < best0) { best0 = b0; arg0 = kb; }
          if (b1 < best1) { best1 = b1; arg1 = kb; }
        }
        const unsigned int i0 = at + q * KM_TILE, i1 = i0 + 32;
        const bool live0 = i0 < end, live1 = i1 < end;
        const bool ch0 = live0 && (p.it == 0 || arg0 != old0), ch1 = live1 && (p.it == 0 || arg1 != old1);
        if (ch0) p.idx_s[i0] = (uint8_t)arg0;
        if (ch1) p.idx_s[i1] = (uint8_t)arg1;
        if (p.it == 0) {
          book(p0, arg0, ch0);
          book(p1, arg1, ch1);
        } else {
          const unsigned int todo0 = __ballot_sync(0xffffffffu, ch0), todo1 = __ballot_sync(0xffffffffu, ch1);
          auto queue = [&](float4 pt, int k, int old, bool go, unsigned int todo) {
            if (go) {
              const int slot = waiting + __popc(todo & ((1u << lane) - 1u));
              wait_s[warp][slot] = pt;
              sides_s[warp][slot] = (uint16_t)(k | old << 8);
            }
            waiting += __popc(todo);
            if (waiting >= 32) flush(waiting - 32);            // (at most 31 waited before: never more than 63)
          };
          if (todo0) queue(p0, arg0, old0, ch0, todo0);
          if (todo1) queue(p1, arg1, old1, ch1, todo1);
        }
        __syncwarp();
      }
    }
  }
  if (waiting) flush(0);
  __syncthreads();
  for (int i = tid; i < 256 * 4; i += KM_THREADS) {
    const int* a = acc_s + (i >> 2) * 9 + (i & 3);
    const long long v = (long long)a[0] * 32768 + a[4];
    if (v) atomicAdd(reinterpret_cast<unsigned long long*>(&p.h->sums[i]), (unsigned long long)v);
  }
  if (tid < 256) {
    const int c = acc_s[tid * 9 + 8];
    if (c) atomicAdd(&p.h->counts[tid], c);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const int last = atomicAdd(&p.h->ticket, 1) == (int)gridDim.x - 1;
    if (last) { atomicExch(&p.h->ticket, 0); atomicExch(&p.h->next_run, 0u); }
    last_s = last;
  }
  __syncthreads();
  if (!last_s) return;
  // ---- the last CTA: centroids = means of their points (empty clusters stay), largest move ----------
  __threadfence();
  bool settled = true;
  if (tid < 256) {
    const int cnt = __ldcg(&p.h->counts[tid]);
    if (cnt > 0) {
      const float4 c = c_s[tid];
      float nv[4];
      const double unit = (double)cnt * (double)qscale;
#pragma unroll
      for (int j = 0; j < 4; ++j) nv[j] = (float)((double)__ldcg(&p.h->sums[4 * tid + j]) / unit);
      if (tid == 0) {
        const unsigned int odd = __ldcg(&p.h->odd);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const unsigned int o = (odd >> (3 * j)) & 7u;
          if (o) nv[j] = o == 1u ? __int_as_float(0x7f800000) : o == 2u ? neg_inf() : __int_as_float(0x7fffffff);
        }
      }
      p.centroids[tid] = make_float4(nv[0], nv[1], nv[2], nv[3]);
      settled = fabsf(nv[0] - c.x) < 1e-4f && fabsf(nv[1] - c.y) < 1e-4f && fabsf(nv[2] - c.z) < 1e-4f && fabsf(nv[3] - c.w) < 1e-4f;
    }
  }
  const int still = __syncthreads_or(!settled);
  if (tid == 0 && !still && p.it >= 5) p.h->done = 1;
}

}  // namespace shard

using namespace shard;

extern "C" size_t shard_b200_kmeans_workspace_bytes(int32_t count, int64_t n) {
  if (count < 1 || count > 65535 || n < 1 || n >= (1ll << 31)) return 0;
  return km_layout(n).bytes * (size_t)count;
}

extern "C" int shard_b200_kmeans(const float* x, int32_t count, int64_t n, float max_abs, int32_t n_iter, float* centroids,
                                 uint8_t* idx_u8, void* workspace, size_t workspace_bytes, void* stream) {
  if (!x || !centroids || !idx_u8 || !workspace || n_iter < 1 || !(max_abs >= 0.f)) return SHARD_E_ARG;
  const size_t need = shard_b200_kmeans_workspace_bytes(count, n);
  if (need == 0) return SHARD_E_ARG;
  if (workspace_bytes < need) return SHARD_E_WORKSPACE;
  if (((uintptr_t)x | (uintptr_t)centroids | (uintptr_t)workspace) & 15) return SHARD_E_ALIGN;
  const KmeansLayout l = km_layout(n);
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* ws = (unsigned char*)workspace;
  KmeansParams p{};
  p.x = (const float4*)x;
  p.n = n;
  p.centroids = (float4*)centroids;
  p.idx = idx_u8;
  p.h = (KmeansHeader*)ws;
  p.cells = (unsigned int*)(ws + l.cells);
  p.totals = (unsigned int*)(ws + l.totals);
  p.xs = (float4*)(ws + l.xs);
  p.perm = (unsigned int*)(ws + l.perm);
  p.boxes = (float4*)(ws + l.boxes);
  p.idx_s = ws + l.idx;
  p.max_abs = max_abs;
  p.bits = l.bits;
  p.ws_stride = l.bytes;
  // header, counters, totals
  cudaError_t e = cudaMemset2DAsync(ws, l.bytes, 0, l.xs, count, st);
  if (e != cudaSuccess) return (int)e;
  const int wide = capped_blocks((n + 255) / 256, count > 4 ? 2 : 8);
  const dim3 g_wide(wide, count);
  if (max_abs == 0.f) kmeans_max_abs_kernel<<<g_wide, 256, 0, st>>>(p);
  kmeans_sort_kernel<false><<<g_wide, 256, 0, st>>>(p);
  kmeans_scan_kernel<<<dim3(1 << (4 * l.bits - 10), count), 1024, 0, st>>>(p, false);
  kmeans_scan_kernel<<<dim3(1, count), 1024, 0, st>>>(p, true);
  kmeans_sort_kernel<true><<<g_wide, 256, 0, st>>>(p);
  const long long tiles = (n + KM_TILE - 1) / KM_TILE;
  kmeans_boxes_kernel<<<dim3(capped_blocks((tiles + 7) / 8, 8), count), 256, 0, st>>>(p);
  // Longer runs share the test against all centroids (a third of a tile's work at run = 1), shorter
  // ones give every warp of the machine work: the longest that still leaves each two runs.
  const int sms = sm_count() > 0 ? sm_count() : 1;
  p.run = 1;
  while (p.run < KM_MAX_RUN && tiles * count / (2 * p.run) >= (long long)sms * 2 * KM_WARPS * 2) p.run *= 2;
  const long long runs = (tiles + p.run - 1) / p.run;
  p.warp_runs = KM_CTA_POINTS / (KM_WARPS * p.run * KM_TILE);
  // two CTAs per SM over all problems, but never fewer than the runs need at warp_runs each
  long long blocks = (2ll * sms + count - 1) / count;
  const long long most = (runs + KM_WARPS - 1) / KM_WARPS, least = (runs + KM_WARPS * p.warp_runs - 1) / ((long long)KM_WARPS * p.warp_runs);
  if (blocks > most) blocks = most;
  if (blocks < least) blocks = least;
  for (int it = 0; it < n_iter; ++it) {
    p.it = it;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned int)blocks, count);
    cfg.blockDim = dim3(KM_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = it > 0 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kmeans_iteration_kernel, p);
    if (e != cudaSuccess) return (int)e;
  }
  kmeans_unsort_kernel<<<g_wide, 256, 0, st>>>(p);
  SHARD_CHECK_LAUNCH();
  return SHARD_OK;
}
