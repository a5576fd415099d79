// kmeans.cu -- KMeansTransform's GPU work: pairwise distances, exact
// assignment, k-means++ seeding and Lloyd iterations.
//
// Replaces src/transforms/kmeans/distance.jl (pairwise_distances! :28-165,
// assign_clusters! :287-310), init.jl (init_random :22-31,
// init_kmeans_plus_plus :56-128), lloyd.jl (lloyd! :36-134, the M-step
// :149-212) and KMeansTransform.jl fit! (:106-161).
//
// Assignment is the exact arg-min (FP64 order of near-ties, lowest centroid id
// on exact ties) through the exact-search path with k = 1.  The M-step sums
// every cluster's points in point order in FP32 -- a stable counting sort
// groups the points first -- so a fit is deterministic and matches the
// oracle's restatement bit for bit from the same initial centroids.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <vector>

#include "kernels.cuh"

namespace mann {
namespace {

constexpr int PP_CHUNK = 1024;  // k-means++ running-sum block (the oracle uses the same)
constexpr int SORT_CHUNK = 1024;

// ------------------------------------------------------------------ pairwise
// D[i][j] = dist(X[i], C[j]) in the FP32 form's arithmetic (sequential over
// dimensions); 64 x 64 tiles, 256 threads, 4 x 4 per thread.
template <int METRIC>
__global__ void __launch_bounds__(256) pairwise_kernel(const float* __restrict__ X, int64_t n,
                                                       const float* __restrict__ C, int k, int d,
                                                       const float* __restrict__ xn,
                                                       const float* __restrict__ cn,
                                                       float* __restrict__ D) {
  __shared__ float xs[16][65];
  __shared__ float cs[16][65];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t i0 = (int64_t)blockIdx.y * 64;
  const int j0 = blockIdx.x * 64;
  float acc[4][4] = {};
  for (int c0 = 0; c0 < d; c0 += 16) {
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {
      const int r = e >> 4, c = e & 15;
      const int64_t gi = i0 + r;
      const int gj = j0 + r;
      xs[c][r] = (gi < n && c0 + c < d) ? X[gi * d + c0 + c] : 0.0f;
      cs[c][r] = (gj < k && c0 + c < d) ? C[(int64_t)gj * d + c0 + c] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      float xv[4], cv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        xv[u] = xs[c][ty + 16 * u];
        cv[u] = cs[c][tx + 16 * u];
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          if (METRIC == MANN_METRIC_COSINE) {
            acc[a][b] = __fmaf_rn(xv[a], cv[b], acc[a][b]);
          } else {
            const float t = __fsub_rn(xv[a], cv[b]);
            acc[a][b] = __fmaf_rn(t, t, acc[a][b]);
          }
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int64_t gi = i0 + ty + 16 * a;
    if (gi >= n) continue;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int gj = j0 + tx + 16 * b;
      if (gj >= k) continue;
      float v = acc[a][b];
      if (METRIC == MANN_METRIC_EUCLIDEAN) {
        v = __fsqrt_rn(v);
      } else if (METRIC == MANN_METRIC_COSINE) {
        const float den = __fmul_rn(__fsqrt_rn(xn[gi]), __fsqrt_rn(cn[gj]));
        v = __fsub_rn(1.0f, __fdiv_rn(v, den));
        if (v < 0.0f) v = 0.0f;
      }
      D[gi * k + gj] = v;
    }
  }
}

// ------------------------------------------------------------------ gathers
__global__ void gather_rows_kernel(const float* __restrict__ X, int d, const int64_t* __restrict__ idx,
                                   int64_t m, float* __restrict__ out) {
  const int64_t r = blockIdx.x;
  if (r >= m) return;
  const float* src = X + idx[r] * d;
  for (int c = threadIdx.x; c < d; c += blockDim.x) out[r * d + c] = src[c];
}

// ------------------------------------------------------------------ k-means++
// A step draws the next centroid: every point's smallest squared distance to
// the centroids chosen so far is brought up to date with the last one, the
// distances are summed in PP_CHUNK-point blocks and over the blocks, and the
// running sum is searched for u * total -- all sums in FP64, in point order.
//
// One CTA, or four, update a block of points; its last one sums it, and the last
// of all searches the blocks' sums.  What bounds a step is the reading of rows
// (134 MB at 262,144 x 128: 20 us) while most points are open, and a chain of
// loads, barriers and tickets (about 16 us) at all times:
// - in large sets a point whose centroid lies too far from the new one to lose
//   it (pp_reach_kernel) is not read at all, and the rest is staged with three
//   slices of columns in flight;
// - FP64 additions are slow and a chain of them slower still (one thread per
//   1024 additions took 110 us per step, as did the one-thread search), so sums
//   are made in 64-bit integers, in parallel, whenever that is exact: with every
//   term a multiple of 2^L and the total at most 2^53 units, each partial sum is
//   a double, so the ordered FP64 sum rounds nowhere and equals the integer one.
//   Where the terms' range does not allow it, one thread adds in order;
// - a step's kernels start while their predecessor still runs and wait for it
//   where they need it (262,144 x 128: 34.3 -> 29.4 ms for 1,023 steps).
// Measured, all steps, against 128-point CTAs that read every point and start one
// after the other: 262,144 x 128 in 1,024 groups, 1,024 centroids 44 -> 29.5 ms;
// 131,072 x 64 22.6 -> 19.1; 60,000 x 64, 256 centroids 5.1 -> 4.1; 20,000 x 48,
// 128 centroids 2.2 -> 2.0.
constexpr int PP_T = 256;     // threads
constexpr int PP_STAGES = 3;  // slices of rows in flight
// The CTAs of a block of points, the rows they stage at a time and the columns
// of a slice (106 and 109 KB in all, two CTAs per SM).
template <int PARTS>
struct PpShape {
  static constexpr int PTS = PP_CHUNK / PARTS, PER = PTS / PP_T;  // points of a CTA, of a thread
  static constexpr int ROWS = PARTS == 1 ? 128 : 256, DC = PARTS == 1 ? 64 : 32, STR = DC + 4;
  static constexpr int TILE = (ROWS + 1) * STR;  // the last row: the centroid's
};
// coordinates from which leaving points out pays for a second kernel per step:
// it costs 3 us, and 32 MB of rows are read in 5 (60,000 x 64 = 15 MB, 255
// steps: 4.5 ms with it, 4.1 without; 131,072 x 64, 1,023 steps: 19.1 and 24.8;
// 262,144 x 128: 29.4 and 40.3)
constexpr int64_t PP_PRUNE = 1ll << 23;
constexpr long long PP_EXACT = 1ll << 53;
static_assert(PP_CHUNK % (4 * PP_T) == 0 && PP_CHUNK < 32768, "points per thread, indices");

// v = mant * 2^exp2 with an odd mantissa (or 0); false for inf and NaN
__device__ __forceinline__ bool pp_split(double v, long long& mant, int& exp2) {
  const long long bits = __double_as_longlong(v);
  const int e = (int)((bits >> 52) & 0x7FF);
  mant = (bits & 0xFFFFFFFFFFFFFll) | (e ? (1ll << 52) : 0ll);
  exp2 = (e ? e : 1) - 1075;
  if (mant) {
    const int tz = __ffsll(mant) - 1;
    mant >>= tz;
    exp2 += tz;
  }
  return e != 0x7FF && bits >= 0;
}
__device__ __forceinline__ bool pp_split(float v, long long& mant, int& exp2) {
  const int bits = __float_as_int(v), e = (bits >> 23) & 0xFF;  // (bits < 0: refused below)
  int m = (bits & 0x7FFFFF) | (e ? 1 << 23 : 0);
  exp2 = (e ? e : 1) - 150;
  if (m) {
    const int tz = __ffs(m) - 1;
    m >>= tz;
    exp2 += tz;
  }
  mant = m;
  return e != 0xFF && bits >= 0;
}
// 2^e as a double, -1022 <= e <= 1023
__device__ __forceinline__ double pp_pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }

// terms in units of 2^low, or -1 past 2^53
__device__ __forceinline__ long long pp_units(long long mant, int exp2, int low) {
  if (mant == 0) return 0;
  const int sh = exp2 - low;
  if (sh > 52 || mant > (PP_EXACT >> sh)) return -1;
  return mant << sh;
}

__device__ __forceinline__ int pp_block_min(int v, int* red) {
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int w = 1; w < PP_T / 32; ++w) v = min(v, red[w]);
  return v;
}

// exclusive prefix of v over the block; the total in `total`
__device__ __forceinline__ long long pp_block_scan(long long v, long long* red, long long& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const long long x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  __syncthreads();
  if (lane == 31) red[w] = inc;
  __syncthreads();
  long long base = 0;
  total = 0;
  for (int i = 0; i < PP_T / 32; ++i) {
    if (i < w) base += red[i];
    total += red[i];
  }
  return base + inc - v;
}

// The ordered running sum acc, acc + x(0), ... of terms >= 0, each thread
// holding a contiguous run [i0, i1) of them: the total, and the first term of
// the thread's run through which the running sum reaches goal(total) (`at`, or
// -1) with the sum before it (`before`), when every partial sum is exact in
// FP64; false otherwise.
template <typename Term, typename Goal>
__device__ bool pp_exact_sum(double acc, int64_t i0, int64_t i1, Term term, int* redi, long long* redl, double& total,
                             Goal goal, int64_t& at, double& before) {
  constexpr int NO_LOW = 1 << 20;
  int low = NO_LOW;
  bool ok = true;
  auto part = [&](auto v, long long& m, int& e) {
    ok &= pp_split(v, m, e);
    if (m) low = min(low, e);
  };
  long long m;
  int e;
  at = -1;
  part(acc, m, e);
  for (int64_t i = i0; i < i1; ++i) part(term(i), m, e);
  low = pp_block_min(ok ? low : -NO_LOW, redi);
  if (low == -NO_LOW) return false;
  if (low == NO_LOW) low = 0;  // every term is zero
  if (low < -1000) return false;
  pp_split(acc, m, e);
  const long long a0 = pp_units(m, e, low);
  long long mine = 0;
  ok = a0 >= 0;
  for (int64_t i = i0; i < i1 && ok; ++i) {
    pp_split(term(i), m, e);
    const long long u = pp_units(m, e, low);
    mine += u;
    ok = u >= 0 && mine <= PP_EXACT;
  }
  if (!__syncthreads_and(ok)) return false;
  long long sum;
  long long run = a0 + pp_block_scan(mine, redl, sum);
  if (a0 + sum > PP_EXACT) return false;  // at most 257 * 2^53: no overflow
  const double unit = pp_pow2(low);
  total = (double)(a0 + sum) * unit;
  const double g = goal(total);
  if (!((double)(run + mine) * unit >= g)) return true;
  for (int64_t i = i0; i < i1; ++i) {
    pp_split(term(i), m, e);
    const long long next = run + pp_units(m, e, low);
    if ((double)next * unit >= g) {
      at = i;
      before = (double)run * unit;
      break;
    }
    run = next;
  }
  return true;
}

struct PpArgs {
  const float* X;
  int64_t n;
  int d;
  int i;              // the centroid to choose; idx[0 .. i) are chosen
  int vec;            // rows are 16-byte aligned
  const double* u;    // draws
  int64_t* idx;
  float* mind;        // [n]
  double* bsum;       // [blocks]
  unsigned* tickets;  // the step's and the blocks', zero between steps
  int prune;          // leave points out by `reach`
  int* near;          // [n] the centroid mind was measured to (prune)
  float* reach;       // [k] by pp_reach_kernel
};

// reach[m]: a point of centroid m whose squared distance is below it lies at
// least as far from the centroid chosen last.  By the triangle inequality that
// holds below a quarter of the centroids' squared distance; every FP32 sum here
// is within (d + 3) u of the exact one in relative terms (nothing near 1e-30 is
// denormal), which 8 (d + 8) u outweighs, so the point's FP32 distance to the
// new centroid would not be smaller either and mind stays the same, bit by bit.
__global__ void __launch_bounds__(PP_T) pp_reach_kernel(PpArgs a) {
  const int lane = threadIdx.x & 31, m = blockIdx.x * (PP_T / 32) + (threadIdx.x >> 5);
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the step before: its choice
  asm volatile("griddepcontrol.launch_dependents;");
  if (m >= a.i - 1) return;
  const float* x = a.X + a.idx[m] * a.d;
  const float* c = a.X + a.idx[a.i - 1] * a.d;
  float s = 0.0f;
#pragma unroll 4
  for (int e = lane; e < a.d; e += 32) {
    const float v = __fsub_rn(__ldg(x + e), __ldg(c + e));
    s = __fmaf_rn(v, v, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    const float keep = 1.0f - 8.0f * (float)(a.d + 8) * 5.9604644775390625e-08f;
    const float r = __fmul_rd(__fmul_rd(0.25f, keep), s);
    // 0 (no point is below it) where the bound says nothing: overflow, NaN, huge d
    a.reach[m] = keep > 0.5f && r >= 1e-30f && s < __int_as_float(0x7F800000) ? r : 0.0f;
  }
}

// cp.async of n <= ROWS rows' columns [c0, c0 + DC) -- rows who[0 .. n) of the
// points at x0 -- and of the centroid's (row ROWS); columns past d are zero on
// both sides and add nothing.
template <typename S>
__device__ __forceinline__ void pp_stage(float* tile, const float* __restrict__ x0, const float* __restrict__ c,
                                         const short* who, int n, int c0, int d, int vec) {
  const int cw = min(S::DC, d - c0);
  if (vec) {
    constexpr int Q = S::DC / 4;
    for (int e = threadIdx.x; e < (n + 1) * Q; e += PP_T) {
      const int r = e / Q, cc = (e % Q) * 4;
      float* dst = tile + (r < n ? r : S::ROWS) * S::STR + cc;
      const float* src = (r < n ? x0 + (int64_t)who[r] * d : c) + c0 + cc;
      if (cc < cw) {
        const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(src) : "memory");
      } else {
        *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  } else {
    for (int e = threadIdx.x; e < (n + 1) * S::DC; e += PP_T) {
      const int r = e / S::DC, cc = e % S::DC;
      const float* src = (r < n ? x0 + (int64_t)who[r] * d : c) + c0 + cc;
      tile[(r < n ? r : S::ROWS) * S::STR + cc] = cc < cw ? __ldg(src) : 0.0f;
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// PARTS CTAs share a block of points; with several, the last of them sums it.
template <int PARTS>
__global__ void __launch_bounds__(PP_T) pp_step_kernel(PpArgs a) {
  extern __shared__ __align__(16) float pp_smem[];  // [PP_STAGES] tiles
  using S = PpShape<PARTS>;
  __shared__ float own[S::PTS];  // the CTA's points' distances
  __shared__ short who[S::PTS];
  float* vals = PARTS == 1 ? own : pp_smem;  // a block's
  __shared__ int redi[PP_T / 32];
  __shared__ long long redl[PP_T / 32];
  __shared__ int s_last;
  __shared__ long long s_pick;
  __shared__ double s_acc;
  constexpr int PER = S::PER;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int64_t n = a.n;
  const int d = a.d;
  const int64_t nb = (n + PP_CHUNK - 1) / PP_CHUNK;
  const int64_t b0 = (int64_t)blockIdx.x * S::PTS;
  const int len = (int)min((int64_t)S::PTS, n - b0);
  // The next kernel's CTAs may take their places; they wait for this kernel's
  // end.  After a reach kernel this one was launched once every CTA of it had
  // seen the step before complete, so all but `reach` is there already.
  asm volatile("griddepcontrol.launch_dependents;");
  const bool prune = a.prune && a.i > 1;
  if (!prune) asm volatile("griddepcontrol.wait;" ::: "memory");
  const float* c = a.X + __ldcg(a.idx + a.i - 1) * d;

  // the points that the new centroid may be nearer to
  int rows = 0;
  {
    unsigned opens[PER];
    float old[PER];
    int near[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = u * PP_T + t;
      old[u] = __int_as_float(0x7F800000);
      near[u] = 0;
      if (a.i > 1 && e < len) {
        old[u] = __ldcg(a.mind + b0 + e);
        if (prune) near[u] = __ldcg(a.near + b0 + e);
      }
    }
    if (prune) asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int e = u * PP_T + t;
      const bool open = e < len && !(prune && old[u] < a.reach[near[u]]);
      own[e] = old[u];
      opens[u] = __ballot_sync(0xffffffffu, open);
    }
    int mine = 0;
#pragma unroll
    for (int u = 0; u < PER; ++u) mine += __popc(opens[u]);
    if (lane == 0) redi[w] = mine;
    __syncthreads();
    int slot = 0;
    for (int v = 0; v < PP_T / 32; ++v) {
      if (v < w) slot += redi[v];
      rows += redi[v];
    }
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      if (opens[u] >> lane & 1u) who[slot + __popc(opens[u] & ((1u << lane) - 1u))] = (short)(u * PP_T + t);
      slot += __popc(opens[u]);
    }
    __syncthreads();
  }

  // squared distances in the FP32 form (dimension order): groups of ROWS
  // rows, a slice of columns at a time; groups of half the CTA take turns
  const int slices = (d + S::DC - 1) / S::DC, steps = (rows + S::ROWS - 1) / S::ROWS * slices;
  auto stage = [&](int it) {
    if (it < steps) {
      const int g = it / slices * S::ROWS;
      pp_stage<S>(pp_smem + it % PP_STAGES * S::TILE, a.X + b0 * d, c, who + g, min(S::ROWS, rows - g),
               it % slices * S::DC, d, a.vec);
    } else {
      asm volatile("cp.async.commit_group;" ::: "memory");  // the waits count groups
    }
  };
  for (int it = 0; it < PP_STAGES - 1; ++it) stage(it);
  float s = 0.0f;
  for (int it = 0; it < steps; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(PP_STAGES - 2) : "memory");
    __syncthreads();  // slice it has landed for every thread; slice it - 1 is read
    stage(it + PP_STAGES - 1);
    const int g = it / slices, sl = it - g * slices, r = g * S::ROWS + t % S::ROWS;
    if (t / S::ROWS != g % (PP_T / S::ROWS) || r >= rows) continue;
    const float* tile = pp_smem + it % PP_STAGES * S::TILE;
    const float *x = tile + t % S::ROWS * S::STR, *cs = tile + S::ROWS * S::STR;
    const int cw = min(S::DC, d - sl * S::DC);
    if (sl == 0) s = 0.0f;
#pragma unroll 4
    for (int cc = 0; cc < cw; cc += 4) {
      const float4 xv = *reinterpret_cast<const float4*>(x + cc), cv = *reinterpret_cast<const float4*>(cs + cc);
      float v = __fsub_rn(xv.x, cv.x);
      s = __fmaf_rn(v, v, s);
      v = __fsub_rn(xv.y, cv.y);
      s = __fmaf_rn(v, v, s);
      v = __fsub_rn(xv.z, cv.z);
      s = __fmaf_rn(v, v, s);
      v = __fsub_rn(xv.w, cv.w);
      s = __fmaf_rn(v, v, s);
    }
    if (sl == slices - 1) {
      const int e = who[r];
      const float old = own[e];
      if (a.i == 1 || s < old) {
        const float now = s < old ? s : old;
        own[e] = now;
        a.mind[b0 + e] = now;
        if (a.prune) a.near[b0 + e] = a.i - 1;
      }
    }
  }
  __syncthreads();

  // the block's sum
  const int64_t blk = blockIdx.x / PARTS, s0 = blk * PP_CHUNK;
  const int slen = (int)min((int64_t)PP_CHUNK, n - s0);
  if constexpr (PARTS > 1) {
    __threadfence();
    __syncthreads();
    if (t == 0) {
      s_last = atomicAdd(a.tickets + 1 + blk, 1u) + 1u == (unsigned)((slen + S::PTS - 1) / S::PTS);
      if (s_last) a.tickets[1 + blk] = 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int e = t; e < slen; e += PP_T) vals[e] = __ldcg(a.mind + s0 + e);
    __syncthreads();
  }
  constexpr int RUN = PP_CHUNK / PP_T;
  auto value = [&](int64_t e) { return vals[e]; };
  double total = 0.0, before = 0.0;
  int64_t at;
  const double never = __longlong_as_double(0x7FF8000000000000ll);  // a goal that no sum reaches
  if (!pp_exact_sum(0.0, min(slen, t * RUN), min(slen, (t + 1) * RUN), value, redi, redl, total,
                    [&](double) { return never; }, at, before)) {
    total = 0.0;
    if (t == 0)
      for (int e = 0; e < slen; ++e) total += (double)vals[e];
  }
  __threadfence();
  __syncthreads();
  if (t == 0) {
    a.bsum[blk] = total;
    __threadfence();
    s_last = atomicAdd(a.tickets, 1u) + 1u == (unsigned)nb;
    if (s_last) *a.tickets = 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();

  // searchsortedfirst(cumsum(mind), u * total) with the blocked running sums
  if (t == 0) {
    s_pick = nb;
    s_acc = 0.0;
  }
  __syncthreads();
  const int64_t per = (nb + PP_T - 1) / PP_T;
  const double draw = a.u[a.i];
  auto block_sum = [&](int64_t b) { return __ldcg(a.bsum + b); };
  const bool exact = pp_exact_sum(0.0, min(nb, t * per), min(nb, (t + 1) * per), block_sum, redi, redl, total,
                                  [&](double sum) { return draw * sum; }, at, before);
  double thr = draw * total;
  if (exact) {
    if (at >= 0) atomicMin(&s_pick, (long long)at);
    __syncthreads();
    if (at >= 0 && s_pick == at) s_acc = before;
  } else if (t == 0) {
    total = 0.0;
    for (int64_t b = 0; b < nb; ++b) total += __ldcg(a.bsum + b);
    thr = draw * total;
    double acc = 0.0;
    for (int64_t b = 0; b < nb; ++b) {
      if (acc + __ldcg(a.bsum + b) >= thr) {
        s_pick = b;
        break;
      }
      acc += __ldcg(a.bsum + b);
    }
    s_acc = acc;
    redl[0] = __double_as_longlong(thr);
  }
  __syncthreads();
  if (!exact) thr = __longlong_as_double(redl[0]);
  const int64_t pb = s_pick;
  const double acc = s_acc;
  if (pb >= nb) {
    if (t == 0) a.idx[a.i] = n - 1;
    return;
  }
  const int64_t f0 = pb * PP_CHUNK;
  const int flen = (int)min((int64_t)PP_CHUNK, n - f0);
  for (int e = t; e < flen; e += PP_T) vals[e] = __ldcg(a.mind + f0 + e);
  __syncthreads();  // s_pick is read
  if (t == 0) s_pick = n - 1;
  __syncthreads();
  if (pp_exact_sum(acc, min(flen, t * RUN), min(flen, (t + 1) * RUN), value, redi, redl, total,
                   [&](double) { return thr; }, at, before)) {
    if (at >= 0) atomicMin(&s_pick, (long long)(f0 + at));
  } else if (t == 0) {
    double a2 = acc;
    for (int e = 0; e < flen; ++e) {
      a2 += (double)vals[e];
      if (a2 >= thr) {
        s_pick = f0 + e;
        break;
      }
    }
  }
  __syncthreads();
  if (t == 0) a.idx[a.i] = s_pick;
}

// ------------------------------------------------------------------ M-step
// hist[c * nb + b] = points of chunk b assigned to c
__global__ void sort_hist_kernel(const int32_t* __restrict__ assign, int64_t n, int64_t nb,
                                 unsigned* __restrict__ hist) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  atomicAdd(&hist[(int64_t)assign[j] * nb + j / SORT_CHUNK], 1u);
}

// Exclusive scan of m unsigned counts into int64 offsets, SCAN_PER counts per
// block: block totals first, then every block adds up the totals before its
// own and scans its counts (one block walking all k n / 1024 counts took
// 430 us per Lloyd iteration at 262,144 points and 1,024 clusters).
constexpr int SCAN_T = 1024, SCAN_PER = 4 * SCAN_T;
__device__ __forceinline__ int64_t scan_block(int64_t v, int64_t* warp_sum, int64_t& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += x;
  }
  __syncthreads();
  if (lane == 31) warp_sum[w] = inc;
  __syncthreads();
  int64_t base = 0;
  total = 0;
  for (int i = 0; i < SCAN_T / 32; ++i) {
    if (i < w) base += warp_sum[i];
    total += warp_sum[i];
  }
  return base + inc - v;
}
__global__ void __launch_bounds__(SCAN_T) scan_totals_kernel(const unsigned* __restrict__ in, int64_t m,
                                                            int64_t* __restrict__ totals) {
  __shared__ int64_t ws[SCAN_T / 32];
  int64_t s = 0, total;
#pragma unroll
  for (int u = 0; u < SCAN_PER / SCAN_T; ++u) {
    const int64_t i = (int64_t)blockIdx.x * SCAN_PER + u * SCAN_T + threadIdx.x;
    if (i < m) s += in[i];
  }
  scan_block(s, ws, total);
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}
__global__ void __launch_bounds__(SCAN_T) scan_kernel(const unsigned* __restrict__ in, int64_t m,
                                                     const int64_t* __restrict__ totals, int64_t* __restrict__ out) {
  __shared__ int64_t ws[SCAN_T / 32];
  int64_t before = 0, base, total;
  for (int64_t b = threadIdx.x; b < blockIdx.x; b += SCAN_T) before += totals[b];
  scan_block(before, ws, base);
  const int64_t i0 = (int64_t)blockIdx.x * SCAN_PER + (SCAN_PER / SCAN_T) * threadIdx.x;
  unsigned v[SCAN_PER / SCAN_T];
  int64_t s = 0;
#pragma unroll
  for (int u = 0; u < SCAN_PER / SCAN_T; ++u) {
    v[u] = i0 + u < m ? in[i0 + u] : 0u;
    s += v[u];
  }
  int64_t acc = base + scan_block(s, ws, total);
#pragma unroll
  for (int u = 0; u < SCAN_PER / SCAN_T; ++u) {
    if (i0 + u < m) out[i0 + u] = acc;
    acc += v[u];
  }
}

// cluster c's members occupy [start[c], start[c] + count[c])
__global__ void cluster_ranges_kernel(const int64_t* __restrict__ offs, int k, int64_t nb, int64_t n,
                                      int64_t* __restrict__ start, int64_t* __restrict__ count) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= k) return;
  const int64_t s0 = offs[(int64_t)c * nb];
  const int64_t s1 = (c + 1 < k) ? offs[(int64_t)(c + 1) * nb] : n;
  start[c] = s0;
  count[c] = s1 - s0;
}

// stable scatter: one warp per chunk walks its points in order
__global__ void sort_scatter_kernel(const int32_t* __restrict__ assign, int64_t n, int64_t nb,
                                    int64_t* __restrict__ offs, int64_t* __restrict__ members) {
  const int lane = threadIdx.x & 31;
  const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nb) return;
  const int64_t e = min(n, (b + 1) * SORT_CHUNK);
  for (int64_t g = b * SORT_CHUNK; g < e; g += 32) {
    const int64_t j = g + lane;
    const bool valid = j < e;
    const int c = valid ? assign[j] : -1;
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    int64_t* slot = valid ? &offs[(int64_t)c * nb + b] : nullptr;
    const int64_t base = valid ? *slot : 0;
    __syncwarp();
    if (valid) {
      members[base + rank] = j;
      if (rank == 0) *slot = base + __popc(peers);
    }
    __syncwarp();
  }
}

// sums[c][r] = sum over c's members (in point order) of X[m][r], FP32
__global__ void msum_kernel(const float* __restrict__ X, int d, int k,
                            const int64_t* __restrict__ start, const int64_t* __restrict__ count,
                            const int64_t* __restrict__ members, float* __restrict__ sums) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)k * d) return;
  const int c = (int)(t / d), r = (int)(t % d);
  float s = 0.0f;
  const int64_t* mem = members + start[c];
  const int64_t cnt = count[c];
  int64_t m = 0;
  for (; m + 16 <= cnt; m += 16) {  // sixteen rows in flight per thread; the additions keep their order
    float v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = __ldg(X + mem[m + u] * d + r);
#pragma unroll
    for (int u = 0; u < 16; ++u) s = __fadd_rn(s, v[u]);
  }
  for (; m < cnt; ++m) s = __fadd_rn(s, __ldg(X + mem[m] * d + r));
  sums[t] = s;
}

__global__ void mdiv_kernel(const float* __restrict__ sums, const int64_t* __restrict__ count, int d,
                            int k, float* __restrict__ newc) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)k * d) return;
  const int64_t cnt = count[t / d];
  if (cnt > 0) newc[t] = __fdiv_rn(sums[t], (float)cnt);
}

// FP64 distance of every point to its assigned centroid (farthest-point repair)
__global__ void assigned_dist64_kernel(const float* __restrict__ X, int64_t n, int d,
                                       const float* __restrict__ C, const int32_t* __restrict__ assign,
                                       int metric, double* __restrict__ out) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const float* x = X + j * d;
  const float* c = C + (int64_t)assign[j] * d;
  double s = 0.0;
  for (int r = 0; r < d; ++r) {
    const double t = (double)x[r] - (double)c[r];
    s = fma(t, t, s);
  }
  out[j] = metric == MANN_METRIC_EUCLIDEAN ? sqrt(s) : s;
}

// first index of the maximum (single block)
__global__ void argmax_first_kernel(const double* __restrict__ v, int64_t n, int64_t* __restrict__ out) {
  __shared__ double bv[1024];
  __shared__ int64_t bi[1024];
  double best = -INFINITY;
  int64_t bj = 0;
  for (int64_t j = threadIdx.x; j < n; j += blockDim.x)
    if (v[j] > best) {
      best = v[j];
      bj = j;
    }
  bv[threadIdx.x] = best;
  bi[threadIdx.x] = bj;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      const double ov = bv[threadIdx.x + o];
      const int64_t oi = bi[threadIdx.x + o];
      if (ov > bv[threadIdx.x] || (ov == bv[threadIdx.x] && oi < bi[threadIdx.x])) {
        bv[threadIdx.x] = ov;
        bi[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = bi[0];
}

__global__ void repair_kernel(const float* __restrict__ X, int d, const int64_t* __restrict__ far,
                              int c, float* __restrict__ newc, int64_t* __restrict__ count,
                              double* __restrict__ dist) {
  const int64_t f = *far;
  for (int r = threadIdx.x; r < d; r += blockDim.x) newc[(int64_t)c * d + r] = X[f * d + r];
  __syncthreads();
  if (threadIdx.x == 0) {
    count[c] = 1;
    dist[f] = -INFINITY;
  }
}

// Relative bound of an FP32-form Euclidean distance's error: (d + 3) u on the
// square, so half of it and two more roundings on its root.
__device__ __forceinline__ float dist_rel(int d) { return (float)(d + 8) * 5.9604645e-08f; }
// what squares lost to underflow can hide
constexpr float DIST_ABS = 1e-17f;

// per-cluster movement in the fit's metric (FP32 form), max over clusters; and
// upper bounds of the Euclidean movements with their maximum (float bits)
__global__ void movement_kernel(const float* __restrict__ oldc, const float* __restrict__ newc, int k,
                                int d, int metric, double* __restrict__ out_max, float* __restrict__ moved,
                                unsigned* __restrict__ moved_max) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (c < k) {
    float s = 0.0f;
#pragma unroll 16
    for (int r = 0; r < d; ++r) {
      const float t = __fsub_rn(__ldg(oldc + (int64_t)c * d + r), __ldg(newc + (int64_t)c * d + r));
      s = __fmaf_rn(t, t, s);
    }
    m = metric == MANN_METRIC_EUCLIDEAN ? (double)__fsqrt_rn(s) : (double)s;
    const float up = __fadd_ru(__fmul_ru(__fsqrt_ru(s), __fadd_ru(1.0f, dist_rel(d))), DIST_ABS);
    moved[c] = up;
    atomicMax(moved_max, __float_as_uint(up));
  }
  // max over the block, then atomically over blocks (non-negative doubles)
  __shared__ double red[64];
  red[threadIdx.x] = m;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0)
    atomicMax(reinterpret_cast<unsigned long long*>(out_max),
              (unsigned long long)__double_as_longlong(red[0]));
}

// Bounds for Lloyd's assignments: ub[j] >= the distance of point j to its
// centroid, lb[j] <= its distance to every other centroid (true Euclidean
// distances).  While ub stays below lb the assignment cannot change, so only
// the other points are searched again.

// bounds from a search's two nearest centroids; point of result i: rows[i], or i
__global__ void bounds_from_top2_kernel(const int32_t* __restrict__ ids, const float* __restrict__ dists, int64_t m,
                                        const int32_t* __restrict__ rows, int d, int metric,
                                        int32_t* __restrict__ assign, float* __restrict__ ub, float* __restrict__ lb) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const int64_t j = rows ? (int64_t)rows[i] : i;
  float d1 = dists[2 * i], d2 = dists[2 * i + 1];
  if (metric != MANN_METRIC_EUCLIDEAN) {
    d1 = __fsqrt_ru(d1);
    d2 = __fsqrt_rd(d2);
  }
  // a square that overflowed says no more than that the distance is at least
  // the root of the largest float: that centroid may come near
  if (d2 == INFINITY) d2 = __fsqrt_rd(FLT_MAX);
  const float rel = dist_rel(d);
  assign[j] = ids[2 * i];
  ub[j] = __fadd_ru(__fmul_ru(d1, __fadd_ru(1.0f, rel)), DIST_ABS);
  // the two nearest may stand in FP64 order: either may be the FP32 second
  lb[j] = __fsub_rd(__fmul_rd(d2, __fsub_rd(1.0f, 2.0f * rel)), DIST_ABS);
}

// The centroids moved: widen every point's bounds, sharpen ub by the distance
// itself where they meet, and list the points that stay undecided.
__global__ void __launch_bounds__(256)
    bounds_moved_kernel(const float* __restrict__ X, int64_t n, int d, const float* __restrict__ C,
                        const int32_t* __restrict__ assign, const float* __restrict__ moved,
                        const unsigned* __restrict__ moved_max, float* __restrict__ ub, float* __restrict__ lb,
                        int32_t* __restrict__ active, int* __restrict__ n_active) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool open = false;
  if (j < n) {
    const int a = assign[j];
    float u = __fadd_ru(ub[j], moved[a]);
    const float l = __fsub_rd(lb[j], __uint_as_float(*moved_max));
    // a gap of 1e-5 is far past the rounding of the FP64 order of near-ties
    open = !(u < __fmul_rd(l, 0.99999f));
    if (open) {
      const float* x = X + j * d;
      const float* c = C + (int64_t)a * d;
      float s = 0.0f;
#pragma unroll 16
      for (int r = 0; r < d; ++r) {
        const float t = __fsub_rn(__ldg(x + r), __ldg(c + r));
        s = __fmaf_rn(t, t, s);
      }
      u = __fadd_ru(__fmul_ru(__fsqrt_ru(s), __fadd_ru(1.0f, dist_rel(d))), DIST_ABS);
      open = !(u < __fmul_rd(l, 0.99999f));
    }
    ub[j] = u;
    lb[j] = l;
  }
  const unsigned m = __ballot_sync(0xFFFFFFFFu, open);
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0 && m) base = atomicAdd(n_active, __popc(m));
  base = __shfl_sync(0xFFFFFFFFu, base, 0);
  if (open) active[base + __popc(m & ((1u << lane) - 1u))] = (int32_t)j;
}

__global__ void gather_rows32_kernel(const float* __restrict__ X, int d, const int32_t* __restrict__ idx, int64_t m,
                                     float* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m * d) return;
  out[e] = __ldg(X + (int64_t)idx[e / d] * d + e % d);
}

// ------------------------------------------------------------------ RNG
// splitmix64-seeded xoshiro256** (host)
struct Rng {
  uint64_t s[4];
  explicit Rng(uint64_t seed) {
    for (int i = 0; i < 4; ++i) {
      seed += 0x9E3779B97F4A7C15ull;
      uint64_t z = seed;
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
      s[i] = z ^ (z >> 31);
    }
  }
  static uint64_t rotl(uint64_t x, int k) { return (x << k) | (x >> (64 - k)); }
  uint64_t next() {
    const uint64_t r = rotl(s[1] * 5, 7) * 9;
    const uint64_t t = s[1] << 17;
    s[2] ^= s[0];
    s[3] ^= s[1];
    s[1] ^= s[2];
    s[0] ^= s[3];
    s[2] ^= t;
    s[3] = rotl(s[3], 45);
    return r;
  }
  double uniform() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
  uint64_t below(uint64_t m) { return m ? next() % m : 0; }
};

// first m of a seeded Fisher-Yates permutation of 0..n-1
std::vector<int64_t> sample_indices(Rng& rng, int64_t n, int64_t m) {
  std::vector<int64_t> perm(n);
  for (int64_t i = 0; i < n; ++i) perm[i] = i;
  for (int64_t i = 0; i < m; ++i) {
    const int64_t j = i + (int64_t)rng.below((uint64_t)(n - i));
    std::swap(perm[i], perm[j]);
  }
  perm.resize(m);
  return perm;
}

}  // namespace

// ---------------------------------------------------------------- launchers

mann_status pairwise_device(Context* ctx, cudaStream_t s, const float* X, int64_t n, const float* C,
                            int k, int d, int metric, float* D) {
  const float* xn = nullptr;
  const float* cn = nullptr;
  if (metric == MANN_METRIC_COSINE) {
    float *a = nullptr, *b = nullptr;
    MANN_TRY(ctx->scratch_t(SLOT_NORMS_Q, (size_t)n, &a));
    MANN_TRY(ctx->scratch_t(SLOT_NORMS_B, (size_t)k, &b));
    MANN_TRY(launch_row_sqnorm(X, n, d, a, s));
    MANN_TRY(launch_row_sqnorm(C, k, d, b, s));
    xn = a;
    cn = b;
  }
  dim3 grid((unsigned)ceil_div(k, 64), (unsigned)ceil_div(n, 64));
  if (grid.y > 65535) return fail(MANN_EINVAL_ARG, "too many rows for one pairwise call");
  if (metric == MANN_METRIC_EUCLIDEAN)
    pairwise_kernel<MANN_METRIC_EUCLIDEAN><<<grid, 256, 0, s>>>(X, n, C, k, d, xn, cn, D);
  else if (metric == MANN_METRIC_SQEUCLIDEAN)
    pairwise_kernel<MANN_METRIC_SQEUCLIDEAN><<<grid, 256, 0, s>>>(X, n, C, k, d, xn, cn, D);
  else
    pairwise_kernel<MANN_METRIC_COSINE><<<grid, 256, 0, s>>>(X, n, C, k, d, xn, cn, D);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// Exact assignment of n points to k centroids (arg-min, FP64 order of
// near-ties, lowest id on exact ties); dist = FP32-form distance (may be NULL).
mann_status kmeans_assign_device(Context* ctx, cudaStream_t s, const float* X, int64_t n,
                                 const float* C, int k, int d, int metric, int32_t* assign,
                                 float* dist) {
  mann_knn_params p{};
  p.metric = metric;
  p.k = 1;
  p.precision = MANN_PREC_AUTO;
  p.flags = MANN_FLAG_FP64_TIES;
  float* dd = dist;
  if (!dd) MANN_TRY(ctx->scratch_t(SLOT_KM_DIST, (size_t)n, &dd));
  // a point seldom has more than a few centroids within rounding of its
  // nearest, and every list entry costs insertions in each of the n rows: 8
  // entries against 33 take 262,144 x 1,024 x 128 from 5.7 to 2.8 ms (host call
  // 6.5 -> 3.6).  Points whose nearest centroid is repeated 8 to 32 times take
  // both scans: 16.5 -> 19.2 ms with 9 of each, where 33 entries in the former
  // tile kernel took 21.2
  return exact_search_device(ctx, s, &p, C, k, X, n, d, -1, 1, 1, assign, dd, nullptr, 7);
}

mann_status kmeanspp_device(Context* ctx, cudaStream_t s, const float* X, int64_t n, int d, int k,
                            int64_t first, const double* u_host, int64_t* idx_dev) {
  float* mind = nullptr;
  double *bsum = nullptr, *u = nullptr;
  unsigned* tickets = nullptr;
  const int64_t nb = ceil_div(n, PP_CHUNK);
  MANN_TRY(ctx->scratch_t(SLOT_KM_A, (size_t)n * 2 + k, &mind));  // mind, near, reach
  MANN_TRY(ctx->scratch_t(SLOT_KM_B, (size_t)nb * 2 + 1, &bsum));
  tickets = reinterpret_cast<unsigned*>(bsum + nb);
  MANN_TRY(ctx->scratch_t(SLOT_KM_C, (size_t)k, &u));
  MANN_CUDA_TRY(cudaMemcpyAsync(u, u_host, sizeof(double) * k, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(idx_dev, &first, sizeof(int64_t), cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemsetAsync(tickets, 0, sizeof(unsigned) * (nb + 1), s));
  PpArgs a{X, n, d, 0, (d % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0) ? 1 : 0, u, idx_dev, mind, bsum,
           tickets, n * d >= PP_PRUNE ? 1 : 0, reinterpret_cast<int*>(mind + n), mind + 2 * n};
  // four CTAs per block while all of them run at once: one reads its 1,024 rows
  // with the bandwidth of one SM (60,000 x 64, 256 centroids: 6.2 ms with one CTA,
  // 4.1 with four; 131,072 x 64, 1,024: 19.1 and 21.0)
  const int parts = nb * 4 <= ctx->num_sms * 2 ? 4 : 1;
  const auto step = parts == 1 ? pp_step_kernel<1> : pp_step_kernel<4>;
  const int smem = (int)sizeof(float) * PP_STAGES * (parts == 1 ? PpShape<1>::TILE : PpShape<4>::TILE);
  MANN_CUDA_TRY(cudaFuncSetAttribute(step, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  for (a.i = 1; a.i < k; ++a.i) {
    // (a launch with the attribute starts while its predecessor still runs, as
    // far as the kernels' own waits let it)
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(PP_T);
    cfg.stream = s;
    cfg.attrs = &early;
    cfg.numAttrs = a.i > 1 ? 1 : 0;
    if (a.prune && a.i > 1) {
      cfg.gridDim = dim3((unsigned)ceil_div(a.i - 1, PP_T / 32));
      MANN_CUDA_TRY(cudaLaunchKernelEx(&cfg, pp_reach_kernel, a));
      MANN_CHECK_LAUNCH();
    }
    cfg.gridDim = dim3((unsigned)ceil_div(n, PP_CHUNK / parts));
    cfg.dynamicSmemBytes = smem;
    MANN_CUDA_TRY(cudaLaunchKernelEx(&cfg, step, a));
    MANN_CHECK_LAUNCH();
  }
  return MANN_OK;
}

mann_status gather_rows_device(cudaStream_t s, const float* X, int d, const int64_t* idx_dev,
                               int64_t m, float* out) {
  if (m <= 0) return MANN_OK;
  gather_rows_kernel<<<(unsigned)m, 128, 0, s>>>(X, d, idx_dev, m, out);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// The scan's block totals sit behind the offsets.
static size_t offs_len(int k, int64_t nb) { return (size_t)k * nb + (size_t)ceil_div((int64_t)k * nb, SCAN_PER); }

// Stable counting sort of the points by cluster (hist [k][nb], offs [offs_len]).
static mann_status sort_by_cluster(cudaStream_t s, const int32_t* assign, int64_t n, int k, int64_t nb, unsigned* hist,
                                   int64_t* offs, int64_t* start, int64_t* count, int64_t* members) {
  const int64_t m = (int64_t)k * nb;
  int64_t* totals = offs + m;
  MANN_CUDA_TRY(cudaMemsetAsync(hist, 0, sizeof(unsigned) * m, s));
  sort_hist_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(assign, n, nb, hist);
  MANN_CHECK_LAUNCH();
  scan_totals_kernel<<<(unsigned)ceil_div(m, SCAN_PER), SCAN_T, 0, s>>>(hist, m, totals);
  MANN_CHECK_LAUNCH();
  scan_kernel<<<(unsigned)ceil_div(m, SCAN_PER), SCAN_T, 0, s>>>(hist, m, totals, offs);
  MANN_CHECK_LAUNCH();
  cluster_ranges_kernel<<<(unsigned)ceil_div(k, 256), 256, 0, s>>>(offs, k, nb, n, start, count);
  MANN_CHECK_LAUNCH();
  sort_scatter_kernel<<<(unsigned)ceil_div(nb, 4), 128, 0, s>>>(assign, n, nb, offs, members);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// Group points by cluster: cluster c's members (ascending point index) are
// members[start[c] .. start[c] + count[c]).
mann_status group_by_cluster_device(Context* ctx, cudaStream_t s, const int32_t* assign, int64_t n,
                                    int k, int64_t* start, int64_t* count, int64_t* members) {
  const int64_t nb = ceil_div(n, SORT_CHUNK);
  unsigned* hist = nullptr;
  int64_t* offs = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_A, (size_t)k * nb, &hist));
  MANN_TRY(ctx->scratch_t(SLOT_KM_B, offs_len(k, nb), &offs));
  return sort_by_cluster(s, assign, n, k, nb, hist, offs, start, count, members);
}

// State of Lloyd's assignments (bounds above).
struct LloydBounds {
  float *ub = nullptr, *lb = nullptr, *moved = nullptr;
  int32_t* active = nullptr;  // [n]
  int* n_active = nullptr;    // device; behind it the largest movement's bits
  unsigned* moved_max = nullptr;
  int64_t open = -1;          // points to assign anew; -1: all (no bounds yet)
};

// Assigns the open points to their nearest centroids (exactly, as
// kmeans_assign_device) and sets their bounds.
static mann_status assign_open(Context* ctx, cudaStream_t s, const float* X, int64_t n, const float* C, int k, int d,
                               int metric, LloydBounds& lb, int32_t* assign) {
  if (lb.open == 0) return MANN_OK;
  const float* Q = X;
  const int32_t* rows = nullptr;
  int64_t m = n;
  if (lb.open > 0 && lb.open <= n / 2) {  // past half, the whole set costs little more than gathering
    float* g = nullptr;
    m = lb.open;
    rows = lb.active;
    MANN_TRY(ctx->scratch_t(SLOT_KM_GATHER, (size_t)m * d, &g));
    gather_rows32_kernel<<<(unsigned)ceil_div(m * d, 256), 256, 0, s>>>(X, d, rows, m, g);
    MANN_CHECK_LAUNCH();
    Q = g;
  }
  int32_t* ids = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_TOP2, (size_t)4 * m, &ids));
  float* dists = reinterpret_cast<float*>(ids + 2 * m);
  mann_knn_params p{};
  p.metric = metric;
  p.k = 2;
  p.precision = MANN_PREC_AUTO;
  p.flags = MANN_FLAG_FP64_TIES;
  MANN_TRY(exact_search_device(ctx, s, &p, C, k, Q, m, d, -1, std::min(2, k), 2, ids, dists, nullptr, 6));
  bounds_from_top2_kernel<<<(unsigned)ceil_div(m, 256), 256, 0, s>>>(ids, dists, m, rows, d, metric, assign, lb.ub,
                                                                    lb.lb);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// Lloyd from the centroids in C (device, updated in place).  Assignments are
// exact in every iteration; after the first only the points whose bounds do
// not rule out a change are searched (262,144 x 128 points, 1,024 clusters: an
// iteration 3.1 -> 0.5 ms once the centroids settle).
mann_status lloyd_device(Context* ctx, cudaStream_t s, const float* X, int64_t n, int d, int k,
                         float* C, int max_iters, double tol, int metric, int32_t* assign,
                         int* iters_out) {
  const int am = metric == MANN_METRIC_EUCLIDEAN ? MANN_METRIC_EUCLIDEAN : MANN_METRIC_SQEUCLIDEAN;
  const int64_t nb = ceil_div(n, SORT_CHUNK);
  unsigned* hist = nullptr;
  int64_t *offs = nullptr, *start = nullptr, *count = nullptr, *members = nullptr;
  float *sums = nullptr, *newc = nullptr;
  double *dist64 = nullptr, *move = nullptr;
  int64_t* far = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_A, (size_t)k * nb, &hist));
  MANN_TRY(ctx->scratch_t(SLOT_KM_B, offs_len(k, nb), &offs));
  MANN_TRY(ctx->scratch_t(SLOT_KM_C, (size_t)2 * k + 8, &start));
  count = start + k;
  move = reinterpret_cast<double*>(start + 2 * k);
  far = start + 2 * k + 3;
  MANN_TRY(ctx->scratch_t(SLOT_KM_D, (size_t)n, &members));
  MANN_TRY(ctx->scratch_t(SLOT_KM_E, (size_t)2 * k * d, &sums));
  newc = sums + (size_t)k * d;
  LloydBounds lb;
  MANN_TRY(ctx->scratch_t(SLOT_KM_BOUNDS, (size_t)2 * n + k, &lb.ub));
  lb.lb = lb.ub + n;
  lb.moved = lb.lb + n;
  MANN_TRY(ctx->scratch_t(SLOT_KM_ACTIVE, (size_t)n, &lb.active));
  // one 16-byte record for the host: the movement, the open points, the largest movement's bits
  lb.n_active = reinterpret_cast<int*>(move + 1);
  lb.moved_max = reinterpret_cast<unsigned*>(lb.n_active + 1);
  int it = 0;
  for (int step = 1; step <= max_iters; ++step) {
    it = step;
    MANN_TRY(assign_open(ctx, s, X, n, C, k, d, am, lb, assign));
    MANN_TRY(sort_by_cluster(s, assign, n, k, nb, hist, offs, start, count, members));
    msum_kernel<<<(unsigned)ceil_div((int64_t)k * d, 256), 256, 0, s>>>(X, d, k, start, count,
                                                                         members, sums);
    MANN_CHECK_LAUNCH();
    MANN_CUDA_TRY(cudaMemcpyAsync(newc, C, sizeof(float) * k * d, cudaMemcpyDeviceToDevice, s));
    mdiv_kernel<<<(unsigned)ceil_div((int64_t)k * d, 256), 256, 0, s>>>(sums, count, d, k, newc);
    MANN_CHECK_LAUNCH();
    // empty clusters: farthest point (first maximum), marked once taken
    std::vector<int64_t> hcount(k);
    MANN_CUDA_TRY(cudaMemcpyAsync(hcount.data(), count, sizeof(int64_t) * k, cudaMemcpyDeviceToHost, s));
    MANN_CUDA_TRY(cudaStreamSynchronize(s));
    bool any_empty = false;
    for (int c = 0; c < k; ++c) any_empty |= hcount[c] == 0;
    if (any_empty) {
      MANN_TRY(ctx->scratch_t(SLOT_KM_F, (size_t)n, &dist64));
      assigned_dist64_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(X, n, d, C, assign, am, dist64);
      MANN_CHECK_LAUNCH();
      for (int c = 0; c < k; ++c) {
        if (hcount[c] != 0) continue;
        argmax_first_kernel<<<1, 1024, 0, s>>>(dist64, n, far);
        MANN_CHECK_LAUNCH();
        repair_kernel<<<1, 128, 0, s>>>(X, d, far, c, newc, count, dist64);
        MANN_CHECK_LAUNCH();
      }
    }
    MANN_CUDA_TRY(cudaMemsetAsync(move, 0, 2 * sizeof(double), s));
    movement_kernel<<<(unsigned)ceil_div(k, 64), 64, 0, s>>>(C, newc, k, d, am, move, lb.moved, lb.moved_max);
    MANN_CHECK_LAUNCH();
    MANN_CUDA_TRY(cudaMemcpyAsync(C, newc, sizeof(float) * k * d, cudaMemcpyDeviceToDevice, s));
    bounds_moved_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(X, n, d, C, assign, lb.moved, lb.moved_max, lb.ub,
                                                                  lb.lb, lb.active, lb.n_active);
    MANN_CHECK_LAUNCH();
    struct {
      double move;
      int open;
      unsigned moved_max;
    } h{};
    MANN_CUDA_TRY(cudaMemcpyAsync(&h, move, sizeof(h), cudaMemcpyDeviceToHost, s));
    MANN_CUDA_TRY(cudaStreamSynchronize(s));
    lb.open = h.open;
    if (h.move < tol) break;
  }
  MANN_TRY(assign_open(ctx, s, X, n, C, k, d, am, lb, assign));
  if (iters_out) *iters_out = it;
  return MANN_OK;
}

// KMeansTransform.fit! : optional subsample, random or k-means++ seeding,
// Lloyd, then the full assignment when a subsample was used.
mann_status kmeans_fit_device(Context* ctx, cudaStream_t s, const float* X, int64_t n, int d, int k,
                              int metric, int init, int max_iters, double tol, int64_t subsample,
                              uint64_t seed, float* C, int32_t* assign, int* iters_out) {
  if (k <= 0 || k > n)
    return fail(MANN_EINVAL_ARG, "Cannot fit " + std::to_string(k) + " clusters with only " +
                                     std::to_string(n) + " points");
  Rng rng(seed);
  const bool use_sub = subsample > 0 && subsample < n;
  const float* Xt = X;
  int64_t nt = n;
  if (use_sub) {
    nt = std::max<int64_t>(subsample, k);
    std::vector<int64_t> idx = sample_indices(rng, n, nt);
    int64_t* didx = nullptr;
    float* xs = nullptr;
    MANN_TRY(ctx->scratch_t(SLOT_KM_G, (size_t)nt, &didx));
    MANN_TRY(ctx->scratch_t(SLOT_KM_H, (size_t)nt * d, &xs));
    MANN_CUDA_TRY(cudaMemcpyAsync(didx, idx.data(), sizeof(int64_t) * nt, cudaMemcpyHostToDevice, s));
    MANN_TRY(gather_rows_device(s, X, d, didx, nt, xs));
    MANN_CUDA_TRY(cudaStreamSynchronize(s));  // idx (host) must outlive the copy
    Xt = xs;
  }
  int64_t* cidx = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_I, (size_t)k, &cidx));
  if (init == 0) {
    std::vector<int64_t> idx = sample_indices(rng, nt, k);
    MANN_CUDA_TRY(cudaMemcpyAsync(cidx, idx.data(), sizeof(int64_t) * k, cudaMemcpyHostToDevice, s));
    MANN_CUDA_TRY(cudaStreamSynchronize(s));
  } else {
    const int64_t first = (int64_t)rng.below((uint64_t)nt);
    std::vector<double> u(k);
    for (int i = 0; i < k; ++i) u[i] = rng.uniform();
    MANN_TRY(kmeanspp_device(ctx, s, Xt, nt, d, k, first, u.data(), cidx));
    MANN_CUDA_TRY(cudaStreamSynchronize(s));
  }
  MANN_TRY(gather_rows_device(s, Xt, d, cidx, k, C));
  int32_t* atrain = assign;
  if (use_sub) MANN_TRY(ctx->scratch_t(SLOT_KM_J, (size_t)nt, &atrain));
  MANN_TRY(lloyd_device(ctx, s, Xt, nt, d, k, C, max_iters, tol, metric, atrain, iters_out));
  if (use_sub) {
    const int am = metric == MANN_METRIC_EUCLIDEAN ? MANN_METRIC_EUCLIDEAN : MANN_METRIC_SQEUCLIDEAN;
    MANN_TRY(kmeans_assign_device(ctx, s, X, n, C, k, d, am, assign, nullptr));
  }
  return MANN_OK;
}

// ---------------------------------------------------------------- C ABI

namespace {

mann_status check_points(const float* X, int64_t n, int d) {
  if (d <= 0) return fail(MANN_EINVAL_ARG, "Dataset must have at least one dimension");
  if (n <= 0) return fail(MANN_EINVAL_ARG, "Dataset must contain at least one point");
  if (n > 0x7FFFFFFFll) return fail(MANN_EINVAL_ARG, "at most 2^31-1 points (int32 ids)");
  if (!X) return fail(MANN_EINVAL_ARG, "NULL buffer");
  return MANN_OK;
}

bool l2_metric(int m) { return m == MANN_METRIC_EUCLIDEAN || m == MANN_METRIC_SQEUCLIDEAN; }

}  // namespace
}  // namespace mann

using namespace mann;

extern "C" {

mann_status mann_pairwise_distances(const float* X, int64_t n, const float* C, int32_t k, int32_t d,
                                    int32_t metric, float* D) {
  clear_error();
  MANN_TRY(check_points(X, n, d));
  if (k <= 0 || !C || !D) return fail(MANN_EINVAL_ARG, "need k > 0 centroids and an output");
  if (!l2_metric(metric) && metric != MANN_METRIC_COSINE) return fail(MANN_EINVAL_ARG, "unknown metric code");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr, *dd = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_X, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)k * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_OUT_DISTS, (size_t)n * k, &dd));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, X, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dc, C, sizeof(float) * k * d, cudaMemcpyHostToDevice, s));
  MANN_TRY(pairwise_device(ctx, s, dx, n, dc, k, d, metric, dd));
  MANN_CUDA_TRY(cudaMemcpyAsync(D, dd, sizeof(float) * n * k, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  return MANN_OK;
}

mann_status mann_kmeans_assign(const float* X, int64_t n, const float* C, int32_t k, int32_t d,
                               int32_t metric, int32_t* out_assign, float* out_dist) {
  clear_error();
  MANN_TRY(check_points(X, n, d));
  if (k <= 0 || !C || !out_assign) return fail(MANN_EINVAL_ARG, "need k > 0 centroids and an output");
  if (!l2_metric(metric) && metric != MANN_METRIC_COSINE) return fail(MANN_EINVAL_ARG, "unknown metric code");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr, *dd = nullptr;
  int32_t* da = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_X, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)k * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_KM_ASSIGN, (size_t)n, &da));
  MANN_TRY(ctx->scratch_t(SLOT_OUT_DISTS, (size_t)n, &dd));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, X, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dc, C, sizeof(float) * k * d, cudaMemcpyHostToDevice, s));
  MANN_TRY(kmeans_assign_device(ctx, s, dx, n, dc, k, d, metric, da, dd));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_assign, da, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
  if (out_dist) MANN_CUDA_TRY(cudaMemcpyAsync(out_dist, dd, sizeof(float) * n, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  return MANN_OK;
}

mann_status mann_kmeanspp(const float* X, int64_t n, int32_t d, int32_t k, int64_t first,
                          const double* u, int64_t* out_idx) {
  clear_error();
  MANN_TRY(check_points(X, n, d));
  if (k <= 0 || k > n) return fail(MANN_EINVAL_ARG, "Cannot initialize " + std::to_string(k) +
                                                        " clusters with only " + std::to_string(n) + " points");
  if (first < 0 || first >= n || !u || !out_idx) return fail(MANN_EINVAL_ARG, "bad first index or buffers");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float* dx = nullptr;
  int64_t* di = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_X, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_I, (size_t)k, &di));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, X, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  MANN_TRY(kmeanspp_device(ctx, s, dx, n, d, k, first, u, di));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_idx, di, sizeof(int64_t) * k, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  return MANN_OK;
}

mann_status mann_kmeans_lloyd(const float* X, int64_t n, int32_t d, int32_t k, float* centroids,
                              int32_t max_iters, double tol, int32_t metric, int32_t* out_assign,
                              int32_t* out_iters) {
  clear_error();
  MANN_TRY(check_points(X, n, d));
  if (k <= 0 || !centroids || !out_assign) return fail(MANN_EINVAL_ARG, "need k > 0 centroids and outputs");
  if (max_iters <= 0 || !(tol > 0)) return fail(MANN_EINVAL_ARG, "max_iters and tol must be positive");
  if (!l2_metric(metric)) return fail(MANN_EINVAL_ARG, "Lloyd runs on Euclidean / SqEuclidean");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr;
  int32_t* da = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_X, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)k * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_KM_ASSIGN, (size_t)n, &da));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, X, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dc, centroids, sizeof(float) * k * d, cudaMemcpyHostToDevice, s));
  int iters = 0;
  MANN_TRY(lloyd_device(ctx, s, dx, n, d, k, dc, max_iters, tol, metric, da, &iters));
  MANN_CUDA_TRY(cudaMemcpyAsync(centroids, dc, sizeof(float) * k * d, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_assign, da, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  if (out_iters) *out_iters = iters;
  return MANN_OK;
}

mann_status mann_kmeans_fit(const mann_kmeans_params* p, const float* X, int64_t n, int32_t d,
                            float* out_centroids, int32_t* out_assign, int32_t* out_iters) {
  clear_error();
  if (!p) return fail(MANN_EINVAL_ARG, "params must not be NULL");
  MANN_TRY(check_points(X, n, d));
  if (p->k <= 0) return fail(MANN_EINVAL_ARG, "Number of clusters must be positive");
  if (p->init != 0 && p->init != 1) return fail(MANN_EINVAL_ARG, "init must be random (0) or k-means++ (1)");
  if (p->max_iters <= 0 || !(p->tol > 0)) return fail(MANN_EINVAL_ARG, "max_iters and tol must be positive");
  if (p->subsample < 0) return fail(MANN_EINVAL_ARG, "subsample_size must be positive or 0 (none)");
  if (!l2_metric(p->metric)) return fail(MANN_EINVAL_ARG, "KMeans runs on Euclidean / SqEuclidean");
  if (!out_centroids || !out_assign) return fail(MANN_EINVAL_ARG, "NULL buffer");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr;
  int32_t* da = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_KM_X, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)p->k * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_KM_ASSIGN, (size_t)n, &da));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, X, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  int iters = 0;
  MANN_TRY(kmeans_fit_device(ctx, s, dx, n, d, p->k, p->metric, p->init, p->max_iters, p->tol,
                             p->subsample, p->seed, dc, da, &iters));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_centroids, dc, sizeof(float) * p->k * d, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_assign, da, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  if (out_iters) *out_iters = iters;
  return MANN_OK;
}

}  // extern "C"
