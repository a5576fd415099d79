// knn_fp32.cu -- exact FP32 kNN with fused per-row top-k (the plain form).
//
// Replaces the per-query scan of src/indices/bruteforce.jl:59-65 (one
// Distances.jl evaluation per point, then partialsortperm) and the batch loop
// of src/ann_index.jl:91-98.  A CTA owns a block of queries and walks tiles of
// 128 points: it computes the tile's distances in registers (difference form,
// one fused multiply-add per dimension in order 0..d-1 -- bit-identical to the
// oracle's sequential sum) and folds those below a row's k-th best into the
// row's sorted top-k list in shared memory.  The (query block, tile) units are
// shared out evenly over the CTAs; a row's partial lists are merged by a
// second kernel.  Order: (distance, id) as partialsortperm (bruteforce.jl:65).
#include <algorithm>

#include "kernels.cuh"
#include "f32x2.cuh"
#include "warp_list.cuh"

namespace mann {

namespace {

constexpr int K1_THREADS = 256;
constexpr int K1_BN = 128;  // points per tile
constexpr int K1_DK = 16;   // dimensions per shared-memory stage
constexpr uint32_t K1_NAN = 0x7FFFFFFFu;  // every NaN distance in the threshold tests
constexpr int K1_QCAP = 32;  // candidates a row's queue holds
constexpr int K1_DRAIN = 8;  // ... and the number at which it is merged into the row's list
constexpr unsigned FULL = 0xFFFFFFFFu;
using wl::list_get;
using wl::list_insert;
using wl::cmpex;
using wl::merge32;
using wl::sort32;

// Squared row norms as the FP32 form's sequential sum (dimension order, one
// fmaf per term).  One warp per 32 rows: 32 x 32 tiles come in through
// shared memory with coalesced loads (a row's 32 columns per load
// instruction), then lane l adds row l's squares in order; the next tile's
// loads are issued before the current tile's sums.
__global__ void __launch_bounds__(256) row_sqnorm_kernel(const float* __restrict__ x, int64_t n, int d,
                                                         float* __restrict__ out) {
  __shared__ float tile[8][32][33];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t r0 = ((int64_t)blockIdx.x * 8 + w) * 32;
  if (r0 >= n) return;
  const int nr = (int)min((int64_t)32, n - r0);
  float nxt[32];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      nxt[i] = (i < nr && c0 + lane < d) ? __ldg(&x[(r0 + i) * d + c0 + lane]) : 0.0f;
  };
  fetch(0);
  float s = 0.0f;
  for (int c0 = 0; c0 < d; c0 += 32) {
    const int cw = min(32, d - c0);
#pragma unroll
    for (int i = 0; i < 32; ++i) tile[w][i][lane] = nxt[i];
    __syncwarp();
    if (c0 + 32 < d) fetch(c0 + 32);
    if (lane < nr)
      for (int c = 0; c < cw; ++c) s = __fmaf_rn(tile[w][lane][c], tile[w][lane][c], s);
    __syncwarp();
  }
  if (lane < nr) out[r0 + lane] = s;
}

// Thread-tile row/column maps.  TQ rows per thread, 4 or 2: ty*TQ+i.  Eight columns per thread: {tx*4+j, 64+tx*4+j}.
template <int TQ>
__device__ __forceinline__ int tile_row(int ty, int i) {
  return ty * TQ + i;
}
__device__ __forceinline__ int tile_col(int tx, int j) {
  return (j < 4) ? tx * 4 + j : 64 + tx * 4 + (j - 4);
}

template <int TQ>
__device__ __forceinline__ void load_q_frag(const float* p, int ty, float (&v)[TQ]) {
  if constexpr (TQ == 4) {
    float4 a = *reinterpret_cast<const float4*>(p + ty * 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  } else {
    float2 a = *reinterpret_cast<const float2*>(p + ty * 2);
    v[0] = a.x; v[1] = a.y;
  }
}

__device__ __forceinline__ void load_b_frag(const float* p, int tx, float (&v)[8]) {
  float4 a = *reinterpret_cast<const float4*>(p + tx * 4);
  float4 b = *reinterpret_cast<const float4*>(p + 64 + tx * 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// Stage loader: rows [r0, r0+R) x dims [c0, c0+16) of a row-major [*][d]
// matrix into registers (VEC: float4 per thread-slot, else scalars).
template <int R, bool VEC>
struct StageLoader {
  static constexpr int NV = VEC ? (R * 4 + K1_THREADS - 1) / K1_THREADS
                                : (R * 16 + K1_THREADS - 1) / K1_THREADS;
  float4 v4[VEC ? NV : 1];
  float v1[VEC ? 1 : NV];

  __device__ __forceinline__ void load(const float* __restrict__ src, const int32_t* rows,
                                       int64_t r0, int64_t rend, int d, int c0, int tid) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if constexpr (VEC) {
        const int e = tid + i * K1_THREADS;
        float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < R * 4) {
          const int r = e >> 2, c = c0 + (e & 3) * 4;
          const int64_t gr = r0 + r;
          if (gr < rend && c < d) {
            const int64_t row = rows ? (int64_t)rows[gr] : gr;
            val = __ldg(reinterpret_cast<const float4*>(src + row * (int64_t)d + c));
          }
        }
        v4[i] = val;
      } else {
        const int e = tid + i * K1_THREADS;
        float val = 0.f;
        if (e < R * 16) {
          const int r = e >> 4, c = c0 + (e & 15);
          const int64_t gr = r0 + r;
          if (gr < rend && c < d) {
            const int64_t row = rows ? (int64_t)rows[gr] : gr;
            val = __ldg(src + row * (int64_t)d + c);
          }
        }
        v1[i] = val;
      }
    }
  }

  // transpose into dst[dim][row] (row stride `str`)
  __device__ __forceinline__ void store(float* dst, int str, int tid) const {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      if constexpr (VEC) {
        const int e = tid + i * K1_THREADS;
        if (e < R * 4) {
          const int r = e >> 2, c = (e & 3) * 4;
          dst[(c + 0) * str + r] = v4[i].x;
          dst[(c + 1) * str + r] = v4[i].y;
          dst[(c + 2) * str + r] = v4[i].z;
          dst[(c + 3) * str + r] = v4[i].w;
        }
      } else {
        const int e = tid + i * K1_THREADS;
        if (e < R * 16) dst[(e & 15) * str + (e >> 4)] = v1[i];
      }
    }
  }
};

// Shared-memory footprint of one CTA of the tile kernels: the sorted list of
// every row, its queue of admitted candidates and their count, the row's
// threshold (two words for Euclidean), and the two staged slices.
template <int BQ, int KW>
__host__ __device__ constexpr size_t k1_smem_bytes() {
  return sizeof(uint64_t) * BQ * (32 * KW + K1_QCAP) + sizeof(uint32_t) * 4 * BQ +
         sizeof(float) * 2 * K1_DK * ((BQ + 4) + (K1_BN + 4));
}

// CTAs per SM that the tile kernels are compiled for.  The tile phase is
// bound by the FP32 pipe and the fold by latency, so a second and third CTA
// fill the pipe while one folds: three where the lists leave room (k <= 32), else two.
template <int BQ, int KW>
__host__ __device__ constexpr int k1_ctas() {
  return KW == 1 ? 3 : 2;
}

// v[j] for a lane-varying j in [0, N), N a power of two: a select tree on the bits of j
template <int N>
__device__ __forceinline__ float select_tree(const float (&v)[N], int j) {
  float t[N];
#pragma unroll
  for (int i = 0; i < N; ++i) t[i] = v[i];
#pragma unroll
  for (int w = N / 2, bit = 1; w >= 1; w >>= 1, bit <<= 1) {
#pragma unroll
    for (int i = 0; i < w; ++i) t[i] = (j & bit) ? t[2 * i + 1] : t[2 * i];
  }
  return t[0];
}

// The cnt <= 32 queued candidates of a row into its sorted list of 32 KW
// entries.  KW = 1: the candidates are sorted across the lanes (16-wide when
// that holds them) and merged in one bitonic step -- reverse, lane-wise
// minimum, five half-cleaners -- whatever their number; longer lists take
// them one by one.
template <int KW>
__device__ __forceinline__ void k1_drain_row(uint64_t* __restrict__ list, const uint64_t* __restrict__ queue, int cnt,
                                             int k, int lane, uint64_t& kth) {
  uint64_t c = lane < cnt ? queue[lane] : KEY_NONE;
  if constexpr (KW == 1) {
    uint64_t L = list[lane];
#pragma unroll
    for (int w = 2; w <= 16; w <<= 1)
#pragma unroll
      for (int j = w >> 1; j > 0; j >>= 1) c = cmpex(c, j, ((lane & j) == 0) == ((lane & w) == 0));
    if (cnt > 16) {  // the halves are sorted up and down: merge them
#pragma unroll
      for (int j = 16; j > 0; j >>= 1) c = cmpex(c, j, (lane & j) == 0);
    }
    const uint64_t r = __shfl_sync(FULL, (unsigned long long)c, 31 - lane);
    L = r < L ? r : L;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) L = cmpex(L, j, (lane & j) == 0);
    list[lane] = L;
    kth = __shfl_sync(FULL, (unsigned long long)L, k - 1);
  } else {
    uint64_t L[KW];
#pragma unroll
    for (int s = 0; s < KW; ++s) L[s] = list[s * 32 + lane];
    uint64_t thr = list_get<KW>(L, k - 1);
    for (int e = 0; e < cnt; ++e) {
      const uint64_t cnd = __shfl_sync(FULL, (unsigned long long)c, e);
      if (cnd < thr) {
        list_insert<KW>(L, cnd, lane);
        thr = list_get<KW>(L, k - 1);
      }
    }
#pragma unroll
    for (int s = 0; s < KW; ++s) list[s * 32 + lane] = L[s];
    kth = thr;
  }
}

// One CTA's work: queries [q0, min(q0 + BQ, nq)) against points [nb0, nb1);
// the sorted list of query row gq goes to dst + gq * dst_stride.
//
// Tile phase: BQ x 128 distances in registers, TQ x 8 per thread, one sub and
// one fma per dimension and pair, two pairs per f32x2 instruction.  Bound by the
// FP32 pipe and the reads of its operands from shared memory (20,011 x 100: 25 of
// the 33.8 T lane-operations/s of that mix; issue slots 57 % busy, shared memory
// 53 %; per issue 2.1 warps wait for operands, 1.3 for the pipe).  The global loads of the next 16-dimension slice -- of
// the next tile after a tile's last -- are in flight during the current one.
//
// Fold: distances are never staged.  Every distance is compared in its
// register with the row's k-th best so far (as raw bits: distances are not
// negative, and NaN sorts last); the few that pass go to the row's queue in
// shared memory, and the warp that owns the row merges the queue into the
// row's list once it holds K1_DRAIN candidates.  A queue that runs full ends
// the round: its rows are merged, and the candidates left are tested again.
// Points come in ascending id order, so in a tile's first round a distance
// equal to the k-th belongs to a later id and is refused (strict test; the
// threshold holds earlier tiles only); later rounds of the tile admit equals
// and the merge orders them by id.
//
// Measured on one GB300 against the former kernel (128-row tiles, one CTA per
// SM, distances staged in shared memory, one warp-wide insertion per
// candidate, a grid of whole query blocks): 1,000 x 10,000 x 64, k = 10:
// 291 -> 133 us; self graph of 20,011 x 100, k = 15: 7.69 -> 3.23 ms (25 of
// the 40 T lane-operations/s of the FP32 pipe); 10,000 x 60,000 x 784:
// 55.1 -> 31.9 ms (29.5 T); graphs of 24 clouds, 32 dimensions, k = 15:
// 29.4 -> 22.7 ms (26 T).
template <int METRIC, int BQ, int KW, bool VEC>
__device__ __forceinline__ void k1_body(const float* __restrict__ base, int64_t nb0, int64_t nb1,
                                        const float* __restrict__ qs, const int32_t* __restrict__ qrows,
                                        int64_t q0, int64_t nq, int d, const float* __restrict__ qnorm,
                                        const float* __restrict__ bnorm, int k, uint64_t* __restrict__ dst0,
                                        int64_t dst_stride, uint64_t* smem) {
  constexpr int TQ = BQ / 16;
  constexpr int TN = 8;
  constexpr int RPW = BQ / 8;
  constexpr int QSTR = BQ + 4;
  constexpr int BSTR = K1_BN + 4;
  constexpr uint32_t ALL = 0xFFFFFFFFu;
  uint64_t* lists = smem;                                        // [BQ][32 KW]
  uint64_t* queues = lists + BQ * 32 * KW;                       // [BQ][QCAP]
  float* Qs = reinterpret_cast<float*>(queues + BQ * K1_QCAP);   // [2][DK][QSTR]
  float* Bs = Qs + 2 * K1_DK * QSTR;                             // [2][DK][BSTR]
  uint32_t* thr = reinterpret_cast<uint32_t*>(Bs + 2 * K1_DK * BSTR);  // [BQ] bits of the k-th distance (ALL: none)
  uint32_t* thr_sq = thr + BQ;                                   // [BQ] Euclidean: bits no passing square exceeds
  int* qcnt = reinterpret_cast<int*>(thr_sq + BQ);               // [BQ]

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = tid >> 4, tx = tid & 15;
  const int nchunks = (d + K1_DK - 1) / K1_DK;

  for (int e = tid; e < BQ * 32 * KW; e += K1_THREADS) lists[e] = KEY_NONE;
  for (int e = tid; e < BQ; e += K1_THREADS) {
    thr[e] = ALL;
    thr_sq[e] = ALL;
    qcnt[e] = 0;
  }

  StageLoader<BQ, VEC> qload;
  StageLoader<K1_BN, VEC> bload;
  qload.load(qs, qrows, q0, nq, d, 0, tid);
  bload.load(base, nullptr, nb0, min(nb1, nb0 + K1_BN), d, 0, tid);
  qload.store(Qs, QSTR, tid);
  bload.store(Bs, BSTR, tid);
  __syncthreads();
  int buf = 0;

  for (int64_t t0 = nb0; t0 < nb1; t0 += K1_BN) {
    const int64_t tend = min(nb1, t0 + K1_BN);
    // accumulators of columns 2j, 2j+1 packed in one f32x2 pair
    uint64_t acc2[TQ][TN / 2];
#pragma unroll
    for (int i = 0; i < TQ; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) acc2[i][j] = 0ull;

    for (int c = 0; c < nchunks; ++c) {
      const bool last = c + 1 == nchunks;
      const bool more = !last || tend < nb1;
      if (more) {
        const int64_t tn = last ? tend : t0;
        const int c0 = last ? 0 : (c + 1) * K1_DK;
        qload.load(qs, qrows, q0, nq, d, c0, tid);
        bload.load(base, nullptr, tn, min(nb1, tn + K1_BN), d, c0, tid);
      }
      const float* qsb = Qs + buf * K1_DK * QSTR;
      const float* bsb = Bs + buf * K1_DK * BSTR;
      const int kend = min(K1_DK, d - c * K1_DK);  // dimensions past d hold zeros on both sides
#pragma unroll
      for (int k4 = 0; k4 < K1_DK; k4 += 4) {
        if (k4 >= kend) break;
#pragma unroll
        for (int kk = k4; kk < k4 + 4; ++kk) {
          float qv[TQ], bv[TN];
          load_q_frag<TQ>(qsb + kk * QSTR, ty, qv);
          load_b_frag(bsb + kk * BSTR, tx, bv);
          uint64_t b2[TN / 2];
#pragma unroll
          for (int j = 0; j < TN / 2; ++j) b2[j] = f2::pack(bv[2 * j], bv[2 * j + 1]);
#pragma unroll
          for (int i = 0; i < TQ; ++i) {
            const uint64_t q2 = f2::pack(qv[i], qv[i]);
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) {
              if constexpr (METRIC == MANN_METRIC_COSINE) {
                acc2[i][j] = f2::fma(q2, b2[j], acc2[i][j]);
              } else {
                const uint64_t t = f2::sub(q2, b2[j]);
                acc2[i][j] = f2::fma(t, t, acc2[i][j]);
              }
            }
          }
        }
      }
      if (more) {
        qload.store(Qs + (buf ^ 1) * K1_DK * QSTR, QSTR, tid);
        bload.store(Bs + (buf ^ 1) * K1_DK * BSTR, BSTR, tid);
      }
      __syncthreads();
      buf ^= 1;
    }

    float acc[TQ * TN];  // element i * 8 + j: row tile_row(ty, i), column tile_col(tx, j)
#pragma unroll
    for (int i = 0; i < TQ; ++i)
#pragma unroll
      for (int j = 0; j < TN / 2; ++j) f2::unpack(acc2[i][j], acc[i * TN + 2 * j], acc[i * TN + 2 * j + 1]);
    if constexpr (METRIC == MANN_METRIC_COSINE) {
#pragma unroll
      for (int i = 0; i < TQ; ++i) {
        const int64_t gq = q0 + tile_row<TQ>(ty, i);
        const float qn = (gq < nq) ? qnorm[qrows ? qrows[gq] : gq] : 1.0f;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          const int64_t gb = t0 + tile_col(tx, j);
          const float bn = (gb < tend) ? bnorm[gb] : 1.0f;
          const float den = __fmul_rn(__fsqrt_rn(qn), __fsqrt_rn(bn));
          float v = __fsub_rn(1.0f, __fdiv_rn(acc[i * TN + j], den));
          if (v < 0.0f) v = 0.0f;
          acc[i * TN + j] = v;
        }
      }
    }
    // candidates of this thread: one bit per element
    const bool partial_tile = tend - t0 < K1_BN;
    uint32_t pend = 0;
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
      const int r = tile_row<TQ>(ty, i);
      const uint32_t lim = METRIC == MANN_METRIC_EUCLIDEAN ? thr_sq[r] : thr[r];
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < TN; ++j) m |= (__float_as_uint(acc[i * TN + j]) < lim ? 1u : 0u) << j;
      if (q0 + r >= nq) m = 0;
      pend |= m << (i * TN);
    }
    if (partial_tile) {
      uint32_t cm = 0;
#pragma unroll
      for (int j = 0; j < TN; ++j) cm |= (t0 + tile_col(tx, j) < tend ? 1u : 0u) << j;
#pragma unroll
      for (int i = 1; i < TQ; ++i) cm |= (cm & 0xFFu) << (i * TN);
      pend &= cm;
    }
    for (bool first = true;; first = false) {
      uint32_t todo = pend;
      while (todo) {
        const int e = __ffs(todo) - 1;
        todo &= todo - 1;
        const int r = tile_row<TQ>(ty, e >> 3);
        float v = select_tree<TQ * TN>(acc, e);
        if constexpr (METRIC == MANN_METRIC_EUCLIDEAN) v = __fsqrt_rn(v);
        const uint32_t lim = thr[r], vb = v == v ? __float_as_uint(v) : K1_NAN;
        if (first ? vb < lim : vb <= lim) {
          const int pos = atomicAdd(&qcnt[r], 1);
          if (pos >= K1_QCAP) continue;  // full: tested again in the next round
          queues[r * K1_QCAP + pos] = make_key(v, (uint32_t)(t0 + tile_col(tx, e & 7)));
        }
        pend &= ~(1u << e);
      }
      const bool again = __syncthreads_or(pend != 0);
      // merge the queues of this warp's rows: all that hold K1_DRAIN
      // candidates, and in the last round of the last tile every one
      const int least = tend < nb1 || again ? K1_DRAIN : 1;
      for (int r = warp * RPW; r < warp * RPW + RPW; ++r) {
        const int cnt = min(qcnt[r], K1_QCAP);
        if (cnt < least) continue;  // warp-uniform
        uint64_t kth;
        k1_drain_row<KW>(lists + r * 32 * KW, queues + r * K1_QCAP, cnt, k, lane, kth);
        __syncwarp();
        if (lane == 0) {
          qcnt[r] = 0;
          if (kth != KEY_NONE) {
            const float t = key_dist(kth);
            thr[r] = t == t ? __float_as_uint(t) : K1_NAN;
            // sqrt(v) < t needs v < t^2 (1 + 2^-21): a square at or past that
            // bound has a larger root however both round
            if constexpr (METRIC == MANN_METRIC_EUCLIDEAN)
              thr_sq[r] = __float_as_uint(__fadd_ru(__fmul_ru(__fmul_ru(t, t), 1.0000005f), 1e-44f));
          }
        }
      }
      if (!again) break;
      __syncthreads();
    }
  }
  // write this split's lists (each warp its own rows)
  for (int r = warp * RPW; r < warp * RPW + RPW; ++r) {
    const int64_t gq = q0 + r;
    if (gq >= nq) break;
    uint64_t* dst = dst0 + gq * dst_stride;
    for (int e = lane; e < k; e += 32) dst[e] = lists[r * 32 * KW + e];
  }
}

// How the tile kernel's CTAs share the (query block, point tile) units.
// Unit u is tile u % tiles of query block u / tiles.
//   splits == 0: CTA c takes units [c per, (c + 1) per) -- an equal share of
//     the whole work, whatever the block and tile counts.  Going from unit to
//     unit either the CTA or the query block (or both) moves on, so CTA c's
//     list of query row q is row q + c BQ of `partial`: one list per row and BQ
//     more per CTA.  (A place in every row for each CTA that may meet its block
//     was two lists per row: 100,000 rows, k = 128, 201 MB and now 122.  The
//     search takes as long either way: 20,011 x 20,011 x 100, k = 15, 3,188 and
//     3,120 us; 10,000 x 60,000 x 256, k = 10, 10.76 and 10.73 ms; 100,000 x
//     3,000 x 8, k = 128, 10.06 and 9.99 ms.)
//   splits > 0: CTA c takes split c % splits (tiles_per tiles) of query block
//     c / splits; its list of row q is list c % splits of the row's `slots`.
struct K1Walk {
  int64_t total, per;
  int tiles, splits, tiles_per;
  int slots;  // lists per query row (splits == 0: at most)
  int step;      // lists from a CTA's first to the next one's (splits == 0; 0: one list per row)
  int stride;    // ... from a row's first to the next row's
  int64_t rows;  // lists in all
};

template <int METRIC, int BQ, int KW, bool VEC>
__global__ void __launch_bounds__(K1_THREADS, k1_ctas<BQ, KW>())
    k1_tile_topk(const float* __restrict__ base, int64_t n, const float* __restrict__ qs,
                 const int32_t* __restrict__ qrows, int64_t nq, int d,
                 const float* __restrict__ qnorm, const float* __restrict__ bnorm, int k, K1Walk w,
                 uint64_t* __restrict__ partial) {
  extern __shared__ __align__(16) uint64_t k1_smem[];
  int64_t u = (int64_t)blockIdx.x * w.per, uend = min(w.total, u + w.per);
  if (w.splits > 0) {
    const int64_t qb = blockIdx.x / w.splits;
    const int t0 = (int)(blockIdx.x % w.splits) * w.tiles_per;
    u = qb * w.tiles + t0;
    uend = qb * w.tiles + min(w.tiles, t0 + w.tiles_per);
  }
  while (u < uend) {
    const int64_t qb = u / w.tiles;
    const int t0 = (int)(u - qb * w.tiles);
    const int t1 = (int)min((int64_t)w.tiles, t0 + (uend - u));
    // (the CTA as the unit's: with blockIdx.x here the compiler schedules the tile
    // phase differently, 10.73 -> 10.92 ms at 10,000 x 60,000 x 256)
    const int first = w.splits > 0 ? (int)(blockIdx.x % w.splits) : (int)(u / w.per) * w.step;
    k1_body<METRIC, BQ, KW, VEC>(base, (int64_t)t0 * K1_BN, min(n, (int64_t)t1 * K1_BN), qs, qrows, qb * BQ, nq, d,
                                 qnorm, bnorm, k, partial + (int64_t)first * k, (int64_t)w.stride * k, k1_smem);
    u += t1 - t0;
    __syncthreads();  // the next block's set-up overwrites the lists
  }
}

// Segmented persistent form over a device work queue: the work items of many
// independent point sets stored back to back -- item i covers queries
// [q0, qend) of one set against that set's points [nb0, nb1) (global rows,
// so the keys carry global ids) and writes split slot `split` of each
// query's lists.  A grid of resident CTAs takes the items (largest first) from the queue
// by an atomic counter until the queue is exhausted.  Before taking work a
// CTA waits until the queue of this call is published (q->epoch == epoch,
// written with the plan ahead of the kernel in stream order); the wait is
// bounded by `wait_cycles`, after which the CTA records MANN_ETIMEOUT in
// q->status and returns without touching any list.  `qrows` is null; with the
// constant in its place the compiler spills in the inner loop (338,792 rows x 32:
// 22.7 -> 23.6 ms).
template <int METRIC, int BQ, int KW, bool VEC>
__global__ void __launch_bounds__(K1_THREADS, k1_ctas<BQ, KW>())
    k1_persistent(const float* __restrict__ data, const SegItem* __restrict__ items, SegQueue* q, unsigned epoch,
                  long long wait_cycles, int d, int k, int nsplit, uint64_t* __restrict__ partial,
                  const int32_t* __restrict__ qrows) {
  extern __shared__ __align__(16) uint64_t k1_smem[];
  __shared__ int s_item;
  __shared__ int s_count;
  if (threadIdx.x == 0) {
    volatile SegQueue* vq = q;
    const long long t0 = clock64();
    int ok = 1;
    while (vq->epoch != epoch) {
      if (clock64() - t0 > wait_cycles) {
        atomicCAS(&q->status, 0, (int)MANN_ETIMEOUT);
        ok = 0;
        break;
      }
      __nanosleep(64);
    }
    __threadfence();
    s_count = ok ? vq->count : 0;
  }
  __syncthreads();
  const int count = s_count;
  for (;;) {
    if (threadIdx.x == 0) {
      const unsigned long long i = atomicAdd(&q->head, 1ull);
      s_item = i < (unsigned long long)count ? (int)i : -1;
    }
    __syncthreads();
    const int idx = s_item;
    if (idx < 0) break;
    const SegItem it = items[idx];
    k1_body<METRIC, BQ, KW, VEC>(data, it.nb0, it.nb1, data, qrows, it.q0, it.qend, d, nullptr, nullptr, k,
                                 partial + (int64_t)it.split * k, (int64_t)nsplit * k, k1_smem);
    __syncthreads();  // s_item is rewritten only after every thread read it
  }
}

// Exact FP32 scan for a handful of query rows (nq <= 32, e.g. the rows the
// BF16 form could not certify): one point per thread, blocks striding over
// 256-point chunks, every distance the FP32 form's sequential sum in
// dimension order (queries staged 32 dimensions at a time in shared memory,
// the point's slice in registers); warp w keeps the lists of rows w, w+8,
// w+16, w+24; one list per (row, block), merged afterwards.
constexpr int FEW_Q = 32;
constexpr int FEW_T = 256;
constexpr int FEW_DC = 32;
// up to FEW_QS rows with d <= FEW_STAGED_D: the rows are staged whole in shared
// memory once, and each thread streams its point with no barrier per chunk
constexpr int FEW_QS = 4;
constexpr int FEW_STAGED_D = 2048;

// the FP32 form's distance from the sequential sum `acc` (row qrow, point pi)
template <int METRIC>
__device__ __forceinline__ float few_distance(float acc, const float* __restrict__ qnorm, int64_t qrow,
                                              const float* __restrict__ bnorm, int64_t pi, bool valid) {
  float v = acc;
  if constexpr (METRIC == MANN_METRIC_EUCLIDEAN) {
    v = __fsqrt_rn(v);
  } else if constexpr (METRIC == MANN_METRIC_COSINE) {
    const float qnv = qnorm[qrow];
    const float bnv = valid ? bnorm[pi] : 1.0f;
    const float den = __fmul_rn(__fsqrt_rn(qnv), __fsqrt_rn(bnv));
    v = __fsub_rn(1.0f, __fdiv_rn(v, den));
    if (v < 0.0f) v = 0.0f;
  }
  return v;
}

// the block's distances dsm[j][0, np) (points p0 ...) into the lists of rows
// j = warp + 8 m, held by that warp
template <int KW, int M>
__device__ __forceinline__ void few_fold(const float (*dsm)[FEW_T + 1], uint64_t (&L)[M][KW], int nq, int warp,
                                         int lane, int64_t p0, int np, int k) {
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int j = warp + 8 * m;
    if (j >= nq) continue;  // warp-uniform
    uint64_t thr = list_get<KW>(L[m], k - 1);
    for (int c8 = 0; c8 < FEW_T; c8 += 32) {
      const int col = c8 + lane;
      const uint64_t key = col < np ? make_key(dsm[j][col], (uint32_t)(p0 + col)) : KEY_NONE;
      unsigned pend = __ballot_sync(FULL, key < thr);
      while (pend) {
        const int src = __ffs(pend) - 1;
        pend &= pend - 1;
        const uint64_t cnd = __shfl_sync(FULL, key, src);
        if (cnd < thr) {
          list_insert<KW>(L[m], cnd, lane);
          thr = list_get<KW>(L[m], k - 1);
        }
      }
    }
  }
}

template <int METRIC, int KW, bool VEC>
__global__ void __launch_bounds__(FEW_T, 2)
    few_rows_kernel(const float* __restrict__ base, int64_t n, const float* __restrict__ qs,
                    const int32_t* __restrict__ qrows, int nq, int d, const float* __restrict__ qnorm,
                    const float* __restrict__ bnorm, int k, uint64_t* __restrict__ partial) {
  __shared__ __align__(16) float qsm[FEW_Q][FEW_DC];
  __shared__ float dsm[FEW_Q][FEW_T + 1];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint64_t L[4][KW];
#pragma unroll
  for (int m = 0; m < 4; ++m)
#pragma unroll
    for (int s = 0; s < KW; ++s) L[m][s] = KEY_NONE;
  for (int64_t p0 = (int64_t)blockIdx.x * FEW_T; p0 < n; p0 += (int64_t)gridDim.x * FEW_T) {
    const int64_t pi = p0 + t;
    const bool valid = pi < n;
    const float* prow = base + (valid ? pi : 0) * d;
    float acc[FEW_Q];
#pragma unroll
    for (int j = 0; j < FEW_Q; ++j) acc[j] = 0.0f;
    for (int c0 = 0; c0 < d; c0 += FEW_DC) {
      const int dc = min(FEW_DC, d - c0);
      __syncthreads();
      for (int e = t; e < FEW_Q * FEW_DC; e += FEW_T) {
        const int r = e / FEW_DC, c = e % FEW_DC;
        float v = 0.0f;
        if (r < nq && c < dc) v = __ldg(&qs[(int64_t)(qrows ? qrows[r] : r) * d + c0 + c]);
        qsm[r][c] = v;
      }
      float pv[FEW_DC];
      if (VEC && dc == FEW_DC) {
#pragma unroll
        for (int c = 0; c < FEW_DC; c += 4) {
          const float4 v = valid ? __ldg(reinterpret_cast<const float4*>(prow + c0 + c)) : make_float4(0, 0, 0, 0);
          pv[c] = v.x;
          pv[c + 1] = v.y;
          pv[c + 2] = v.z;
          pv[c + 3] = v.w;
        }
      } else {
#pragma unroll
        for (int c = 0; c < FEW_DC; ++c) pv[c] = (valid && c < dc) ? __ldg(prow + c0 + c) : 0.0f;
      }
      __syncthreads();
      // dimensions past d are zero on both sides and add nothing
#pragma unroll
      for (int j = 0; j < FEW_Q; ++j) {
        if (j < nq) {
          float a = acc[j];
#pragma unroll
          for (int c = 0; c < FEW_DC; c += 4) {
            const float4 q4 = *reinterpret_cast<const float4*>(&qsm[j][c]);
            if constexpr (METRIC == MANN_METRIC_COSINE) {
              a = __fmaf_rn(q4.x, pv[c], a);
              a = __fmaf_rn(q4.y, pv[c + 1], a);
              a = __fmaf_rn(q4.z, pv[c + 2], a);
              a = __fmaf_rn(q4.w, pv[c + 3], a);
            } else {
              float u = __fsub_rn(q4.x, pv[c]);
              a = __fmaf_rn(u, u, a);
              u = __fsub_rn(q4.y, pv[c + 1]);
              a = __fmaf_rn(u, u, a);
              u = __fsub_rn(q4.z, pv[c + 2]);
              a = __fmaf_rn(u, u, a);
              u = __fsub_rn(q4.w, pv[c + 3]);
              a = __fmaf_rn(u, u, a);
            }
          }
          acc[j] = a;
        }
      }
    }
#pragma unroll
    for (int j = 0; j < FEW_Q; ++j)
      if (j < nq) dsm[j][t] = few_distance<METRIC>(acc[j], qnorm, qrows ? qrows[j] : j, bnorm, pi, valid);
    __syncthreads();
    few_fold<KW, 4>(dsm, L, nq, warp, lane, p0, (int)min((int64_t)FEW_T, n - p0), k);
  }
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int j = warp + 8 * m;
    if (j >= nq) continue;
    uint64_t* dst = partial + ((int64_t)j * gridDim.x + blockIdx.x) * k;
#pragma unroll
    for (int s = 0; s < KW; ++s) {
      const int e = s * 32 + lane;
      if (e < k) dst[e] = L[m][s];
    }
  }
}

// Where a search's results go: its keys, or -- with ids set -- the ids and
// distances of its rows (launch_finish's rules, row i to output row i).
struct FewOut {
  uint64_t* keys;  // [nq][k]
  int32_t* ids;    // [nq][kout]
  float* dists;
  int kout;
  int64_t graph_self;
};

// The last of the sets starting at offs[0 .. nsets) that starts at or before the
// row: 32 candidates a step.
__device__ __forceinline__ int set_of(const int64_t* __restrict__ offs, int nsets, int64_t row, int lane) {
  int lo = 0;
  for (int len = nsets; len > 1;) {
    const int st = (len + 31) / 32, p = lane * st;
    const unsigned le = __ballot_sync(FULL, p < len && offs[lo + p] <= row);
    const int hit = (31 - __clz(le)) * st;  // lane 0's always is
    lo += hit;
    len = min(st, len - hit);
  }
  return lo;
}

// One row's sorted keys (lane e: entry e, k <= 32 of them) as ids, counted from
// `first`, and distances.
__device__ __forceinline__ void finish_row32(const FewOut& o, int64_t q, uint64_t key, int k, int lane,
                                             int32_t first = 0) {
  const bool keep = lane < k && key != KEY_NONE && !(o.graph_self >= 0 && (int64_t)key_id(key) == o.graph_self + q);
  const unsigned have = __ballot_sync(FULL, keep);
  const int pos = __popc(have & ((1u << lane) - 1u));
  if (keep && pos < o.kout) {
    o.ids[q * o.kout + pos] = (int32_t)key_id(key) - first;
    o.dists[q * o.kout + pos] = key_dist(key);
  }
  for (int e = __popc(have) + lane; e < o.kout; e += 32) {
    o.ids[q * o.kout + e] = -1;
    o.dists[q * o.kout + e] = __int_as_float(0x7F800000);
  }
}

// four more terms of a sum, in dimension order
template <int METRIC>
__device__ __forceinline__ void few_add(float& a, const float4& q4, const float4& v) {
  if constexpr (METRIC == MANN_METRIC_COSINE) {
    a = __fmaf_rn(q4.x, v.x, a);
    a = __fmaf_rn(q4.y, v.y, a);
    a = __fmaf_rn(q4.z, v.z, a);
    a = __fmaf_rn(q4.w, v.w, a);
  } else {
    float u = __fsub_rn(q4.x, v.x);
    a = __fmaf_rn(u, u, a);
    u = __fsub_rn(q4.y, v.y);
    a = __fmaf_rn(u, u, a);
    u = __fsub_rn(q4.z, v.z);
    a = __fmaf_rn(u, u, a);
    u = __fsub_rn(q4.w, v.w);
    a = __fmaf_rn(u, u, a);
  }
}

// few_rows_kernel for nq <= FEW_QS rows of d <= FEW_STAGED_D: the rows sit in
// shared memory ([FEW_QS][d], staged once), and no barrier falls between a
// point's columns (the chunked form waits for its loads 25 times per point at
// d = 784); the same sequential sums in dimension order.  Every warp keeps its
// own list of every row -- 32 new distances are sorted and merged at once when
// many of them count, so no warp waits for another's insertions -- and a block
// merges its warps' lists at the end.
//
// With a ticket (lists of at most 32) the last block to finish merges all the
// blocks' lists and writes the results: a single query is one launch instead
// of three (1 x 10,000 x 64: 22 us of kernels with two gaps, now 11).
//
// VEC (d a multiple of 4, 16-byte rows): the points come in through shared
// memory, 32 columns of a warp's 32 rows at a time with eight lanes to a row and
// the next slice in flight.  A thread that reads its own row touches 32 lines
// per load, and the line lookups bound it: one row against 290,000 x 256 points
// (297 MB, 44 us at the copy rate) took 98 us, now 78 from a cold cache; four
// rows 145, now 109; 60,000 x 784 70, now 61; 10,000 x 64 14.3, now 12.3.
constexpr int FEW_SD = 32, FEW_SS = FEW_SD + 4;  // columns of a slice, their stride
constexpr size_t FEW_SLICE_BYTES = sizeof(float) * 2 * (FEW_T / 32) * 32 * FEW_SS;
template <int METRIC, int KW, bool VEC>
__global__ void __launch_bounds__(FEW_T, 2)
    few_rows_staged_kernel(const float* __restrict__ base, int64_t n, const float* __restrict__ qs,
                           const int32_t* __restrict__ qrows, int nq, int d, const float* __restrict__ qnorm,
                           const float* __restrict__ bnorm, int k, uint64_t* __restrict__ partial,
                           unsigned* __restrict__ ticket, FewOut out, int slice_at) {
  extern __shared__ __align__(16) float fq[];  // [nq][d], then the warps' lists
  uint64_t(*wl)[FEW_QS][32 * KW] = reinterpret_cast<uint64_t(*)[FEW_QS][32 * KW]>(fq);
  __shared__ int last;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int e = t; e < nq * d; e += FEW_T) {
    const int r = e / d, c = e % d;
    fq[e] = __ldg(&qs[(int64_t)(qrows ? qrows[r] : r) * d + c]);
  }
  __syncthreads();
  uint64_t L[FEW_QS][KW], thr[FEW_QS];
#pragma unroll
  for (int j = 0; j < FEW_QS; ++j) {
    thr[j] = KEY_NONE;
#pragma unroll
    for (int s = 0; s < KW; ++s) L[j][s] = KEY_NONE;
  }
  for (int64_t p0 = (int64_t)blockIdx.x * FEW_T; p0 < n; p0 += (int64_t)gridDim.x * FEW_T) {
    const int64_t pi = p0 + t;
    const bool valid = pi < n;
    const float* prow = base + (valid ? pi : 0) * d;
    float acc[FEW_QS];
#pragma unroll
    for (int j = 0; j < FEW_QS; ++j) acc[j] = 0.0f;
    if constexpr (VEC) {
      const int64_t w0 = p0 + warp * 32;  // the warp's first point
      float* slices = fq + slice_at + warp * 2 * 32 * FEW_SS;
      auto fetch = [&](int c0) {
        const int c = (lane & 7) * 4;
        float* dst = slices + (c0 / FEW_SD & 1) * 32 * FEW_SS;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int r = it * 4 + (lane >> 3);
          if (w0 + r < n && c0 + c < d) {
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst + r * FEW_SS + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(base + (w0 + r) * d + c0 + c)
                         : "memory");
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      fetch(0);
      for (int c0 = 0; c0 < d; c0 += FEW_SD) {
        fetch(c0 + FEW_SD);  // nothing past d
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const float* x = slices + (c0 / FEW_SD & 1) * 32 * FEW_SS + lane * FEW_SS;
        const int cw = min(FEW_SD, d - c0);
#pragma unroll 4
        for (int c = 0; c < cw; c += 4) {
          const float4 v = *reinterpret_cast<const float4*>(x + c);
#pragma unroll
          for (int j = 0; j < FEW_QS; ++j)
            if (j < nq) few_add<METRIC>(acc[j], *reinterpret_cast<const float4*>(&fq[j * d + c0 + c]), v);
        }
        __syncwarp();
      }
    } else if (valid) {
#pragma unroll 8
      for (int c = 0; c < d; ++c) {
        const float pv = __ldg(prow + c);
#pragma unroll
        for (int j = 0; j < FEW_QS; ++j) {
          if (j < nq) {
            const float qv = fq[j * d + c];
            if constexpr (METRIC == MANN_METRIC_COSINE) {
              acc[j] = __fmaf_rn(qv, pv, acc[j]);
            } else {
              const float u = __fsub_rn(qv, pv);
              acc[j] = __fmaf_rn(u, u, acc[j]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < FEW_QS; ++j) {
      if (j >= nq) break;  // uniform
      const float v = few_distance<METRIC>(acc[j], qnorm, qrows ? qrows[j] : j, bnorm, pi, valid);
      uint64_t key = valid ? make_key(v, (uint32_t)pi) : KEY_NONE;
      unsigned pend = __ballot_sync(FULL, key < thr[j]);
      if (pend == 0) continue;
      if (KW == 1 && __popc(pend) > 3) {
        L[j][0] = merge32(L[j][0], sort32(key < thr[j] ? key : KEY_NONE, lane), lane);
        thr[j] = list_get<KW>(L[j], k - 1);
        continue;
      }
      while (pend) {
        const int src = __ffs(pend) - 1;
        pend &= pend - 1;
        const uint64_t cnd = __shfl_sync(FULL, (unsigned long long)key, src);
        if (cnd < thr[j]) {
          list_insert<KW>(L[j], cnd, lane);
          thr[j] = list_get<KW>(L[j], k - 1);
        }
      }
    }
  }
  // the block's lists: row j's by warp j
  __syncthreads();
#pragma unroll
  for (int j = 0; j < FEW_QS; ++j)
#pragma unroll
    for (int s = 0; s < KW; ++s) wl[warp][j][s * 32 + lane] = L[j][s];
  __syncthreads();
  if (warp < nq) {
    uint64_t B[KW];
#pragma unroll
    for (int s = 0; s < KW; ++s) B[s] = wl[0][warp][s * 32 + lane];
    for (int w = 1; w < FEW_T / 32; ++w) {
      if constexpr (KW == 1) {
        B[0] = merge32(B[0], wl[w][warp][lane], lane);
      } else {
        uint64_t th = list_get<KW>(B, k - 1);
        for (int e = 0; e < k; ++e) {
          const uint64_t cnd = wl[w][warp][e];  // ascending: the rest cannot enter either
          if (!(cnd < th)) break;
          list_insert<KW>(B, cnd, lane);
          th = list_get<KW>(B, k - 1);
        }
      }
    }
    uint64_t* dst = partial + ((int64_t)warp * gridDim.x + blockIdx.x) * k;
#pragma unroll
    for (int s = 0; s < KW; ++s) {
      const int e = s * 32 + lane;
      if (e < k) dst[e] = B[s];
    }
  }
  if constexpr (KW == 1) {
    if (!ticket) return;
    __threadfence();
    __syncthreads();
    if (t == 0) {
      last = atomicAdd(ticket, 1u) + 1u == gridDim.x;
      if (last) *ticket = 0u;  // for the next search
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // every warp merges a share of the blocks' lists of every row
    const int nb = gridDim.x;
    __syncthreads();
    for (int j = 0; j < nq; ++j) {
      const uint64_t* src = partial + (int64_t)j * nb * k;
      uint64_t B = KEY_NONE;
#pragma unroll 4
      for (int g = warp; g < nb; g += FEW_T / 32)
        B = merge32(B, lane < k ? __ldcg(src + (int64_t)g * k + lane) : KEY_NONE, lane);
      wl[warp][j][lane] = B;
    }
    __syncthreads();
    if (warp >= nq) return;
    uint64_t B = wl[0][warp][lane];
    for (int w = 1; w < FEW_T / 32; ++w) B = merge32(B, wl[w][warp][lane], lane);
    if (out.ids)
      finish_row32(out, warp, B, k, lane);
    else if (lane < k)
      out.keys[(int64_t)warp * k + lane] = B;
  }
}

// Exact lists of single rows, each against its own set: CTA (i, c) scans points
// [c chunk, (c + 1) chunk) of the set that holds row rows[i] of `data`, and
// writes the 32 nearest to partial[i][c].  A warp takes 64 points at a time,
// brought in 16 columns at a time with four lanes to a row (a thread that reads
// its own row touches 32 lines per load), and keeps its own list; the slices are
// the warp's own, so no barrier falls inside.  Bound by the latency of the
// slices, which the 40 warps of an SM cover.  Replaces 32-row tiles holding one
// row each (124 rows of sets of up to 50,000 x 32: 295 to 445 us, now 57).
constexpr int SR_T = 256, SR_W = SR_T / 32, SR_DC = 16, SR_XS = SR_DC + 4;
template <int METRIC, bool VEC>
__global__ void __launch_bounds__(SR_T, 5)
    seg_rows_kernel(const float* __restrict__ data, const int32_t* __restrict__ rows, const int64_t* __restrict__ offs,
                    int nsets, int nsplit, int64_t chunk, int d, uint64_t* __restrict__ partial) {
  __shared__ __align__(16) float xs[SR_W][64][SR_XS];
  __shared__ __align__(16) float qs[SR_W][SR_DC];
  __shared__ uint64_t lists[SR_W][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t i = blockIdx.x / nsplit;
  const int64_t row = rows[i];
  const int lo = set_of(offs, nsets, row, lane);
  const int64_t end = offs[lo + 1];
  const int64_t p_begin = min(end, offs[lo] + (int64_t)(blockIdx.x % nsplit) * chunk), p_end = min(end, p_begin + chunk);
  const float* q = data + row * d;
  uint64_t L = KEY_NONE, thr = KEY_NONE;
  for (int64_t p0 = p_begin + w * 64; p0 < p_end; p0 += SR_W * 64) {
    const int np = (int)min((int64_t)64, p_end - p0);
    float acc[2] = {0.0f, 0.0f};
    for (int c0 = 0; c0 < d; c0 += SR_DC) {
      __syncwarp();
      if constexpr (VEC) {
        const int c = (lane & 3) * 4;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int r = it * 8 + (lane >> 2);
          if (r < np && c0 + c < d) {
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(&xs[w][r][c]);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(data + (p0 + r) * d + c0 + c)
                         : "memory");
          } else {
            *reinterpret_cast<float4*>(&xs[w][r][c]) = make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      } else {
        const int c = lane & 15;
#pragma unroll 8
        for (int it = 0; it < 32; ++it) {
          const int r = it * 2 + (lane >> 4);
          xs[w][r][c] = r < np && c0 + c < d ? __ldg(data + (p0 + r) * d + c0 + c) : 0.0f;
        }
      }
      if (lane < SR_DC) qs[w][lane] = c0 + lane < d ? __ldg(q + c0 + lane) : 0.0f;
      if constexpr (VEC) asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      // columns past d are zero on both sides and add nothing
#pragma unroll
      for (int c = 0; c < SR_DC; c += 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(&qs[w][c]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = *reinterpret_cast<const float4*>(&xs[w][32 * h + lane][c]);
          float u = __fsub_rn(q4.x, v.x);
          acc[h] = __fmaf_rn(u, u, acc[h]);
          u = __fsub_rn(q4.y, v.y);
          acc[h] = __fmaf_rn(u, u, acc[h]);
          u = __fsub_rn(q4.z, v.z);
          acc[h] = __fmaf_rn(u, u, acc[h]);
          u = __fsub_rn(q4.w, v.w);
          acc[h] = __fmaf_rn(u, u, acc[h]);
        }
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 32 * h + lane;
      const float v = few_distance<METRIC>(acc[h], nullptr, 0, nullptr, 0, false);
      const uint64_t key = r < np ? make_key(v, (uint32_t)(p0 + r)) : KEY_NONE;
      if (!__any_sync(FULL, key < thr)) continue;
      L = merge32(L, sort32(key < thr ? key : KEY_NONE, lane), lane);
      thr = __shfl_sync(FULL, (unsigned long long)L, 31);
    }
  }
  lists[w][lane] = L;
  __syncthreads();
  if (w > 0) return;
  for (int v = 1; v < SR_W; ++v) L = merge32(L, lists[v][lane], lane);
  partial[(int64_t)blockIdx.x * 32 + lane] = L;
}

constexpr size_t few_list_bytes(int kw) { return sizeof(uint64_t) * (FEW_T / 32) * FEW_QS * 32 * kw; }

// fused: the kernel itself merges the blocks' lists into `out` (with a ticket)
bool few_fused(int nq, int d, int kk, const unsigned* ticket) {
  return ticket && nq <= FEW_QS && d <= FEW_STAGED_D && kk <= 32;
}

template <int METRIC, bool VEC>
mann_status launch_few_m(int grid, const float* base, int64_t n, const float* qs, const int32_t* rows, int nq,
                         int d, const float* qn, const float* bn, int kk, uint64_t* partial, unsigned* ticket,
                         const FewOut& out, cudaStream_t s) {
  if (nq <= FEW_QS && d <= FEW_STAGED_D) {
    const size_t smem = std::max(sizeof(float) * nq * d, few_list_bytes(kk <= 32 ? 1 : 2));  // <= 32 KB
    const size_t slices = VEC ? FEW_SLICE_BYTES : 0;
    const auto kern = kk <= 32 ? few_rows_staged_kernel<METRIC, 1, VEC> : few_rows_staged_kernel<METRIC, 2, VEC>;
    MANN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(float) * FEW_QS * FEW_STAGED_D + slices)));
    kern<<<grid, FEW_T, smem + slices, s>>>(base, n, qs, rows, nq, d, qn, bn, kk, partial,
                                            kk <= 32 ? ticket : nullptr, out, (int)(smem / sizeof(float)));
  } else if (kk <= 32) {
    few_rows_kernel<METRIC, 1, VEC><<<grid, FEW_T, 0, s>>>(base, n, qs, rows, nq, d, qn, bn, kk, partial);
  } else {
    few_rows_kernel<METRIC, 2, VEC><<<grid, FEW_T, 0, s>>>(base, n, qs, rows, nq, d, qn, bn, kk, partial);
  }
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// The few-row scan for any metric and alignment.
mann_status run_few(int metric, int grid, const float* base, int64_t n, const float* qs, const int32_t* rows, int nq,
                    int d, const float* qn, const float* bn, int kk, uint64_t* partial, unsigned* ticket,
                    const FewOut& out, cudaStream_t s) {
  const bool vec = (d % 4 == 0) && ((reinterpret_cast<uintptr_t>(base) & 15) == 0);
#define FEW_METRIC(M)                                                                                        \
  return vec ? launch_few_m<M, true>(grid, base, n, qs, rows, nq, d, qn, bn, kk, partial, ticket, out, s)    \
             : launch_few_m<M, false>(grid, base, n, qs, rows, nq, d, qn, bn, kk, partial, ticket, out, s)
  if (metric == MANN_METRIC_EUCLIDEAN) FEW_METRIC(MANN_METRIC_EUCLIDEAN);
  if (metric == MANN_METRIC_SQEUCLIDEAN) FEW_METRIC(MANN_METRIC_SQEUCLIDEAN);
  FEW_METRIC(MANN_METRIC_COSINE);
#undef FEW_METRIC
}

// Merge up to `slots` sorted lists of k keys per query into one sorted list
// of k.  One warp per query; lane s walks list s (and s+32, ...).  After a
// balanced walk of the tile kernel (per > 0, bq rows per block) a row has one
// list for every CTA that its query block met, placed as K1Walk says.  With
// o.ids the results are written as finish_kernel writes them, without a launch
// of its own.  `shared`: several lists may hold the same key (inverted lists
// with points in common); it counts once.
__global__ void merge_lists_kernel(const uint64_t* __restrict__ partial, int64_t nq, int slots,
                                   int k, FewOut o, int64_t tiles, int64_t per, int bq, bool shared) {
  const int lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q >= nq) return;
  const uint64_t* src = partial + q * (int64_t)slots * k;
  int64_t next = k;  // from a list of the row to the next
  int nsplit = slots;
  if (per > 0) {
    const int64_t qb = q / bq, c0 = qb * tiles / per;
    nsplit = (int)(((qb + 1) * tiles - 1) / per - c0) + 1;
    src = partial + (q + c0 * bq) * k;
    next = (int64_t)bq * k;
  }
  // Short lists of few splits, one entry per lane, merge in bitonic steps (about
  // 55 instructions a list); many splits take the head-by-head form below
  // (about 75 an entry).  Two splits of 338,792 rows, k = 16: 857 us head by head.
  if (k <= 32 && nsplit * 55 < k * 75) {
    uint64_t B = lane < k ? src[lane] : KEY_NONE;
    for (int g = 1; g < nsplit; g += 4) {
      uint64_t v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = g + u < nsplit && lane < k ? src[(g + u) * next + lane] : KEY_NONE;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (g + u >= nsplit) break;  // uniform
        uint64_t M = merge32(B, v[u], lane);
        if (shared) {
          // equal keys stand side by side: entries that B holds already leave the list first
          const uint64_t left = __shfl_up_sync(FULL, (unsigned long long)M, 1);
          if (__any_sync(FULL, lane > 0 && left == M && M != KEY_NONE)) {
            const bool twice = wl::contains32(B, v[u], lane);
            M = merge32(B, sort32(twice ? KEY_NONE : v[u], lane), lane);
          }
        }
        B = M;
      }
    }
    if (o.ids)
      finish_row32(o, q, B, k, lane);
    else if (lane < k)
      o.keys[q * k + lane] = B;
    return;
  }
  constexpr int MAXL = 8;  // lists per lane (nsplit <= 256)
  int head[MAXL];
  uint64_t cur[MAXL];
#pragma unroll
  for (int t = 0; t < MAXL; ++t) {
    const int s = lane + 32 * t;
    head[t] = 0;
    cur[t] = (s < nsplit) ? src[s * next] : KEY_NONE;
  }
  int found = 0;
  for (int e = 0; e < k; ++e) {
    uint64_t m = cur[0];
#pragma unroll
    for (int t = 1; t < MAXL; ++t) m = min(m, cur[t]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, (uint64_t)__shfl_xor_sync(FULL, m, o));
    if (!o.ids) {
      if (lane == 0) o.keys[q * k + e] = m;
    } else if (m != KEY_NONE && found < o.kout && !(o.graph_self >= 0 && (int64_t)key_id(m) == o.graph_self + q)) {
      if (lane == 0) {
        o.ids[q * o.kout + found] = key_id(m);
        o.dists[q * o.kout + found] = key_dist(m);
      }
      ++found;
    }
    if (m == KEY_NONE) continue;
#pragma unroll
    for (int t = 0; t < MAXL; ++t) {
      if (cur[t] == m) {  // one owner, or every list that shares the key
        const int s = lane + 32 * t;
        ++head[t];
        cur[t] = head[t] < k ? src[s * next + head[t]] : KEY_NONE;
      }
    }
  }
  if (o.ids)
    for (int e = found + lane; e < o.kout; e += 32) {
      o.ids[q * o.kout + e] = -1;
      o.dists[q * o.kout + e] = __int_as_float(0x7F800000);
    }
}

__global__ void finish_kernel(const uint64_t* __restrict__ keys, int64_t nq, int kk, FewOut o,
                              const int64_t* __restrict__ offs, int nsets) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nq) return;
  const uint64_t* src = keys + q * (int64_t)kk;
  int32_t* oid = o.ids + q * o.kout;
  float* odist = o.dists + q * o.kout;
  int32_t first = 0;
  if (offs) {
    int lo = 0, hi = nsets - 1;
    while (lo < hi) {  // last set whose offset <= q
      const int mid = (lo + hi + 1) >> 1;
      if (offs[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    first = (int32_t)offs[lo];
  }
  int m = 0;
  for (int e = 0; e < kk && m < o.kout; ++e) {
    const uint64_t key = src[e];
    if (key == KEY_NONE) break;
    if (o.graph_self >= 0 && (int64_t)key_id(key) == o.graph_self + q) continue;
    oid[m] = (int32_t)key_id(key) - first;
    odist[m] = key_dist(key);
    ++m;
  }
  for (; m < o.kout; ++m) {
    oid[m] = -1;
    odist[m] = __int_as_float(0x7F800000);
  }
}

// finish_kernel for lists of at most 32: a warp per row, so that keys, ids and
// distances move in whole lines, and the set's first row found by its lanes
// (338,792 rows of 15 in 24 sets: 70 us and 26 for the offsets of the ids, now 41).
__global__ void finish32_kernel(const uint64_t* __restrict__ keys, int64_t nq, int kk, FewOut o,
                                const int64_t* __restrict__ offs, int nsets) {
  const int lane = threadIdx.x & 31;
  const int64_t q = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (q >= nq) return;
  const uint64_t key = lane < kk ? keys[q * kk + lane] : KEY_NONE;
  finish_row32(o, q, key, kk, lane, offs ? (int32_t)offs[set_of(offs, nsets, q, lane)] : 0);
}

// query rows per CTA of the tile kernel
int k1_rows(int64_t nq, int k) { return nq > 32 && k <= 128 ? 64 : 32; }

// The tile kernel's walk.  splits > 0: that many splits per query block.
// splits == 0: an equal share of the units for every CTA that the device
// holds at once -- a grid of whole query blocks leaves a nearly empty last
// wave (20,011 rows: 313 blocks on 456 places) or, with few blocks, idle SMs
// -- unless there are so many query blocks that whole ones balance to within
// an eighth, which needs no merge.
K1Walk k1_walk(int num_sms, int64_t n, int64_t nq, int k, int splits) {
  const int bq = k1_rows(nq, k);
  const int64_t qblocks = ceil_div(nq, bq);
  K1Walk w{};
  w.tiles = (int)ceil_div(n, K1_BN);
  w.total = qblocks * w.tiles;
  const int64_t places = (int64_t)num_sms * (k <= 32 ? k1_ctas<64, 1>() : k1_ctas<64, 2>());
  if (splits == 0 && qblocks >= 8 * places) splits = 1;
  if (splits > 0) {
    w.tiles_per = (int)ceil_div(w.tiles, splits);
    w.splits = (int)ceil_div(w.tiles, w.tiles_per);
    w.slots = w.splits;
    w.stride = w.slots;
    w.rows = nq * w.slots;
    return w;
  }
  w.per = std::max(ceil_div(w.total, places), ceil_div(w.tiles, 96));  // at most 97 lists per row
  w.slots = w.per % w.tiles == 0 ? 1 : (w.tiles % w.per == 0 ? (int)(w.tiles / w.per) : (int)((w.tiles - 2) / w.per) + 2);
  w.step = w.slots > 1 ? bq : 0;
  w.stride = 1;
  w.rows = nq + (ceil_div(w.total, w.per) - 1) * w.step;
  return w;
}

template <int METRIC, int BQ, int KW, bool VEC>
mann_status launch_k1(Context* ctx, const float* base, int64_t n, const float* qs, const int32_t* rows,
                      int64_t nq, int d, const float* qn, const float* bn, int k, const K1Walk& w, uint64_t* partial,
                      cudaStream_t s) {
  constexpr size_t smem = k1_smem_bytes<BQ, KW>();
  auto kern = k1_tile_topk<METRIC, BQ, KW, VEC>;
  MANN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int64_t grid = w.splits > 0 ? ceil_div(nq, BQ) * w.splits : ceil_div(w.total, w.per);
  ctx->time_begin(s);
  kern<<<(unsigned)grid, K1_THREADS, smem, s>>>(base, n, qs, rows, nq, d, qn, bn, k, w, partial);
  ctx->time_end(s);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

template <int METRIC, bool VEC>
mann_status dispatch_k1(Context* ctx, int k, const float* base, int64_t n, const float* qs, const int32_t* rows,
                        int64_t nq, int d, const float* qn, const float* bn, const K1Walk& w, uint64_t* partial,
                        cudaStream_t s) {
  if (k1_rows(nq, k) == 32)
    return launch_k1<METRIC, 32, 8, VEC>(ctx, base, n, qs, rows, nq, d, qn, bn, k, w, partial, s);
  if (k <= 32) return launch_k1<METRIC, 64, 1, VEC>(ctx, base, n, qs, rows, nq, d, qn, bn, k, w, partial, s);
  if (k <= 64) return launch_k1<METRIC, 64, 2, VEC>(ctx, base, n, qs, rows, nq, d, qn, bn, k, w, partial, s);
  return launch_k1<METRIC, 64, 4, VEC>(ctx, base, n, qs, rows, nq, d, qn, bn, k, w, partial, s);
}

// The tile kernel for any metric and alignment.
mann_status run_k1(Context* ctx, int metric, int k, const float* base, int64_t n, const float* qs, const int32_t* rows,
                   int64_t nq, int d, const float* qn, const float* bn, const K1Walk& w, uint64_t* partial,
                   cudaStream_t s) {
  const bool vec = (d % 4 == 0) && ((reinterpret_cast<uintptr_t>(base) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(qs) & 15) == 0);
#define K1_METRIC(M)                                                                                    \
  return vec ? dispatch_k1<M, true>(ctx, k, base, n, qs, rows, nq, d, qn, bn, w, partial, s)            \
             : dispatch_k1<M, false>(ctx, k, base, n, qs, rows, nq, d, qn, bn, w, partial, s)
  if (metric == MANN_METRIC_EUCLIDEAN) K1_METRIC(MANN_METRIC_EUCLIDEAN);
  if (metric == MANN_METRIC_SQEUCLIDEAN) K1_METRIC(MANN_METRIC_SQEUCLIDEAN);
  K1_METRIC(MANN_METRIC_COSINE);
#undef K1_METRIC
}

}  // namespace

template <int METRIC, int BQ, int KW, bool VEC>
static mann_status launch_pers_t(int num_sms, const float* data, const SegItem* items, SegQueue* q, unsigned epoch,
                                 long long wait_cycles, int d, int k, int nsplit, uint64_t* partial,
                                 cudaStream_t s) {
  constexpr size_t smem = k1_smem_bytes<BQ, KW>();
  auto kern = k1_persistent<METRIC, BQ, KW, VEC>;
  MANN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  MANN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, K1_THREADS, smem));
  const int grid = std::max(1, per_sm) * num_sms;  // every CTA resident: the queue needs no co-scheduling
  kern<<<(unsigned)grid, K1_THREADS, smem, s>>>(data, items, q, epoch, wait_cycles, d, k, nsplit, partial, nullptr);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

mann_status launch_k1_persistent(int num_sms, const float* data, const SegItem* items, SegQueue* q, unsigned epoch,
                                 long long wait_cycles, int d, int metric, int bq, int k, int nsplit,
                                 uint64_t* partial, cudaStream_t s) {
  if (k < 1 || k > 64) return fail(MANN_EINVAL_ARG, "batched graphs support 1 <= k <= 64 (k+1 with self)");
  const bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
#define PERS_CASE(M, B, KW)                                                                                      \
  return vec ? launch_pers_t<M, B, KW, true>(num_sms, data, items, q, epoch, wait_cycles, d, k, nsplit, partial, \
                                             s)                                                                 \
             : launch_pers_t<M, B, KW, false>(num_sms, data, items, q, epoch, wait_cycles, d, k, nsplit, partial, \
                                              s)
  if (metric == MANN_METRIC_EUCLIDEAN) {
    if (k > 32) {
      if (bq == 32) PERS_CASE(MANN_METRIC_EUCLIDEAN, 32, 2);
      PERS_CASE(MANN_METRIC_EUCLIDEAN, 64, 2);
    }
    if (bq == 32) PERS_CASE(MANN_METRIC_EUCLIDEAN, 32, 1);
    PERS_CASE(MANN_METRIC_EUCLIDEAN, 64, 1);
  }
  if (metric == MANN_METRIC_SQEUCLIDEAN) {
    if (k > 32) {
      if (bq == 32) PERS_CASE(MANN_METRIC_SQEUCLIDEAN, 32, 2);
      PERS_CASE(MANN_METRIC_SQEUCLIDEAN, 64, 2);
    }
    if (bq == 32) PERS_CASE(MANN_METRIC_SQEUCLIDEAN, 32, 1);
    PERS_CASE(MANN_METRIC_SQEUCLIDEAN, 64, 1);
  }
#undef PERS_CASE
  return fail(MANN_EINVAL_ARG, "batched graphs: Euclidean or SqEuclidean");
}

mann_status launch_seg_rows(const float* data, const int32_t* rows, int cnt, const int64_t* offs, int nsets, int nsplit,
                            int64_t chunk, int d, int metric, uint64_t* partial, cudaStream_t s) {
  if (cnt <= 0) return MANN_OK;
  const int64_t grid = (int64_t)cnt * nsplit;
  if (grid > INT32_MAX) return fail(MANN_EINVAL_ARG, "batched graphs: too many rows to scan");
  const bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
#define SEG_ROWS(M)                                                                                                 \
  (vec ? seg_rows_kernel<M, true> : seg_rows_kernel<M, false>)<<<(unsigned)grid, SR_T, 0, s>>>(data, rows, offs, nsets, \
                                                                                      nsplit, chunk, d, partial)
  if (metric == MANN_METRIC_EUCLIDEAN)
    SEG_ROWS(MANN_METRIC_EUCLIDEAN);
  else if (metric == MANN_METRIC_SQEUCLIDEAN)
    SEG_ROWS(MANN_METRIC_SQEUCLIDEAN);
  else
    return fail(MANN_EINVAL_ARG, "batched graphs: Euclidean or SqEuclidean");
#undef SEG_ROWS
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

mann_status launch_merge_lists(const uint64_t* partial, int64_t nq, int nsplit, int k, uint64_t* out,
                               cudaStream_t s, bool shared) {
  if (nq <= 0) return MANN_OK;
  if (nsplit > 128) return fail(MANN_EINVAL_ARG, "at most 128 lists per query can be merged");
  merge_lists_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, s>>>(partial, nq, nsplit, k, FewOut{out, nullptr, nullptr, 0, -1}, 0,
                                                               0, 1, shared);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

mann_status launch_row_sqnorm(const float* x, int64_t n, int d, float* out, cudaStream_t s) {
  if (n <= 0) return MANN_OK;
  row_sqnorm_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, s>>>(x, n, d, out);  // 8 warps x 32 rows
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

mann_status launch_finish(const uint64_t* keys, int64_t nq, int kk, int kout, int64_t graph_self,
                          int32_t* ids, float* dists, cudaStream_t s, const int64_t* offs, int nsets) {
  if (nq <= 0 || kout <= 0) return MANN_OK;
  const FewOut o{nullptr, ids, dists, kout, graph_self};
  if (kk <= 32)
    finish32_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, s>>>(keys, nq, kk, o, offs, nsets);
  else
    finish_kernel<<<(unsigned)ceil_div(nq, 128), 128, 0, s>>>(keys, nq, kk, o, offs, nsets);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

// knn_fp32_keys, or with o.ids set the finished results (nothing in *out_keys).
static mann_status fp32_search(Context* ctx, cudaStream_t s, const float* base, int64_t n, const float* qs, int64_t nq,
                               int d, int metric, int kk, const int32_t* rows, const float* qn, const float* bn,
                               FewOut o, uint64_t** out_keys, int slot_partial, int slot_keys) {
  if (kk < 1 || kk > KMAX_FUSED)
    return fail(MANN_EINVAL_ARG, "fused top-k supports 1 <= k <= " + std::to_string(KMAX_FUSED));
  if (nq <= 0) return MANN_OK;
  if (metric == MANN_METRIC_COSINE && (qn == nullptr || bn == nullptr))
    return fail(MANN_EINVAL_ARG, "cosine search needs row norms");
  const bool few = nq <= FEW_Q && kk <= 64;
  // a handful of rows: one point per thread across the whole GPU (one pass for n <= 65536)
  const int grid = few ? (int)std::min<int64_t>(256, ceil_div(n, FEW_T)) : 0;
  const K1Walk w = few ? K1Walk{} : k1_walk(ctx->num_sms, n, nq, kk, 0);
  const int slots = few ? grid : w.slots;
  const bool fused = few && few_fused((int)nq, d, kk, ctx->few_ticket);
  uint64_t* partial = nullptr;
  MANN_TRY(ctx->scratch_t(slot_partial, (size_t)(few ? nq * slots : w.rows) * kk, &partial));
  if (!o.ids && (fused || slots > 1)) MANN_TRY(ctx->scratch_t(slot_keys, (size_t)nq * kk, &o.keys));
  if (few) {
    ctx->time_begin(s);
    MANN_TRY(run_few(metric, grid, base, n, qs, rows, (int)nq, d, qn, bn, kk, partial, fused ? ctx->few_ticket : nullptr,
                     o, s));
    ctx->time_end(s);
  } else {
    MANN_TRY(run_k1(ctx, metric, kk, base, n, qs, rows, nq, d, qn, bn, w, partial, s));
  }
  if (!fused) {
    if (slots == 1) {
      if (o.ids) return launch_finish(partial, nq, kk, o.kout, o.graph_self, o.ids, o.dists, s);
      *out_keys = partial;
      return MANN_OK;
    }
    merge_lists_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, s>>>(partial, nq, slots, kk, o, few ? 0 : w.tiles,
                                                                 few ? 0 : w.per, few ? 1 : k1_rows(nq, kk), false);
    MANN_CHECK_LAUNCH();
  }
  if (!o.ids) *out_keys = o.keys;
  return MANN_OK;
}

mann_status knn_fp32_keys(Context* ctx, cudaStream_t s, const float* base, int64_t n,
                          const float* qs, int64_t nq, int d, int metric, int kk,
                          const int32_t* rows, const float* qn, const float* bn,
                          uint64_t** out_keys, int slot_partial, int slot_keys) {
  return fp32_search(ctx, s, base, n, qs, nq, d, metric, kk, rows, qn, bn, FewOut{nullptr, nullptr, nullptr, 0, -1},
                     out_keys, slot_partial, slot_keys);
}

mann_status knn_fp32_finished(Context* ctx, cudaStream_t s, const float* base, int64_t n, const float* qs, int64_t nq,
                              int d, int metric, int kk, const float* qn, const float* bn, int kout,
                              int64_t graph_self, int32_t* ids, float* dists) {
  return fp32_search(ctx, s, base, n, qs, nq, d, metric, kk, nullptr, qn, bn,
                     FewOut{nullptr, ids, dists, kout, graph_self}, nullptr, SLOT_PARTIAL, SLOT_KEYS);
}

}  // namespace mann

namespace mann {

// Plan of the FP32 form for (n, nq, kk) on a device with num_sms SMs, as
// knn_fp32_keys_on makes it: a few rows (nq <= FEW_Q, kk <= 64) go to the
// few-row kernel with `*nsplit_out` = its grid of point slices; otherwise the
// tile kernel with `*nsplit_out` point splits: one CTA per SM if its blocks had
// 128 rows, so two of the three that an SM holds with the 64 rows they have (k <=
// 64).  More splits would fill those places but take more scratch, of which the
// entry point has a fixed amount: a search that fits must go on fitting.
// `*words_out` = the uint64
// words of scratch (per-split lists, then merged lists when there is more
// than one split).
void knn_fp32_plan(int num_sms, int64_t n, int64_t nq, int kk, int* nsplit_out,
                   size_t* words_out) {
  int nsplit = 1;
  if (nq <= FEW_Q && kk <= 64) {
    nsplit = (int)std::min<int64_t>(256, ceil_div(n, FEW_T));
  } else {
    const int bq = nq <= 32 ? 32 : (kk <= 64 ? 128 : (kk <= 128 ? 64 : 32));
    const int64_t qblocks = ceil_div(nq, bq);
    const int64_t tiles = ceil_div(n, K1_BN);
    int64_t want = std::max<int64_t>(1, ceil_div(num_sms, qblocks));
    want = std::min<int64_t>(want, std::min<int64_t>(tiles, 128));
    const int64_t tiles_per = ceil_div(tiles, want);
    nsplit = (int)ceil_div(tiles, tiles_per);
  }
  *nsplit_out = nsplit;
  *words_out = (size_t)nq * nsplit * kk + (nsplit > 1 ? (size_t)nq * kk : 0);
}

// knn_fp32_keys on caller-provided scratch (`words` uint64 at `scratch`,
// laid out as knn_fp32_plan says); no allocation.
mann_status knn_fp32_keys_on(int num_sms, cudaStream_t s, const float* base, int64_t n,
                             const float* qs, int64_t nq, int d, int metric, int kk,
                             const float* qn, const float* bn, uint64_t* scratch, size_t words,
                             uint64_t** out_keys) {
  if (kk < 1 || kk > KMAX_FUSED)
    return fail(MANN_EINVAL_ARG, "fused top-k supports 1 <= k <= " + std::to_string(KMAX_FUSED));
  if (nq <= 0) return MANN_OK;
  if (metric == MANN_METRIC_COSINE && (qn == nullptr || bn == nullptr))
    return fail(MANN_EINVAL_ARG, "cosine search needs row norms");
  int nsplit = 1;
  size_t need = 0;
  knn_fp32_plan(num_sms, n, nq, kk, &nsplit, &need);
  if (need > words) return fail(MANN_EINVAL_ARG, "scratch too small for this search");
  uint64_t* partial = scratch;
  mann_status st;
  if (nq <= FEW_Q && kk <= 64) {
    // the few-row kernel, as knn_fp32_keys runs it (grid = nsplit), its lists merged by a launch of their own
    st = run_few(metric, nsplit, base, n, qs, nullptr, (int)nq, d, qn, bn, kk, partial, nullptr,
                 FewOut{nullptr, nullptr, nullptr, 0, -1}, s);
  } else {
    Context plain;  // carries the SM count; no timing, no scratch
    plain.num_sms = num_sms;
    st = run_k1(&plain, metric, kk, base, n, qs, nullptr, nq, d, qn, bn, k1_walk(num_sms, n, nq, kk, nsplit), partial,
                s);
  }
  MANN_TRY(st);
  if (nsplit == 1) {
    *out_keys = partial;
    return MANN_OK;
  }
  uint64_t* keys = partial + (size_t)nq * nsplit * kk;
  merge_lists_kernel<<<(unsigned)ceil_div(nq, 8), 256, 0, s>>>(partial, nq, nsplit, kk,
                                                               FewOut{keys, nullptr, nullptr, 0, -1}, 0, 0, 1, false);
  MANN_CHECK_LAUNCH();
  *out_keys = keys;
  return MANN_OK;
}

}  // namespace mann
