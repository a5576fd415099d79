// ivf.cu -- IVF-Flat on the GPU: build (KMeans + inverted lists) and search
// (route to nprobe lists, scan them, top-k).
//
// Replaces src/indices/ivf_flat.jl: build_index (:30-93), _centroid_distances
// + partialsortperm routing (:103-131, :150) and the list scan into a bounded
// heap (:153-167); the routing hook is select_indices(TopKRouting)
// (src/indices/multilevel/routing.jl:94-118), and mann_ivf_scan takes any
// routing (the learned probe supplies its own).
//
// The scan runs "inverted" like the reference's batched multi-level query
// (src/indices/multilevel/query.jl:363-396): queries are grouped by the list
// they probe, and one CTA scans one list, or a part of a long one, for up to 16
// of its queries, the points read in place through the list's ids, every
// distance in the FP32 form's sequential arithmetic, keeping each query's
// top-k.  Order: (distance,
// id); the reference's heap keeps an arbitrary member of an exact tie at the
// k-th place, this keeps the lower id.
#include <algorithm>
#include <type_traits>
#include <vector>

#include "f32x2.cuh"
#include "kernels.cuh"
#include "warp_list.cuh"

namespace mann {

namespace {

// Queries per CTA (at most).  32 at three CTAs per SM, for lists that see more
// than a dozen queries, were slower at every size: 220 lists of 600 x 64, 59
// queries each 649 us against 450; 195 of 370 x 96, 412 each 2.14 ms and 1.76.
constexpr int SCAN_Q = 16;
constexpr int SCAN_T = 128;   // threads
constexpr int SCAN_P = 256;   // points per pass: two per thread
constexpr int SCAN_DC = 16;   // dimensions per staged slice of a point row

__global__ void ivf_lists_kernel(const int64_t* __restrict__ start, const int64_t* __restrict__ members,
                                 int k, int64_t n, int64_t* __restrict__ offsets,
                                 int32_t* __restrict__ ids) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ids[i] = (int32_t)members[i];
  if (i <= k) offsets[i] = i < k ? start[i] : n;
}

__global__ void probe_count_kernel(const int32_t* __restrict__ probes, int64_t np, int nlist,
                                   unsigned* __restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  const int l = probes[i];
  if (l >= 0 && l < nlist) atomicAdd(&cnt[l], 1u);
}

// Exclusive prefix sums of the per-list query counts and of their qc-query
// chunks; one block of 1024 threads, each owning a contiguous run of lists.
__global__ void __launch_bounds__(1024) probe_scan_kernel(const unsigned* __restrict__ cnt, int nlist, int qc,
                                                          int64_t* __restrict__ qoff,
                                                          int64_t* __restrict__ choff) {
  __shared__ int64_t wa[32], wb[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int per = (nlist + 1023) / 1024;
  const int l0 = min(nlist, t * per), l1 = min(nlist, l0 + per);
  int64_t a = 0, b = 0;
  for (int l = l0; l < l1; ++l) {
    a += cnt[l];
    b += (cnt[l] + qc - 1) / qc;
  }
  int64_t ia = a, ib = b;  // inclusive scans within the warp
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t xa = __shfl_up_sync(0xffffffffu, ia, o), xb = __shfl_up_sync(0xffffffffu, ib, o);
    if (lane >= o) {
      ia += xa;
      ib += xb;
    }
  }
  if (lane == 31) {
    wa[w] = ia;
    wb[w] = ib;
  }
  __syncthreads();
  if (w == 0) {
    int64_t va = wa[lane], vb = wb[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t xa = __shfl_up_sync(0xffffffffu, va, o), xb = __shfl_up_sync(0xffffffffu, vb, o);
      if (lane >= o) {
        va += xa;
        vb += xb;
      }
    }
    wa[lane] = va;
    wb[lane] = vb;
  }
  __syncthreads();
  int64_t ea = ia - a + (w ? wa[w - 1] : 0), eb = ib - b + (w ? wb[w - 1] : 0);
  for (int l = l0; l < l1; ++l) {
    qoff[l] = ea;
    choff[l] = eb;
    ea += cnt[l];
    eb += (cnt[l] + qc - 1) / qc;
  }
  if (t == 1023) {
    qoff[nlist] = ea;
    choff[nlist] = eb;
  }
}

// (query, probe rank) pairs grouped by list, and the list of every chunk (a
// search for it in each scan block was a chain of a dozen dependent loads)
__global__ void probe_scatter_kernel(const int32_t* __restrict__ probes, int64_t nq, int nprobe,
                                     int nlist, const int64_t* __restrict__ qoff, const int64_t* __restrict__ choff,
                                     unsigned* __restrict__ cursor, int32_t* __restrict__ pair_q,
                                     int32_t* __restrict__ pair_r, int32_t* __restrict__ chunk_list) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t l = i; l < nlist; l += (int64_t)gridDim.x * blockDim.x)
    for (int64_t c = choff[l]; c < choff[l + 1]; ++c) chunk_list[c] = (int32_t)l;
  if (i >= nq * nprobe) return;
  const int l = probes[i];
  if (l < 0 || l >= nlist) return;
  const int64_t pos = qoff[l] + atomicAdd(&cursor[l], 1u);
  pair_q[pos] = (int32_t)(i / nprobe);
  pair_r[pos] = (int32_t)(i % nprobe);
}

// One stage of a warp's bitonic network over 32-bit values (lane holds one).
__device__ __forceinline__ uint32_t cmpex32(uint32_t v, int j, bool keep_min) {
  const uint32_t o = __shfl_xor_sync(wl::FULL, v, j);
  return keep_min ? min(v, o) : max(v, o);
}

// One pass's distances of one query (dist[0, np), bits not negative) into its
// sorted list of at most 32 keys.  The k-th smallest of the lanes' minima is
// an upper bound of the pass's k-th distance, so a list that is not full sees
// about k distances instead of all of them (at k = 10, 12 of 256); those that
// pass are sorted and merged 32 at a time.  Entering them one by one took more
// instructions than the distances themselves.
__device__ __forceinline__ void pass_topk32(const float* __restrict__ dist, int np, const int32_t* __restrict__ ids,
                                            uint64_t& L, int k, uint64_t* __restrict__ buf, int lane) {
  constexpr int G = SCAN_P / 32;
  uint32_t v[G];
  uint32_t low = 0xFFFFFFFFu;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int col = 32 * g + lane;
    const float f = col < np ? dist[col] : 0.0f;
    v[g] = col < np ? (f == f ? __float_as_uint(f) : 0x7FC00000u) : 0xFFFFFFFFu;
    low = min(low, v[g]);
  }
  const uint64_t kth = __shfl_sync(wl::FULL, (unsigned long long)L, k - 1);
  uint32_t thr;  // bits of the largest distance that may still enter
  if (kth != KEY_NONE) {
    thr = __float_as_uint(key_dist(kth));
  } else {
#pragma unroll
    for (int w = 2; w <= 32; w <<= 1)
#pragma unroll
      for (int j = w >> 1; j > 0; j >>= 1) low = cmpex32(low, j, ((lane & j) == 0) == ((lane & w) == 0));
    thr = __shfl_sync(wl::FULL, low, k - 1);  // all bits set: fewer than k lanes hold a point
  }
  unsigned pend = 0;
#pragma unroll
  for (int g = 0; g < G; ++g) pend |= (v[g] <= thr && 32 * g + lane < np ? 1u : 0u) << g;
  while (__any_sync(wl::FULL, pend != 0)) {
    int base = 0;
    __syncwarp();
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const bool mine = (pend >> g) & 1u;
      const unsigned m = __ballot_sync(wl::FULL, mine);
      const int pos = base + __popc(m & ((1u << lane) - 1u));
      if (mine && pos < 32) {
        const int col = 32 * g + lane;
        buf[pos] = make_key(__uint_as_float(v[g]), (uint32_t)ids[col]);
        pend &= ~(1u << g);
      }
      base += __popc(m);
    }
    __syncwarp();
    L = wl::merge32(L, wl::sort32(lane < base ? buf[lane] : KEY_NONE, lane), lane);
    if (base > 32) {  // the rest is tested again against the list's new k-th
      const uint64_t now = __shfl_sync(wl::FULL, (unsigned long long)L, k - 1);
      if (now != KEY_NONE) {
        const uint32_t t = __float_as_uint(key_dist(now));
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (v[g] > t) pend &= ~(1u << g);
      }
    }
  }
}

// Shared memory of a scan CTA: the staged queries, then a slice of every row, over which the pass's distances are laid when the arithmetic is done.
struct ScanSmem {
  static constexpr int QC = SCAN_Q;
  static constexpr int SDQ = 128;                  // query dimensions per stage
  static constexpr int QS = QC + 4;                // stride (floats), a multiple of 4
  static constexpr int XS = SCAN_DC + 4;           // stride of a staged row slice
  static constexpr int DS = SCAN_P + 1;            // stride of a query's distances
  static constexpr size_t QUERIES = (size_t)SDQ * QS;
  static constexpr size_t ROWS = (size_t)SCAN_P * XS;
  static constexpr size_t DISTS = (size_t)QC * DS;
  static constexpr size_t BYTES = sizeof(float) * (QUERIES + (ROWS > DISTS ? ROWS : DISTS));
};

// One CTA: up to SCAN_Q of list l's queries and a part of the list (blockIdx.y).  Each thread takes
// two points of the list per pass (read in place through the list's ids) and
// computes their distances to every query of the CTA, each distance the
// sequential difference-form sum over dimensions 0..d-1 of the FP32 form.
// Warp w keeps the sorted top-k of queries w, w+4, ... as warp-distributed lists.
//
// A warp brings in its 64 rows a 16-dimension slice at a time, four lanes to a
// row (cp.async), and each thread reads its own rows back from shared memory;
// the slices are the warp's own, so no block barrier falls inside the
// arithmetic (past 128 dimensions two per 128, where the queries are staged
// anew), and six CTAs per SM cover each other's loads.  A pair of points per
// thread halves the reads of the queries, one 16-byte broadcast per four queries
// and dimension.  What bounds it is waiting: at 10,000 queries in 4 of 4,096
// lists of 1M x 128 (338 us) issue slots are 52 % busy, the FMA pipe 31 %, shared
// memory 24 % and DRAM 20 %; of the 8 warps waiting per issue 2.7 stand at the
// barriers around the selection, 1.8 on fixed latencies, 1.5 on shared memory and
// 1.3 on rows.
template <int METRIC, int KW, bool VEC>
__global__ void __launch_bounds__(SCAN_T, 6)
    ivf_scan_kernel(const float* __restrict__ data, const int64_t* __restrict__ loff,
                    const int32_t* __restrict__ lids, const float* __restrict__ qs, int d,
                    const int64_t* __restrict__ qoff, const int32_t* __restrict__ pair_q,
                    const int32_t* __restrict__ pair_r, const int64_t* __restrict__ choff,
                    const int32_t* __restrict__ chunk_list, int nlist,
                    int k, int nprobe, uint64_t* __restrict__ partial) {
  // queries staged transposed, [dimension][query] with a padded stride, so one
  // 16-byte broadcast read gives four queries' value at one dimension
  using S = ScanSmem;
  constexpr int QC = SCAN_Q, SDQ = S::SDQ, QS = S::QS, XS = S::XS;
  constexpr int NW = SCAN_T / 32;
  extern __shared__ __align__(16) float scan_smem[];
  float* qsm = scan_smem;
  float* rows = qsm + S::QUERIES;  // [SCAN_P][XS]
  float* dsm = rows;               // [QC][DS]
  __shared__ int32_t s_q[QC];
  __shared__ uint64_t s_buf[NW][32];

  const int64_t w = blockIdx.x;
  if (w >= choff[nlist]) return;
  const int l = chunk_list[w];
  const int64_t e0 = qoff[l] + (w - choff[l]) * QC;
  const int nqe = (int)min((int64_t)QC, qoff[l + 1] - e0);
  const int64_t l_end = loff[l + 1];
  const int64_t part = ((l_end - loff[l] + gridDim.y - 1) / gridDim.y + SCAN_P - 1) / SCAN_P * SCAN_P;
  const int64_t p_begin = min(l_end, loff[l] + blockIdx.y * part), p_end = min(l_end, p_begin + part);
  if (blockIdx.y > 0 && p_begin == p_end) return;  // its lists are empty already
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (t < nqe) s_q[t] = pair_q[e0 + t];

  constexpr int MW = QC / NW;  // queries per warp
  uint64_t L[MW][KW];
#pragma unroll
  for (int m = 0; m < MW; ++m)
#pragma unroll
    for (int s = 0; s < KW; ++s) L[m][s] = KEY_NONE;

  float* wrows = rows + warp * 64 * XS;  // the warp's 64 rows: lane's are lane and lane + 32
  for (int64_t p0 = p_begin; p0 < p_end; p0 += SCAN_P) {
    int32_t row[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t pi = p0 + warp * 64 + 32 * h + lane;
      row[h] = pi < p_end ? lids[pi] : -1;
    }
    // dimensions [c0, c0 + SCAN_DC) of the warp's rows (VEC: what lies below d)
    auto fetch = [&](int c0) {
      float* dst = wrows;
      if constexpr (VEC) {
        const int c = (lane & 3) * 4;
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int r = it * 8 + (lane >> 2);
          const int32_t src = __shfl_sync(wl::FULL, row[it >> 2], r & 31);
          if (src >= 0 && c0 + c < d) {
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst + r * XS + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(data + (int64_t)src * d + c0 + c)
                         : "memory");
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      } else {
        const int c = c0 + (lane & 15);
        for (int it = 0; it < 32; ++it) {
          const int r = it * 2 + (lane >> 4);
          const int32_t a = __shfl_sync(wl::FULL, row[0], r & 31), b = __shfl_sync(wl::FULL, row[1], r & 31);
          const int32_t src = r < 32 ? a : b;
          dst[r * XS + (lane & 15)] = src >= 0 && c < d ? __ldg(data + (int64_t)src * d + c) : 0.0f;
        }
      }
    };
    // the arithmetic is what the scan costs, so it stops where the list does:
    // a warp past the end computes nothing, one with at most 32 rows one half
    const int halves = (int)min((int64_t)2, max((int64_t)0, (p_end - p0 - warp * 64 + 31) / 32));
    if (p0 > p_begin) __syncthreads();  // the last pass's distances lie over the slices
    if (halves > 0) fetch(0);
    // queries 2i and 2i+1 in one f32x2 pair: each lane rounds as the scalar
    // difference form, dimension by dimension in order
    uint64_t acc2[2][QC / 2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < QC / 2; ++i) acc2[h][i] = 0ull;
    const int ng4 = (nqe + 3) >> 2;  // groups of four staged queries in use
    for (int c0 = 0; c0 < d; c0 += SCAN_DC) {
      const int cq = c0 % SDQ;  // within the staged queries
      if (cq == 0 && (d > SDQ || p0 == p_begin)) {
        const int dq = min(SDQ, d - c0);
        __syncthreads();
        // consecutive threads take consecutive queries: distinct banks
        for (int e = t; e < QC * SDQ / 4; e += SCAN_T) {
          const int r = e % QC, c = e / QC * 4;
          float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          if (r < nqe) {
            const float* q = qs + (int64_t)s_q[r] * d + c0 + c;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (c + i < dq) v[i] = __ldg(q + i);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) qsm[(c + i) * QS + r] = v[i];
        }
        __syncthreads();
      }
      if (halves == 0) continue;
      if (c0 > 0) fetch(c0);
      if constexpr (VEC) asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      const float* own = wrows + lane * XS;
      const int dc = min(SCAN_DC, d - c0);
      // four dimensions of NH points against the staged queries
      auto four = [&](int c4, auto nh) {
        constexpr int NH = decltype(nh)::value;
        float x[NH][4];
#pragma unroll
        for (int h = 0; h < NH; ++h) {
          const float4 v = *reinterpret_cast<const float4*>(own + 32 * h * XS + c4);
          x[h][0] = v.x;
          x[h][1] = v.y;
          x[h][2] = v.z;
          x[h][3] = v.w;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4* qrow4 = reinterpret_cast<const float4*>(&qsm[(cq + c4 + i) * QS]);
#pragma unroll
          for (int g = 0; g < QC / 4; ++g) {
            if (g < ng4) {  // block-uniform
              const float4 q4 = qrow4[g];
              const uint64_t lo = f2::pack(q4.x, q4.y), hi = f2::pack(q4.z, q4.w);
#pragma unroll
              for (int h = 0; h < NH; ++h) {
                const uint64_t x2 = f2::pack(x[h][i], x[h][i]);
                uint64_t u = f2::sub(lo, x2);
                acc2[h][2 * g] = f2::fma(u, u, acc2[h][2 * g]);
                u = f2::sub(hi, x2);
                acc2[h][2 * g + 1] = f2::fma(u, u, acc2[h][2 * g + 1]);
              }
            }
          }
        }
      };
      // past d (VEC: no such dimension) both sides hold zeros
      if (halves == 2) {
#pragma unroll 1
        for (int c4 = 0; c4 < dc; c4 += 4) four(c4, std::integral_constant<int, 2>());
      } else {
#pragma unroll 1
        for (int c4 = 0; c4 < dc; c4 += 4) four(c4, std::integral_constant<int, 1>());
      }
      __syncwarp();  // every lane has read the slice before it is replaced
    }
    __syncthreads();  // every warp has read its slices
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < QC / 2; ++i) {
        float a, b;
        f2::unpack(acc2[h][i], a, b);
        const int col = warp * 64 + 32 * h + lane;
        if (2 * i < nqe) dsm[(2 * i) * S::DS + col] = METRIC == MANN_METRIC_EUCLIDEAN ? __fsqrt_rn(a) : a;
        if (2 * i + 1 < nqe) dsm[(2 * i + 1) * S::DS + col] = METRIC == MANN_METRIC_EUCLIDEAN ? __fsqrt_rn(b) : b;
      }
    __syncthreads();
    const int np = (int)min((int64_t)SCAN_P, p_end - p0);
#pragma unroll
    for (int m = 0; m < MW; ++m) {
      const int j = warp + NW * m;
      if (j >= nqe) continue;  // warp-uniform
      const float* dist = dsm + j * S::DS;
      if constexpr (KW == 1) {
        pass_topk32(dist, np, lids + p0, L[m][0], k, s_buf[warp], lane);
      } else {
        uint64_t thr = wl::list_get<KW>(L[m], k - 1);
        for (int c8 = 0; c8 < SCAN_P; c8 += 32) {
          const int col = c8 + lane;
          const uint64_t key = col < np ? make_key(dist[col], (uint32_t)lids[p0 + col]) : KEY_NONE;
          unsigned pend = __ballot_sync(wl::FULL, key < thr);
          while (pend) {
            const int src = __ffs(pend) - 1;
            pend &= pend - 1;
            const uint64_t cnd = __shfl_sync(wl::FULL, key, src);
            if (cnd < thr) {
              wl::list_insert<KW>(L[m], cnd, lane);
              thr = wl::list_get<KW>(L[m], k - 1);
            }
          }
        }
      }
    }
  }
  __syncthreads();  // an empty list ran no pass
#pragma unroll
  for (int m = 0; m < MW; ++m) {
    const int j = warp + NW * m;
    if (j >= nqe) continue;
    uint64_t* dst = partial + (((int64_t)s_q[j] * nprobe + pair_r[e0 + j]) * gridDim.y + blockIdx.y) * k;
#pragma unroll
    for (int s = 0; s < KW; ++s) {
      const int e = s * 32 + lane;
      if (e < k) dst[e] = L[m][s];
    }
  }
}

template <int METRIC, int KW, bool VEC>
mann_status launch_scan_t(cudaStream_t s, dim3 grid, const float* data, const int64_t* loff, const int32_t* lids,
                          const float* qs, int d, const int64_t* qoff, const int32_t* pair_q, const int32_t* pair_r,
                          const int64_t* choff, const int32_t* chunk_list, int nlist, int k, int nprobe,
                          uint64_t* partial) {
  auto kern = ivf_scan_kernel<METRIC, KW, VEC>;
  constexpr size_t smem = ScanSmem::BYTES;
  MANN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  kern<<<grid, SCAN_T, smem, s>>>(data, loff, lids, qs, d, qoff, pair_q, pair_r, choff, chunk_list, nlist, k, nprobe,
                                  partial);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

template <int METRIC>
mann_status launch_scan_m(cudaStream_t s, dim3 grid, bool vec, const float* data, const int64_t* loff,
                          const int32_t* lids, const float* qs, int d, const int64_t* qoff,
                          const int32_t* pair_q, const int32_t* pair_r, const int64_t* choff,
                          const int32_t* chunk_list, int nlist, int k, int nprobe, uint64_t* partial) {
  if (k <= 32)
    return vec ? launch_scan_t<METRIC, 1, true>(s, grid, data, loff, lids, qs, d, qoff, pair_q, pair_r, choff,
                                                chunk_list, nlist, k, nprobe, partial)
               : launch_scan_t<METRIC, 1, false>(s, grid, data, loff, lids, qs, d, qoff, pair_q, pair_r, choff,
                                                 chunk_list, nlist, k, nprobe, partial);
  return vec ? launch_scan_t<METRIC, 2, true>(s, grid, data, loff, lids, qs, d, qoff, pair_q, pair_r, choff,
                                              chunk_list, nlist, k, nprobe, partial)
             : launch_scan_t<METRIC, 2, false>(s, grid, data, loff, lids, qs, d, qoff, pair_q, pair_r, choff,
                                               chunk_list, nlist, k, nprobe, partial);
}

}  // namespace

// Scan of the given probes [nq][nprobe] (list ids, -1 = none): the points of
// the probed lists are read in place through list_ids; results as ids/dists
// [nq][k] (-1 / +inf padding).
mann_status ivf_scan_device(Context* ctx, cudaStream_t s, const float* data, int64_t n, int d,
                            int metric, const int64_t* loff, const int32_t* lids, int nlist,
                            const float* qs, int64_t nq, const int32_t* probes, int nprobe, int k,
                            int32_t* out_ids, float* out_dists) {
  (void)n;
  if (k < 1 || k > 64) return fail(MANN_EINVAL_ARG, "IVF search supports 1 <= k <= 64");
  if (nprobe < 1 || nprobe > 128) return fail(MANN_EINVAL_ARG, "IVF search supports 1 <= nprobe <= 128");
  if (metric == MANN_METRIC_COSINE) return fail(MANN_EINVAL_ARG, "IVF search: Euclidean / SqEuclidean");
  if (nq <= 0) return MANN_OK;
  unsigned* cnt = nullptr;
  int64_t *qoff = nullptr, *choff = nullptr;
  int32_t *pair_q = nullptr, *pair_r = nullptr;
  uint64_t *partial = nullptr, *keys = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_CNT, (size_t)2 * nlist + 4, &cnt));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_OFF, (size_t)2 * (nlist + 1), &qoff));
  choff = qoff + (nlist + 1);
  // chunks <= pairs / SCAN_Q + lists; blocks past the real count return at once
  const int64_t pairs = nq * nprobe;
  const int64_t max_chunks = ceil_div(pairs, SCAN_Q) + nlist;
  // Lists are cut into parts while the chunks fill the chip's six CTAs per SM
  // less than twice over: one CTA walks a long list alone (300 queries, 9 of 228
  // lists of 476 x 128, uneven: 544 us whole, 250 in parts; 4,356 queries, 3 of
  // 220 lists of 598 x 64: 450 and 363).
  const int64_t chunks = ceil_div(pairs, SCAN_Q) + std::min<int64_t>(pairs, nlist);
  const int parts = (int)std::max<int64_t>(
      1, std::min<int64_t>({8, 128 / nprobe, ceil_div((int64_t)12 * ctx->num_sms, std::max<int64_t>(chunks, 1))}));
  int32_t* chunk_list = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_PAIRS, (size_t)2 * nq * nprobe + (size_t)max_chunks, &pair_q));
  pair_r = pair_q + nq * nprobe;
  chunk_list = pair_r + nq * nprobe;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_PARTIAL, (size_t)nq * nprobe * parts * k, &partial));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_KEYS, (size_t)nq * k, &keys));
  MANN_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(unsigned) * (2 * nlist + 4), s));
  MANN_CUDA_TRY(cudaMemsetAsync(partial, 0xFF, sizeof(uint64_t) * nq * nprobe * parts * k, s));
  probe_count_kernel<<<(unsigned)ceil_div(nq * nprobe, 256), 256, 0, s>>>(probes, nq * nprobe, nlist, cnt);
  MANN_CHECK_LAUNCH();
  probe_scan_kernel<<<1, 1024, 0, s>>>(cnt, nlist, SCAN_Q, qoff, choff);
  MANN_CHECK_LAUNCH();
  probe_scatter_kernel<<<(unsigned)ceil_div(nq * nprobe, 256), 256, 0, s>>>(
      probes, nq, nprobe, nlist, qoff, choff, cnt + nlist, pair_q, pair_r, chunk_list);
  MANN_CHECK_LAUNCH();
  const bool vec = (d % 4) == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
  const dim3 grid((unsigned)max_chunks, (unsigned)parts);
  ctx->time_begin(s);
  if (metric == MANN_METRIC_EUCLIDEAN)
    MANN_TRY(launch_scan_m<MANN_METRIC_EUCLIDEAN>(s, grid, vec, data, loff, lids, qs, d, qoff, pair_q, pair_r,
                                                  choff, chunk_list, nlist, k, nprobe, partial));
  else
    MANN_TRY(launch_scan_m<MANN_METRIC_SQEUCLIDEAN>(s, grid, vec, data, loff, lids, qs, d, qoff, pair_q,
                                                    pair_r, choff, chunk_list, nlist, k, nprobe, partial));
  ctx->time_end(s);
  // (lists may have points in common: a point found in two of them is one result)
  MANN_TRY(launch_merge_lists(partial, nq, nprobe * parts, k, keys, s, true));
  MANN_TRY(launch_finish(keys, nq, k, k, -1, out_ids, out_dists, s));
  return MANN_OK;
}

// top-nprobe centroids of every query (TopKRouting on exact centroid distances)
mann_status ivf_route_device(Context* ctx, cudaStream_t s, const float* centroids, int nlist, int d,
                             int centroid_metric, const float* qs, int64_t nq, int nprobe,
                             int32_t* probes) {
  mann_knn_params p{};
  p.metric = centroid_metric;
  p.k = nprobe;
  // a short search is over in the FP32 form before the tensor-core form's
  // dozen launches are.  FP32 and AUTO at the line's sides, 4 probes, call by
  // call: 5e8 multiply-adds 100 and 174 us (953 queries x 4,096 x 128), 98 and
  // 183 (476 x 4,096 x 256), 127 and 215 (77 x 8,192 x 784); 1e9 181 and 235,
  // 142 and 185, 184 and 219; 2e9 262 and 179, 275 and 236, 257 and 220
  p.precision = (double)nq * nlist * d < 1e9 ? MANN_PREC_FP32 : MANN_PREC_AUTO;
  float* dd = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_ROUTE_D, (size_t)nq * nprobe, &dd));
  return exact_search_device(ctx, s, &p, centroids, nlist, qs, nq, d, -1, std::min(nprobe, nlist),
                             nprobe, probes, dd, nullptr);
}

mann_status ivf_build_device(Context* ctx, cudaStream_t s, const float* data, int64_t n, int d,
                             int nlist, int centroid_metric, int max_iters, double tol,
                             int64_t subsample, uint64_t seed, float* centroids, int64_t* offsets,
                             int32_t* ids, int* iters) {
  int32_t* assign = nullptr;
  int64_t *start = nullptr, *members = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_ASSIGN, (size_t)n, &assign));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_START, (size_t)2 * nlist, &start));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_MEMBERS, (size_t)n, &members));
  MANN_TRY(kmeans_fit_device(ctx, s, data, n, d, nlist, centroid_metric, 1, max_iters, tol, subsample,
                             seed, centroids, assign, iters));
  MANN_TRY(group_by_cluster_device(ctx, s, assign, n, nlist, start, start + nlist, members));
  ivf_lists_kernel<<<(unsigned)ceil_div(std::max<int64_t>(n, nlist + 1), 256), 256, 0, s>>>(
      start, members, nlist, n, offsets, ids);
  MANN_CHECK_LAUNCH();
  return MANN_OK;
}

}  // namespace mann

using namespace mann;

extern "C" {

mann_status mann_ivf_build(const mann_ivf_build_params* p, const float* data, int64_t n, int32_t d,
                           float* out_centroids, int64_t* out_offsets, int32_t* out_ids,
                           int32_t* out_iters) {
  clear_error();
  if (!p) return fail(MANN_EINVAL_ARG, "params must not be NULL");
  if (d <= 0) return fail(MANN_EINVAL_ARG, "Dataset must have at least one dimension");
  if (n <= 0) return fail(MANN_EINVAL_ARG, "Dataset must contain at least one point");
  if (p->nlist <= 0) return fail(MANN_EINVAL_ARG, "nlist must be positive");
  if (p->nlist > n) return fail(MANN_EINVAL_ARG, "Cannot fit " + std::to_string(p->nlist) +
                                                     " clusters with only " + std::to_string(n) + " points");
  if (p->centroid_metric != MANN_METRIC_EUCLIDEAN && p->centroid_metric != MANN_METRIC_SQEUCLIDEAN)
    return fail(MANN_EINVAL_ARG, "centroid metric: Euclidean or SqEuclidean");
  if (!data || !out_centroids || !out_offsets || !out_ids) return fail(MANN_EINVAL_ARG, "NULL buffer");
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr;
  int64_t* doff = nullptr;
  int32_t* dids = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_BASE, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)p->nlist * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_LOFF, (size_t)p->nlist + 1, &doff));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_LIDS, (size_t)n, &dids));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, data, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  int iters = 0;
  MANN_TRY(ivf_build_device(ctx, s, dx, n, d, p->nlist, p->centroid_metric,
                            p->kmeans_max_iters > 0 ? p->kmeans_max_iters : 25,
                            p->kmeans_tol > 0 ? p->kmeans_tol : 1e-4, p->kmeans_subsample, p->seed,
                            dc, doff, dids, &iters));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_centroids, dc, sizeof(float) * p->nlist * d, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_offsets, doff, sizeof(int64_t) * (p->nlist + 1), cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_ids, dids, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  if (out_iters) *out_iters = iters;
  return MANN_OK;
}

static mann_status ivf_check(const mann_knn_params* p, int32_t nprobe, const float* data, int64_t n,
                             int32_t d, int32_t nlist, const int64_t* offs, const int32_t* ids,
                             const float* qs, int64_t q) {
  if (!p) return fail(MANN_EINVAL_ARG, "params must not be NULL");
  if (d <= 0) return fail(MANN_EINVAL_ARG, "Dataset must have at least one dimension");
  if (n <= 0) return fail(MANN_EINVAL_ARG, "Dataset must contain at least one point");
  if (nlist <= 0 || nprobe <= 0) return fail(MANN_EINVAL_ARG, "nlist and nprobe must be positive");
  if (q < 0) return fail(MANN_EINVAL_ARG, "negative query count");
  if (!data || !offs || !ids || (q > 0 && !qs)) return fail(MANN_EINVAL_ARG, "NULL buffer");
  return MANN_OK;
}

mann_status mann_ivf_search_device(const mann_knn_params* p, int32_t nprobe, int32_t centroid_metric,
                                   const float* data, int64_t n, int32_t d, const float* centroids,
                                   int32_t nlist, const int64_t* list_offsets,
                                   const int32_t* list_ids, const float* queries, int64_t q,
                                   int32_t* out_ids, float* out_dists, void* stream) {
  clear_error();
  MANN_TRY(ivf_check(p, nprobe, data, n, d, nlist, list_offsets, list_ids, queries, q));
  if (p->k <= 0 || q == 0) return MANN_OK;
  nprobe = std::min(nprobe, nlist);  // clamp(nprobe, 1, nlist) (ivf_flat.jl:146)
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CallScope scope(ctx, s);
  int32_t* probes = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_IVF_PROBES, (size_t)q * nprobe, &probes));
  MANN_TRY(ivf_route_device(ctx, s, centroids, nlist, d, centroid_metric, queries, q, nprobe, probes));
  return ivf_scan_device(ctx, s, data, n, d, p->metric, list_offsets, list_ids, nlist, queries, q,
                         probes, nprobe, p->k, out_ids, out_dists);
}

mann_status mann_ivf_scan_device(const mann_knn_params* p, const int32_t* probes, int32_t nprobe,
                                 const float* data, int64_t n, int32_t d, int32_t nlist,
                                 const int64_t* list_offsets, const int32_t* list_ids,
                                 const float* queries, int64_t q, int32_t* out_ids,
                                 float* out_dists, void* stream) {
  clear_error();
  MANN_TRY(ivf_check(p, nprobe, data, n, d, nlist, list_offsets, list_ids, queries, q));
  if (!probes && q > 0) return fail(MANN_EINVAL_ARG, "NULL probes");
  if (p->k <= 0 || q == 0) return MANN_OK;
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CallScope scope(ctx, s);
  return ivf_scan_device(ctx, s, data, n, d, p->metric, list_offsets, list_ids, nlist, queries, q,
                         probes, nprobe, p->k, out_ids, out_dists);
}

mann_status mann_ivf_search(const mann_knn_params* p, int32_t nprobe, int32_t centroid_metric,
                            const float* data, int64_t n, int32_t d, const float* centroids,
                            int32_t nlist, const int64_t* list_offsets, const int32_t* list_ids,
                            const float* queries, int64_t q, int32_t* out_ids, float* out_dists) {
  clear_error();
  MANN_TRY(ivf_check(p, nprobe, data, n, d, nlist, list_offsets, list_ids, queries, q));
  if (p->k <= 0 || q == 0) return MANN_OK;
  nprobe = std::min(nprobe, nlist);
  Context* ctx = nullptr;
  MANN_TRY(get_context(&ctx));
  cudaStream_t s = ctx->stream;
  CallScope scope(ctx, s);
  float *dx = nullptr, *dc = nullptr, *dq = nullptr, *dd = nullptr;
  int64_t* doff = nullptr;
  int32_t *dids = nullptr, *dout = nullptr, *probes = nullptr;
  MANN_TRY(ctx->scratch_t(SLOT_BASE, (size_t)n * d, &dx));
  MANN_TRY(ctx->scratch_t(SLOT_KM_CENT, (size_t)nlist * d, &dc));
  MANN_TRY(ctx->scratch_t(SLOT_QUERIES, (size_t)q * d, &dq));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_LOFF, (size_t)nlist + 1, &doff));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_LIDS, (size_t)n, &dids));
  MANN_TRY(ctx->scratch_t(SLOT_OUT_IDS, (size_t)q * p->k, &dout));
  MANN_TRY(ctx->scratch_t(SLOT_OUT_DISTS, (size_t)q * p->k, &dd));
  MANN_TRY(ctx->scratch_t(SLOT_IVF_PROBES, (size_t)q * nprobe, &probes));
  MANN_CUDA_TRY(cudaMemcpyAsync(dx, data, sizeof(float) * n * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dc, centroids, sizeof(float) * nlist * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dq, queries, sizeof(float) * q * d, cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(doff, list_offsets, sizeof(int64_t) * (nlist + 1), cudaMemcpyHostToDevice, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(dids, list_ids, sizeof(int32_t) * n, cudaMemcpyHostToDevice, s));
  MANN_TRY(ivf_route_device(ctx, s, dc, nlist, d, centroid_metric, dq, q, nprobe, probes));
  MANN_TRY(ivf_scan_device(ctx, s, dx, n, d, p->metric, doff, dids, nlist, dq, q, probes, nprobe,
                           p->k, dout, dd));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_ids, dout, sizeof(int32_t) * q * p->k, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaMemcpyAsync(out_dists, dd, sizeof(float) * q * p->k, cudaMemcpyDeviceToHost, s));
  MANN_CUDA_TRY(cudaStreamSynchronize(s));
  return MANN_OK;
}

}  // extern "C"
