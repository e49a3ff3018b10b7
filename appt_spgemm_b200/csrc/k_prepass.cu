// Structural pre-pass, input validation, stable row binning and prefix scans.
//
// The pre-pass replaces k_flops (src/spgemm_engine.cuh:47-50) — one thread per
// row with a serial loop — by one warp per row reading the row's entries and
// the referenced B row bounds in parallel; it also records the output row's
// column span, which selects between hash tables and dense column windows.
// The binning replaces k_caps (src/spgemm_engine.cuh:51-57), which only chose
// between one 1024-slot shared table and a global arena.
#include <climits>

#include "kernels.h"

namespace spg {

// ---------------------------------------------------------------------------
// validation
// ---------------------------------------------------------------------------
__global__ void k_validate(MatView A, uint32_t* status) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if (warp == 0 && lane == 0) {
    if (A.rowptr[0] != 0 || (int64_t)A.rowptr[A.n] != A.nnz) report(status, DEV_ERR_INVALID_CSR);
  }
  for (int64_t i = warp; i < A.n; i += nwarps) {
    const int32_t s = A.rowptr[i], e = A.rowptr[i + 1];
    if (s < 0 || e < s || (int64_t)e > A.nnz) {
      if (lane == 0) report(status, DEV_ERR_INVALID_CSR);
      continue;
    }
    bool bad = false;
    for (Pos p = s + lane; p < (Pos)e; p += 32) {
      const int32_t j = A.col[p];
      if (j < 0 || j >= A.n) bad = true;
      if (p > (Pos)s && A.col[p - 1] >= j) bad = true;
    }
    if (__any_sync(0xffffffffu, bad) && lane == 0) report(status, DEV_ERR_INVALID_CSR);
  }
}

cudaError_t launch_validate(const MatView& A, uint32_t* status, cudaStream_t s) {
  const int threads = 256;
  int64_t warps = A.n > 0 ? A.n : 1;
  int64_t blocks = (warps * 32 + threads - 1) / threads;
  if (blocks > 65535 * 8) blocks = 65535 * 8;
  k_validate<<<(unsigned)blocks, threads, 0, s>>>(A, status);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// pre-pass: products and output column span per row (one warp per row)
// ---------------------------------------------------------------------------
// Every index is checked before it is used, so the kernel may run before the
// host has seen the validation verdict: a row that meets a row pointer or
// column outside its range gets f = −1, and the later kernels of the
// one-readback plan skip it.  It is also the validation of A (k_validate's checks,
// in the same read of A's rows): a violation sets DEV_ERR_INVALID_CSR in `status`.
__global__ void k_prepass(MatView A, MatView B, int64_t* __restrict__ f, int32_t* __restrict__ lo,
                          int32_t* __restrict__ hi, uint32_t* status, int64_t fcap) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if (warp == 0 && lane == 0 &&
      (A.rowptr[0] != 0 || (int64_t)A.rowptr[A.n] != A.nnz))
    report(status, DEV_ERR_INVALID_CSR);
  for (int64_t i = warp; i < A.n; i += nwarps) {
    int32_t s = A.rowptr[i], e = A.rowptr[i + 1];
    bool bad = s < 0 || e < s || (int64_t)e > A.nnz;
    if (bad) s = e = 0;
    long long prod = 0;
    int mn = INT_MAX, mx = -1;
    bool unsorted = false;
    // four entries per lane at a time, each step's loads issued together (a hub
    // row is a chain of them: R-MAT 2^15 113 -> 53 µs)
    for (Pos p0 = s + lane; p0 < (Pos)e; p0 += 128) {
      int32_t k[4], bs[4], be[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const Pos p = p0 + 32 * u;
        const bool in = p < (Pos)e;
        k[u] = in ? A.col[p] : 0;
        if (in && p > (Pos)s && A.col[p - 1] >= k[u]) unsorted = true;
        const bool ok = in && k[u] >= 0 && k[u] < B.n;
        bad = bad || (in && !ok);
        bs[u] = ok ? 0 : -1;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool ok = bs[u] == 0;
        bs[u] = ok ? B.rowptr[k[u]] : 0;
        be[u] = ok ? B.rowptr[k[u] + 1] : 0;
        if (bs[u] < 0 || be[u] < bs[u] || (int64_t)be[u] > B.nnz) {
          bad = true;
          bs[u] = be[u] = 0;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        prod += be[u] - bs[u];
        if (be[u] > bs[u]) {
          mn = min(mn, B.col[bs[u]]);
          mx = max(mx, B.col[be[u] - 1]);
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      prod += __shfl_xor_sync(0xffffffffu, prod, o);
      mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    bad = __any_sync(0xffffffffu, bad);
    unsorted = __any_sync(0xffffffffu, unsorted);
    if (lane == 0 && (bad || unsorted)) report(status, DEV_ERR_INVALID_CSR);
    if (lane == 0 && !bad && prod > fcap) report(status, DEV_ERR_SMALL_CAP);
    if (lane == 0) {
      f[i] = bad ? -1 : prod;
      lo[i] = bad ? INT_MAX : mn;
      hi[i] = bad ? -1 : mx;
    }
  }
}

cudaError_t launch_prepass(const MatView& A, const MatView& B, int64_t* f, int32_t* lo,
                           int32_t* hi, cudaStream_t s, uint32_t* status, int64_t fcap) {
  // no rows: the validation is rowptr[0] == 0 and nnz == 0 alone
  if (A.n == 0) return launch_validate(A, status, s);
  const int threads = 256;
  int64_t blocks = ((int64_t)A.n * 32 + threads - 1) / threads;
  if (blocks > 148 * 64) blocks = 148 * 64;
  k_prepass<<<(unsigned)blocks, threads, 0, s>>>(A, B, f, lo, hi, status, fcap);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// binning
// ---------------------------------------------------------------------------
// Two launches: the bin of every row, kept in a byte, with the bins' totals; then
// each block of rows reserves its places in the bins' lists and writes its rows
// there, in order within the block (the lists' order does not matter to the
// results).  A histogram per block with a scan over bins and blocks between the
// two, which kept the lists sorted, took 78 against 29 µs on a million rows: the
// scan ran in one CTA.
__global__ void __launch_bounds__(256) k_bin_count(BinSource src, uint8_t* __restrict__ bin,
                                                   unsigned long long* __restrict__ work,
                                                   const int* skip) {
  if (skip && *skip) return;
  __shared__ int cnt[kNumBins];
  __shared__ unsigned long long blocks, slices;
  if (threadIdx.x < kNumBins) cnt[threadIdx.x] = 0;
  if (threadIdx.x == 0) blocks = slices = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kBinRowsPerBlock;
  for (int t = threadIdx.x; t < kBinRowsPerBlock; t += blockDim.x) {
    const int64_t i = base + t;
    int b = i < src.n ? row_bin(src, (int)i) : -1;
    unsigned nb = 0;
    unsigned long long ns = 0;
    if (b == kHeavyBin || b == kPanelBin0) {
      if (src.mode == 0 || b == kPanelBin0) nb = (src.hi[i] >> 10) - (src.lo[i] >> 10) + 1;
      if (b == kPanelBin0) ns = (unsigned long long)nb * (src.arowptr[i + 1] - src.arowptr[i]);
      b += heavy_class(src.f[i]);
    }
    if (__any_sync(0xffffffffu, nb > 0)) {  // (an atomic per row: 30 µs on 2,000 heavy rows)
      nb = __reduce_add_sync(0xffffffffu, nb);
      for (int o = 16; o > 0; o >>= 1) ns += __shfl_xor_sync(0xffffffffu, ns, o);
      if ((threadIdx.x & 31) == 0) {
        atomicAdd(&blocks, (unsigned long long)nb);
        if (ns) atomicAdd(&slices, ns);
      }
    }
    const unsigned same = __match_any_sync(0xffffffffu, b);
    if (b < 0) continue;
    bin[i] = (uint8_t)b;
    if ((same & lanemask_lt()) == 0u) atomicAdd(&cnt[b], __popc(same));
  }
  __syncthreads();
  if (threadIdx.x < kNumBins && cnt[threadIdx.x])
    atomicAdd(&work[threadIdx.x], (unsigned long long)cnt[threadIdx.x]);
  if (threadIdx.x == 0 && blocks) atomicAdd(&work[kNumBins], blocks);
  if (threadIdx.x == 0 && slices) atomicAdd(&work[kNumBins + 1], slices);
}

__global__ void __launch_bounds__(256) k_bin_scatter(int64_t n, const uint8_t* __restrict__ bin,
                                                     unsigned long long* __restrict__ work,
                                                     int32_t* __restrict__ rows_out,
                                                     const int* skip) {
  if (skip && *skip) return;
  __shared__ int place[kNumBins];        // next place of each bin's rows of this block
  __shared__ int warp_cnt[8][kNumBins];
  __shared__ int cnt[kNumBins];
  const int tid = threadIdx.x, w = tid >> 5;
  constexpr int kPer = kBinRowsPerBlock / 256;
  if (tid < kNumBins) cnt[tid] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kBinRowsPerBlock;
  int b[kPer];
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    const int64_t i = base + u * 256 + tid;
    b[u] = i < n ? bin[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, b[u]);
    if (b[u] >= 0 && (same & lanemask_lt()) == 0u) atomicAdd(&cnt[b[u]], __popc(same));
  }
  __syncthreads();
  if (tid < kNumBins) {
    unsigned long long start = 0;
    for (int k = 0; k < tid; ++k) start += work[k];
    place[tid] = cnt[tid] ? (int)(start + atomicAdd(&work[kBinBack + tid],
                                                    (unsigned long long)cnt[tid]))
                          : 0;
  }
#pragma unroll
  for (int u = 0; u < kPer; ++u) {
    for (int t = tid; t < 8 * kNumBins; t += 256) (&warp_cnt[0][0])[t] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, b[u]);
    const int rank = __popc(same & lanemask_lt());
    if (b[u] >= 0 && rank == 0) warp_cnt[w][b[u]] = __popc(same);
    __syncthreads();
    if (b[u] >= 0) {
      int pos = place[b[u]] + rank;
      for (int ww = 0; ww < w; ++ww) pos += warp_cnt[ww][b[u]];
      rows_out[pos] = (int32_t)(base + u * 256 + tid);
    }
    __syncthreads();
    if (tid < kNumBins) {
      int add = 0;
      for (int ww = 0; ww < 8; ++ww) add += warp_cnt[ww][tid];
      place[tid] += add;
    }
    __syncthreads();  // the counts are zeroed next
  }
}

cudaError_t launch_bin_rows(const BinSource& src, uint8_t* bin, int64_t* work, int32_t* rows_out,
                            cudaStream_t s, const int* skip) {
  cudaError_t e = cudaMemsetAsync(work, 0, sizeof(int64_t) * kBinWork, s);
  const int nblocks = (int)((src.n + kBinRowsPerBlock - 1) / kBinRowsPerBlock);
  if (e != cudaSuccess || nblocks == 0) return e;
  k_bin_count<<<nblocks, 256, 0, s>>>(src, bin, (unsigned long long*)work, skip);
  SPG_COUNT_LAUNCH();
  k_bin_scatter<<<nblocks, 256, 0, s>>>(src.n, bin, (unsigned long long*)work, rows_out, skip);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// exclusive scans (three phases: tile sums, scan of tile sums, apply)
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ long long block_exclusive_scan64(long long v, long long* scratch,
                                                           long long* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  long long incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    long long t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  __syncthreads();
  if (lane == 31) scratch[w] = incl;
  __syncthreads();
  long long before = 0, all = 0;
  for (int i = 0; i < nw; ++i) {
    long long s = scratch[i];
    if (i < w) before += s;
    all += s;
  }
  *total = all;
  return before + incl - v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const int32_t* __restrict__ in,
                                                             int64_t n, long long* tile_sums) {
  __shared__ long long scratch[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += in[base + k];
  s = block_sum64(s, scratch);
  if (threadIdx.x == 0) tile_sums[blockIdx.x] = s;
}

__global__ void __launch_bounds__(1024) k_scan_tile_sums(long long* tile_sums, int64_t ntiles) {
  __shared__ long long scratch[32];
  __shared__ long long carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b = 0; b < ntiles; b += blockDim.x) {
    const int64_t idx = b + threadIdx.x;
    long long v = idx < ntiles ? tile_sums[idx] : 0;
    long long tot;
    long long ex = block_exclusive_scan64(v, scratch, &tot);
    if (idx < ntiles) tile_sums[idx] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile_sums[ntiles] = carry;
}

template <typename OutT>
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(const int32_t* __restrict__ in,
                                                             OutT* __restrict__ out, int64_t n,
                                                             const long long* tile_sums,
                                                             int64_t ntiles) {
  __shared__ long long scratch[32];
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int32_t v[kScanItems];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  long long tot;
  long long run = tile_sums[blockIdx.x] + block_exclusive_scan64(s, scratch, &tot);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = (OutT)run;
    run += v[k];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = (OutT)tile_sums[ntiles];
}

// One tile (n <= kScanTile): the whole scan in one launch.
template <typename OutT>
__global__ void __launch_bounds__(kScanThreads) k_scan_single(const int32_t* __restrict__ in,
                                                              OutT* __restrict__ out, int64_t n) {
  __shared__ long long scratch[32];
  const int64_t base = (int64_t)threadIdx.x * kScanItems;
  int32_t v[kScanItems];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? in[base + k] : 0;
    s += v[k];
  }
  long long tot;
  long long run = block_exclusive_scan64(s, scratch, &tot);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = (OutT)run;
    run += v[k];
  }
  if (threadIdx.x == 0) out[n] = (OutT)tot;
}

// Row pointers of C with the row statistics, in two launches (one tile: one).
// The first takes a follower's count from its run's first row, sums each tile and
// gathers the statistics; in the second each tile sums the tiles before it.
// (A scan of three launches, the run counts and the statistics as launches of
// their own took 58 against 19 µs on a million rows.)
//   stats: Σ products, max products, max row count, max span, Σ row counts, the
//     two device status words, so that one copy brings a plan's verdict, and the
//     rows looked at for crowding
struct RowStats {
  unsigned long long sf = 0, mf = 0, mc = 0, ms = 0;
  unsigned long long crowd = 0;  // rows looked at, and 2^32 times those found crowded
  __device__ __forceinline__ void add(unsigned long long f, int c, int lo, int hi) {
    sf += f;
    mf = f > mf ? f : mf;
    mc = (unsigned)c > mc ? (unsigned)c : mc;
    const unsigned long long span = hi >= lo ? (unsigned long long)((long long)hi - lo + 1) : 0;
    ms = span > ms ? span : ms;
  }
  // per warp, then one atomic each per CTA (of one CTA: plain stores)
  __device__ __forceinline__ void store(unsigned long long* stats, bool single) {
    __shared__ unsigned long long acc[5];
    if (threadIdx.x < 5) acc[threadIdx.x] = 0;
    __syncthreads();
    if (crowd) atomicAdd(&acc[4], crowd);
    for (int o = 16; o > 0; o >>= 1) {
      sf += __shfl_xor_sync(0xffffffffu, sf, o);
      const unsigned long long a = __shfl_xor_sync(0xffffffffu, mf, o);
      const unsigned long long b = __shfl_xor_sync(0xffffffffu, mc, o);
      const unsigned long long c = __shfl_xor_sync(0xffffffffu, ms, o);
      mf = a > mf ? a : mf;
      mc = b > mc ? b : mc;
      ms = c > ms ? c : ms;
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&acc[0], sf);
      atomicMax(&acc[1], mf);
      atomicMax(&acc[2], mc);
      atomicMax(&acc[3], ms);
    }
    __syncthreads();
    if (single) {
      if (threadIdx.x < 4) stats[threadIdx.x] = acc[threadIdx.x];
      if (threadIdx.x == 4) stats[6] = acc[4];
    } else if (threadIdx.x == 0) {
      if (acc[4]) atomicAdd(&stats[6], acc[4]);
      atomicAdd(&stats[0], acc[0]);
      atomicMax(&stats[1], acc[1]);
      atomicMax(&stats[2], acc[2]);
      atomicMax(&stats[3], acc[3]);
    }
  }
};

// A sorted row looked at: 1, and 2^32 more when six of eight of its
// columns lie within 2^-kCrowdLog2 of its span.  (Up to kCrowdMin products fit a bucket.)
__device__ __noinline__ unsigned long long crowd_look(const MatView& A, const MatView& B,
                                                      int64_t i, int64_t f, int cnt, int32_t lo,
                                                      int32_t hi) {
  if (f <= kCrowdMin || f > kSortMaxProducts || 2 * f > kSortMaxMerge2 * cnt) return 0;
  const int32_t ps = A.rowptr[i], len = A.rowptr[i + 1] - ps, window = (hi - lo) >> kCrowdLog2;
  int32_t c[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) c[u] = crowd_column(A.col + ps, len, B.rowptr, B.col, u);
  int most = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    int near = 0;
#pragma unroll
    for (int v = 0; v < 8; ++v) near += c[v] >= c[u] && c[v] - c[u] <= window;
    most = max(most, c[u] < 0 ? 0 : near);
  }
  return most >= 6 ? 1ull << 32 | 1ull : 1ull;
}

template <bool SINGLE>
__global__ void __launch_bounds__(kScanThreads) k_count_tiles(
    MatView A, MatView B, int32_t* cnt, const uint8_t* __restrict__ lead, const int64_t* __restrict__ f,
    const int32_t* __restrict__ lo, const int32_t* __restrict__ hi, int64_t n,
    int64_t* __restrict__ rowptr, long long* __restrict__ tile_sums,
    unsigned long long* __restrict__ stats, const uint32_t* __restrict__ status) {
  __shared__ long long scratch[32];
  const int64_t tile = (int64_t)blockIdx.x * kScanTile;
  RowStats st;
  if (SINGLE) {
    const int64_t base = tile + (int64_t)threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    long long s = 0;
    if (!lead && base + kScanItems <= n) {  // (the arrays are 16-byte aligned)
      int32_t l[kScanItems], h[kScanItems];
      int64_t p[kScanItems];
#pragma unroll
      for (int k = 0; k < kScanItems; k += 4) {
        *(int4*)(v + k) = *(const int4*)(cnt + base + k);
        *(int4*)(l + k) = *(const int4*)(lo + base + k);
        *(int4*)(h + k) = *(const int4*)(hi + base + k);
        *(longlong2*)(p + k) = *(const longlong2*)(f + base + k);
        *(longlong2*)(p + k + 2) = *(const longlong2*)(f + base + k + 2);
      }
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        s += v[k];
        st.add((unsigned long long)p[k], v[k], l[k], h[k]);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; ++k) {
        const int64_t i = base + k;
        v[k] = 0;
        if (i >= n) continue;
        v[k] = cnt[lead && lead[i] ? i - lead[i] : i];
        if (lead && lead[i]) cnt[i] = v[k];
        s += v[k];
        st.add((unsigned long long)f[i], v[k], lo[i], hi[i]);
      }
    }
    long long tot;
    long long run = block_exclusive_scan64(s, scratch, &tot);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      if (base + k < n) rowptr[base + k] = run;
      run += v[k];
    }
    if (threadIdx.x == 0) {
      rowptr[n] = tot;
      stats[4] = (unsigned long long)tot;
      stats[5] = status[0] | (unsigned long long)status[1] << 32;
    }
  } else {
    long long s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {  // coalesced: the order does not matter here
      const int64_t i = tile + k * kScanThreads + threadIdx.x;
      if (i >= n) continue;
      const int d = lead ? lead[i] : 0;
      const int32_t c = cnt[i - d];
      if (d) cnt[i] = c;
      s += c;
      st.add((unsigned long long)f[i], c, lo[i], hi[i]);
      // (eight threads of the tile look at one row each, so that it costs them one chain
      // of loads; a single tile's rows are not looked at)
      if ((threadIdx.x & 63) == 32 && (threadIdx.x >> 6) == k)
        st.crowd = crowd_look(A, B, i, f[i], c, lo[i], hi[i]);
    }
    s = block_sum64(s, scratch);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = s;
  }
  st.store(stats, SINGLE);
}

__global__ void __launch_bounds__(kScanThreads) k_count_apply(const int32_t* __restrict__ cnt,
                                                              int64_t n, int64_t ntiles,
                                                              const long long* __restrict__ tiles,
                                                              int64_t* __restrict__ rowptr,
                                                              unsigned long long* stats,
                                                              const uint32_t* __restrict__ status) {
  __shared__ long long scratch[32];
  long long before = 0;
  for (int64_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) before += tiles[t];
  before = block_sum64(before, scratch);
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int32_t v[kScanItems];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = (base + k < n) ? cnt[base + k] : 0;
    s += v[k];
  }
  long long tot;
  long long run = before + block_exclusive_scan64(s, scratch, &tot);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) rowptr[base + k] = run;
    run += v[k];
  }
  if (blockIdx.x == ntiles - 1 && threadIdx.x == 0) {
    rowptr[n] = before + tot;
    stats[4] = (unsigned long long)(before + tot);
    stats[5] = status[0] | (unsigned long long)status[1] << 32;
  }
}

// (beyond this many tiles, 16.8 M rows, the tiles before a tile are scanned by
// the three-launch scan)
constexpr int64_t kMaxCountTiles = 4096;

cudaError_t launch_row_pointers(const MatView& A, const MatView& B, int32_t* cnt,
                                const uint8_t* lead, const int64_t* f,
                                const int32_t* lo, const int32_t* hi, int64_t n, int64_t* rowptr,
                                unsigned long long* stats, const uint32_t* status, void* tmp,
                                cudaStream_t s) {
  long long* tiles = (long long*)tmp;
  const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
  if (ntiles == 1) {
    k_count_tiles<true><<<1, kScanThreads, 0, s>>>(A, B, cnt, lead, f, lo, hi, n, rowptr, tiles, stats,
                                                   status);
    SPG_COUNT_LAUNCH();
    return cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(stats, 0, sizeof(unsigned long long) * kRowStats, s);
  if (e != cudaSuccess) return e;
  if (n <= 0) {
    e = cudaMemcpyAsync(stats + 5, status, 2 * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s);
    return e != cudaSuccess ? e : cudaMemsetAsync(rowptr, 0, sizeof(int64_t), s);
  }
  k_count_tiles<false><<<(unsigned)ntiles, kScanThreads, 0, s>>>(A, B, cnt, lead, f, lo, hi, n, rowptr,
                                                                 tiles, stats, status);
  SPG_COUNT_LAUNCH();
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (ntiles > kMaxCountTiles) {
    if ((e = launch_scan_i32_i64(cnt, rowptr, n, tmp, s)) != cudaSuccess) return e;
    e = cudaMemcpyAsync(stats + 4, rowptr + n, sizeof(int64_t), cudaMemcpyDeviceToDevice, s);
    return e != cudaSuccess ? e
                            : cudaMemcpyAsync(stats + 5, status, 2 * sizeof(uint32_t),
                                              cudaMemcpyDeviceToDevice, s);
  }
  k_count_apply<<<(unsigned)ntiles, kScanThreads, 0, s>>>(cnt, n, ntiles, tiles, rowptr, stats,
                                                          status);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

size_t scan_tmp_bytes(int64_t n) {
  int64_t ntiles = (n + kScanTile - 1) / kScanTile;
  return sizeof(long long) * (size_t)(ntiles + 1);
}

template <typename OutT>
static cudaError_t scan_impl(const int32_t* in, OutT* out, int64_t n, void* tmp, cudaStream_t s) {
  long long* tile = (long long*)tmp;
  const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
  if (ntiles == 0) return cudaMemsetAsync(out, 0, sizeof(OutT), s);
  if (ntiles == 1) {
    k_scan_single<OutT><<<1, kScanThreads, 0, s>>>(in, out, n);
    SPG_COUNT_LAUNCH();
    return cudaGetLastError();
  }
  k_scan_tiles<<<(unsigned)ntiles, kScanThreads, 0, s>>>(in, n, tile);
  SPG_COUNT_LAUNCH();
  k_scan_tile_sums<<<1, 1024, 0, s>>>(tile, ntiles);
  SPG_COUNT_LAUNCH();
  k_scan_apply<OutT><<<(unsigned)ntiles, kScanThreads, 0, s>>>(in, out, n, tile, ntiles);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_scan_i32_i64(const int32_t* in, int64_t* out, int64_t n, void* tmp,
                                cudaStream_t s) {
  return scan_impl<int64_t>(in, out, n, tmp, s);
}
cudaError_t launch_scan_i32_i32(const int32_t* in, int32_t* out, int64_t n, void* tmp,
                                cudaStream_t s) {
  return scan_impl<int32_t>(in, out, n, tmp, s);
}

// ---------------------------------------------------------------------------
// column histogram and structural descriptors
// ---------------------------------------------------------------------------
__global__ void k_col_count(MatView A, int32_t* __restrict__ cnt) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < A.nnz; p += stride) {
    const int32_t k = A.col[p];
    if (k >= 0 && k < A.n) atomicAdd(&cnt[k], 1);  // others: invalid input, never counted
  }
}

cudaError_t launch_col_count(const MatView& A, int32_t* cnt, cudaStream_t s) {
  if (A.nnz == 0) return cudaSuccess;
  int64_t blocks = (A.nnz + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_col_count<<<(unsigned)blocks, 256, 0, s>>>(A, cnt);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

__global__ void k_describe(MatView A, const int32_t* __restrict__ colcount, DescAccum* acc) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long deg2 = 0, paa = 0, paat = 0, sym = 0;
  int maxdeg = 0, maxcol = 0, band = 0;
  for (int64_t i = warp; i < A.n; i += nwarps) {
    const int32_t s = A.rowptr[i], e = A.rowptr[i + 1];
    if (lane == 0) {
      deg2 += (unsigned long long)(e - s) * (unsigned long long)(e - s);
      maxdeg = max(maxdeg, e - s);
      const unsigned long long c = colcount[i];
      paat += c * c;
      maxcol = max(maxcol, (int)c);
    }
    for (Pos p = s + lane; p < (Pos)e; p += 32) {
      const int32_t j = A.col[p];
      paa += (unsigned long long)(A.rowptr[j + 1] - A.rowptr[j]);
      band = max(band, (int)(j > i ? j - i : i - j));
      // is (j, i) present?  binary search for i in row j
      int32_t lo = A.rowptr[j], hi = A.rowptr[j + 1];
      while (lo < hi) {
        const int32_t mid = lo + ((hi - lo) >> 1);  // (lo + hi may exceed 2^31)
        if (A.col[mid] < i) lo = mid + 1; else hi = mid;
      }
      if (lo < A.rowptr[j + 1] && A.col[lo] == i) ++sym;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    deg2 += __shfl_xor_sync(0xffffffffu, deg2, o);
    paa += __shfl_xor_sync(0xffffffffu, paa, o);
    paat += __shfl_xor_sync(0xffffffffu, paat, o);
    sym += __shfl_xor_sync(0xffffffffu, sym, o);
    maxdeg = max(maxdeg, __shfl_xor_sync(0xffffffffu, maxdeg, o));
    maxcol = max(maxcol, __shfl_xor_sync(0xffffffffu, maxcol, o));
    band = max(band, __shfl_xor_sync(0xffffffffu, band, o));
  }
  if (lane == 0) {
    atomicAdd(&acc->sum_deg2, deg2);
    atomicAdd(&acc->prod_aa, paa);
    atomicAdd(&acc->prod_aat, paat);
    atomicAdd(&acc->sym_hits, sym);
    atomicMax(&acc->max_deg, maxdeg);
    atomicMax(&acc->max_col_deg, maxcol);
    atomicMax(&acc->bandwidth, band);
  }
}

cudaError_t launch_describe(const MatView& A, const int32_t* colcount, DescAccum* acc,
                            cudaStream_t s) {
  if (A.n == 0) return cudaSuccess;
  int64_t blocks = ((int64_t)A.n * 32 + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  k_describe<<<(unsigned)blocks, 256, 0, s>>>(A, colcount, acc);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace spg
