// Runs of shifted rows: consecutive rows of C whose products have the same
// places, each a copy of the row before with every column one further on.
//
// On a structured grid, row i + 1 of A is row i shifted by one column wherever
// both points have the same neighbours, and so are the rows of B it reads:
// product for product, row i + 1 of C is row i shifted.  The hash kernels found
// the place of every one of the 729 products of a 27-point row by a probe (920
// SM cycles a row on the 96³ grid).  Here a run's places are found once, for
// its first row, and its other rows only multiply and add:
//  - the pre-pass marks the rows of A that are their predecessor shifted by one;
//    a row of C follows its predecessor when its row of A and every row of B
//    that it reads do (k_find_runs, which cuts the runs at 256 rows);
//  - only the first row of a run goes through the symbolic phase (the others
//    take its count), and the numeric phase takes a run per CTA;
//  - the CTA lists the products of each output entry in k order (a bitmap of
//    the span ranks the columns, one warp places the products), then takes 32
//    rows at a time, a lane per row: the rows of B that they read lie side by
//    side in memory (k, k + 1, … of the same length) and are copied to shared
//    memory once, and an output entry of all 32 rows is one walk over its list,
//    the same for every lane.  Sums start from 0.0 and take the products in k
//    order, so the values are those of the other kernels, bit for bit.
// 27-point stencil 96³, A·A: numeric phase 2.99 -> 1.42 ms (runs 1.26 ms, the
// rows at the grid's faces in the hash kernels), symbolic 1.04 -> 0.09 ms, call
// 4.51 -> 1.88 ms; 5-point grid 1009²: call 1.27 -> 0.38 ms.  The run kernel
// issues on 44% of cycles and moves wavefronts on 56% (two 64-bit shared-memory
// loads a product), with two CTAs (16 warps) per SM, 109 KB each: latency is
// what is left.  Measured and not kept (against 1.11 ms for the largest launch in
// those runs): two entries' sums at a time 1.16, entries drawn by list length 1.16,
// neighbouring runs to one CTA 1.16 ms;
// the entries shared out by list length, or 16 warps a team (32 per SM): no change.
#include <algorithm>
#include <climits>

#include "kernels.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kRunOut = 8;                    // output entries a warp stages at a time
constexpr int kStageRow = 33;                 // doubles between staged entries (32 rows)
constexpr int kMaxLen = 126;                  // entries of A's row

// A launch's CTA by team size: threads, and the limits of its runs' rows.  The
// runs of few entries a row (teams of one warp) have small CTAs, five per SM
// instead of two: a run's own steps (its entries, its rows of B, the check of
// its columns) are a chain of loads that only other CTAs hide.  5-point grid
// 1009²: 145 -> 127 µs.
template <int T>
struct RunShape {
  static constexpr int kThreads = T == 1 ? 128 : 256;
  static constexpr int kWarps = kThreads / 32, kTeams = kWarps / T;
  static constexpr int kTeamBuffer = T == 1 ? kRunSmallBuffer : kRunBuffer * T / 8;  // doubles
  static constexpr int kProducts = T == 1 ? kRunSmallProducts : kRunMaxProducts;
  static constexpr int kSpan = T == 1 ? kRunSmallSpan : kRunMaxSpan;
  static constexpr int kList = 2 * kProducts;  // lists start at even places
  static constexpr size_t kBufferBytes = (size_t)kTeams * kTeamBuffer * 8;
  static constexpr size_t kStageBytes = (size_t)kWarps * kRunOut * kStageRow * 8;
  // team buffers (also the bitmap while the places are found), the staging area
  // (also the products then), the lists, their starts, the output columns and the
  // products' columns
  static constexpr size_t kSmem = kBufferBytes + kStageBytes + (size_t)kList * 4 +
                                  (size_t)kProducts * 12;
  static_assert(kStageBytes >= (size_t)kProducts * 10, "products fit the staging area");
  static_assert(kBufferBytes >= (size_t)kSpan / 32 * 5 + 64, "bitmap fits");
};

__device__ __forceinline__ void copy_async8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src));
}

// Shared-memory loads by 32-bit address: the operand addresses are sums of a
// lane's base and an offset from a list (volatile: they stay between the barriers).
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ double lds_f64(uint32_t addr) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint2 lds_pair(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}

__device__ __forceinline__ void team_sync(int team, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(threads) : "memory");
}

// Consecutive rows of B that a row of C reads: `rows` of them, of `len` entries,
// from entry `src` for the run's first row; at `off` in the team's buffer.
struct RowGroup {
  int src;
  uint16_t off, rows, len, t;  // t: the group's first entry of A's row
};

template <int T>  // warps per team of 32 rows
__global__ void __launch_bounds__(RunShape<T>::kThreads, T == 1 ? 5 : 2) k_runs(RowArgs a) {
  using S = RunShape<T>;
  constexpr int kRunThreads = S::kThreads, kRunWarps = S::kWarps, kTeams = S::kTeams;
  constexpr int kTeamThreads = T * 32, kMaxProducts = S::kProducts;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ RowGroup groups[kMaxLen];
  __shared__ int t_src[kMaxLen], t_rel[kMaxLen];
  __shared__ uint16_t t_len[kMaxLen], t_off[kMaxLen], t_first[kMaxLen + 2];
  __shared__ int scratch[33];
  __shared__ int s_groups, s_distinct, s_stride;
  double* buffer = (double*)smem;
  double* stage_all = buffer + kTeams * S::kTeamBuffer;
  uint32_t* list = (uint32_t*)((unsigned char*)stage_all + S::kStageBytes);
  uint32_t* start = list + S::kList;  // an output entry's first place << 8 | products
  int* out_col = (int*)(start + kMaxProducts);  // its column, from the row's index
  int* prod_col = out_col + kMaxProducts;       // the products' columns, likewise
  // while the places are found
  uint32_t* bitmap = (uint32_t*)buffer;
  uint32_t* desc = (uint32_t*)stage_all;  // per product: where its operands will lie
  int* cur = (int*)(desc + kMaxProducts);
  uint16_t* rank = (uint16_t*)(cur + kMaxProducts);

  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int team = wid / T, tw = wid % T, team_tid = tid % kTeamThreads;
  double* buf = buffer + (size_t)team * S::kTeamBuffer;
  double* stage = stage_all + (size_t)wid * kRunOut * kStageRow;
  int have_len = -1, have_m = 0;  // the lists at hand are of a row of this many entries

  for (int r = blockIdx.x; r < a.nrows; r += gridDim.x) {
    const int row0 = a.rows[r];
    const int nrun = a.runlen[row0];
    const int32_t ps = a.A.rowptr[row0];
    const int len_a = a.A.rowptr[row0 + 1] - ps;
    const int lo = a.lo[row0];
    const int span = a.hi[row0] - lo + 1;
    const int m = a.cnt_in[row0];
    const int stride_a = len_a | 1;
    // (what the pre-pass has checked; a plan whose structure was changed since
    // must not write past the arrays)
    if (len_a > kMaxLen || m > kMaxProducts || span > S::kSpan) {
      if (tid == 0) report(a.status, DEV_ERR_OVERFLOW);
      continue;
    }

    __syncthreads();  // the previous run is finished
    bool differ = len_a != have_len || m != have_m;
    for (int t = tid; t < len_a; t += kRunThreads) {
      const int32_t k = a.A.col[ps + t];
      const int src = a.B.rowptr[k], len = a.B.rowptr[k + 1] - src;
      differ = differ || k - row0 != t_rel[t] || len != t_len[t];
      t_src[t] = src;
      t_rel[t] = k - row0;
      t_len[t] = (uint16_t)min(len, 65535);
    }
    bool same = !__syncthreads_or(differ);

    int ng = s_groups, stride = s_stride;
    auto load_tile = [&](int row_t, int nt) {  // rows row_t … of the run, nt of them
      const double* av = a.A.val + ps + (int64_t)row_t * len_a;
      if (len_a == stride_a) {
        for (int i = team_tid; i < nt * len_a; i += kTeamThreads) copy_async8(buf + i, av + i);
      } else {
        for (int j = tw; j < nt; j += T)
          for (int t = lane; t < len_a; t += 32)
            copy_async8(buf + j * stride_a + t, av + (int64_t)j * len_a + t);
      }
      for (int g = 0; g < ng; ++g) {
        const RowGroup gr = groups[g];
        const int rows = gr.rows + nt - 1, len = gr.len;
        const double* bv = a.B.val + (int64_t)gr.src + (int64_t)row_t * len;
        double* dst = buf + gr.off;
        if (len == stride) {  // one piece
          const int n = rows * len;
          for (int i = team_tid; i < n; i += kTeamThreads) copy_async8(dst + i, bv + i);
        } else if (len > 16) {
          for (int j = tw; j < rows; j += T)
            for (int q = lane; q < len; q += 32)
              copy_async8(dst + j * stride + q, bv + (int64_t)j * len + q);
        } else {  // several short rows per warp
          const int lg = len > 1 ? 32 - __clz(len - 1) : 0;
          const int q = lane & ((1 << lg) - 1);
          if (q < len)
            for (int j = tw << (5 - lg) | lane >> lg; j < rows; j += T << (5 - lg))
              copy_async8(dst + j * stride + q, bv + (int64_t)j * len + q);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int row_t = team * 32;

    if (same) {
      // the lists of the last run hold if the rows of B have its columns too;
      // the first rows' operands are on their way meanwhile
      for (int g = tid; g < ng; g += kRunThreads) groups[g].src = t_src[groups[g].t];
      __syncthreads();
      if (row_t < nrun) load_tile(row_t, min(32, nrun - row_t));
      differ = false;
      for (int t = wid; t < len_a; t += kRunWarps) {
        const int e0 = t_first[t], len = t_len[t];
        for (int q = lane; q < len; q += 32)
          differ = differ || a.B.col[t_src[t] + q] - row0 != prod_col[e0 + q];
      }
      same = !__syncthreads_or(differ);
      if (!same) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
    }
    if (!same) {
      have_len = -1;
      const int words = (span + 31) >> 5, words4 = (words + 3) >> 2;
      for (int i = tid; i < words4 * 4; i += kRunThreads) bitmap[i] = 0u;
      for (int i = tid; i < m; i += kRunThreads) cur[i] = 0;
      if (tid == 0) {
        int st = 0, n = 0, e = 0, off = 32 * stride_a, t0 = 0;
        for (int t = 0; t < len_a; ++t) st = max(st, t_len[t] | 1);
        for (int t = 0; t < len_a; ++t) {
          if (t == 0 || t_rel[t] != t_rel[t - 1] + 1) {
            t0 = t;
            groups[n].src = t_src[t];
            groups[n].len = t_len[t];
            groups[n].off = (uint16_t)off;
            groups[n].rows = 0;
            groups[n].t = (uint16_t)t;
            off += 31 * st;
            ++n;
          }
          t_off[t] = (uint16_t)(groups[n - 1].off + (t - t0) * st);
          off += st;
          ++groups[n - 1].rows;
          t_first[t] = (uint16_t)e;
          e += t_len[t];
          if (off > S::kTeamBuffer || e > kMaxProducts) {  // as above
            n = -1;
            break;
          }
        }
        if (n >= 0) t_first[len_a] = (uint16_t)e;
        s_groups = n;
        s_stride = st;
      }
      __syncthreads();
      ng = s_groups;
      stride = s_stride;
      if (ng < 0) {
        if (tid == 0) report(a.status, DEV_ERR_OVERFLOW);
        continue;
      }
      const int f = t_first[len_a];

      // 1. the products: columns, operand places, and the bitmap of the columns
      for (int t = wid; t < len_a; t += kRunWarps) {
        const int e0 = t_first[t], len = t_len[t];
        for (int q = lane; q < len; q += 32) {
          const unsigned x = min((unsigned)(a.B.col[t_src[t] + q] - lo), (unsigned)span - 1u);
          prod_col[e0 + q] = (int)x + lo - row0;
          desc[e0 + q] = (uint32_t)(t_off[t] + q) << 3 | (uint32_t)t << 20;  // bytes, t · 8 << 17
          atomicOr(&bitmap[x >> 5], 1u << (x & 31));
        }
      }
      __syncthreads();
      // 2. ranks of the columns
      int* pre4 = (int*)(bitmap + words4 * 4);
      {
        const int per = (words4 + kRunThreads - 1) / kRunThreads;
        const int gb = min(words4, tid * per), ge = min(words4, gb + per);
        int local = 0;
        for (int g = gb; g < ge; ++g)
          local += __popc(bitmap[4 * g]) + __popc(bitmap[4 * g + 1]) + __popc(bitmap[4 * g + 2]) +
                   __popc(bitmap[4 * g + 3]);
        int tot;
        int run = block_exclusive_scan(local, scratch, &tot);
        for (int g = gb; g < ge; ++g) {
          pre4[g] = run;
          run += __popc(bitmap[4 * g]) + __popc(bitmap[4 * g + 1]) + __popc(bitmap[4 * g + 2]) +
                 __popc(bitmap[4 * g + 3]);
        }
        if (tid == 0) s_distinct = tot;
      }
      __syncthreads();
      if (s_distinct != m) {
        if (tid == 0) report(a.status, DEV_ERR_OVERFLOW);
        continue;
      }
      for (int e = tid; e < f; e += kRunThreads) {
        const int c = prod_col[e];
        const unsigned x = (unsigned)(c + row0 - lo);
        const int i = (int)(x >> 5);
        int k = pre4[i >> 2];
        for (int w = i & ~3; w < i; ++w) k += __popc(bitmap[w]);
        k += __popc(bitmap[i] & ((1u << (x & 31)) - 1u));
        rank[e] = (uint16_t)k;
        out_col[k] = c;
        atomicAdd(&cur[k], 1);
      }
      __syncthreads();
      // 3. the lists' places
      {
        const int per = (m + kRunThreads - 1) / kRunThreads;
        const int b = min(m, tid * per), e = min(m, b + per);
        int local = 0;
        for (int i = b; i < e; ++i) local += (cur[i] + 1) & ~1;
        int tot;
        int run = block_exclusive_scan(local, scratch, &tot);
        for (int i = b; i < e; ++i) {
          const int n = cur[i];
          start[i] = (uint32_t)run << 8 | (uint32_t)n;
          cur[i] = run;
          run += (n + 1) & ~1;
        }
      }
      __syncthreads();
      // 4. one warp places the products in k order, while the others copy the first
      // rows' operands
      if (row_t < nrun) load_tile(row_t, min(32, nrun - row_t));
      if (wid == 0) {
        for (int e0 = 0; e0 < f; e0 += 32) {
          const int e = e0 + lane;
          const int k = e < f ? (int)rank[e] : -1 - lane;
          const unsigned peers = __match_any_sync(kFull, k) ;
          if (e < f) list[cur[k] + __popc(peers & lanemask_lt())] = desc[e];
          __syncwarp();
          if (e < f && (peers & lanemask_lt()) == 0u) cur[k] += __popc(peers);
          __syncwarp();
        }
      }
      have_len = len_a;
      have_m = m;
      __syncthreads();  // the lists are complete, the staging area is free
    }

    // 5. 32 rows at a time, a lane per row
    for (; row_t < nrun; row_t += 32 * kTeams) {
      const int nt = min(32, nrun - row_t);
      asm volatile("cp.async.wait_all;" ::: "memory");
      team_sync(team, kTeamThreads);
      const uint32_t pa = smem_addr(buf + lane * stride_a), pb = smem_addr(buf + lane * stride);
      const uint32_t list0 = smem_addr(list);
      const int64_t base = a.rowptr[row0 + row_t];
      for (int k0 = tw * kRunOut; k0 < m; k0 += T * kRunOut) {
        const int nk = min(kRunOut, m - k0);
        for (int k = 0; k < nk; ++k) {
          const uint32_t se = start[k0 + k];
          uint32_t l = list0 + (se >> 8) * 4u;
          int n = (int)(se & 255u);
          double sum = 0.0;
          for (; n >= 4; n -= 4, l += 16) {
            const uint2 d = lds_pair(l), e = lds_pair(l + 8);
            const double a0 = lds_f64(pa + (d.x >> 17)), b0 = lds_f64(pb + (d.x & 0x1ffffu));
            const double a1 = lds_f64(pa + (d.y >> 17)), b1 = lds_f64(pb + (d.y & 0x1ffffu));
            const double a2 = lds_f64(pa + (e.x >> 17)), b2 = lds_f64(pb + (e.x & 0x1ffffu));
            const double a3 = lds_f64(pa + (e.y >> 17)), b3 = lds_f64(pb + (e.y & 0x1ffffu));
            sum = __dadd_rn(sum, __dmul_rn(a0, b0));
            sum = __dadd_rn(sum, __dmul_rn(a1, b1));
            sum = __dadd_rn(sum, __dmul_rn(a2, b2));
            sum = __dadd_rn(sum, __dmul_rn(a3, b3));
          }
          if (n & 2) {
            const uint2 d = lds_pair(l);
            l += 8;
            const double a0 = lds_f64(pa + (d.x >> 17)), b0 = lds_f64(pb + (d.x & 0x1ffffu));
            const double a1 = lds_f64(pa + (d.y >> 17)), b1 = lds_f64(pb + (d.y & 0x1ffffu));
            sum = __dadd_rn(sum, __dmul_rn(a0, b0));
            sum = __dadd_rn(sum, __dmul_rn(a1, b1));
          }
          if (n & 1) {
            const uint32_t d = lds_pair(l).x;
            sum = __dadd_rn(sum, __dmul_rn(lds_f64(pa + (d >> 17)), lds_f64(pb + (d & 0x1ffffu))));
          }
          stage[k * kStageRow + lane] = sum;
        }
        __syncwarp();
        // eight entries of four rows at a time
        const int k = lane & 7;
        if (k < nk) {
          int j = lane >> 3;
          int c = out_col[k0 + k] + row0 + row_t + j;
          int64_t d = base + (int64_t)j * m + k0 + k;
          for (; j < nt; j += 4, c += 4, d += 4 * m) {
            a.ccol[d] = a.colbase ? c - a.colbase[row0 + row_t + j] : c;
            a.cval[d] = stage[k * kStageRow + j];
          }
        }
        __syncwarp();
      }
      team_sync(team, kTeamThreads);  // every warp is done with the operands
      const int next = row_t + 32 * kTeams;
      if (next < nrun) load_tile(next, min(32, nrun - next));
    }
  }
}

template <int T>
cudaError_t launch_runs_t(const RowArgs& a, int num_sms, cudaStream_t s) {
  auto kernel = k_runs<T>;
  constexpr int kThreads = RunShape<T>::kThreads;
  constexpr size_t kSmem = RunShape<T>::kSmem;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)kSmem);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, kSmem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (int64_t)per_sm * num_sms;
  if (grid > a.nrows) grid = a.nrows;
  kernel<<<(unsigned)grid, kThreads, kSmem, s>>>(a);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// the pre-pass, and finding the runs
// ---------------------------------------------------------------------------

// What the pre-pass reads of a row of B: {first entry, end, first column, last
// column}, one 16-byte gather per entry of A instead of four loads (end < first:
// a row pointer out of range).
__global__ void k_row_info(MatView B, int4* __restrict__ info, const int* skip) {
  if (skip && *skip) return;
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= B.n) return;
  const int32_t s = B.rowptr[k], e = B.rowptr[k + 1];
  int4 r = make_int4(0, -1, 0, 0);
  if (s >= 0 && e >= s && (int64_t)e <= B.nnz)
    r = make_int4(s, e, e > s ? B.col[s] : INT_MAX, e > s ? B.col[e - 1] : -1);
  info[k] = r;
}

// Sums over entries p0, p0 + step, … below p1 of the row of A that starts at s;
// `shifted`: every entry is one further on than the row before (at s1) has it.
struct RowSums {
  unsigned lo16 = 0, hi16 = 0;  // products: Σ of the row lengths' halves
  int mn = INT_MAX, mx = -1;
  bool bad = false;

  template <bool SHIFT>
  __device__ __forceinline__ bool add(const MatView& A, const int4* __restrict__ info, int32_t n_b,
                                      Pos s, Pos p0, Pos p1, int step, int32_t back) {
    bool shifted = SHIFT;
#pragma unroll 2
    for (Pos p = p0; p < p1; p += step) {
      const int32_t k = A.col[p];
      if (p > s && A.col[p - 1] >= k) bad = true;
      if (SHIFT && back > 0 && A.col[p - back] != k - 1) shifted = false;
      if (k < 0 || k >= n_b) {
        bad = true;
        continue;
      }
      const int4 b = info[k];
      const unsigned len = (unsigned)(b.y - b.x);
      bad = bad || (int)len < 0;
      lo16 += len & 0xffffu;
      hi16 += len >> 16;
      mn = min(mn, b.z);
      mx = max(mx, b.w);
    }
    return shifted;
  }
  __device__ __forceinline__ void reduce(const WarpGroup& g) {
    if (g.G == 32) {
      lo16 = __reduce_add_sync(kFull, lo16);
      hi16 = __reduce_add_sync(kFull, hi16);
      mn = __reduce_min_sync(kFull, mn);
      mx = __reduce_max_sync(kFull, mx);
    } else {
      for (int o = g.G >> 1; o > 0; o >>= 1) {
        lo16 += __shfl_xor_sync(g.mask, lo16, o);
        hi16 += __shfl_xor_sync(g.mask, hi16, o);
        mn = min(mn, __shfl_xor_sync(g.mask, mn, o));
        mx = max(mx, __shfl_xor_sync(g.mask, mx, o));
      }
    }
    bad = g.ballot(bad) != 0u;
  }
  __device__ __forceinline__ long long products() const {
    return (long long)lo16 + ((long long)hi16 << 16);
  }
};

constexpr int kLongRow = 256;      // longer rows of A are cut into pieces
constexpr int kLongPiece = 1024;
constexpr int kRowsAhead = 4;      // rows whose loads a group has in flight together

// Products and column span per row of C = A·B, the validation of A
// (launch_validate's checks), and flag[i] = 1 when row i of A is row i − 1 with
// every column one further on.  G lanes per row, `rows` (at most 256) rows per
// CTA; every index is checked before it is used, and a row that meets one out
// of range gets f = −1.  Rows of more than kLongRow entries are listed, a piece
// {row, first entry} at a time, for k_prepass_long.  marks: {pieces listed,
// rows flagged, rows listed}.  Bound by the latency of entry -> row of B, hence four rows of
// a group at a time where none is longer than the group.
constexpr int kRunBlock = 256;
constexpr int kShortLanes = 8;  // lanes per row of the matrices that take k_prepass_short
__global__ void __launch_bounds__(256) k_prepass_rows(
    MatView A, int32_t n_b, const int4* __restrict__ info, int G, int rows,
    int64_t* __restrict__ f, int32_t* __restrict__ lo, int32_t* __restrict__ hi,
    uint8_t* __restrict__ flag, int2* __restrict__ pieces, int64_t max_pieces,
    int32_t* __restrict__ marks, uint32_t* status, const int* skip) {
  if (skip && *skip) return;
  __shared__ int s_flagged;
  __shared__ int32_t ptr[kRunBlock + 2];  // row pointers of rows row0 − 1 … row0 + rows
  const WarpGroup g(G);
  const int64_t row0 = (int64_t)blockIdx.x * rows;
  if (threadIdx.x == 0) s_flagged = 0;
  for (int t = threadIdx.x; t < rows + 2; t += 256) {
    const int64_t i = row0 - 1 + t;
    ptr[t] = i < 0 ? -1 : A.rowptr[min(i, (int64_t)A.n)];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 &&
      (A.rowptr[0] != 0 || (int64_t)A.rowptr[A.n] != A.nnz))
    report(status, DEV_ERR_INVALID_CSR);
  __syncthreads();
  const int nrows = (int)min((int64_t)rows, A.n - row0), ngroups = 256 / G;
  int flagged = 0;
  // sums of row r (of this CTA's) reduced over the group, and what follows from them
  auto finish = [&](int r, bool on, RowSums& t, bool same, bool wrong) {
    same = g.ballot(!same) == 0u;
    t.reduce(g);
    const bool bad = t.bad || wrong;
    if (on && g.lane == 0) {
      const int64_t i = row0 + r;
      if (bad) report(status, DEV_ERR_INVALID_CSR);
      f[i] = bad ? -1 : t.products();
      lo[i] = bad ? INT_MAX : t.mn;
      hi[i] = bad ? -1 : t.mx;
      flag[i] = same && !bad;
      flagged += same && !bad;
    }
  };
  for (int r0 = threadIdx.x / G; r0 - (threadIdx.x & 31) / G < nrows;
       r0 += ngroups * kRowsAhead) {  // whole warps
    int32_t s[kRowsAhead], len[kRowsAhead];
    bool candidate[kRowsAhead], wrong[kRowsAhead], on[kRowsAhead];
    bool fast = true;
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) {
      const int r = r0 + u * ngroups;
      on[u] = r < nrows;
      const int32_t s0 = on[u] ? ptr[r + 1] : 0, e0 = on[u] ? ptr[r + 2] : 0;
      wrong[u] = s0 < 0 || e0 < s0 || (int64_t)e0 > A.nnz;
      s[u] = wrong[u] ? 0 : s0;
      len[u] = wrong[u] ? 0 : e0 - s0;
      const int32_t s1 = on[u] ? ptr[r] : -1;
      candidate[u] = len[u] > 0 && len[u] <= kMaxLen && s1 >= 0 && s[u] - s1 == len[u];
      fast = fast && len[u] <= G;
    }
    if (__all_sync(kFull, fast)) {
      int32_t k[kRowsAhead], before[kRowsAhead], above[kRowsAhead];
      int4 b[kRowsAhead];
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u) {
        const int32_t p = s[u] + g.lane;
        const bool in = g.lane < len[u];
        k[u] = in ? A.col[p] : -1;
        above[u] = in && candidate[u] ? A.col[p - len[u]] : -2;
      }
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u) {
        before[u] = __shfl_up_sync(kFull, k[u], 1);
        if (g.lane == 0) before[u] = -1;
      }
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u)
        b[u] = k[u] >= 0 && k[u] < n_b ? info[k[u]] : make_int4(0, 0, INT_MAX, -1);
#pragma unroll
      for (int u = 0; u < kRowsAhead; ++u) {
        const bool in = g.lane < len[u];
        RowSums t;
        const unsigned n = (unsigned)(b[u].y - b[u].x);
        t.bad = in && (k[u] < 0 || k[u] >= n_b || before[u] >= k[u] || (int)n < 0);
        t.lo16 = n & 0xffffu;
        t.hi16 = n >> 16;
        t.mn = b[u].z;
        t.mx = b[u].w;
        finish(r0 + u * ngroups, on[u], t, candidate[u] && (!in || above[u] == k[u] - 1),
               wrong[u]);
      }
      continue;
    }
#pragma unroll 1
    for (int u = 0; u < kRowsAhead; ++u) {
      const int r = r0 + u * ngroups;
      // (read again rather than kept: u is not a constant here)
      const bool on_u = r < nrows;
      const int32_t s0 = on_u ? ptr[r + 1] : 0, e0 = on_u ? ptr[r + 2] : 0;
      const int32_t s1 = on_u ? ptr[r] : -1;
      const bool wrong_u = s0 < 0 || e0 < s0 || (int64_t)e0 > A.nnz;
      const bool listed = !wrong_u && e0 - s0 > kLongRow;
      const int32_t sr = wrong_u || listed ? 0 : s0, er = wrong_u || listed ? 0 : e0;
      const int n = er - sr;
      const bool cand = n > 0 && n <= kMaxLen && s1 >= 0 && sr - s1 == n;
      RowSums t;
      const bool same = t.add<true>(A, info, n_b, sr, sr + g.lane, er, G, cand ? n : 0);
      finish(r, on_u, t, same && cand, wrong_u);
      if (listed && g.lane == 0) {
        const int pc = (e0 - s0 + kLongPiece - 1) / kLongPiece;
        const int64_t at = (unsigned)atomicAdd(&marks[0], pc);
        // (rows of a valid A cannot list more)
        if (at + pc > max_pieces) report(status, DEV_ERR_INVALID_CSR);
        else
          for (int c = 0; c < pc; ++c)
            pieces[at + c] = make_int2((int)(row0 + r), s0 + c * kLongPiece);
      }
    }
  }
  if (flagged) atomicAdd(&s_flagged, flagged);
  __syncthreads();
  if (threadIdx.x == 0 && s_flagged) atomicAdd(&marks[1], s_flagged);
}

// The same with a thread per row, for matrices of few entries a row: a group of
// eight lanes spends its instructions on the reductions (5-point grid 1009²:
// 94 -> 20 µs with the row's entries in turn, four loads in flight).  Rows of
// more than kThreadRow entries are listed for the warps of k_prepass_long (a warp
// that took its own 32 rows' one after another: 120 against 24 µs where 2,000 rows
// of 64 entries lie together among 100,000).
constexpr int kThreadRow = 16;
__global__ void __launch_bounds__(256) k_prepass_short(
    MatView A, int32_t n_b, const int4* __restrict__ info, int64_t* __restrict__ f,
    int32_t* __restrict__ lo, int32_t* __restrict__ hi, uint8_t* __restrict__ flag,
    int2* __restrict__ pieces, int64_t max_pieces, int32_t* __restrict__ marks,
    int32_t* __restrict__ mid, uint32_t* status, const int* skip) {
  if (skip && *skip) return;
  const int lane = threadIdx.x & 31;
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const bool on = i < A.n;
  if (i == 0 && (A.rowptr[0] != 0 || (int64_t)A.rowptr[A.n] != A.nnz))
    report(status, DEV_ERR_INVALID_CSR);
  int32_t s = on ? A.rowptr[i] : 0, e = on ? A.rowptr[i + 1] : 0;
  const int32_t s1 = on && i > 0 ? A.rowptr[i - 1] : -1;
  const bool wrong = s < 0 || e < s || (int64_t)e > A.nnz;
  if (wrong) s = e = 0;
  const int len = e - s;
  const bool candidate = len > 0 && len <= kMaxLen && s1 >= 0 && s - s1 == len;
  bool same = candidate;
  RowSums t;
  if (len <= kThreadRow) {
    int before = -1;
    for (int q = 0; q < len; q += 4) {
      int32_t k[4], above[4];
      int4 b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool in = q + u < len;
        k[u] = in ? A.col[s + q + u] : -1;
        above[u] = in && candidate ? A.col[s + q + u - len] : -2;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        b[u] = k[u] >= 0 && k[u] < n_b ? info[k[u]] : make_int4(0, 0, INT_MAX, -1);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (q + u >= len) break;
        const unsigned n = (unsigned)(b[u].y - b[u].x);
        t.bad = t.bad || k[u] < 0 || k[u] >= n_b || before >= k[u] || (int)n < 0;
        t.lo16 += n & 0xffffu;
        t.hi16 += n >> 16;
        t.mn = min(t.mn, b[u].z);
        t.mx = max(t.mx, b[u].w);
        same = same && above[u] == k[u] - 1;
        before = k[u];
      }
    }
  }
  const bool is_mid = len > kThreadRow && len <= kLongRow;
  const unsigned mids = __ballot_sync(kFull, is_mid);
  if (mids) {
    int at = 0;
    if (lane == 0) at = atomicAdd(&marks[2], __popc(mids));
    at = __shfl_sync(kFull, at, 0) + __popc(mids & lanemask_lt());
    if (is_mid) mid[at] = (int32_t)i;
  }
  if (len > kLongRow) {
    const int pc = (len + kLongPiece - 1) / kLongPiece;
    const int64_t at = (unsigned)atomicAdd(&marks[0], pc);
    // (rows of a valid A cannot list more)
    if (at + pc > max_pieces) report(status, DEV_ERR_INVALID_CSR);
    else
      for (int c = 0; c < pc; ++c) pieces[at + c] = make_int2((int)i, s + c * kLongPiece);
  }
  const bool bad = t.bad || wrong;
  if (on && !is_mid) {
    if (bad) report(status, DEV_ERR_INVALID_CSR);
    f[i] = bad ? -1 : t.products();
    lo[i] = bad ? INT_MAX : t.mn;
    hi[i] = bad ? -1 : t.mx;
    flag[i] = same && !bad;
  }
  const int flagged = __syncthreads_count(on && !is_mid && same && !bad);
  if (threadIdx.x == 0 && flagged) atomicAdd(&marks[1], flagged);
}

// The listed pieces, a CTA each, and the listed rows, a warp each.
__global__ void __launch_bounds__(256) k_prepass_long(
    MatView A, int32_t n_b, const int4* __restrict__ info, int64_t* f, int32_t* lo, int32_t* hi,
    uint8_t* __restrict__ flag, const int2* __restrict__ pieces, int64_t max_pieces,
    const int32_t* __restrict__ mid, int32_t* marks, uint32_t* status) {
  const int lane = threadIdx.x & 31;
  int n = marks[0];
  if (n < 0 || n > max_pieces) n = 0;  // A is invalid, and some pieces are not listed
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    const int2 piece = pieces[c];
    const Pos s = A.rowptr[piece.x];
    const Pos e = min((Pos)A.rowptr[piece.x + 1], (Pos)piece.y + kLongPiece);
    RowSums t;
    t.add<false>(A, info, n_b, s, (Pos)piece.y + threadIdx.x, e, blockDim.x, 0);
    t.reduce(WarpGroup(32));
    if (lane == 0) {
      if (t.bad) report(status, DEV_ERR_INVALID_CSR);
      atomicAdd((unsigned long long*)&f[piece.x], (unsigned long long)t.products());
      atomicMin(&lo[piece.x], t.mn);
      atomicMax(&hi[piece.x], t.mx);
    }
  }
  const int rows = marks[2];
  int flagged = 0;
  for (int r = (blockIdx.x * 256 + threadIdx.x) >> 5; r < rows; r += gridDim.x * 8) {
    const int32_t i = mid[r];  // (its row pointers were checked)
    const int32_t s = A.rowptr[i], e = A.rowptr[i + 1], s1 = i > 0 ? A.rowptr[i - 1] : -1;
    const bool candidate = e - s <= kMaxLen && s1 >= 0 && s - s1 == e - s;
    RowSums t;
    bool same = t.add<true>(A, info, n_b, s, (Pos)s + lane, e, 32, candidate ? e - s : 0);
    same = __all_sync(kFull, same) && candidate;
    t.reduce(WarpGroup(32));
    if (lane == 0) {
      if (t.bad) report(status, DEV_ERR_INVALID_CSR);
      f[i] = t.bad ? -1 : t.products();
      lo[i] = t.bad ? INT_MAX : t.mn;
      hi[i] = t.bad ? -1 : t.mx;
      flag[i] = same && !t.bad;
      flagged += same && !t.bad;
    }
  }
  if (flagged) atomicAdd(&marks[1], flagged);
}

// Too few rows of A are their predecessor shifted for runs to matter.
__device__ __forceinline__ bool few_shifted(const int32_t* marks, int32_t n) {
  return marks[1] < n / 16;
}

// flag[i] as above for a matrix of valid rows (Aᵀ); not needed where A has
// few shifted rows.
__global__ void __launch_bounds__(256) k_shift_flags(MatView M, int G, uint8_t* __restrict__ flag,
                                                     const int32_t* __restrict__ marks) {
  if (few_shifted(marks, M.n)) return;
  const WarpGroup g(G);
  const int64_t row0 = (int64_t)blockIdx.x * kRunBlock;
  for (int r = threadIdx.x / G; r < kRunBlock; r += kRunBlock / G) {
    const int64_t i = row0 + r;
    const bool on = i < M.n;
    bool same = false;
    if (on && i > 0) {
      const int32_t s1 = M.rowptr[i - 1], s = M.rowptr[i], len = M.rowptr[i + 1] - s;
      same = len > 0 && s - s1 == len;
      if (same)
        for (int q = g.lane; q < len; q += G) same = same && M.col[s1 + q] == M.col[s + q] - 1;
    }
    same = g.ballot(!same) == 0u;
    if (on && g.lane == 0) flag[i] = same;
  }
}

// The runs of 256 rows per CTA:
//   lead[i]: rows back to the first row of i's run (0: i is one, or in no run)
//   runlen[i], need[i]: in a run its rows, and the doubles that 32 of them take
//     in shared memory; 0 in no run
__global__ void __launch_bounds__(256) k_find_runs(
    MatView A, const int4* __restrict__ info, int G, const uint8_t* __restrict__ flag_a,
    const uint8_t* __restrict__ flag_b, const int64_t* __restrict__ f,
    const int32_t* __restrict__ lo, const int32_t* __restrict__ hi, uint8_t* __restrict__ lead,
    uint16_t* __restrict__ runlen, uint16_t* __restrict__ need,
    const int32_t* __restrict__ marks, const int* skip) {
  if (skip && *skip) return;
  __shared__ uint32_t firsts[kRunBlock / 32];  // rows that start a run, one bit each
  __shared__ uint16_t sneed[kRunBlock];
  __shared__ uint8_t list[kRunBlock / kRunMinRows], sflag[kRunBlock];
  __shared__ int32_t ptr[kRunBlock + 1];
  __shared__ int s_count;
  const WarpGroup g(G);
  const int tid = threadIdx.x;
  const int64_t row0 = (int64_t)blockIdx.x * kRunBlock;
  const int rows = (int)min((int64_t)kRunBlock, A.n - row0);
  if (few_shifted(marks, A.n) || !__syncthreads_or(tid < rows && flag_a[row0 + tid])) {
    if (tid < rows) {
      lead[row0 + tid] = 0;
      runlen[row0 + tid] = 0;
      need[row0 + tid] = 0;
    }
    return;
  }
  if (tid < kRunBlock / 32) firsts[tid] = 0u;
  if (tid == 0) s_count = 0;
  sneed[tid] = 0;
  sflag[tid] = tid < rows ? flag_a[row0 + tid] : 0;
  for (int t = tid; t < rows + 1; t += kRunBlock) ptr[t] = A.rowptr[row0 + t];
  __syncthreads();
  // a row of C follows its predecessor when its row of A and the rows of B that
  // it reads do
  if (G == kShortLanes) {  // few entries a row: a thread per row
    bool follows = tid > 0 && tid < rows && sflag[tid];
    if (follows)
      for (Pos q = ptr[tid], e = ptr[tid + 1]; q < e && follows; q += 4) {
        int32_t k[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) k[u] = A.col[min(q + u, e - 1)];
#pragma unroll
        for (int u = 0; u < 4; ++u) follows = flag_b[k[u]] && follows;
      }
    const unsigned starts = __ballot_sync(kFull, tid < rows && !follows);
    if ((tid & 31) == 0) firsts[tid >> 5] = starts;
  } else for (int r0 = tid / G; r0 < kRunBlock; r0 += kRunBlock / G * kRowsAhead) {  // whole warps
    Pos p[kRowsAhead], e[kRowsAhead];
    int32_t k[kRowsAhead];
    bool follows[kRowsAhead];
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) {
      const int r = r0 + u * (kRunBlock / G);
      follows[u] = r > 0 && r < rows && sflag[r];  // (a flagged row is a valid one)
      p[u] = follows[u] ? ptr[r] + g.lane : 0;
      e[u] = follows[u] ? ptr[r + 1] : 0;
    }
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) k[u] = p[u] < e[u] ? A.col[p[u]] : -1;
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u)
      if (k[u] >= 0) follows[u] = follows[u] && flag_b[k[u]];
#pragma unroll
    for (int u = 0; u < kRowsAhead; ++u) {
      for (Pos q = p[u] + G; q < e[u]; q += G) follows[u] = follows[u] && flag_b[A.col[q]];
      const bool all = g.ballot(!follows[u]) == 0u;
      const int r = r0 + u * (kRunBlock / G);
      if (g.lane == 0 && r < rows && !all) atomicOr(&firsts[r >> 5], 1u << (r & 31));
    }
  }
  __syncthreads();
  // the first row of this row's run, and the run's length
  int first = 0, next = 0;
  if (tid < rows) {
    int w = tid >> 5;
    uint32_t bits = firsts[w] & ((2u << (tid & 31)) - 1u);
    while (!bits) bits = firsts[--w];  // row 0 of the block starts a run
    first = 32 * w + 31 - __clz((int)bits);
    next = rows;
    for (int v = first >> 5; v < kRunBlock / 32; ++v) {
      const uint32_t after =
          v == first >> 5 ? firsts[v] & ~((2u << (first & 31)) - 1u) : firsts[v];
      if (after) {
        next = 32 * v + __ffs((int)after) - 1;
        break;
      }
    }
    const int least = first == 0 || next == rows ? kRunMinRows
                      : G == kShortLanes         ? kRunMinWholeShort
                                                 : kRunMinWhole;
    if (tid == first && next - first >= least) list[atomicAdd(&s_count, 1)] = (uint8_t)tid;
  }
  __syncthreads();
  // what 32 rows of each run take, a group of lanes per run
  for (int l = tid / G; l - (tid & 31) / G < s_count; l += kRunBlock / G) {
    const bool on = l < s_count;
    const int r = on ? list[l] : 0;
    const int64_t i = row0 + r;
    const int64_t products = f[i];
    const int32_t s = A.rowptr[i];
    const int len = A.rowptr[i + 1] - s;
    const bool small = on && len <= kMaxLen && products > 0 && products <= kRunMaxProducts &&
                       hi[i] - lo[i] < kRunMaxSpan;
    int brows = 0, longest = 0;
    if (small)
      for (int t = g.lane; t < len; t += G) {
        const int32_t k = A.col[s + t];
        const int4 b = info[k];
        longest = max(longest, b.y - b.x);
        brows += t == 0 || A.col[s + t - 1] != k - 1 ? 32 : 1;
      }
    for (int o = G >> 1; o > 0; o >>= 1) {
      brows += __shfl_xor_sync(g.mask, brows, o);
      longest = max(longest, __shfl_xor_sync(g.mask, longest, o));
    }
    const int total = brows * (longest | 1) + 32 * (len | 1);  // (below 2^24 for a small row)
    if (small && total <= kRunBuffer && g.lane == 0) sneed[r] = (uint16_t)total;
  }
  __syncthreads();
  if (tid >= rows) return;
  const bool run = sneed[first] > 0;
  const int64_t i = row0 + tid;
  lead[i] = run ? (uint8_t)(tid - first) : 0;
  runlen[i] = run ? (uint16_t)(next - first) : 0;
  need[i] = sneed[first];
}

int lanes_for(const MatView& A) {
  const double mean = A.n > 0 ? (double)A.nnz / A.n : 1.0;
  return mean <= 8 ? kShortLanes : mean <= 16 ? 16 : 32;
}

}  // namespace

cudaError_t launch_runs(int team, const RowArgs& a, int num_sms, cudaStream_t s) {
  if (a.nrows <= 0) return cudaSuccess;
  switch (team) {
    case 0: return launch_runs_t<1>(a, num_sms, s);
    case 1: return launch_runs_t<2>(a, num_sms, s);
    case 2: return launch_runs_t<4>(a, num_sms, s);
    case 3: return launch_runs_t<8>(a, num_sms, s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_prepass_rows(const MatView& A, const MatView& B, const PrepassArrays& w,
                                int num_sms, uint32_t* status, cudaStream_t s, const int* skip) {
  if (A.n == 0) return launch_validate(A, status, s);
  cudaError_t e = cudaMemsetAsync(w.marks, 0, 3 * sizeof(int32_t), s);
  if (e != cudaSuccess) return e;
  const int G = lanes_for(A);
  const unsigned blocks = (unsigned)(((int64_t)A.n + kRunBlock - 1) / kRunBlock);
  k_row_info<<<blocks, 256, 0, s>>>(B, w.info, skip);
  SPG_COUNT_LAUNCH();
  // fewer rows per CTA where 256 would leave SMs without one
  int rows = kRunBlock;
  while (rows > kRowsAhead * (256 / G) && rows > 32 && A.n / rows < num_sms * 8) rows >>= 1;
  if (G == kShortLanes)
    k_prepass_short<<<blocks, 256, 0, s>>>(A, B.n, w.info, w.f, w.lo, w.hi, w.flag_a, w.pieces,
                                           prepass_pieces(A.nnz), w.marks, w.mid, status,
                                           skip);
  else
    k_prepass_rows<<<(unsigned)((A.n + rows - 1) / rows), 256, 0, s>>>(
        A, B.n, w.info, G, rows, w.f, w.lo, w.hi, w.flag_a, w.pieces, prepass_pieces(A.nnz),
        w.marks, status, skip);
  SPG_COUNT_LAUNCH();
  if (A.nnz > kThreadRow) {
    // (grid_sms asks for many CTAs, and few have anything to do)
    k_prepass_long<<<std::min(num_sms * 4, 148 * 64), 256, 0, s>>>(A, B.n, w.info, w.f, w.lo, w.hi, w.flag_a,
                                               w.pieces, prepass_pieces(A.nnz), w.mid, w.marks,
                                               status);
    SPG_COUNT_LAUNCH();
  }
  if (!w.lead) return cudaGetLastError();
  const uint8_t* flag_b = w.flag_a;
  if (B.col != A.col) {
    k_shift_flags<<<blocks, 256, 0, s>>>(B, G, w.flag_b, w.marks);
    SPG_COUNT_LAUNCH();
    flag_b = w.flag_b;
  }
  k_find_runs<<<blocks, 256, 0, s>>>(A, w.info, G, w.flag_a, flag_b, w.f, w.lo, w.hi, w.lead,
                                     w.runlen, w.need, w.marks, skip);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace spg
