// Heavy rows, numeric phase: a warp per (row, panel), a panel being a fixed
// range of 2^pan_log2 output columns whose values the warp holds densely in
// shared memory.
//
// The CTA-per-row kernel adds every product in place in C, one CTA barrier per
// entry of A's row, and the windowed warp kernel walks a whole row alone: a
// power-law graph's hub rows then set the time (R-MAT 2^14: 6.1 ms of the
// call's 9.9 ms in single warps, 2^16: 6.8 of 10.7 ms in CTAs waiting for
// barriers and for L2).  Cutting a row into panels makes its parts independent:
//  - slice bounds: ptr[k·(npan+1) + p] is the first entry of B row k at or past
//    panel p, found once by binary search (the rows are sorted), so a warp
//    reads exactly the entries of its panel, two adjacent ints per entry of A;
//  - the entries of 32 slices are loaded as one flattened run, all lanes busy
//    even when the slices hold a few entries each; the additions then go slice
//    by slice (a slice's columns are distinct), one __syncwarp per slice, so
//    every value is the k-ordered sum of the other kernels, bit for bit;
//  - a product is added straight to its column's place: no bitmap, no rank, no
//    hash.  Places start as −0.0, which no sum can be: the kernels' sums start
//    from +0.0, and x + y is −0.0 only when both are.  A product has 0.0 added
//    first (−0.0 becomes +0.0; nothing else changes), so the first addition
//    gives 0.0 + product and the places still holding −0.0 at the end are the
//    columns without an entry;
//  - warps draw panels until none is left; in launches that are to leave their SMs to
//    others now and then (grid_sms) there are as many warps as panels, up to the
//    grid's limit, and each leaves after its share;
//  - the symbolic phase's distinct-column counts per block give the panel's
//    first slot in C, and the panel is written in column order.
// R-MAT 2^16: the launches of the rows that were in CTAs 2.7 ms against 6.8
// there, and 3.2 ms now that rows of fewer products come here too.  Bound by the shared
// and L1 pipe (LSU wavefronts 79%: a 64-bit read and write of a place per product,
// the columns and values of the slices) and by issue (65%).  Panels of 2048 columns
// 3.36 against 2.68 ms (fewer warps per SM), of 512 3.02 (more slices per entry of
// A); eight tasks drawn at a time, before that, 6.4 against 3.5 ms (one warp was left
// with a hub row's neighbouring panels).
#include <algorithm>
#include <climits>

#include "kernels.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPanelUnroll = 4;     // groups of 32 products loaded ahead
constexpr long long kAbsent = (long long)0x8000000000000000ull;  // −0.0

// First and one-past-last panel of the row's output columns.
__device__ __forceinline__ int2 row_panels(const HeavyArgs& h, int row) {
  const int lo = h.lo[row];
  const int hi = h.hi[row];
  if (lo > hi) return make_int2(0, 0);
  return make_int2(lo >> h.pan_log2, (hi >> h.pan_log2) + 1);
}

// First position in [l, u) whose column is at or past c.
__device__ __forceinline__ int32_t column_bound(const int32_t* __restrict__ col, int32_t l,
                                                int32_t u, int64_t c) {
  while (l < u) {
    const int32_t mid = l + ((u - l) >> 1);  // (l + u may exceed 2^31)
    if (col[mid] < c) l = mid + 1; else u = mid;
  }
  return l;
}

// The slice of B row k in panel p.
__device__ __forceinline__ int2 panel_slice(const HeavyArgs& h, int32_t k, int p) {
  if (h.ptr) {
    const int32_t* q = h.ptr + (int64_t)k * (h.npan + 1) + p;
    return make_int2(q[0], q[1]);
  }
  const MatView& B = h.r.B;
  const int32_t u = B.rowptr[k + 1];
  const int32_t l = column_bound(B.col, B.rowptr[k], u, (int64_t)p << h.pan_log2);
  return make_int2(l, column_bound(B.col, l, u, (int64_t)(p + 1) << h.pan_log2));
}

__global__ void k_panel_bounds(MatView B, int pan_log2, int npan, int32_t* __restrict__ ptr) {
  const int64_t total = (int64_t)B.n * (npan + 1);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int64_t k = i / (npan + 1);
    const int p = (int)(i - k * (npan + 1));
    ptr[i] = column_bound(B.col, B.rowptr[k], B.rowptr[k + 1], (int64_t)p << pan_log2);
  }
}

// One CTA: the task offsets of the rows, a task per panel; off[nrows] is the number
// of tasks.  The rows are listed by product
// count, largest first, so a hub row's tasks start early and none of them is
// left to the end.
constexpr int kOffsetThreads = 1024, kOffsetRows = 8;
__global__ void __launch_bounds__(kOffsetThreads) k_panel_offsets(HeavyArgs h,
                                                                  int64_t* __restrict__ off) {
  __shared__ int scratch[33];
  __shared__ long long carry;
  const int tid = threadIdx.x, nrows = h.r.nrows;
  if (tid == 0) carry = 0;
  __syncthreads();
  for (int r0 = 0; r0 < nrows; r0 += kOffsetThreads * kOffsetRows) {
    // each step's loads issued together (rows past the end count the last one)
    int n[kOffsetRows], lo[kOffsetRows], hi[kOffsetRows], sum = 0;
#pragma unroll
    for (int u = 0; u < kOffsetRows; ++u)
      n[u] = h.r.rows[min(r0 + tid * kOffsetRows + u, nrows - 1)];
#pragma unroll
    for (int u = 0; u < kOffsetRows; ++u) {
      lo[u] = h.lo[n[u]];
      hi[u] = h.hi[n[u]];
    }
#pragma unroll
    for (int u = 0; u < kOffsetRows; ++u) {
      n[u] = r0 + tid * kOffsetRows + u < nrows
                 ? (hi[u] >> h.pan_log2) - (lo[u] >> h.pan_log2) + 1
                 : 0;
      sum += n[u];
    }
    int tot;
    long long at = carry + block_exclusive_scan(sum, scratch, &tot);
#pragma unroll
    for (int u = 0; u < kOffsetRows; ++u) {
      const int r = r0 + tid * kOffsetRows + u;
      if (r < nrows) off[r] = at;
      at += n[u];
    }
    __syncthreads();
    if (tid == 0) carry += tot;
    __syncthreads();
  }
  if (tid == 0) off[nrows] = carry;
}

// The row of task t: the last r with off[r] <= t, by a 32-way search.
__device__ __forceinline__ int task_row(const int64_t* off, int nrows, int64_t t) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = nrows;  // off[lo] <= t < off[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) >> 5;
    const int i = lo + lane * step;
    const unsigned le = __ballot_sync(kFull, i < hi && off[i] <= t);
    lo += (__popc(le) - 1) * step;  // off is non-decreasing: a prefix of the lanes
    hi = min(hi, lo + step);
  }
  return lo;
}

__global__ void __launch_bounds__(512) k_panel_num(HeavyArgs h, const int64_t* __restrict__ off) {
  extern __shared__ __align__(16) unsigned char smem[];
  const RowArgs& a = h.r;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int W = 1 << h.pan_log2;
  double* acc = (double*)(smem + (size_t)wid * panel_warp_bytes(h.pan_log2));
  double2* slice = (double2*)(acc + W);  // 32 of {a_ik, B position of the run's product 0}
  const int64_t total = off[a.nrows];
  int64_t share = total;
  if (h.retire) {
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    if ((int64_t)blockIdx.x * (blockDim.x >> 5) + wid >= total) return;
    share = (total + warps - 1) / warps;
  }
  for (int x = lane; x < W; x += 32) acc[x] = __longlong_as_double(kAbsent);
  __syncwarp();

  for (; share > 0; --share) {
    int64_t t = 0;
    if (lane == 0) t = (int64_t)atomicAdd((unsigned long long*)h.task_queue, 1ull);
    t = __shfl_sync(kFull, t, 0);
    if (t >= total) break;
    const int r = task_row(off, a.nrows, t);
    const int row = a.rows[r];
    const int2 pr = row_panels(h, row);
    const int p = pr.x + (int)(t - off[r]);
    const Pos ps = a.A.rowptr[row], pe = a.A.rowptr[row + 1];
    const int cb = a.colbase ? a.colbase[row] : 0;
    const int w0 = p << h.pan_log2;

    // 32 entries of A's row at a time: the next 32's slice bounds and the columns
    // of the 32 after them are on their way meanwhile
    int2 bnd = make_int2(0, 0);
    double av = 0.0;
    int32_t k = 0;
    if (ps + lane < pe) {
      bnd = panel_slice(h, a.A.col[ps + lane], p);
      av = a.A.val[ps + lane];
    }
    if (ps + 32 + lane < pe) k = a.A.col[ps + 32 + lane];
    Pos pb = ps;                     // next 32 entries
    int run = 0, c0 = 0, first = 0;  // products of the current 32, next one, this lane's first
    auto advance = [&]() -> bool {   // to the next products, if any
      while (c0 >= run) {
        if (pb >= pe) return false;
        const int bs = bnd.x, len = bnd.y - bnd.x;
        const double at = av;
        bnd = make_int2(0, 0);
        if (pb + 32 + lane < pe) {
          bnd = panel_slice(h, k, p);
          av = a.A.val[pb + 32 + lane];
        }
        if (pb + 64 + lane < pe) k = a.A.col[pb + 64 + lane];
        pb += 32;
        const unsigned live = __ballot_sync(kFull, len > 0);
        if (!live) continue;
        int incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += v;
        }
        run = __shfl_sync(kFull, incl, 31);
        c0 = 0;
        first = len > 0 ? incl - len : INT_MAX;
        __syncwarp();  // the previous products' lookups are done
        if (len > 0)
          slice[__popc(live & lanemask_lt())] =
              make_double2(at, __longlong_as_double((long long)(bs - first)));
        __syncwarp();
      }
      return true;
    };
    // the next products, kPanelUnroll groups of 32: loaded here, used one step later
    int col[kPanelUnroll];
    unsigned starts[kPanelUnroll];
    double lv[kPanelUnroll], rv[kPanelUnroll];
    auto fetch = [&]() {
#pragma unroll
      for (int u = 0; u < kPanelUnroll; ++u) {
        const int c = c0 + u * 32;
        col[u] = -1;
        starts[u] = 0u;
        lv[u] = 0.0;
        rv[u] = 0.0;
        if (c < run) {
          // slices that start in this group of 32 products, one bit each
          const int d = first - c;
          starts[u] = __reduce_or_sync(kFull, d > 0 && d < 32 ? 1u << d : 0u);
          const int t0 = __popc(__ballot_sync(kFull, d <= 0)) - 1;
          const double2 sl = slice[t0 + __popc(starts[u] & (lanemask_lt() * 2u + 1u))];
          if (c + lane < run) {
            const int q = (int)__double_as_longlong(sl.y) + c + lane;
            col[u] = a.B.col[q];
            rv[u] = a.B.val[q];
            lv[u] = sl.x;
          }
        }
      }
      c0 += 32 * kPanelUnroll;
    };
    bool more = advance();
    if (more) fetch();
    while (more) {
      int x[kPanelUnroll];
      unsigned st[kPanelUnroll];
      double v[kPanelUnroll];
#pragma unroll
      for (int u = 0; u < kPanelUnroll; ++u) {
        const unsigned j = (unsigned)(col[u] - w0);
        x[u] = col[u] >= 0 && j < (unsigned)W ? (int)j : -1;
        v[u] = __dadd_rn(__dmul_rn(lv[u], rv[u]), 0.0);
        st[u] = starts[u];
      }
      more = advance();
      if (more) fetch();
#pragma unroll
      for (int u = 0; u < kPanelUnroll; ++u) {
        const int n = __popc(st[u]);
        if (n <= 4) {
          const int mine = __popc(st[u] & (lanemask_lt() * 2u + 1u));
          for (int i = 0; i <= n; ++i) {  // slice by slice: the k order
            if (mine == i && x[u] >= 0) acc[x[u]] = __dadd_rn(acc[x[u]], v[u]);
            __syncwarp();
          }
        } else {
          // many short slices, few of whose products share a column: those that
          // do go in lane order, the others at once
          const unsigned same = __match_any_sync(kFull, x[u]) & lanemask_lt();
          const int rank = x[u] >= 0 ? __popc(same) : 0;
          if (x[u] >= 0 && rank == 0) acc[x[u]] = __dadd_rn(acc[x[u]], v[u]);
          __syncwarp();
          for (int i = 1; __any_sync(kFull, rank >= i); ++i) {
            if (rank == i) acc[x[u]] = __dadd_rn(acc[x[u]], v[u]);
            __syncwarp();
          }
        }
      }
    }

    // the panel's first slot: the distinct columns of the blocks before it
    int64_t before = 0;
    if (p > pr.x) {
      const int nb = (p << (h.pan_log2 - h.blk_log2)) - (h.lo[row] >> h.blk_log2);
      const uint16_t* cnt = h.blk_cnt + h.blk_off[row];
      int s = 0;
      for (int i = lane; i < nb; i += 32) s += cnt[i];
      before = __reduce_add_sync(kFull, s);
    }
    const int64_t base = a.rowptr[row] + before;
    const int64_t room = (int64_t)a.cnt_in[row] - before;

    // write the panel in column order and leave its places absent
    int64_t written = 0;
    for (int c = 0; c < W; c += 64) {
      const double2 v = *(const double2*)(acc + c + 2 * lane);
      const bool h0 = __double_as_longlong(v.x) != kAbsent;
      const bool h1 = __double_as_longlong(v.y) != kAbsent;
      const unsigned b0 = __ballot_sync(kFull, h0), b1 = __ballot_sync(kFull, h1);
      if (!(b0 | b1)) continue;
      *(double2*)(acc + c + 2 * lane) =
          make_double2(__longlong_as_double(kAbsent), __longlong_as_double(kAbsent));
      int64_t pos = written + __popc(b0 & lanemask_lt()) + __popc(b1 & lanemask_lt());
      written += __popc(b0) + __popc(b1);
      const int j = w0 + c + 2 * lane;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (!(e ? h1 : h0)) continue;
        if (pos < room) {
          a.ccol[base + pos] = j + e - cb;
          a.cval[base + pos] = e ? v.y : v.x;
        }
        ++pos;
      }
    }
    if (lane == 0 && (written > room || (p + 1 == pr.y && written != room)))
      report(a.status, DEV_ERR_OVERFLOW);
    __syncwarp();
  }
}

}  // namespace

static int64_t align256(int64_t b) { return (b + 255) & ~(int64_t)255; }

int64_t panel_workspace(int64_t n, int npan, int64_t nrows, bool table) {
  return (table ? align256(4 * n * (npan + 1)) : 0) + align256(8 * (nrows + 1)) + 256;
}

cudaError_t launch_panels(HeavyArgs& h, void* workspace, bool table, int num_sms,
                          cudaStream_t s) {
  if (h.r.nrows <= 0) return cudaSuccess;
  char* w = (char*)workspace;
  const int64_t nptr = (int64_t)h.r.B.n * (h.npan + 1);
  int32_t* ptr = table ? (int32_t*)w : nullptr;
  if (table) w += align256(4 * nptr);
  int64_t* off = (int64_t*)w;
  w += align256(8 * ((int64_t)h.r.nrows + 1));
  h.ptr = ptr;
  h.task_queue = (int64_t*)w;
  cudaError_t e = cudaMemsetAsync(h.task_queue, 0, sizeof(int64_t), s);
  if (e != cudaSuccess) return e;
  if (table) {
    const int64_t blocks = std::min<int64_t>((nptr + 255) / 256, (int64_t)num_sms * 32);
    k_panel_bounds<<<(unsigned)blocks, 256, 0, s>>>(h.r.B, h.pan_log2, h.npan, ptr);
    SPG_COUNT_LAUNCH();
  }
  k_panel_offsets<<<1, kOffsetThreads, 0, s>>>(h, off);
  SPG_COUNT_LAUNCH();
  if ((e = cudaGetLastError()) != cudaSuccess) return e;

  auto kernel = k_panel_num;
  const size_t per = panel_warp_bytes(h.pan_log2);
  // two CTAs per SM, each of as many warps as half of its shared memory holds
  constexpr size_t kMostBytes = (size_t)112 * 1024;
  const int warps = (int)std::max<size_t>(1, std::min<size_t>(16, kMostBytes / per));
  const size_t bytes = per * warps;
  e = allow_shared_memory(kernel, kMostBytes);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, bytes);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  const int64_t grid =
      std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * num_sms, (h.tasks + warps - 1) / warps));
  kernel<<<(unsigned)grid, warps * 32, bytes, s>>>(h, off);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace spg
