// Sorted rows, numeric phase: rows whose products hardly merge (sparse random
// graphs, power-law rows of middling size) have all of their products in flight
// at once and are ordered by a bucket sort, without a hash table.
//
// In the hash kernels such a row claims a slot per product, with a chain of
// B-row loads in front of each group of three, and then compacts and
// radix-sorts as many entries as it had products, in a table of up to 24 KB a
// row (nine warps per SM).  Erdős–Rényi, 40,009 rows of mean degree 20 (400
// products a row, 398 distinct): numeric launch 810 -> 240 µs (20 -> 66 G
// products/s; reading A and writing C alone takes 31 µs).  What is left is
// instruction issue and its latencies (52% of issue slots, shared-memory
// wavefronts 52%, about 9 warp instructions a product), not memory.
//
// A row's products are expanded into shared memory in k order, each as a
// packed word (column − lo) << eb | e with e its place in that order, 20
// bytes a product in all.  Word order is (column, k) order, so the row is done
// once the words are sorted:
//  - F buckets over the column span (F the row capacity; monotone in the
//    column) count their words, an exclusive scan of the counts places the
//    buckets, and a second pass drops each word into its bucket;
//  - a word's final place is its bucket's start plus the words below it in the
//    bucket: one or two of them unless columns cluster;
//  - rows whose fullest bucket holds more than kBucketMax words (clustered
//    columns: the places would cost the square of it) sort the words with the
//    stable radix sort instead.
// The first word of a run of equal columns adds the run's products in k order,
// starting from 0.0, so every value is the same sum, bit for bit, as in the
// hash kernels; no synchronisation per k is needed.  Rows of up to 512 products
// take one warp, larger ones a CTA of a warp per 512 products (one warp up to
// 1024 products: 344 against 240 µs on the graph above; a warp per 256: 260;
// half as many buckets: 255).
#include <climits>

#include "kernels.h"

namespace spg {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kBucketMax = 48;

// Warps per row of the F-product kernel: a CTA of several from 513 products on.
__host__ __device__ constexpr int sort_warps(int f) { return f <= 512 ? 1 : (f + 511) / 512; }
// Shared memory of one row: values, two word buffers, bucket counters.
constexpr size_t sort_row_bytes(int f) { return (size_t)20 * f; }

__device__ __forceinline__ int warp_exclusive_scan(int v, int* total) {
  const int lane = threadIdx.x & 31;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  *total = __shfl_sync(kFull, incl, 31);
  return incl - v;
}

// Bucket of a column offset below the row's span: monotone, below F.  `mult`
// is (2^32 − 1) / span · F, or 0 when the span has at most F columns.
__device__ __forceinline__ unsigned bucket_of(uint32_t x, uint32_t mult) {
  return mult ? __umulhi(x, mult) : x;
}

// Sorts w0[0..m) on the column bits with the stable radix sort; the result
// ends in w0.  Its counters (7-bit digits) take 128 · NW of the F in cnt.
template <int NW>
__device__ __noinline__ void clustered_sort(uint32_t* w0, uint32_t* w1, int m, int lo_bit,
                                            int nbits, int* cnt, int* scratch) {
  const uint32_t* r = radix_sort_words<NW, 7>(w0, w1, m, lo_bit, nbits, cnt, scratch);
  if (r != w0) {
    const int tid = NW == 1 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
    for (int i = tid; i < m; i += NW * 32) w0[i] = w1[i];
  }
  nw_sync<NW>();
}

// One row of up to F products (a multiple of 128, at most 512 per warp) by a
// group of NW warps; 2^eb >= F.  `part` holds NW + 1 ints (NW > 1).
template <int NW>
__device__ __forceinline__ void sort_row(const RowArgs& a, const int row, const int F,
                                         const int eb, double* vals, uint32_t* w0, uint32_t* w1,
                                         int* cnt, int* part) {
  constexpr int GT = NW * 32;
  const uint32_t emask = (1u << eb) - 1u;
  const int lane = threadIdx.x & 31;
  const int wid = NW == 1 ? 0 : (int)(threadIdx.x >> 5);
  const int tid = NW == 1 ? lane : (int)threadIdx.x;
  const Pos ps = a.A.rowptr[row], pe = a.A.rowptr[row + 1];
  const int lo = a.lo[row], hi = a.hi[row];
  const uint32_t span = (uint32_t)(hi - lo) + 1u;
  const int64_t base = a.rowptr[row];
  const int expect = a.cnt_in[row];
  const int cb = a.colbase ? a.colbase[row] : 0;
  const uint32_t mult = span > (uint32_t)F ? (0xffffffffu / span) * (uint32_t)F : 0u;
  for (int s = tid * 4; s < F; s += GT * 4) *(int4*)(cnt + s) = make_int4(0, 0, 0, 0);
  nw_sync<NW>();

  // expand: 32 entries of A's row at a time, their products 32 at a time; with
  // several warps each takes its share of those
  int done = 0;
  for (Pos pb = ps; pb < pe; pb += 32) {
    int bs = 0, len = 0;
    double av = 0.0;
    if (pb + lane < pe) {
      const int32_t k = a.A.col[pb + lane];
      bs = a.B.rowptr[k];
      len = a.B.rowptr[k + 1] - bs;
      av = a.A.val[pb + lane];
    }
    unsigned live = __ballot_sync(kFull, len > 0);
    if (live & (live + 1u)) {  // empty B rows between others: close the gaps
      const int from = (int)__fns(live, 0, lane + 1);
      bs = __shfl_sync(kFull, bs, from & 31);
      av = __shfl_sync(kFull, av, from & 31);
      len = __shfl_sync(kFull, len, from & 31);
      if (lane >= __popc(live)) len = 0;
      live = (1u << __popc(live)) - 1u;
    }
    int total;
    const int excl = warp_exclusive_scan(len, &total);
    const int src = bs - excl;  // B position of the chunk's product 0, had it lain in this row
    const int first = len > 0 ? excl : INT_MAX;
    if (done + total > F) {  // more products than the plan counted
      if (tid == 0) report(a.status, DEV_ERR_OVERFLOW);
      nw_sync<NW>();
      return;
    }
    for (int e0 = wid * 32; e0 < total; e0 += GT * 4) {
      int col[4];
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        col[u] = -1;
        const int c0 = e0 + u * GT;
        if (c0 >= total) continue;
        // entries that start in this group of 32 products, one bit each; the
        // product's entry is the last that starts at or before it
        const int d = first - c0;
        const unsigned starts =
            __reduce_or_sync(kFull, d > 0 && d < 32 ? 1u << d : 0u) & (lanemask_lt() * 2u + 1u);
        const int t = __popc(__ballot_sync(kFull, d <= 0)) - 1 + __popc(starts);
        const int q = __shfl_sync(kFull, src, t) + c0 + lane;
        const double at = __shfl_sync(kFull, av, t);
        if (c0 + lane < total) {
          col[u] = a.B.col[q];
          v[u] = __dmul_rn(at, a.B.val[q]);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (col[u] < 0) continue;
        const int e = done + e0 + u * GT + lane;
        uint32_t x = (uint32_t)(col[u] - lo);
        if (x >= span) {  // not a column that the plan saw
          report(a.status, DEV_ERR_OVERFLOW);
          x = span - 1;
        }
        vals[e] = v[u];
        w0[e] = x << eb | (uint32_t)e;
        atomicAdd(&cnt[bucket_of(x, mult)], 1);
      }
    }
    done += total;
  }
  nw_sync<NW>();

  // places of the buckets (each warp a contiguous part of them), and whether
  // one of them is too full
  const int c_begin = NW == 1 ? 0 : wid * 512, c_end = NW == 1 ? F : min(F, c_begin + 512);
  int fullest = 0, carry = 0, tot;
  if (NW > 1) {
    int sum = 0;
    for (int s = c_begin + lane * 4; s < c_end; s += 128) {
      const int4 c = *(const int4*)(cnt + s);
      sum += c.x + c.y + c.z + c.w;
      fullest = max(fullest, max(max(c.x, c.y), max(c.z, c.w)));
    }
    sum = __reduce_add_sync(kFull, sum);
    if (lane == 0) part[wid] = sum;
    fullest = __syncthreads_or(fullest > kBucketMax) ? kBucketMax + 1 : 0;
    for (int i = 0; i < wid; ++i) carry += part[i];
  }
  for (int s = c_begin + lane * 4; s < c_end; s += 128) {
    const int4 c = *(const int4*)(cnt + s);
    const int ex = carry + warp_exclusive_scan(c.x + c.y + c.z + c.w, &tot);
    if (NW == 1) fullest = max(fullest, max(max(c.x, c.y), max(c.z, c.w)));
    *(int4*)(cnt + s) = make_int4(ex, ex + c.x, ex + c.x + c.y, ex + c.x + c.y + c.z);
    carry += tot;
  }
  if (NW == 1) fullest = __reduce_max_sync(kFull, fullest);
  nw_sync<NW>();

  if (fullest > kBucketMax) {
    clustered_sort<NW>(w0, w1, done, eb, span_bits(lo, hi), cnt, part);
  } else {
#pragma unroll 1
    for (int e = tid; e < done; e += GT) {
      const uint32_t w = w0[e];
      w1[atomicAdd(&cnt[bucket_of(w >> eb, mult)], 1)] = w;
    }
    nw_sync<NW>();
    // cnt[b] is now the end of bucket b, and so the start of bucket b + 1
#pragma unroll 1
    for (int p = tid; p < done; p += GT) {
      const uint32_t w = w1[p];
      const int b = (int)bucket_of(w >> eb, mult);
      const int s = b ? cnt[b - 1] : 0, e = cnt[b];
      int r = s;
#pragma unroll 1
      for (int q = s; q < e; ++q) r += w1[q] < w;
      w0[r] = w;
    }
    nw_sync<NW>();
  }
  const uint32_t* sorted = w0;

  // the head of each run of equal columns adds the run in k order
  if (done == expect) {  // every column once
#pragma unroll 1
    for (int p = tid; p < done; p += GT) {
      const uint32_t w = sorted[p];
      a.ccol[base + p] = lo + (int)(w >> eb) - cb;
      a.cval[base + p] = __dadd_rn(0.0, vals[w & emask]);
    }
    nw_sync<NW>();  // the buffers are reused by the next row
    return;
  }
  // each warp takes a contiguous part of the words; with several warps the
  // heads are counted first (lane i keeps the head bits of the part's i-th 32)
  const int per = NW == 1 ? done : ((done + GT - 1) / GT) * 32;
  const int p_begin = min(done, wid * per), p_end = min(done, p_begin + per);
  unsigned heads = 0;
  int written = 0;
  if (NW > 1) {
    int count = 0;
#pragma unroll 1
    for (int c = p_begin; c < p_end; c += 32) {
      const int p = c + lane;
      const bool head = p < p_end && (p == 0 || ((sorted[p] ^ sorted[p - 1]) >> eb) != 0);
      const unsigned bal = __ballot_sync(kFull, head);
      if (lane == (c - p_begin) >> 5) heads = bal;
      count += __popc(bal);
    }
    if (lane == 0) part[wid] = count;
    __syncthreads();
    for (int i = 0; i < wid; ++i) written += part[i];
  }
#pragma unroll 1
  for (int c = p_begin; c < p_end; c += 32) {
    const int p = c + lane;
    const uint32_t w = p < p_end ? sorted[p] : 0u;
    unsigned bal;
    if (NW == 1)
      bal = __ballot_sync(kFull, p < p_end && (p == 0 || ((w ^ sorted[p - 1]) >> eb) != 0));
    else
      bal = __shfl_sync(kFull, heads, (c - p_begin) >> 5);
    const int pos = written + __popc(bal & lanemask_lt());
    if ((bal >> lane & 1u) && pos < expect) {
      double v = __dadd_rn(0.0, vals[w & emask]);
#pragma unroll 1
      for (int q = p + 1; q < done; ++q) {
        const uint32_t y = sorted[q];
        if ((y ^ w) >> eb) break;
        v = __dadd_rn(v, vals[y & emask]);
      }
      a.ccol[base + pos] = lo + (int)(w >> eb) - cb;
      a.cval[base + pos] = v;
    }
    written += __popc(bal);
  }
  if (wid == NW - 1 && lane == 0 && written != expect) report(a.status, DEV_ERR_OVERFLOW);
  nw_sync<NW>();
}

template <int NW>
__global__ void __launch_bounds__(NW == 1 ? 256 : NW * 32, NW == 1 ? 5 : 32 / NW) k_sort_rows(RowArgs a, int F, int eb) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int part[NW > 1 ? 33 : 1];
  // NW == 1: a row per warp; else a row per CTA
  const int w = NW == 1 ? (int)(threadIdx.x >> 5) : 0;
  const int nw = NW == 1 ? (int)(blockDim.x >> 5) : 1;
  double* vals = (double*)(smem + (size_t)w * 20 * F);
  uint32_t* w0 = (uint32_t*)(vals + F);
  uint32_t* w1 = w0 + F;
  int* cnt = (int*)(w1 + F);
  for (int r = blockIdx.x * nw + w; r < a.nrows; r += gridDim.x * nw)
    sort_row<NW>(a, a.rows ? a.rows[r] : r, F, eb, vals, w0, w1, cnt, part);
}

template <int NW>
cudaError_t launch_sort_nw(int F, const RowArgs& a, int num_sms, cudaStream_t s) {
  auto kernel = k_sort_rows<NW>;
  const int rows = NW > 1 ? 1 : (F <= 256 ? 8 : 4);  // rows per CTA
  const int threads = NW > 1 ? NW * 32 : rows * 32;
  const size_t smem = sort_row_bytes(F) * rows;
  cudaError_t e;
  if (NW > 1 && sort_row_bytes(512 * NW) > 48 * 1024) {
    e = allow_shared_memory(kernel, sort_row_bytes(512 * NW));
    if (e != cudaSuccess) return e;
  }
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                           cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (int64_t)per_sm * num_sms;
  const int64_t need = (a.nrows + rows - 1) / rows;
  if (grid > need) grid = need;
  kernel<<<(unsigned)grid, threads, smem, s>>>(a, F, ceil_log2_64(F));
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_sort_rows(int max_products, const RowArgs& a, int num_sms, cudaStream_t s) {
  if (a.nrows <= 0) return cudaSuccess;
  const int F = max_products <= 128 ? 128 : (max_products + 127) / 128 * 128;
  switch (sort_warps(F)) {
    case 1: return launch_sort_nw<1>(F, a, num_sms, s);
    case 2: return launch_sort_nw<2>(F, a, num_sms, s);
    case 3: return launch_sort_nw<3>(F, a, num_sms, s);
    case 4: return launch_sort_nw<4>(F, a, num_sms, s);
    case 5: return launch_sort_nw<5>(F, a, num_sms, s);
    case 6: return launch_sort_nw<6>(F, a, num_sms, s);
    case 7: return launch_sort_nw<7>(F, a, num_sms, s);
    case 8: return launch_sort_nw<8>(F, a, num_sms, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace spg
