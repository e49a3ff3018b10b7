// Host-side launchers of the engine's kernels (defined in the k_*.cu files).
// Every launcher is asynchronous on `stream` and returns the launch error.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "device_common.cuh"
#include "internal.h"

namespace spg {

// Kernels launched by the engine on this thread (every <<<>>> site counts).
extern thread_local long long g_kernel_launches;
#define SPG_COUNT_LAUNCH() (++::spg::g_kernel_launches)

// What a kernel may be launched with at most belongs to its function in the
// process's device context, which the engine contexts of all threads share: a
// launcher sets it to one value, the most it ever asks for, never to what the
// launch at hand needs (a thread that lowered it between another's call and launch
// made that launch fail).
template <typename K>
cudaError_t allow_shared_memory(K kernel, size_t most) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

// ---- validation / pre-pass / binning (k_prepass.cu) --------------------------

// Flags DEV_ERR_BAD_INDEX / sets *bad (device int) when A is not a square CSR
// with rowptr[0]=0, monotone rowptr, rowptr[n]=nnz, columns in [0,n) strictly
// increasing within each row.
cudaError_t launch_validate(const MatView& A, uint32_t* status, cudaStream_t s);

// Per row i of C = A·B: products f_i = Σ_{k∈A_i} nnz(B_k) and the column span
// [lo_i, hi_i] of the output row (B rows sorted).  Rows with f_i = 0 get
// lo = INT_MAX, hi = -1; rows that meet an index out of range f_i = −1.  A is
// validated in the same pass (launch_validate's checks), and a row of more than
// fcap products reports DEV_ERR_SMALL_CAP.
cudaError_t launch_prepass(const MatView& A, const MatView& B, int64_t* f, int32_t* lo,
                           int32_t* hi, cudaStream_t s, uint32_t* status, int64_t fcap);

// Sorted rows: the fewest and the most products, the most products per two entries.
// Measured per call, Erdős–Rényi 262,147 (81 products a row) A·Aᵀ / R-MAT 2^14 A·A:
// rows from 96 products on 1.71 ms / -, from 48 1.19 / 1.17, 24 1.14 / 1.14, 8 1.12 /
// 1.12.  Rows that merge more are hashed: sorting up to 2.5 or 4.5 products an entry
// took banded rows 706 and 878 µs against 673 (hashed), the 48-matrix batch 9.2 and
// 9.6 ms against 9.26.  Beyond the warp kernels' largest table the alternative is
// slower: R-MAT 2^15's rows there 174 µs in windows, 10 µs more sorted rows.
constexpr int64_t kSortMinProducts = 8;
constexpr int64_t kSortMaxProducts = 4096;
constexpr int64_t kSortMaxMerge2 = 3;
constexpr int64_t kSortMaxMerge2Large = 6;  // beyond the warp kernels' largest table

// Paneled rows: the narrowest span and the fewest products, in all and per 1024
// columns (a panel costs its task, its slice bounds and a walk over its columns
// whatever it holds).
//
// Rows beyond the sorted rows' range have heavy kernels as their alternative.  From
// kPanelManyProducts a panel on, panels win whatever the row looks like; below, where
// the entries of A have slices worth it (kPanelMinSlice products a panel on average)
// and, over many panels, there are entries enough (the alternative's cost is a barrier
// per entry).  Measured per call, panels / heavy kernels, 2,000 rows over 200,000
// columns: 32 entries of 500 products (82 a panel) 2.40 / 1.25 ms, 32 of 1,000 (163)
// 2.75 / 2.09, 64 of 1,000 (326) 2.28 / 4.80; hub rows of an R-MAT-like graph, 388
// entries over 17 panels (358 products, less than one a slice) 0.52 / 3.24 ms; the hub
// row of an arrowhead of 40,000 went to a single warp, 12.6 -> 4.4 ms.  R-MAT 2^16
// (64 panels) / 2^17 / 2^18, without the condition on the entries 5.26 / 16.5 / 47.3
// ms, with it 5.87 / 15.5 / 43.2, beyond 64 panels only (as below) 5.25 / 15.5 / 43.2.
//
// Smaller rows could be sorted or hashed.  Panels serve them where B's rows are long
// (hubs: kPanelMinMean), or where slices are (kPanelMinSliceSmall) and the row keeps
// kPanelMinEntries entries a panel: a table of few entries is small.  Few are kept
// where the columns of A's row are neighbours (a mesh with several unknowns per node),
// which is all that the symbolic phase can see of it.  Per call, panels / tables,
// 5-point grid of 150 x 150 with six unknowns a node 3.39 / 1.05 ms, four 0.65 / 0.48;
// 27-point grid 34^3 with two 2.97 / 2.49; Erdos-Renyi 3,000 rows of 40 0.26 / 0.34 ms,
// 1,100 of 28 0.20 / 0.29; none of these rows in panels: R-MAT 2^12 0.65 -> 0.82 ms.
// Over three panels or more from kPanelMinMidRow products on: from 256 / 400 / 800 /
// 1600, R-MAT 2^12 0.46 / 0.50 / 0.59 / 0.70 ms and Erdos-Renyi 4,000 rows of 30 0.25 /
// 0.28 / 0.32 / 0.29, but the rows of a 27-point mesh with its nodes renumbered (24^3)
// 0.43 / 0.45 / 0.35 / 0.35 and a thin band of 20,000 (half width 1,300) 0.51 / 0.49 /
// 0.43 / 0.43.  With short rows of B also over one or two panels (a CTA per row in the
// symbolic phase): 40 such meshes of 16^3 in a batch 2.29 -> 1.18 ms, 50 Erdos-Renyi
// matrices of 1,500 rows of 25 1.37 -> 1.19; but not where the matrix has too few rows
// to fill the GPU and launches count: R-MAT 2^11 0.40 -> 0.51 ms, Erdos-Renyi 1,100
// rows of 28 0.22 -> 0.27.
constexpr int32_t kPanelMinSpan = 600;
constexpr int64_t kPanelMinProducts = 64;
constexpr int64_t kPanelManyProducts = 192;
constexpr int64_t kPanelMinSlice = 2;
constexpr int64_t kPanelFewPanels = 64;
constexpr int64_t kPanelMinRow = 256;
constexpr int64_t kPanelMinMidRow = 800;
constexpr int32_t kPanelFewRows = 8192;
constexpr int64_t kPanelMinSliceSmall = 5;
constexpr int64_t kPanelMinMean = 64;
constexpr int64_t kPanelMinEntries = 48;
// Slice bounds are tabulated for every row of B and panel where that is at most so
// many bounds per slice that the paneled rows read (each saves its two searches).  Per
// call with / without the table at 0.08 bounds a slice (R-MAT 2^16) 5.25 / 8.71 ms,
// 1.6 (long rows over 100,000 columns) 1.43 / 2.06, 3.2 1.22 / 1.32, 7.6 10.54 / 10.62,
// 30 and 600 (a few hub rows) no difference beyond 10 µs, for 57 MB.
constexpr int64_t kPanelTableEntries = 8;
// one warp walks a windowed heavy row alone: a larger row would set its tail
constexpr int64_t kWarpRowMaxProducts = (int64_t)1 << 17;

// Narrow rows: the fewest products per entry of A's row (mean B-row length; up
// to kNarrowHalfMean half a warp takes the row), the fewest products per column
// spanned (1 / kNarrowFill), and the fewest and the most products.  Measured per
// call, band of 50,021 / 48-matrix batch / replay of 24: half warps up to a mean of 7
// 402 µs / 7.48 / 3.79 ms, 10 400 / 7.45 / 3.77, 20 416 / 7.50 / 3.82, 40 448 / 7.70 /
// 3.92.  The other lines matter little there (a mean of 3 or 12, one or a sixteenth
// of a product per column, 24 products: all within 1.5%, the run-to-run spread, but
// R-MAT 2^16 5.45 ms against 5.36 with a sixteenth).
constexpr int64_t kNarrowMinMean = 6;
constexpr int64_t kNarrowHalfMean = 10;
constexpr int64_t kNarrowFill = 4;
constexpr int64_t kNarrowMinProducts = 48;
// Rows of up to kNarrowTinySpan columns have small tables, of which a warp takes
// several: summed densely only where B's rows fill more than half of the lanes.
// Numeric phase, dense blocks of 7 / 8 / 10 / 12 / 16 / 20 on the diagonal, narrow
// against tables: 232 / 162, 266 / 169, 322 / 336, 363 / 332, 335 / 300, 313 / 525 µs.
constexpr int64_t kNarrowTinySpan = 16;
constexpr int64_t kNarrowMaxProducts = 1 << 16;

// What a row's bin is computed from.
struct BinSource {
  int mode;                 // 0: symbolic (from products and span), 1: numeric (from counts)
  int32_t n;
  const int64_t* f;
  const int32_t* lo;
  const int32_t* hi;
  const int32_t* rownnz;    // numeric: entries of the row
  int max_log2;             // largest shared table (log2 slots) before the heavy path
  int force_heavy;
  int load_pct;             // table sized for at most this load (percent)
  // symbolic: rows with min(products, span) >= heavy_min also go heavy, so
  // every row the numeric binning sends to the heavy path has block counts
  // from the heavy symbolic kernel (0: no such rule)
  int64_t heavy_min;
  // rows fed by short B rows (products < short_split × nnz(A row); 0: no such
  // rule) go heavy already above 2^short_max_log2 slots (numeric) or from
  // min(products, span) >= short_min (symbolic): the windowed warp kernel
  // serves them better than the CTA-per-row tables, whose per-k barrier idles
  // most of the CTA on short B rows
  const int32_t *arowptr, *acol;
  const unsigned long long* crowd;  // rows looked at, and 2^32 times those found crowded
  int64_t short_split;
  int short_max_log2;
  int64_t short_min;
  // rows whose output span fits 2^dense_max_log2w bitmap words and is at most
  // 8 columns per product, with at least 64 products (and, numeric, at most
  // kDenseVals entries) take the bitmap bins; dense_max_log2w < kDenseMinLog2W:
  // never
  int dense_max_log2w;
  // numeric: rows of up to kSortMaxProducts products of which few
  // merge take the sorted-row kernels
  int sort_rows;
  // rows for the panel kernel, whatever their table (0: none)
  int panels;
  // runs of shifted rows (nullptr: none): rows back to the run's first row, and
  // at that row the run's length and the doubles 32 of its rows need
  const uint8_t* lead;
  const uint16_t* runlen;
  const uint16_t* need;
};

// A row of f products from `len` entries of A over `span` columns: summed densely?
// (The same answer for the symbolic and the numeric binning.)
__host__ __device__ __forceinline__ bool narrow_row_rule(int64_t f, int32_t len, int64_t span) {
  const int64_t lanes = f > kNarrowHalfMean * len ? 32 : 16;
  return (span > kNarrowTinySpan || 2 * f > lanes * len) &&
         span <= kNarrowMin << (kNarrowBins / 2 - 1) && f >= kNarrowMinMean * len &&
         f * kNarrowFill >= span && f >= kNarrowMinProducts &&
         f <= (span > kPanelMinSpan ? kSortMaxProducts : kNarrowMaxProducts);  // (else panels)
}
__host__ __device__ __forceinline__ int narrow_bin(int64_t f, int32_t len, int64_t span) {
  int w = 0;
  while (span > (kNarrowMin << w)) ++w;
  return kNarrowBin0 + 2 * w + (f > kNarrowHalfMean * len ? 1 : 0);
}

// Runs: the fewest rows, and the limits of a row (products, columns spanned) and
// of its operands for 32 rows (doubles), split over the teams of a CTA: two CTAs
// share an SM's 227 KB.  Runs from 32 rows on only: 96³ stencil 2.04 ms against 1.88,
// 47³ 617 against 599 µs; from 4 on: no faster (597 against 587 µs), so 8.  Rows of
// more products were not tried; the lists of 1,024 are the most that leave room for
// the second CTA.
// A run that is whole (not cut at a block of rows, where its other part reuses what
// was found for it) has to be longer: its own steps and idle lanes cost more than they
// save.  Numeric phase of batches of 27-point grids of side 12 / 14 / 16 / 18 / 20 / 24
// (runs of the side less four), runs against tables: 1086 / 452, 1237 / 665, 1269 /
// 958, 1595 / 2480, 1417 / 1424, 990 / 1047 µs; 5-point grids (few entries a row) of 12
// / 16 / 20 / 24 / 30: 201 / 101, 159 / 119, 201 / 170, 200 / 180, 179 / 174.
constexpr int kRunMinRows = 8;
constexpr int kRunMinWhole = 14;
constexpr int kRunMinWholeShort = 24;
constexpr int kRunMaxProducts = 768;
constexpr int kRunMaxSpan = 1 << 18;
constexpr int kRunBuffer = 9216;

// … and of the runs that teams of one warp take.
constexpr int kRunSmallProducts = 192;
constexpr int kRunSmallSpan = 1 << 15;
constexpr int kRunSmallBuffer = 704;

// Team size (log2 warps) of a run whose rows have m entries of f products over
// `span` columns: a warp per 16 entries, and a share of the buffer that holds
// the operands.
__host__ __device__ __forceinline__ int run_team(int64_t m, int need, int64_t f, int64_t span) {
  int t = m <= 16 && f <= kRunSmallProducts && span <= kRunSmallSpan && need <= kRunSmallBuffer ? 0
          : m <= 32                                                                              ? 1
          : m <= 64                                                                              ? 2
                                                                                                 : 3;
  while (t > 0 && t < 3 && need > (kRunBuffer >> (3 - t))) ++t;
  return t;
}

__host__ __device__ __forceinline__ int ceil_log2_64(int64_t x) {
  if (x <= 1) return 0;
#ifdef __CUDA_ARCH__
  return 64 - __clzll(x - 1);
#else
  return 64 - __builtin_clzll((unsigned long long)(x - 1));
#endif
}

// log2 slots of the table that holds `size` entries at `load` percent: the
// smallest L with 2^L >= size · 100 / load + 1 (integer division), that is with
// size · 100 < load · 2^L.
__host__ __device__ __forceinline__ int table_log2(int64_t size, int load) {
  int l = ceil_log2_64(size);
  while (size * 100 >= ((int64_t)load << l)) ++l;
  return l < kMinTableLog2 ? kMinTableLog2 : l;
}

// Products of a row in sorted-row bin b: 128, 256, 512 (a warp), then 768, 1024,
// 1536, 2048, 4096 (a CTA).  Six bins (powers of two) measured 8.74 against
// 8.52 ms on the 48-matrix batch, ten bins no faster than eight.
__host__ __device__ __forceinline__ int sort_bin_products(int b) {
  return b < 3 ? 128 << b : b == 7 ? 4096 : (b & 1 ? 768 : 1024) << ((b - 3) >> 1);
}

// A row of f products and m entries whose columns span `span`: sorted rather
// than hashed?  The words (column − lo) << log2 F | place must fit 32 bits.
__host__ __device__ __forceinline__ bool sorted_row(int64_t f, int64_t m, int64_t span,
                                                    int64_t merge2 = kSortMaxMerge2) {
  return f >= kSortMinProducts && f <= kSortMaxProducts && 2 * f <= merge2 * m &&
         span <= ((int64_t)1 << (32 - ceil_log2_64(f < 128 ? 128 : f)));
}

// Class of a heavy row's products: 0 (2^20 and more) … kHeavyClasses − 1.
__host__ __device__ __forceinline__ int heavy_class(int64_t f) {
  int c = 0;
  while (c < kHeavyClasses - 1 && f < (int64_t)1 << (20 - 2 * c)) ++c;
  return c;
}

// Sorted rows most of whose columns crowd into a small part of their span (a community
// of a graph, with a few links to elsewhere) fill single buckets, and the radix sort
// that takes over is slower than the tables: communities of 400 among 200,000 columns
// 1.71 against 1.48 ms, of 1,000 among 100,000 2.15 against 1.81, of 100 among 60,000
// 194 against 124 µs; with communities of 2,000 among 100,000 sorting is still faster
// (4.4 against 5.8 ms).  One row in 512 is looked at (k_count_tiles; with 64 of them the
// plan of Erdos-Renyi 40,009 took 15 µs more), and where most of those have six of eight
// columns within 2^-kCrowdLog2 of the span none of the matrix's rows are sorted.
constexpr int kCrowdLog2 = 7;
constexpr int kCrowdMin = 48;
__host__ __device__ __forceinline__ bool crowded(unsigned long long crowd) {
  return 2 * (crowd >> 32) > (crowd & 0xffffffffull);
}
// Column t of eight that are spread over a row's products: from the B row of an entry
// at t / 8 of A's row, the entry at t / 8 of it (-1: none).
__device__ __forceinline__ int32_t crowd_column(const int32_t* cols, int32_t len,
                                                const int32_t* browptr, const int32_t* bcol,
                                                int t) {
  const int32_t k = cols[(int64_t)len * (2 * t + 1) >> 4];
  const int32_t bs = browptr[k], m = browptr[k + 1] - bs;
  return m > 0 ? bcol[bs + ((int64_t)m * (2 * t + 1) >> 4)] : -1;
}

// Are the row's columns (len of them, sorted) mostly runs of neighbours?  By eight
// of its entries.  Neighbouring rows of B then hold much the same columns: the
// unknowns of a mesh's node, or the neighbours of a grid point.
__host__ __device__ __forceinline__ bool clumped_columns(const int32_t* cols, int32_t len) {
  int next = 0;
  for (int t = 0; t < 8; ++t) {
    const int32_t p = (int32_t)((int64_t)(len - 1) * t >> 3);
    next += p + 1 < len && cols[p + 1] == cols[p] + 1;
  }
  return next >= 4;
}

// A row of f products from `len` entries of A (their columns: cols) over columns
// [lo, hi] of a matrix of n rows: cut into panels?  `entries`: its entries, -1 while they are not known
// (symbolic phase: a row that is heavy there for its panels may be hashed in the
// numeric phase, but not the reverse, for want of its column counts).
__host__ __device__ __forceinline__ bool paneled_row(int64_t f, int32_t len, const int32_t* cols,
                                                     int32_t lo, int32_t hi, int64_t entries,
                                                     int32_t n) {
  if (f < kPanelMinRow || hi - lo < kPanelMinSpan) return false;
  const int64_t panels = (hi >> 10) - (lo >> 10) + 1;
  if (f < kPanelMinProducts * panels) return false;
  if (f > kSortMaxProducts)
    return f >= kPanelManyProducts * panels ||
           (f >= kPanelMinSlice * panels * len &&
            (panels <= kPanelFewPanels || 2 * (int64_t)len >= panels));
  const bool long_b = f >= kPanelMinMean * len;
  if (f < kPanelMinSliceSmall * panels * len) return false;
  if (f < kPanelMinMidRow && (panels > 2 || (!long_b && n > kPanelFewRows))) return false;
  if (long_b) return true;
  if (entries >= 0 && entries < kPanelMinEntries * panels) return false;
  return !clumped_columns(cols, len);
}

// Table size rule: symbolic tables hold keys only and are sized for the load
// limit (default 75%) of min(products, span); numeric tables hold key+value
// and are sized for the load limit (default 66%) of the exact row count.
// Bin b in 1..kNumTableBins means 2^(b+kMinTableLog2−1) slots.
__host__ __device__ __forceinline__ int row_bin(const BinSource& s, int i) {
  int64_t size;
  if (s.lead && s.lead[i]) return kEmptyBin;  // its run's first row stands for it
  if (s.mode == 0) {
    int64_t f = s.f[i];
    if (f <= 0) return kEmptyBin;
    int64_t span = (int64_t)s.hi[i] - (int64_t)s.lo[i] + 1;
    size = f < span ? f : span;
  } else {
    int64_t m = s.rownnz[i];
    if (m <= 0) return kEmptyBin;
    size = m;
  }
  if (!s.force_heavy) {
    const int32_t len = s.arowptr[i + 1] - s.arowptr[i];
    const int64_t span = (int64_t)s.hi[i] - s.lo[i] + 1;
    if (!(s.mode == 1 && s.lead && s.runlen[i]) && narrow_row_rule(s.f[i], len, span))
      return narrow_bin(s.f[i], len, span);
  }
  if (s.mode == 1 && s.lead && s.runlen[i])
    return kRunBin0 + run_team(size, s.need[i], s.f[i], (int64_t)s.hi[i] - s.lo[i] + 1);
  if (s.panels && paneled_row(s.f[i], s.arowptr[i + 1] - s.arowptr[i], s.acol + s.arowptr[i],
                              s.lo[i], s.hi[i], s.mode == 1 ? size : -1, s.n))
    return s.mode == 1 ? kPanelBin0 : kHeavyBin;
  if (s.force_heavy) return kHeavyBin;
  int lg = table_log2(size, s.load_pct);
  if (s.mode == 1 && s.sort_rows && lg <= s.max_log2 && !crowded(*s.crowd) &&
      sorted_row(s.f[i], size, (int64_t)s.hi[i] - s.lo[i] + 1,
                 lg > s.short_max_log2 ? kSortMaxMerge2Large : kSortMaxMerge2)) {
    int b = 0;
    while (sort_bin_products(b) < s.f[i]) ++b;
    return kSortBin0 + b;
  }
  if (s.mode == 0 && s.heavy_min > 0 && size >= s.heavy_min) return kHeavyBin;
  if (s.dense_max_log2w >= kDenseMinLog2W) {
    const int64_t words = ((int64_t)s.hi[i] - s.lo[i] + 32) >> 5;
    const int64_t f = s.f[i];
    // (symbolic: only rows the numeric binning can never send heavy, which
    // need the heavy symbolic kernel's block counts)
    // the bitmap's bookkeeping (clearing, counting, prefixes) grows with the
    // span: worth it only where the span is at most 8 columns per product
    if (f >= 64 && words * 4 <= f && words <= ((int64_t)1 << s.dense_max_log2w) &&
        (s.mode == 0 ? (s.short_split <= 0 || size < s.short_min) : size <= kDenseVals)) {
      int lw = ceil_log2_64(words);
      if (lw < kDenseMinLog2W) lw = kDenseMinLog2W;
      return kDenseBin0 + lw - kDenseMinLog2W;
    }
  }
  if (lg > s.max_log2) return kHeavyBin;
  if (s.short_split > 0 &&
      s.f[i] < s.short_split * ((int64_t)s.arowptr[i + 1] - s.arowptr[i]) &&
      (s.mode == 0 ? size >= s.short_min : lg > s.short_max_log2))
    return kHeavyBin;
  return lg - kMinTableLog2 + 1;
}

constexpr int kBinRowsPerBlock = 256;  // rows per block of the binning kernels

// Binning: the rows of each bin listed one bin after another (in row order within
// blocks of kBinRowsPerBlock rows).
//   bin: a byte per row; work: kBinWork int64 on the device, of which the first
//   kBinBack come back: the rows of each bin; the blocks of 1024 columns that the
//   heavy (symbolic phase) or the paneled rows (numeric) span, and the slices of B
//   rows that the latter read there (blocks times entries of A)
constexpr int kBinBack = kNumBins + 2;
constexpr int kBinWork = kBinBack + kNumBins;
// `skip` (device, may be null): where it is not 0 nothing is done (work stays 0).
cudaError_t launch_bin_rows(const BinSource& src, uint8_t* bin, int64_t* work, int32_t* rows_out,
                            cudaStream_t s, const int* skip = nullptr);

// Exclusive scan of int32 counts into int64 offsets out[0..n], out[n] = total.
// `tmp` needs scan_tmp_bytes(n) bytes.
size_t scan_tmp_bytes(int64_t n);
cudaError_t launch_scan_i32_i64(const int32_t* in, int64_t* out, int64_t n, void* tmp,
                                cudaStream_t s);
// Same with int32 output (caller guarantees the total fits in int32).
cudaError_t launch_scan_i32_i32(const int32_t* in, int32_t* out, int64_t n, void* tmp,
                                cudaStream_t s);

// ---- shared-memory hash rows (k_rows.cu) ------------------------------------

struct RowArgs {
  MatView A, B;
  const int32_t* rows;      // this bin's rows (nullptr: rows 0..nrows-1)
  int32_t nrows;
  int32_t G;                // lanes per row (warp bins); CTA bins use blockDim
  // symbolic outputs
  int32_t* rownnz;
  // numeric inputs / outputs
  const int64_t* rowptr;    // C row pointers
  const int32_t* cnt_in;    // symbolic counts (expected entries)
  int32_t* ccol;
  double* cval;
  uint32_t* status;
  // output column span per row (pre-pass): keys of row i lie in [lo[i], hi[i]]
  const int32_t* lo;
  const int32_t* hi;
  // batched plans: first column of the row's instance, subtracted from every
  // column index written (nullptr for a single matrix)
  const int32_t* colbase;
  // CTA-per-row bins: in a persistent launch rows are drawn from this counter
  // (zeroed by the launcher) as CTAs free up; nullptr: dealt out in turn
  int32_t* queue;
  // the one-readback plan's symbolic launch (warp kernels): rows whose
  // pre-pass product count is negative (an invalid index met) or above fcap
  // (beyond the table) are skipped with a zero count, the latter reported as
  // DEV_ERR_SMALL_CAP; nullptr: every row is processed
  const int64_t* fsmall;
  int64_t fcap;
  const uint16_t* runlen;   // runs of shifted rows: rows of the run that starts here
};

// Writes m sorted packed words ((col − lo) << LOG2T | slot) as a row's columns
// and the values of their table slots, lanes first, first + stride, … (so the
// stores are coalesced).
template <int LOG2T>
__device__ __forceinline__ void emit_packed(const RowArgs& a, int row, int lo, int m,
                                            const uint32_t* sorted, const double* vals,
                                            int64_t base, int first, int stride) {
  const int cb = a.colbase ? a.colbase[row] : 0;
  for (int e = first; e < m; e += stride) {
    const uint32_t pk = sorted[e];
    const int j = lo + (int)(pk >> LOG2T);
    const double v = vals[pk & ((1u << LOG2T) - 1u)];
    a.ccol[base + e] = j - cb;
    a.cval[base + e] = v;
  }
}

// Marks the columns of a row's products, column − lo < span, with a byte each
// (symbolic phase): plain stores of 1, in no order.  G lanes per row; the B rows
// are walked in pieces of G entries, eight pieces' loads in flight.
template <int G>
__device__ __forceinline__ void narrow_mark(const RowArgs& a, const WarpGroup& g, int row, int lo,
                                            int span, unsigned char* seen) {
  constexpr int kAhead = 8;
  const Pos ps = a.A.rowptr[row], pe = a.A.rowptr[row + 1];
  for (Pos pb = ps; pb < pe; pb += G) {
    const int cnt = min(G, pe - pb);
    int bs = 0, len = 0;
    if (g.lane < cnt) {
      const int32_t k = a.A.col[pb + g.lane];
      bs = a.B.rowptr[k];
      len = a.B.rowptr[k + 1] - bs;
    }
    for (int t0 = 0; t0 < cnt; t0 += kAhead) {
      int b[kAhead], l[kAhead], x[kAhead];
      int longest = 0;
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int t = min(t0 + u, G - 1);
        b[u] = __shfl_sync(g.mask, bs, t, G);
        l[u] = __shfl_sync(g.mask, len, t, G);
        if (t0 + u >= cnt) l[u] = 0;
        longest = max(longest, l[u]);
        x[u] = g.lane < l[u] ? a.B.col[b[u] + g.lane] - lo : -1;
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if ((unsigned)x[u] < (unsigned)span) seen[x[u]] = 1;
      for (int q = G; q < longest; q += G) {  // what is left of the longer ones
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          x[u] = q + g.lane < l[u] ? a.B.col[b[u] + q + g.lane] - lo : -1;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if ((unsigned)x[u] < (unsigned)span) seen[x[u]] = 1;
      }
    }
  }
}

// Number of bits needed for the column field of a row spanning [lo, hi].
__device__ __forceinline__ int span_bits(int lo, int hi) {
  const uint32_t span = (uint32_t)(hi - lo);
  return span ? 32 - __clz((int)span) : 0;
}

// Numeric-zero compaction (k_compact.cu): kept (non-zero) entries per row of
// C, and the kept entries of rows [r0, r1) gathered in order into tcol/tval
// at newptr[row] − newptr[r0].
cudaError_t launch_count_kept(const int64_t* rowptr, const double* val, int32_t n, int32_t* kept,
                              cudaStream_t s);
cudaError_t launch_gather_kept(const int64_t* rowptr, const int32_t* col, const double* val,
                               const int64_t* newptr, int32_t r0, int32_t r1, int32_t* tcol,
                               double* tval, cudaStream_t s);

// Warp-per-row kernels (k_rows_w32.cu) for table bins of up to 2048 slots
// with 32 lanes per row; returns cudaErrorNotSupported for other bins.
cudaError_t launch_hash_w32(int log2t, bool numeric, const RowArgs& a, int num_sms,
                            cudaStream_t s);

// Launch the kernel of one table bin (1..kNumTableBins).
cudaError_t launch_hash_bin(int bin, bool numeric, const RowArgs& a, int num_sms,
                            cudaStream_t s);
// Warp-per-row bitmap kernels of the dense bins (k_dense_w32.cu).
cudaError_t launch_dense_bin(int bin, bool numeric, const RowArgs& a, int num_sms,
                             cudaStream_t s);
int hash_bin_lanes(int bin, int lanes_cfg);
// Narrow rows of up to W columns, `lanes` (16 or 32) per row (k_narrow.cu).
cudaError_t launch_narrow(bool numeric, int W, int lanes, const RowArgs& a, int num_sms,
                          cudaStream_t s);
// The pre-pass of the regular plans (k_runs.cu): products and column span per
// row, the validation of A and, with `lead`, the runs of shifted rows.  Per row
// of B: info; per row of A: the others (mid: scratch); marks: three ints; pieces:
// prepass_pieces(nnz).
// (rows of more than 256 entries, in pieces of 1024: at most 1.25 nnz / 256)
constexpr int64_t prepass_pieces(int64_t nnz) { return nnz / 200 + 1; }
struct PrepassArrays {
  int4* info;
  int64_t* f;
  int32_t *lo, *hi, *marks, *mid;
  int2* pieces;
  uint8_t *flag_a, *flag_b, *lead;
  uint16_t *need, *runlen;
};
cudaError_t launch_prepass_rows(const MatView& A, const MatView& B, const PrepassArrays& w,
                                int num_sms, uint32_t* status, cudaStream_t s,
                                const int* skip = nullptr);
// Runs of shifted rows: the numeric phase of the runs whose first rows are listed
// (teams of 2^team warps).
cudaError_t launch_runs(int team, const RowArgs& a, int num_sms, cudaStream_t s);
// Sorted rows of up to max_products <= kSortMaxProducts products each, numeric
// phase (k_sort_rows.cu).
cudaError_t launch_sort_rows(int max_products, const RowArgs& a, int num_sms, cudaStream_t s);

// ---- heavy rows: dense column windows (k_heavy.cu) --------------------------
struct HeavyArgs {
  RowArgs r;                // rows = heavy list, outputs as in RowArgs
  const int32_t* lo;        // output column span per row
  const int32_t* hi;
  int32_t window_bits;      // W (multiple of 32 * threads)
  // column blocks: heavy row i's span [lo, hi] is cut at multiples of
  // 2^blk_log2 columns; blk_cnt[blk_off[i] + b] is the number of distinct output
  // columns in its b-th block (saturated at 65535), written by the
  // symbolic kernel when blk_cnt is set and read by the windowed numeric one
  const int64_t* blk_off;   // per row (n + 1), 0 blocks for rows not heavy
  uint16_t* blk_cnt;
  int32_t blk_log2;
  int32_t cap;              // numeric: most distinct columns per window
  int32_t sub_log2;         // numeric: window width inside a block above cap
  int4* hcur;               // numeric: per entry of A {B cursor, B row end, next column, 0}
  int32_t vcap;             // shared-value CTA kernel: most values per window
  int32_t wcap_bits;        // shared-value CTA kernel: widest window (bitmap bits)
  // numeric: rows fed by many short B rows (mean length below `split`) take
  // the windowed warp kernel, rows dominated by long B rows the CTA kernel,
  // whose 1024 threads stream each long B row (each kernel skips the other's
  // rows); split 0: all to the CTA kernel
  int64_t split;
  const int64_t* f;         // products per row (pre-pass)
  // CTA kernels: in a persistent launch (fewer CTAs than rows) a CTA takes its
  // next row from this counter (launch_heavy zeroes it on the stream first),
  // so a CTA that drew hub rows does not hold the others back; required
  int32_t* queue;
  // panel kernel (k_panel.cu): panels of 2^pan_log2 columns, npan of them over
  // n columns; slice bounds (nullptr: searched for) and task counter set by
  // launch_panels
  int32_t pan_log2, npan;
  const int32_t* ptr;
  int64_t* task_queue;
  int64_t tasks;            // at most so many panels
  bool retire;              // a warp leaves after its share of them (grid_sms)
};

// The heavy row goes to the windowed warp kernel: mean B-row length
// f / nnz(A row) below split, and at most kWarpRowMaxProducts products.
__device__ __forceinline__ bool heavy_row_windowed(const HeavyArgs& h, int row) {
  if (h.split <= 0 || h.f[row] > kWarpRowMaxProducts) return false;
  const int64_t len = (int64_t)h.r.A.rowptr[row + 1] - h.r.A.rowptr[row];
  return h.f[row] < h.split * len;
}
cudaError_t launch_heavy(bool numeric, const HeavyArgs& a, int threads, int num_sms,
                         cudaStream_t s);
size_t heavy_smem_bytes(bool numeric, int threads, int window_bits);

// Blocks per row for the heavy rows of `bsym` (0 for the others), scanned into
// blk_off[0..n] (launch_scan_i32_i64 with tmp of scan_tmp_bytes(n)).
cudaError_t launch_heavy_blocks(const BinSource& bsym, int blk_log2, int32_t* nblk,
                                int64_t* blk_off, void* scan_tmp, cudaStream_t s);

// Numeric phase of the CTA rows with their values in shared memory, window by
// window (k_heavy_win.cu); needs blk_cnt, hcur and queue.
cudaError_t launch_heavy_win(const HeavyArgs& a, int threads, int num_sms,
                             cudaStream_t s);
size_t heavy_win_smem_bytes(int threads, int vcap, int wcap_bits);

// Windowed numeric phase of heavy rows (k_heavy_w32.cu): a warp per row walks
// the row's column blocks in windows of at most `cap` distinct columns.
cudaError_t launch_heavy_w32(const HeavyArgs& a, int num_sms, cudaStream_t s);
// Numeric phase of the rows cut into panels (k_panel.cu), in `workspace` of
// panel_workspace bytes (with or without the table of slice bounds); sets h.ptr
// and h.task_queue.
__host__ __device__ constexpr size_t panel_warp_bytes(int pan_log2) { return ((size_t)8 << pan_log2) + 512; }
int64_t panel_workspace(int64_t n, int npan, int64_t nrows, bool table);
cudaError_t launch_panels(HeavyArgs& h, void* workspace, bool table, int num_sms,
                          cudaStream_t s);
constexpr int kHeavyTableLog2 = 10;  // its shared table: 1024 slots per warp

// ---- transpose and segment sort (k_transpose.cu) ----------------------------

// Counting-sort transpose: t_rowptr (n+1) gets the column histogram scan,
// entries are appended per column with atomic cursors into (tmp_col, tmp_val),
// then each column is sorted by row into (t_col, t_val).
// Workspace: cnt/cursor int32[n], scan tmp, tmp_col/tmp_val [nnz], long list.
struct TransposeWork {
  int32_t* cnt;
  int32_t* cursor;
  void* scan_tmp;
  int32_t* tmp_col;
  double* tmp_val;
  int32_t* long_list;   // int32[n]
  int32_t* long_count;  // int32[1]
  uint32_t* status;
};
cudaError_t launch_transpose(const MatView& A, int32_t* t_rowptr, int32_t* t_col, double* t_val,
                             const TransposeWork& w, int num_sms, cudaStream_t s);
// Values of Aᵀ for a structurally symmetric A (Aᵀ keeps A's rowptr and col);
// sets *asym (device int, pre-zeroed) when some entry has no mirror.
cudaError_t launch_sym_transpose_vals(const MatView& A, double* t_val, int* asym, cudaStream_t s);

// Sort segments of unique int keys (with double payloads) from a source store
// into a destination store.  Segment s: source [src_off[s], +len), destination
// [dst_off[s], +len), len = lens ? lens[s] : src_off[s+1] − src_off[s].
struct SegSortArgs {
  int32_t nseg;
  const int32_t* off;    // segment s: entries off[s] … off[s + 1] of both sides
  const int32_t* src_key;
  const double* src_val;
  int32_t* dst_key;
  double* dst_val;
  int32_t key_bound;     // keys lie in [0, key_bound)
  int32_t* long_list;
  int32_t* long_count;
  uint32_t* status;
};
cudaError_t launch_segsort(const SegSortArgs& a, int num_sms, cudaStream_t s);

// ---- batched plans (k_batch.cu) ---------------------------------------------
struct BatchDesc {          // one instance, as uploaded to the device
  const int32_t* rowptr;
  const int32_t* col;
  const double* val;
  int32_t n;
  int32_t pad;
  int64_t nnz;
  int64_t row_off;          // first row (and column) of the instance in the block diagonal
  int64_t nnz_off;          // first entry of the instance
};
// Block-diagonal concatenation: rowptr (N+1), col/val (NNZ) with columns offset
// by the instance's row_off, colbase[r] = row_off of row r's instance.  Sets
// *bad when an instance's rowptr does not run 0..nnz or a column leaves its block.
cudaError_t launch_batch_concat(const BatchDesc* d, const int64_t* row_off, const int64_t* nnz_off,
                                int count, int64_t N, int64_t NNZ, int32_t* rowptr, int32_t* col,
                                double* val, int32_t* colbase, uint32_t* bad, int num_sms,
                                cudaStream_t s);
// Refresh only the values of the block-diagonal copy from the instances.
cudaError_t launch_batch_vals(const BatchDesc* d, const int64_t* nnz_off, int count, int64_t NNZ,
                              double* val, int num_sms, cudaStream_t s);
// out[b] = rowptr_c[row_off[b]] for b = 0..count.
cudaError_t launch_gather_offsets(const int64_t* rowptr_c, const int64_t* row_off, int count,
                                  int64_t* out, cudaStream_t s);

// ---- descriptors ------------------------------------------------------------
struct DescAccum {        // device accumulators of spg_describe
  unsigned long long sum_deg2;   // Σ deg²
  unsigned long long prod_aa;    // Σ_{(i,k)} deg(k)
  unsigned long long prod_aat;   // Σ_k colcount²
  unsigned long long sym_hits;   // entries (i,j) with (j,i) present
  int max_deg;
  int max_col_deg;
  int bandwidth;
  int pad;
};
cudaError_t launch_describe(const MatView& A, const int32_t* colcount, DescAccum* acc,
                            cudaStream_t s);
// Row pointers of C from the row counts (with `lead`, a run's rows take its
// first row's count first), and kRowStats statistics: Σ products, max products,
// max row count, max column span, nnz(C), and the device status words as they are
// then, and the rows looked at for crowding with 2^32 times those found so.  cnt, f, lo, hi: 16-byte aligned.  tmp: scan_tmp_bytes(n).
constexpr int kRowStats = 7;
cudaError_t launch_row_pointers(const MatView& A, const MatView& B, int32_t* cnt,
                                const uint8_t* lead, const int64_t* f, const int32_t* lo,
                                const int32_t* hi, int64_t n, int64_t* rowptr,
                                unsigned long long* stats, const uint32_t* status, void* tmp,
                                cudaStream_t s);
cudaError_t launch_col_count(const MatView& A, int32_t* cnt, cudaStream_t s);

}  // namespace spg
