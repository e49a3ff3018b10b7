// Narrow rows: rows of C whose columns span at most 1024 columns (banded
// matrices), summed densely in shared memory by a warp or half of one.
//
// In the hash kernels every product probes for its column and a row ends with a
// sort, although a banded row's columns are already places: 1,500 products over
// 190 columns took 1,500 probes.  Here a product is added at column − lo: no
// probe, no sort, and the row is written in column order.  The places start as
// −0.0, which no sum can be (the sums start from +0.0, and x + y is −0.0 only
// when both are), and a product has 0.0 added first (−0.0 becomes +0.0, nothing
// else changes): the places that still hold −0.0 at the end have no entry.  One
// group synchronisation per B-row segment keeps the k order of every sum, so the
// values are those of the other kernels, bit for bit.  The symbolic phase marks
// a byte per column with plain stores (every store writes 1, so they need no
// order and no atomics) and counts the bytes.
//
// Random band of 50,021 rows and half-bandwidth 48: numeric 347 -> 157 µs, symbolic
// 154 -> 117 µs, call 652 -> 385 µs.  Bound by issue (74% of slots) and
// shared-memory wavefronts (73%): about 2.5 warp instructions a product.  Walking
// the B rows without the list of segments took 207 against 145 µs (its loop
// control was most of its 3.7 instructions a product).
#include "kernels.h"

namespace spg {

namespace {

constexpr int kAhead = 4;       // segments loaded ahead
constexpr int kSegments = 64;   // segments listed at a time
constexpr long long kAbsent = (long long)0x8000000000000000ull;  // −0.0

// Up to G consecutive entries of a B row and the entry of A that they multiply.
struct __align__(16) Segment {
  double a;
  int32_t start, count;
};

template <int G>
__device__ __forceinline__ void narrow_row(const RowArgs& a, const WarpGroup& g, int row,
                                           double* acc, Segment* segs, int W) {
  const int lo = a.lo[row];
  const int span = min(a.hi[row] - lo + 1, W);
  const Pos ps = a.A.rowptr[row], pe = a.A.rowptr[row + 1];
  const int32_t* bcol = a.B.col + g.lane;
  const double* bval = a.B.val + g.lane;
  for (Pos pb = ps; pb < pe;) {
    // the segments of the next entries of A's row, as many whole entries as the
    // list takes (a B row lies within the span: at most 1024 / G segments)
    int start = 0, len = 0;
    double av = 0.0;
    if (pb + g.lane < pe) {
      const int32_t k = a.A.col[pb + g.lane];
      start = a.B.rowptr[k];
      len = a.B.rowptr[k + 1] - start;
      av = a.A.val[pb + g.lane];
    }
    const int n = (len + G - 1) / G;
    int incl = n;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const int t = __shfl_up_sync(g.mask, incl, o, G);
      if (g.lane >= o) incl += t;
    }
    const unsigned taken = g.ballot(pb + g.lane < pe && incl <= kSegments);  // a prefix
    const int entries = __popc(taken);
    if (entries == 0) {  // not what the plan saw
      if (g.lane == 0) report(a.status, DEV_ERR_OVERFLOW);
      break;
    }
    const int total = __shfl_sync(g.mask, incl, entries - 1, G);
    g.sync();  // the previous segments are used up
    if (g.lane < entries)
      for (int i = 0; i < n; ++i) {
        Segment sg;
        sg.a = av;
        sg.start = start + i * G;
        sg.count = min(G, len - i * G);
        segs[incl - n + i] = sg;
      }
    if (g.lane < kAhead) {
      Segment none;
      none.a = 0.0;
      none.start = none.count = 0;
      segs[total + g.lane] = none;
    }
    g.sync();
    pb += entries;
    int col[kAhead];
    bool in[kAhead];
    double lv[kAhead], rv[kAhead];
    auto fetch = [&](int s) {
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const Segment sg = segs[s + u];
        in[u] = g.lane < sg.count;
        col[u] = in[u] ? bcol[sg.start] : 0;
        rv[u] = in[u] ? bval[sg.start] : 0.0;
        lv[u] = sg.a;
      }
    };
    fetch(0);
    for (int s = 0; s < total; s += kAhead) {
      int x[kAhead];
      bool on[kAhead];
      double v[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        x[u] = (col[u] - lo) & (W - 1);
        on[u] = in[u];
        v[u] = __dadd_rn(__dmul_rn(lv[u], rv[u]), 0.0);
      }
      if (s + kAhead < total) fetch(s + kAhead);
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        if (on[u]) acc[x[u]] = __dadd_rn(acc[x[u]], v[u]);
        g.sync();  // k-order of the accumulation
      }
    }
  }
  // write the row in column order and leave its places absent
  const int64_t base = a.rowptr[row];
  const int expect = a.cnt_in[row];
  const int cb = a.colbase ? a.colbase[row] : 0;
  int written = 0;
  for (int c = 0; c < span; c += G) {
    const int x = c + g.lane;
    const double v = x < span ? acc[x] : __longlong_as_double(kAbsent);
    const bool have = __double_as_longlong(v) != kAbsent;
    const unsigned bal = g.ballot(have);
    const int pos = written + __popc(bal & ((1u << g.lane) - 1u));
    if (have) {
      acc[x] = __longlong_as_double(kAbsent);
      if (pos < expect) {
        a.ccol[base + pos] = lo + x - cb;
        a.cval[base + pos] = v;
      }
    }
    written += __popc(bal);
  }
  if (g.lane == 0 && written != expect) report(a.status, DEV_ERR_OVERFLOW);
  g.sync();
}

// Numeric: W places (a power of two) per row, 32 / G rows per warp.
template <int G>
__global__ void __launch_bounds__(256) k_narrow_num(RowArgs a, int W) {
  extern __shared__ __align__(16) unsigned char smem[];
  const WarpGroup g(G);
  const int per_cta = blockDim.x / G, gi = threadIdx.x / G;
  double* acc = (double*)smem + (size_t)gi * W;
  Segment* segs =
      (Segment*)((double*)smem + (size_t)per_cta * W) + (size_t)gi * (kSegments + kAhead);
  for (int x = g.lane; x < W; x += G) acc[x] = __longlong_as_double(kAbsent);
  g.sync();
  for (int r = blockIdx.x * per_cta + gi; r < a.nrows; r += gridDim.x * per_cta)
    narrow_row<G>(a, g, a.rows ? a.rows[r] : r, acc, segs, W);
}

// Symbolic: a byte per column.
template <int G>
__global__ void __launch_bounds__(256) k_narrow_sym(RowArgs a, int W) {
  extern __shared__ __align__(16) unsigned char smem[];
  const WarpGroup g(G);
  const int per_cta = blockDim.x / G, gi = threadIdx.x / G;
  unsigned char* seen = smem + (size_t)gi * W;
  for (int x = g.lane * 4; x < W; x += G * 4) *(uint32_t*)(seen + x) = 0u;
  g.sync();
  for (int r = blockIdx.x * per_cta + gi; r < a.nrows; r += gridDim.x * per_cta) {
    const int row = a.rows[r];
    const int lo = a.lo[row];
    const int span = min(a.hi[row] - lo + 1, W);
    narrow_mark<G>(a, g, row, lo, span, seen);
    g.sync();
    int c = 0;
    for (int x = g.lane * 4; x < span; x += G * 4) {
      c += __popc(*(const uint32_t*)(seen + x));
      *(uint32_t*)(seen + x) = 0u;
    }
    c = g.sum(c);
    if (g.lane == 0) a.rownnz[row] = c;
    g.sync();
  }
}

template <typename K>
cudaError_t launch_narrow_k(K kernel, int rows, int threads, size_t smem, const RowArgs& a, int W,
                            int num_sms, cudaStream_t s) {
  // (smem is at most 48 KB: two rows of 1024 columns take 18 KB)
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  int64_t grid = (int64_t)per_sm * num_sms;
  const int64_t need = (a.nrows + rows - 1) / rows;
  if (grid > need) grid = need;
  kernel<<<(unsigned)grid, threads, smem, s>>>(a, W);
  SPG_COUNT_LAUNCH();
  return cudaGetLastError();
}

template <int G>
cudaError_t launch_narrow_g(bool numeric, int W, const RowArgs& a, int num_sms, cudaStream_t s) {
  const size_t per = numeric ? (size_t)W * 8 + (kSegments + kAhead) * sizeof(Segment) : (size_t)W;
  int rows = 256 / G;  // per CTA
  while (rows > 32 / G && per * rows > 48 * 1024) rows >>= 1;
  if (numeric) return launch_narrow_k(k_narrow_num<G>, rows, rows * G, per * rows, a, W, num_sms, s);
  return launch_narrow_k(k_narrow_sym<G>, rows, rows * G, per * rows, a, W, num_sms, s);
}

}  // namespace

cudaError_t launch_narrow(bool numeric, int W, int lanes, const RowArgs& a, int num_sms,
                          cudaStream_t s) {
  if (a.nrows <= 0) return cudaSuccess;
  return lanes == 16 ? launch_narrow_g<16>(numeric, W, a, num_sms, s)
                     : launch_narrow_g<32>(numeric, W, a, num_sms, s);
}

}  // namespace spg
