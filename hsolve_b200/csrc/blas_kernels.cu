// HBM-bound kernels of the Krylov loop (sm_100a, FP64):
//  * CSR SpMM  Y = M X  (replaces hsolve's spmm, src/sparse/kernels.cpp:797);
//  * fused shifted residual R = B (X + sigma Y) - A Y with its column norms (shifted_residual,
//    src/sparse/kernels.cpp:850; contract include/hsolve/sparse.hpp:157-174);
//  * tall-skinny Gram G = X^T Y with a fixed-order two-stage reduction (bitwise reproducible), and
//    Y = beta Y + alpha X S for the block Gram-Schmidt / CholQR updates and Ritz vectors
//    (BlockOrthonormalizer, src/eigen/block_ortho.cpp:165,270; orthogonalize_block_cgs2,
//    src/linalg/dense_ops.hpp:180).
#include <algorithm>
#include <cstdint>
#include <mutex>

#include <math_constants.h>

#include "blas_kernels.cuh"
#include "common.hpp"
#include "device.cuh"

namespace hsg {

void cuda_check(cudaError_t e, const char* what);

namespace {

// Rows of a CSR product: a CTA takes a chunk of 64 rows (16 where the matrix has few) and sums each by four
// lanes: the entries of a row are read by neighbouring lanes, the gathers of neighbouring rows fall into the same
// lines, and the partial sums take two shuffle steps. A curl-curl row has at most 13 entries: a warp per row left
// 19 lanes idle and spent most of its time in five-step reductions (the call for the residual of 8 columns at
// n = 21,660: 135 us, now 23).
//
// Longer rows want more lanes: chunks above most_entries a row take sixteen lanes a row, rows above kLongRow a
// warp each. With four lanes up to 128 entries and the warp's own eight rows one after another above, the
// residual of 8 columns took 33 us at n = 3,000 with 64 entries a row (now 24; a warp per row 42), 107 with 192
// entries (38; 57) and 1,104 where 8 of the 3,000 rows were full (160; 214); a product of 8 columns 523 us there
// (60; 95).
constexpr int kRowThreads = 256;
constexpr int kRowWarps = kRowThreads / 32;
constexpr int kChunk = kRowThreads / 4, kSmallChunk = kRowThreads / 16;
constexpr int kSmallRows = 444 * kSmallChunk;  // 16 lanes a row fill three CTAs an SM
constexpr int kLongRow = 512;

// Entries a row up to which a chunk takes four lanes a row. In few rows they leave the device idle (n = 3,000,
// residual of 8 columns, four and sixteen lanes: 13 entries 22 and 20 us, 30 entries 28 and 21; one column
// 17.4 and 18.4, 17.3 and 17.7); in many rows they move less (n = 100,000, 8 columns, 96 entries: 173 and
// 308 us, 128 entries 211 and 397; a product of one column 42 and 39, 51 and 44).
template <int P>
__device__ __forceinline__ int most_entries(int chunk) {
  return chunk == kSmallChunk ? 24 : (P == 1 ? 96 : 128);
}

// f(value, column) for this lane's entries of the row [q0, q1): every G-th, kAhead of them read before the
// gathers (a curl-curl row is one batch).
template <int G, int kAhead, bool kWhole, class Fn>
__device__ __forceinline__ void group_entries(std::int64_t q0, std::int64_t q1, const std::int32_t* ci, const double* v,
                                              Fn&& f) {
  std::int64_t q = q0 + (threadIdx.x & (G - 1));
  // rows of many batches: the whole ones without tests (not with eight columns, whose sums leave no registers for
  // a second copy of the batch: a product of 3,000 rows with 128 entries took 24 us, 18 without)
  if constexpr (G > 4 && kWhole) {
    for (; q + G * (kAhead - 1) < q1; q += G * kAhead) {
      double a[kAhead];
      std::int32_t j[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        a[u] = v[q + G * u];
        j[u] = ci[q + G * u];
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) f(a[u], j[u]);
    }
  }
  for (; q < q1; q += G * kAhead) {
    double a[kAhead];
    std::int32_t j[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      a[u] = q + G * u < q1 ? v[q + G * u] : 0.0;
      j[u] = q + G * u < q1 ? ci[q + G * u] : -1;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (j[u] >= 0) f(a[u], j[u]);
  }
}

// The G lanes' sums of P columns, scattered: a lane keeps columns first .. first + kCols in a[0 ..] (several
// lanes the same column where P < G: `writer` is one of them); a halving of the columns a step while there
// are columns to halve, which is half the shuffles of a full reduction.
constexpr int log2i(int v) { return v <= 1 ? 0 : 1 + log2i(v / 2); }
template <int P, int G>
struct GroupCols {
  static constexpr int kHalvings = log2i(P) < log2i(G) ? log2i(P) : log2i(G);
  static constexpr int kCols = P >> kHalvings, kShare = G >> kHalvings;
  int first;
  bool writer;
  __device__ __forceinline__ GroupCols() {
    const int sub = threadIdx.x & (G - 1);
    first = sub / kShare * kCols;
    writer = sub % kShare == 0;
  }
  __device__ __forceinline__ static void sum(double (&a)[P]) {
    int width = P;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const bool up = (threadIdx.x & o) != 0;
      if (width > 1) {
        width /= 2;
#pragma unroll
        for (int c = 0; c < P / 2; ++c)
          if (c < width) {
            const double send = up ? a[c] : a[c + width], keep = up ? a[c + width] : a[c];
            a[c] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
      } else {
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
      }
    }
  }
};

// The rows of a matrix, chunk by chunk: quad(i, span(i, end)) for this lane's row i of a chunk that ends at `end`,
// by four lanes (i may lie beyond), or wide(row0, end) for a chunk of many entries; entries(a, b) are those of the
// rows [a, b). Both leave out the long rows, which take a warp each, long_row(i): a CTA's warps share those of
// eight groups spread over the matrix, so that neighbouring long rows meet as many CTAs as there are groups of
// them (1,000 rows of 1,000 entries at the end of 100,000 of 13, a product of 8 columns: 365 us by the warps of
// the rows' own chunks, now 83).
template <int P, class Span, class Entries, class Quad, class Wide, class LongRow>
__device__ __forceinline__ void for_rows(std::int64_t n, int chunk, Span&& span, Entries&& entries, Quad&& quad,
                                         Wide&& wide, LongRow&& long_row) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group_rows = chunk / kRowWarps, group_lanes = kRowThreads / chunk;
  const auto group = [&](int w) { return (w * static_cast<std::int64_t>(gridDim.x) + blockIdx.x) * group_rows; };
  const std::int64_t row0 = blockIdx.x * static_cast<std::int64_t>(chunk), end = row0 + chunk < n ? row0 + chunk : n;
  const std::int64_t i = row0 + (threadIdx.x >> 2), k = group(warp) + lane / group_lanes;
  // (all row pointers are read at once, before the chunk's kind is known)
  const auto mine = span(i, end);
  const bool is_long = k < n && entries(k, k + 1) > kLongRow;
  if (entries(row0, end) > most_entries<P>(chunk) * (end - row0)) wide(row0, end);
  else if (__any_sync(0xffffffffu, i < end)) quad(i, mine);
  if (!__syncthreads_or(is_long)) return;
  __shared__ unsigned mask[kRowWarps];
  const unsigned found = __ballot_sync(0xffffffffu, lane % group_lanes == 0 && is_long);
  if (lane == 0) mask[warp] = found;
  __syncthreads();
  int turn = 0;
  for (int w = 0; w < kRowWarps; ++w)
    for (unsigned m = mask[w]; m; m &= m - 1)
      if (turn++ % kRowWarps == warp) long_row(group(w) + (__ffs(m) - 1) / group_lanes);
}

struct SpmmArgs {
  std::int64_t n;
  const std::int64_t* rp;
  const std::int32_t* ci;
  const double* v;
  const double* x;
  std::int64_t ldx;
  double* y;
  std::int64_t ldy;
  int p;
  double alpha, beta;
};

// Row i of y = alpha M x + beta y by G lanes; [q0, q1): its entries. All lanes of a warp come here; the rows of
// those without `store` are not written.
template <int P, int G, int kAhead>
__device__ __forceinline__ void spmm_row(const SpmmArgs& g, std::int64_t i, std::int64_t q0, std::int64_t q1,
                                         bool store) {
  std::int64_t off[P];  // columns beyond p repeat column 0: read, never stored
#pragma unroll
  for (int c = 0; c < P; ++c) off[c] = c < g.p ? c * g.ldx : 0;
  double acc[P];
#pragma unroll
  for (int c = 0; c < P; ++c) acc[c] = 0.0;
  group_entries<G, kAhead, (P < 8)>(q0, q1, g.ci, g.v, [&](double a, std::int64_t j) {
    const double* xj = g.x + j;
#pragma unroll
    for (int c = 0; c < P; ++c) acc[c] = fma(a, xj[off[c]], acc[c]);
  });
  const GroupCols<P, G> cols;
  cols.sum(acc);
#pragma unroll
  for (int u = 0; u < cols.kCols; ++u) {
    const int c = cols.first + u;
    if (c < g.p && store && cols.writer)
      g.y[i + c * g.ldy] = g.alpha * acc[u] + (g.beta == 0.0 ? 0.0 : g.beta * g.y[i + c * g.ldy]);
  }
}

// entries that a lane of sixteen or more reads ahead: the loads in flight are these times the columns
template <int P>
constexpr int kRowAhead = P >= 4 ? 2 : 4;

template <int P>
__device__ __noinline__ void spmm_long_row(const SpmmArgs& g, std::int64_t i) {
  spmm_row<P, 32, kRowAhead<P>>(g, i, g.rp[i], g.rp[i + 1], true);
}

// the entries of row i < end that its lanes sum: none of a long row
struct SpmmSpan {
  std::int64_t q0 = 0, q1 = 0;
  bool mine = false;
  __device__ __forceinline__ SpmmSpan(const SpmmArgs& g, std::int64_t i, std::int64_t end) {
    if (i >= end) return;
    q0 = g.rp[i];
    q1 = g.rp[i + 1];
    mine = q1 - q0 <= kLongRow;
    if (!mine) q1 = q0;
  }
};

template <int P>
__device__ __noinline__ void spmm_wide_rows(const SpmmArgs& g, std::int64_t row0, std::int64_t end) {
  for (std::int64_t i = row0 + threadIdx.x / 16; row0 < end; row0 += kRowThreads / 16, i += kRowThreads / 16) {
    const SpmmSpan e(g, i, end);
    spmm_row<P, 16, kRowAhead<P>>(g, i, e.q0, e.q1, e.mine);
  }
}

template <int P>
__global__ void __launch_bounds__(kRowThreads, P == 1 ? 5 : (P == 2 ? 4 : 3))
    k_spmm(const __grid_constant__ SpmmArgs g, int chunk) {
  for_rows<P>(g.n, chunk, [&](std::int64_t i, std::int64_t end) { return SpmmSpan(g, i, end); },
              [&](std::int64_t a, std::int64_t b) { return g.rp[b] - g.rp[a]; },
              [&](std::int64_t i, const SpmmSpan& e) { spmm_row<P, 4, 4>(g, i, e.q0, e.q1, e.mine); },
              [&](std::int64_t row0, std::int64_t end) { spmm_wide_rows<P>(g, row0, end); },
              [&](std::int64_t i) { spmm_long_row<P>(g, i); });
}

// Partial Gram sums: CTA b covers rows [b*chunk, (b+1)*chunk); warp w handles columns i = w, w+8,..
// of X; the result part[b][i + c*m] = sum_rows X[row,i] Y[row,c].
__global__ void k_gram_partial(std::int64_t n, int m, int p, const double* x, std::int64_t ldx, const double* y,
                               std::int64_t ldy, std::int64_t chunk, double* part) {
  extern __shared__ double ys[];  // chunk x p
  const std::int64_t r0 = blockIdx.x * chunk;
  const std::int64_t r1 = r0 + chunk < n ? r0 + chunk : n;
  const int rows = static_cast<int>(r1 - r0);
  for (int t = threadIdx.x; t < rows * p; t += blockDim.x) {
    const int rr = t % rows, c = t / rows;
    ys[c * chunk + rr] = y[r0 + rr + c * ldy];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* out = part + static_cast<std::int64_t>(blockIdx.x) * m * p;
  for (int i = warp; i < m; i += nw) {
    double acc[kMaxBlock];
#pragma unroll
    for (int c = 0; c < kMaxBlock; ++c) acc[c] = 0.0;
    const double* xi = x + static_cast<std::int64_t>(i) * ldx + r0;
    for (int rr = lane; rr < rows; rr += 32) {
      const double xv = xi[rr];
#pragma unroll
      for (int c = 0; c < kMaxBlock; ++c)
        if (c < p) acc[c] += xv * ys[c * chunk + rr];
    }
#pragma unroll
    for (int c = 0; c < kMaxBlock; ++c) {
      if (c >= p) break;
      const double s = warp_sum(acc[c]);
      if (lane == 0) out[i + c * m] = s;
    }
  }
}

// Fixed-order sum of the partials: g[t] = sum_b part[b][t]. A block takes 32 consecutive outputs;
// its 8 thread rows stride over the partials (reads coalesced over the outputs) and their 8 sums are
// added in shared memory in row order, so the result does not depend on the launch.
constexpr int kReduceRows = 8;
__global__ void __launch_bounds__(32 * kReduceRows) k_gram_reduce(int nparts, int mp, const double* part, double* g) {
  __shared__ double acc[kReduceRows][33];
  const int tl = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int t = blockIdx.x * 32 + tl;
  double s = 0.0;
  if (t < mp)
    for (int b = row; b < nparts; b += kReduceRows) s += part[static_cast<std::int64_t>(b) * mp + t];
  acc[row][tl] = s;
  __syncthreads();
  if (row == 0 && t < mp) {
    double v = 0.0;
#pragma unroll
    for (int r = 0; r < kReduceRows; ++r) v += acc[r][tl];
    g[t] = v;
  }
}

// Y[:, c0:c0+q] = beta Y + alpha X S[:, c0:c0+q] (X n x m, S m x q in shared memory), 16 columns a pass.
// y (n x q) = alpha X S + beta y: one thread per row, S staged in shared memory QC columns at a time
// (QC = 8 for the Krylov block width, 16 for wider products).
template <int QC>
__global__ void k_gemm_tall(std::int64_t n, int m, int q, const double* x, std::int64_t ldx, const double* s, int lds,
                            double* y, std::int64_t ldy, double alpha, double beta) {
  extern __shared__ double ss[];  // m x QC
  for (int c0 = 0; c0 < q; c0 += QC) {
    const int qc = q - c0 < QC ? q - c0 : QC;
    __syncthreads();
    for (int t = threadIdx.x; t < m * QC; t += blockDim.x) {
      const int i = t % m, c = t / m;
      ss[c * m + i] = c < qc ? s[i + static_cast<std::int64_t>(c0 + c) * lds] : 0.0;
    }
    __syncthreads();
    for (std::int64_t row = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; row < n;
         row += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
      double acc[QC];
#pragma unroll
      for (int c = 0; c < QC; ++c) acc[c] = 0.0;
#pragma unroll 4
      for (int i = 0; i < m; ++i) {
        const double xv = x[row + static_cast<std::int64_t>(i) * ldx];
#pragma unroll
        for (int c = 0; c < QC; ++c) acc[c] += xv * ss[c * m + i];
      }
#pragma unroll
      for (int c = 0; c < QC; ++c) {
        if (c >= qc) break;
        double* yp = y + row + static_cast<std::int64_t>(c0 + c) * ldy;
        *yp = alpha * acc[c] + (beta == 0.0 ? 0.0 : beta * *yp);
      }
    }
  }
}

__global__ void k_diag_scale(std::int64_t n, int p, const double* d, const double* x, std::int64_t ldx, double* y,
                             std::int64_t ldy) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    y[i + c * ldy] = d[i] * x[i + c * ldx];
  }
}

__global__ void k_copy_cols(std::int64_t n, int p, const double* x, std::int64_t ldx, double* y, std::int64_t ldy) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    y[i + c * ldy] = x[i + c * ldx];
  }
}

// Standard normal entries y(i, c) from a counter-based stream: a SplitMix64 hash of (seed, element
// index) gives two uniforms, Box-Muller turns them into one normal deviate. Deterministic in the
// seed and independent of the launch shape.
__device__ __forceinline__ std::uint64_t splitmix64(std::uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void k_fill_normal(std::int64_t n, int p, double* y, std::int64_t ldy, std::uint64_t seed) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::uint64_t h1 = splitmix64(seed ^ (static_cast<std::uint64_t>(t) * 2 + 1));
    const std::uint64_t h2 = splitmix64(h1 ^ 0xD1B54A32D192ED03ull);
    const double u1 = (static_cast<double>(h1 >> 11) + 0.5) * 0x1.0p-53;  // (0, 1)
    const double u2 = static_cast<double>(h2 >> 11) * 0x1.0p-53;          // [0, 1)
    const std::int64_t i = t % n, c = t / n;
    y[i + c * ldy] = sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
  }
}

// Shifted residual of a shift-invert solve, all P columns at once:
//   r(i, c) = (B w_c)(i) - (A y_c)(i),  w = x + sigma y  (B = null: B = I),
//   s(i, c) = (|B| |w_c|)(i) + (|A| |y_c|)(i),
// and the componentwise backward error omega_c = max_i |r(i, c)| / s(i, c) with 0/0 = 0, r/0 = inf and
// inf for a row whose r or s is not finite (the contract of hsolve's shifted_residual,
// include/hsolve/sparse.hpp:157-174). omega must hold zeros at launch; the maximum is taken by an
// integer atomic max on the bit patterns of non-negative doubles (order independent).
struct ResidualArgs {
  std::int64_t n;
  const std::int64_t* arp;
  const std::int32_t* aci;
  const double* av;
  const std::int64_t* brp;
  const std::int32_t* bci;
  const double* bv;
  double sigma;
  const double* x;
  std::int64_t ldx;
  const double* y;
  std::int64_t ldy;
  double* r;
  std::int64_t ldr;
  int p;
};

// Row i by G lanes ([a0, a1), [b0, b1): its entries of A and B): r stored and om raised to the row's backward
// errors where `store` (the lanes' columns, see GroupCols).
template <int P, int G, int kAhead, class Om>
__device__ __forceinline__ void residual_row(const ResidualArgs& g, std::int64_t i, std::int64_t a0, std::int64_t a1,
                                             std::int64_t b0, std::int64_t b1, bool store, Om&& om) {
  const auto xoff = [&](int c) { return c < g.p ? c * g.ldx : 0; };  // columns beyond p repeat column 0
  std::int64_t yoff[P];
#pragma unroll
  for (int c = 0; c < P; ++c) yoff[c] = c < g.p ? c * g.ldy : 0;
  double ra[P], sa[P];
#pragma unroll
  for (int c = 0; c < P; ++c) { ra[c] = 0.0; sa[c] = 0.0; }
  group_entries<G, kAhead, (P < 8)>(a0, a1, g.aci, g.av, [&](double a, std::int64_t j) {
    const double* yj = g.y + j;
#pragma unroll
    for (int c = 0; c < P; ++c) {
      const double t = yj[yoff[c]];
      ra[c] = fma(-a, t, ra[c]);
      sa[c] = fma(fabs(a), fabs(t), sa[c]);
    }
  });
  if (g.brp)
    group_entries<G, kAhead, (P < 8)>(b0, b1, g.bci, g.bv, [&](double b, std::int64_t j) {
#pragma unroll
      for (int c = 0; c < P; ++c) {
        const double w = fma(g.sigma, g.y[j + yoff[c]], g.x[j + xoff(c)]);
        ra[c] = fma(b, w, ra[c]);
        sa[c] = fma(fabs(b), fabs(w), sa[c]);
      }
    });
  const GroupCols<P, G> cols;
  cols.sum(ra);
  cols.sum(sa);
#pragma unroll
  for (int u = 0; u < cols.kCols; ++u) {
    const int c = cols.first + u;
    if (c >= g.p || !store) continue;
    double rs = ra[u], ss = sa[u];
    if (!g.brp) {
      const double w = fma(g.sigma, g.y[i + c * g.ldy], g.x[i + c * g.ldx]);
      rs += w;
      ss += fabs(w);
    }
    if (g.r && cols.writer) g.r[i + c * g.ldr] = rs;
    const double ar = fabs(rs);
    double w;
    if (!isfinite(rs) || !isfinite(ss)) w = CUDART_INF;
    else if (ss > 0.0) w = ar / ss;
    else w = ar > 0.0 ? CUDART_INF : 0.0;
    om(u, w);
  }
}

// (om: the warp's own column maxima in shared memory)
template <int P>
__device__ __noinline__ void residual_long_row(const ResidualArgs& g, std::int64_t i, double* om) {
  const GroupCols<P, 32> cols;
  residual_row<P, 32, kRowAhead<P>>(g, i, g.arp[i], g.arp[i + 1], g.brp ? g.brp[i] : 0, g.brp ? g.brp[i + 1] : 0, true,
                                    [&](int u, double w) {
                                      if (cols.writer) om[cols.first + u] = fmax(om[cols.first + u], w);
                                    });
  __syncwarp();
}

// the entries of row i < end that its lanes sum: none of a long row
struct ResidualSpan {
  std::int64_t a0 = 0, a1 = 0, b0 = 0, b1 = 0;
  bool mine = false;
  __device__ __forceinline__ ResidualSpan(const ResidualArgs& g, std::int64_t i, std::int64_t end) {
    if (i >= end) return;
    a0 = g.arp[i];
    a1 = g.arp[i + 1];
    if (g.brp) {
      b0 = g.brp[i];
      b1 = g.brp[i + 1];
    }
    mine = a1 - a0 <= kLongRow && b1 - b0 <= kLongRow;
    if (!mine) {
      a1 = a0;
      b1 = b0;
    }
  }
};

// the lanes' column maxima to the warp's (part)
template <int P, int G>
__device__ __forceinline__ void keep_maxima(const double (&om)[GroupCols<P, G>::kCols], double* part) {
  const GroupCols<P, G> cols;
#pragma unroll
  for (int u = 0; u < cols.kCols; ++u) {
    double w = om[u];
#pragma unroll
    for (int o = G; o < 32; o <<= 1) w = fmax(w, __shfl_xor_sync(0xffffffffu, w, o));
    if ((threadIdx.x & 31) < G && cols.writer) part[cols.first + u] = fmax(part[cols.first + u], w);
  }
  __syncwarp();
}
template <int P>
__device__ __noinline__ void residual_wide_rows(const ResidualArgs& g, std::int64_t row0, std::int64_t end,
                                                double* part) {
  double om[GroupCols<P, 16>::kCols] = {};
  for (std::int64_t i = row0 + threadIdx.x / 16; row0 < end; row0 += kRowThreads / 16, i += kRowThreads / 16) {
    const ResidualSpan e(g, i, end);
    residual_row<P, 16, kRowAhead<P>>(g, i, e.a0, e.a1, e.b0, e.b1, e.mine,
                                      [&](int u, double w) { om[u] = fmax(om[u], w); });
  }
  keep_maxima<P, 16>(om, part);
}

template <int P>
__global__ void __launch_bounds__(kRowThreads, P == 1 ? 4 : 3)
    k_shifted_residual(const __grid_constant__ ResidualArgs g, int chunk, unsigned long long* omega) {
  __shared__ double part[kRowWarps][P];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane < P) part[warp][lane] = 0.0;
  __syncwarp();
  const auto entries = [&](std::int64_t a, std::int64_t b) {
    const std::int64_t in_a = g.arp[b] - g.arp[a], in_b = g.brp ? g.brp[b] - g.brp[a] : 0;
    return in_a > in_b ? in_a : in_b;
  };
  for_rows<P>(g.n, chunk, [&](std::int64_t i, std::int64_t end) { return ResidualSpan(g, i, end); }, entries,
           [&](std::int64_t i, const ResidualSpan& e) {
             double om[GroupCols<P, 4>::kCols] = {};
             residual_row<P, 4, 4>(g, i, e.a0, e.a1, e.b0, e.b1, e.mine, [&](int u, double w) { om[u] = w; });
             keep_maxima<P, 4>(om, part[warp]);
           },
           [&](std::int64_t row0, std::int64_t end) { residual_wide_rows<P>(g, row0, end, part[warp]); },
           [&](std::int64_t i) { residual_long_row<P>(g, i, part[warp]); });
  if (omega) {
    // one atomic per column and CTA
    __syncthreads();
    if (threadIdx.x < P && static_cast<int>(threadIdx.x) < g.p) {
      double w = 0.0;
      for (int q = 0; q < kRowWarps; ++q) w = fmax(w, part[q][threadIdx.x]);
      // (it only grows: most CTAs find a larger one there)
      const double there = __longlong_as_double(static_cast<long long>(__ldcg(&omega[threadIdx.x])));
      if (w > there) atomic_max_nonneg(&omega[threadIdx.x], w);
    }
  }
}

// z = x + y (p columns)
__global__ void k_add_cols(std::int64_t n, int p, const double* x, std::int64_t ldx, const double* y,
                           std::int64_t ldy, double* z, std::int64_t ldz) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    z[i + c * ldz] = x[i + c * ldx] + y[i + c * ldy];
  }
}

// y(:, c) = x(:, c) for the columns with mask bit c set (p <= 32)
__global__ void k_copy_cols_masked(std::int64_t n, int p, unsigned mask, const double* x, std::int64_t ldx, double* y,
                                   std::int64_t ldy) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    if ((mask >> c) & 1u) y[i + c * ldy] = x[i + c * ldx];
  }
}


// r = a - lam .* b (column c uses lam[c]); y holds r
__global__ void k_residual_cols(std::int64_t n, int p, const double* ax, std::int64_t lda, const double* bx,
                                std::int64_t ldb, const double* lam, double* r, std::int64_t ldr) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    r[i + c * ldr] = ax[i + c * lda] - lam[c] * bx[i + c * ldb];
  }
}

__global__ void k_scale_cols(std::int64_t n, int p, double a, double* y, std::int64_t ldy) {
  const std::int64_t total = n * p;
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < total;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t i = t % n, c = t / n;
    y[i + c * ldy] *= a;
  }
}

// out[j] = sum_i x[i, j] y[i, j] (one CTA per column, fixed-order tree reduction)
__global__ void k_col_dots(std::int64_t n, const double* x, std::int64_t ldx, const double* y, std::int64_t ldy,
                           double* out) {
  __shared__ double red[32];
  const double* xc = x + static_cast<std::int64_t>(blockIdx.x) * ldx;
  const double* yc = y + static_cast<std::int64_t>(blockIdx.x) * ldy;
  double s = 0.0;
  for (std::int64_t i = threadIdx.x; i < n; i += blockDim.x) s += xc[i] * yc[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) out[blockIdx.x] = t;
  }
}

int grid_for(std::int64_t work, int threads) {
  const std::int64_t b = (work + threads - 1) / threads;
  return static_cast<int>(b < 1 ? 1 : (b > 148 * 32 ? 148 * 32 : b));
}

// rows of a CTA's chunk: short while the matrix has too few rows for three CTAs an SM
int row_chunk(std::int64_t n) { return n <= kSmallRows ? kSmallChunk : kChunk; }

}  // namespace

void spmm(const CsrDev& M, const double* x, std::int64_t ldx, double* y, std::int64_t ldy, int p, double alpha,
          double beta, cudaStream_t s) {
  if (p <= 0 || M.n == 0) return;
  const int chunk = row_chunk(M.n), blocks = static_cast<int>((M.n + chunk - 1) / chunk);
  for (int c0 = 0; c0 < p; c0 += 8) {
    const int pc = p - c0 < 8 ? p - c0 : 8;
    const double* xc = x + c0 * ldx;
    const SpmmArgs g{M.n, M.rp, M.ci, M.v, xc, ldx, y + c0 * ldy, ldy, pc, alpha, beta};
    if (pc == 1) { note_launches(1); k_spmm<1><<<blocks, kRowThreads, 0, s>>>(g, chunk); }
    else if (pc <= 2) { note_launches(1); k_spmm<2><<<blocks, kRowThreads, 0, s>>>(g, chunk); }
    else if (pc <= 4) { note_launches(1); k_spmm<4><<<blocks, kRowThreads, 0, s>>>(g, chunk); }
    else { note_launches(1); k_spmm<8><<<blocks, kRowThreads, 0, s>>>(g, chunk); }
  }
}

void gram(std::int64_t n, int m, int p, const double* x, std::int64_t ldx, const double* y, std::int64_t ldy,
          double* g, double* part, std::int64_t part_cap, cudaStream_t s) {
  if (m <= 0 || p <= 0) return;
  // p > kMaxBlock: column chunks of Y
  for (int c0 = 0; c0 < p; c0 += kMaxBlock) {
    const int pc = p - c0 < kMaxBlock ? p - c0 : kMaxBlock;
    std::int64_t chunk = (n + 295) / 296;
    const std::int64_t cap_rows = 6144 / pc;  // Y chunk <= 48 KB of shared memory
    if (chunk > cap_rows) chunk = cap_rows;
    if (chunk < 64) chunk = 64;
    const std::int64_t nparts = (n + chunk - 1) / chunk;
    if (nparts * m * pc > part_cap) return;  // caller sized part_cap with gram_part_size()
    const std::size_t smem = static_cast<std::size_t>(chunk) * pc * sizeof(double);
    note_launches(1);
    k_gram_partial<<<static_cast<int>(nparts), 256, smem, s>>>(n, m, pc, x, ldx, y + c0 * ldy, ldy, chunk, part);
    note_launches(1);
    k_gram_reduce<<<(m * pc + 31) / 32, 32 * kReduceRows, 0, s>>>(static_cast<int>(nparts), m * pc, part,
                                                               g + static_cast<std::int64_t>(c0) * m);
  }
}

void gemm_tall(std::int64_t n, int m, int q, const double* x, std::int64_t ldx, const double* sdev, int lds, double* y,
               std::int64_t ldy, double alpha, double beta, cudaStream_t s) {
  if (q <= 0 || n <= 0) return;
  if (m <= 0) {
    if (beta != 1.0) { note_launches(1); k_scale_cols<<<grid_for(n * q, 256), 256, 0, s>>>(n, q, beta, y, ldy); }
    return;
  }
  static std::once_flag configured;
  std::call_once(configured, [&] {
    cudaFuncSetAttribute(k_gemm_tall<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    cudaFuncSetAttribute(k_gemm_tall<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  note_launches(1);
  if (q <= 8) {
    const std::size_t smem = static_cast<std::size_t>(m) * 8 * sizeof(double);
    k_gemm_tall<8><<<grid_for(n, 256), 256, smem, s>>>(n, m, q, x, ldx, sdev, lds, y, ldy, alpha, beta);
  } else {
    const std::size_t smem = static_cast<std::size_t>(m) * 16 * sizeof(double);
    k_gemm_tall<16><<<grid_for(n, 256), 256, smem, s>>>(n, m, q, x, ldx, sdev, lds, y, ldy, alpha, beta);
  }
}

std::int64_t gram_part_size(std::int64_t n, int m, int p) {
  const int pc = p < kMaxBlock ? p : kMaxBlock;
  std::int64_t chunk = (n + 295) / 296;
  const std::int64_t cap_rows = 6144 / (pc > 0 ? pc : 1);
  if (chunk > cap_rows) chunk = cap_rows;
  if (chunk < 64) chunk = 64;
  return ((n + chunk - 1) / chunk) * static_cast<std::int64_t>(m) * pc;
}

void col_dots(std::int64_t n, int m, const double* x, std::int64_t ldx, const double* y, std::int64_t ldy, double* out,
              cudaStream_t s) {
  if (m <= 0) return;
  note_launches(1);
  k_col_dots<<<m, 512, 0, s>>>(n, x, ldx, y, ldy, out);
}

void scale_cols(std::int64_t n, int p, double a, double* y, std::int64_t ldy, cudaStream_t s) {
  note_launches(1);
  k_scale_cols<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, a, y, ldy);
}

void diag_scale(std::int64_t n, int p, const double* d, const double* x, std::int64_t ldx, double* y,
                std::int64_t ldy, cudaStream_t s) {
  note_launches(1);
  k_diag_scale<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, d, x, ldx, y, ldy);
}

void copy_cols(std::int64_t n, int p, const double* x, std::int64_t ldx, double* y, std::int64_t ldy, cudaStream_t s) {
  note_launches(1);
  k_copy_cols<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, x, ldx, y, ldy);
}

namespace {
// Lanczos recurrence with device-resident coefficients (ab[j]: alpha_j = v_j^T A v_j; ab[kLanczosMax + j]:
// beta_j^2 = ||w_j||^2): w -= alpha_j v_j + beta_{j-1} v_{j-1}
__global__ void k_lanczos_orth(std::int64_t n, double* w, const double* v, const double* vp, const double* ab, int j,
                               int stride) {
  const double alpha = ab[j];
  const double beta = j > 0 ? sqrt(fmax(ab[stride + j - 1], 0.0)) : 0.0;
  for (std::int64_t i = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    w[i] -= alpha * v[i] + (j > 0 ? beta * vp[i] : 0.0);
}
// v = w / sqrt(nrm2[0]) (zero when the norm is zero: the Krylov space is invariant)
__global__ void k_scale_by_norm(std::int64_t n, const double* w, double* v, const double* nrm2) {
  const double q = nrm2[0];
  const double f = q > 0.0 ? 1.0 / sqrt(q) : 0.0;
  for (std::int64_t i = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    v[i] = w[i] * f;
}
}  // namespace

void lanczos_orth(std::int64_t n, double* w, const double* v, const double* vp, const double* ab, int j, int stride,
                  cudaStream_t s) {
  note_launches(1);
  k_lanczos_orth<<<grid_for(n, 256), 256, 0, s>>>(n, w, v, vp, ab, j, stride);
}

void scale_by_norm(std::int64_t n, const double* w, double* v, const double* nrm2, cudaStream_t s) {
  note_launches(1);
  k_scale_by_norm<<<grid_for(n, 256), 256, 0, s>>>(n, w, v, nrm2);
}

void fill_normal(std::int64_t n, int p, double* y, std::int64_t ldy, std::uint64_t seed, cudaStream_t s) {
  note_launches(1);
  k_fill_normal<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, y, ldy, seed);
}

void shifted_residual(const CsrDev& A, const CsrDev* B, double sigma, const double* x, std::int64_t ldx,
                      const double* y, std::int64_t ldy, double* r, std::int64_t ldr, int p, double* omega,
                      cudaStream_t s) {
  if (p <= 0 || A.n == 0) return;
  const int chunk = row_chunk(A.n), blocks = static_cast<int>((A.n + chunk - 1) / chunk);
  if (omega) cuda_check(cudaMemsetAsync(omega, 0, static_cast<std::size_t>(p) * sizeof(double), s), "memset omega");
  for (int c0 = 0; c0 < p; c0 += 8) {
    const int pc = p - c0 < 8 ? p - c0 : 8;
    const double* xc = x + c0 * ldx;
    const double* yc = y + c0 * ldy;
    double* rc = r ? r + c0 * ldr : nullptr;
    unsigned long long* oc = omega ? reinterpret_cast<unsigned long long*>(omega + c0) : nullptr;
    const ResidualArgs g{A.n, A.rp, A.ci, A.v, B ? B->rp : nullptr, B ? B->ci : nullptr, B ? B->v : nullptr, sigma,
                         xc, ldx, yc, ldy, rc, ldr, pc};
    note_launches(1);
    if (pc == 1)
      k_shifted_residual<1><<<blocks, kRowThreads, 0, s>>>(g, chunk, oc);
    else if (pc <= 2)
      k_shifted_residual<2><<<blocks, kRowThreads, 0, s>>>(g, chunk, oc);
    else if (pc <= 4)
      k_shifted_residual<4><<<blocks, kRowThreads, 0, s>>>(g, chunk, oc);
    else
      k_shifted_residual<8><<<blocks, kRowThreads, 0, s>>>(g, chunk, oc);
  }
}

void add_cols(std::int64_t n, int p, const double* x, std::int64_t ldx, const double* y, std::int64_t ldy, double* z,
              std::int64_t ldz, cudaStream_t s) {
  if (p <= 0 || n <= 0) return;
  note_launches(1);
  k_add_cols<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, x, ldx, y, ldy, z, ldz);
}

void copy_cols_masked(std::int64_t n, int p, unsigned mask, const double* x, std::int64_t ldx, double* y,
                      std::int64_t ldy, cudaStream_t s) {
  if (p <= 0 || n <= 0 || mask == 0u) return;
  note_launches(1);
  k_copy_cols_masked<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, mask, x, ldx, y, ldy);
}

void residual_cols(std::int64_t n, int p, const double* ax, std::int64_t lda, const double* bx, std::int64_t ldb,
                   const double* lam, double* r, std::int64_t ldr, cudaStream_t s) {
  note_launches(1);
  k_residual_cols<<<grid_for(n * p, 256), 256, 0, s>>>(n, p, ax, lda, bx, ldb, lam, r, ldr);
}

}  // namespace hsg
