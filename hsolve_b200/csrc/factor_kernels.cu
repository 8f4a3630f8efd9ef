// Numeric multifrontal LDL^T kernels for sm_100a (FP64).
//
// What replaces MUMPS JOB=2 (hsolve src/factor/mumps_factorization.cpp:300-356; the arithmetic of
// MUMPS dfac_front_LDLT_type1.F / dfac_front_aux.F / dfac_asm.F): symmetric equilibration of
// K = alpha A + beta B, scatter of K into the fronts' panels, assembly of children's contribution
// blocks, and the partial factorization of every front with 1x1 / 2x2 threshold pivots restricted
// to its fully-summed columns. Inertia (neg / zero / pos) is counted from D as pivots are accepted.
//
// Fronts are processed level by level (height in the assembly tree). Small fronts (m <= 64) are
// factorized entirely in shared memory by one CTA with right-looking threshold Bunch-Kaufman.
// Larger fronts use a-posteriori threshold pivoting by panels of NB columns: the diagonal block is
// factorized with Bunch-Kaufman restricted to the block, the rows below are solved against it while
// the largest |l| of every column is recorded, the longest acceptable prefix of pivots is kept
// (|l| <= 1/u), rejected columns are restored from a backup and moved behind the candidates, and
// the trailing matrix receives the rank-q update. Columns no candidate order can pivot are reported
// (failed) so that the host can move them into the parent front and factorize again.
#include <cooperative_groups.h>
#include <cstdint>
#include <mutex>

#include "common.hpp"
#include "device.cuh"
#include "factor_kernels.cuh"

namespace hsg {

namespace {

constexpr double kAlphaBK = 0.6403882032022076;  // (1 + sqrt(17)) / 8

// Determinant of a 2x2 pivot [a b; b c] in the factor's arithmetic R (the pivot test and the
// elimination use the same value).
template <class R>
__device__ __forceinline__ double pivot_det(double a, double b, double c) {
  const R ra = static_cast<R>(a), rb = static_cast<R>(b), rc = static_cast<R>(c);
  return static_cast<double>(ra * rc - rb * rb);
}

// two consecutive shared-memory values in one vector load (16-byte aligned pairs of doubles,
// 8-byte aligned pairs of floats)
__device__ __forceinline__ double2 load_pair(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ float2 load_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }

// cp_async_elem to a shared-memory address, of `size` bytes (sizeof(R), or 0: filled with zero)
template <class R>
__device__ __forceinline__ void cp_async_sized(unsigned dst, const R* src, int size) {
  if constexpr (sizeof(R) == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}

// ------------------------------------------------------------------ scaling and assembly

__global__ void k_fill(double* x, std::int64_t n, double v) {
  for (std::int64_t i = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    x[i] = v;
}

// The kernels that form K = alpha A + beta B read (alpha, beta) = ab[0..1] from device memory, so that a
// captured factorization serves every shift.
// r[i] = max_j |d_i K_ij d_j| over both triangles (atomic max on non-negative doubles)
__global__ void k_scale_rowmax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                               const double* b, const double* ab, const double* d, unsigned long long* r) {
  const double alpha = ab[0], beta = ab[1];
  for (std::int64_t p = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; p < nnz;
       p += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int32_t i = row[p], j = col[p];
    const double v = fabs((alpha * a[p] + beta * b[p]) * d[i] * d[j]);
    atomic_max_nonneg(&r[i], v);
    if (i != j) atomic_max_nonneg(&r[j], v);
  }
}

__global__ void k_scale_update(std::int64_t n, double* d, unsigned long long* r) {
  for (std::int64_t i = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const double v = __longlong_as_double(static_cast<long long>(r[i]));
    if (v > 0.0) d[i] = d[i] / sqrt(v);
    r[i] = 0ull;
  }
}

// panels[dest[p]] = d_i d_j (alpha a_p + beta b_p) (rounded to the factor type R); records max |.|
// for the null-pivot threshold
template <class R>
__global__ void k_scatter(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                          const double* b, const double* ab, const double* d, const std::int64_t* dest,
                          R* panels, FactorCounters* cnt) {
  const double alpha = ab[0], beta = ab[1];
  double mx = 0.0;
  for (std::int64_t p = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; p < nnz;
       p += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int32_t i = row[p], j = col[p];
    const double v = (alpha * a[p] + beta * b[p]) * d[i] * d[j];
    panels[dest[p]] = static_cast<R>(v);
    mx = fmax(mx, fabs(v));
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&cnt->amax_bits, mx);
}

// max |d_i d_j (alpha a_p + beta b_p)| alone (the null-pivot threshold of an inertia-only count,
// whose entries are scattered level by level)
__global__ void k_amax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                       const double* b, const double* ab, const double* d, FactorCounters* cnt) {
  const double alpha = ab[0], beta = ab[1];
  double mx = 0.0;
  for (std::int64_t p = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; p < nnz;
       p += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
    mx = fmax(mx, fabs((alpha * a[p] + beta * b[p]) * d[row[p]] * d[col[p]]));
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&cnt->amax_bits, mx);
}

// panels[dest[p]] = d_i d_j (alpha a_p + beta b_p) for the listed entries p = idx[t] (one level's)
template <class R>
__global__ void k_scatter_list(const std::int64_t* idx, std::int64_t count, const std::int32_t* row,
                               const std::int32_t* col, const double* a, const double* b, const double* ab,
                               const double* d, const std::int64_t* dest, R* panels) {
  const double alpha = ab[0], beta = ab[1];
  for (std::int64_t t = blockIdx.x * static_cast<std::int64_t>(blockDim.x) + threadIdx.x; t < count;
       t += static_cast<std::int64_t>(gridDim.x) * blockDim.x) {
    const std::int64_t p = idx[t];
    panels[dest[p]] = static_cast<R>((alpha * a[p] + beta * b[p]) * d[row[p]] * d[col[p]]);
  }
}

// Assembly of a level's fronts, a warp per column (item: front, first of eight columns): the column of the
// contribution block is zeroed (lower triangle; no kernel reads above the diagonal), then the children's
// columns that fall on it are added in child order (econt[cptr[..]..]: child, column of its block). One
// launch instead of one to zero and one per child rank, each of which read and wrote the parent again;
// an entry's additions come from one warp, in a fixed order. Of 21 + 7 launches at n = 3,021 seven
// are left (0.65 -> 0.58 ms a factorization); n = 109,744: 1.14 ms of zeroing and adding, now 0.93.
template <class R>
__global__ void __launch_bounds__(256) k_assemble(const int2* items, const SnDev* sn, const std::int32_t* cptr,
                                                  const int2* econt, const std::int32_t* rmap, R* panels, R* cb) {
  constexpr int kBatch = 4;
  const int2 it = items[blockIdx.x];
  const SnDev p = sn[it.x];
  const int lane = threadIdx.x & 31, j = it.y + (threadIdx.x >> 5);
  if (j >= p.m) return;
  const std::int32_t pc = p.m - p.k;
  const std::int32_t e0 = cptr[p.cptr_off + j], e1 = cptr[p.cptr_off + j + 1];
  R* dst = panels + p.panel_off + static_cast<std::int64_t>(j) * p.m;
  if (j >= p.k) {
    dst = cb + p.cb_off + static_cast<std::int64_t>(j - p.k) * pc;
    for (std::int32_t i = j - p.k + lane; i < pc; i += 32) dst[i] = R(0);
    dst -= p.k;  // rows of a contribution-block column are numbered from p.k
    __syncwarp();
  }
  for (std::int32_t e = e0; e < e1; ++e) {
    const int2 c = econt[e];
    const SnDev ch = sn[c.x];
    const std::int32_t mc = ch.m - ch.k;
    const R* src = cb + ch.cb_off + static_cast<std::int64_t>(c.y) * mc;
    const std::int32_t* rm = rmap + ch.rmap_off;
    // sources and destinations are read before the stores, which could alias them for the compiler
    for (std::int32_t r0 = c.y + lane; r0 < mc; r0 += 32 * kBatch) {
      R v[kBatch];
      std::int32_t at[kBatch];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const std::int32_t r = r0 + 32 * u;
        at[u] = r < mc ? rm[r] : -1;
        v[u] = r < mc ? src[r] : R(0);
      }
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
        if (at[u] >= 0) v[u] += dst[at[u]];
#pragma unroll
      for (int u = 0; u < kBatch; ++u)
        if (at[u] >= 0) dst[at[u]] = v[u];
    }
    __syncwarp();  // the next child's additions may meet entries that another lane has just written
  }
}

// ------------------------------------------------------------ dense pivoting in shared memory

// Decision of one pivot step (computed by warp 0).
enum : int { kFail = 0, kOneJ = 1, kOneR = 2, kTwoR = 3, kNull = 4 };

struct StepShared {
  int j, lim, prog, force, dec, r, stop;
  int neg, pos, zero, two, forced;
};

// Warp 0: decide the pivot at column j of the lower-stored matrix F (order m, ld ld) with
// candidates [j, nfs). Row maxima cover all rows [j, m).
template <class R>
__device__ void decide_pivot(const R* F, int ld, int m, int nfs, int j, double u, double thr, bool force,
                             StepShared& st) {
  const int lane = threadIdx.x & 31;
  const R* cj = F + static_cast<std::int64_t>(j) * ld;
  double gc = 0.0, best = 0.0;
  int r = -1;
  for (int i = j + 1 + lane; i < m; i += 32) {
    const double v = fabs(cj[i]);
    gc = fmax(gc, v);
    if (i < nfs && v > best) { best = v; r = i; }
  }
  gc = warp_max(gc);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int orr = __shfl_xor_sync(0xffffffffu, r, o);
    if (ob > best || (ob == best && orr >= 0 && (r < 0 || orr < r))) { best = ob; r = orr; }
  }
  const double dcc = fabs(cj[j]);
  int dec = kFail;
  if (thr >= 0.0 && fmax(dcc, gc) <= thr) dec = kNull;
  else if (dcc > 0.0 && dcc >= u * gc) dec = kOneJ;
  else if (force && (r < 0 || best == 0.0 || dcc >= kAlphaBK * gc)) dec = dcc > 0.0 ? kOneJ : kNull;
  if (dec == kFail && r >= 0 && best > 0.0) {
    // maxima of columns j and r excluding rows {j, r}
    const R* cr = F + static_cast<std::int64_t>(r) * ld;
    double gc2 = 0.0, gr2 = 0.0;
    for (int i = j + 1 + lane; i < m; i += 32) {
      if (i != r) gc2 = fmax(gc2, static_cast<double>(fabs(cj[i])));
      if (i < r && i != j) gr2 = fmax(gr2, static_cast<double>(fabs(F[r + static_cast<std::int64_t>(i) * ld])));
      if (i > r) gr2 = fmax(gr2, static_cast<double>(fabs(cr[i])));
    }
    gc2 = warp_max(gc2);
    gr2 = warp_max(gr2);
    const double a = cj[j], b = cj[r], c = cr[r];
    const double det = pivot_det<R>(a, b, c);
    if (force) {
      dec = det != 0.0 ? kTwoR : (dcc > 0.0 ? kOneJ : kNull);
    } else {
      if (det != 0.0) {
        const double ia = fabs(c / det), ib = fabs(b / det), ic = fabs(a / det);
        if (ia * gc2 + ib * gr2 <= 1.0 / u && ib * gc2 + ic * gr2 <= 1.0 / u) dec = kTwoR;
      }
      if (dec == kFail) {
        const double drr = fabs(c);
        if (drr > 0.0 && drr >= u * fmax(fabs(b), gr2)) dec = kOneR;
      }
    }
  }
  if (lane == 0) { st.dec = dec; st.r = r; }
}

// symmetric swap of positions p, q (< m) of the lower-stored matrix; labels follow
template <class R>
__device__ void sym_swap(R* F, int ld, int m, int p, int q, int* lab) {
  if (p == q) return;
  if (p > q) { const int t = p; p = q; q = t; }
  const int n1 = p, n2 = q - p - 1, n3 = m - q - 1;
  for (int t = threadIdx.x; t < n1 + n2 + n3 + 1; t += blockDim.x) {
    R *x, *y;
    if (t < n1) { x = F + p + static_cast<std::int64_t>(t) * ld; y = F + q + static_cast<std::int64_t>(t) * ld; }
    else if (t < n1 + n2) { const int c = p + 1 + (t - n1); x = F + c + static_cast<std::int64_t>(p) * ld; y = F + q + static_cast<std::int64_t>(c) * ld; }
    else if (t < n1 + n2 + n3) { const int i = q + 1 + (t - n1 - n2); x = F + i + static_cast<std::int64_t>(p) * ld; y = F + i + static_cast<std::int64_t>(q) * ld; }
    else { x = F + p + static_cast<std::int64_t>(p) * ld; y = F + q + static_cast<std::int64_t>(q) * ld; }
    const R v = *x; *x = *y; *y = v;
  }
  if (threadIdx.x == 0 && lab) { const int t = lab[p]; lab[p] = lab[q]; lab[q] = t; }
}

// eliminate a 1x1 (or null) pivot at j: column scaled to l, trailing rows/cols [j+1, m) updated
template <class R>
__device__ void elim1(R* F, int ld, int m, int j, bool null_piv, R* tmp) {
  const R d = F[j + static_cast<std::int64_t>(j) * ld];
  R* cj = F + static_cast<std::int64_t>(j) * ld;
  for (int i = j + 1 + threadIdx.x; i < m; i += blockDim.x) {
    const R x = cj[i];
    tmp[i] = null_piv ? R(0) : x;
    cj[i] = null_piv ? R(0) : x / d;
  }
  __syncthreads();
  if (!null_piv) {
    const int w = m - j - 1;
    const R inv = R(1) / d;
    for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
      const int i = j + 1 + t % w, c = j + 1 + t / w;
      if (i >= c) F[i + static_cast<std::int64_t>(c) * ld] -= tmp[i] * tmp[c] * inv;
    }
  }
  __syncthreads();
}

// eliminate the 2x2 pivot (j, j+1)
template <class R>
__device__ void elim2(R* F, int ld, int m, int j, R* tmp0, R* tmp1) {
  const R a = F[j + static_cast<std::int64_t>(j) * ld], b = F[j + 1 + static_cast<std::int64_t>(j) * ld];
  const R c = F[j + 1 + static_cast<std::int64_t>(j + 1) * ld];
  const R det = a * c - b * b;
  const R ia = c / det, ib = -b / det, ic = a / det;
  R* c0 = F + static_cast<std::int64_t>(j) * ld;
  R* c1 = F + static_cast<std::int64_t>(j + 1) * ld;
  for (int i = j + 2 + threadIdx.x; i < m; i += blockDim.x) {
    const R x0 = c0[i], x1 = c1[i];
    tmp0[i] = x0;
    tmp1[i] = x1;
    c0[i] = ia * x0 + ib * x1;
    c1[i] = ib * x0 + ic * x1;
  }
  __syncthreads();
  const int w = m - j - 2;
  for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
    const int i = j + 2 + t % w, cc = j + 2 + t / w;
    if (i >= cc) F[i + static_cast<std::int64_t>(cc) * ld] -= c0[i] * tmp0[cc] + c1[i] * tmp1[cc];
  }
  __syncthreads();
}

// One elimination of threshold Bunch-Kaufman on a lower-stored dense matrix in shared memory, from the
// state in st: candidates [st.j, nfs), rows [0, m). root: pivots may be forced (never fail). Ends after
// a pivot (st.j advanced) or with st.stop = 1 (nothing left, or positions [st.j, nfs) failed); pv[t] in
// {0 null, 1 1x1, 2/3 2x2}; lab follows the swaps. The general step: runs of plain 1x1 pivots go
// through fast_pivots.
template <class R>
__device__ void dense_bk_step(R* F, int ld, int m, int nfs, bool root, double u, double thr, int* lab, signed char* pv,
                              R* tmp0, R* tmp1, StepShared& st) {
  while (true) {
    if (threadIdx.x == 0) {
      st.stop = 0;
      while (st.j >= st.lim) {
        if (st.j < nfs && st.prog) { st.lim = nfs; st.prog = 0; }
        else if (st.j < nfs && root && !st.force) { st.force = 1; st.lim = nfs; }
        else { st.stop = 1; break; }
      }
    }
    __syncthreads();
    if (st.stop) break;
    const int j = st.j;
    if (threadIdx.x < 32) decide_pivot(F, ld, m, nfs, j, u, thr, st.force != 0, st);
    __syncthreads();
    const int dec = st.dec, r = st.r;
    if (dec == kFail) {
      sym_swap(F, ld, m, j, st.lim - 1, lab);
      __syncthreads();
      if (threadIdx.x == 0) st.lim -= 1;
      __syncthreads();
      continue;
    }
    if (dec == kOneR) { sym_swap(F, ld, m, j, r, lab); __syncthreads(); }
    if (dec == kTwoR) { sym_swap(F, ld, m, j + 1, r, lab); __syncthreads(); }
    if (dec == kTwoR) {
      if (threadIdx.x == 0) {
        const R a = F[j + static_cast<std::int64_t>(j) * ld], b = F[j + 1 + static_cast<std::int64_t>(j) * ld];
        const R c = F[j + 1 + static_cast<std::int64_t>(j + 1) * ld];
        const R det = a * c - b * b;
        if (det < 0) { st.neg++; st.pos++; } else if (a + c < 0) st.neg += 2; else st.pos += 2;
        st.two++;
        if (st.force) st.forced++;
        pv[j] = 2; pv[j + 1] = 3;
      }
      elim2(F, ld, m, j, tmp0, tmp1);
      if (threadIdx.x == 0) {
        st.j = j + 2; st.prog = 1; st.force = 0;
        if (st.lim < st.j) st.lim = st.j;
        if (st.lim == j + 1) st.lim = j + 2;
      }
    } else {
      const bool nul = dec == kNull;
      if (threadIdx.x == 0) {
        const double d = F[j + static_cast<std::int64_t>(j) * ld];
        if (nul) { st.zero++; pv[j] = 0; }
        else { if (d < 0) st.neg++; else st.pos++; pv[j] = 1; }
        if (st.force) st.forced++;
      }
      elim1(F, ld, m, j, nul, tmp0);
      if (threadIdx.x == 0) {
        st.j = j + 1; st.prog = 1; st.force = 0;
        if (st.lim < st.j) st.lim = st.j;
      }
    }
    break;
  }
  __syncthreads();
}

constexpr double kRcpMin = 1e-280, kRcpMax = 1e280;  // |d| whose reciprocal is away from the ends of the range

// The bits of |v| that order like the values (the upper word of a double), and a bound of every
// value with those bits.
__device__ __forceinline__ unsigned mag_bits(double v) { return static_cast<unsigned>(__double2hiint(v)) & 0x7fffffffu; }
__device__ __forceinline__ unsigned mag_bits(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ double mag_upper(unsigned b, double) { return __hiloint2double(static_cast<int>(b) + 1, 0); }
__device__ __forceinline__ double mag_upper(unsigned b, float) { return static_cast<double>(__uint_as_float(b)); }
constexpr double kMagSlack = 1.0 + 4e-6;  // mag_upper is at most this factor above the value

// The lower triangle of a matrix of order MAXM in the registers of NT threads, by 8 x 8 blocks dealt to
// the warps in the layout of the FP64 tensor instruction's accumulator (lane: row lane / 4, columns
// 2 (lane % 4), + 1 of the block).
template <int MAXM, int NT, class R>
struct RegTri {
  static constexpr int NW = NT / 32, NB8 = MAXM / 8, NBLK = NB8 * (NB8 + 1) / 2, PER = (NBLK + NW - 1) / NW;
  static constexpr int kNone = 1 << 20;
  R v[PER][2];
  int r0[PER], c0[PER];  // this lane's row and first column of the warp's blocks (kNone: no block)
  __device__ __forceinline__ void place() {
    const int warp = threadIdx.x >> 5;
#pragma unroll
    for (int s = 0; s < PER; ++s) {
      int b = NW - 1 - warp + NW * s, bj = 0;
      while (bj < NB8 && b >= NB8 - bj) { b -= NB8 - bj; ++bj; }
      r0[s] = 8 * (bj + b) + ((threadIdx.x & 31) >> 2);
      c0[s] = bj < NB8 ? 8 * bj + 2 * (threadIdx.x & 3) : kNone;
    }
  }
  // f(value, row, column) for this lane's entries on or below the diagonal
  template <class Fn>
  __device__ __forceinline__ void each(Fn&& f) {
#pragma unroll
    for (int s = 0; s < PER; ++s)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (c0[s] != kNone && r0[s] >= c0[s] + e) f(v[s][e], r0[s], c0[s] + e);
  }
};

// Shared memory of fast_pivots: four columns before their elimination, their L and W = L D (row-major).
template <int MAXM, class R>
struct __align__(16) QuadSmem {
  R col[4 * MAXM + 16], l[4 * MAXM], x[4 * MAXM];
  int npass;
};

// Runs of plain 1x1 pivots, the common case, by the whole CTA: the matrix is in registers (y; entries
// of rows and columns beyond its order are zero), four pivots a step. The owners publish the four
// columns; warp 0 (a row per lane, the 4 x 4 block's own elimination in every lane) eliminates them and
// tests each: 1x1 against the largest entry below, rounded up, so a pivot that passes here passes the
// exact test; every warp applies the pivots up to the first failure to its blocks (FP64: one tensor
// instruction a block). The eliminated columns, L with D on the diagonal, go to F (order ld, shared).
// Ends at st.lim or before the first column whose test fails.
//
// A pivot is a chain of dependent operations (1 / d, scale, update, the next d), not work. A 32 x 32
// block takes 9,500 cycles: 16,900 with every row divided by d, 36,100 with one warp for the whole block.
template <int MAXM, int NT, class R>
__device__ __forceinline__ void fast_pivots(RegTri<MAXM, NT, R>& y, QuadSmem<MAXM, R>& sm, R* F, int ld, double u,
                                            double thr, signed char* pv, StepShared& st) {
  constexpr int NR = MAXM / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t4 = lane & 3, g = lane >> 2;
  int j = st.j;
  const int lim = st.lim;
  const double nul = thr >= 0.0 ? thr * kMagSlack : -1.0;
  int np = 4;
  while (np == 4 && j < lim) {
#pragma unroll
    for (int s = 0; s < y.PER; ++s)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int t = y.c0[s] + e - j;
        if (static_cast<unsigned>(t) < 4u) sm.col[y.r0[s] * 4 + t] = y.v[s][e];
      }
    __syncthreads();
    // (rows above j hold leftovers: they reach only entries above the diagonal or of eliminated columns)
    R x[4][NR], l[4][NR];
    if (warp == 0) {
      R a[4][4];
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int t = 0; t <= s; ++t) a[t][s] = sm.col[(j + s) * 4 + t];
#pragma unroll
      for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t][r] = sm.col[(lane + 32 * r) * 4 + t];
      double gc[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const R inv = R(1) / a[t][t];
        R la[4];
#pragma unroll
        for (int s = t + 1; s < 4; ++s) la[s] = a[t][s] * inv;
#pragma unroll
        for (int r = 0; r < NR; ++r) l[t][r] = x[t][r] * inv;
#pragma unroll
        for (int s2 = t + 1; s2 < 4; ++s2) {
#pragma unroll
          for (int s = s2; s < 4; ++s) a[s2][s] -= la[s] * a[t][s2];
#pragma unroll
          for (int r = 0; r < NR; ++r) x[s2][r] -= l[t][r] * a[t][s2];
        }
        unsigned gb = 0;
#pragma unroll
        for (int r = 0; r < NR; ++r) gb = max(gb, lane + 32 * r > j + t ? mag_bits(x[t][r]) : 0u);
        gc[t] = mag_upper(__reduce_max_sync(0xffffffffu, gb), a[0][0]);
      }
#pragma unroll
      for (int r = 0; r < NR; ++r)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          sm.l[(lane + 32 * r) * 4 + t] = l[t][r];
          sm.x[(lane + 32 * r) * 4 + t] = x[t][r];
        }
      unsigned pass = 0, negs = 0;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const double dcc = fabs(static_cast<double>(a[t][t]));
        const bool ok = (j + t < lim) & (dcc >= kRcpMin) & (dcc <= kRcpMax) & (dcc >= u * gc[t]) &
                        ((dcc > nul) | (gc[t] > nul));
        pass |= ok ? 1u << t : 0u;
        negs |= a[t][t] < R(0) ? 1u << t : 0u;
      }
      const int n = __ffs(~pass) - 1;
      if (lane < n) pv[j + lane] = 1;
      if (lane == 0) {
        sm.npass = n;
        const int neg = __popc(negs & ((1u << n) - 1u));
        st.neg += neg;
        st.pos += n - neg;
      }
    }
    __syncthreads();
    np = sm.npass;
#pragma unroll
    for (int s = 0; s < y.PER; ++s) {
      const int rb = y.r0[s] - g, cb = y.c0[s] - 2 * t4;
      if (y.c0[s] != y.kNone && cb + 7 > j) {
        if constexpr (sizeof(R) == 8) {
          const R a = sm.l[(rb + g) * 4 + t4], b = sm.x[(cb + g) * 4 + t4];
          dmma_m8n8k4(y.v[s][0], y.v[s][1], t4 < np ? -a : R(0), t4 < np ? b : R(0));
        } else {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const R a = sm.l[(rb + g) * 4 + t];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const R b = sm.x[(y.c0[s] + e) * 4 + t];
              y.v[s][e] = t < np ? fma(-a, b, y.v[s][e]) : y.v[s][e];
            }
          }
        }
      }
    }
    if (warp == 0) {
#pragma unroll
      for (int t = 0; t < 4; ++t)
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const int i = lane + 32 * r;
          if (i >= j + t && i < ld && t < np) F[i + (j + t) * ld] = i == j + t ? x[t][r] : l[t][r];
        }
    }
    j += np;
  }
  if (threadIdx.x == 0 && j > st.j) {
    st.j = j;
    st.prog = 1;
  }
  __syncthreads();
}

// Warp maximum of non-negative floats: their bit patterns order like the values, so one integer
// warp reduction replaces a shuffle tree.
__device__ __forceinline__ float warp_maxf(float v) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}

// One warp: one elimination of threshold Bunch-Kaufman on the panel's diagonal block (order w <= 32,
// shared memory, ld kNB, all rows candidates), from the state in st: the general step, for the columns
// where fast_pivots stops. The acceptance rules of dense_bk_step, up to the column maxima's rounding to
// single precision (the panel's rows test every pivot again); the argmax for a 2 x 2 partner is taken only
// where the 1 x 1 test fails; columns are scaled by 1 / d or by the inverse of the 2 x 2 pivot. The update of a step reads the pivot column(s) into
// registers first, so its column read-modify-writes are independent and pipeline. Not inlined: as a
// function of its own it is register-allocated apart from the panel kernels' other phases.
// Warp-synchronous: no block barriers. Ends after a pivot or with st.stop = 1 ([st.j, w) could not be
// pivoted).
template <class R>
__device__ __noinline__ void warp_block_step(R* F, int w, bool root, double u, double thr, int* lab, signed char* pv,
                                             StepShared& st) {
  const int lane = threadIdx.x & 31;
  constexpr int ld = kNB;
  __shared__ R s_c0[kNB], s_c1[kNB];
  int j = st.j, lim = st.lim, prog = st.prog, force = st.force, stop = 0;
  int neg = 0, pos = 0, zero = 0, two = 0, forced = 0;
  while (j < w) {
    if (j >= lim) {
      if (prog) { lim = w; prog = 0; continue; }
      if (root && !force) { force = 1; lim = w; continue; }
      stop = 1;
      break;
    }
    const R* cj = F + j * ld;
    const double xj = lane > j && lane < w ? cj[lane] : 0.0;
    const float gcf = warp_maxf(static_cast<float>(fabs(xj)));
    const double gc = static_cast<double>(gcf);
    const double dj = cj[j];
    const double dcc = fabs(dj);
    int dec = kFail, r = -1;
    if (thr >= 0.0 && fmax(dcc, gc) <= thr) dec = kNull;
    else if (dcc > 0.0 && dcc >= u * gc) dec = kOneJ;
    else {
      // partner candidate: argmax over rows (j, w) of |F(i, j)|
      // (not a number counts as no candidate: the lanes have to agree on the partner)
      float best = lane > j && lane < w && xj == xj ? static_cast<float>(fabs(xj)) : -1.0f;
      int bi = best >= 0.0f ? lane : -1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi >= 0 && (bi < 0 || oi < bi))) { best = ob; bi = oi; }
      }
      r = bi;
      if (force && (r < 0 || best <= 0.0f || dcc >= kAlphaBK * gc)) dec = dcc > 0.0 ? kOneJ : kNull;
      else if (r >= 0 && best > 0.0f) {
        const R* cr = F + r * ld;
        const double xr = lane > j && lane < w && lane != r ? (lane < r ? F[r + lane * ld] : cr[lane]) : 0.0;
        const float gr2f = warp_maxf(static_cast<float>(fabs(xr)));
        const float gc2f = warp_maxf(lane != r ? static_cast<float>(fabs(xj)) : 0.0f);
        const double gr2 = gr2f, gc2 = gc2f;
        const double a = dj, b = cj[r], c = cr[r];
        const double det = pivot_det<R>(a, b, c);
        if (force) dec = det != 0.0 ? kTwoR : (dcc > 0.0 ? kOneJ : kNull);
        else {
          if (det != 0.0) {
            const double ia = fabs(c / det), ib = fabs(b / det), ic = fabs(a / det);
            if (ia * gc2 + ib * gr2 <= 1.0 / u && ib * gc2 + ic * gr2 <= 1.0 / u) dec = kTwoR;
          }
          if (dec == kFail && fabs(c) > 0.0 && fabs(c) >= u * fmax(fabs(b), gr2)) dec = kOneR;
        }
      }
    }
    // swaps (rare)
    int sp = -1, sq = -1;
    if (dec == kFail) { sp = j; sq = lim - 1; }
    else if (dec == kOneR) { sp = j; sq = r; }
    else if (dec == kTwoR) { sp = j + 1; sq = r; }
    if (sp >= 0 && sp != sq) {
      int p = sp < sq ? sp : sq, q = sp < sq ? sq : sp;
      for (int t = lane; t < w + 1; t += 32) {
        R *x = nullptr, *y = nullptr;
        if (t < p) { x = F + p + t * ld; y = F + q + t * ld; }
        else if (t > p && t < q) { x = F + t + p * ld; y = F + q + t * ld; }
        else if (t > q && t < w) { x = F + t + p * ld; y = F + t + q * ld; }
        else if (t == p) { x = F + p + p * ld; y = F + q + q * ld; }
        if (x) { const R v = *x; *x = *y; *y = v; }
      }
      if (lane == 0) { const int tl = lab[p]; lab[p] = lab[q]; lab[q] = tl; }
      __syncwarp();
    }
    if (dec == kFail) { lim -= 1; continue; }
    const int i = lane;
    if (dec == kTwoR) {
      const R a = F[j + j * ld], b = F[j + 1 + j * ld], c = F[j + 1 + (j + 1) * ld];
      const R det = a * c - b * b;
      const R idet = R(1) / det;
      const R ia = c * idet, ib = -b * idet, ic = a * idet;
      const R x0 = (i >= j + 2 && i < w) ? F[i + j * ld] : R(0);
      const R x1 = (i >= j + 2 && i < w) ? F[i + (j + 1) * ld] : R(0);
      const R l0 = ia * x0 + ib * x1, l1 = ib * x0 + ic * x1;
      // the pivot columns go through shared memory into registers first, so that the column
      // updates below are independent of each other (no store can alias a later load)
      s_c0[i] = x0;
      s_c1[i] = x1;
      __syncwarp();
      R y0[kNB], y1[kNB];
#pragma unroll
      for (int c2 = 0; c2 < kNB; ++c2) { y0[c2] = s_c0[c2]; y1[c2] = s_c1[c2]; }
#pragma unroll
      for (int c2 = 0; c2 < kNB; ++c2)
        if (c2 >= j + 2 && i >= c2 && i < w) F[i + c2 * ld] -= l0 * y0[c2] + l1 * y1[c2];
      __syncwarp();
      if (i >= j + 2 && i < w) { F[i + j * ld] = l0; F[i + (j + 1) * ld] = l1; }
      if (lane == 0) { pv[j] = 2; pv[j + 1] = 3; }
      if (det < 0) { neg++; pos++; } else if (a + c < 0) neg += 2; else pos += 2;
      two++;
      if (force) forced++;
      j += 2;
    } else {
      const bool nul = dec == kNull;
      const R d = F[j + j * ld];
      const R inv = nul ? R(0) : R(1) / d;
      const R x = (i > j && i < w) ? F[i + j * ld] : R(0);
      const R xs = x * inv;
      s_c0[i] = x;
      __syncwarp();
      if (!nul) {
        R y[kNB];
#pragma unroll
        for (int c2 = 0; c2 < kNB; ++c2) y[c2] = s_c0[c2];
#pragma unroll
        for (int c2 = 0; c2 < kNB; ++c2)
          if (c2 > j && i >= c2 && i < w) F[i + c2 * ld] -= xs * y[c2];
      }
      __syncwarp();
      if (i > j && i < w) F[i + j * ld] = xs;
      if (lane == 0) pv[j] = nul ? 0 : 1;
      if (nul) zero++;
      else if (d < 0) neg++;
      else pos++;
      if (force) forced++;
      j += 1;
    }
    __syncwarp();
    prog = 1;
    force = 0;
    if (lim < j) lim = j;
    break;
  }
  if (lane == 0) {
    st.neg += neg; st.pos += pos; st.zero += zero; st.two += two; st.forced += forced;
    st.j = j; st.lim = lim; st.prog = prog; st.force = force; st.stop = stop;
  }
  // the lanes return together: the caller's block barrier counts the warp once, whichever lanes arrive
  __syncwarp();
}

__device__ __forceinline__ void bk_begin(StepShared& st, int lim) {
  st.j = 0; st.lim = lim; st.prog = 0; st.force = 0; st.stop = 0;
  st.neg = st.pos = st.zero = st.two = st.forced = 0;
}

// The panel's diagonal block by the whole CTA: y holds its lower triangle (zero from order w on); st was
// begun (and a block barrier passed) before. The factored block is left in F (shared, ld kNB, lower
// triangle).
template <class R>
__device__ void block_bk(RegTri<kNB, kAppThreads, R>& y, R* F, QuadSmem<kNB, R>& qs, int w, bool root, double u,
                         double thr, int* lab, signed char* pv, StepShared& st) {
  while (true) {
    if (!st.force && st.j < st.lim) fast_pivots<kNB, kAppThreads>(y, qs, F, kNB, u, thr, pv, st);
    const int j = st.j;
    if (j >= w) break;
    y.each([&](R& v, int i, int c) { if (c >= j && i < w) F[i + c * kNB] = v; });
    __syncthreads();
    if (threadIdx.x < 32) warp_block_step(F, w, root, u, thr, lab, pv, st);
    __syncthreads();
    if (st.stop || st.j >= w) break;
    y.each([&](R& v, int i, int c) { if (i < w) v = F[i + c * kNB]; });
    __syncthreads();  // every entry is read before F changes again
  }
}

}  // namespace

// ---------------------------------------------------------------------- small fronts (smem)

// A front in registers (fast_pivots); shared memory holds its eliminated columns, and all of it for the
// general pivot steps (2x2 pivots, swaps, null and forced pivots).
template <int MAXM, int NT, class R>
__global__ void __launch_bounds__(NT) k_front_small(const std::int32_t* list, const SnDev* sn, R* panels, R* cb,
                                                    signed char* piv_out, std::int32_t* pidx_out, FactorParams prm,
                                                    FactorCounters* cnt, std::int32_t* failed) {
  extern __shared__ __align__(16) unsigned char small_dyn[];
  R* F = reinterpret_cast<R*>(small_dyn);
  __shared__ R tmp0[MAXM], tmp1[MAXM];
  __shared__ QuadSmem<MAXM, R> qs;
  __shared__ int lab[MAXM];
  __shared__ signed char pv[MAXM];
  __shared__ StepShared st;
  const SnDev d = sn[list[blockIdx.x]];
  const int m = d.m, k = d.k, ld = m;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  R* panel = panels + d.panel_off;
  R* cbb = cb + d.cb_off;
  auto at = [&](int i, int c) -> R& {
    return c < k ? panel[static_cast<std::int64_t>(c) * m + i] : cbb[static_cast<std::int64_t>(c - k) * (m - k) + (i - k)];
  };
  RegTri<MAXM, NT, R> y;
  y.place();
#pragma unroll
  for (int s = 0; s < y.PER; ++s) y.v[s][0] = y.v[s][1] = R(0);
  y.each([&](R& v, int i, int c) { if (i < m) v = at(i, c); });
  for (int t = threadIdx.x; t < m; t += NT) lab[t] = t;
  if (threadIdx.x == 0) bk_begin(st, k);
  __syncthreads();
  const double thr = null_threshold(prm);
  while (true) {
    if (!st.force && st.j < st.lim) fast_pivots<MAXM, NT>(y, qs, F, ld, prm.u, thr, pv, st);
    const int j = st.j;
    if (j >= k) break;
    y.each([&](R& v, int i, int c) { if (c >= j && i < m) F[i + c * ld] = v; });
    __syncthreads();
    dense_bk_step(F, ld, m, k, d.parent < 0, prm.u, thr, lab, pv, tmp0, tmp1, st);
    y.each([&](R& v, int i, int c) { if (i < m) v = F[i + c * ld]; });
    if (st.stop) break;
    __syncthreads();  // every entry is read before F changes again
  }
  const int e = st.j;
  for (int c = warp; c < e; c += NT / 32)
    for (int i = c + lane; i < m; i += 32) panel[static_cast<std::int64_t>(c) * m + i] = F[i + c * ld];
  y.each([&](R& v, int i, int c) { if (c >= e && i < m) at(i, c) = v; });
  for (int t = threadIdx.x; t < k; t += blockDim.x) {
    pidx_out[d.first + t] = lab[t];
    piv_out[d.first + t] = t < e ? pv[t] : static_cast<signed char>(-1);
  }
  if (threadIdx.x == 0) {
    if (st.neg) atomicAdd(&cnt->neg, static_cast<unsigned long long>(st.neg));
    if (st.pos) atomicAdd(&cnt->pos, static_cast<unsigned long long>(st.pos));
    if (st.zero) atomicAdd(&cnt->zero, static_cast<unsigned long long>(st.zero));
    if (st.two) atomicAdd(&cnt->two_by_two, static_cast<unsigned long long>(st.two));
    if (st.forced) atomicAdd(&cnt->forced, static_cast<unsigned long long>(st.forced));
    if (e < k) {
      const unsigned long long at = atomicAdd(&cnt->failed, static_cast<unsigned long long>(k - e));
      for (int t = e; t < k; ++t)
        if (at + (t - e) < static_cast<unsigned long long>(prm.failed_cap)) failed[at + (t - e)] = d.first + lab[t];
    }
  }
}

// ------------------------------------------------------------- larger fronts: a-posteriori pivoting
//
// One front is processed by nr CTAs (nr = 1 for the one-CTA-per-front kernel; nr >= 1 per front in the
// cooperative kernel, where every step is separated by a grid-wide barrier). The pivoting state of a
// front lives in its global scratch (AppCtrl + block + labels + column maxima + backup), written by
// the front's rank-0 CTA and read by all its CTAs after the barrier.

namespace {

template <class R>
struct FrontView {
  R* panel;  // m x k, ld m
  R* cbb;    // (m-k)^2, ld m-k
  int m, k;
  __device__ R* col(int c) const {
    return c < k ? panel + static_cast<std::int64_t>(c) * m : cbb + static_cast<std::int64_t>(c - k) * (m - k) - k;
  }
  __device__ R& at(int i, int c) const { return col(c)[i]; }
};

struct AppCtrl {
  int p, lim, prog, force, stop, w, eb, q;
  int neg, pos, zero, two, forced, finished, fb, bar;  // fb: first pivot whose trailing update is pending;
                                                       // bar: arrivals at the front's barrier
};

// The fields of the control block that a panel step reads, copied by every CTA of the front right
// after a barrier: rank 0 may already change the control block for the next panel while slower
// CTAs still work on this one.
struct StepView {
  int p, w, lim, fb, eb, force, stop;
};

// The scratch of a front is laid out in units of doubles whatever the factor type R; the R-typed
// arrays (B, Borig, backup) occupy the first sizeof(R) / 8 of their double-sized regions.
template <class R>
struct AppFront {
  FrontView<R> f;
  int first;
  bool root;
  AppCtrl* ctrl;
  double* slots;   // two sets of the per-panel arrays below, used by alternate panels
  R* B;            // factored diagonal block, kNB x kNB col-major
  R* Borig;        // the block before factorization
  int* lab;        // block permutation
  signed char* pv; // block pivot types
  unsigned long long* cmax;
  unsigned long long* rmax;
  R* backup;       // kNB columns of m rows
  R* wd;           // W = L D of the pending pivots: column s is pivot fb + s, m rows each
  std::int32_t* plab;
  signed char* ppv;
};

// point the per-panel arrays at set `slot` (0 or 1)
template <class R>
__device__ __forceinline__ void set_slot(AppFront<R>& F, int slot) {
  double* s = F.slots + slot * kAppSlotDoubles;
  F.B = reinterpret_cast<R*>(s);
  s += kNB * kNB;
  F.Borig = reinterpret_cast<R*>(s);
  s += kNB * kNB;
  F.lab = reinterpret_cast<int*>(s);
  s += kNB / 2;
  F.pv = reinterpret_cast<signed char*>(s);
  s += kNB / 8;
  F.cmax = reinterpret_cast<unsigned long long*>(s);
  s += kNB;
  F.rmax = reinterpret_cast<unsigned long long*>(s);
}

__device__ __forceinline__ StepView step_view(const AppCtrl* c) {
  StepView v;
  v.p = __ldcg(&c->p);
  v.w = __ldcg(&c->w);
  v.lim = __ldcg(&c->lim);
  v.fb = __ldcg(&c->fb);
  v.eb = __ldcg(&c->eb);
  v.force = __ldcg(&c->force);
  v.stop = __ldcg(&c->stop);
  return v;
}

template <class R>
__device__ AppFront<R> make_front(const SnDev& d, R* panels, R* cb, double* scratch, signed char* piv_out,
                                  std::int32_t* pidx_out) {
  AppFront<R> F;
  F.f = FrontView<R>{panels + d.panel_off, d.cb_off >= 0 ? cb + d.cb_off : nullptr, d.m, d.k};
  F.first = d.first;
  F.root = d.parent < 0;
  double* s = scratch + d.scratch_off;
  F.ctrl = reinterpret_cast<AppCtrl*>(s);
  s += kAppCtrlDoubles;
  F.slots = s;
  s += 2 * kAppSlotDoubles;
  F.backup = reinterpret_cast<R*>(s);
  s += static_cast<std::int64_t>(d.m) * kNB;
  F.wd = reinterpret_cast<R*>(s);
  F.plab = pidx_out + d.first;
  F.ppv = piv_out + d.first;
  set_slot(F, 0);
  return F;
}

// symmetric swap of fully-summed positions a, b (< k) of the front in global memory
template <class R>
__device__ void front_swap(const FrontView<R>& f, int a, int b, std::int32_t* lab) {
  if (a == b) return;
  if (a > b) { const int t = a; a = b; b = t; }
  const int n1 = a, n2 = b - a - 1, n3 = f.m - b - 1;
  for (int t = threadIdx.x; t < n1 + n2 + n3 + 1; t += blockDim.x) {
    R *x, *y;
    if (t < n1) { x = &f.at(a, t); y = &f.at(b, t); }
    else if (t < n1 + n2) { const int c = a + 1 + (t - n1); x = &f.at(c, a); y = &f.at(b, c); }
    else if (t < n1 + n2 + n3) { const int i = b + 1 + (t - n1 - n2); x = &f.at(i, a); y = &f.at(i, b); }
    else { x = &f.at(a, a); y = &f.at(b, b); }
    const R v = *x; *x = *y; *y = v;
  }
  if (threadIdx.x == 0) { const std::int32_t t = lab[a]; lab[a] = lab[b]; lab[b] = t; }
}

// Init (all ranks split the label work; rank 0 the control block).
template <class R>
__device__ void app_init(AppFront<R>& F, int rank, int nr) {
  const int k = F.f.k;
  for (int t = rank * blockDim.x + threadIdx.x; t < k; t += nr * blockDim.x) { F.plab[t] = t; F.ppv[t] = -1; }
  if (rank == 0 && threadIdx.x == 0) {
    AppCtrl c{};
    c.lim = k;
    *F.ctrl = c;
  }
}

// Rank 0: the factored block at column p (order w, in Bs) to the front and to the panel's arrays.
template <class R>
__device__ void app_publish_block(AppFront<R>& F, int p, int w, const R* Bs, const int* slab, const signed char* spv,
                                  const StepShared& bst) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (__syncthreads_or(threadIdx.x < w && slab[threadIdx.x] != static_cast<int>(threadIdx.x))) {
    // the block's rows were swapped: its pivot labels follow
    int old = 0;
    if (threadIdx.x < w) old = F.plab[p + slab[threadIdx.x]];
    __syncthreads();
    if (threadIdx.x < w) F.plab[p + threadIdx.x] = old;
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const int c2 = warp + 8 * s;
    if (lane >= c2 && lane < w) F.f.at(p + lane, p + c2) = Bs[lane + c2 * kNB];
    F.B[lane + c2 * kNB] = Bs[lane + c2 * kNB];
  }
  for (int t = threadIdx.x; t < kNB; t += blockDim.x) {
    F.lab[t] = slab[t];
    F.pv[t] = spv[t];
    F.cmax[t] = 0ull;
    F.rmax[t] = 0ull;
  }
  if (threadIdx.x == 0) F.ctrl->eb = bst.j;
}

// Rank 0: decide what the next panel is (stop = 1: front finished), and factorize its diagonal block
// with block-restricted threshold Bunch-Kaufman; permute the L rows of the block; publish to scratch.
template <class R>
__device__ void app_control_and_block(AppFront<R>& F, const FactorParams& prm, double thr, R* Bs, QuadSmem<kNB, R>& qs,
                                      int* slab, signed char* spv, StepShared& bst, int* shared_stop,
                                      FactorCounters* cnt, std::int32_t* failed, int* level_done) {
  AppCtrl* c = F.ctrl;
  const int k = F.f.k;
  if (threadIdx.x == 0) {
    int stop = 1;
    if (!c->finished) {
      while (true) {
        if (c->p >= k) { stop = 1; break; }
        if (c->p >= c->lim) {
          if (c->prog) { c->lim = k; c->prog = 0; continue; }
          if (F.root && !c->force) { c->force = 1; c->lim = k; continue; }
          stop = 1;
          break;
        }
        stop = 0;
        c->w = min(kNB, c->lim - c->p);
        break;
      }
    }
    c->stop = stop;
    *shared_stop = stop;
    if (stop && !c->finished) {
      c->finished = 1;
      const int e = c->p;
      if (c->neg) atomicAdd(&cnt->neg, static_cast<unsigned long long>(c->neg));
      if (c->pos) atomicAdd(&cnt->pos, static_cast<unsigned long long>(c->pos));
      if (c->zero) atomicAdd(&cnt->zero, static_cast<unsigned long long>(c->zero));
      if (c->two) atomicAdd(&cnt->two_by_two, static_cast<unsigned long long>(c->two));
      if (c->forced) atomicAdd(&cnt->forced, static_cast<unsigned long long>(c->forced));
      if (e < k) {
        const unsigned long long at = atomicAdd(&cnt->failed, static_cast<unsigned long long>(k - e));
        for (int t = e; t < k; ++t)
          if (at + (t - e) < static_cast<unsigned long long>(prm.failed_cap)) failed[at + (t - e)] = F.first + F.plab[t];
      }
      if (level_done) atomicAdd(level_done, 1);
    }
  }
  __syncthreads();
  if (*shared_stop) return;
  const int p = c->p, w = c->w;
  const bool force = c->force != 0;
  if (force && p + 1 < k) {
    // A root front that made no progress over all its remaining columns: Bunch-Kaufman's choice
    // for column p without threshold, with the partner searched among all remaining fully-summed
    // rows (not only the block's), is brought next to p before the block is factorized.
    __shared__ double s_bv[32], s_gc[32];
    __shared__ int s_bi[32], s_r;
    double bv = -1.0, gc = 0.0;
    int bi = -1;
    for (int i = p + 1 + threadIdx.x; i < F.f.m; i += blockDim.x) {
      const double v = fabs(F.f.at(i, p));
      gc = fmax(gc, v);
      if (i < k && v > bv) { bv = v; bi = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      gc = fmax(gc, __shfl_xor_sync(0xffffffffu, gc, o));
      if (ov > bv || (ov == bv && oi >= 0 && (bi < 0 || oi < bi))) { bv = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { s_bv[threadIdx.x >> 5] = bv; s_bi[threadIdx.x >> 5] = bi; s_gc[threadIdx.x >> 5] = gc; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double b = -1.0, g = 0.0;
      int r = -1;
      for (int q = 0; q < static_cast<int>(blockDim.x >> 5); ++q) {
        g = fmax(g, s_gc[q]);
        if (s_bv[q] > b || (s_bv[q] == b && s_bi[q] >= 0 && (r < 0 || s_bi[q] < r))) { b = s_bv[q]; r = s_bi[q]; }
      }
      const double dcc = fabs(F.f.at(p, p));
      s_r = (r < 0 || b <= 0.0 || dcc >= kAlphaBK * g) ? -1 : r;
    }
    __syncthreads();
    const int r = s_r;
    if (r > p + 1) front_swap(F.f, p + 1, r, F.plab);
    __syncthreads();
  }
  RegTri<kNB, kAppThreads, R> y;
  y.place();
#pragma unroll
  for (int s = 0; s < y.PER; ++s) y.v[s][0] = y.v[s][1] = R(0);
  y.each([&](R& v, int i, int c2) { if (i < w) v = F.f.at(p + i, p + c2); });
  y.each([&](R& v, int i, int c2) { if (i < w) F.Borig[i + c2 * kNB] = v; });
  for (int t = threadIdx.x; t < w; t += blockDim.x) slab[t] = t;
  if (threadIdx.x == 0) bk_begin(bst, w);
  __syncthreads();
  block_bk(y, Bs, qs, w, force, prm.u, thr, slab, spv, bst);
  app_publish_block(F, p, w, Bs, slab, spv, bst);
}

// All ranks: rows [p+w, m) solved against the block (L21 = F21 P L11^-T D^-1), backup, column maxima.
// The rows of a rank go through shared memory in chunks of kRowChunk: the copies of the chunk are
// issued before the block's arrays are read, four lanes run a row's substitution (lane q owns columns
// q, q + 4, ..; a finished value goes to the other three by shuffle, every sum in the order of its
// columns) and write the backup, and a warp per four columns applies D^-1 through per-column
// coefficients (no branch on the pivot type), writes L and W = L D back (coalesced) and reduces the
// column maxima. The phase is a chain of latencies (a rank of the n = 109,744 box's root holds at most
// 20 rows): with 64 CTAs there, at most 45 rows each, one thread a row (496 dependent-load FMAs, 3.3 us) and
// the copies after the block took 7.9 us a panel, this form 5.3; with 148 CTAs it is 5.5.
template <class R>
__device__ void app_rows(AppFront<R>& F, const StepView& v, int rank, int nr, R* Bs, int* slab, signed char* spv,
                         R* Lm) {
  const int p = v.p, w = v.w, eb = v.eb, m = F.f.m;
  // D^-1 as three coefficients per column: l(t) = k0 y(t-1) + k1 y(t) + k2 y(t+1); ksel says
  // which value the column maximum takes: 0 |l|, 1 |y| (null pivot, l = 0), 2 none (t >= eb)
  R* k0 = Lm + kNB * kNB;
  R* k1 = k0 + kNB;
  R* k2 = k1 + kNB;
  int* ksel = reinterpret_cast<int*>(k2 + kNB);
  R* Y = Lm + kRowStage;  // kNB columns of kRowChunk rows
  const int rtotal = m - (p + w);
  const int rchunk = (rtotal + nr - 1) / nr;
  const int rbeg = p + w + rank * rchunk, rend = min(m, rbeg + rchunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warp `warp` copies, writes back and reduces the maxima of columns 4 warp .. 4 warp + 3 (eight warps)
  static_assert(kAppThreads / 32 * 4 == kNB, "a warp takes four columns");
  auto stage = [&](int c0, int nrow) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int t = 4 * warp + c;
      if (t >= w) break;
      const R* col = F.f.panel + static_cast<std::int64_t>(p + t) * m + c0;
      for (int r = lane; r < nrow; r += 32) cp_async_elem(&Y[t * kRowChunk + r], col + r, true);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __syncthreads();  // the staging area's last users are done
  if (rbeg < rend) stage(rbeg, min(kRowChunk, rend - rbeg));
  // the block: Bs as it is; Lm(t, s) = L11(t, s) for s < min(t, eb), zero otherwise (2x2 couplings
  // belong to D)
#pragma unroll
  for (int u = 0; u < kNB * kNB / kAppThreads; ++u) {
    const int e = threadIdx.x + u * kAppThreads, t = e & (kNB - 1), s = e / kNB;
    const R x = __ldcg(&F.B[e]);
    const signed char ty = __ldcg(&F.pv[s]);
    Bs[e] = x;
    Lm[e] = t > s && t < w && s < eb && !(ty == 2 && t == s + 1) ? x : R(0);
  }
  bool moved = false;
  if (threadIdx.x < kNB) {
    const int t = threadIdx.x;
    const signed char ty = __ldcg(&F.pv[t]);
    const int from = __ldcg(&F.lab[t]);
    const R* b = F.B;
    R a0 = R(0), a1 = R(1), a2 = R(0);
    int sel = 2;
    if (t < eb) {
      sel = 0;
      if (ty == 0) { a1 = R(0); sel = 1; }
      else if (ty == 1) a1 = R(1) / __ldcg(&b[t + t * kNB]);
      else {
        const int f0 = ty == 2 ? t : t - 1;
        const R a = __ldcg(&b[f0 + f0 * kNB]), c = __ldcg(&b[f0 + 1 + f0 * kNB]);
        const R cc = __ldcg(&b[f0 + 1 + (f0 + 1) * kNB]);
        const R idet = R(1) / (a * cc - c * c);
        // first of the pair: l = (c y_t - b y_{t+1}) / det; second: l = (a y_t - b y_{t-1}) / det
        if (ty == 2) { a1 = cc * idet; a2 = -c * idet; }
        else { a0 = -c * idet; a1 = a * idet; }
      }
    }
    k0[t] = a0;
    k1[t] = a1;
    k2[t] = a2;
    ksel[t] = sel;
    slab[t] = from;
    spv[t] = ty;
    moved = t < w && from != t;
  }
  // did the block factorization swap any of its rows? (rarely: then the permutation below moves data)
  const bool permuted = __syncthreads_or(moved) != 0;
  // permute the L rows p..p+w-1 of the eliminated columns c < p (a thread owns a column; the
  // columns are split into contiguous chunks over the ranks)
  const int cchunk = (p + nr - 1) / nr;
  const int cend = permuted ? min(p, (rank + 1) * cchunk) : 0;
  for (int cc = rank * cchunk + threadIdx.x; cc < cend; cc += blockDim.x) {
    R x[kNB];
    R* colp = F.f.col(cc) + p;
#pragma unroll
    for (int a = 0; a < kNB; ++a) x[a] = a < w ? colp[slab[a]] : R(0);
#pragma unroll
    for (int a = 0; a < kNB; ++a)
      if (a < w) colp[a] = x[a];
  }
  constexpr int kBatch = 4;
  // column maxima in FP32 (rounding is monotone: the maximum of the rounded values is the rounded
  // maximum), reduced over the warp with one integer max on the bit patterns of the non-negative floats
  float cm[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  for (int c0 = rbeg; c0 < rend; c0 += kRowChunk) {
    const int nrow = min(kRowChunk, rend - c0);
    if (c0 > rbeg) {
      __syncthreads();
      stage(c0, nrow);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // four lanes per row, eight rows per warp; lanes without a row follow along for the shuffles
    const int q = lane & 3;
    for (int r0 = 0; r0 < nrow; r0 += kAppThreads / 4) {
      const int r = r0 + (threadIdx.x >> 2);
      const bool in = r < nrow;
      if (r0 + 8 * warp >= nrow) break;
      R y[kNB / 4];
#pragma unroll
      for (int j = 0; j < kNB / 4; ++j) {
        const int t = q + 4 * j;
        y[j] = in && t < w ? Y[slab[t] * kRowChunk + r] : R(0);
        if (in && t < w) F.backup[static_cast<std::int64_t>(t) * m + c0 + r] = y[j];
      }
#pragma unroll
      for (int s = 0; s < kNB - 1; ++s) {
        const R ys = __shfl_sync(0xffffffffu, y[s / 4], s & 3, 4);
#pragma unroll
        for (int j = s / 4; j < kNB / 4; ++j) y[j] = fma(-ys, Lm[s * kNB + q + 4 * j], y[j]);
      }
#pragma unroll
      for (int j = 0; j < kNB / 4; ++j)
        if (in && q + 4 * j < w) Y[(q + 4 * j) * kRowChunk + r] = y[j];
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int t = 4 * warp + c;
      if (t >= w) break;
      const int sel = ksel[t];
      const R a0 = k0[t], a1 = k1[t], a2 = k2[t];
      const bool first = a0 != R(0), second = a2 != R(0);
      const R* yt = Y + t * kRowChunk;
      R* colp = F.f.panel + static_cast<std::int64_t>(p + t) * m + c0;
      R* wcol = F.wd + static_cast<std::int64_t>(p - v.fb + t) * m + c0;
      // a batch of shared-memory reads before the global stores (which could alias them)
      for (int r0 = lane; r0 < nrow; r0 += 32 * kBatch) {
        R x[kBatch], l[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int r = r0 + 32 * u;
          x[u] = r < nrow ? yt[r] : R(0);
          l[u] = a1 * x[u];
          // (only the pair's own column is read: its neighbours may lie outside the panel)
          if (second && r < nrow) l[u] = fma(a2, yt[r + kRowChunk], l[u]);
          if (first && r < nrow) l[u] = fma(a0, yt[r - kRowChunk], l[u]);
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
          const int r = r0 + 32 * u;
          if (r < nrow) {
            colp[r] = sel == 1 ? R(0) : l[u];
            // the substituted row is W = L D, the update's second operand (zero for a null pivot)
            if (sel != 2) wcol[r] = sel == 1 ? R(0) : x[u];
          }
          if (sel != 2) cm[c] = fmaxf(cm[c], static_cast<float>(fabs(sel == 1 ? x[u] : l[u])));
        }
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float x = warp_maxf(cm[c]);
    const int t = 4 * warp + c;
    // the column maximum of |l| (|y| for a null pivot), rounded up by 1e-7 to stay conservative;
    // the accept step reads the maxima of all ranks
    if (lane == 0 && t < w && x > 0.0f) {
      const double ad = static_cast<double>(x) * (1.0 + 1e-7);
      const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(ad));
      atomicMax(&F.cmax[t], bits);
      atomicMax(&F.rmax[t], bits);
    }
  }
}

// All ranks: the accepted prefix q (identical in every CTA); rank 0 books the inertia. The small
// per-panel arrays are staged in shared memory first (one parallel load) so that warp 0's tests
// below touch no global memory. Bs / spv already hold the panel's block and pivot types (app_rows).
template <class R>
__device__ int app_accept(AppFront<R>& F, const StepView& v, int rank, double thr, double inv_u, int* sq,
                          const R* Bs, const signed char* spv, unsigned long long* scm,
                          unsigned long long* srm) {
  const int eb = v.eb;
  const int p = v.p;
  const bool force = v.force != 0;
  for (int t = threadIdx.x; t < kNB; t += blockDim.x) {
    scm[t] = __ldcg(&F.cmax[t]);
    srm[t] = __ldcg(&F.rmax[t]);
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    // warp 0: lane t tests the pivot that starts at t (the second of a 2x2 pair starts none); the
    // accepted prefix ends at the first failing start. A forced step accepts its first pivot
    // without the threshold; the block's later pivots were chosen from the block alone and pass the
    // a-posteriori tests like any other.
    const int t = threadIdx.x;
    const signed char ty = t < eb ? spv[t] : static_cast<signed char>(3);
    const bool start = t < eb && ty != 3;
    bool fail = false;
    if (start && !(force && t == 0)) {
      const double cm = __longlong_as_double(static_cast<long long>(scm[t]));
      if (ty == 0) fail = __longlong_as_double(static_cast<long long>(srm[t])) > thr;
      else if (ty == 1) fail = cm > inv_u;
      else {
        const double cm2 = t + 1 < kNB ? __longlong_as_double(static_cast<long long>(scm[t + 1])) : 0.0;
        fail = fmax(cm, cm2) > inv_u;
      }
    }
    const unsigned fails = __ballot_sync(0xffffffffu, fail);
    const unsigned over = __ballot_sync(0xffffffffu, start && ty != 0 && ty != 1 && t + 1 >= eb);
    const int q = fails ? __ffs(fails) - 1 : (over ? eb + 1 : eb);
    if (t == 0) *sq = q;
    if (rank == 0) {
      // inertia of the accepted pivots: lane t books the pivot that starts at t
      int neg = 0, pos = 0, zero = 0, two = 0;
      if (start && t < q) {
        if (ty == 0) zero = 1;
        else if (ty == 1) { if (Bs[t + t * kNB] < 0) neg = 1; else pos = 1; }
        else if (ty == 2) {
          const R a = Bs[t + t * kNB], b = Bs[t + 1 + t * kNB], cc = Bs[t + 1 + (t + 1) * kNB];
          const R det = a * cc - b * b;
          if (det < 0) { neg = 1; pos = 1; } else if (a + cc < 0) neg = 2; else pos = 2;
          two = 1;
        }
      }
      neg = __reduce_add_sync(0xffffffffu, neg);
      pos = __reduce_add_sync(0xffffffffu, pos);
      zero = __reduce_add_sync(0xffffffffu, zero);
      two = __reduce_add_sync(0xffffffffu, two);
      if (t == 0) {
        AppCtrl* cw = F.ctrl;
        cw->q = q;
        cw->neg += neg;
        cw->pos += pos;
        cw->zero += zero;
        cw->two += two;
        if (force && q > 0) cw->forced += spv[0] == 2 ? 2 : 1;
      }
    }
  }
  __syncthreads();
  const int q = *sq;
  if (rank == 0)
    for (int t = threadIdx.x; t < q; t += blockDim.x) F.ppv[p + t] = spv[t];
  return q;
}

// All ranks: restore the rejected block columns [q, w) from the backup / original block.
template <class R>
__device__ void app_restore(AppFront<R>& F, const StepView& v, int rank, int nr, int q, const R* Bs,
                            const signed char* spv) {
  const int p = v.p, w = v.w, m = F.f.m;
  const int rtotal = m - (p + w);
  const int rchunk = (rtotal + nr - 1) / nr;
  const int rbeg = p + w + rank * rchunk, rend = min(m, rbeg + rchunk);
  for (int i = rbeg + threadIdx.x; i < rend; i += blockDim.x)
    for (int t = q; t < w; ++t) F.f.at(i, p + t) = F.backup[static_cast<std::int64_t>(t) * m + i];
  if (rank == 0) {
    for (int t = threadIdx.x; t < w * w; t += blockDim.x) {
      const int a = t % w, b = t / w;
      if (b >= q && a >= b) {
        const int la = F.lab[a], lb = F.lab[b];
        F.f.at(p + a, p + b) = la >= lb ? F.Borig[la + lb * kNB] : F.Borig[lb + la * kNB];
      }
      if (a >= q && b < q) {
        // W = L D of the rejected rows, which the row step did not see (a 2x2 pivot's coupling is D)
        const R l = Bs[a + b * kNB];
        const signed char ty = spv[b];
        R x = R(0);
        if (ty == 1) x = l * Bs[b + b * kNB];
        else if (ty == 2) x = fma(Bs[b + b * kNB], l, Bs[b + 1 + b * kNB] * Bs[a + (b + 1) * kNB]);
        else if (ty == 3) x = fma(Bs[b + (b - 1) * kNB], Bs[a + (b - 1) * kNB], Bs[b + b * kNB] * l);
        F.wd[static_cast<std::int64_t>(p - v.fb + b) * m + p + a] = x;
      }
    }
  }
}

// Blocked step. The pivots [fb, p + q) eliminated since the last full update are pending: their
// Schur update has reached only the panels factorized since. After a panel the pending update goes
// either to the whole trailing matrix (a flush: the panel rejected columns, the candidate range
// ends, or more than pending_max(m) pivots would be pending after the next panel) or to the next panel's columns only.
// A column is therefore up to date when its panel is factorized, and every other trailing column
// receives the pending pivots in one rank-(<= pending_max(m)) update instead of one update per panel.
__device__ __forceinline__ bool app_flushes(int m, int p, int w, int q, int lim, int fb) {
  return q < w || p + q >= lim || p + q + kNB - fb > pending_max(m);
}

// All ranks: C(i, c) -= sum_{s in [fb, p+q)} L(i, s) W(c, s), W = L D, over the lower triangle
// c <= i < m of the columns c in [p+q, col_hi): all trailing columns when the step flushes, else the
// next panel's. Rejected columns [p+q, p+w) of a flushing panel already hold the updates of
// [fb, p) (they were part of the panel) and take only those of [p, p+q). W is what the row step's
// substitution leaves before D^-1 (kept in the front's scratch); null pivots have L = 0.
//
// The update runs on the FP64 tensor cores (mma.sync m8n8k4, D = A B + C with A 8 x 4, B 4 x 8) by
// 64 x 64 tiles of C dealt round-robin to the ranks. The tile's rows of L and its columns' rows of
// W come in chunks of kUpdChunk pivots by cp.async (zero-filled outside the front), column-major with
// stride kUpdLd = 4 (mod 16): copies of consecutive rows are contiguous and every fragment read of a
// half-warp hits 32 distinct banks. kUpdStages chunks are in flight across tile boundaries, so the
// next tile arrives while this one is computed (a 64 x 64 x 128 tile is 4.2 us of FP64 tensor work on
// an SM; staged as a whole, scaled by D and only then multiplied, the update phase of a root panel of
// the n = 109,744 box took 20.0 us with 64 CTAs, this form 16.1; with 148 CTAs it is 10.4).
// Warp w (of 8) computes rows 16 (w % 4) .. +16 and columns 32 (w / 4) .. +32
// of the tile as 2 x 4 blocks of 8 x 8. A thread's fragment element (g, t) is row g = lane / 4,
// column t = lane % 4 of A; row t, column g of B; row g, columns 2t, 2t + 1 of C.
// FP32 factors (the operator factorization of the mixed-precision path) keep the same staging and
// the same output ownership per thread, and accumulate with FP32 FMAs (there is no FP32 tensor
// instruction with full FP32 operands; the FP64 refinement of every solve absorbs FP32 rounding).
//
// With look-ahead (la: the panel was accepted whole and the next one follows directly), rank 0 updates
// and factorizes the next panel's diagonal block first (app_next_block): that block is left out here, and
// rank 0 takes the last tiles of the list, fewer than the others by what its block costs (about 9.5 us: two
// tiles of 128 pivots, five of 32; of 224 pivots it is rather one, which gains 0.6 % at n = 291,359).
struct UpdTile {
  int tile, ti, tj;
};

template <class R>
__device__ void app_update(AppFront<R>& F, const StepView& v, int rank, int nr, int q, bool la, R* stage) {
  const int p = v.p, w = v.w, lim = v.lim, fb = v.fb, m = F.f.m;
  const int from = p + q;
  const int K = from - fb;
  const int rows = m - from;
  if (rows <= 0 || K <= 0) return;
  const bool flush = app_flushes(m, p, w, q, lim, fb);
  const int col_hi = flush ? m : min(m, from + min(kNB, lim - from));
  const int rej_hi = flush && q < w ? p + w : 0;  // columns below this take only the pivots >= p
  const int nt = (rows + kTile - 1) / kTile;
  const int nct = (col_hi - from + kTile - 1) / kTile;
  const int ntiles = nct * nt - nct * (nct - 1) / 2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int rbase = (warp & 3) * 16, cbase = (warp >> 2) * 32;
  const int Kpad = (K + 3) & ~3;
  const int nk = (K + kUpdChunk - 1) / kUpdChunk;
  // tiles [tfirst, tend) of this rank by tstep: round-robin, or with look-ahead the last t0 for rank 0
  // and the others over ranks 1..
  const bool split = la && nr > 1;
  const int behind = K > 64 ? 2 : (K > 32 ? 3 : 5);
  const int t0 = split ? max(0, (ntiles + behind) / nr - behind) : 0;
  const int tfirst = split ? (rank == 0 ? ntiles - t0 : rank - 1) : rank;
  const int tend = split && rank > 0 ? ntiles - t0 : ntiles;
  const int tstep = split ? (rank == 0 ? 1 : nr - 1) : nr;
  if (tfirst >= tend) return;
  const int skip = la ? min(kNB, lim - from) + from : from;  // rows (and columns) below: the next block
  // the tile `step` further on, column by column: (ti, tj) with tj <= ti < nt
  auto forward = [&](UpdTile& t, int step) {
    t.tile += step;
    t.ti += step;
    while (t.ti >= nt && t.tj < nct) {
      ++t.tj;
      t.ti += t.tj - nt;
    }
  };
  // a thread copies tile row r, pivots sg, sg + 4, ... of a chunk: pointers that advance by four columns,
  // the validity of the row in the copies' sizes
  const int r = threadIdx.x & (kTile - 1), sg = threadIdx.x >> 6;
  const std::int64_t step4 = 4 * static_cast<std::int64_t>(m);
  const R* lsrc = nullptr;
  const R* wsrc = nullptr;
  int lsize = 0, wsize = 0, smin = 0;
  auto aim = [&](const UpdTile& t) {
    const int i = from + t.ti * kTile + r, c = from + t.tj * kTile + r;
    lsize = i < m ? static_cast<int>(sizeof(R)) : 0;
    wsize = c < col_hi ? static_cast<int>(sizeof(R)) : 0;
    smin = c < rej_hi ? p - fb : 0;
    lsrc = F.f.panel + static_cast<std::int64_t>(fb + sg) * m + (i < m ? i : from);
    wsrc = F.wd + static_cast<std::int64_t>(sg) * m + (c < col_hi ? c : from);
  };
  const unsigned stage0 = static_cast<unsigned>(__cvta_generic_to_shared(stage)) +
                          static_cast<unsigned>((sg * kUpdLd + r) * sizeof(R));
  constexpr unsigned kStageBytes = 2 * kUpdChunk * kUpdLd * sizeof(R), kHalf = kUpdChunk * kUpdLd * sizeof(R);
  auto issue = [&](int kc, int st) {
    unsigned dst = stage0 + st * kStageBytes;
    int s = kc * kUpdChunk + sg;
    const int send = min(Kpad, (kc + 1) * kUpdChunk);
#pragma unroll 8
    for (; s < send; s += 4) {
      const bool in = s < K;  // (a copy of no bytes reads nothing: the pointer is not followed)
      cp_async_sized<R>(dst, lsrc, in ? lsize : 0);
      cp_async_sized<R>(dst + kHalf, wsrc, in && s >= smin ? wsize : 0);
      dst += 4 * kUpdLd * sizeof(R);
      lsrc += step4;
      wsrc += step4;
    }
  };
  UpdTile ft{0, 0, 0}, ct;  // the tile being fetched, and the one computed
  forward(ft, tfirst);
  aim(ft);
  ct = ft;
  int fk = 0, fst = 0, cst = 0;
  auto fetch_next = [&]() {
    if (ft.tile < tend) {
      issue(fk, fst);
      fst = fst + 1 == kUpdStages ? 0 : fst + 1;
      if (++fk == nk) {
        fk = 0;
        forward(ft, tstep);
        if (ft.tile < tend) aim(ft);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __syncthreads();  // the staging area's last users are done
#pragma unroll
  for (int u = 0; u < kUpdStages - 1; ++u) fetch_next();
  while (ct.tile < tend) {
    const int i0 = from + ct.ti * kTile, j0 = from + ct.tj * kTile;
    // warps whose 32 columns all lie at or beyond col_hi (the second half of a panel's tile) or
    // whose 16 rows all lie above their first column or in the next block have nothing to update
    const bool idle = j0 + cbase >= col_hi || i0 + rbase + 15 < max(j0 + cbase, skip);
    // this thread's C entries (rows rbase + 8a + g, columns cbase + 8b + 2 t4 + e)
    R* colp[4][2];
    R cv[2][4][2], acc[2][4][2];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cc = j0 + cbase + 8 * b + 2 * t4 + e;
        colp[b][e] = !idle && cc < col_hi ? F.f.col(cc) : nullptr;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int i = i0 + rbase + 8 * a + g;
          cv[a][b][e] = (colp[b][e] && i < m && cc <= i && i >= skip) ? colp[b][e][i] : R(0);
          acc[a][b][e] = R(0);
        }
      }
    for (int kc = 0; kc < nk; ++kc) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kUpdStages - 2) : "memory");
      __syncthreads();  // the chunk has arrived for every thread, and the stage fetched next is free
      fetch_next();
      const R* Ls = stage + cst * (2 * kUpdChunk * kUpdLd);
      const R* Ws = Ls + kUpdChunk * kUpdLd;
      cst = cst + 1 == kUpdStages ? 0 : cst + 1;
      if (idle) continue;
      if constexpr (sizeof(R) == 8) {
        const int send = min(kUpdChunk, Kpad - kc * kUpdChunk);
#pragma unroll 2
        for (int s0 = 0; s0 < send; s0 += 4) {
          double af[2], bf[4];
#pragma unroll
          for (int a = 0; a < 2; ++a) af[a] = Ls[(s0 + t4) * kUpdLd + rbase + 8 * a + g];
#pragma unroll
          for (int b = 0; b < 4; ++b) bf[b] = Ws[(s0 + t4) * kUpdLd + cbase + 8 * b + g];
#pragma unroll
          for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) dmma_m8n8k4(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
        }
      } else {
        // FP32: the thread's own 2 x 8 outputs by rank-1 steps (two L values, four W pairs per pivot)
        const int send = min(kUpdChunk, K - kc * kUpdChunk);
#pragma unroll 4
        for (int s = 0; s < send; ++s) {
          const R* ls = Ls + s * kUpdLd + rbase + g;
          const R* ws = Ws + s * kUpdLd + cbase + 2 * t4;
          const R l0 = ls[0], l1 = ls[8];
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const auto w2 = load_pair(ws + 8 * b);
            acc[0][b][0] = fma(l0, w2.x, acc[0][b][0]);
            acc[0][b][1] = fma(l0, w2.y, acc[0][b][1]);
            acc[1][b][0] = fma(l1, w2.x, acc[1][b][0]);
            acc[1][b][1] = fma(l1, w2.y, acc[1][b][1]);
          }
        }
      }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cc = j0 + cbase + 8 * b + 2 * t4 + e;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
          const int i = i0 + rbase + 8 * a + g;
          if (colp[b][e] && i < m && cc <= i && i >= skip) colp[b][e][i] = cv[a][b][e] - acc[a][b][e];
        }
      }
    forward(ct, tstep);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The rejected columns np + t (t < r = w - q, np = p + q) change places with the last candidates lim - r + t.
// Where the two ranges are disjoint all ranks do it at once: an entry (i, c) changes places with
// (pi(i), pi(c)), pi the exchange, so the entries of the exchanged rows and columns move in pairs, each pair
// by one thread. (One column after another on rank 0, each waiting for the one before, the seven rejecting
// panels at n = 21,660 cost 0.2 ms of a 2.78 ms factorization, those at n = 109,744 0.3 of 12.05.) Not
// inlined: rarely run, and inside the panel loop it costs the update registers.
__device__ __forceinline__ bool app_swaps_at_once(const StepView& v, int q) {
  const int np = v.p + q, r = v.w - q;
  return r > 0 && np + r < v.lim && np + r <= v.lim - r;
}

template <class R>
__device__ __noinline__ void app_swap_rejected(AppFront<R>& F, const StepView& v, int q, int rank, int nr) {
  const int m = F.f.m, r = v.w - q, na = v.p + q, nb = v.lim - r;
  const int total = r * m;
  for (int idx = rank * blockDim.x + threadIdx.x; idx < total; idx += nr * blockDim.x) {
    const int t = idx % r, x = idx / r, a = na + t, b = nb + t;
    int y = x;  // pi(x); exchanges between two exchanged indices are taken by the smaller t
    if (x >= na && x < na + r) {
      if (x - na < t) continue;
      y = x - na + nb;
    } else if (x >= nb && x < nb + r) {
      if (x - nb <= t) continue;
      y = x - nb + na;
    }
    R* e = &F.f.at(max(a, x), min(a, x));
    R* f = &F.f.at(max(b, y), min(b, y));
    const R u = *e;
    *e = *f;
    *f = u;
  }
  if (rank == 0)
    for (int t = threadIdx.x; t < r; t += blockDim.x) {
      const std::int32_t l = F.plab[na + t];
      F.plab[na + t] = F.plab[nb + t];
      F.plab[nb + t] = l;
    }
}

// Rank 0: advance past the accepted pivots; move rejected columns behind the candidates (moved: done
// already, by all ranks).
template <class R>
__device__ void app_advance(AppFront<R>& F, int q, bool moved) {
  AppCtrl* c = F.ctrl;
  const int p = c->p, w = c->w;
  const int np = p + q, r = w - q;
  const int lim = c->lim;
  const bool flushed = app_flushes(F.f.m, p, w, q, lim, c->fb);
  if (r > 0 && np + r < lim && !moved) {
    for (int t = 0; t < r; ++t) {
      front_swap(F.f, np + t, lim - r + t, F.plab);
      __syncthreads();
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    c->p = np;
    if (flushed) c->fb = np;
    if (q > 0) { c->prog = 1; c->force = 0; }
    if (r > 0) c->lim = np + r < lim ? lim - r : np;
  }
  __syncthreads();
}

template <class R>
struct AppSmem {
  R Bs[kNB * kNB];
  QuadSmem<kNB, R> qs;
  int slab[kNB];
  signed char spv[kNB];
  unsigned long long scm[kNB], srm[kNB];
  StepShared bst;
  int stop, q, ok;
};

// Rank 0, look-ahead: the panel at v was accepted whole and the next one follows directly. Applies the
// pending pivots to the next panel's diagonal block in the registers that its factorization works in (the
// accumulator layout of the tensor instruction), factorizes it and publishes the next step. Done before the
// rank's share of the update: the block is on the panel chain, the update is not. (As the first 64 x 64
// tile of the update, written back and read again, it took 5.8 us of a root panel, and the control block's
// global reads and the swap logic 2 more.)
template <class R>
__device__ void app_next_block(AppFront<R>& F, const StepView& v, int slot, const FactorParams& prm, double thr,
                               AppSmem<R>& sm, R* stage) {
  constexpr int kLd = kNB + 4;  // 4 (mod 16): conflict-free fragment reads
  const int m = F.f.m, fb = v.fb, p = v.p + v.w, w = min(kNB, v.lim - p), K = p - fb;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
  const int Kpad = (K + 7) & ~7;
  set_slot(F, slot);
  R* Ls = stage;
  static_assert(2 * kKB * kLd <= kAppDynDoubles, "the pending pivots' rows fit the staging area");
  R* Ws = stage + kKB * kLd;
  __syncthreads();  // the staging area's last users are done
  for (int s = warp; s < Kpad; s += kAppThreads / 32) {
    const bool in = s < K && lane < w;
    const std::int64_t at = static_cast<std::int64_t>(in ? s : 0) * m + (in ? p + lane : p);
    cp_async_elem(&Ls[s * kLd + lane], F.f.panel + static_cast<std::int64_t>(fb) * m + at, in);
    cp_async_elem(&Ws[s * kLd + lane], F.wd + at, in);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  RegTri<kNB, kAppThreads, R> y;
  y.place();
#pragma unroll
  for (int s = 0; s < y.PER; ++s) y.v[s][0] = y.v[s][1] = R(0);
  y.each([&](R& x, int i, int c) { if (i < w) x = F.f.at(p + i, p + c); });
  for (int t = threadIdx.x; t < w; t += blockDim.x) sm.slab[t] = t;
  if (threadIdx.x == 0) {
    AppCtrl* c = F.ctrl;
    c->p = p;
    c->w = w;
    c->prog = 1;
    c->force = 0;
    c->stop = 0;
    if (app_flushes(m, v.p, v.w, v.w, v.lim, fb)) c->fb = p;
    bk_begin(sm.bst, w);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int s = 0; s < y.PER; ++s) {
    if (y.c0[s] == y.kNone) continue;
    const int rb = y.r0[s] - g, cb = y.c0[s] - 2 * t4;
    R acc[2][2] = {};  // even and odd groups of four pivots: two chains
    if constexpr (sizeof(R) == 8) {
      for (int s0 = 0; s0 < Kpad; s0 += 8)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = (s0 + 4 * h + t4) * kLd;
          dmma_m8n8k4(acc[h][0], acc[h][1], Ls[k + rb + g], Ws[k + cb + g]);
        }
    } else {
      for (int k = 0; k < K; ++k) {
        const R l = Ls[k * kLd + y.r0[s]];
#pragma unroll
        for (int e = 0; e < 2; ++e) acc[0][e] = fma(l, Ws[k * kLd + y.c0[s] + e], acc[0][e]);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) y.v[s][e] -= acc[0][e] + acc[1][e];
  }
  y.each([&](R& x, int i, int c) { if (i < w) F.Borig[i + c * kNB] = x; });
  __syncthreads();
  block_bk(y, sm.Bs, sm.qs, w, false, prm.u, thr, sm.slab, sm.spv, sm.bst);
  app_publish_block(F, p, w, sm.Bs, sm.slab, sm.spv, sm.bst);
}

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier of the nr CTAs of one front (all co-resident: cooperative launch). Arrivals count up in
// the front's control block; a CTA waits until the count reaches the next multiple of nr. The wait
// gives up after kBarrierTimeoutNs (or when another front has given up), books the timeout in the
// counters and returns false, so that a stuck front ends the kernel instead of hanging it.
constexpr unsigned long long kBarrierTimeoutNs = 5ull * 1000 * 1000 * 1000;

__device__ bool front_barrier(int* bar, int nr, unsigned long long* timeouts, int* s_ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    if (nr > 1) {
      // arrival with release semantics (the CTA's writes, ordered before it by the block barrier,
      // become visible to every rank that acquires the count) and acquire for the later reads
      int old;
      asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
      const int target = (old / nr + 1) * nr;
      unsigned long long t0 = 0;
      for (unsigned it = 0;; ++it) {
        int arrived;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(arrived) : "l"(bar) : "memory");
        if (arrived >= target) break;
        if ((it & 63u) == 63u) {
          if (*reinterpret_cast<volatile unsigned long long*>(timeouts) != 0ull) { ok = 0; break; }
          const unsigned long long t = global_ns();
          if (t0 == 0) t0 = t;
          else if (t - t0 > kBarrierTimeoutNs) { atomicAdd(timeouts, 1ull); ok = 0; break; }
          __nanosleep(64);
        }
      }
    }
    *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

// The panel loop of one front, run by its nr CTAs (rank 0 .. nr-1). A step is
//   [control: rank 0 advances past the previous panel and factorizes the next block] barrier
//   rows (all) barrier  accept (all, identical)  [restore (all) barrier]  update (all) barrier
// and when a panel is accepted whole and the next one follows directly (look-ahead), rank 0
// advances and factorizes the next block before its share of the update, so that the control phase
// and its barrier are skipped. Alternate panels use alternate per-panel arrays, so the next
// block's arrays never overlap the ones slower CTAs still read.
template <bool kCoop, class R>
__device__ void app_front(AppFront<R>& F, int rank, int nr, const FactorParams& prm, FactorCounters* cnt,
                          std::int32_t* failed, int* level_done, AppSmem<R>& sm, R* stage) {
  const double thr = null_threshold(prm);
  const double inv_u = 1.0 / prm.u;
  int* bar = &F.ctrl->bar;
  auto sync = [&]() -> bool {
    if (kCoop) return front_barrier(bar, nr, &cnt->sync_timeouts, &sm.ok);
    __syncthreads();
    return true;
  };
  bool la = false;
  int j = 0, qprev = 0;
  StepView vprev{};
  while (true) {
    if (!la) {
      const bool moved = j > 0 && app_swaps_at_once(vprev, qprev);
      if (moved) {
        app_swap_rejected(F, vprev, qprev, rank, nr);
        if (!sync()) break;
      }
      if (rank == 0) {
        if (j > 0) app_advance(F, qprev, moved);
        set_slot(F, j & 1);
        app_control_and_block(F, prm, thr, sm.Bs, sm.qs, sm.slab, sm.spv, sm.bst, &sm.stop, cnt, failed,
                              level_done);
      }
      if (!sync()) break;
    }
    set_slot(F, j & 1);
    const StepView v = step_view(F.ctrl);
    if (v.stop) break;
    app_rows(F, v, rank, nr, sm.Bs, sm.slab, sm.spv, stage);
    if (!sync()) break;
    const int q = app_accept(F, v, rank, thr, inv_u, &sm.q, sm.Bs, sm.spv, sm.scm, sm.srm);
    if (q < v.w) {
      app_restore(F, v, rank, nr, q, sm.Bs, sm.spv);
      if (!sync()) break;
    }
    la = q == v.w && v.p + v.w < v.lim;
    if (la && rank == 0) app_next_block(F, v, (j + 1) & 1, prm, thr, sm, stage);
    app_update(F, v, rank, nr, q, la, stage);
    if (!sync()) break;
    qprev = q;
    vprev = v;
    ++j;
  }
}

}  // namespace

// One CTA per front (nr = 1), fronts listed in `list`.
template <class R>
__global__ void __launch_bounds__(kAppThreads) k_front_app(const std::int32_t* list, const SnDev* sn, R* panels,
                                                           R* cb, double* scratch, signed char* piv_out,
                                                           std::int32_t* pidx_out, FactorParams prm,
                                                           FactorCounters* cnt, std::int32_t* failed) {
  extern __shared__ __align__(16) unsigned char app_dyn[];
  R* stage = reinterpret_cast<R*>(app_dyn);
  __shared__ AppSmem<R> sm;
  const SnDev d = sn[list[blockIdx.x]];
  AppFront<R> F = make_front(d, panels, cb, scratch, piv_out, pidx_out);
  app_init(F, 0, 1);
  __syncthreads();
  app_front<false>(F, 0, 1, prm, cnt, failed, nullptr, sm, stage);
}

// Cooperative: the fronts of a level share the grid; front f owns CTAs [cta_start[f], cta_start[f+1])
// and runs its panel loop with its own barriers, independently of the other fronts.
template <class R>
__global__ void __launch_bounds__(kAppThreads) k_front_coop(const std::int32_t* list, const std::int32_t* cta_start,
                                                            int nfronts, const SnDev* sn, R* panels, R* cb,
                                                            double* scratch, signed char* piv_out,
                                                            std::int32_t* pidx_out, FactorParams prm,
                                                            FactorCounters* cnt, std::int32_t* failed,
                                                            int* level_done) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  extern __shared__ __align__(16) unsigned char app_dyn[];
  R* stage = reinterpret_cast<R*>(app_dyn);
  __shared__ AppSmem<R> sm;
  int fi = 0;
  while (fi + 1 < nfronts && cta_start[fi + 1] <= static_cast<int>(blockIdx.x)) ++fi;
  const int rank = static_cast<int>(blockIdx.x) - cta_start[fi];
  const int nr = cta_start[fi + 1] - cta_start[fi];
  const SnDev d = sn[list[fi]];
  AppFront<R> F = make_front(d, panels, cb, scratch, piv_out, pidx_out);
  app_init(F, rank, nr);
  grid.sync();  // the control blocks (and their barrier counts) are initialized
  app_front<true>(F, rank, nr, prm, cnt, failed, level_done, sm, stage);
}

// ------------------------------------------------------------------------------ launchers

void launch_fill(double* x, std::int64_t n, double v, cudaStream_t s) {
  if (n <= 0) return;
  const int blocks = static_cast<int>(std::min<std::int64_t>((n + 255) / 256, 148 * 16));
  note_launches(1);
  k_fill<<<blocks, 256, 0, s>>>(x, n, v);
}

void launch_scale_rowmax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                         const double* b, const double* ab, const double* d, unsigned long long* r,
                         cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<std::int64_t>((nnz + 255) / 256, 148 * 16));
  note_launches(1);
  k_scale_rowmax<<<blocks, 256, 0, s>>>(nnz, row, col, a, b, ab, d, r);
}

void launch_scale_update(std::int64_t n, double* d, unsigned long long* r, cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<std::int64_t>((n + 255) / 256, 148 * 16));
  note_launches(1);
  k_scale_update<<<blocks, 256, 0, s>>>(n, d, r);
}

template <class R>
void launch_scatter(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                    const double* b, const double* ab, const double* d, const std::int64_t* dest,
                    R* panels, FactorCounters* cnt, cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<std::int64_t>((nnz + 255) / 256, 148 * 16));
  note_launches(1);
  k_scatter<R><<<blocks, 256, 0, s>>>(nnz, row, col, a, b, ab, d, dest, panels, cnt);
}

void launch_amax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a, const double* b,
                 const double* ab, const double* d, FactorCounters* cnt, cudaStream_t s) {
  const int blocks = static_cast<int>(std::min<std::int64_t>((nnz + 255) / 256, 148 * 16));
  note_launches(1);
  k_amax<<<blocks, 256, 0, s>>>(nnz, row, col, a, b, ab, d, cnt);
}

template <class R>
void launch_scatter_list(const std::int64_t* idx, std::int64_t count, const std::int32_t* row, const std::int32_t* col,
                         const double* a, const double* b, const double* ab, const double* d,
                         const std::int64_t* dest, R* panels, cudaStream_t s) {
  if (count <= 0) return;
  const int blocks = static_cast<int>(std::min<std::int64_t>((count + 255) / 256, 148 * 16));
  note_launches(1);
  k_scatter_list<R><<<blocks, 256, 0, s>>>(idx, count, row, col, a, b, ab, d, dest, panels);
}

template <class R>
void launch_assemble(const int2* items, int nitems, const SnDev* sn, const std::int32_t* cptr, const int2* econt,
                     const std::int32_t* rmap, R* panels, R* cb, cudaStream_t s) {
  if (nitems <= 0) return;
  note_launches(1);
  k_assemble<R><<<nitems, 256, 0, s>>>(items, sn, cptr, econt, rmap, panels, cb);
}

template <class R>
void launch_front_small(int maxm, const std::int32_t* list, int nlist, const SnDev* sn, R* panels, R* cb,
                        signed char* piv, std::int32_t* pidx, const FactorParams& prm, FactorCounters* cnt,
                        std::int32_t* failed, cudaStream_t s) {
  if (nlist <= 0) return;
  const std::size_t smem = static_cast<std::size_t>(maxm) * maxm * sizeof(R);
  note_launches(1);
  if (maxm <= 32) k_front_small<32, 128, R><<<nlist, 128, smem, s>>>(list, sn, panels, cb, piv, pidx, prm, cnt, failed);
  else k_front_small<kSmallMax, 256, R><<<nlist, 256, smem, s>>>(list, sn, panels, cb, piv, pidx, prm, cnt, failed);
}

template <class R>
constexpr std::size_t app_dyn_bytes() { return static_cast<std::size_t>(kAppDynDoubles) * sizeof(R); }

template <class R>
void launch_front_app(const std::int32_t* list, int nlist, const SnDev* sn, R* panels, R* cb, double* scratch,
                      signed char* piv, std::int32_t* pidx, const FactorParams& prm, FactorCounters* cnt,
                      std::int32_t* failed, cudaStream_t s) {
  if (nlist <= 0) return;
  constexpr std::size_t smem = app_dyn_bytes<R>();
  static std::once_flag configured;
  std::call_once(configured, [&] {
    cudaFuncSetAttribute(k_front_app<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  });
  note_launches(1);
  k_front_app<R><<<nlist, kAppThreads, smem, s>>>(list, sn, panels, cb, scratch, piv, pidx, prm, cnt, failed);
}

namespace {
template <class R>
int coop_max_ctas_of(int device) {
  constexpr std::size_t smem = app_dyn_bytes<R>();
  cudaFuncSetAttribute(k_front_coop<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  int per_sm = 0, sms = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_front_coop<R>, kAppThreads, smem);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return per_sm * sms;
}
}  // namespace

// co-resident CTAs of the cooperative panel kernel, valid for both factor types (one plan serves a
// factorization object of either precision)
int coop_max_ctas(int device) { return std::min(coop_max_ctas_of<double>(device), coop_max_ctas_of<float>(device)); }

template <class R>
cudaError_t launch_front_coop(const std::int32_t* list, const std::int32_t* cta_start, int nfronts, int nctas,
                              const SnDev* sn, R* panels, R* cb, double* scratch, signed char* piv, std::int32_t* pidx,
                              const FactorParams& prm, FactorCounters* cnt, std::int32_t* failed, int* level_done,
                              cudaStream_t s) {
  if (nfronts <= 0) return cudaSuccess;
  constexpr std::size_t smem = app_dyn_bytes<R>();
  FactorParams p = prm;
  void* args[] = {const_cast<std::int32_t**>(&list), const_cast<std::int32_t**>(&cta_start), &nfronts,
                  const_cast<SnDev**>(&sn), &panels, &cb, &scratch, &piv, &pidx, &p, &cnt, &failed, &level_done};
  note_launches(1);
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(k_front_coop<R>), dim3(nctas), dim3(kAppThreads), args,
                                     smem, s);
}

#define HSG_FACTOR_INSTANTIATE(R)                                                                                     \
  template void launch_scatter<R>(std::int64_t, const std::int32_t*, const std::int32_t*, const double*,             \
                                  const double*, const double*, const double*, const std::int64_t*, R*,              \
                                  FactorCounters*, cudaStream_t);                                                     \
  template void launch_scatter_list<R>(const std::int64_t*, std::int64_t, const std::int32_t*, const std::int32_t*,   \
                                       const double*, const double*, const double*, const double*,                  \
                                       const std::int64_t*, R*, cudaStream_t);                                       \
  template void launch_assemble<R>(const int2*, int, const SnDev*, const std::int32_t*, const int2*,                  \
                                   const std::int32_t*, R*, R*, cudaStream_t);                                        \
  template void launch_front_small<R>(int, const std::int32_t*, int, const SnDev*, R*, R*, signed char*,              \
                                      std::int32_t*, const FactorParams&, FactorCounters*, std::int32_t*,             \
                                      cudaStream_t);                                                                  \
  template void launch_front_app<R>(const std::int32_t*, int, const SnDev*, R*, R*, double*, signed char*,            \
                                    std::int32_t*, const FactorParams&, FactorCounters*, std::int32_t*, cudaStream_t); \
  template cudaError_t launch_front_coop<R>(const std::int32_t*, const std::int32_t*, int, int, const SnDev*, R*, R*, \
                                            double*, signed char*, std::int32_t*, const FactorParams&,                 \
                                            FactorCounters*, std::int32_t*, int*, cudaStream_t);
HSG_FACTOR_INSTANTIATE(double)
HSG_FACTOR_INSTANTIATE(float)
#undef HSG_FACTOR_INSTANTIATE

}  // namespace hsg
