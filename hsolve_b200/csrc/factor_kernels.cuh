// Launchers of the factorization kernels (factor_kernels.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "device.cuh"

namespace hsg {

constexpr int kSmallMax = 64;          // fronts up to this order are factorized in shared memory
constexpr int kNB = 32;                // panel width of the a-posteriori pivoting kernel
constexpr int kTile = 64;              // trailing-update tile (rows = cols)
// Pending pivots whose trailing update is applied at once (blocked step). More of them spread a tile's fixed
// costs and its pass over C over more products, but lengthen the next panel's own updates, which are on
// the chain: n = 291,359 (fronts to 5,861) 53.7 ms a factorization with 128, 52.3 with 192, 51.9 with 224;
// n = 21,660 (fronts to 1,279) 2.61, 2.63, 2.65. With 224 in no front, from an order of 2,048 on and from
// 1,400 on (ms): n = 48,750 (fronts to 1,961) 5.22, 5.22, 5.30; 58,885 (1,966) 5.63, 5.63, 5.68; 75,690
// (2,713) 8.92, 8.93, 8.91; 109,744 (2,965) 12.01, 11.95, 11.93; 291,359 53.7, 52.2, 51.8.
constexpr int kKB = 224;               // most of any front
constexpr int kKBLargeFront = 2048;
#if defined(__CUDACC__)
__host__ __device__
#endif
inline int pending_max(int m) { return m >= kKBLargeFront ? kKB : 128; }
constexpr int kUpdLd = kTile + 4;      // column stride of the staged update operands (conflict-free fragment reads)
constexpr int kUpdChunk = 32;          // pivots of a tile's operands staged at once
constexpr int kUpdStages = 4;          // staged chunks (one computed, the others in flight)
constexpr int kAppDynDoubles = kUpdStages * 2 * kUpdChunk * kUpdLd;  // dynamic shared memory of the panel kernels
constexpr int kRowStage = kNB * kNB + 4 * kNB;   // panel row step: the block's L and the D^-1 coefficients
constexpr int kRowChunk = (kAppDynDoubles - kRowStage) / kNB;  // rows staged at once by the panel row step
constexpr int kAppThreads = 256;
constexpr int kCoopMinFront = 192;     // levels whose largest panel front is at least this use the cooperative kernel
constexpr int kAssembleCols = 8;       // columns per assembly CTA (a warp each)
// per-front scratch of the panel kernels (doubles): control block, two sets (alternate panels) of
// block, original block, labels, pivot types and column maxima, backup of the panel's rows, W = L D
// of the pending pivots (at most pending_max, and at most the front's k)
constexpr int kAppCtrlDoubles = 8;
constexpr int kAppSlotDoubles = 2 * kNB * kNB + kNB / 2 + kNB / 8 + 2 * kNB;
inline std::int64_t app_scratch_doubles(int m, int k) {
  return kAppCtrlDoubles + 2 * kAppSlotDoubles + static_cast<std::int64_t>(m) * (kNB + (k < pending_max(m) ? k : pending_max(m)));
}

void launch_fill(double* x, std::int64_t n, double v, cudaStream_t s);
void launch_scale_rowmax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                         const double* b, const double* ab, const double* d, unsigned long long* r,
                         cudaStream_t s);
void launch_scale_update(std::int64_t n, double* d, unsigned long long* r, cudaStream_t s);
// The front kernels are instantiated for R = double (the FP64 factorization that certifies inertia)
// and R = float (the FP32 operator factorization of the mixed-precision path): panels and
// contribution blocks hold R, the pivot scratch stays in units of doubles.
template <class R>
void launch_scatter(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a,
                    const double* b, const double* ab, const double* d, const std::int64_t* dest,
                    R* panels, FactorCounters* cnt, cudaStream_t s);
// inertia-only counts: the largest scaled entry alone, and the scatter of one level's entries
void launch_amax(std::int64_t nnz, const std::int32_t* row, const std::int32_t* col, const double* a, const double* b,
                 const double* ab, const double* d, FactorCounters* cnt, cudaStream_t s);
template <class R>
void launch_scatter_list(const std::int64_t* idx, std::int64_t count, const std::int32_t* row, const std::int32_t* col,
                         const double* a, const double* b, const double* ab, const double* d,
                         const std::int64_t* dest, R* panels, cudaStream_t s);
template <class R>
void launch_assemble(const int2* items, int nitems, const SnDev* sn, const std::int32_t* cptr, const int2* econt,
                     const std::int32_t* rmap, R* panels, R* cb, cudaStream_t s);
template <class R>
void launch_front_small(int maxm, const std::int32_t* list, int nlist, const SnDev* sn, R* panels, R* cb,
                        signed char* piv, std::int32_t* pidx, const FactorParams& prm, FactorCounters* cnt,
                        std::int32_t* failed, cudaStream_t s);
template <class R>
void launch_front_app(const std::int32_t* list, int nlist, const SnDev* sn, R* panels, R* cb, double* scratch,
                      signed char* piv, std::int32_t* pidx, const FactorParams& prm, FactorCounters* cnt,
                      std::int32_t* failed, cudaStream_t s);

// cooperative launch over the large fronts of a level (see factor_kernels.cu); the co-resident grid
// is the smaller of the two instantiations'
int coop_max_ctas(int device);
template <class R>
cudaError_t launch_front_coop(const std::int32_t* list, const std::int32_t* cta_start, int nfronts, int nctas,
                              const SnDev* sn, R* panels, R* cb, double* scratch, signed char* piv, std::int32_t* pidx,
                              const FactorParams& prm, FactorCounters* cnt, std::int32_t* failed, int* level_done,
                              cudaStream_t s);

}  // namespace hsg
