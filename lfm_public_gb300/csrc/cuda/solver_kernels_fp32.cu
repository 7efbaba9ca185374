// Kernels of the FP32-bulk form, one thread per cell, ghost or face: thin
// wrappers over the device functions of solver_fp32.cuh (which the batched
// multi-case kernel shares).
#include "solver_fp32.cuh"
#include "solver_launch.h"

namespace lfm {
namespace dev {

// Threads per block. These kernels wait for loads or (M2AUSM's flux) for
// divisions and square roots; small blocks leave and enter an SM one by one, so
// the last wave is short and a boundary cell's ghost work holds few threads.
// Measured on GB300, us a step at 256, 128 and 64 threads: 768 x 512 cylinder,
// update 58.5, 55.4, 53.8, M1 flux 45.4, 43.8, 67.2; 331 x 217 M2AUSM flux
// 70.7, 54.4, 48.1; 192 x 128 x 48 wake, update 287, 269, 266.
constexpr int kCellThreads = 128;
template <int SCH>
constexpr int kFaceThreads = SCH == kSchemeAUSM ? 64 : 128;

// Primitives of cells, ghosts and halos [first, a.nt): first = 0 where all are
// stale, else nc + ng (halos only: the update keeps the others current).
template <int D>
__global__ void __launch_bounds__(256) k_prep32(const __grid_constant__ Args<float> a, int first) {
    const int t = first + LFM_GLOBAL_ID();
    PdlWait{a.pdl}();
    if (t < a.nt) prep32<D>(a, t);
}

template <int D, bool ELL>
__global__ void __launch_bounds__(kCellThreads) k_grad32(const __grid_constant__ Args<float> a) {
    const int c = LFM_GLOBAL_ID();
    if (c < a.nc) grad32<D, ELL>(a, c, PdlWait{a.pdl});
}

template <int D, bool LES, bool ELL>
__global__ void __launch_bounds__(kCellThreads) k_vis32(const __grid_constant__ Args<float> a) {
    const int c = LFM_GLOBAL_ID();
    if (c < a.nc) vis32<D, LES, ELL>(a, c, PdlWait{a.pdl});
}

template <int D, int SCH, bool LES>
__global__ void __launch_bounds__(kFaceThreads<SCH>) k_flux32(const __grid_constant__ Args<float> a) {
    const int f = LFM_GLOBAL_ID();
    if (f < a.nf) flux32<D, SCH, true, LES, true>(a, f, PdlWait{a.pdl});
}

// Cell-centred form (flux32_cell): one thread per cell over the faces it
// owns, at 768 threads per SM (80 registers; the cell keeps its own 23 values
// across its faces, 3D spills 24 bytes). Off by default: fluxCellOption gives
// both sides' measurements.
template <int D, int SCH>
__global__ void __launch_bounds__(kCellThreads, 768 / kCellThreads) k_flux32_cell(const __grid_constant__ Args<float> a) {
    const int c = LFM_GLOBAL_ID();
    if (c < a.nc) flux32_cell<D, SCH>(a, c, PdlWait{a.pdl});
}

// Warp-interleaved cells: warp j of block b updates the 32 cells of chunk
// j * gridDim.x + b (coalesced within the warp), so a block's warps lie in
// chunks spread over the mesh. The cells with boundary faces come first in
// the solver order and write their ghosts' next state in FP64 (on an FP64 pipe
// that issues about two instructions per clock per SM); interleaved, their
// warps land on different SMs instead of filling the first few blocks, whose
// SMs would otherwise finish last. Beyond kSpreadCells a block keeps consecutive
// cells, which gathers from HBM prefer; the first blocks start first there and
// are done long before the last.
template <int D>
constexpr int kSpreadCells = D == 2 ? 1 << 20 : 1 << 18;

template <int D, bool RES, bool ELL>
__device__ __forceinline__ void update_thread(const Args<float>& a, double Ak, double Bk, int first) {
    const bool spread = a.nc <= kSpreadCells<D>;
    const int c = spread ? (int)(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) << 5) + (int)(threadIdx.x & 31u)
                         : (int)LFM_GLOBAL_ID();
    if (c < a.nc) update32<D, ELL ? kEntriesEll : kEntriesList>(a, c, Ak, Bk, a.step->dt32, first, RES, PdlWait{a.pdl});
}

template <int D, bool RES, bool ELL>
__global__ void __launch_bounds__(kCellThreads) k_update32(const __grid_constant__ Args<float> a, double Ak, double Bk,
                                                            int first) {
    update_thread<D, RES, ELL>(a, Ak, Bk, first);
}

// Fused flux + update (fluxupdate32): one thread per cell, cells mapped as
// in the update kernel that writes ghosts (warp-interleaved chunks).
template <int D, int SCH, bool VIS, bool RES, bool ELL>
__global__ void __launch_bounds__(kCellThreads) k_fluxupdate32(const __grid_constant__ Args<float> a, double Ak, double Bk,
                                                                int first) {
    const int c = (int)(((threadIdx.x >> 5) * gridDim.x + blockIdx.x) << 5) + (int)(threadIdx.x & 31u);
    if (c < a.nc) fluxupdate32<D, SCH, VIS, ELL>(a, c, Ak, Bk, a.step->dt32, first, RES, PdlWait{a.pdl});
}

template <int D, int SCH, bool VIS, bool ELL>
void launch_fluxupdate32_kernel(const Args<float>& a, const StageConfig& s, cudaStream_t st) {
    const unsigned nb = (unsigned)((a.nc + kCellThreads - 1) / kCellThreads);
    if (s.withRes) launch_kernel_pdl(s.pdl && a.pdl, k_fluxupdate32<D, SCH, VIS, true, ELL>, nb, kCellThreads, st, a, s.A, s.B, s.first);
    else launch_kernel_pdl(s.pdl && a.pdl, k_fluxupdate32<D, SCH, VIS, false, ELL>, nb, kCellThreads, st, a, s.A, s.B, s.first);
}

template <int D, int SCH>
void launch_fluxupdate32_scheme(const Args<float>& a, const StageConfig& s, cudaStream_t st) {
    if (SCH != kSchemeAUSM && !s.needVis) {   // no viscous terms, no viscous rows
        if (a.cfEll) launch_fluxupdate32_kernel<D, SCH, false, true>(a, s, st);
        else launch_fluxupdate32_kernel<D, SCH, false, false>(a, s, st);
    } else {
        if (a.cfEll) launch_fluxupdate32_kernel<D, SCH, true, true>(a, s, st);
        else launch_fluxupdate32_kernel<D, SCH, true, false>(a, s, st);
    }
}

template <int D, bool ELL>
void launch_update32(const Args<float>& a, const StageConfig& s, cudaStream_t st) {
    const unsigned nb = (unsigned)((a.nc + kCellThreads - 1) / kCellThreads);   // a 32-cell chunk per warp
    if (s.withRes) launch_kernel_pdl(s.pdl && a.pdl, k_update32<D, true, ELL>, nb, kCellThreads, st, a, s.A, s.B, s.first);
    else launch_kernel_pdl(s.pdl && a.pdl, k_update32<D, false, ELL>, nb, kCellThreads, st, a, s.A, s.B, s.first);
}

template <int D>
__global__ void __launch_bounds__(256) k_set_state32(const __grid_constant__ Args<float> a, const double* q,
                                                     int64_t stride) {
    const int c = LFM_GLOBAL_ID();
    if (c == 0) *a.flag = 0;   // a new state starts with a clear non-finite flag
    if (c < a.nc) set_state32<D>(a, q, stride, c);
}

// Preparation for one residual of a caller's state (k_prep_residual64): the
// primitives of every cell and ghost; q' itself is not kept, the fluxes read the
// primitives alone.
template <int D>
__global__ void __launch_bounds__(128) k_prep_residual32(const __grid_constant__ Args<float> a, const double* q,
                                                         int64_t stride, int vWords, int gradWords, int cellGrad) {
    const int t = LFM_GLOBAL_ID();
    PdlRelease{a.pdl}();
    if (t >= a.nt) return;
    constexpr int NQ = D + 2;
    const int c = t < a.nc ? t : a.gCell[t - a.nc];
    double qp[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) qp[v] = q[(size_t)v * stride + c] - a.qRef[v];
    if (t >= a.nc || cellGrad)
        for (int k = 0; k < gradWords; ++k) a.grad[(size_t)t * gradWords + k] = 0.0f;
    if (t < a.nc) {
        prims32<D>(a, t, qp, a.prim);
        return;
    }
#pragma unroll
    for (int v = 0; v < NQ; ++v) qp[v] += a.qRef[v];
    ghost32<D>(a, t - a.nc, a.gKind[t - a.nc], ghost_in<float, D>(a, qp), a.prim);
    for (int k = 0; k < vWords; ++k) a.V[(size_t)t * vWords + k] = 0.0f;
}

// ---------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------
static inline unsigned nblocks(int n, int b) { return (unsigned)((n + b - 1) / b); }

template <int D>
void launch_fp32(const Args<float>& a, const StageConfig& s, int which, cudaStream_t st) {
    switch (which) {
        case 0: {
            const int first = s.fullPrep ? 0 : a.nc + a.ng;
            // not as a dependent: few blocks of FP64 work, crowded when released early
            if (a.nt > first) launch_kernel_pdl(false, k_prep32<D>, nblocks(a.nt - first, 256), 256, st, a, first);
            break;
        }
        case 1:
            if (s.needGrad && a.cfEll) launch_kernel_pdl(s.pdl && a.pdl, k_grad32<D, true>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            else if (s.needGrad) launch_kernel_pdl(s.pdl && a.pdl, k_grad32<D, false>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            break;
        case 2:
            if (!s.needVis) break;
            if (a.smagC && a.cfEll) launch_kernel_pdl(s.pdl && a.pdl, k_vis32<D, true, true>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            else if (a.smagC) launch_kernel_pdl(s.pdl && a.pdl, k_vis32<D, true, false>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            else if (a.cfEll) launch_kernel_pdl(s.pdl && a.pdl, k_vis32<D, false, true>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            else launch_kernel_pdl(s.pdl && a.pdl, k_vis32<D, false, false>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            break;
        case 3:
            if (s.fluxStaging.stages > 0) {   // staged kernel (configured for this scheme, laminar)
                launch_flux32_staged(a, s, st);
            } else if (a.nf == 0) {
            } else if (a.fOwn && !a.smagC && s.scheme != kSchemeAUSM) {   // cell-centred
                if (s.scheme == kSchemeM1) launch_kernel_pdl(s.pdl && a.pdl, k_flux32_cell<D, kSchemeM1>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
                else launch_kernel_pdl(s.pdl && a.pdl, k_flux32_cell<D, kSchemeM2>, nblocks(a.nc, kCellThreads), kCellThreads, st, a);
            } else if (a.smagC) {   // Smagorinsky LES variants
                if (s.scheme == kSchemeM1) launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeM1, true>, nblocks(a.nf, kFaceThreads<kSchemeM1>), kFaceThreads<kSchemeM1>, st, a);
                else if (s.scheme == kSchemeM2) launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeM2, true>, nblocks(a.nf, kFaceThreads<kSchemeM2>), kFaceThreads<kSchemeM2>, st, a);
                else launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeAUSM, true>, nblocks(a.nf, kFaceThreads<kSchemeAUSM>), kFaceThreads<kSchemeAUSM>, st, a);
            } else {
                if (s.scheme == kSchemeM1) launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeM1, false>, nblocks(a.nf, kFaceThreads<kSchemeM1>), kFaceThreads<kSchemeM1>, st, a);
                else if (s.scheme == kSchemeM2) launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeM2, false>, nblocks(a.nf, kFaceThreads<kSchemeM2>), kFaceThreads<kSchemeM2>, st, a);
                else launch_kernel_pdl(s.pdl && a.pdl, k_flux32<D, kSchemeAUSM, false>, nblocks(a.nf, kFaceThreads<kSchemeAUSM>), kFaceThreads<kSchemeAUSM>, st, a);
            }
            break;
        case 4:
            if (a.cfEll) launch_update32<D, true>(a, s, st);
            else launch_update32<D, false>(a, s, st);
            break;
        default: break;
    }
}

void launch_kernel_fp32(const Args<float>& a, const StageConfig& s, int which, cudaStream_t st) {
    if (a.D == 2)
        launch_fp32<2>(a, s, which, st);
    else
        launch_fp32<3>(a, s, which, st);
}

void launch_fluxupdate32(const Args<float>& a, const StageConfig& s, cudaStream_t st) {
    if (a.D == 2) {
        if (s.scheme == kSchemeM1) launch_fluxupdate32_scheme<2, kSchemeM1>(a, s, st);
        else if (s.scheme == kSchemeM2) launch_fluxupdate32_scheme<2, kSchemeM2>(a, s, st);
        else launch_fluxupdate32_scheme<2, kSchemeAUSM>(a, s, st);
    } else {
        if (s.scheme == kSchemeM1) launch_fluxupdate32_scheme<3, kSchemeM1>(a, s, st);
        else if (s.scheme == kSchemeM2) launch_fluxupdate32_scheme<3, kSchemeM2>(a, s, st);
        else launch_fluxupdate32_scheme<3, kSchemeAUSM>(a, s, st);
    }
}

void launch_set_state32(const Args<float>& a, const double* q, int64_t stride, cudaStream_t st) {
    if (a.D == 2)
        k_set_state32<2><<<nblocks(a.nc, 256), 256, 0, st>>>(a, q, stride);
    else
        k_set_state32<3><<<nblocks(a.nc, 256), 256, 0, st>>>(a, q, stride);
}

void launch_prep_residual32(const Args<float>& a, const double* q, int64_t stride, int vWords, int gradWords, int cellGrad,
                            cudaStream_t st) {
    if (a.D == 2)
        k_prep_residual32<2><<<nblocks(a.nt, 128), 128, 0, st>>>(a, q, stride, vWords, gradWords, cellGrad);
    else
        k_prep_residual32<3><<<nblocks(a.nt, 128), 128, 0, st>>>(a, q, stride, vWords, gradWords, cellGrad);
}

}  // namespace dev
}  // namespace lfm

// ---------------------------------------------------------------------------
// Self-test of the integer-pipe conversions (lfm_selftest_fp_convert).
// ---------------------------------------------------------------------------
namespace {

__global__ void k_convert_selftest(int64_t n, const unsigned* f32, const unsigned long long* f64,
                                   unsigned long long* f64_of_f32, unsigned* f32_of_f64) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    f64_of_f32[i] = (unsigned long long)__double_as_longlong(lfm::dev::f32_to_f64(__uint_as_float(f32[i])));
    f32_of_f64[i] = __float_as_uint(lfm::dev::f64_to_f32(__longlong_as_double((long long)f64[i])));
}

}  // namespace

extern "C" int lfm_selftest_fp_convert(int64_t n, const uint32_t* f32_bits, const uint64_t* f64_bits,
                                       uint64_t* f64_of_f32, uint32_t* f32_of_f64) {
    if (n <= 0 || !f32_bits || !f64_bits || !f64_of_f32 || !f32_of_f64) return -1;
    unsigned *d32 = nullptr, *o32 = nullptr;
    unsigned long long *d64 = nullptr, *o64 = nullptr;
    cudaError_t e = cudaMalloc(&d32, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&o32, (size_t)n * 4);
    if (e == cudaSuccess) e = cudaMalloc(&d64, (size_t)n * 8);
    if (e == cudaSuccess) e = cudaMalloc(&o64, (size_t)n * 8);
    if (e == cudaSuccess) e = cudaMemcpy(d32, f32_bits, (size_t)n * 4, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d64, f64_bits, (size_t)n * 8, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_convert_selftest<<<(unsigned)((n + 255) / 256), 256>>>(n, d32, d64, o64, o32);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(f64_of_f32, o64, (size_t)n * 8, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(f32_of_f64, o32, (size_t)n * 4, cudaMemcpyDeviceToHost);
    cudaFree(d32);
    cudaFree(o32);
    cudaFree(d64);
    cudaFree(o64);
    return e == cudaSuccess ? 0 : -3;
}
