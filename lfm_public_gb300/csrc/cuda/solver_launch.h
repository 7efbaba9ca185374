// Host-side launch interface of the time-step kernels.
#pragma once

#include <cuda_runtime.h>

#include "solver_kernels.cuh"
#include "tile_desc.h"

namespace lfm {
namespace dev {

// Staged FP32-bulk flux kernel (flux_staged_fp32.cu): faces per block (one
// chunk), shared-memory buffers per thread (the staging depth, 0 = the plain
// flux kernel), and the persistent grid and dynamic shared memory set by
// configure_flux_staging.
struct FluxStaging {
    int stages = 0;
    int faces = 128;
    int grid = 0;
    size_t smem = 0;
};

// Whether a case's step launches its kernels as programmatic dependents
// (PdlWait, solver_device.cuh). A dependent's blocks go where room appears
// first; one with fewer blocks than the chip holds at once is crowded onto part
// of the SMs, and FP64 work then waits for their FP64 pipes, while a larger one
// fills every SM anyway and a smaller one finds idle SMs. FP32 kernels wait for
// loads, which crowded SMs serve as well. Where the line lies depends on the blocks
// an SM holds: with the 2D update at 79 registers (6 blocks) for 72 (7) 47k cells
// took 90 us in place of 72. Measured on GB300, us a step without and with (one unit
// of the timer is 2 us):
//   FP64 2D M1   2k cells  44.9  38.8 |  36k  65.5  59.3 | 51.5k 83.9 75.7 | 52.0k 83.9 94.1
//             65.5k cells  96.2 114.6 |  81k 112.6 118.7 | viscous 51.2k 151.5 139.2
//             52.1k 151.5 178.8 | 101k 240.6 253.9 | 135k 295.9 294.8 | 144k 319.4 309.2
//   FP64 2D M2AUSM 15k cells 163.8 153.5 | 24.1k 215.0 206.8 | 24.6k 215.0 249.8 | 33k 251.9 292.2
//              135k cells 749.0 750.5
//   FP64 3D      5k cells 133.1 122.8 | 8.1k 133.1 126.9 | 10k 133.1 147.4 | 61k 323.6 384.9
//              117k cells 560.1 563.1 | 134k 624.6 616.4 | 171k 773.1 747.6
//   FP64 3D M2AUSM 6.0k cells 235.5 227.3 | 6.8k 237.5 307.1
//   FP32 2D      2k cells  36.8  34.7 |  46k  57.2  49.9 | 135k 73.7 67.5
//   FP32 3D      5k cells  61.4  53.2 |  51k  81.9  83.9 | 83k 98.2 99.9 | 134k 118.7 116.7 | 171k 147.4 137.1
// FP32 3D from 50k to 100k cells is even, within the timer's unit, and goes with the
// sizes around it.
inline bool pdl_pays(bool fp64, int D, int scheme, int nc) {
    if (!fp64 || nc >= 131072) return true;
    if (D == 3) return nc <= (scheme == kSchemeAUSM ? 6000 : 8192);
    return nc <= (scheme == kSchemeAUSM ? 24192 : 51200);
}

// Launches k, with `pdl` as a programmatic dependent of the stream's previous
// kernel (PdlWait, solver_device.cuh).
template <class... P, class... V>
inline void launch_kernel_pdl(bool pdl, void (*k)(P...), unsigned grid, unsigned block, cudaStream_t st, V... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k, P(args)...);
}

// What one RK stage runs (src/mesh_solver.cpp:500-672).
struct StageConfig {
    // the kernel follows another of the same chain (or nothing) on its stream:
    // with Args::pdl it is launched as its programmatic dependent
    bool pdl = false;
    int scheme = 0;       // kSchemeM1 / M2 / AUSM
    bool needGrad = false;
    bool needVis = true;
    double A = 0, B = 1;  // low-storage RK coefficients of this stage
    int first = 0;        // stage 0: dq starts from zero (prepare_for_timestep)
    int withRes = 0;      // record the stage-0 residual
    // FP32-bulk: the update writes the next stage's cell primitives, so the
    // preparation pass covers the ghosts only unless the cell primitives are
    // stale (a new state was set).
    bool fullPrep = true;
    // FP32-bulk flux: the staged kernel when stages > 0
    FluxStaging fluxStaging;
};

template <typename T>
void launch_stage(const Args<T>& a, const StageConfig& s, cudaStream_t st);
template <typename T>
void launch_kernel(const Args<T>& a, const StageConfig& s, int which, cudaStream_t st);
template <>
void launch_stage<float>(const Args<float>& a, const StageConfig& s, cudaStream_t st);
template <>
void launch_kernel<float>(const Args<float>& a, const StageConfig& s, int which, cudaStream_t st);
// FP32-bulk kernels (perturbation form).
void launch_kernel_fp32(const Args<float>& a, const StageConfig& s, int which, cudaStream_t st);
// FP32-bulk fused flux + update of every cell (laminar): the face rhs
// evaluated by the cells themselves; the next stage's primitives go to a.primW, which must not be a.prim.
void launch_fluxupdate32(const Args<float>& a, const StageConfig& s, cudaStream_t st);
// Staged flux kernel: for M1 / M2 without the LES terms; configure sets the
// kernel's shared-memory limit (outside graph capture) and fs.grid, fs.smem.
bool flux_staging_supported(int scheme, bool les);
cudaError_t configure_flux_staging(int D, int scheme, int nf, FluxStaging& fs);
void launch_flux32_staged(const Args<float>& a, const StageConfig& s, cudaStream_t st);
// Preparation for one residual of the state q ([nq][stride] on the device):
// primitives (FP64: the stored rows too) of the cells and ghosts, the ghosts' V
// rows (vRows / vWords per cell) and gradients (cellGrad: the cells' too) cleared.
void launch_prep_residual64(const Args<double>& a, const double* q, int64_t stride, int vRows, int gradRows, int cellGrad,
                            cudaStream_t st);
void launch_prep_residual32(const Args<float>& a, const double* q, int64_t stride, int vWords, int gradWords, int cellGrad,
                            cudaStream_t st);
// The address at which kernels read and write the page-locked host memory
// [p, p + bytes), or null for other memory, for a p that is not aligned for
// doubles and for a range that is not page-locked to its end: the copy calls serve
// those. A state in page-locked memory is read and written by the
// kernels that convert it: the C2C link moves it at the copy engines' rate, and
// the stream does not change between engine and kernels, which costs a batch
// of eight cases about 30 us a case.
double* kernel_address(const double* p, size_t bytes);
// A new FP64 state from an absolute one (or from the stored rows, stride nt).
void launch_set_state64(const Args<double>& a, const double* q, int64_t stride, cudaStream_t st);
// A new FP32-bulk state from an absolute one: q', the cells' primitives and
// their boundary ghosts' primitives.
void launch_set_state32(const Args<float>& a, const double* q, int64_t stride, cudaStream_t st);

// Rows of the per-cell primitive array: FP64 keeps 1/rho, u[D], R psi, c;
// the FP32 perturbation form keeps rho', m'[D], u'[D], R psi', c.
template <typename T>
constexpr int primRows(int D) {
    return sizeof(T) == sizeof(double) ? D + 3 : 2 * D + 3;
}
// Values per cell of the viscous array and of M2AUSM's gradients (FP64: rows of
// nt; FP32-bulk: whole 16-byte parts per cell).
template <typename T>
constexpr size_t visWords(int D, bool les) {
    return sizeof(T) == sizeof(double) ? (size_t)(D * D + 2 * D + (les ? D * D : 0)) : (size_t)visStride32(D, les);
}
template <typename T>
constexpr size_t gradWords(int D) {
    return sizeof(T) == sizeof(double) ? (size_t)(2 * D + D * D) : (size_t)gradStride32(D);
}
// Offset added to the stored state before use (the FP32-bulk form stores
// q - q_ref; zero for the FP64 path).
struct QOffset {
    double v[5];
};
// FP64 path, at set-up: the face, entry and cell constants of a (wN, cfSoN,
// cellSoW and, where allocated, mS .. kl) from its geometry.
void launch_fp64_constants(const Args<double>& a, cudaStream_t st);
// mode 0: max CFL, mode 1: min dt; *arrived 0 before and after, out may be
// page-locked host memory
void launch_cfl(int D, const double* q, QOffset qo, int nt, int nc, const double* volInv, const int* sOff, const double* cellS,
                double dt, int mode, double maxCo, double* partial, unsigned* arrived, double* out, cudaStream_t st);
// Sets the time step the single-case kernels read.
void launch_set_step(StepDt* step, double dt, cudaStream_t st);
void launch_res_sum(const double* res, int nc, double* partial, double* out, cudaStream_t st);
void launch_set_flag(int* flag, int v, cudaStream_t st);
// dst[v][c] = src[v][c] + sign * off.v[v], v < nq, c < n (row strides in elements).
void launch_offset_rows(double* dst, int64_t dstStride, const double* src, int64_t srcStride, int n, int nq,
                        QOffset off, double sign, cudaStream_t st);
// Halo slots [first, first + nh) of dst (row stride dstNt) take `rows` values
// of cell srcCell[h] of partition srcPart[h] (base srcBase[p], stride srcNt[p]).
template <typename X>
void launch_halo_gather(X* dst, int dstNt, int first, int rows, int nh, const int* srcPart, const int* srcCell,
                        X* const* srcBase, const int* srcNt, cudaStream_t st);
// The same for an array of `words` floats per cell (a multiple of 4).
void launch_halo_gather_cells(float* dst, int first, int words, int nh, const int* srcPart, const int* srcCell,
                              float* const* srcBase, cudaStream_t st);

// Post-processing (post_kernels.cu).
void launch_stats(int D, const double* q, int64_t nt, QOffset qo, int nc, double gm1, int n, double* avg,
                  double* rms, cudaStream_t st);
void launch_probe(int D, const double* q, int64_t nt, QOffset qo, const int* cells, int n, double gm1, double pInf,
                  double* out, cudaStream_t st);
enum { kGhostFresh = 0, kGhostUndo = 1 };
template <typename T>
void launch_forces(const Args<T>& a, QOffset qo, const double* gS, const double* gD, const int* gPatch, int mode,
                   double Blast, const int* patches, int nPatches, double* terms, double* fp, double* fv,
                   cudaStream_t st);

// Fused FP32-bulk stage over tiles (tile_kernels.cu).
struct TileArgs {
    const TileDesc* tiles;
    const int* ints;
    const float* floats;
    const float* primIn;   // primitives at the stage start (the update writes the other buffer)
    int nTiles;
    int block;             // threads of a block
    size_t smemBytes;      // dynamic shared memory of a block
    int needGrad, needVis; // passes to run
    int haveV, haveGrad;   // arrays the fluxes read (zero where not computed)
};
size_t tile_smem_bytes(int D, int maxL, int maxLF, bool haveV, bool haveGrad);
// g: the solver's arguments with prim = the output primitive buffer.
cudaError_t launch_tile_stage(const Args<float>& g, const TileArgs& t, const StageConfig& s, cudaStream_t st);

constexpr int kKernelsPerStage = 5;  // prep, grad, vis, flux, update
// Timing slots of lfm_solver_profile_step: the five kernels, then the fused
// tile stage (which does the work of the five), then the fused flux + update
// (which does the work of the last two).
constexpr int kKernelSlots = 7;
constexpr int kSlotTileStage = 5;
constexpr int kSlotFluxUpdate = 6;
inline const char* kernelName(int i) {
    static const char* names[] = {"k_prep", "k_grad", "k_vis", "k_flux", "k_update", "k_tile_stage",
                                  "k_flux_update"};
    return (i >= 0 && i < kKernelSlots) ? names[i] : "";
}

}  // namespace dev
}  // namespace lfm
