// Persistent multi-case stage kernel of the batch engine (batch.cuh).
#include <algorithm>

#include "batch.cuh"
#include "solver_fp32.cuh"
#include "solver_launch.h"

namespace lfm {
namespace dev {

namespace {

// A grid barrier gives up after kBarrierTimeoutNs of waiting (read from the
// GPU's global nanosecond timer), or after kBarrierSpinLimit polls should
// that timer not advance.
constexpr unsigned long long kBarrierTimeoutNs = 1000000000ull;   // 1 s
constexpr unsigned kBarrierSpinLimit = 1u << 25;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier of the blocks of one launch (all resident: the launch is
// cooperative, or its grid is sized to the resident capacity). Arrival is an
// atomic increment after a release fence; between its arrival and its wait the
// block runs `meanwhile` (loads of what no phase writes). Waiting is bounded:
// after about a second, or once another block has given up, the block sets the
// error flag and the caller returns without touching further data. The flag
// and the timer are read every 64th poll only: with every poll they doubled
// the time from the last arrival to the wake-up.
template <class F>
__device__ __forceinline__ bool grid_barrier(unsigned* counter, unsigned target, int* error, F meanwhile) {
    __shared__ int sOk;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
    }
    meanwhile();
    if (threadIdx.x == 0) {
        int ok = 1;
        unsigned spins = 0;
        const unsigned long long t0 = global_ns();
        while (*(volatile unsigned*)counter < target) {
            if ((++spins & 63u) == 0 && (*(volatile int*)error != 0 || spins > kBarrierSpinLimit ||
                                         global_ns() - t0 > kBarrierTimeoutNs)) {
                atomicOr(error, 1);
                ok = 0;
                break;
            }
            __nanosleep(20);
        }
        __threadfence();
        sOk = ok;
    }
    __syncthreads();
    return sOk != 0;
}

// One item of a phase: a cell or ghost (prep, only in a case's first step
// after a new state: afterwards the update writes the next stage's primitives
// of each cell and of its boundary ghosts), a cell (grad + vis, update) or a
// face (flux) of the case in shared memory. FULL = false is the variant
// for batches of M1/M2 cases without viscosity: no gradient or viscous code
// is compiled in, which keeps the kernel's register count (and so its
// occupancy) down.
template <int PH, int D, bool FULL, bool PLAIN, class Sync>
__device__ __forceinline__ void item(const BatchCase& bc, int stage, int i, Sync sync) {
    const Args<float>& a = bc.a;
    if (PH == 0) {
        sync();
        prep32<D>(a, i);
    } else if (PH == 1) {
        if (FULL) {
            if (!PLAIN && bc.needGrad) {
                if (a.cfEll) grad32<D, true>(a, i, sync);
                else grad32<D, false>(a, i, sync);
            }
            if (bc.needVis) {
                if (PLAIN || a.cfEll) vis32<D, false, true>(a, i, sync);
                else vis32<D, false, false>(a, i, sync);
            }
        }
    } else if (PH == 2) {
        if (bc.scheme == kSchemeM1)
            flux32<D, kSchemeM1, FULL, false, false>(a, i, sync);
        else if (!FULL || PLAIN || bc.scheme == kSchemeM2)
            flux32<D, kSchemeM2, FULL, false, false>(a, i, sync);
        else
            flux32<D, kSchemeAUSM, FULL, false, false>(a, i, sync);
    } else {
        const int first = stage == 0;
        const bool res = bc.residuals && first;
        update32<D, PLAIN ? kEntriesEll : kEntriesEither>(a, i, bc.rkA[stage], bc.rkB[stage], bc.dt32, first, res, sync);
    }
}

// Makes case `slot` the block's current one (in shared memory), its primitive
// buffers as the stage reads (in) and writes (out) them: 0 or 1 of its two (a
// case that is never fused has the same one twice).
template <int BLOCK>
__device__ __forceinline__ void load_case(const BatchArgs& b, int slot, int in, int out, BatchCase& sc, int& sSlot) {
    // every thread of the block comes here with the same slot, and sSlot is
    // written between barriers, so the warps of a block need not wait for one
    // another until the case changes
    if (slot == sSlot) return;
    __syncthreads();
    const int4* src = reinterpret_cast<const int4*>(b.cases + slot);
    int4* dst = reinterpret_cast<int4*>(&sc);
    constexpr int n16 = (int)(sizeof(BatchCase) / 16);
    for (int k = threadIdx.x; k < n16; k += BLOCK) dst[k] = src[k];
    if (threadIdx.x == 0) sSlot = slot;
    __syncthreads();
    if (threadIdx.x == 0) {
        float* buf[2] = {sc.a.prim, sc.a.primW};
        sc.a.prim = in ? buf[1] : buf[0];
        sc.a.primW = out ? buf[1] : buf[0];
    }
    __syncthreads();
}

// The tiles of phase PH assigned to this block: a contiguous range of the
// phase's tile list (neighbouring tiles of a case share cached neighbours).
struct BlockTiles {
    int t0, t1;
    BatchTile first;
};

// The block's range of phase PH, its first tile and that tile's case: what the
// host wrote before the step, so a block loads it while it still waits for the
// phase before.
template <int PH, int BLOCK>
__device__ __forceinline__ BlockTiles block_tiles(const BatchArgs& b, int in, int out, BatchCase& sc, int& sSlot) {
    const int nT = b.nTiles[PH];
    BlockTiles r;
    r.t0 = (int)((long long)nT * blockIdx.x / gridDim.x);
    r.t1 = (int)((long long)nT * (blockIdx.x + 1) / gridDim.x);
    if (r.t0 < r.t1) {
        r.first = b.tiles[PH][r.t0];
        load_case<BLOCK>(b, r.first.slot, in, out, sc, sSlot);
    }
    return r;
}

template <int PH, int BLOCK, int DIMS, bool FULL, bool PLAIN, class Sync = NoWait>
__device__ __forceinline__ void phase_tiles(const BatchArgs& b, int stage, const BlockTiles& r, BatchCase& sc,
                                            int& sSlot, Sync sync = Sync()) {
    for (int t = r.t0; t < r.t1; ++t) {
        const BatchTile td = t == r.t0 ? r.first : b.tiles[PH][t];
        load_case<BLOCK>(b, td.slot, b.parity, b.parity, sc, sSlot);
        const int end = td.start + td.count;
        for (int k = 0; k < b.itemsPerThread; ++k) {
            const int i = td.start + (int)threadIdx.x + k * BLOCK;
            if (i < end) {
                if (DIMS == 2 || sc.a.D == 2)
                    item<PH, 2, FULL, PLAIN>(sc, stage, i, sync);
                else
                    item<PH, 3, FULL, PLAIN>(sc, stage, i, sync);
            }
        }
    }
}

// Resident blocks per SM the stage kernel is compiled for: its registers are
// those of its largest phase, and every phase waits for loads, so threads
// count: 1024 per SM for the 2D inviscid variant (64 registers), 768 with the
// viscous terms and M2AUSM in 2D (80), 512 with 3D cases (128).
constexpr int stage_blocks(int block, int dims, bool full) {
    const int threads = dims == 2 ? (full ? 768 : 1024) : 512;
    return threads >= block ? threads / block : 1;
}

// Stage `stage` of every case: [prep] | [grad + vis] | flux | update, with a
// grid barrier between phases (none after the last; the bracketed phases and
// their barriers only when they have tiles). Within the launch every array
// is written by one phase and read only by later ones, so no block reads a
// line it cached before another block rewrote it.
// DIMS = 2: every case is 2D; DIMS = 0: 2D and 3D cases. FULL: see item().
template <int BLOCK, int DIMS, bool FULL>
__global__ void __launch_bounds__(BLOCK, stage_blocks(BLOCK, DIMS, FULL)) k_batch_stage(const __grid_constant__ BatchArgs b,
                                                                                       int stage) {
    __shared__ BatchCase sc;
    __shared__ int sSlot;
    if (threadIdx.x == 0) sSlot = -1;
    __syncthreads();
    unsigned* counter = &b.ctl->barrier[stage];
    unsigned target = b.barrierExtra;   // 0 except under lfm_batch_debug_barrier
    BlockTiles r;
    auto barrier = [&](auto next) {
        target += gridDim.x;
        return grid_barrier(counter, target, b.error, next);
    };
    auto next1 = [&] { r = block_tiles<1, BLOCK>(b, b.parity, b.parity, sc, sSlot); };
    auto next2 = [&] { r = block_tiles<2, BLOCK>(b, b.parity, b.parity, sc, sSlot); };
    auto next3 = [&] { r = block_tiles<3, BLOCK>(b, b.parity, b.parity, sc, sSlot); };
    const bool grad = FULL && b.nTiles[1] > 0;
    auto after_prep = [&] { grad ? next1() : next2(); };
    if (b.nTiles[0] > 0) {
        r = block_tiles<0, BLOCK>(b, b.parity, b.parity, sc, sSlot);
        phase_tiles<0, BLOCK, DIMS, FULL, false>(b, stage, r, sc, sSlot);
        if (!barrier(after_prep)) return;
    } else {
        after_prep();
    }
    if (grad) {
        phase_tiles<1, BLOCK, DIMS, FULL, false>(b, stage, r, sc, sSlot);
        if (!barrier(next2)) return;
    }
    phase_tiles<2, BLOCK, DIMS, FULL, false>(b, stage, r, sc, sSlot);
    if (!barrier(next3)) return;
    phase_tiles<3, BLOCK, DIMS, FULL, false>(b, stage, r, sc, sSlot);
}

// Flux and update of cell i of a case that can do both at once (fluxupdate32).
__device__ __forceinline__ void fused_item(const BatchCase& bc, int stage, int i) {
    const int first = stage == 0;
    const bool res = bc.residuals && first;
    if (bc.scheme == kSchemeM1)
        fluxupdate32<2, kSchemeM1, false, true>(bc.a, i, bc.rkA[stage], bc.rkB[stage], bc.dt32, first, res);
    else
        fluxupdate32<2, kSchemeM2, false, true>(bc.a, i, bc.rkA[stage], bc.rkB[stage], bc.dt32, first, res);
}

// A stage of a batch whose cases can all do flux and update at once
// (CaseLayout::fusable) and have current primitives: one phase, no barrier, so stages follow one another as programmatic dependents (each loads
// its first tile's case before it waits for the stage before).
// 768 threads per SM (80 registers, 56 bytes spilled) beat 512 without spills
// and 1024 (64, 120 bytes): 143, 150 and 149 us a step of eight cases.
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK > 256 ? 1 : 768 / BLOCK) k_batch_fused(const __grid_constant__ BatchArgs b,
                                                                                     int stage) {
    __shared__ BatchCase sc;
    __shared__ int sSlot;
    if (threadIdx.x == 0) sSlot = -1;
    __syncthreads();
    const int in = (b.parity + stage) & 1;
    const BlockTiles r = block_tiles<3, BLOCK>(b, in, in ^ 1, sc, sSlot);
    PdlWait{1}();
    for (int t = r.t0; t < r.t1; ++t) {
        const BatchTile td = t == r.t0 ? r.first : b.tiles[3][t];
        load_case<BLOCK>(b, td.slot, in, in ^ 1, sc, sSlot);
        for (int k = 0; k < b.itemsPerThread; ++k) {
            const int i = td.start + (int)threadIdx.x + k * BLOCK;
            if (i < td.start + td.count) fused_item(sc, stage, i);
        }
    }
}

// One phase of a stage over every case, for the phased launch mode. PLAIN: no
// case is M2AUSM and all have fixed-width tables (PhasedShape::plain). A phase
// waits for loads, and without M2AUSM's reconstruction and the face lists it
// fits 1024 threads on an SM (64 registers; the 3D update then spills 212
// bytes, and is faster all the same); with them 512 (128). Us a step, GB300, of
// the general phases, of plain ones at 768 threads and at 1024: 2D and 3D of
// 14k cells each 88, 72, 74; viscous 2D of 289k 172, 156, 149; 3D of 365k 552,
// 414, 434; 2D and 3D of 308k 478, 399, 385.
template <bool PLAIN>
constexpr int phase_blocks(int block) {
    constexpr int threads = PLAIN ? 1024 : 512;
    return threads >= block ? threads / block : 1;
}

template <int PH, int BLOCK, int DIMS, bool FULL, bool PLAIN>
__global__ void __launch_bounds__(BLOCK, phase_blocks<PLAIN>(BLOCK)) k_batch_phase(const __grid_constant__ BatchArgs b, int stage) {
    __shared__ BatchCase sc;
    __shared__ int sSlot;
    if (threadIdx.x == 0) sSlot = -1;
    __syncthreads();
    const BlockTiles r = block_tiles<PH, BLOCK>(b, b.parity, b.parity, sc, sSlot);
    phase_tiles<PH, BLOCK, DIMS, FULL, PLAIN>(b, stage, r, sc, sSlot, PdlWait{1});
    PdlWait{1}();   // also where a block had no item: the next phase waits for this one alone
}

// New states of several cases, and their states out, in one launch each: one
// row of blocks per case, so that the copies over the C2C link overlap.
__global__ void __launch_bounds__(256) k_batch_set(const BatchCase* cases, const __grid_constant__ BatchStates m,
                                                   int parity) {
    __shared__ Args<float> a;
    const BatchCase& bc = cases[m.slot[blockIdx.y]];
    if ((int)(blockIdx.x * blockDim.x) >= bc.a.nc) return;
    if (threadIdx.x == 0) {
        a = bc.a;
        if (parity) a.prim = a.primW;   // the buffer the next step reads
    }
    __syncthreads();
    const int c = LFM_GLOBAL_ID();
    const double* q = m.q[blockIdx.y];
    if (c == 0) *a.flag = 0;   // a new state starts with a clear non-finite flag
    if (c >= a.nc) return;
    if (a.D == 2) set_state32<2>(a, q, a.nc, c);
    else set_state32<3>(a, q, a.nc, c);
}

// Primitives of one case's cells and ghosts from its stored state.
__global__ void __launch_bounds__(256) k_batch_prims(const BatchCase* cases, int slot, int parity) {
    __shared__ Args<float> a;
    if (threadIdx.x == 0) {
        a = cases[slot].a;
        if (parity) a.prim = a.primW;
    }
    __syncthreads();
    const int t = LFM_GLOBAL_ID();
    if (t >= a.nt) return;
    if (a.D == 2) prep32<2>(a, t);
    else prep32<3>(a, t);
}

__global__ void __launch_bounds__(256) k_batch_get(const BatchCase* cases, const __grid_constant__ BatchStates m) {
    const Args<float>& a = cases[m.slot[blockIdx.y]].a;
    const int c = LFM_GLOBAL_ID(), nc = a.nc;
    if (c >= nc) return;
    double* out = m.q[blockIdx.y];
    for (int v = 0; v < a.nq; ++v) out[(size_t)v * nc + c] = a.q[(size_t)v * a.nt + c] + a.qRef[v];
}

// The phases of a stage that have tiles, one kernel each, every one but the
// step's first a programmatic dependent of the one before.
template <int PH, int BLOCK, int DIMS, bool FULL, bool PLAIN>
cudaError_t launch_phase(const BatchArgs& b, int stage, const PhasedShape& p, bool* chained, cudaStream_t st) {
    if (p.tiles[PH] == 0) return cudaSuccess;
    static thread_local int fit = -1;   // resident blocks per SM of this kernel
    auto k = k_batch_phase<PH, BLOCK, DIMS, FULL, PLAIN>;
    if (fit < 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, BLOCK, 0);
        if (e != cudaSuccess || fit < 1) {
            fit = -1;
            return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
        }
    }
    const int per = p.blocksPerSm > 0 ? std::min(p.blocksPerSm, fit) : fit;
    // up to four grids' worth of blocks: their tiles differ in work, and a block
    // that ends early makes room for another (2D and 3D of 368k cells, one, two
    // and four grids: 438, 385, 377 us a step; M2AUSM and M1 of 150k 363, 266, 260)
    launch_kernel_pdl(*chained, k, (unsigned)std::min(p.tiles[PH], 4 * per * p.sms), BLOCK, st, b, stage);
    *chained = true;
    return cudaGetLastError();
}

template <int BLOCK, int DIMS, bool FULL, bool PLAIN>
cudaError_t launch_phases(const BatchArgs& b, int stage, const PhasedShape& p, cudaStream_t st) {
    bool chained = stage > 0;
    cudaError_t e = launch_phase<0, BLOCK, DIMS, FULL, PLAIN>(b, stage, p, &chained, st);
    if (e == cudaSuccess && FULL) e = launch_phase<1, BLOCK, DIMS, FULL, PLAIN>(b, stage, p, &chained, st);
    if (e == cudaSuccess) e = launch_phase<2, BLOCK, DIMS, FULL, PLAIN>(b, stage, p, &chained, st);
    if (e == cudaSuccess) e = launch_phase<3, BLOCK, DIMS, FULL, PLAIN>(b, stage, p, &chained, st);
    return e;
}

template <int BLOCK>
cudaError_t launch_phases_variant(const BatchArgs& b, int stage, int variant, const PhasedShape& p, cudaStream_t st) {
    switch (variant) {
        case kBatchVariant2DInviscid: return launch_phases<BLOCK, 2, false, false>(b, stage, p, st);
        case kBatchVariant2D:
            return p.plain ? launch_phases<BLOCK, 2, true, true>(b, stage, p, st)
                           : launch_phases<BLOCK, 2, true, false>(b, stage, p, st);
        default:
            return p.plain ? launch_phases<BLOCK, 0, true, true>(b, stage, p, st)
                           : launch_phases<BLOCK, 0, true, false>(b, stage, p, st);
    }
}

// Kernel of a launch shape and variant (kBatchVariant*).
template <int BLOCK>
auto kernel_of(int variant) -> void (*)(BatchArgs, int) {
    switch (variant) {
        case kBatchVariant2DInviscid: return k_batch_stage<BLOCK, 2, false>;
        case kBatchVariant2D: return k_batch_stage<BLOCK, 2, true>;
        default: return k_batch_stage<BLOCK, 0, true>;
    }
}

template <int BLOCK>
cudaError_t launch_block(const BatchArgs& b, int stage, int variant, int grid, bool cooperative, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(BLOCK);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = cooperative ? attr : nullptr;
    cfg.numAttrs = cooperative ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel_of<BLOCK>(variant), b, stage);
}

}  // namespace

cudaError_t launch_batch_stage(const BatchArgs& b, int stage, int block, int variant, int grid, bool cooperative,
                               cudaStream_t st) {
    switch (block) {
        case 128: return launch_block<128>(b, stage, variant, grid, cooperative, st);
        case 512: return launch_block<512>(b, stage, variant, grid, cooperative, st);
        default: return launch_block<256>(b, stage, variant, grid, cooperative, st);
    }
}

template <int BLOCK>
static cudaError_t launch_fused(const BatchArgs& b, int stage, const PhasedShape& p, cudaStream_t st) {
    static thread_local int fit = -1;   // resident blocks per SM
    if (fit < 0) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_batch_fused<BLOCK>, BLOCK, 0);
        if (e != cudaSuccess || fit < 1) {
            fit = -1;
            return e != cudaSuccess ? e : cudaErrorInvalidConfiguration;
        }
    }
    // Up to 32 grids' worth of blocks: one that ends early makes room for
    // another, and few tiles a block leave its warps out of step. At 128 threads,
    // us a step with two, eight and 32 grids: 2.5M cells 850, 698, 706; 9.7M cells
    // with eight and 32: 2806, 2536. Below 230k cells there is a tile a block.
    const int per = p.blocksPerSm > 0 ? std::min(p.blocksPerSm, fit) : fit;
    launch_kernel_pdl(stage > 0, k_batch_fused<BLOCK>, (unsigned)std::min(p.tiles[3], 32 * per * p.sms), BLOCK, st, b,
                      stage);
    return cudaGetLastError();
}

cudaError_t launch_batch_fused(const BatchArgs& b, int stage, int block, const PhasedShape& p, cudaStream_t st) {
    switch (block) {
        case 128: return launch_fused<128>(b, stage, p, st);
        case 512: return launch_fused<512>(b, stage, p, st);
        default: return launch_fused<256>(b, stage, p, st);
    }
}

cudaError_t launch_batch_prims(const BatchCase* cases, int slot, int nt, int parity, cudaStream_t st) {
    k_batch_prims<<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(cases, slot, parity);
    return cudaGetLastError();
}

cudaError_t launch_batch_states(const BatchCase* cases, const BatchStates& m, int n, int maxCells, bool set, int parity,
                                cudaStream_t st) {
    const dim3 grid((unsigned)((maxCells + 255) / 256), (unsigned)n);
    if (set) k_batch_set<<<grid, 256, 0, st>>>(cases, m, parity);
    else k_batch_get<<<grid, 256, 0, st>>>(cases, m);
    return cudaGetLastError();
}

cudaError_t launch_batch_phased(const BatchArgs& b, int stage, int block, int variant, const PhasedShape& p,
                                cudaStream_t st) {
    switch (block) {
        case 128: return launch_phases_variant<128>(b, stage, variant, p, st);
        case 512: return launch_phases_variant<512>(b, stage, variant, p, st);
        default: return launch_phases_variant<256>(b, stage, variant, p, st);
    }
}

int batch_blocks_per_sm(int block, int variant) {
    int n = 0;
    cudaError_t e;
    switch (block) {
        case 128: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_of<128>(variant), 128, 0); break;
        case 512: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_of<512>(variant), 512, 0); break;
        default: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_of<256>(variant), 256, 0); break;
    }
    return e == cudaSuccess ? n : 0;
}

}  // namespace dev
}  // namespace lfm
