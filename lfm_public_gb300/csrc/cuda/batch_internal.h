// Host-side internals of the batch engine shared by the batch C ABI
// (capi_batch.cu) and the request server (capi_server.cu).
#pragma once

#include <cstddef>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "args_setup.h"
#include "batch.cuh"
#include "lfm_gpu.h"
#include "solver_launch.h"

namespace lfm {
namespace batch {

constexpr size_t kAlign = 256;
inline size_t roundUp(size_t b) { return (b + kAlign - 1) & ~(kAlign - 1); }

// First-fit allocator over [0, size) in 256-byte granules; free ranges are
// kept sorted by offset and coalesced on release.
class Arena {
public:
    void reset(size_t size) {
        free_.clear();
        size_ = size & ~(kAlign - 1);
        if (size_) free_[0] = size_;
    }
    bool alloc(size_t bytes, size_t* off) {
        bytes = roundUp(bytes);
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second >= bytes) {
                *off = it->first;
                const size_t rest = it->second - bytes;
                const size_t at = it->first + bytes;
                free_.erase(it);
                if (rest) free_[at] = rest;
                return true;
            }
        }
        return false;
    }
    void release(size_t off, size_t bytes) {
        bytes = roundUp(bytes);
        auto it = free_.emplace(off, bytes).first;
        auto nx = std::next(it);
        if (nx != free_.end() && it->first + it->second == nx->first) {
            it->second += nx->second;
            free_.erase(nx);
        }
        if (it != free_.begin()) {
            auto pv = std::prev(it);
            if (pv->first + pv->second == it->first) {
                pv->second += it->second;
                free_.erase(it);
            }
        }
    }
    size_t largest() const {
        size_t m = 0;
        for (auto& kv : free_) m = std::max(m, kv.second);
        return m;
    }
    size_t total() const {
        size_t m = 0;
        for (auto& kv : free_) m += kv.second;
        return m;
    }
    size_t size() const { return size_; }

private:
    std::map<size_t, size_t> free_;
    size_t size_ = 0;
};

// Byte offsets of every array of one case inside its arena block.
struct CaseLayout {
    size_t total = 0;
    bool fusable;   // flux and update at once (fluxupdate32)
    size_t q, dq, res, prim, prim1, V, grad, flux, fG0, fG1, d, dinv, dnorm, fP, fN, volInv32, sponge, cfOff, cfList,
        cfNbr, cfEll, cfEllN, cellGhosts, gCell, gKind, gFace;

    explicit CaseLayout(const lfm_solver_desc* d) {
        const size_t D = (size_t)d->dim, nq = (size_t)d->nq, nc = (size_t)d->n_cells, ng = (size_t)d->n_ghosts;
        const size_t nt = nc + ng, nf = (size_t)d->n_faces, ne = (size_t)d->cell_face_offsets[nc];
        const bool ausm = d->solver == LFM_SOLVER_M2AUSM;
        q = add(nq * nt * 8);
        dq = add(nq * nc * 4);
        res = d->residuals ? add(nq * nc * 8) : npos();
        prim = add((size_t)lfm::dev::primRows<float>(d->dim) * nt * 4);
        // As in the single-case solver, evaluating each face twice pays where
        // the flux is short (2D inviscid M1 / M2): a stage then is one phase
        // without a grid barrier. The second primitive buffer takes the space that
        // rows of single values and a second copy of the face lists would: callers
        // size arenas by that footprint, and no case may outgrow it (one of mostly
        // isolated cells would, with far more ghosts than cells).
        const size_t one = roundUp(nf), fours = roundUp(nf * 4), eights = roundUp(nf * 8);
        const size_t rows = 4 * eights + 5 * fours + one + roundUp(nc * 8) + roundUp((nc + 1) * 4) + 2 * roundUp(ne * 4);
        const size_t parts = 2 * roundUp(nf * 16) + roundUp(nc * 16);
        const size_t second = roundUp((size_t)lfm::dev::primRows<float>(d->dim) * nt * 4);
        fusable = D == 2 && !lfm::setup::needVis(d) && !ausm && lfm::setup::ellFits(d) && parts + second <= rows;
        prim1 = fusable ? add((size_t)lfm::dev::primRows<float>(d->dim) * nt * 4) : npos();
        V = lfm::setup::needVis(d) ? add((size_t)lfm::dev::visStride32(d->dim, false) * nt * 4) : npos();
        grad = ausm ? add((size_t)lfm::dev::gradStride32(d->dim) * nt * 4) : npos();
        flux = add(nq * nf * 4);
        fG0 = add(nf * 16);
        fG1 = add(nf * 16);
        this->d = ausm ? add(D * nf * 4) : npos();
        // the two-point gradients of viscous boundary faces
        dinv = d->mu != 0.0 ? add(nf * 4) : npos();
        dnorm = d->mu != 0.0 ? add(D * nf * 4) : npos();
        fP = D == 3 ? add(nf * 4) : npos();   // 2D: in fG1
        fN = D == 3 ? add(nf * 4) : npos();
        volInv32 = add(nc * 4);
        sponge = add(nc * 4);
        // the fixed-width cell -> face tables when every cell fits them, else
        // the face lists
        const bool fits = lfm::setup::ellFits(d);
        cfOff = fits ? npos() : add((nc + 1) * 4);
        cfList = fits ? npos() : add(ne * 4);
        cfNbr = fits ? npos() : add(ne * 4);
        const size_t W = (size_t)(D == 2 ? lfm::dev::kEllWidth<2> : lfm::dev::kEllWidth<3>);
        cfEll = fits ? add(W * nc * 4) : npos();
        cfEllN = fits ? add(W * nc * 4) : npos();
        cellGhosts = add(nc);
        gCell = add(ng * 4);
        gKind = add(ng * 4);
        gFace = add(ng * 4);
    }
    static size_t npos() { return ~(size_t)0; }

private:
    size_t add(size_t bytes) {
        const size_t at = total;
        total += roundUp(bytes ? bytes : 1);
        return at;
    }
};

struct Slot {
    bool used = false;
    size_t off = 0, bytes = 0;
    int D = 2, nq = 4, nc = 0, ng = 0, nf = 0, nt = 0;
    bool needGradVis = false, fusable = false, plain = false;
    bool primsValid = false;   // cells' primitives current (kept so by the update phase)
    double qRef[5] = {0, 0, 0, 0, 0};   // the device state is q - qRef
    double* q = nullptr;   // device
    lfm::dev::Args<float> a{};   // the case's kernel arguments (host copy)
};

// A case ready for admission: its arena block image (constant arrays and
// initial state in device layout) and its kernel constants. Built on the host
// only, so a server can prepare requests on the submitting thread.
struct PreparedCase {
    CaseLayout layout;
    std::vector<unsigned char> image;
    dev::BatchCase bc{};          // constants; device pointers filled at admission
    int D = 2, nq = 4, nc = 0, ng = 0, nf = 0;
    bool needGradVis = false;
    explicit PreparedCase(const lfm_solver_desc* d) : layout(d) {}
};

// Validates a description against the batch's RK order and builds its image.
int prepareCase(const lfm_solver_desc* d, double dt, int rkOrder, PreparedCase** out);
// Admits a prepared case: arena block, upload, case table. LFM_ERR_NOMEM when
// no slot or no arena block of its size is free.
int commitCase(lfm_batch* b, const PreparedCase& pc, int* slot);

}  // namespace batch
}  // namespace lfm

struct lfm_batch {
    int device = 0;
    cudaStream_t stream = nullptr;
    int rkOrder = 5;
    int maxCases = 0;
    unsigned char* arenaBase = nullptr;
    lfm::batch::Arena arena;
    lfm::dev::BatchCase* dCases = nullptr;
    int* dFlags = nullptr;
    int* dError = nullptr;
    lfm::dev::BatchCtl* dCtl = nullptr;
    lfm::dev::BatchTile* dTiles[lfm::dev::kBatchPhases] = {};
    size_t tileCap[lfm::dev::kBatchPhases] = {};
    int* dNTiles = nullptr;
    std::vector<lfm::batch::Slot> slots;
    int sms = 0;
    // One kernel per phase at 128 threads until a shape is asked for: small
    // batches are latency-bound, and their phases then overlap as programmatic
    // dependents where the persistent kernel waits at its grid barriers (three
    // cases of 11k-29k cells, 2D and 3D: 139 -> 112 us a step, GB300).
    lfm_batch_tuning tune{128, 1, 0, 1, 1};
    int variant = lfm::dev::kBatchVariantGeneral;   // stage-kernel variant of the current cases
    bool plain = false;                 // its phases' (PhasedShape::plain)
    bool untuned = true;        // no launch shape was asked for
    int nTiles[lfm::dev::kBatchPhases] = {};
    int grid = 0;
    bool tilesDirty = true;
    bool lean = false;          // every case is fusable and has current primitives
    int parity = 0;             // the fusable cases' current primitive buffer
    cudaGraphExec_t graph[2][2] = {};   // a step's graph, by [lean][parity]
    bool graphStale[2][2] = {};         // its kernels, grids or arguments have changed
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    void* scrub = nullptr;
    size_t scrubBytes = 0;
    double* dStage = nullptr;   // a case's absolute state in transit to or from the host
    size_t stageBytes = 0;
    unsigned barrierExtra = 0;  // lfm_batch_debug_barrier
};
