// Host-side packing of the FP32-bulk face geometry (plain C++: used by the
// solver and batch set-up and by the tile builder).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>

#include "lfm_gpu.h"

namespace lfm {
namespace setup {

// FP32-bulk face geometry of face f in its 16-byte parts (Args::fG0, fG1;
// solver_fp32.cuh gives the layout), its cells p and n as given. Each value is
// the FP64 one rounded to FP32.
inline void packFace32(const lfm_solver_desc* d, size_t f, int p, int n, float* g0, float* g1) {
    const size_t nf = (size_t)d->n_faces;
    const float w = (float)d->w[f], lapc = (float)(d->delta_mag[f] * d->dmag_inv[f]);
    for (size_t k = 0; k < (size_t)d->dim; ++k) {
        g0[k] = (float)d->S[k * nf + f];
        g1[k] = (float)d->K[k * nf + f];
    }
    if (d->dim == 2) {
        g0[2] = w;
        g0[3] = lapc;
        std::memcpy(&g1[2], &p, 4);
        std::memcpy(&g1[3], &n, 4);
    } else {
        g0[3] = w;
        g1[3] = lapc;
    }
}
// A face's N side n with the face's boundary flag in the top bit.
inline int flaggedN(const lfm_solver_desc* d, size_t f, int n) {
    return (int)((uint32_t)n | (d->face_ghost[f] ? 0x80000000u : 0u));
}
inline int flaggedN(const lfm_solver_desc* d, size_t f) { return flaggedN(d, f, (int)d->face_n[f]); }

}  // namespace setup
}  // namespace lfm
