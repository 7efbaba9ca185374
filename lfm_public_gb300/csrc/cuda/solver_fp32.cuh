// FP32-bulk form of the time step: face fluxes, limiter, residual sums and
// the RK increment register dq in FP32; the accumulation of the conserved
// state, boundary ghost states, geometry precompute and the dt reduction in
// FP64.
//
// Perturbation form. The FP64 state is stored as its deviation from a
// constant reference state q_ref = (rho_inf, rho_inf U_inf, rho_inf E_inf):
// q' = q - q_ref (exact differences of nearby numbers, and no cancellation
// when it is rounded to FP32). Every FP32 quantity is a perturbation too:
// r' = rho - rho_inf, m' = rho u - rho_inf U_inf, u' = u - U_inf and
// R psi' = p/rho - p_ref/rho_inf, derived by expressions whose terms are all
// perturbation-sized. Each face rhs is F(q_f).S - F(q_ref).S. The
// reference-state flux through the faces of a cell sums to
// F(q_ref).(sum_f S_f) = 0 because the face vectors of a closed cell cancel,
// so dropping it leaves every cell residual unchanged while FP32 rounding only
// ever scales perturbations. Evaluated on absolute values, FP32 would round
// the pressure (~1e5 Pa) by ~1e-2 Pa per face, the size of an acoustic wave;
// here the rounding is ~1e-7 of the perturbation.
//
// GB300 runs FP64 instructions (conversions included) at about two per clock
// per SM, so the FP64 work is kept to one FMA per component, the
// accumulation of the conserved state: conversions between FP32 and FP64 run on the
// integer pipes (fp_convert.cuh), and the update kernel derives the next
// stage's primitives from the new state while it holds it in registers
// (prims32), so a stage reads q' once. The primitive formulas use explicitly
// rounded operations, so they give the same bits wherever they are inlined.
//
// The schemes are those of the FP64 kernels (solver_kernels.cu), which follow
// the reference (src/cfd_v0.cpp:1896-2822): M1 as the central flux its
// Kurganov-Tadmor formula reduces to, M2 and M2AUSM as written, with the
// perfect-gas enthalpy h = e + p/rho = gamma/(gamma-1) R psi.
#pragma once

#include "fp_convert.cuh"
#include "solver_device.cuh"

namespace lfm {
namespace dev {

// ---------------------------------------------------------------------------
// Layout. What a thread reads of one cell, ghost or face lies together, in
// 16-byte parts, so that a gather is one to six vector loads where rows of
// single values take 6 to 15 loads with their address arithmetic (a 2D viscous
// face: 10 loads instead of 37):
//   prim   [nt] float4 A, then [nt] B, then [nt] c (sound speed, M2AUSM only)
//          2D: A = u'[2], R psi', rho'   B = m'[2]
//          3D: A = u'[3], R psi'         B = m'[3], rho'
//          (the viscous pass reads A alone)
//   V      [nt] kVisStride floats: dudx, dTdx, sigmaU, then the LES stress
//   grad   [nt] kGradStride floats: rho, p, u gradients
//   flux   [nf] float4: the first four rhs, then (3D) [nf] the fifth
//   fG0    [nf] float4  2D: S[2], w, |delta|/|d|   3D: S[3], w
//   fG1    [nf] float4  2D: K[2], P, N (integers)  3D: K[3], |delta|/|d|
//   fN, N  the N side, its top bit set on boundary faces
//   cfEll, cfEllN  [nc][kEllWidth]: a cell's face entries and the cells across
// Values and their order of evaluation do not depend on the layout. The kernels
// wait for loads (ncu: long scoreboard), so what counts is the bytes a thread
// has in flight and the round trips it makes. Measured on GB300 against rows
// of single values, us a step: 768 x 512 M1 cylinder (in L2) 184 -> 164, of it
// the flux 72 -> 54; 331 x 217 M2AUSM cylinder 118 -> 101; 192 x 128 x 48 wake
// (HBM) 986 -> 920; 256 x 256 vortex 51 -> 45.
// ---------------------------------------------------------------------------
template <int D>
struct Prim32 {
    float r, m[D], u[D], R;   // rho', m', u', R psi'
};

template <int D>
struct Face32 {
    float S[D], w, K[D], lapc;
};

template <int D, bool LES>
constexpr int kVisStride = visStride32(D, LES);
template <int D>
constexpr int kGradStride = gradStride32(D);

// Floats from the start of prim to its B part and to its sound speeds.
__device__ __forceinline__ size_t prim_b(size_t nt) { return 4 * nt; }
template <int D>
__device__ __forceinline__ size_t prim_c(size_t nt) {
    return (size_t)(2 * D + 2) * nt;
}

template <int D>
__device__ __forceinline__ void load_prim(const Args<float>& a, int t, Prim32<D>& p) {
    const float4 A = reinterpret_cast<const float4*>(a.prim)[t];
    const float* b = a.prim + prim_b((size_t)a.nt);
    p.u[0] = A.x;
    p.u[1] = A.y;
    if constexpr (D == 2) {
        const float2 B = reinterpret_cast<const float2*>(b)[t];
        p.R = A.z;
        p.r = A.w;
        p.m[0] = B.x;
        p.m[1] = B.y;
    } else {
        const float4 B = reinterpret_cast<const float4*>(b)[t];
        p.u[2] = A.z;
        p.R = A.w;
        p.m[0] = B.x;
        p.m[1] = B.y;
        p.m[2] = B.z;
        p.r = B.w;
    }
}

// u' and R psi' of cell t (and rho' in 2D).
template <int D>
__device__ __forceinline__ void load_uR(const Args<float>& a, int t, float* u, float& R) {
    const float4 A = reinterpret_cast<const float4*>(a.prim)[t];
    u[0] = A.x;
    u[1] = A.y;
    if constexpr (D == 2) {
        R = A.z;
    } else {
        u[2] = A.z;
        R = A.w;
    }
}

template <int D>
__device__ __forceinline__ void store_prim(const Args<float>& a, float* dst, int t, const Prim32<D>& p) {
    float* b = dst + prim_b((size_t)a.nt);
    if constexpr (D == 2) {
        reinterpret_cast<float4*>(dst)[t] = make_float4(p.u[0], p.u[1], p.R, p.r);
        reinterpret_cast<float2*>(b)[t] = make_float2(p.m[0], p.m[1]);
    } else {
        reinterpret_cast<float4*>(dst)[t] = make_float4(p.u[0], p.u[1], p.u[2], p.R);
        reinterpret_cast<float4*>(b)[t] = make_float4(p.m[0], p.m[1], p.m[2], p.r);
    }
}

template <int N>
__device__ __forceinline__ void load_vec4(const float* p, float* out) {
#pragma unroll
    for (int k = 0; k < N / 4; ++k) {
        const float4 x = reinterpret_cast<const float4*>(p)[k];
        out[4 * k] = x.x;
        out[4 * k + 1] = x.y;
        out[4 * k + 2] = x.z;
        out[4 * k + 3] = x.w;
    }
}
template <int N>
__device__ __forceinline__ void store_vec4(float* p, const float* v) {
#pragma unroll
    for (int k = 0; k < N / 4; ++k)
        reinterpret_cast<float4*>(p)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}

// Viscous rows of a cell: kVisRows values, padded to whole float4 (3D: 16).
template <int D>
constexpr int kVisVec = D == 2 ? 8 : 16;
template <int D, bool LES>
__device__ __forceinline__ void load_vis(const Args<float>& a, int t, float* v) {
    load_vec4<kVisVec<D>>(a.V + (size_t)t * kVisStride<D, LES>, v);
}

// Face f: geometry, and its cells i (P) and j (N); ghost: a boundary face.
template <int D>
__device__ __forceinline__ void load_face(const Args<float>& a, int f, Face32<D>& g, int& i, int& j, bool& ghost) {
    const float4 g0 = a.fG0[f], g1 = a.fG1[f];
    int n;
    g.S[0] = g0.x;
    g.S[1] = g0.y;
    g.K[0] = g1.x;
    g.K[1] = g1.y;
    if constexpr (D == 2) {
        g.w = g0.z;
        g.lapc = g0.w;
        i = __float_as_int(g1.z);
        n = __float_as_int(g1.w);
    } else {
        g.S[2] = g0.z;
        g.w = g0.w;
        g.K[2] = g1.z;
        g.lapc = g1.w;
        i = a.fP[f];
        n = a.fN[f];
    }
    ghost = n < 0;
    j = n & 0x7fffffff;
}

// S and w of face f.
template <int D>
__device__ __forceinline__ float load_Sw(const Args<float>& a, int f, float* S) {
    const float4 g0 = a.fG0[f];
    S[0] = g0.x;
    S[1] = g0.y;
    if constexpr (D == 2) {
        return g0.z;
    } else {
        S[2] = g0.z;
        return g0.w;
    }
}

// The kEllWidth entries of cell c in a fixed-width table.
template <int D>
__device__ __forceinline__ void load_ell(const int* table, int c, int* out) {
    if constexpr (D == 2) {
        const int4 x = reinterpret_cast<const int4*>(table)[c];
        out[0] = x.x;
        out[1] = x.y;
        out[2] = x.z;
        out[3] = x.w;
    } else {
        const int2* p = reinterpret_cast<const int2*>(table) + 3 * (size_t)c;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int2 x = p[k];
            out[2 * k] = x.x;
            out[2 * k + 1] = x.y;
        }
    }
}

template <int D>
__device__ __forceinline__ void load_flux(const Args<float>& a, int f, float* v) {
    load_vec4<4>(a.flux + 4 * (size_t)f, v);
    if constexpr (D == 3) v[4] = a.flux[4 * (size_t)a.nf + f];
}
template <int D>
__device__ __forceinline__ void store_flux(const Args<float>& a, int f, const float* v) {
    store_vec4<4>(a.flux + 4 * (size_t)f, v);
    if constexpr (D == 3) a.flux[4 * (size_t)a.nf + f] = v[4];
}

// p - p_ref of a state with perturbations r', R psi':
// rho R psi - rho_inf R psi_inf = rho_inf R psi' + r' (R psi_inf + R psi').
__device__ __forceinline__ float pressure_dev(const RefState32& R, float r, float Rpsi) {
    return R.rho * Rpsi + r * (R.Rpsi + Rpsi);
}

// ---------------------------------------------------------------------------
// prims32: FP32 primitives of interior cell t from its FP64 perturbation state
// qp = q - q_ref. Explicitly rounded operations only (no contraction), so the
// preparation and update kernels produce identical bits.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void prims32(const Args<float>& a, int t, const double* qp, float* dst) {
    const RefState32& R = a.ref;
    const size_t nt = (size_t)a.nt;
    const float r = f64_to_f32(qp[0]);
    float m[D];
#pragma unroll
    for (int k = 0; k < D; ++k) m[k] = f64_to_f32(qp[k + 1]);
    const float E = f64_to_f32(qp[D + 1]);
    const float rho = __fadd_rn(R.rho, r);
    const float rinv = __frcp_rn(rho);
    float u[D], Uu = 0.0f, uu = 0.0f, U2 = 0.0f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        u[k] = __fmul_rn(__fmaf_rn(-R.U[k], r, m[k]), rinv);   // (m' - U_inf r') / rho
        Uu = __fmaf_rn(R.U[k], u[k], Uu);
        uu = __fmaf_rn(u[k], u[k], uu);
        U2 = __fmaf_rn(R.U[k], R.U[k], U2);
    }
    // kinetic energy: rho|u|^2/2 - rho_inf|U_inf|^2/2 = r'|U_inf|^2/2 + rho (U_inf.u' + |u'|^2/2)
    const float K = __fmaf_rn(rho, __fmaf_rn(0.5f, uu, Uu), __fmul_rn(__fmul_rn(0.5f, r), U2));
    const float p = __fmul_rn(R.gm1, __fsub_rn(E, K));            // p - p_ref
    const float Rpsi = __fmul_rn(__fmaf_rn(-R.Rpsi, r, p), rinv);  // p/rho - p_ref/rho_inf
    Prim32<D> p32;
    p32.r = r;
    p32.R = Rpsi;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        p32.m[k] = m[k];
        p32.u[k] = u[k];
    }
    store_prim<D>(a, dst, t, p32);
    if (a.primC) dst[prim_c<D>(nt) + t] = __fsqrt_rn(__fmul_rn(R.gamma, __fadd_rn(R.Rpsi, Rpsi)));
}

// ---------------------------------------------------------------------------
// ghost32: boundary state of ghost g (FP64) from the absolute state qi of its
// interior cell, and its FP32 primitives. A ghost state can lie far from the
// free stream (a wall mirrors the momentum, u' = -2 U_inf - u'), where the
// FP32 kinetic-energy difference of prims32 would cancel; ghosts are few, so
// theirs is FP64.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void ghost32(const Args<float>& a, int g, int kind, const GhostIn<D>& in, float* dst) {
    const int t = a.nc + g;
    GhostState<D> o;
    ghost_state<float, D>(a, g, kind, in, o);
    Prim32<D> p32;
    p32.r = (float)(o.q[0] - a.qRef[0]);
#pragma unroll
    for (int k = 0; k < D; ++k) {
        p32.m[k] = (float)(o.q[k + 1] - a.qRef[k + 1]);
        p32.u[k] = (float)(o.u[k] - a.UInf[k]);
    }
    p32.R = (float)(o.R - a.RpsiRef);
    store_prim<D>(a, dst, t, p32);
    if (a.primC) dst[prim_c<D>((size_t)a.nt) + t] = sqrtf(a.ref.gamma * (a.ref.Rpsi + p32.R));
}

// ---------------------------------------------------------------------------
// prep32: primitives of cell or halo t from the stored perturbation state, or,
// for a ghost, its boundary state (FP64, from the interior cell) and primitives.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void prep32(const Args<float>& a, int t) {
    constexpr int NQ = D + 2;
    const size_t nt = (size_t)a.nt;
    if (t < a.nc || t >= a.nc + a.ng) {
        double qp[NQ];
#pragma unroll
        for (int v = 0; v < NQ; ++v) qp[v] = a.q[(size_t)v * nt + t];
        prims32<D>(a, t, qp, a.prim);
        return;
    }
    const int g = t - a.nc;
    const int in = a.gCell[g];
    double qi[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) qi[v] = a.q[(size_t)v * nt + in] + a.qRef[v];
    ghost32<D>(a, g, a.gKind[g], ghost_in<float, D>(a, qi), a.prim);
}

// ---------------------------------------------------------------------------
// update32: gather of the face rhs of cell c in ascending face order (the
// reference's scatter order; the sum is the cell residual RES), sponge source
// and low-storage RK update of the FP64 perturbation state
// (src/cfd_v0.cpp:2800-2822), then the next stage's primitives of the cell.
// The increment dt/V RES, the sponge source and the RK register
// dq = A dq + increment are FP32: dq restarts at every step (A = 0 in stage
// 0) and holds only that step's increments, so its rounding is that of the
// FP32 rhs it sums. The conserved state accumulates in FP64,
// q' = q' + B dq (one FP64 FMA per component), so rounding does not build up
// over the steps. The sponge pulls q towards q_ref:
// dt sigma (q_ref - q) = -dt sigma q'.
// The cell also writes the next stage's state of its boundary ghosts
// (a ghost depends on its interior cell only), so no preparation pass over
// the ghosts is needed; the values are those prep32 computes.
// ---------------------------------------------------------------------------
// ghosts_of32: the FP32 primitives of the boundary ghosts of cell c, from FP64
// states formed from its perturbation state qp (those prep32 computes).
template <int D>
__device__ __forceinline__ void ghosts_of32(const Args<float>& a, int c, const CellGhosts& g, const double* qp,
                                            float* dst) {
    constexpr int NQ = D + 2;
    double qa[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) qa[v] = qp[v] + a.qRef[v];
    const GhostIn<D> in = ghost_in<float, D>(a, qa);
    for_ghosts<float, D>(a, c, g, [&](int j, int kind) { ghost32<D>(a, j - a.nc, kind, in, dst); });
}

// gather32: the face rhs sum of cell c (ascending face order). The face's sign
// (+ where c is P, - where N) is a sign-bit flip of the loaded value, so an
// entry costs one add (a - b is a + (-b) in IEEE arithmetic: the same bits).
template <int D>
__device__ __forceinline__ void gather32(const Args<float>& a, int c, float* sum) {
    constexpr int NQ = D + 2;
#pragma unroll
    for (int v = 0; v < NQ; ++v) sum[v] = 0.0f;
    for (int e = a.cfOff[c]; e < a.cfOff[c + 1]; ++e) {
        const int code = a.cfList[e];
        float x[NQ];
        load_flux<D>(a, code >= 0 ? code : ~code, x);
#pragma unroll
        for (int v = 0; v < NQ; ++v) sum[v] += code >= 0 ? x[v] : neg_bits(x[v]);
    }
}

// gather32_ell: gather32 through the fixed-width table. Every face index of
// the cell is loaded at once, then every face's rhs, so the gather costs two
// memory round trips instead of one per face; the sum runs in the same
// (ascending face) order, so it has gather32's bits.
template <int D, class F>
__device__ __forceinline__ void gather32_ell(const Args<float>& a, const int* code, float* sum, F meanwhile) {
    constexpr int NQ = D + 2, W = kEllWidth<D>;
    float x[W][NQ];
#pragma unroll
    for (int k = 0; k < W; ++k)
        if (code[k] != kEllPad) load_flux<D>(a, code[k] >= 0 ? code[k] : ~code[k], x[k]);
    meanwhile();   // while they are in flight
#pragma unroll
    for (int v = 0; v < NQ; ++v) sum[v] = 0.0f;
#pragma unroll
    for (int k = 0; k < W; ++k) {
        if (code[k] == kEllPad) continue;
#pragma unroll
        for (int v = 0; v < NQ; ++v) sum[v] += code[k] >= 0 ? x[k][v] : neg_bits(x[k][v]);
    }
}

// The cell's own values the update reads, loaded before its rhs gather so
// that they are in flight together with it.
template <int D>
struct CellIn32 {
    double qp[D + 2];   // q'
    float dq[D + 2];
    float vi, sg;       // 1/V, sponge sigma
    int ghosts;         // it has boundary faces
    CellGhosts gh;
};

template <int D, class Sync = NoWait>
__device__ __forceinline__ void load_cell32(const Args<float>& a, int c, int first, CellIn32<D>& in,
                                            Sync sync = Sync()) {
    const size_t nt = (size_t)a.nt, nc = (size_t)a.nc;
    in.vi = a.volInv32[c];
    in.sg = a.sponge[c];
    in.ghosts = a.cellGhosts[c];
    sync();
#pragma unroll
    for (int v = 0; v < D + 2; ++v) {
        in.qp[v] = a.q[v * nt + c];
        in.dq[v] = first ? 0.0f : a.dq[v * nc + c];
    }
}

// apply32: the update of cell c from its rhs sum and its loaded values
// (see update32).
template <int D>
__device__ __forceinline__ void apply32(const Args<float>& a, int c, const float* sum, const CellIn32<D>& in,
                                        double Ak, double Bk, float dt32, int first, bool res) {
    constexpr int NQ = D + 2;
    const size_t nt = (size_t)a.nt, nc = (size_t)a.nc;
    const float dtvi = __fmul_rn(dt32, in.vi);
    const float sg = in.sg;
    const float dts = -__fmul_rn(dt32, sg);
    const float A32 = __double2float_rn(Ak);
    double qn[NQ];
    bool finite = true;
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
        const float inc = __fmul_rn(dtvi, sum[v]);
        float acc = first ? inc : __fmaf_rn(A32, in.dq[v], inc);
        const double qp = in.qp[v];
        if (sg != 0.0f) acc = __fmaf_rn(dts, f64_to_f32(qp), acc);
        a.dq[v * nc + c] = acc;
        qn[v] = fma(Bk, f32_to_f64(acc), qp);
        a.q[v * nt + c] = qn[v];
        finite = finite && isfinite(sum[v]);
        if (res) a.res[v * nc + c] = f32_to_f64(sum[v]);
    }
    if (!finite) atomicOr(a.flag, 1);
    prims32<D>(a, c, qn, a.primW);
    if (in.ghosts) ghosts_of32<D>(a, c, in.gh, qn, a.primW);
}

// ELL: the fixed-width table, the face list, or (the batch, one copy of whose
// code serves every case) whichever the case has.
enum Entries32 { kEntriesList, kEntriesEll, kEntriesEither };
template <int D, Entries32 ELL, class Sync = NoWait>
__device__ __forceinline__ void update32(const Args<float>& a, int c, double Ak, double Bk, float dt32, int first,
                                         bool res, Sync sync = Sync()) {
    constexpr int W = kEllWidth<D>;
    int code[ELL != kEntriesList ? W : 1];
    if (ELL == kEntriesEll || (ELL == kEntriesEither && a.cfEll)) load_ell<D>(a.cfEll, c, code);
    CellIn32<D> in;
    load_cell32<D>(a, c, first, in, sync);
    float sum[D + 2];
    auto ghosts = [&] {
        if (in.ghosts) in.gh = cell_ghosts<float, D>(a, c);
    };
    if (ELL == kEntriesEll || (ELL == kEntriesEither && a.cfEll)) {
        gather32_ell<D>(a, code, sum, ghosts);
    } else {
        ghosts();
        gather32<D>(a, c, sum);
    }
    apply32<D>(a, c, sum, in, Ak, Bk, dt32, first, res);
}

// A new state: q' = q - q_ref of cell c from a caller's absolute state q
// ([nq][stride] doubles), its primitives and its boundary ghosts' -- the values the preparation pass
// derives from the stored q', from registers.
template <int D>
__device__ __forceinline__ void set_state32(const Args<float>& a, const double* q, int64_t stride, int c) {
    double qp[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) {
        qp[v] = q[(size_t)v * stride + c] - a.qRef[v];
        a.q[(size_t)v * a.nt + c] = qp[v];
    }
    prims32<D>(a, c, qp, a.prim);
    if (a.cellGhosts[c]) ghosts_of32<D>(a, c, cell_ghosts<float, D>(a, c), qp, a.prim);
}

// Calls f(code, o, S, w) for every face entry of cell c in ascending face
// order (code: the face, one's complement where c is N; o: the cell across; the
// face's S and w): through the fixed-width tables (ELL), unrolled so that the
// entries' loads overlap, or the face list. sync() comes after the loads of
// constants (in 2D the geometry too; in 3D it would take 24 registers more)
// and before the first f.
template <int D, bool ELL, class Sync, class F>
__device__ __forceinline__ void for_entries32(const Args<float>& a, int c, Sync sync, F f) {
    if constexpr (ELL) {
        constexpr int W = kEllWidth<D>;
        int code[W], nb[W];
        load_ell<D>(a.cfEll, c, code);
        load_ell<D>(a.cfEllN, c, nb);
        float S[W][D], w[W];
        if constexpr (D == 2) {
#pragma unroll
            for (int k = 0; k < W; ++k)
                if (code[k] != kEllPad) w[k] = load_Sw<D>(a, code[k] >= 0 ? code[k] : ~code[k], S[k]);
        }
        sync();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (code[k] == kEllPad) continue;
            if constexpr (D == 3) w[k] = load_Sw<D>(a, code[k] >= 0 ? code[k] : ~code[k], S[k]);
            f(code[k], nb[k], S[k], w[k]);
        }
    } else {
        sync();
        for (int e = a.cfOff[c]; e < a.cfOff[c + 1]; ++e) {
            const int code = a.cfList[e];
            float S[D];
            const float w = load_Sw<D>(a, code >= 0 ? code : ~code, S);
            f(code, a.cfNbr[e], S, w);
        }
    }
}

// ---------------------------------------------------------------------------
// grad32: Gauss gradients of rho', p' and u' (those of rho, p and u up to
// the reference state's closed-cell sum) for M2AUSM's minmod reconstruction.
// ---------------------------------------------------------------------------
template <int D, bool ELL, class Sync = NoWait>
__device__ __forceinline__ void grad32(const Args<float>& a, int c, Sync sync = Sync()) {
    const RefState32& R = a.ref;
    float G[kGradStride<D>];   // rho, p, u gradients
#pragma unroll
    for (int k = 0; k < kGradStride<D>; ++k) G[k] = 0.0f;
    const float vi = a.volInv32[c];
    Prim32<D> self;
    float cpr;
    auto own_values = [&] {
        sync();
        load_prim<D>(a, c, self);
        cpr = pressure_dev(R, self.r, self.R);
    };
    for_entries32<D, ELL>(a, c, own_values, [&](int code, int o, const float* S, float w) {
        const bool own = code >= 0;   // c is the face's P side
        float uu[D];
        Prim32<D> oth;
        load_prim<D>(a, o, oth);
        const float opr = pressure_dev(R, oth.r, oth.R);
        float so[D];
#pragma unroll
        for (int k = 0; k < D; ++k) {
            so[k] = own ? S[k] * vi : -S[k] * vi;
            uu[k] = own ? interp(w, self.u[k], oth.u[k]) : interp(w, oth.u[k], self.u[k]);
        }
        const float ri = own ? self.r : oth.r, rj = own ? oth.r : self.r;
        const float pi = own ? cpr : opr;
        const float pj = own ? opr : cpr;
        const float rho = interp(w, ri, rj);
        const float p = interp(w, pi, pj);
#pragma unroll
        for (int x = 0; x < D; ++x) {
            G[D + x] += p * so[x];
            G[x] += rho * so[x];
#pragma unroll
            for (int b = 0; b < D; ++b) G[2 * D + b * D + x] += uu[b] * so[x];
        }
    });
    store_vec4<kGradStride<D>>(a.grad + (size_t)c * kGradStride<D>, G);
}

// ---------------------------------------------------------------------------
// vis32: dudx and dTdx from u' and T', sigmaU = (U_inf + u') . tau.
// ---------------------------------------------------------------------------
// LES compiles in the Smagorinsky SGS stress (cases with a.smagC).
template <int D, bool LES, bool ELL, class Sync = NoWait>
__device__ __forceinline__ void vis32(const Args<float>& a, int c, Sync sync = Sync()) {
    float g[D][D], gT[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        gT[k] = 0.0f;
#pragma unroll
        for (int l = 0; l < D; ++l) g[k][l] = 0.0f;
    }
    const float vi = a.volInv32[c];
    const float Rinv = a.ref.Rinv;
    float cu[D], cR;
    auto own_values = [&] {
        sync();
        load_uR<D>(a, c, cu, cR);
    };
    for_entries32<D, ELL>(a, c, own_values, [&](int code, int o, const float* S, float w) {
        const bool own = code >= 0;   // c is the face's P side
        float ou[D], oR, so[D], fU[D];
        load_uR<D>(a, o, ou, oR);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            so[k] = own ? S[k] * vi : -S[k] * vi;
            fU[k] = own ? interp(w, cu[k], ou[k]) : interp(w, ou[k], cu[k]);
        }
        const float fT = (own ? interp(w, cR, oR) : interp(w, oR, cR)) * Rinv;
#pragma unroll
        for (int x = 0; x < D; ++x) {
#pragma unroll
            for (int y = 0; y < D; ++y) g[x][y] += fU[x] * so[y];
            gT[x] += fT * so[x];
        }
    });
    const float mu = a.ref.mu;
    float tau[D][D];
    stress<float, D>(g, mu, tau);
    float U[D], out[kVisVec<D>];
#pragma unroll
    for (int k = 0; k < D; ++k) U[k] = a.ref.U[k] + cu[k];
#pragma unroll
    for (int x = 0; x < D; ++x) {
#pragma unroll
        for (int y = 0; y < D; ++y) out[x * D + y] = g[x][y];
        out[D * D + x] = gT[x];
        out[D * D + D + x] = dotv<float, D>(U, tau[x]);
    }
#pragma unroll
    for (int k = kVisRows<D>; k < kVisVec<D>; ++k) out[k] = 0.0f;
    float* row = a.V + (size_t)c * kVisStride<D, LES>;
    if (LES && a.smagC) {   // Smagorinsky LES: the cell's SGS stress
        float sg[D][D];
        sgs_stress<float, D>(g, a.smagC[c], sg);
#pragma unroll
        for (int x = 0; x < D; ++x)
#pragma unroll
            for (int y = 0; y < D; ++y) {
                const int k = kVisRows<D> + x * D + y;
                if (k < kVisVec<D>) out[k < kVisVec<D> ? k : 0] = sg[x][y];
                else row[k] = sg[x][y];
            }
    }
    store_vec4<kVisVec<D>>(row, out);
}

// d(M) = p5pos(M) - p5neg(M) is, for |M| < 1, the odd polynomial
// (3M - M^3)/2 + 2 alpha M (1 - M^2)^2. Its divided difference
// (d(a) - d(b)) / (a - b), so that d(MN) - d(MP) is formed as a product with
// MN - MP instead of a difference of two O(1) numbers.
__device__ __forceinline__ float p5diff_dd(float a, float b, float alpha) {
    const float s2 = a * a + a * b + b * b;                                   // (a^3 - b^3)/(a - b)
    const float s4 = a * a * a * a + a * a * a * b + a * a * b * b + a * b * b * b + b * b * b * b;
    return 1.5f - 0.5f * s2 + 2.0f * alpha * (1.0f - 2.0f * s2 + s4);
}

// ---------------------------------------------------------------------------
// flux32: perturbation rhs of face f, F(q_f).S - F(q_ref).S, plus the
// viscous terms (linear in the gradients, so unchanged in form).
// ---------------------------------------------------------------------------
// VIS = false compiles the viscous terms out (for callers that know mu = 0).
// EARLYV loads the viscous rows of both cells together with the primitives, so
// the gathers overlap instead of following one another: the stand-alone flux
// kernel (measured with rows of single values in place of the 16-byte parts: 3D
// flux 4.05 -> 3.43 ms per step on the 9.4M-cell wake, whose gathers come from
// HBM; 2 % in 2D, whose gathers hit L2). The batch's kernels, whose registers
// other code already fills, keep the late loads.
//
// face_rhs32_core takes the face's geometry and both cells' primitives as
// values and loadV(Vi, Vj), which fills their viscous rows; `a` gives the
// constants and what only some faces read. So a caller that holds a cell's
// values in registers, or reads them from shared memory (the staged flux
// kernel, flux_staged_fp32.cu), gets the same bits.
template <int D, int SCH, bool VIS, bool LES, bool EARLYV, class A, class LV>
__device__ __forceinline__ void face_rhs32_core(const A& a, int f, int i, int j, bool ghost, const Face32<D>& geo,
                                                const Prim32<D>& pi_, const Prim32<D>& pj_, LV loadV, float* rhs) {
    const RefState32& R = a.ref;
    const float w = geo.w;
    const float* S = geo.S;
    const float ri = pi_.r, rj = pj_.r, Ri = pi_.R, Rj = pj_.R;
    const float *mi = pi_.m, *mj = pj_.m, *ui = pi_.u, *uj = pj_.u;
    constexpr bool needV = VIS || SCH == kSchemeAUSM;
    float Vi[needV ? kVisVec<D> : 1], Vj[needV ? kVisVec<D> : 1];
    const bool visc = VIS && a.ref.mu != 0.0f;
    if (needV && (SCH == kSchemeAUSM || (EARLYV && visc && !ghost))) loadV(Vi, Vj);
    // Face state: linear interpolation for M1, the mid-point for M2 / M2AUSM.
    const float wf = (SCH == kSchemeM1) ? w : 0.5f;
    const float rf = interp(wf, ri, rj);
    const float rinv = 1.0f / (R.rho + rf);
    float mf[D], uf[D];
    float mS = 0.0f, ufS = 0.0f, UrS = 0.0f, mrS = 0.0f;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        mf[k] = interp(wf, mi[k], mj[k]);
        uf[k] = (mf[k] - R.U[k] * rf) * rinv;      // u_f - U_inf with u_f = m_f / rho_f
        mS += mf[k] * S[k];
        ufS += uf[k] * S[k];
        UrS += R.U[k] * S[k];
        mrS += R.m[k] * S[k];
    }
    const float phi = UrS + ufS;                    // u_f . S
    const float Rf = interp(wf, Ri, Rj);
    float pf = pressure_dev(R, rf, Rf);             // rho_f R psi_f - p_ref
    float Hf;                                       // H - H_ref
    if (SCH == kSchemeM1) {
        // H_f = e_f + |u_f|^2/2 + R psi_f with e_f = R psi_f / (gamma - 1)
        float Uu = 0.0f, uu = 0.0f;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            Uu += R.U[k] * uf[k];
            uu += uf[k] * uf[k];
        }
        Hf = R.gh * Rf + Uu + 0.5f * uu;
    } else {
        // mean of the cells' H = gamma/(gamma-1) R psi + |u|^2/2
        float Hi = R.gh * Ri, Hj = R.gh * Rj;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            Hi += R.U[k] * ui[k] + 0.5f * ui[k] * ui[k];
            Hj += R.U[k] * uj[k] + 0.5f * uj[k] * uj[k];
        }
        Hf = 0.5f * (Hi + Hj);
    }
    if constexpr (SCH == kSchemeAUSM) {
        // shock sensor, minmod reconstructions and AUSM+ pressure dissipation
        // (src/cfd_v0.cpp:2288-2339) on the perturbation variables; minmod is
        // invariant under a common shift of both sides.
        const float* pc = a.prim + prim_c<D>((size_t)a.nt);
        const float cavg = 0.5f * (pc[i] + pc[j]);
        float d[D], Gi[kGradStride<D>], Gj[kGradStride<D>];
#pragma unroll
        for (int k = 0; k < D; ++k) d[k] = a.d[(size_t)k * a.nf + f];
        load_vec4<kGradStride<D>>(a.grad + (size_t)i * kGradStride<D>, Gi);
        load_vec4<kGradStride<D>>(a.grad + (size_t)j * kGradStride<D>, Gj);
        float cdiv = 0.0f, ndiv = 0.0f, ccurl = 0.0f, ncurl = 0.0f, unPos = 0.0f, unNeg = 0.0f, dUn = 0.0f,
              norm = 0.0f;
#pragma unroll
        for (int x = 0; x < D; ++x) {
            cdiv += Vi[x * D + x];
            ndiv += Vj[x * D + x];
#pragma unroll
            for (int y = x + 1; y < D; ++y) {
                const float cc = Vi[x * D + y] - Vi[y * D + x];
                const float nn = Vj[x * D + y] - Vj[y * D + x];
                ccurl += cc * cc;
                ncurl += nn * nn;
            }
            const float *gi = Gi + 2 * D + x * D, *gj = Gj + 2 * D + x * D;
            const float uP = minmod_interp<D, true>(ui[x], uj[x], gi, d, w);
            const float uN = minmod_interp<D, false>(ui[x], uj[x], gj, d, w);
            unPos += (R.U[x] + uP) * S[x];
            unNeg += (R.U[x] + uN) * S[x];
            dUn += (uN - uP) * S[x];
            norm += S[x] * S[x];
        }
        float ct = -(cdiv / sqrtf(cdiv * cdiv + ccurl + 4e-2f));
        ct = (ct < 0.0f) ? 0.0f : ct;
        float nt_ = -(ndiv / sqrtf(ndiv * ndiv + ncurl + 4e-2f));
        nt_ = (nt_ < 0.0f) ? 0.0f : nt_;
        const float theta = 0.5f * (ct + nt_);
        const float pi = pressure_dev(R, ri, Ri), pj = pressure_dev(R, rj, Rj);
        const float *gri = Gi, *grj = Gj, *gpi = Gi + D, *gpj = Gj + D;
        const float rhoPos = R.rho + minmod_interp<D, true>(ri, rj, gri, d, w);
        const float rhoNeg = R.rho + minmod_interp<D, false>(ri, rj, grj, d, w);
        const float pPos = minmod_interp<D, true>(pi, pj, gpi, d, w);    // p - p_ref
        const float pNeg = minmod_interp<D, false>(pi, pj, gpj, d, w);
        const float Msq = (unPos * unPos + unNeg * unNeg) / (2.0f * cavg * cavg * norm);
        const float sc = 1.0f / (sqrtf(norm) * cavg);
        const float MPos = unPos * sc, MNeg = unNeg * sc;
        const float Minf = 0.2f;
        float mm = (Msq < Minf * Minf) ? Minf * Minf : Msq;
        mm = (mm < 1.0f) ? mm : 1.0f;
        const float M0 = sqrtf(mm);
        const float fa = M0 * (2.0f - M0);
        const float alpha = 3.0f * (5.0f * fa * fa - 4.0f) / 16.0f;
        const float ppP = p5pos(MPos, alpha), pnP = p5neg(MPos, alpha);
        const float ppN = p5pos(MNeg, alpha), pnN = p5neg(MNeg, alpha);
        const float dN = ppN - pnN, dP = ppP - pnP;
        const float dNdP = (fabsf(MPos) < 1.0f && fabsf(MNeg) < 1.0f) ? dUn * sc * p5diff_dd(MNeg, MPos, alpha)
                                                                       : dN - dP;
        // pNeg dN - pPos dP with p = p_ref + p'
        const float phalf = R.p * dNdP + pNeg * dN - pPos * dP;
        const float pu = -0.75f * ppP * pnN * (rhoPos + rhoNeg) * cavg * fa * dUn;
        pf += theta * (pu - 0.5f * phalf);
    }
    // F(q_f).S - F(q_ref).S
    rhs[0] = -mS;
#pragma unroll
    for (int k = 0; k < D; ++k) rhs[k + 1] = -(R.m[k] * ufS + mf[k] * phi + pf * S[k]);
    rhs[D + 1] = -(mS * R.H + (mrS + mS) * Hf);

    // Viscous face terms (src/cfd_v0.cpp:2682-2796), as in the FP64 kernel.
    const float mu = a.ref.mu;
    if (visc) {
        const float Rinv = a.ref.Rinv;
        const float Ti = Ri * Rinv, Tj = Rj * Rinv;   // T - T_ref
        const float lapc = geo.lapc;
        const float* Kf = geo.K;
        float g[D][D], gT[D], sU[D];
        if (!ghost) {
            if (!EARLYV && SCH != kSchemeAUSM) loadV(Vi, Vj);
#pragma unroll
            for (int x = 0; x < D; ++x) {
#pragma unroll
                for (int y = 0; y < D; ++y) g[x][y] = interp(w, Vi[x * D + y], Vj[x * D + y]);
                gT[x] = interp(w, Vi[D * D + x], Vj[D * D + x]);
                sU[x] = interp(w, Vi[D * D + D + x], Vj[D * D + D + x]);
            }
        } else {
            const float dinv = a.dinv[f];
            float dn[D], tau[D][D], Uf[D];
#pragma unroll
            for (int k = 0; k < D; ++k) dn[k] = a.dnorm[(size_t)k * a.nf + f];
#pragma unroll
            for (int x = 0; x < D; ++x) {
#pragma unroll
                for (int y = 0; y < D; ++y) g[x][y] = (uj[x] - ui[x]) * dn[y] * dinv;
                gT[x] = (Tj - Ti) * dn[x] * dinv;
                Uf[x] = R.U[x] + interp(w, ui[x], uj[x]);
            }
            stress<float, D>(g, mu, tau);
#pragma unroll
            for (int x = 0; x < D; ++x) sU[x] = dotv<float, D>(Uf, tau[x]);
        }
        float tr = g[0][0];
#pragma unroll
        for (int x = 1; x < D; ++x) tr += g[x][x];
        const float dsum = -(mu * 2.0f / 3.0f) * tr;
        const float kc = a.ref.kcond;
#pragma unroll
        for (int x = 0; x < D; ++x) {
            float gtS = g[0][x] * S[0];
#pragma unroll
            for (int y = 1; y < D; ++y) gtS += g[y][x] * S[y];
            rhs[x + 1] += mu * gtS + dsum * S[x] + mu * (lapc * (uj[x] - ui[x]) + dotv<float, D>(Kf, g[x]));
        }
        rhs[D + 1] += dotv<float, D>(sU, S) + kc * (lapc * (Tj - Ti) + dotv<float, D>(Kf, gT));
        if constexpr (LES) {
            if (a.smagC && !ghost) {   // Smagorinsky LES, as in the FP64 kernel
                const float* si = a.V + (size_t)i * kVisStride<D, true> + kVisRows<D>;
                const float* sj = a.V + (size_t)j * kVisStride<D, true> + kVisRows<D>;
#pragma unroll
                for (int x = 0; x < D; ++x) {
                    float s = 0.0f;
#pragma unroll
                    for (int y = 0; y < D; ++y) s += interp(w, si[x * D + y], sj[x * D + y]) * S[y];
                    rhs[x + 1] += s;
                }
            }
        }
    }
}

template <int D, int SCH, bool VIS = true, bool LES = false, bool EARLYV = false, class Sync = NoWait>
__device__ __forceinline__ void flux32(const Args<float>& a, int f, Sync sync = Sync()) {
    Face32<D> geo;
    Prim32<D> pi, pj;
    int i, j;
    bool ghost;
    load_face<D>(a, f, geo, i, j, ghost);
    sync();
    load_prim<D>(a, i, pi);
    load_prim<D>(a, j, pj);
    float rhs[D + 2];
    face_rhs32_core<D, SCH, VIS, LES, EARLYV>(
        a, f, i, j, ghost, geo, pi, pj,
        [&](float* Vi, float* Vj) {
            load_vis<D, LES>(a, i, Vi);
            load_vis<D, LES>(a, j, Vj);
        },
        rhs);
    store_flux<D>(a, f, rhs);
}

// ---------------------------------------------------------------------------
// flux32_cell: the rhs of the faces cell c owns (it is their P side), one
// after another in face order. The cell's own primitive and viscous rows are
// read once, into registers, for all its faces (a face-per-thread kernel
// reads them once per face); the cell across each face is read per face, its
// index one face ahead. The rhs is face_rhs32_core's, so it keeps flux32's
// bits. M1 / M2 without the LES terms.
// ---------------------------------------------------------------------------
template <int D, int SCH, class Sync = NoWait>
__device__ __forceinline__ void flux32_cell(const Args<float>& a, int c, Sync sync = Sync()) {
    static_assert(SCH != kSchemeAUSM, "the cell-centred flux holds no sound speed or gradients");
    const int f0 = a.fOwn[c], f1 = a.fOwn[c + 1];
    if (f0 >= f1) return;
    const bool vis = a.ref.mu != 0.0f;
    int nn = a.fN[f0];
    sync();
    Prim32<D> self;
    load_prim<D>(a, c, self);
    float Vc[kVisVec<D>];
    if (vis) load_vis<D, false>(a, c, Vc);
    for (int f = f0; f < f1; ++f) {
        const int n = nn;
        if (f + 1 < f1) nn = a.fN[f + 1];
        const int j = n & 0x7fffffff;
        const bool ghost = n < 0;
        Face32<D> geo;
        const float4 g0 = a.fG0[f], g1 = a.fG1[f];
        geo.S[0] = g0.x;
        geo.S[1] = g0.y;
        geo.K[0] = g1.x;
        geo.K[1] = g1.y;
        if constexpr (D == 2) {
            geo.w = g0.z;
            geo.lapc = g0.w;
        } else {
            geo.S[2] = g0.z;
            geo.w = g0.w;
            geo.K[2] = g1.z;
            geo.lapc = g1.w;
        }
        Prim32<D> oth;
        load_prim<D>(a, j, oth);
        float rhs[D + 2];
        face_rhs32_core<D, SCH, true, false, true>(
            a, f, c, j, ghost, geo, self, oth,
            [&](float* Vi, float* Vj) {
                load_vis<D, false>(a, j, Vj);
#pragma unroll
                for (int k = 0; k < kVisVec<D>; ++k) Vi[k] = Vc[k];
            },
            rhs);
        store_flux<D>(a, f, rhs);
    }
}

// ---------------------------------------------------------------------------
// fluxupdate32: the rhs of every face of cell c, evaluated by the cell itself
// (each face is evaluated by both of its cells, from the face's own data, so
// both get the bits flux32 stores), summed in ascending face order as the
// update's gather sums the stored values, then the update of apply32. The
// face rhs never reaches memory and a stage needs one kernel less; the next
// stage's primitives go to a.primW, the other of two buffers (the cells of
// this launch still read a.prim). The cell's own values are read once.
// ---------------------------------------------------------------------------
template <int D, int SCH, bool VIS, bool ELL, class Sync = NoWait>
__device__ __forceinline__ void fluxupdate32(const Args<float>& a, int c, double Ak, double Bk, float dt32, int first,
                                             bool res, Sync sync = Sync()) {
    constexpr int NQ = D + 2;
    CellIn32<D> in;
    Prim32<D> self;
    constexpr bool needV = VIS || SCH == kSchemeAUSM;
    float Vc[needV ? kVisVec<D> : 1];
    auto own_values = [&] {
        load_cell32<D>(a, c, first, in, sync);
        load_prim<D>(a, c, self);
        if constexpr (needV) load_vis<D, false>(a, c, Vc);
        if (in.ghosts) in.gh = cell_ghosts<float, D>(a, c);
    };
    float sum[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) sum[v] = 0.0f;
    for_entries32<D, ELL>(a, c, own_values, [&](int code, int o, const float* S, float w) {
        const bool own = code >= 0;
        const int f = own ? code : ~code;
        Face32<D> geo;
        bool ghost = false;
        if constexpr (VIS) {
            int i, j;
            load_face<D>(a, f, geo, i, j, ghost);
        } else {   // S and w suffice without the viscous terms
#pragma unroll
            for (int k = 0; k < D; ++k) geo.S[k] = S[k];
            geo.w = w;
        }
        Prim32<D> oth, pi, pj;
        load_prim<D>(a, o, oth);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            pi.m[k] = own ? self.m[k] : oth.m[k];
            pj.m[k] = own ? oth.m[k] : self.m[k];
            pi.u[k] = own ? self.u[k] : oth.u[k];
            pj.u[k] = own ? oth.u[k] : self.u[k];
        }
        pi.r = own ? self.r : oth.r;
        pj.r = own ? oth.r : self.r;
        pi.R = own ? self.R : oth.R;
        pj.R = own ? oth.R : self.R;
        float r[NQ];
        face_rhs32_core<D, SCH, VIS, false, true>(
            a, f, own ? c : o, own ? o : c, ghost, geo, pi, pj,
            [&](float* Vi, float* Vj) {
                float Vo[kVisVec<D>];
                load_vis<D, false>(a, o, Vo);
#pragma unroll
                for (int k = 0; k < kVisRows<D>; ++k) {
                    Vi[k] = own ? Vc[needV ? k : 0] : Vo[k];
                    Vj[k] = own ? Vo[k] : Vc[needV ? k : 0];
                }
            },
            r);
#pragma unroll
        for (int v = 0; v < NQ; ++v) sum[v] += own ? r[v] : neg_bits(r[v]);
    });
    apply32<D>(a, c, sum, in, Ak, Bk, dt32, first, res);
}

}  // namespace dev
}  // namespace lfm
