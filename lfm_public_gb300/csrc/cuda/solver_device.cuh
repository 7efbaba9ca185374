// Device helpers shared by the FP64 and FP32-bulk time-step kernels.
#pragma once

#include "solver_kernels.cuh"

namespace lfm {
namespace dev {

#define LFM_GLOBAL_ID() ((int)(blockIdx.x * blockDim.x + threadIdx.x))

// Programmatic dependent launch. The kernels of a time step are launched so
// that a kernel's blocks may become resident once every block of its
// predecessor has passed its own wait, instead of after the predecessor has
// drained; each first loads what no kernel of the step writes (face lists,
// geometry, cell constants) and then waits here for the predecessor's results.
// Since a kernel releases its successor only after its wait, at most two
// kernels of the chain overlap, and everything before the predecessor is
// complete. Without it each kernel of a 2D case spends 2 to 4 of its 8 to 15 us
// launching, loading indices and draining. Args::pdl says which cases launch
// their kernels that way (pdl_pays, solver_launch.h); one launched plainly all
// the same passes at once.
struct PdlWait {
    int pdl;
    __device__ __forceinline__ void operator()() const {
        if (!pdl) return;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
};
// The first kernel of a chain has nothing to wait for.
struct PdlRelease {
    int pdl;
    __device__ __forceinline__ void operator()() const {
        if (pdl) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
};
// For device functions called inside one kernel (the batch, the tiles).
struct NoWait {
    __device__ __forceinline__ void operator()() const {}
};

template <typename T>
__device__ __forceinline__ T interp(T w, T a, T b) {
    return w * a + (T(1) - w) * b;
}

// 1/x in FP64 from the series 1/x = y / (1 - e) = y (1 + e + e^2 + ...),
// e = 1 - xy, with y the single-precision reciprocal approximation of x
// truncated to binary32 (PTX rcp.approx.ftz.f32; |e| is at most about 2^-22
// with the truncation): the terms up to e^2 leave a relative error of e^3, far
// below the rounding of the last operation, for three FP64 FMAs -- GB300
// issues about two FP64 instructions per clock per SM, and a full-precision
// division takes several more. Values outside binary32's normal range take
// the division.
__device__ __forceinline__ double rcp64(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7ffu) - 896;   // binary32 biased exponent
    if (ex < 2 || ex > 252) return 1.0 / x;
    const unsigned fb = ((unsigned)(b >> 32) & 0x80000000u) | ((unsigned)ex << 23) | (unsigned)((b >> 29) & 0x7fffffu);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
    // widen r exactly: rebias its (normal) exponent, move its mantissa up
    const unsigned rb = __float_as_uint(r);
    double y = __longlong_as_double((long long)(((unsigned long long)(rb & 0x80000000u) << 32) |
                                                ((unsigned long long)(((rb >> 23) & 0xffu) + 896u) << 52) |
                                                ((unsigned long long)(rb & 0x7fffffu) << 29)));
    double e = fma(-x, y, 1.0);
    e = fma(e, e, e);
    return fma(y, e, y);
}

// -x and isfinite(x) of an FP64 value on the integer pipe (a sign-bit flip;
// an exponent test), leaving GB300's FP64 pipe to the arithmetic.
__device__ __forceinline__ double neg_bits(double x) {
    return __hiloint2double(__double2hiint(x) ^ (int)0x80000000u, __double2loint(x));
}
__device__ __forceinline__ float neg_bits(float x) { return __uint_as_float(__float_as_uint(x) ^ 0x80000000u); }
__device__ __forceinline__ bool finite_bits(double x) {
    return ((unsigned)__double2hiint(x) & 0x7ff00000u) != 0x7ff00000u;
}

// interp with the weight of N given (1 - w, precomputed per face).
template <typename T>
__device__ __forceinline__ T interp2(T w, T wN, T a, T b) {
    return w * a + wN * b;
}

template <typename T, int D>
__device__ __forceinline__ T dotv(const T* a, const T* b) {
    T s = a[0] * b[0];
#pragma unroll
    for (int k = 1; k < D; ++k) s += a[k] * b[k];
    return s;
}

// Deviatoric stress of a velocity gradient g (row a = gradient of u_a), in the
// reference's evaluation order (src/cfd_v0.cpp:1813-1822).
template <typename T, int D>
__device__ __forceinline__ void stress(const T g[D][D], T mu, T tau[D][D]) {
#pragma unroll
    for (int a = 0; a < D; ++a) {
        tau[a][a] = T(2) * g[a][a];
#pragma unroll
        for (int b1 = a + 1; b1 < D + a; ++b1) {
            const int b = b1 % D;
            tau[a][b] = mu * (g[a][b] + g[b][a]);
            tau[a][a] -= g[b][b];
        }
        tau[a][a] *= T(2.0 / 3.0) * mu;
    }
}

// Smagorinsky subgrid stress added to a cell's tauMC (calc_VIS_Smagorinsky,
// src/cfd_v0.cpp:1675-1695): -C |S| S_ab + (C |S| div u / 3) delta_ab with
// S the symmetric part of the velocity gradient g, |S| = sqrt(2 S_ab S_ab)
// and C = -2 (0.16 Delta)^2 the cell's model constant.
template <typename T, int D>
__device__ __forceinline__ void sgs_stress(const T g[D][D], T C, T out[D][D]) {
    T sm = T(0), divu = T(0);
#pragma unroll
    for (int x = 0; x < D; ++x) {
#pragma unroll
        for (int y = 0; y < D; ++y) {
            const T s = T(0.5) * (g[x][y] + g[y][x]);
            sm += s * s;
        }
        divu += g[x][x];
    }
    sm = sqrt(T(2) * sm);
    const T cs = C * sm;
#pragma unroll
    for (int x = 0; x < D; ++x) {
#pragma unroll
        for (int y = 0; y < D; ++y) out[x][y] = -(cs * (T(0.5) * (g[x][y] + g[y][x])));
        out[x][x] += cs * divu / T(3);
    }
}

// Rows of the per-cell viscous array: dudx (D x D), dTdx, sigmaU, then with
// Smagorinsky LES the SGS stress (D x D).
template <int D>
constexpr int kVisRows = D * D + 2 * D;

// Minmod-limited face reconstruction from the upwind side (calc_r and
// interp_minmod, api/cfdv0_solver.h:310-370), FP32: FROMP from P with its
// gradient, else from N. The limiter 2 (gradcf / gradf) - 1, held to [0, 1], is
// 1 or 0 unless the quotient is between 1/2 and 1, which the comparisons tell
// exactly (the reference's largest quotient, 1000, lies beyond): only then it is
// divided. (|gradf| is 0 or at least 2^-123, so its half is exact.) The flux of
// a 331 x 217 M2AUSM cylinder executed 1200 instructions a face, many of them
// the long form of a division, of the very small differences of a uniform flow:
// 53 -> 36 us a step from uniform flow, 1 % of the step in a disturbed one; with
// branches in place of the selects that one was 4 % slower (GB300). Values that
// are no numbers come to the quotient.
template <int D, bool FROMP>
__device__ __forceinline__ float minmod_interp(float cp, float ap, const float* grad, const float* d, float w) {
    const float gradf = ap - cp + 1.0e-30f;
    float gradcf = d[0] * grad[0];
#pragma unroll
    for (int k = 1; k < D; ++k) gradcf += d[k] * grad[k];
    // the quotient's sign moved to its upper part
    const float af = fabsf(gradf);
    const float gc = __uint_as_float(__float_as_uint(gradcf) ^ (__float_as_uint(gradf) & 0x80000000u));
    const bool zero = gc < 0.5f * af, fixed = zero || gc >= af;   // 1 / 1 in a fixed one's place
    float lim = 2.0f * ((fixed ? 1.0f : gc) / (fixed ? 1.0f : af)) - 1.0f;
    if (zero) lim = 0.0f;
    const float weight = FROMP ? lim * w + (1.0f - lim) : lim * w;
    return weight * cp + (1.0f - weight) * ap;
}

// Comparisons of a double on the integer pipe, from its upper word (an FP64
// comparison takes an FP64 issue slot). Not a number is neither.
__device__ __forceinline__ bool neg64(double x) {   // x < 0, or -0
    return (unsigned)__double2hiint(x) - 0x80000000u <= 0x7ff00000u;
}
__device__ __forceinline__ bool atleast1(double x) {   // x >= 1
    return (unsigned)__double2hiint(x) - 0x3ff00000u <= 0x40000000u;
}
__device__ __forceinline__ double pos_part(double x) { return neg64(x) ? 0.0 : x; }

// 1/sqrt(x) in FP64, as rcp64: from the single-precision approximation y of
// the truncated argument, 1/sqrt(x) = y (1 - e)^(-1/2) with e = 1 - x y^2, the
// terms up to e^2 (PTX rsqrt.approx.ftz.f32).
__device__ __forceinline__ double rsqrt64(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(b >> 52) - 896;   // with the sign: negative numbers are out of range
    if (ex < 2 || ex > 252) return rsqrt(x);
    const unsigned fb = ((unsigned)ex << 23) | ((unsigned)(b >> 29) & 0x7fffffu);
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
    const unsigned rb = __float_as_uint(r);
    const double y = __longlong_as_double((long long)(((unsigned long long)((rb >> 23) + 896u) << 52) |
                                                      ((unsigned long long)(rb & 0x7fffffu) << 29)));
    const double e = fma(-x * y, y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// Both limited reconstructions of a face value in FP64 (minmod_interp with
// flux = +1 from P's gradient and -1 from N's): the two share the difference
// across the face, so one reciprocal serves both, and the weights
// lim w + (1 - lim)(1 +- 1) / 2 multiply out to an increment lim (1 - w) from
// P and lim w from N. The limiter is 1 or 0 wherever |gradcf| > |gradf|, so the
// case of a quotient too large to form (minmod_interp's 1000; 0 / 0 counts as one)
// is told by the exponents. With the sensor's and the Mach numbers' divisions replaced alike
// the M2AUSM flux of a 331 x 217 cylinder took 413 us a step where it took 681,
// and 301 with the comparisons on the integer pipe, the sensor's roots by
// rsqrt64 and the pressure polynomials by p5half (GB300).
template <int D>
__device__ __forceinline__ void minmod_pair(double cp, double ap, const double* gradP, const double* gradN,
                                            const double* d, double w, double wN, double& fromP, double& fromN) {
    const double df = ap - cp;
    const double gradf = df + 1.0e-30;
    const double rf = rcp64(gradf);
    const unsigned hg = (unsigned)__double2hiint(gradf) & 0x7fffffffu;
    const unsigned hf = hg ? hg + 0x00100000u : 0u;   // beyond |gradf|; any value beside 0
    double lim[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const double* grad = s ? gradN : gradP;
        double gradcf = d[0] * grad[0];
#pragma unroll
        for (int k = 1; k < D; ++k) gradcf += d[k] * grad[k];
        const int hc = __double2hiint(gradcf);
        double r = fma(2.0, gradcf * rf, -1.0);
        if (hf <= 0x7ff00000u && ((unsigned)hc & 0x7fffffffu) - hf <= 0x7ff00000u - hf)
            r = ((unsigned)hc > 0x80000000u) != (__double2hiint(gradf) < 0) ? 0.0 : 1.0;   // -0 is not negative
        r = atleast1(r) ? 1.0 : r;
        lim[s] = pos_part(r);
    }
    fromP = fma(lim[0] * wN, df, cp);
    fromN = fma(-(lim[1] * w), df, ap);
}

// Half the difference of the AUSM+ pressure polynomials below, which add up to
// 1: p5pos = 1/2 + p5half, p5neg = 1/2 - p5half, for |M| < 1
// M (3/4 - M^2 / 4 + alpha (1 - M^2)^2).
__device__ __forceinline__ double p5half(double M, double alpha) {
    const double M2 = M * M, t = 1.0 - M2;
    const double s = M * fma(alpha, t * t, fma(-0.25, M2, 0.75));
    const int h = __double2hiint(M);
    // |M| from 1 up to the largest number: one side alone
    if (((unsigned)h & 0x7fffffffu) - 0x3ff00000u < 0x40000000u) return h < 0 ? -0.5 : 0.5;
    return s;
}

// AUSM+ fifth-order pressure polynomials (p5Pos / p5Neg, src/cfd_v0.cpp:1863-1895).
template <typename T>
__device__ __forceinline__ T p5pos(T M, T alpha) {
    const T M2Pos = T(0.25) * (M + T(1)) * (M + T(1));
    const T M2Neg = T(-0.25) * (M - T(1)) * (M - T(1));
    if (fabs(M) < T(1)) return M2Pos * ((T(2) - M) - T(16) * alpha * M * M2Neg);
    return T(0.5) * (M + fabs(M)) / M;
}

template <typename T>
__device__ __forceinline__ T p5neg(T M, T alpha) {
    const T M2Pos = T(0.25) * (M + T(1)) * (M + T(1));
    const T M2Neg = T(-0.25) * (M - T(1)) * (M - T(1));
    if (fabs(M) < T(1)) return M2Neg * ((T(-2) - M) + T(16) * alpha * M * M2Pos);
    return T(0.5) * (M - fabs(M)) / M;
}

// x component of the area vector of face f.
__device__ __forceinline__ double face_sx(const Args<double>& a, int f) { return a.S[f]; }
__device__ __forceinline__ double face_sx(const Args<float>& a, int f) { return (double)a.fG0[f].x; }

// Boundary ghosts (set_boundary_conditions, src/cfd_v0.cpp:1009-1221), state
// and primitives from those of the interior cell (FP64). The reference's
// expressions (TInt = pInt / (R rhoInt), rhoExt = rhoInt TInt / TInf, rhoExt EExt
// with EExt = p / (rhoExt (gamma - 1)) + |u|^2 / 2, then 1/rhoExt, uExt and
// p/rhoExt) with the divisions that cancel left out and those by constants
// turned into host-side factors.
//
// What counts is the depth of the chain: it is the last serial part of a
// boundary cell's update, an FP64 operation takes 65 cycles from operand to
// result, and the update kernel of a small case waits for the cell at a corner,
// which has two ghosts. What depends on the interior cell is therefore formed
// once for all its ghosts (ghost_in), and a ghost takes at most three operations
// more: its primitives follow from the interior's, not from its own state.
// Measured on GB300 against a state and primitives per ghost, us a step: 48 x 48
// FP64 vortex 45.0 -> 40.9, 256 x 256 vortex FP64 106.4 -> 100.3 and FP32-bulk
// 43.0 -> 36.8 (16 of which the ghosts took, in a copy without them).
template <int D>
struct GhostIn {
    double rho, rinv, m[D], u[D], E;
    double p, pinv, R, ke;   // pressure, its reciprocal, R psi, |u|^2 / 2
};
template <int D>
struct GhostState {
    double q[D + 2], rinv, u[D], R;
};

template <typename T, int D>
__device__ __forceinline__ GhostIn<D> ghost_in(const Args<T>& a, const double* qi) {
    GhostIn<D> g;
    g.rho = qi[0];
    g.E = qi[D + 1];
    g.rinv = rcp64(qi[0]);
    double s = 0.0;   // rho |u|^2
#pragma unroll
    for (int k = 0; k < D; ++k) {
        g.m[k] = qi[k + 1];
        g.u[k] = qi[k + 1] * g.rinv;
        s = k ? fma(g.m[k], g.u[k], s) : g.m[0] * g.u[0];
    }
    const double e = fma(-0.5, s, g.E);
    g.p = e * a.gm1;
    g.pinv = rcp64(g.p);
    g.R = e * (a.gm1 * g.rinv);
    g.ke = s * (0.5 * g.rinv);
    return g;
}

// One sequence for the three kinds, operands selected by kind (on the integer
// pipe): the boundary cells of a warp alternate between inlet and outlet on a
// row-ordered mesh, and branches would run one after another. A wall mirrors the
// momentum, an inlet takes pInt, TInf, UInf, an outlet pInf, TInt, uInt.
template <typename T, int D>
__device__ __forceinline__ void ghost_state(const Args<T>& a, int g, int kind, const GhostIn<D>& in, GhostState<D>& o) {
    if (kind < 1 || kind > 4) {
        // Patches without a boundary condition keep a zero ghost state, as
        // in the reference (src/cfd_v0.cpp:406-416): its primitives are not finite.
#pragma unroll
        for (int v = 0; v < D + 2; ++v) o.q[v] = 0.0;
        o.rinv = rcp64(o.q[0]);
#pragma unroll
        for (int k = 0; k < D; ++k) o.u[k] = o.q[k + 1] * o.rinv;
        o.R = o.q[D + 1] * o.rinv;
        return;
    }
    const bool wall = kind == 1;
    bool inlet = kind == 2;
    if (kind == 4) inlet = face_sx(a, a.gFace[g]) <= 0.0;  // free stream along +x enters
    // rho: p / (R TInf) | rho pInf / p | rho;  1/rho: R TInf / p | p / (rho pInf) | 1/rho
    o.q[0] = (wall ? in.rho : inlet ? in.p : in.rho * a.pInf) * (wall ? 1.0 : inlet ? a.RTInv : in.pinv);
    o.rinv = (wall ? in.rinv : inlet ? a.RT : in.rinv * a.pInfInv) * (wall ? 1.0 : inlet ? in.pinv : in.p);
    const double Rout = a.pInf * o.rinv;
    o.R = wall ? in.R : inlet ? a.RT : Rout;
    const double e = fma(inlet ? a.keInf : in.ke, o.q[0], (inlet ? in.p : a.pInf) * a.gm1Inv);
    o.q[D + 1] = wall ? in.E : e;
#pragma unroll
    for (int k = 0; k < D; ++k) {
        o.u[k] = wall ? neg_bits(in.u[k]) : inlet ? a.UInf[k] : in.u[k];
        const double m = o.q[0] * o.u[k];
        o.q[k + 1] = wall ? neg_bits(in.m[k]) : m;
    }
}

// The state alone, of ghost g from its interior cell's state qi.
template <typename T, int D>
__device__ __forceinline__ void ghost_bc(const Args<T>& a, int g, const double* qi, double* qv) {
    GhostState<D> o;
    ghost_state<T, D>(a, g, a.gKind[g], ghost_in<T, D>(a, qi), o);
#pragma unroll
    for (int v = 0; v < D + 2; ++v) qv[v] = o.q[v];
}

// FP64 path: the primitives every face reads (1/rho, u, R psi = p/rho, c) of
// cell, ghost or halo t from its conservative state qv (compute_Rpsi,
// api/cfdv0_solver.h:252-261).
template <int D>
__device__ __forceinline__ void prims64(const Args<double>& a, int t, const double* qv) {
    const size_t nt = (size_t)a.nt;
    const double rinv = rcp64(qv[0]);
    double u[D], s = 0.0;   // s = rho |u|^2
#pragma unroll
    for (int k = 0; k < D; ++k) {
        u[k] = qv[k + 1] * rinv;
        s = k ? fma(qv[k + 1], u[k], s) : qv[1] * u[0];
    }
    const double Rpsi = fma(-0.5, s, qv[D + 1]) * (a.gm1 * rinv);
    a.prim[t] = rinv;
#pragma unroll
    for (int k = 0; k < D; ++k) a.prim[(size_t)(1 + k) * nt + t] = u[k];
    a.prim[(size_t)(D + 1) * nt + t] = Rpsi;
    if (a.primC) a.prim[(size_t)(D + 2) * nt + t] = sqrt(a.gamma * Rpsi);   // read by M2AUSM only
}

// The boundary ghosts of a cell with boundary faces. A ghost is only ever across
// a face of its own cell, so the neighbour column alone names it; the entries of
// an ordinary cell are loaded together, where following the face list to the
// face's N side costs two dependent loads per face. The first two ghosts (a corner
// has two) and their kinds are loaded ahead of the cell's new state, so
// that the update's last serial part is arithmetic alone.
struct CellGhosts {
    int j[2] = {-1, -1}, kind[2] = {0, 0};   // the first two ghosts and their kinds
    int count = 0;
};

template <typename T, int D>
__device__ __forceinline__ int entry_cell(const Args<T>& a, int c, int k) {   // the cell across entry k, -1 past the last
    if constexpr (sizeof(T) == sizeof(float)) {
        if (a.cfEllN) return k < kEllWidth<D> ? a.cfEllN[(size_t)c * kEllWidth<D> + k] : -1;
    }
    return a.cfOff[c] + k < a.cfOff[c + 1] ? a.cfNbr[a.cfOff[c] + k] : -1;
}

template <typename T, int D>
__device__ __forceinline__ CellGhosts cell_ghosts(const Args<T>& a, int c) {
    constexpr int W = kEllWidth<D>;
    CellGhosts g;
    int nb[W];
#pragma unroll
    for (int k = 0; k < W; ++k) nb[k] = entry_cell<T, D>(a, c, k);
    auto found = [&](int j) {
        if (j < a.nc || j >= a.nc + a.ng) return;
        if (g.count == 0) g.j[0] = j;
        if (g.count == 1) g.j[1] = j;
        ++g.count;
    };
#pragma unroll
    for (int k = 0; k < W; ++k) found(nb[k]);
    if (nb[W - 1] >= 0)   // a cell of more faces
        for (int k = W, j; (j = entry_cell<T, D>(a, c, k)) >= 0; ++k) found(j);
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (g.count > k) g.kind[k] = a.gKind[g.j[k] - a.nc];
    return g;
}

// f(j, kind) for each of them: the first two, then (a cell with more boundary
// faces) the others in entry order. Faces may share a ghost, so that fewer than
// `count` are left: the walk ends with the entries. (Telling them by their place
// among the ghosts passed takes two counters more, and the batch's update phases
// spilled 8 bytes more.)
template <typename T, int D, class F>
__device__ __forceinline__ void for_ghosts(const Args<T>& a, int c, const CellGhosts& g, F f) {
    int left = g.count;
#pragma unroll 1
    for (int k = 0; left > 0; ++k) {
        int j = k == 0 ? g.j[0] : g.j[1], kind = k == 0 ? g.kind[0] : g.kind[1];
        if (k >= 2) {
            j = entry_cell<T, D>(a, c, k - 2);
            if (j < 0) break;   // past the last entry
            if (j < a.nc || j >= a.nc + a.ng || j == g.j[0] || j == g.j[1]) continue;
            kind = a.gKind[j - a.nc];
        }
        f(j, kind);
        --left;
    }
}

// FP64 path: state and primitives of ghost g into the stored arrays.
template <int D>
__device__ __forceinline__ void ghost64(const Args<double>& a, int g, int kind, const GhostIn<D>& in) {
    const size_t nt = (size_t)a.nt, t = (size_t)(a.nc + g);
    GhostState<D> o;
    ghost_state<double, D>(a, g, kind, in, o);
#pragma unroll
    for (int v = 0; v < D + 2; ++v) a.q[v * nt + t] = o.q[v];
    a.prim[t] = o.rinv;
#pragma unroll
    for (int k = 0; k < D; ++k) a.prim[(1 + k) * nt + t] = o.u[k];
    a.prim[(D + 1) * nt + t] = o.R;
    if (a.primC) a.prim[(D + 2) * nt + t] = sqrt(a.gamma * o.R);
}

// FP64 path: the states and primitives of the boundary ghosts of cell c from
// its conservative state qc (those k_prep computes for the next stage).
template <int D>
__device__ __forceinline__ void ghosts_of64(const Args<double>& a, int c, const CellGhosts& g, const double* qc) {
    const GhostIn<D> in = ghost_in<double, D>(a, qc);
    for_ghosts<double, D>(a, c, g, [&](int j, int kind) { ghost64<D>(a, j - a.nc, kind, in); });
}

// FP64 path: gather of the face rhs of cell c, sponge source and low-storage
// RK update (src/cfd_v0.cpp:2800-2822). The rhs are summed in ascending face
// order (the order in which the reference's scatter reaches the cell); the
// sum is the cell residual RES. PRIM: the cell also writes the next stage's
// primitives from the registers it holds, and the next stage's
// states and primitives of its boundary ghosts -- a ghost depends on its
// interior cell only -- so that no preparation pass runs between the stages.
template <typename T, int D, bool RES, bool PRIM = false, class Sync = NoWait>
__device__ __forceinline__ void update_cell(const Args<T>& a, int c, double Ak, double Bk, double dt, int first,
                                            Sync sync = Sync()) {
    constexpr int NQ = D + 2;
    const size_t nt = (size_t)a.nt, nf = (size_t)a.nf, nc = (size_t)a.nc;
    constexpr int W = kEllWidth<D>;
    const int e0 = a.cfOff[c], e1 = a.cfOff[c + 1];
    int code[W];
#pragma unroll
    for (int k = 0; k < W; ++k) code[k] = e0 + k < e1 ? a.cfList[e0 + k] : kEllPad;
    const double vi = a.volInv[c], sg = a.sponge[c];
    // (ng > 0 first: a uniform branch around the load, without which the 2D kernel
    // keeps 79 registers for 72, six blocks an SM for seven)
    const bool ghosts = PRIM && a.ng > 0 && a.cellGhosts[c];
    CellGhosts gh;
    sync();
    double qv[NQ], dq[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
        qv[v] = a.q[v * nt + c];
        dq[v] = first ? 0.0 : a.dq[v * nc + c];
    }
    T sum[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) sum[v] = T(0);
    if (e1 - e0 <= W) {
        // every face index of the cell, then every rhs value, in flight at
        // once; summed in the same (ascending face) order as the loop below
        // The face's sign (+ where c is P, - where N) goes on the value as a
        // sign-bit flip on the integer pipe, so each entry costs one FP64 add
        // (a - b is a + (-b) in IEEE arithmetic: the same bits)
        T fl[W][NQ];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const int f = code[k] >= 0 ? code[k] : ~code[k];
#pragma unroll
            for (int v = 0; v < NQ; ++v) {
                const T x = code[k] != kEllPad ? a.flux[v * nf + f] : T(0);
                fl[k][v] = code[k] >= 0 ? x : neg_bits(x);
            }
        }
        if (ghosts) gh = cell_ghosts<T, D>(a, c);   // while the rhs are in flight
        // the first face starts the sum (a cell has at least one face)
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (code[k] == kEllPad) continue;
#pragma unroll
            for (int v = 0; v < NQ; ++v) sum[v] = k ? sum[v] + fl[k][v] : fl[0][v];
        }
    } else {
        if (ghosts) gh = cell_ghosts<T, D>(a, c);
        for (int e = e0; e < e1; ++e) {
            const int code = a.cfList[e];
            if (code >= 0) {
#pragma unroll
                for (int v = 0; v < NQ; ++v) sum[v] += a.flux[v * nf + code];
            } else {
                const int f = ~code;
#pragma unroll
                for (int v = 0; v < NQ; ++v) sum[v] -= a.flux[v * nf + f];
            }
        }
    }
    double acc[NQ];
    bool finite = true;
    const double dtvi = dt * vi;
#pragma unroll
    for (int v = 0; v < NQ; ++v) acc[v] = Ak * dq[v] + dtvi * (double)sum[v];
    if (sg != 0.0) {
        acc[0] += dt * sg * (a.rhoInf - qv[0]);
#pragma unroll
        for (int k = 0; k < D; ++k) acc[k + 1] += dt * sg * (a.rhoInf * a.UInf[k] - qv[k + 1]);
        acc[D + 1] += dt * sg * (a.rhoInf * a.EInf - qv[D + 1]);
    }
    double qn[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
        a.dq[v * nc + c] = acc[v];
        qn[v] = qv[v] + Bk * acc[v];
        finite = finite && finite_bits(qn[v]);
        a.q[v * nt + c] = qn[v];
        if (RES) a.res[v * nc + c] = (double)sum[v];
    }
    if (!finite) atomicOr(a.flag, 1);
    if constexpr (PRIM) {
        prims64<D>(a, c, qn);
        if (ghosts) ghosts_of64<D>(a, c, gh, qn);
    }
}

}  // namespace dev
}  // namespace lfm
