// Device kernels of the explicit finite-volume time step (see solver_kernels.cuh).
#include <cuda.h>

#include <cstdint>

#include "lfm_gpu.h"
#include "solver_device.cuh"
#include "solver_launch.h"

namespace lfm {
namespace dev {

// Threads per block: small ones share the FP64 pipes evenly to the end (a
// 393k-cell update is 10 blocks of 256 per SM on some, 11 on others) and a
// boundary cell's ghost work holds few threads. Measured on GB300, us a step at
// 256, 128 and 64 threads: update, 48 x 48 vortex 39.9, 27.7, 29.3, 768 x 512
// cylinder 168.2, 160.6, 159.1, 192 x 128 x 48 wake 836, 792, 756; flux of the
// cylinder 442, 432, 431, of the 331 x 217 M2AUSM cylinder 307, 301, 301, of the
// 97 x 61 x 23 wake 360, 358, 360, of the 384 x 256 x 96 wake 22117, 22097, 22101.
template <int D>
constexpr int kCellThreads = D == 2 ? 128 : 64;
template <int D>
constexpr int kFaceThreads = D == 2 ? 128 : 256;
// Blocks per SM that the flux has to fit (0: whatever does): 56 registers in 2D
// without M2AUSM (with 64 a 50k-cell M2 vortex, whose kernels overlap (pdl_pays),
// took 102 us a step for 72, with the LES stress 217 for 168), and with the LES
// stress in 3D 80, with M2AUSM 128, which it exceeds by a few otherwise.
template <int D, int SCH, bool LES>
constexpr int kFluxBlocks = D == 2 ? (SCH != kSchemeAUSM ? 9 : 0)
                                   : (!LES ? 0 : SCH == kSchemeAUSM ? 2 : 3);

// ---------------------------------------------------------------------------
// k_prep: ghost states and per-cell primitives of entries [first, nt). The
// update writes the cells' and ghosts' primitives for the next stage, so
// between stages only processor halos (copied in) need this pass.
// ---------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(256) k_prep(Args<T> a, int first) {
    const int t = first + LFM_GLOBAL_ID();
    PdlWait{a.pdl}();
    if (t >= a.nt) return;
    constexpr int NQ = D + 2;
    const bool ghost = t >= a.nc && t < a.nc + a.ng;
    const int c = ghost ? a.gCell[t - a.nc] : t;   // a halo's state was copied in from its partition
    double qv[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) qv[v] = a.q[(size_t)v * a.nt + c];
    if (ghost) ghost64<D>(a, t - a.nc, a.gKind[t - a.nc], ghost_in<T, D>(a, qv));
    else prims64<D>(a, t, qv);
}

// A new state: the rows of the stored state from the caller's q ([nq][stride];
// the stored rows themselves after a copy, stride nt), the cells' primitives
// and their boundary ghosts' states and primitives, and a clear
// non-finite flag.
template <int D>
__global__ void __launch_bounds__(256) k_set_state64(const __grid_constant__ Args<double> a, const double* q,
                                                     int64_t stride) {
    const int c = LFM_GLOBAL_ID();
    if (c == 0) *a.flag = 0;
    if (c >= a.nc) return;
    double qv[D + 2];
#pragma unroll
    for (int v = 0; v < D + 2; ++v) {
        qv[v] = q[(size_t)v * stride + c];
        a.q[(size_t)v * a.nt + c] = qv[v];
    }
    prims64<D>(a, c, qv);
    if (a.cellGhosts[c]) ghosts_of64<D>(a, c, cell_ghosts<double, D>(a, c), qv);
}

void launch_set_state64(const Args<double>& a, const double* q, int64_t stride, cudaStream_t st) {
    const unsigned nb = (unsigned)((a.nc + 255) / 256);
    if (a.D == 2) k_set_state64<2><<<nb, 256, 0, st>>>(a, q, stride);
    else k_set_state64<3><<<nb, 256, 0, st>>>(a, q, stride);
}

// D consecutive FP64 values starting at an index that is a multiple of D:
// one 16-byte load in 2D (the constants of an incidence entry or a cell).
template <int D>
__device__ __forceinline__ void load_vec(const double* p, size_t i, double* out) {
    if constexpr (D == 2) {
        const double2 v = reinterpret_cast<const double2*>(p)[i];
        out[0] = v.x;
        out[1] = v.y;
    } else {
#pragma unroll
        for (int k = 0; k < D; ++k) out[k] = p[i * D + k];
    }
}

// Calls f(j, so) for every face entry of cell c (the cell j across it and its
// constant cfSoN). The entries of an ordinary cell are loaded together, in 2D
// with their constants, before sync(), so that after it the gathers from the
// cells across start at once.
template <int D, class Sync, class F>
__device__ __forceinline__ void for_entries64(const Args<double>& a, int c, Sync sync, F f) {
    constexpr int W = kEllWidth<D>;
    const int e0 = a.cfOff[c], n = a.cfOff[c + 1] - e0;
    if (n <= W) {
        int nb[W];
        double so[W][D];
#pragma unroll
        for (int k = 0; k < W; ++k) {
            nb[k] = k < n ? a.cfNbr[e0 + k] : 0;
            if (D == 2 && k < n) load_vec<D>(a.cfSoN, (size_t)(e0 + k), so[k]);
        }
        sync();
#pragma unroll
        for (int k = 0; k < W; ++k) {
            if (k >= n) continue;
            if (D == 3) load_vec<D>(a.cfSoN, (size_t)(e0 + k), so[k]);
            f(nb[k], so[k]);
        }
    } else {
        sync();
        for (int e = e0; e < e0 + n; ++e) {
            double so[D];
            load_vec<D>(a.cfSoN, (size_t)e, so);
            f(a.cfNbr[e], so);
        }
    }
}

// ---------------------------------------------------------------------------
// k_grad: gradients read by M2AUSM's minmod reconstruction.
// ---------------------------------------------------------------------------
template <typename T, int D>
__global__ void __launch_bounds__(kCellThreads<D>) k_grad(Args<T> a) {
    const int c = LFM_GLOBAL_ID();
    if (c >= a.nc) return;
    T gr[D], gp[D], gu[D][D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        gr[k] = gp[k] = T(0);
#pragma unroll
        for (int l = 0; l < D; ++l) gu[k][l] = T(0);
    }
    // Gauss gradients of rho, p and u: the cell's own share through its
    // constant cellSoW, each neighbour's through the entry constant cfSoN
    // (the face values w v_P + (1 - w) v_N expanded)
    const size_t nt = (size_t)a.nt;
    auto own = [&] {
        T sw[D], Uc[D];
        load_vec<D>(a.cellSoW, (size_t)c, sw);
        PdlWait{a.pdl}();
#pragma unroll
        for (int k = 0; k < D; ++k) Uc[k] = a.prim[(size_t)(1 + k) * nt + c];
        const T rhoc = a.q[c];
        const T pc = rhoc * a.prim[(size_t)(D + 1) * nt + c];
#pragma unroll
        for (int x = 0; x < D; ++x) {
            gp[x] = pc * sw[x];
            gr[x] = rhoc * sw[x];
#pragma unroll
            for (int b = 0; b < D; ++b) gu[b][x] = Uc[b] * sw[x];
        }
    };
    for_entries64<D>(a, c, own, [&](int j, const T* so) {
        const T rhoj = a.q[j];
        const T pj = rhoj * a.prim[(size_t)(D + 1) * nt + j];
#pragma unroll
        for (int x = 0; x < D; ++x) {
            gp[x] += pj * so[x];
            gr[x] += rhoj * so[x];
#pragma unroll
            for (int b = 0; b < D; ++b) gu[b][x] += a.prim[(size_t)(1 + b) * nt + j] * so[x];
        }
    });
#pragma unroll
    for (int k = 0; k < D; ++k) {
        a.grad[(size_t)k * a.nt + c] = gr[k];
        a.grad[(size_t)(D + k) * a.nt + c] = gp[k];
#pragma unroll
        for (int l = 0; l < D; ++l) a.grad[(size_t)(2 * D + k * D + l) * a.nt + c] = gu[k][l];
    }
}

// ---------------------------------------------------------------------------
// k_vis: dudx, dTdx and sigmaU per cell (tauMC is rebuilt per face from dudx).
// ---------------------------------------------------------------------------
// LES compiles in the Smagorinsky SGS stress (cases with a.smagC).
template <typename T, int D, bool LES>
__global__ void __launch_bounds__(kCellThreads<D>) k_vis(Args<T> a) {
    const int c = LFM_GLOBAL_ID();
    if (c >= a.nc) return;
    T g[D][D], gT[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        gT[k] = T(0);
#pragma unroll
        for (int l = 0; l < D; ++l) g[k][l] = T(0);
    }
    // Gauss gradients of u and of R psi (T = R psi / R: the flux's face
    // constant kK carries the 1/R). With the face value v_f = w v_P + (1 - w) v_N
    // and so = S/V seen from c, sum_f v_f so = v_c cellSoW_c + sum_e v_j
    // cfSoN_e: the cell's own share through one cell constant, each
    // neighbour's through an entry constant (the other cell j = cfNbr[e]).
    T U[D];
    auto own = [&] {
        T sw[D];
        load_vec<D>(a.cellSoW, (size_t)c, sw);
        PdlWait{a.pdl}();
        const T Rc = a.prim[(size_t)(D + 1) * a.nt + c];
#pragma unroll
        for (int x = 0; x < D; ++x) {
            U[x] = a.prim[(size_t)(1 + x) * a.nt + c];
#pragma unroll
            for (int y = 0; y < D; ++y) g[x][y] = U[x] * sw[y];
            gT[x] = Rc * sw[x];
        }
    };
    for_entries64<D>(a, c, own, [&](int j, const T* so) {
        T fU[D];
#pragma unroll
        for (int k = 0; k < D; ++k) fU[k] = a.prim[(size_t)(1 + k) * a.nt + j];
        const T fR = a.prim[(size_t)(D + 1) * a.nt + j];
#pragma unroll
        for (int x = 0; x < D; ++x) {
#pragma unroll
            for (int y = 0; y < D; ++y) g[x][y] += fU[x] * so[y];
            gT[x] += fR * so[x];
        }
    });
    const T mu = (T)a.mu;
    T tau[D][D];
    stress<T, D>(g, mu, tau);
    const size_t nt = (size_t)a.nt;
#pragma unroll
    for (int x = 0; x < D; ++x) {
#pragma unroll
        for (int y = 0; y < D; ++y) a.V[(size_t)(x * D + y) * nt + c] = g[x][y];
        a.V[(size_t)(D * D + x) * nt + c] = gT[x];
        a.V[(size_t)(D * D + D + x) * nt + c] = dotv<T, D>(U, tau[x]);
    }
    if (LES && a.smagC) {   // Smagorinsky LES: the cell's SGS stress
        T sg[D][D];
        sgs_stress<T, D>(g, a.smagC[c], sg);
#pragma unroll
        for (int x = 0; x < D; ++x)
#pragma unroll
            for (int y = 0; y < D; ++y) a.V[(size_t)(kVisRows<D> + x * D + y) * nt + c] = sg[x][y];
    }
}

// ---------------------------------------------------------------------------
// k_flux: rhs of one face.
// ---------------------------------------------------------------------------
template <typename T, int D, int SCH, bool LES>
__global__ void __launch_bounds__(kFaceThreads<D>, kFluxBlocks<D, SCH, LES>) k_flux(Args<T> a) {
    const int f = LFM_GLOBAL_ID();
    if (f >= a.nf) return;
    constexpr int NQ = D + 2;
    const size_t nt = (size_t)a.nt, nf = (size_t)a.nf;
    const int i = a.fP[f], j = a.fN[f];
    const bool ghost = a.fGhost[f] != 0;
    const T w = a.w[f], wN = a.wN[f];
    T S[D];
#pragma unroll
    for (int k = 0; k < D; ++k) S[k] = a.S[k * nf + f];
    PdlWait{a.pdl}();
    T qi[NQ], qj[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) {
        qi[v] = (T)a.q[v * nt + i];
        qj[v] = (T)a.q[v * nt + j];
    }
    const T cri = a.prim[i], ari = a.prim[j];
    T cU[D], aU[D];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        cU[k] = a.prim[(1 + k) * nt + i];
        aU[k] = a.prim[(1 + k) * nt + j];
    }
    const T cRpsi = a.prim[(D + 1) * nt + i], aRpsi = a.prim[(D + 1) * nt + j];
    const T dR = aRpsi - cRpsi;
    // The convective rhs of a momentum component is -(cm cphi + cp S), the
    // energy's -(ea eb + ec ed). They are added to the viscous sum last, largest
    // product last, as one FMA each: the viscous terms then round at their own
    // size, and a momentum component rounds once at the size of p S.
    T cm[D], cphi, cp, ea, eb, ec, ed, mass;

    if (SCH == kSchemeM1) {
        // One_rk_step_M1's Kurganov-Tadmor flux (src/cfd_v0.cpp:2588-2675)
        // builds its "+" and "-" states with the same linear interpolation
        // (w*P + (1-w)*N and (1-w)*N + w*P), so both states are equal, the
        // dissipation terms (q- - q+)*psi+ psi-/(psi+ - psi-) vanish and the
        // wave-speed weights cancel: the flux is the central flux of the
        // interpolated state, F(q_f).S. It is evaluated in that form - one
        // division per face instead of three, no sound speeds - and equals
        // the reference's value up to rounding. The interpolated internal
        // energy per unit mass is that of the interpolated R psi,
        // e = R psi / (gamma - 1) (R psi = (gamma - 1) e in every cell), so
        // e + R psi = gamma / (gamma - 1) R psi.
        const T rho = interp2(w, wN, qi[0], qj[0]);
        T m[D];
#pragma unroll
        for (int k = 0; k < D; ++k) m[k] = interp2(w, wN, qi[k + 1], qj[k + 1]);
        const T Rpsi = aRpsi - w * dR;   // the same interpolation from the difference
        const T rinv = rcp64(rho);
        T mS = T(0), u2 = T(0);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            mS += m[k] * S[k];
            u2 += m[k] * m[k];
        }
        const T phi = mS * rinv;                          // u_f . S
        mass = -mS;
        cphi = phi;
        cp = rho * Rpsi;
#pragma unroll
        for (int k = 0; k < D; ++k) cm[k] = m[k];
        // mS (gh Rpsi + |u|^2 / 2) with mS |u|^2 = phi |m|^2 / rho
        ea = T(0.5) * phi;
        eb = u2 * rinv;
        ec = mS;
        ed = (T)a.gh * Rpsi;
    } else {
        // Pirozzoli kinetic-energy-preserving mid-point flux (src/cfd_v0.cpp:1966-2023)
        // on the sums of the two sides: rho u.S = (m_P + m_N).S / 2 and
        // u = (m_P + m_N) / (rho_P + rho_N), the halves left to the products
        const T rho2 = qi[0] + qj[0];
        T m2[D], mS2 = T(0);
#pragma unroll
        for (int k = 0; k < D; ++k) {
            m2[k] = qi[k + 1] + qj[k + 1];
            mS2 = k ? mS2 + m2[k] * S[k] : m2[0] * S[0];
        }
        T pavg = (T(0.25) * rho2) * (cRpsi + aRpsi);
        const T H2 = (qi[D + 1] * cri + cRpsi) + (qj[D + 1] * ari + aRpsi);
        if (SCH == kSchemeAUSM) {
            // shock sensor, minmod reconstructions and AUSM+ pressure
            // dissipation (src/cfd_v0.cpp:2288-2339)
            const T cavg = T(0.5) * (a.prim[(D + 2) * nt + i] + a.prim[(D + 2) * nt + j]);
            T d[D];
#pragma unroll
            for (int k = 0; k < D; ++k) d[k] = a.d[k * nf + f];
            T cdiv = T(0), ndiv = T(0), ccurl = T(0), ncurl = T(0), unPos = T(0), unNeg = T(0);
#pragma unroll
            for (int x = 0; x < D; ++x) {
                cdiv += a.V[(x * D + x) * nt + i];
                ndiv += a.V[(x * D + x) * nt + j];
#pragma unroll
                for (int y = x + 1; y < D; ++y) {
                    const T cc = a.V[(x * D + y) * nt + i] - a.V[(y * D + x) * nt + i];
                    const T nn = a.V[(x * D + y) * nt + j] - a.V[(y * D + x) * nt + j];
                    ccurl += cc * cc;
                    ncurl += nn * nn;
                }
                T gi[D], gj[D];
#pragma unroll
                for (int y = 0; y < D; ++y) {
                    gi[y] = a.grad[(2 * D + x * D + y) * nt + i];
                    gj[y] = a.grad[(2 * D + x * D + y) * nt + j];
                }
                T uP, uN;
                minmod_pair<D>(cU[x], aU[x], gi, gj, d, w, wN, uP, uN);
                unPos += uP * S[x];
                unNeg += uN * S[x];
            }
            const T ct = pos_part(-cdiv * rsqrt64(cdiv * cdiv + ccurl + T(4e-2)));
            const T nt_ = pos_part(-ndiv * rsqrt64(ndiv * ndiv + ncurl + T(4e-2)));
            const T theta = T(0.5) * (ct + nt_);
            const T pi = qi[0] * cRpsi, pj = qj[0] * aRpsi;   // p = rho R psi
            T gri[D], grj[D], gpi[D], gpj[D];
#pragma unroll
            for (int y = 0; y < D; ++y) {
                gri[y] = a.grad[y * nt + i];
                grj[y] = a.grad[y * nt + j];
                gpi[y] = a.grad[(D + y) * nt + i];
                gpj[y] = a.grad[(D + y) * nt + j];
            }
            T rhoPos, rhoNeg, pPos, pNeg;
            minmod_pair<D>(qi[0], qj[0], gri, grj, d, w, wN, rhoPos, rhoNeg);
            minmod_pair<D>(pi, pj, gpi, gpj, d, w, wN, pPos, pNeg);
            const T sc = rcp64(a.smag[f] * cavg);
            const T MPos = unPos * sc, MNeg = unNeg * sc;
            const T Msq = T(0.5) * (MPos * MPos + MNeg * MNeg);
            const T Minf = T(0.2);
            T m = (Msq < Minf * Minf) ? Minf * Minf : Msq;
            m = (m < T(1)) ? m : T(1);
            const T M0 = sqrt(m);
            const T fa = M0 * (T(2) - M0);
            const T alpha = T(3.0 / 16.0) * (T(5) * fa * fa - T(4));
            const T hP = p5half(MPos, alpha), hN = p5half(MNeg, alpha);
            const T phalf = pNeg * hN - pPos * hP;   // half of p (p5pos - p5neg), N less P
            // Near |M| = 1 one of 1/2 +- h is small and keeps the rounding of 1/2;
            // pu is small against the pressure there. With (1 +- M)^2 taken out of
            // them the flux took 5 % longer, and the momentum residuals were no
            // nearer to extended precision: against the form with both polynomials
            // written out 0.96 of the error, 0.94 as it stands (18 cases, Mach 0.5
            // to 1.5, jumps of 3 to 50 %).
            const T pu = T(-0.75) * (T(0.5) + hP) * (T(0.5) - hN) * (rhoPos + rhoNeg) * cavg * fa * (unNeg - unPos);
            pavg += theta * (pu - phalf);
        }
        const T hphi = T(0.5) * mS2 * rcp64(rho2);   // u_f . S / 2
        const T mS = T(0.5) * mS2;
        mass = -mS;
        cphi = hphi;
        cp = pavg;
#pragma unroll
        for (int k = 0; k < D; ++k) cm[k] = m2[k];
        ea = eb = T(0);
        ec = T(0.5) * mS;
        ed = H2;
    }

    // Viscous face terms (src/cfd_v0.cpp:2682-2796). With mu == 0 every term
    // is an exact zero and the block is skipped.
    // Each is linear in the face's velocity gradient g, in its R psi gradient
    // gR and in the differences across the face, with per-face constants that
    // carry mu, the conductivity and 1/R (solver_kernels.cuh: mS .. kl):
    //   div tauMC + the Laplacian split, component x:
    //     sum_y g[y][x] mu S_y - (2/3) mu tr(g) S_x + mu (K.g[x] + |delta|/|d| du_x)
    //     (the face tauMC, which the reference interpolates from the cells' or
    //     applies to the boundary's two-point gradient, is linear in g)
    //   heat: k/R (K.gR + |delta|/|d| d(R psi)) + sigmaU . S
    // The heat flux and sigmaU.S of each side are summed before they are
    // interpolated (10 instead of 12 operations in 2D). The kernel is bound by
    // the FP64 pipe, and loads are not: seven constants more per face, the
    // convective products joined by FMAs and in all 18 operations less took the flux
    // of the 768 x 512 M1 cylinder from 580 to 431 us a step, of the 97 x 61 x 23 M2
    // wake from 483 to 359 (GB300).
    const T mu = (T)a.mu;
    T vis[D], visE = T(0);
#pragma unroll
    for (int x = 0; x < D; ++x) vis[x] = T(0);
    if (mu != T(0)) {
        T g[D][D];
        if (!ghost) {
            T ei = T(0), ej = T(0);
#pragma unroll
            for (int x = 0; x < D; ++x) {
#pragma unroll
                for (int y = 0; y < D; ++y)
                    g[x][y] = interp2(w, wN, a.V[(x * D + y) * nt + i], a.V[(x * D + y) * nt + j]);
                const T kK = a.kK[x * nf + f];
                ei = x ? ei + a.V[(D * D + x) * nt + i] * kK : a.V[(D * D) * nt + i] * kK;
                ej = x ? ej + a.V[(D * D + x) * nt + j] * kK : a.V[(D * D) * nt + j] * kK;
                ei += a.V[(D * D + D + x) * nt + i] * S[x];
                ej += a.V[(D * D + D + x) * nt + j] * S[x];
            }
            visE = interp2(w, wN, ei, ej);
        } else {
            // explicit two-point gradients on physical boundaries
            const T dinv = a.dinv[f];
            T dn[D], tau[D][D], Uf[D], eV = T(0);
#pragma unroll
            for (int k = 0; k < D; ++k) {
                dn[k] = a.dnorm[k * nf + f] * dinv;
                eV += dR * dn[k] * a.kK[k * nf + f];
            }
#pragma unroll
            for (int x = 0; x < D; ++x) {
#pragma unroll
                for (int y = 0; y < D; ++y) g[x][y] = (aU[x] - cU[x]) * dn[y];
                Uf[x] = interp(w, cU[x], aU[x]);
            }
            stress<T, D>(g, mu, tau);
#pragma unroll
            for (int x = 0; x < D; ++x) eV += dotv<T, D>(Uf, tau[x]) * S[x];
            visE = eV;
        }
        const T ml = a.ml[f];
#pragma unroll
        for (int x = 0; x < D; ++x) {
            T r = g[x][x] * a.mSK[x * nf + f];
            T off = T(0);   // the trace without g[x][x]
            bool any = false;
#pragma unroll
            for (int y = 0; y < D; ++y) {
                if (y == x) continue;
                r += g[y][x] * a.mS[y * nf + f];
                r += g[x][y] * a.mK[y * nf + f];
                off = any ? off + g[y][y] : g[y][y];
                any = true;
            }
            r += off * a.mT[x * nf + f];
            vis[x] = r + ml * (aU[x] - cU[x]);
        }
        visE += a.kl[f] * dR;
        // Smagorinsky LES: the face tauMC also interpolates the cells' SGS
        // stress (boundary faces keep the laminar two-point one, as in the
        // reference)
        if (LES && a.smagC && !ghost) {
#pragma unroll
            for (int x = 0; x < D; ++x) {
                T s = T(0);
#pragma unroll
                for (int y = 0; y < D; ++y)
                    s += interp(w, a.V[(kVisRows<D> + x * D + y) * nt + i], a.V[(kVisRows<D> + x * D + y) * nt + j]) *
                         S[y];
                vis[x] += s;
            }
        }
    }
    T rhs[NQ];
    rhs[0] = mass;
#pragma unroll
    for (int k = 0; k < D; ++k) rhs[k + 1] = fma(-cp, S[k], fma(-cm[k], cphi, vis[k]));
    rhs[D + 1] = fma(-ec, ed, SCH == kSchemeM1 ? fma(-ea, eb, visE) : visE);
#pragma unroll
    for (int v = 0; v < NQ; ++v) a.flux[v * nf + f] = rhs[v];
}

// ---------------------------------------------------------------------------
// k_update: gather, sponge, RK update (update_cell, solver_device.cuh), then
// the next stage's primitives of the cell and the states
// and primitives of its boundary ghosts.
// ---------------------------------------------------------------------------
template <typename T, int D, bool RES>
__global__ void __launch_bounds__(kCellThreads<D>) k_update(const __grid_constant__ Args<T> a, double Ak, double Bk, int first) {
    const int c = LFM_GLOBAL_ID();
    if (c >= a.nc) return;
    update_cell<T, D, RES, true>(a, c, Ak, Bk, a.step->dt, first, PdlWait{a.pdl});
}

// ---------------------------------------------------------------------------
// Reductions: compute_cfl / compute_dt (max / min over cells) and the sum of
// squared cell residuals. Block results go to partials, a single block
// finishes; both levels use a fixed tree, so results are reproducible.
// ---------------------------------------------------------------------------
//
// k_cfl does both levels in one launch: the last block to finish (an arrival
// counter that it resets) reduces the block results and writes the value to
// page-locked host memory, so a caller waits for one launch and no copy. A run
// with adjustTimeStep asks for one of these per step.
template <int D>
__global__ void __launch_bounds__(256) k_cfl(const double* q, QOffset qo, int nt, int nc, const double* volInv,
                                             const int* sOff, const double* cellS, double dt, int mode, double maxCo,
                                             double* partial, unsigned* arrived, double* out) {
    __shared__ double sh[256];
    __shared__ bool last;
    const int c = LFM_GLOBAL_ID();
    const double none = (mode == 0) ? 0.0 : 100.0;
    double v = none;
    if (c < nc) {
        const double rho = q[c] + qo.v[0];
        double m[D];
#pragma unroll
        for (int k = 0; k < D; ++k) m[k] = q[(size_t)(k + 1) * nt + c] + qo.v[k + 1];
        double sum = 0.0;
        for (int e = sOff[c]; e < sOff[c + 1]; ++e) {
            double flux = 0.0, s2 = 0.0;
#pragma unroll
            for (int k = 0; k < D; ++k) {
                const double S = cellS[(size_t)e * D + k];
                flux += m[k] * S;
                s2 += S * S;
            }
            // min dt: the flux through the unit area vector
            sum += (mode == 0) ? fabs(flux) : fabs(flux * rsqrt(s2));
        }
        v = (mode == 0) ? sum * ((1.0 / rho) * volInv[c] * dt) : maxCo * rho * 2.0 * (1.0 / volInv[c]) / sum;
    }
    auto reduce = [&](double x) {
        sh[threadIdx.x] = x;
        __syncthreads();
        for (int s = blockDim.x / 2; s > 0; s >>= 1) {
            if (threadIdx.x < s) {
                const double o = sh[threadIdx.x + s];
                sh[threadIdx.x] = (mode == 0) ? fmax(sh[threadIdx.x], o) : fmin(sh[threadIdx.x], o);
            }
            __syncthreads();
        }
    };
    reduce(v);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = sh[0];
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    v = none;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += blockDim.x) {
        const double o = *(volatile double*)(partial + k);
        v = (mode == 0) ? fmax(v, o) : fmin(v, o);
    }
    __syncthreads();
    reduce(v);
    if (threadIdx.x == 0) {
        *out = sh[0];
        *arrived = 0;
    }
}

// The sum of the block results of k_res_sq.
__global__ void __launch_bounds__(256) k_sum_final(const double* partial, int n, double* out) {
    __shared__ double sh[256];
    double v = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) v = v + partial[k];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

__global__ void __launch_bounds__(256) k_res_sq(const double* res, int nc, double* partial) {
    __shared__ double sh[256];
    const int c = LFM_GLOBAL_ID();
    const double v = (c < nc) ? res[c] * res[c] : 0.0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void k_set_flag(int* flag, int v) { *flag = v; }

// Preparation for one residual of a caller's state q ([nq][stride], read only):
// the stored rows, the primitives of every cell and the states and primitives of
// the ghosts, whose viscous rows and gradients (read as zeros; cellGrad: the
// cells' too, which no pass computes then) are cleared --
// what a memset, a copy and a preparation pass did in three launches, each about
// as long as the residual's own kernels on a small mesh.
template <int D>
__global__ void __launch_bounds__(128) k_prep_residual64(const __grid_constant__ Args<double> a, const double* q,
                                                         int64_t stride, int vRows, int gradRows, int cellGrad) {
    const int t = LFM_GLOBAL_ID();
    PdlRelease{a.pdl}();
    if (t >= a.nt) return;
    constexpr int NQ = D + 2;
    const size_t nt = (size_t)a.nt;
    const int c = t < a.nc ? t : a.gCell[t - a.nc];
    double qv[NQ];
#pragma unroll
    for (int v = 0; v < NQ; ++v) qv[v] = q[(size_t)v * stride + c];
    if (t >= a.nc || cellGrad)
        for (int r = 0; r < gradRows; ++r) a.grad[r * nt + t] = 0.0;
    if (t >= a.nc) {
        for (int r = 0; r < vRows; ++r) a.V[r * nt + t] = 0.0;
        ghost64<D>(a, t - a.nc, a.gKind[t - a.nc], ghost_in<double, D>(a, qv));
        return;
    }
#pragma unroll
    for (int v = 0; v < NQ; ++v) a.q[(size_t)v * nt + t] = qv[v];
    prims64<D>(a, t, qv);
}

void launch_prep_residual64(const Args<double>& a, const double* q, int64_t stride, int vRows, int gradRows, int cellGrad,
                            cudaStream_t st) {
    const unsigned nb = (unsigned)((a.nt + 127) / 128);
    if (a.D == 2) k_prep_residual64<2><<<nb, 128, 0, st>>>(a, q, stride, vRows, gradRows, cellGrad);
    else k_prep_residual64<3><<<nb, 128, 0, st>>>(a, q, stride, vRows, gradRows, cellGrad);
}

double* kernel_address(const double* p, size_t bytes) {
    // a copy engine takes any address, a kernel's loads only aligned ones
    if (reinterpret_cast<uintptr_t>(p) % alignof(double) != 0) return nullptr;
    // One query for all that is asked (a batch asks for every state it moves);
    // what is page-locked and mapped ends with its allocation or registration.
    static const auto query = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &found) !=
            cudaSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<CUresult (*)(unsigned, CUpointer_attribute*, void**, CUdeviceptr)>(f);
    }();
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    unsigned type = 0, managed = 0;
    CUdeviceptr d = 0, start = 0;
    size_t size = 0;
    void* into[] = {&type, &managed, &d, &start, &size};   // zeros where p is unknown to the driver
    if (!query || query(5, what, into, reinterpret_cast<CUdeviceptr>(p)) != CUDA_SUCCESS) return nullptr;
    if (type != CU_MEMORYTYPE_HOST || managed || d == 0) return nullptr;
    if (d < start || d - start > size || bytes > size - (size_t)(d - start)) return nullptr;
    return reinterpret_cast<double*>(d);
}

// ---------------------------------------------------------------------------
// Launchers.
// ---------------------------------------------------------------------------
static inline unsigned blocks(int n, int b) { return (unsigned)((n + b - 1) / b); }

template <typename T, int D, int SCH, bool LES>
void launch_flux(const Args<T>& a, const StageConfig& s, cudaStream_t st) {
    launch_kernel_pdl(s.pdl && a.pdl, k_flux<T, D, SCH, LES>, blocks(a.nf, kFaceThreads<D>), kFaceThreads<D>, st, a);
}

template <typename T, int D, bool LES>
void launch_fp64(const Args<T>& a, const StageConfig& s, int which, cudaStream_t st) {
    switch (which) {
        case 0: {
            // the update keeps the cells' and the ghosts' primitives
            // current: only halos remain, unless all are stale
            const int first = s.fullPrep ? 0 : a.nc + a.ng;
            if (a.nt > first) launch_kernel_pdl(s.pdl && a.pdl, k_prep<T, D>, blocks(a.nt - first, 256), 256, st, a, first);
            break;
        }
        case 1:
            if (s.needGrad) launch_kernel_pdl(s.pdl && a.pdl, k_grad<T, D>, blocks(a.nc, kCellThreads<D>), kCellThreads<D>, st, a);
            break;
        case 2:
            if (s.needVis) launch_kernel_pdl(s.pdl && a.pdl, k_vis<T, D, LES>, blocks(a.nc, kCellThreads<D>), kCellThreads<D>, st, a);
            break;
        case 3:
            if (s.scheme == kSchemeM1) launch_flux<T, D, kSchemeM1, LES>(a, s, st);
            else if (s.scheme == kSchemeM2) launch_flux<T, D, kSchemeM2, LES>(a, s, st);
            else launch_flux<T, D, kSchemeAUSM, LES>(a, s, st);
            break;
        case 4:
            if (s.withRes) launch_kernel_pdl(s.pdl && a.pdl, k_update<T, D, true>, blocks(a.nc, kCellThreads<D>), kCellThreads<D>, st, a, s.A, s.B, s.first);
            else launch_kernel_pdl(s.pdl && a.pdl, k_update<T, D, false>, blocks(a.nc, kCellThreads<D>), kCellThreads<D>, st, a, s.A, s.B, s.first);
            break;
        default: break;
    }
}

// Individual kernels (a stage is kernels 0..kKernelsPerStage-1 in order).
template <typename T>
void launch_kernel(const Args<T>& a, const StageConfig& s, int which, cudaStream_t st) {
    const bool les = a.smagC != nullptr;
    if (a.D == 2)
        les ? launch_fp64<T, 2, true>(a, s, which, st) : launch_fp64<T, 2, false>(a, s, which, st);
    else
        les ? launch_fp64<T, 3, true>(a, s, which, st) : launch_fp64<T, 3, false>(a, s, which, st);
}

template <typename T>
void launch_stage(const Args<T>& a, const StageConfig& s, cudaStream_t st) {
    for (int k = 0; k < kKernelsPerStage; ++k) launch_kernel<T>(a, s, k, st);
}
template void launch_stage<double>(const Args<double>&, const StageConfig&, cudaStream_t);
// The FP32-bulk form runs its own kernels (solver_kernels_fp32.cu).
template <>
void launch_stage<float>(const Args<float>& a, const StageConfig& s, cudaStream_t st) {
    for (int k = 0; k < kKernelsPerStage; ++k) launch_kernel_fp32(a, s, k, st);
}
template void launch_kernel<double>(const Args<double>&, const StageConfig&, int, cudaStream_t);
template <>
void launch_kernel<float>(const Args<float>& a, const StageConfig& s, int which, cudaStream_t st) {
    launch_kernel_fp32(a, s, which, st);
}

void launch_cfl(int D, const double* q, QOffset qo, int nt, int nc, const double* volInv, const int* sOff, const double* cellS,
                double dt, int mode, double maxCo, double* partial, unsigned* arrived, double* out, cudaStream_t st) {
    const unsigned nb = blocks(nc, 256);
    if (D == 2)
        k_cfl<2><<<nb, 256, 0, st>>>(q, qo, nt, nc, volInv, sOff, cellS, dt, mode, maxCo, partial, arrived, out);
    else
        k_cfl<3><<<nb, 256, 0, st>>>(q, qo, nt, nc, volInv, sOff, cellS, dt, mode, maxCo, partial, arrived, out);
}

__global__ void k_set_step(StepDt* step, double dt, float dt32) {
    step->dt = dt;
    step->dt32 = dt32;
}

void launch_set_step(StepDt* step, double dt, cudaStream_t st) { k_set_step<<<1, 1, 0, st>>>(step, dt, (float)dt); }

void launch_res_sum(const double* res, int nc, double* partial, double* out, cudaStream_t st) {
    const unsigned nb = blocks(nc, 256);
    k_res_sq<<<nb, 256, 0, st>>>(res, nc, partial);
    k_sum_final<<<1, 256, 0, st>>>(partial, (int)nb, out);
}

// The constants of the FP64 path, each the value its kernels would otherwise
// form on every visit. Formed here because a mesh's geometry is uploaded once
// while its host loops would double the set-up time of a case.
template <int D>
__global__ void __launch_bounds__(256) k_fp64_face_constants(const Args<double> a, double* wN, double* mS, double* mK,
                                                             double* mT, double* mSK, double* kK, double* ml,
                                                             double* kl) {
    const int f = LFM_GLOBAL_ID();
    if (f >= a.nf) return;
    wN[f] = 1.0 - a.w[f];
    if (!mS) return;
    const double kR = a.kcond * a.Rinv, lap = a.dmag[f] * a.dinv[f];
#pragma unroll
    for (int k = 0; k < D; ++k) {
        const size_t at = (size_t)k * a.nf + f;
        const double S = a.S[at], K = a.K[at];
        mS[at] = a.mu * S;
        mK[at] = a.mu * K;
        mT[at] = -a.mu23 * S;
        mSK[at] = a.mu * (S * (1.0 / 3.0) + K);
        kK[at] = kR * K;
    }
    ml[f] = a.mu * lap;
    kl[f] = kR * lap;
}

// With the face value v_f = w v_P + (1 - w) v_N and so_e = S/V of entry e's
// face seen from its cell c, the Gauss gradient is
//   sum_e v_f so_e = v_c sum_e w_own so_e + sum_e v_across w_across so_e,
// the first sum a cell constant, w_across so_e an entry constant (w_own = w
// where c is P, 1 - w where c is N).
template <int D>
__global__ void __launch_bounds__(256) k_fp64_cell_constants(const Args<double> a, double* soN, double* soW) {
    const int c = LFM_GLOBAL_ID();
    if (c >= a.nc) return;
    double own[D];
#pragma unroll
    for (int k = 0; k < D; ++k) own[k] = 0.0;
    for (int e = a.cfOff[c]; e < a.cfOff[c + 1]; ++e) {
        const int code = a.cfList[e], f = code >= 0 ? code : ~code;
        const double w = a.w[f], wOwn = code >= 0 ? w : 1.0 - w, wAcross = code >= 0 ? 1.0 - w : w;
#pragma unroll
        for (int k = 0; k < D; ++k) {
            const double Sv = a.S[(size_t)k * a.nf + f] * a.volInv[c], so = code >= 0 ? Sv : -Sv;
            soN[(size_t)e * D + k] = wAcross * so;   // entry-major: one entry's D values together
            own[k] += wOwn * so;
        }
    }
#pragma unroll
    for (int k = 0; k < D; ++k) soW[(size_t)c * D + k] = own[k];
}

template <int D>
static void fp64_constants(const Args<double>& a, cudaStream_t st) {
    auto w = [](const double* p) { return const_cast<double*>(p); };
    k_fp64_face_constants<D><<<blocks(a.nf, 256), 256, 0, st>>>(a, w(a.wN), w(a.mS), w(a.mK), w(a.mT), w(a.mSK), w(a.kK),
                                                               w(a.ml), w(a.kl));
    k_fp64_cell_constants<D><<<blocks(a.nc, 256), 256, 0, st>>>(a, w(a.cfSoN), w(a.cellSoW));
}

void launch_fp64_constants(const Args<double>& a, cudaStream_t st) {
    a.D == 2 ? fp64_constants<2>(a, st) : fp64_constants<3>(a, st);
}

void launch_set_flag(int* flag, int v, cudaStream_t st) { k_set_flag<<<1, 1, 0, st>>>(flag, v); }

// dst[v][c] = src[v][c] + sign * off[v] for nq rows of n cells (converts
// between the FP32-bulk form's stored q - q_ref and the absolute state).
__global__ void __launch_bounds__(256) k_offset_rows(double* dst, int64_t dstStride, const double* src,
                                                     int64_t srcStride, int n, int nq, QOffset off, double sign) {
    const int c = LFM_GLOBAL_ID();
    if (c >= n) return;
    for (int v = 0; v < nq; ++v) dst[(size_t)v * dstStride + c] = src[(size_t)v * srcStride + c] + sign * off.v[v];
}

void launch_offset_rows(double* dst, int64_t dstStride, const double* src, int64_t srcStride, int n, int nq,
                        QOffset off, double sign, cudaStream_t st) {
    if (n > 0) k_offset_rows<<<blocks(n, 256), 256, 0, st>>>(dst, dstStride, src, srcStride, n, nq, off, sign);
}

// Halo copies between the partitions of a decomposed case: halo slot h (index
// first + h of the destination) takes `rows` values of cell srcCell[h] of
// partition srcPart[h] -- the on-device form of the reference's MPI halo
// exchange (src/cfd_v0.cpp:3283-3374, 3607-3692).
template <typename X>
__global__ void __launch_bounds__(256) k_halo_gather(X* dst, int dstNt, int first, int rows, int nh,
                                                     const int* srcPart, const int* srcCell, X* const* srcBase,
                                                     const int* srcNt) {
    const int h = LFM_GLOBAL_ID();
    if (h >= nh) return;
    const int p = srcPart[h], c = srcCell[h];
    const X* src = srcBase[p];
    const size_t snt = (size_t)srcNt[p];
    for (int r = 0; r < rows; ++r) dst[(size_t)r * dstNt + first + h] = src[(size_t)r * snt + c];
}

template <typename X>
void launch_halo_gather(X* dst, int dstNt, int first, int rows, int nh, const int* srcPart, const int* srcCell,
                        X* const* srcBase, const int* srcNt, cudaStream_t st) {
    if (nh > 0)
        k_halo_gather<X><<<blocks(nh, 256), 256, 0, st>>>(dst, dstNt, first, rows, nh, srcPart, srcCell, srcBase,
                                                          srcNt);
}
template void launch_halo_gather<double>(double*, int, int, int, int, const int*, const int*, double* const*,
                                         const int*, cudaStream_t);

// Halo slots [first, first + nh) of an array of `words` floats per cell, one
// thread per 16 bytes.
__global__ void __launch_bounds__(256) k_halo_gather_cells(float4* dst, int first, int parts, int nh,
                                                           const int* srcPart, const int* srcCell,
                                                           float* const* srcBase) {
    const int k = LFM_GLOBAL_ID();
    if (k >= nh * parts) return;
    const int h = k / parts, r = k - h * parts;
    const float4* src = reinterpret_cast<const float4*>(srcBase[srcPart[h]]);
    dst[(size_t)(first + h) * parts + r] = src[(size_t)srcCell[h] * parts + r];
}

void launch_halo_gather_cells(float* dst, int first, int words, int nh, const int* srcPart, const int* srcCell,
                              float* const* srcBase, cudaStream_t st) {
    const int parts = words / 4;
    if (nh > 0)
        k_halo_gather_cells<<<blocks(nh * parts, 256), 256, 0, st>>>(reinterpret_cast<float4*>(dst), first, parts, nh,
                                                                    srcPart, srcCell, srcBase);
}

}  // namespace dev
}  // namespace lfm

// ---------------------------------------------------------------------------
// Self-test of the FP64 path's own arithmetic (lfm_selftest_fp64).
// ---------------------------------------------------------------------------
namespace {

// Inputs a function takes (lfm_selftest_fp64), 0: no such function.
int selftest_inputs(int fn) {
    static const int n[] = {1, 1, 1, 1, 2, 9, 9};
    return fn >= 0 && fn < (int)(sizeof(n) / sizeof(n[0])) ? n[fn] : 0;
}

__global__ void k_selftest_fp64(int fn, int64_t n, const double* in, double* out) {
    using namespace lfm::dev;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    auto x = [&](int k) { return in[k * n + i]; };
    switch (fn) {
        case 0: out[i] = rcp64(x(0)); break;
        case 1: out[i] = rsqrt64(x(0)); break;
        case 2: out[i] = pos_part(x(0)); break;
        case 3: out[i] = atleast1(x(0)) ? 1.0 : 0.0; break;
        case 4: out[i] = p5half(x(0), x(1)); break;
        default: {
            const double gP[2] = {x(2), x(3)}, gN[2] = {x(4), x(5)}, d[2] = {x(6), x(7)};
            double fromP, fromN;
            minmod_pair<2>(x(0), x(1), gP, gN, d, x(8), 1.0 - x(8), fromP, fromN);
            out[i] = fn == 5 ? fromP : fromN;
        }
    }
}

}  // namespace

extern "C" int lfm_selftest_fp64(int fn, int64_t n, const double* in, double* out) {
    const int rows = selftest_inputs(fn);
    if (rows == 0 || n <= 0 || !in || !out) return LFM_ERR_INVALID;
    double *di = nullptr, *dout = nullptr;
    cudaError_t e = cudaMalloc(&di, (size_t)rows * (size_t)n * sizeof(double));
    if (e == cudaSuccess) e = cudaMalloc(&dout, (size_t)n * sizeof(double));
    if (e == cudaSuccess) e = cudaMemcpy(di, in, (size_t)rows * (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        k_selftest_fp64<<<(unsigned)((n + 255) / 256), 256>>>(fn, n, di, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, (size_t)n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaFree(di);
    cudaFree(dout);
    return e == cudaSuccess ? LFM_OK : LFM_ERR_CUDA;
}

extern "C" int lfm_selftest_kernel_range(const void* p, size_t bytes) {
    return lfm::dev::kernel_address(static_cast<const double*>(p), bytes) ? 1 : 0;
}
