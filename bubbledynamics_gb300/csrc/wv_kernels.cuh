// Device side of the Westervelt solver: one fused kernel per time step, one pass over the
// Mur faces and one over the DFT planes, templated on the storage/arithmetic type.
//
// Reference: W:139-236 (interior update), W:62-85 (source plane), W:88-135
// (Mur), W:242-265 (water power), W:268-345 (harmonic power via FFT; here an
// on-the-fly DFT), W:575-584 (time-level rotation; here a pointer ring).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/bubbledyn.h"

namespace bd {

#define BD_PI 3.14159265358979323846


// Per-material constants in a form that needs no division per cell, in the
// arithmetic type of the kernel.
template <class real>
struct MatConst {
    real c0;
    real delta_2dt;            // delta / (2 dt)            -> kd = delta_2dt / c^2   (W:216)
    real beta2_rho;            // 2 beta / rho              -> kn = beta2_rho / c^2   (W:217)
    real ra_num[BD_MAX_RELAX]; // 2dt*2*c_v*tau_v / (2dt^3 (2dt+3tau_v)) -> ra = ra_num / c^3 (W:226-227)
    real rb[BD_MAX_RELAX];     // tau_v / (2dt + 3 tau_v)                 (W:227)
    int n_relax;
    int pad;
    // what cell_update() forms from c, for c = c0 (wv_derive_kernel fills these on the
    // device with the operations of cell_coef(), so a cell without a c map reads the
    // bits it would compute)
    real kxy, kz, kd, kn, kr;  // stencil xy and z, diffusivity, nonlinearity, (c dt)^2
    real xr;                   // x / (1 - x), x = 3 kr sum a (semi-implicit relaxation)
    real av[BD_MAX_RELAX];     // a_v
};

template <class real>
struct WvConst {
    MatConst<real> mat[BD_MAX_MATERIALS];
};

template <class real>
struct WvArgs {
    int nx, ny, nz;
    int zb;                    // z-chunk per CTA
    int px;                    // row pitch in cells
    int rev;                   // two-cell kernel: march from the high end
    int acc_n;                 // two-cell and DFT kernels: steps this one accumulates (itself and acc_n - 1 before it)
    long long plane;           // px*ny
    // time levels: p^n (stencil), p^{n-1..n-3}, and the p^{n-4} buffer that receives p^{n+1}
    const real* __restrict__ p0;
    const real* __restrict__ p1;
    const real* __restrict__ p2;
    const real* __restrict__ p3;
    real* __restrict__ p4;
    // relaxation: R^{n-1} and the R^{n-2} buffer that receives R^n, per process
    const real* __restrict__ rcur[BD_MAX_RELAX];
    real* __restrict__ rold[BD_MAX_RELAX];
    int max_relax;
    // medium
    const float* __restrict__ cmap;
    const uint8_t* __restrict__ matmap;
    const int* __restrict__ plane_mat;
    // geometry of the update
    int xhi, yhi, zlo, zhi;    // box of the stencil update (inclusive)
    int src_iz;                // source plane or -1
    int mir_x, mir_y;
    int mur_xp, mur_yp, mur_zp, mur_zm, L, Lzm;
    const real* __restrict__ wx;    // sponge factors per axis (nullptr = none)
    const real* __restrict__ wy;
    const real* __restrict__ wz;
    real dt, kxy180, kz180, dt2;   // dt, dt^2/(180 dx^2), dt^2/(180 dz^2), dt^2
    real dtdx, dtdz;               // dt/dx, dt/dz (Mur)
    // source (W:62-85)
    const double* __restrict__ sA;      // p0*amp_e / var (FP32 path) or p0*amp_e (FP64 path)
    const double* __restrict__ sVar;    // var (FP64 path)
    const double* __restrict__ sTau;    // geometric delay
    const float* __restrict__ sAf;      // FP32 path amplitude p0*amp_e/var
    const float* __restrict__ sPsi;     // FP32 path per-tone phase offset [n_tones][plane]
    const float* __restrict__ sTauf;    // FP32 path delay (burst window)
    const double* __restrict__ sPhi;    // element phase (FP64 path)
    int n_tones;
    int burst;
    double freq[BD_MAX_TONES], tamp[BD_MAX_TONES], tphase[BD_MAX_TONES];
    float tampf[BD_MAX_TONES];
    double tau_max, burst_len;
    float burst_lenf;
    // step tables
    const long long* __restrict__ step_base;   // device step counter of the chunk start
    const double* __restrict__ t_src;          // per-step source time
    const float* __restrict__ theta;           // FP32 path: per step per tone 2 pi frac(f (t - shift))
    const float* __restrict__ tb0;             // FP32 path: per step t - tau_max
    // accumulators
    real* __restrict__ peak;
    real* __restrict__ energy;
    real* __restrict__ dre;
    real* __restrict__ dim;
    const real* __restrict__ tw;               // DFT twiddles [dft step][n_dft][2]
    long long peak_start, peak_end, energy_start, energy_end, dft_start, dft_len;
    real ke;                   // FP64: weight of p^2 (dt) or of (p^{n+1} - p^{n-1})^2 (1 / 4dt) in the energy
    int energy_mode, n_dft, dz_lo, dz_hi;
    int relax_scheme;
    int mat_tile;              // 1: the two-cell kernel receives the material map as a TMA tile per plane
};

// Explicitly rounded arithmetic: the compiler never re-contracts these, so
// every kernel variant that calls cell_update() produces the same bits.
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
// FP32 divisions use the fast hardware path (max 2 ulp), FP64 ones are IEEE.
__device__ __forceinline__ float div_(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double div_(double a, double b) { return __ddiv_rn(a, b); }

template <class real>
__device__ __forceinline__ real ld(const real* p) { return __ldg(p); }

template <class real>
__device__ __forceinline__ real source_value(const WvArgs<real>& a, long long step, int j);

template <>
__device__ __forceinline__ double source_value<double>(const WvArgs<double>& a, long long step, int j) {
    // FP64 path: the arithmetic of W:78-82 (plus tones / bursts / elements).
    const double A = a.sA[j];
    if (A == 0.0) return 0.0;
    double tt = a.t_src[step] + a.sTau[j];
    if (a.burst) {
        const double tb = tt - a.tau_max;
        if (tb < 0.0 || tb >= a.burst_len) return 0.0;
        tt = tb;
    }
    double sum = 0.0;
    for (int k = 0; k < a.n_tones; ++k) sum += a.tamp[k] * sin(2 * BD_PI * a.freq[k] * tt + a.tphase[k] + a.sPhi[j]);
    return A * sum / a.sVar[j];
}

template <>
__device__ __forceinline__ float source_value<float>(const WvArgs<float>& a, long long step, int j) {
    // FP32 path: phases reduced on the host to [0, 2 pi) per step and per cell.
    const float A = a.sAf[j];
    if (A == 0.0f) return 0.0f;
    if (a.burst) {
        const float tb = a.tb0[step] + a.sTauf[j];
        if (tb < 0.0f || tb >= a.burst_lenf) return 0.0f;
    }
    float sum = 0.0f;
    for (int k = 0; k < a.n_tones; ++k)
        sum = fma_(a.tampf[k], sinf(add_(a.theta[step * BD_MAX_TONES + k], a.sPsi[(long long)k * a.plane + j])), sum);
    return mul_(A, sum);
}

template <class real>
__device__ __forceinline__ bool is_mur_cell(const WvArgs<real>& a, int ix, int iy, int iz) {
    return (a.mur_yp && iy >= a.ny - a.L) || (a.mur_xp && ix >= a.nx - a.L) ||
           (a.mur_zp && iz >= a.nz - a.L) || (a.mur_zm && iz < a.Lzm);
}

// max(|v|, pk).  FP64 values compare as integers: a double compare takes the FP64
// unit, 64 cycles a warp, like every FP64 instruction here.
__device__ __forceinline__ float peak_max(float v, float pk) {
    const float av = fabsf(v);
    return av > pk ? av : pk;
}
__device__ __forceinline__ double peak_max(double v, double pk) {
    const long long av = __double_as_longlong(v) & 0x7fffffffffffffffLL;
    return av <= 0x7ff0000000000000LL && av > __double_as_longlong(pk) ? __longlong_as_double(av) : pk;
}

// Energy accumulator update: E + p^2 dt, or E + ((p^{n+1}-p^{n-1})/2dt)^2 dt (W:253-257).
template <class real>
__device__ __forceinline__ real energy_add(const WvArgs<real>& a, real old, real v, real vm1) {
    if constexpr (sizeof(real) == 8) {             // three FP64 instructions, no division
        const real d = a.energy_mode == BD_ENERGY_DPDT2 ? add_(v, -vm1) : v;
        return fma_(mul_(d, d), a.ke, old);
    }
    real e;
    if (a.energy_mode == BD_ENERGY_DPDT2) {
        const real dp = div_(add_(v, -vm1), mul_(real(2.0), a.dt));     // W:253
        e = mul_(mul_(dp, dp), a.dt);                                    // W:257
    } else {
        e = mul_(mul_(v, v), a.dt);
    }
    return add_(old, e);
}

// Peak / energy accumulation on the final p^{n+1} of a cell.
template <class real>
__device__ __forceinline__ void accumulate(const WvArgs<real>& a, long long step, long long i, real v, real vm1) {
    if (step >= a.peak_start && step < a.peak_end) a.peak[i] = peak_max(v, a.peak[i]);
    if (step >= a.energy_start && step < a.energy_end) a.energy[i] = energy_add(a, a.energy[i], v, vm1);
}

template <class real>
__device__ __forceinline__ real cell_c(const WvArgs<real>& a, const WvConst<real>& K, long long i, int m) {
    return a.cmap ? (real)__ldg(a.cmap + i) : K.mat[m].c0;
}

template <class real>
__device__ __forceinline__ int cell_mat(const WvArgs<real>& a, long long i, int iz) {
    if (a.matmap) return __ldg(a.matmap + i);
    if (a.plane_mat) return __ldg(a.plane_mat + iz);
    return 0;
}

// 6th-order second difference times 180 (W:203-205): -490 p + 270 s1 - 27 s2 + 2 s3
template <class real>
__device__ __forceinline__ real d2x180(real pc, real s1, real s2, real s3) {
    return fma_(real(2), s3, fma_(real(-27), s2, fma_(real(270), s1, mul_(real(-490), pc))));
}

// Coefficients of the cell update at sound speed c, into M's derived fields.
template <class real, int NRMAX>
__device__ __forceinline__ void cell_coef(const WvArgs<real>& a, MatConst<real>& M, real c) {
    const real c2 = mul_(c, c);
    const real ic = div_(real(1), c);
    const real ic2 = mul_(ic, ic);
    M.kxy = mul_(c2, a.kxy180);
    M.kz = mul_(c2, a.kz180);
    M.kd = mul_(M.delta_2dt, ic2);
    M.kn = mul_(M.beta2_rho, ic2);
    M.kr = mul_(c2, a.dt2);
    if (a.relax_scheme == BD_RELAX_SEMI_IMPLICIT) {
        const real ic3 = mul_(ic2, ic);
        real sa = real(0);
#pragma unroll
        for (int v = 0; v < NRMAX; ++v)
            if (v < M.n_relax) {
                M.av[v] = mul_(M.ra_num[v], ic3);
                sa = add_(sa, M.av[v]);
            }
        // p = num / (1 - x) with x = 3 kr sum a small: written as num + num x / (1 - x) so
        // the (possibly approximate) division only touches the small correction
        const real x = mul_(mul_(real(3), M.kr), sa);
        M.xr = div_(x, add_(real(1), -x));
    } else {
#pragma unroll
        for (int v = 0; v < NRMAX; ++v)
            if (v < M.n_relax) M.av[v] = mul_(mul_(M.ra_num[v], ic2), ic);
    }
}

template <class real>
__global__ void wv_derive_kernel(const WvArgs<real> a, WvConst<real>* K) {
    const int m = threadIdx.x;
    if (m < BD_MAX_MATERIALS && K->mat[m].c0 > real(0)) {
        MatConst<real> M = K->mat[m];
        cell_coef<real, BD_MAX_RELAX>(a, M, M.c0);
        K->mat[m] = M;
    }
}

// The update of one cell (W:203-234, or the semi-implicit relaxation coupling).
// sx1..sy3: sums of the +-1, +-2, +-3 neighbours along x / y; w[0..6]: p^n at
// iz-3..iz+3 (or iz+3..iz-3); q1..q4: p^{n-1..n-4}; rc / ro: R^{n-1} / R^{n-2} per
// process, ro returns R^n; M: material with the derived coefficients of the cell's
// sound speed.  Returns p^{n+1} before the sponge factor.
template <class real, int NRMAX = BD_MAX_RELAX>
__device__ __forceinline__ real cell_update(const WvArgs<real>& a, const MatConst<real>& M, real pc, real sx1, real sx2,
                                            real sx3, real sy1, real sy2, real sy3, const real* w, real q1, real q2,
                                            real q3, real q4, const real* rc, real* ro) {
    // W:207: 5 p - 18 p1 + 24 p2 - 14 p3 + 3 p4
    const real Dttt = fma_(real(3), q4, fma_(real(-14), q3, fma_(real(24), q2, fma_(real(-18), q1, mul_(real(5), pc)))));
    const real s3 = fma_(real(3), pc, fma_(real(-4), q1, q2));
    const real D1 = mul_(mul_(s3, s3), real(0.25));                                                   // W:208
    const real D2 = mul_(pc, fma_(real(2), pc, fma_(real(-5), q1, fma_(real(4), q2, -q3))));          // W:209
    // W:234 without the relaxation term, as an increment on p^n: Y = p + V with
    // V = (p - p1) + kxy (Dxx + Dyy) + kz Dzz + kd Dttt + kn (D1 + D2).  The terms are
    // summed at the size of the increment (about a quarter of p per step at 8
    // cells per wavelength) and p^{n+1} takes one final rounding: the FP32 field
    // error against FP64 after 3000 cfg1 steps drops from 1.04e-5 to 8.4e-6
    // (summing 2p - p1 + ... directly rounds at the size of p five times).
    // FP64 is bound by its FP64 instructions: there the x and y rings add up before
    // they are weighted (two instructions fewer) and the relaxation terms go straight
    // into V.  Weights that carry kxy and kz save three more (64 x 64 x 201, two
    // processes: 139 us a step instead of 146), but no longer cancel exactly: five
    // times the error after 600 steps.
    real V = add_(pc, -q1);
    const real sz1 = add_(w[4], w[2]), sz2 = add_(w[5], w[1]), sz3 = add_(w[6], w[0]);
    real Dxy;
    if constexpr (sizeof(real) == 8)
        Dxy = fma_(real(2), add_(sx3, sy3), fma_(real(-27), add_(sx2, sy2), fma_(real(270), add_(sx1, sy1), mul_(real(-980), pc))));
    else Dxy = add_(d2x180(pc, sx1, sx2, sx3), d2x180(pc, sy1, sy2, sy3));
    V = fma_(M.kxy, Dxy, V);
    V = fma_(M.kz, d2x180(pc, sz1, sz2, sz3), V);
    V = fma_(M.kd, Dttt, V);
    V = fma_(M.kn, add_(D1, D2), V);
    real pn;
    if (M.n_relax > 0 && a.relax_scheme == BD_RELAX_SEMI_IMPLICIT) {
        // R_v = a_v (3 p^{n+1} + E) + b_v (4 R1 - R2) with the 2nd-order d3p/dt3 at t_n
        // through p^{n+1}..p^{n-3}; p^{n+1} = Y + (c dt)^2 sum_v R_v solved per cell
        const real E = fma_(real(-10), pc, fma_(real(12), q1, fma_(real(-6), q2, q3)));
        real G = real(0);
        real bv[NRMAX > 0 ? NRMAX : 1];
#pragma unroll
        for (int v = 0; v < NRMAX; ++v) {
            if (v < M.n_relax) {
                bv[v] = mul_(M.rb[v], fma_(real(4), rc[v], -ro[v]));
                const real g = fma_(M.av[v], E, bv[v]);
                G = sizeof(real) == 8 && v == 0 ? g : add_(G, g);
            }
        }
        const real Vn = fma_(M.kr, G, V);                        // num = p + Vn
        pn = add_(pc, fma_(add_(pc, Vn), M.xr, Vn));
#pragma unroll
        for (int v = 0; v < NRMAX; ++v)
            if (v < M.n_relax) ro[v] = fma_(M.av[v], fma_(real(3), pn, E), bv[v]);
    } else {
        real sumR = real(0);
#pragma unroll
        for (int v = 0; v < NRMAX; ++v) {
            if (v < M.n_relax) {
                // W:227: R = 2dt 2 c_v tau Dttt/(2dt^3) / ((2dt+3tau) c^3) + tau (4 R1 - R2)/(2dt+3tau)
                const real rn = fma_(M.av[v], Dttt, mul_(M.rb[v], fma_(real(4), rc[v], -ro[v])));
                ro[v] = rn;
                if constexpr (sizeof(real) == 8) V = fma_(rn, M.kr, V);
                else sumR = add_(sumR, rn);
            }
        }
        if constexpr (sizeof(real) == 4) V = fma_(sumR, M.kr, V);
        pn = add_(pc, V);                                                      // W:234
    }
    return pn;
}

// The same at sound speed c (a grid with a c map).
template <class real, int NRMAX = BD_MAX_RELAX>
__device__ __forceinline__ real cell_update_c(const WvArgs<real>& a, MatConst<real> M, real c, real pc, real sx1, real sx2,
                                              real sx3, real sy1, real sy2, real sy3, const real* w, real q1, real q2,
                                              real q3, real q4, const real* rc, real* ro) {
    cell_coef<real, NRMAX>(a, M, c);
    return cell_update<real, NRMAX>(a, M, pc, sx1, sx2, sx3, sy1, sy2, sy3, w, q1, q2, q3, q4, rc, ro);
}

// One time step of the stencil update.  CTA = TX x TY columns; each thread
// marches along z over a chunk of a.zb planes keeping p^n(iz-3..iz+3) of its
// column in registers.  x/y neighbours come through the read-only cache.
template <class real, int TX, int TY>
__global__ void __launch_bounds__(TX* TY) wv_step_kernel(const WvArgs<real> a, const WvConst<real>* __restrict__ Kp,
                                                           int koff) {
    const int ix = blockIdx.x * TX + threadIdx.x;
    const int iy = blockIdx.y * TY + threadIdx.y;
    if (ix >= a.nx || iy >= a.ny) return;
    const WvConst<real>& K = *Kp;
    const long long step = *a.step_base + koff;
    const int z0 = blockIdx.z * a.zb;
    const int z1 = min(a.nz, z0 + a.zb);
    const int nx = a.nx;
    // neighbour offsets along x and y (mirror at index 0) and which are cells (zero ghosts
    // outside; selected, as weights of 0 and 1 cost six FP64 multiplications a cell)
    int xo[6], yo[6];
    bool xw[6], yw[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int o = k < 3 ? k - 3 : k - 2;   // -3,-2,-1,1,2,3
        int jx = ix + o;
        xw[k] = true;
        if (jx < 0) { if (a.mir_x) jx = -jx; else { jx = ix; xw[k] = false; } }
        if (jx >= nx) { jx = ix; xw[k] = false; }
        xo[k] = jx - ix;
        int jy = iy + o;
        yw[k] = true;
        if (jy < 0) { if (a.mir_y) jy = -jy; else { jy = iy; yw[k] = false; } }
        if (jy >= a.ny) { jy = iy; yw[k] = false; }
        yo[k] = (jy - iy) * a.px;
    }
    const bool col_in_box = ix <= a.xhi && iy <= a.yhi;
    const real sw_xy = a.wx ? mul_(a.wx[ix], a.wy[iy]) : real(1);
    const long long col = (long long)iy * a.px + ix;
    // z window of p^n
    real w[7];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int z = z0 - 3 + k;
        w[k] = (z >= 0 && z < a.nz) ? ld(a.p0 + (long long)z * a.plane + col) : real(0);
    }
    for (int iz = z0; iz < z1; ++iz) {
        {
            const int z = iz + 3;
            w[6] = (z < a.nz) ? ld(a.p0 + (long long)z * a.plane + col) : real(0);
        }
        const long long i = (long long)iz * a.plane + col;
        const bool mur = is_mur_cell(a, ix, iy, iz);
        real pn;
        bool have = false;
        if (iz == a.src_iz) {
            pn = source_value<real>(a, step, (int)col);
            have = true;
        } else if (col_in_box && iz >= a.zlo && iz <= a.zhi) {
            const real pc = w[3];
            const real* P = a.p0 + i;
            const auto nb = [](bool in, const real* p) { const real v = ld(p); return in ? v : real(0); };
            const real sx1 = nb(xw[3], P + xo[3]) + nb(xw[2], P + xo[2]);
            const real sx2 = nb(xw[4], P + xo[4]) + nb(xw[1], P + xo[1]);
            const real sx3 = nb(xw[5], P + xo[5]) + nb(xw[0], P + xo[0]);
            const real sy1 = nb(yw[3], P + yo[3]) + nb(yw[2], P + yo[2]);
            const real sy2 = nb(yw[4], P + yo[4]) + nb(yw[1], P + yo[1]);
            const real sy3 = nb(yw[5], P + yo[5]) + nb(yw[0], P + yo[0]);
            const real q1 = ld(a.p1 + i), q2 = ld(a.p2 + i), q3 = ld(a.p3 + i), q4 = a.p4[i];
            const int m = cell_mat(a, i, iz);
            real rc[BD_MAX_RELAX], ro[BD_MAX_RELAX];
            for (int v = 0; v < K.mat[m].n_relax; ++v) { rc[v] = ld(a.rcur[v] + i); ro[v] = a.rold[v][i]; }
            if (a.cmap) pn = cell_update_c(a, K.mat[m], cell_c(a, K, i, m), pc, sx1, sx2, sx3, sy1, sy2, sy3, w, q1, q2, q3, q4, rc, ro);
            else pn = cell_update(a, K.mat[m], pc, sx1, sx2, sx3, sy1, sy2, sy3, w, q1, q2, q3, q4, rc, ro);
            for (int v = 0; v < K.mat[m].n_relax; ++v) a.rold[v][i] = ro[v];
            if (a.wz) pn = mul_(pn, mul_(sw_xy, a.wz[iz]));
            have = true;
        }
        if (have) {
            const real vm1 = (a.energy_mode == BD_ENERGY_DPDT2) ? ld(a.p1 + i) : real(0);
            a.p4[i] = pn;
            if (!mur) accumulate(a, step, i, pn, vm1);
        }
#pragma unroll
        for (int k = 0; k < 6; ++k) w[k] = w[k + 1];
    }
}

template <class real>
__device__ __forceinline__ real mur_k(real c, real dth) {
    const real a = c * dth;
    return (a - real(1)) / (a + real(1));
}

// One layer of the Mur condition (W:101-133): P^{n+1} of the cell from P^{n+1} (nb)
// and P^n (pj) of its inner neighbour and P^n of the cell.
template <class real>
__device__ __forceinline__ real mur_cell(real pj, real nb, real pi, real c, real dth) {
    return pj + (nb - pi) * mur_k(c, dth);
}

// steps the two-cell kernel and the DFT pass accumulate at once, at most: their
// pressures are p^{n+1}..p^{n-3}; the (dp/dt)^2 energy of a step also needs the level
// two before its own, so it stops at four
constexpr int ACC_STEPS = 5, ACC_DPDT = 4;
constexpr int MUR_MAXL = 8;    // layers of an x+, y+ or z+ face

// The z faces where their layers leave no plane between them (Lzm + L >= nz): the z+
// run then starts on a z- cell, the last z- cell reads the first z+ one, or cells
// belong to both.  One thread takes a column, z- first as a serial launch of W:101-113,
// so the order is fixed; wv_mur_kernel follows with the x+ and y+ faces.  A cell of
// both runs accumulates its final value.
template <class real>
__global__ void __launch_bounds__(128) wv_mur_z_kernel(const WvArgs<real> a, const WvConst<real>* __restrict__ Kp, int koff) {
    const WvConst<real>& K = *Kp;
    const int L = a.L;
    const int cx = a.mur_xp ? a.nx - L : a.nx, cy = a.mur_yp ? a.ny - L : a.ny;   // columns outside the x+ / y+ layers
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (t >= (long long)cx * cy) return;
    const long long step = *a.step_base + koff;
    const long long col = (t / cx) * a.px + t % cx;
    const real* Pn = a.p0;
    real* F = a.p4;
    auto put = [&](long long i, real v, bool last) {
        F[i] = v;
        if (last) accumulate(a, step, i, v, a.energy_mode == BD_ENERGY_DPDT2 ? a.p1[i] : real(0));
    };
    for (int iz = 0; iz < a.Lzm; ++iz) {
        const long long i = (long long)iz * a.plane + col, j = i + a.plane;
        put(i, mur_cell(Pn[j], iz + 1 < a.Lzm ? Pn[j] : F[j], Pn[i], cell_c(a, K, i, cell_mat(a, i, iz)), a.dtdz), iz < a.nz - L);
    }
    for (int iz = a.nz - L; iz < a.nz; ++iz) {
        const long long i = (long long)iz * a.plane + col, j = i - a.plane;
        put(i, mur_cell(Pn[j], F[j], Pn[i], cell_c(a, K, i, cell_mat(a, i, iz)), a.dtdz), true);
    }
}

// The Mur faces of a step in one pass, in the order z-, z+, x+, y+ of a serial
// launch of W:88-135.  Every cell's value follows from P^n and from the cells the
// stencil update wrote, which this kernel only reads (the two z runs do not meet,
// Lzm + L < nz; where they do, wv_mur_z_kernel has formed them): a thread takes one run of
// layers (or one z- cell, whose neighbour is P^n or the source plane) and, where
// the run starts on a cell that an earlier face overwrites, forms that cell's
// value itself.  Three kernels, one per face, whose threads re-read each layer
// they had just written took 26 us a step on 107 x 107 x 401 cells; this one 10.4.
template <class real>
__global__ void __launch_bounds__(128) wv_mur_kernel(const WvArgs<real> a, const WvConst<real>* __restrict__ Kp, int koff) {
    const WvConst<real>& K = *Kp;
    const int L = a.L;
    const int cx = a.mur_xp ? a.nx - L : a.nx, cy = a.mur_yp ? a.ny - L : a.ny;   // columns outside the x+ / y+ layers
    const long long n_zm = a.mur_zm ? (long long)cx * cy * a.Lzm : 0, n_zp = a.mur_zp ? (long long)cx * cy : 0;
    const long long n_x = a.mur_xp ? (long long)cy * a.nz : 0, n_y = a.mur_yp ? (long long)a.nx * a.nz : 0;
    long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    // the previous kernel's fields (a no-op for an ordinary launch); the next step's prologue may start
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (t >= n_zm + n_zp + n_x + n_y) return;
    const long long step = *a.step_base + koff;
    const real* __restrict__ Pn = a.p0;
    real* F = a.p4;
    auto c_at = [&](long long i, int iz) { return cell_c(a, K, i, cell_mat(a, i, iz)); };
    // value of a cell of column `col` (outside the x+ / y+ layers) after the z faces
    auto zval = [&](long long col, int iz) -> real {
        const long long i = (long long)iz * a.plane + col;
        if (a.mur_zm && iz < a.Lzm) {
            const long long j = i + a.plane;
            const real pj = Pn[j];
            return mur_cell(pj, iz + 1 < a.Lzm ? pj : F[j], Pn[i], c_at(i, iz), a.dtdz);   // P_next is p^n in W before the face
        }
        if (a.mur_zp && iz >= a.nz - L) {
            const long long i0 = (long long)(a.nz - L) * a.plane + col;
            real f = F[i0 - a.plane];
            for (int z = a.nz - L; z <= iz; ++z) {
                const long long k = (long long)z * a.plane + col;
                f = mur_cell(Pn[k - a.plane], f, Pn[k], c_at(k, z), a.dtdz);
            }
            return f;
        }
        return F[i];
    };
    // the run: nl cells from i0, `st` apart, the first after a cell of value f
    long long i0 = 0, st = 0;
    int iz = 0, nl = L, dzl = 0;
    real f = real(0), dth = a.dtdx;
    if (t < n_zm) {
        const long long col0 = t % ((long long)cx * cy);
        iz = (int)(t / ((long long)cx * cy));
        const long long col = (col0 / cx) * a.px + col0 % cx;
        i0 = (long long)iz * a.plane + col;
        f = zval(col, iz);
        nl = 0;                                     // a single cell, already formed
    } else if ((t -= n_zm) < n_zp) {
        const long long col = (t / cx) * a.px + t % cx;
        iz = a.nz - L;
        i0 = (long long)iz * a.plane + col;
        st = a.plane;
        dzl = 1;
        dth = a.dtdz;
        f = F[i0 - st];
    } else if ((t -= n_zp) < n_x) {
        const int iy = (int)(t % cy);
        iz = (int)(t / cy);
        const long long col = (long long)iy * a.px + a.nx - L;
        i0 = (long long)iz * a.plane + col;
        st = 1;
        f = zval(col - 1, iz);
    } else {
        t -= n_x;
        const int ix = (int)(t % a.nx);
        iz = (int)(t / a.nx);
        const long long col = (long long)(a.ny - L) * a.px + ix;
        i0 = (long long)iz * a.plane + col;
        st = a.px;
        if (ix < cx) f = zval(col - st, iz);
        else {                                      // the row below is an x+ run
            long long k = (long long)iz * a.plane + (col - st) - (ix - (a.nx - L));
            f = zval(k - (long long)iz * a.plane - 1, iz);
            for (int x = a.nx - L; x <= ix; ++x, ++k) f = mur_cell(Pn[k - 1], f, Pn[k], c_at(k, iz), a.dtdx);
        }
    }
    real v[MUR_MAXL];
    v[0] = f;
    if (nl > 0) {
        real pj = Pn[i0 - st];
#pragma unroll
        for (int l = 0; l < MUR_MAXL; ++l) {
            if (l >= nl) break;
            const long long i = i0 + l * st;
            const real pi = Pn[i];
            f = mur_cell(pj, f, pi, c_at(i, iz + l * dzl), dth);
            v[l] = f;
            pj = pi;
        }
    } else nl = 1;
    const bool do_peak = step >= a.peak_start && step < a.peak_end;
    const bool do_energy = step >= a.energy_start && step < a.energy_end;
#pragma unroll
    for (int l = 0; l < MUR_MAXL; ++l) {
        if (l >= nl) break;
        const long long i = i0 + l * st;
        F[i] = v[l];
        if (do_peak) a.peak[i] = peak_max(v[l], a.peak[i]);
        if (do_energy) a.energy[i] = energy_add(a, a.energy[i], v[l], a.energy_mode == BD_ENERGY_DPDT2 ? a.p1[i] : real(0));
    }
}

template <class real, int VEC>
struct alignas(VEC * sizeof(real)) Cells {
    real v[VEC];
};

// The DFT accumulators of this step and the a.acc_n - 1 before it, whose pressures
// are still in the ring, oldest first: one stream over the DFT planes, 8 B (FP32) a
// frequency and cell read and as much written, 20 B of pressures.  Inside the step
// kernels the accumulators took registers and waited for their loads between two
// barriers, and the Mur faces added theirs one cell at a time.  FP32 107 x 107 x
// 401, ten frequencies on 347 planes: a step that accumulated took 253 us instead of
// 62, one in three or four, and the Mur faces 38 instead of 11 in every step; this
// pass takes 102 us (the copy bandwidth) every fifth.  FP64 is bound by its two FMAs a
// frequency, step and cell.  Cells that no step updates hold zeros and add zeros.
// VEC cells a thread; the twiddles sit in shared memory.
template <class real, int VEC>
__global__ void __launch_bounds__(256) wv_dft_kernel(const WvArgs<real> a, int koff) {
    __shared__ real tw[ACC_STEPS][BD_MAX_DFT][2];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long ds = *a.step_base + koff - a.dft_start;
    unsigned mask = 0;                              // bit m: step - m is inside the window
#pragma unroll
    for (int m = 0; m < ACC_STEPS; ++m)
        if (m < a.acc_n && ds - m >= 0 && ds - m < a.dft_len) mask |= 1u << m;
    if (mask == 0) return;
    for (int e = threadIdx.x; e < ACC_STEPS * a.n_dft; e += blockDim.x) {
        const int m = e / a.n_dft, j = e - m * a.n_dft;
        if (!(mask >> m & 1u)) continue;
        const real* t = a.tw + ((ds - m) * a.n_dft + j) * 2;
        tw[m][j][0] = t[0];
        tw[m][j][1] = t[1];
    }
    __syncthreads();
    const long long n = (long long)(a.dz_hi - a.dz_lo) * a.plane;
    const long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * VEC;
    if (i >= n) return;
    const real* const lev[ACC_STEPS] = {a.p4, a.p0, a.p1, a.p2, a.p3};   // p^{n+1} (written by the step), p^n, ...
    using Vec = Cells<real, VEC>;
    auto at = [](const real* p) { return *reinterpret_cast<const Vec*>(p); };
    Vec x[ACC_STEPS];
#pragma unroll
    for (int m = 0; m < ACC_STEPS; ++m)
        if (mask >> m & 1u) x[m] = at(lev[m] + a.dz_lo * a.plane + i);
    constexpr int G = 4;                            // frequencies whose loads are issued together
    for (int j = 0; j < a.n_dft; j += G) {
        Vec r[G], q[G];
#pragma unroll
        for (int u = 0; u < G; ++u)
            if (j + u < a.n_dft) {
                r[u] = at(a.dre + (j + u) * n + i);
                q[u] = at(a.dim + (j + u) * n + i);
            }
#pragma unroll
        for (int m = ACC_STEPS - 1; m >= 0; --m) {
            if (!(mask >> m & 1u)) continue;
#pragma unroll
            for (int u = 0; u < G; ++u)
                if (j + u < a.n_dft) {
                    const real c = tw[m][j + u][0], s = tw[m][j + u][1];
#pragma unroll
                    for (int k = 0; k < VEC; ++k) {
                        r[u].v[k] = fma_(x[m].v[k], c, r[u].v[k]);
                        q[u].v[k] = fma_(-x[m].v[k], s, q[u].v[k]);
                    }
                }
        }
#pragma unroll
        for (int u = 0; u < G; ++u)
            if (j + u < a.n_dft) {
                *reinterpret_cast<Vec*>(a.dre + (j + u) * n + i) = r[u];
                *reinterpret_cast<Vec*>(a.dim + (j + u) * n + i) = q[u];
            }
    }
}

static __global__ void wv_advance_kernel(long long* step_base, int n) {
    if (threadIdx.x == 0 && blockIdx.x == 0) *step_base += n;
}

// NaN / Inf / amplitude probe of a field: flag bit 1 = non-finite, bit 2 = above limit.
template <class real>
__global__ void wv_probe_kernel(const real* __restrict__ p, long long n, double limit, unsigned* flag) {
    unsigned f = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const real v = p[i];
        if (!isfinite(v)) f |= 1u;
        else if (limit > 0 && fabs((double)v) > limit) f |= 2u;
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if (f && (threadIdx.x & 31) == 0) atomicOr(flag, f);
}

}  // namespace bd
