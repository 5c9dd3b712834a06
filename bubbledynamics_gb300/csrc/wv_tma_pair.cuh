// Two-cells-per-thread variant of the TMA-pipelined Westervelt step (sm_103a).
#pragma once

#include <type_traits>

#include "f32x2.cuh"
#include "wv_tma.cuh"

namespace bd {

// cell_coef()'s coefficients of two cells
template <int NR>
struct Coef2 {
    F2 kxy, kz, kd, kn, kr, xr, av[NR > 0 ? NR : 1], rb[NR > 0 ? NR : 1];
};

// of the cells' materials (the same one twice: one set of loads)
template <int NR>
__device__ __forceinline__ Coef2<NR> coef2(const MatConst<float>& A, const MatConst<float>& B) {
    Coef2<NR> c;
    c.kxy = f2(A.kxy, B.kxy); c.kz = f2(A.kz, B.kz); c.kd = f2(A.kd, B.kd);
    c.kn = f2(A.kn, B.kn); c.kr = f2(A.kr, B.kr); c.xr = f2(A.xr, B.xr);
#pragma unroll
    for (int v = 0; v < NR; ++v) { c.av[v] = f2(A.av[v], B.av[v]); c.rb[v] = f2(A.rb[v], B.rb[v]); }
    return c;
}

// at the sound speeds c of the two cells; a process that a cell's material does not
// have gets zero coefficients, which leave the cell's value as it is without it
template <int NR>
__device__ __forceinline__ Coef2<NR> coef2_c(const WvArgs<float>& a, const MatConst<float>& A, const MatConst<float>& B, F2 c) {
    Coef2<NR> k;
    float cx, cy;
    f2_split(c, cx, cy);
    const F2 c2 = f2_mul(c, c), ic = f2(div_(1.0f, cx), div_(1.0f, cy)), ic2 = f2_mul(ic, ic);
    k.kxy = f2_mul(c2, f2(a.kxy180));
    k.kz = f2_mul(c2, f2(a.kz180));
    k.kd = f2_mul(f2(A.delta_2dt, B.delta_2dt), ic2);
    k.kn = f2_mul(f2(A.beta2_rho, B.beta2_rho), ic2);
    k.kr = f2_mul(c2, f2(a.dt2));
    k.xr = f2(0.0f);
    if (NR > 0) {
        if (a.relax_scheme == BD_RELAX_SEMI_IMPLICIT) {
            const F2 ic3 = f2_mul(ic2, ic);
            F2 sa = f2(0.0f);
#pragma unroll
            for (int v = 0; v < NR; ++v) {
                // ptxas leaves this product alone, which is used again (the bits of two processes
                // are tested against the plain kernel's); f2_mul1 costs 0.25 % of a step
                k.av[v] = f2_mul(f2(A.ra_num[v], B.ra_num[v]), ic3);
                sa = f2_add(sa, k.av[v]);
            }
            const F2 x = f2_mul(f2_mul(f2(3.0f), k.kr), sa), d = f2_sub(f2(1.0f), x);
            float x0, x1, d0, d1;
            f2_split(x, x0, x1);
            f2_split(d, d0, d1);
            k.xr = f2(div_(x0, d0), div_(x1, d1));
        } else {
#pragma unroll
            for (int v = 0; v < NR; ++v) k.av[v] = f2_mul(f2_mul(f2(A.ra_num[v], B.ra_num[v]), ic2), ic);
        }
#pragma unroll
        for (int v = 0; v < NR; ++v) k.rb[v] = f2(A.rb[v], B.rb[v]);
    }
    return k;
}

__device__ __forceinline__ F2 d2x180(F2 pc, F2 s1, F2 s2, F2 s3) {
    return f2_fma(f2(2.0f), s3, f2_fma(f2(-27.0f), s2, f2_fma(f2(270.0f), s1, f2_mul(f2(-490.0f), pc))));
}

// cell_update() of two cells: the same operations, so the same bits.  relax: either
// cell's material has relaxation processes.
template <int NR>
__device__ __forceinline__ F2 cell_update2(const WvArgs<float>& a, const Coef2<NR>& k, bool relax, F2 sx1, F2 sx2, F2 sx3,
                                           F2 sy1, F2 sy2, F2 sy3, const F2* w, F2 q1, F2 q2, F2 q3, F2 q4, const F2* rc,
                                           F2* ro) {
    const F2 pc = w[3];
    const F2 Dxx = d2x180(pc, sx1, sx2, sx3);
    const F2 Dyy = d2x180(pc, sy1, sy2, sy3);
    const F2 Dzz = d2x180(pc, f2_add(w[4], w[2]), f2_add(w[5], w[1]), f2_add(w[6], w[0]));
    const F2 Dttt = f2_fma(f2(3.0f), q4, f2_fma(f2(-14.0f), q3, f2_fma(f2(24.0f), q2, f2_fma(f2(-18.0f), q1, f2_mul(f2(5.0f), pc)))));
    const F2 s3 = f2_fma(f2(3.0f), pc, f2_fma(f2(-4.0f), q1, q2));
    const F2 D1 = f2_mul1(f2_mul(s3, s3), f2(0.25f));
    // 4 p2 is exact, so 4 p2 - p3 takes the one rounding of the fma
    const F2 D2 = f2_mul1(pc, f2_fma(f2(2.0f), pc, f2_fma(f2(-5.0f), q1, f2_sub(f2_mul(f2(4.0f), q2), q3))));
    F2 V = f2_sub(pc, q1);
    V = f2_fma(k.kxy, f2_add(Dxx, Dyy), V);
    V = f2_fma(k.kz, Dzz, V);
    V = f2_fma(k.kd, Dttt, V);
    V = f2_fma(k.kn, f2_add(D1, D2), V);
    if (NR == 0 || !relax) return f2_add(pc, V);
    if (a.relax_scheme == BD_RELAX_SEMI_IMPLICIT) {
        const F2 E = f2_fma(f2(-10.0f), pc, f2_fma(f2(12.0f), q1, f2_fma(f2(-6.0f), q2, q3)));
        F2 G = f2(0.0f), bv[NR > 0 ? NR : 1];
#pragma unroll
        for (int v = 0; v < NR; ++v) {
            bv[v] = f2_mul(k.rb[v], f2_sub(f2_mul(f2(4.0f), rc[v]), ro[v]));
            G = f2_add(G, f2_fma(k.av[v], E, bv[v]));
        }
        const F2 Vn = f2_fma(k.kr, G, V);
        const F2 pn = f2_add(pc, f2_fma(f2_add(pc, Vn), k.xr, Vn));
#pragma unroll
        for (int v = 0; v < NR; ++v) ro[v] = f2_fma(k.av[v], f2_fma(f2(3.0f), pn, E), bv[v]);
        return pn;
    }
    F2 sumR = f2(0.0f);
#pragma unroll
    for (int v = 0; v < NR; ++v) {
        ro[v] = f2_fma(k.av[v], Dttt, f2_mul(k.rb[v], f2_sub(f2_mul(f2(4.0f), rc[v]), ro[v])));
        sumR = f2_add(sumR, ro[v]);
    }
    return f2_add(pc, f2_fma(sumR, k.kr, V));
}

// One Westervelt step, TMA-pipelined, two adjacent x cells per thread: the
// same pipeline as wv_tma_kernel (p^n plane ring with halo, pointwise ring,
// bounded mbarrier waits), with every tile and global access of a thread one
// 8- or 16-byte pair (nx must be even, which a 16-byte row pitch gives) and a
// pointwise ring of NQ slots (NQ >= ZU), so that a shallower ring leaves room
// for more CTAs per SM.  The CTA has TX/2 x TY threads; the launch bound asks
// for 24 resident warps per SM (at most 85 registers a thread).  The cell update is
// cell_update(), so the results are the plain kernel's bits.
//
// ACC: which accumulators the step may touch.  ACC_PE: peak and energy (each still
// gated by its window); ACC_PEAK: only the peak map (the energy tile is not loaded,
// 4 B less per cell); ACC_NONE: none (outside the windows, or a step that a later
// one accumulates for: neither tile is loaded, 8 B less per cell).  Planes on which
// every cell of the tile is updated take a copy of the cell code without the
// per-cell conditions.
template <int TX, int TY, int NREL, int ZU, int FL, int NQ, int ACC = ACC_PE>
__global__ void __launch_bounds__(TX* TY / 2, 1536 / (TX * TY)) wv_tma_pair_kernel(const WvArgs<float> a,
                                                                 const WvConst<float>* __restrict__ Kp, int koff,
                                                                 const __grid_constant__ TmaMaps maps,
                                                                 unsigned* __restrict__ err) {
    using real = float;
    constexpr int CX = 2;
    static_assert(NREL >= 0 && NREL <= 2, "compiled for the relaxation count");
    static_assert(NQ >= ZU, "the pointwise ring holds a whole group of planes");
    constexpr int NRMAX = NREL, nrel = NREL;
    using L = TmaLayout<real, TX, TY, NRMAX, NQ>;
    constexpr int TXT = TX / CX;                   // thread columns
    constexpr int NT = TXT * TY;                   // threads
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ MatConst<real> sK[BD_MAX_MATERIALS];
    // FL >= 0: bit 0 = one material everywhere, bit 1 = per-cell c map (compile-time);
    // FL_NOC = no c map, materials read from the arguments; FL = -1: both read from them
    const bool has_c = FL >= 0 ? (FL & 2) != 0 : a.cmap != nullptr;
    real* Pring = reinterpret_cast<real*>(smem);
    unsigned char* Qring = smem + TMA_NP * L::PSLOT;
    uint64_t* barP = reinterpret_cast<uint64_t*>(Qring + NQ * L::QS);
    uint64_t* barQ = barP + TMA_NP;

    const int tx = threadIdx.x, tyt = threadIdx.y;
    const int tid = tyt * TXT + tx;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    // every other step marches from the high end (chunks and planes), so that it
    // starts on what the step before it left in L2; the z stencil is symmetric, so
    // the bits are the same
    const int bz = a.rev ? gridDim.z - 1 - blockIdx.z : blockIdx.z;
    const int z0 = bz * a.zb;
    const int z1 = min(a.nz, z0 + a.zb);
    const int zbn = z1 - z0;
    const int zf = a.rev ? z1 - 1 : z0, zd = a.rev ? -1 : 1;   // first plane, direction
    auto zof = [&](int r) { return zf + zd * r; };             // r-th plane of the march

    for (int e = tid; e < (int)(BD_MAX_MATERIALS * sizeof(MatConst<real>) / 4); e += NT)
        reinterpret_cast<unsigned*>(sK)[e] = reinterpret_cast<const unsigned*>(Kp)[e];

    auto pslot = [&](int q) {
        return reinterpret_cast<real*>(reinterpret_cast<unsigned char*>(Pring) + (q % TMA_NP) * L::PSLOT);
    };
    auto qslot = [&](int r) { return Qring + (r % NQ) * L::QS; };

    // producer (thread 0): march plane q - 3 of p^n, march plane r of the pointwise tiles
    auto issueP = [&](int q) {
        if (q > zbn + 5) return;
        const int plane = zof(q - 3);
        uint64_t* bar = &barP[q % TMA_NP];
        if (plane < 0 || plane >= a.nz) { mbar_arrive(bar); return; }   // read as zeros, nothing to copy
        mbar_expect_tx(bar, L::PW * L::PH * (unsigned)sizeof(real));
        tma_load_3d(pslot(q), &maps.p0, bar, x0 - 4, y0 - 3, plane);
    };
    auto issueQ = [&](int r) {
        if (r >= zbn) return;
        const int plane = zof(r);
        uint64_t* bar = &barQ[r % NQ];
        unsigned char* q = qslot(r);
        constexpr int acc_tiles = ACC == ACC_PE ? 2 : ACC == ACC_PEAK ? 1 : 0;
        mbar_expect_tx(bar, (unsigned)((4 + acc_tiles + 2 * nrel) * L::QTB + (has_c ? L::QTF : 0) +
                                       (a.mat_tile ? L::QT : 0)));
        for (int k = 0; k < 4; ++k) tma_load_3d(q + k * L::QTB, &maps.q[k], bar, x0, y0, plane);
        for (int v = 0; v < nrel; ++v) {
            tma_load_3d(q + (4 + v) * L::QTB, &maps.rc[v], bar, x0, y0, plane);
            tma_load_3d(q + (4 + NRMAX + v) * L::QTB, &maps.ro[v], bar, x0, y0, plane);
        }
        if constexpr (ACC != ACC_NONE) tma_load_3d(q + L::K_PEAK * L::QTB, &maps.peak, bar, x0, y0, plane);
        if constexpr (ACC == ACC_PE)
            tma_load_3d(q + L::K_ENERGY * L::QTB, &maps.energy, bar, x0, y0, plane);
        if (has_c) tma_load_3d(q + L::NQR * L::QTB, &maps.cmap, bar, x0, y0, plane);
        if (a.mat_tile) tma_load_3d(q + L::NQR * L::QTB + L::QTF, &maps.mat, bar, x0, y0, plane);
    };

    if (tid == 0) {
        for (int s = 0; s < TMA_NP; ++s) mbar_init(&barP[s], 1);
        for (int s = 0; s < NQ; ++s) mbar_init(&barQ[s], 1);
        mbar_fence_init();
    }
    __syncthreads();
    // Programmatic dependent launch: with the attribute set by the host, the
    // prologue above (material constants, barrier set-up) overlaps the tail of
    // the previous step's grid; the fields and the step counter it wrote are
    // read only after this wait (a no-op for an ordinary launch).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const long long step = *a.step_base + koff;
    if (tid == 0) {
        for (int q = 0; q < TMA_NP; ++q) issueP(q);
        for (int r = 0; r < NQ; ++r) issueQ(r);
    }
    auto waitP = [&](int q) { mbar_wait(&barP[q % TMA_NP], (unsigned)((q / TMA_NP) & 1), err); };
    auto waitQ = [&](int r) { mbar_wait(&barQ[r % NQ], (unsigned)((r / NQ) & 1), err); };

    // this thread's two cells: row tyt, columns CX * tx and CX * tx + 1 of the tile
    const int ix = x0 + CX * tx, iy = y0 + tyt;
    const int own = (tyt + 3) * L::PW + CX * tx + 4, k = tyt * TX + CX * tx;
    const int col = iy * a.px + ix;                // column index iy * px + ix (a plane has < 2^31 cells)
    bool active[CX], inbox[CX], murxy[CX];
#pragma unroll
    for (int c = 0; c < CX; ++c) {
        active[c] = ix + c < a.nx && iy < a.ny;
        inbox[c] = ix + c <= a.xhi && iy <= a.yhi;
        murxy[c] = (a.mur_yp && iy >= a.ny - a.L) || (a.mur_xp && ix + c >= a.nx - a.L);
    }
    const F2 swxy = f2(a.wx && active[0] ? mul_(a.wx[ix], a.wy[iy]) : 1.0f, a.wx && active[1] ? mul_(a.wx[ix + 1], a.wy[iy]) : 1.0f);
    F2 w[7];                                       // p^n of the two cells, by plane of the march
    auto load_w = [&](const real* tile, bool in) -> F2 { return in ? ld2(tile + own) : f2(0.0f); };
#pragma unroll
    for (int k = 0; k < 6; ++k) {                  // the first plane and three on either side, but the last
        waitP(k);
        const int plane = zof(k - 3);
        w[k] = load_w(pslot(k), plane >= 0 && plane < a.nz);
    }
    // every cell of the tile inside the grid and the update box and on no x / y
    // Mur layer: the planes of the tile inside the z range take the code without
    // per-cell conditions (the same operations on every cell, so the same bits)
    const bool mine = active[0] && active[1] && inbox[0] && inbox[1] && !murxy[0] && !murxy[1];
    const bool tile_fast = __syncthreads_and(mine) != 0;   // also: the slots of the three planes before the first are free again
    if (tid == 0)
        for (int q = TMA_NP; q < TMA_NP + 3; ++q) issueP(q);

    const bool fix_x = a.mir_x && x0 == 0, fix_y = a.mir_y && y0 == 0;
    // Deferred accumulation: a step's peak and energy terms follow from its
    // pressure alone, which stays in the ring, so one step in four or five adds its
    // own terms and those of the steps since the last such step, oldest first (the
    // same operations on every accumulator, so the same bits), and the steps between
    // leave the accumulators alone.  Bit m: step - m is inside the window.
    const int acc_n = ACC == ACC_NONE ? 0 : a.acc_n;
    unsigned peak_m = 0, energy_m = 0;
    if constexpr (ACC != ACC_NONE) {
#pragma unroll
        for (int m = 0; m < ACC_STEPS; ++m) {
            const long long t = step - m;
            if (m >= acc_n) continue;
            if (t >= a.peak_start && t < a.peak_end) peak_m |= 1u << m;
            if (t >= a.energy_start && t < a.energy_end) energy_m |= 1u << m;
        }
    }
    const bool do_peak = peak_m != 0;
    const bool do_energy = ACC == ACC_PE && energy_m != 0;
    const bool single_mat = FL >= 0 && FL != FL_NOC ? (FL & 1) != 0 : (!a.matmap && !a.plane_mat);
    const bool dpdt = a.energy_mode == BD_ENERGY_DPDT2;

    for (int rg = 0; rg < zbn; rg += ZU) {
        // the last planes of this CTA: the next step's grid may start its prologue
        if (rg + ZU >= zbn) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
    for (int u = 0; u < ZU; ++u) {
        const int r = rg + u;
        if (r >= zbn) break;
        const int iz = zof(r);
        const int qc = r + 3;                      // stencil plane
        waitP(qc + 3);
        w[6] = load_w(pslot(qc + 3), (unsigned)zof(r + 3) < (unsigned)a.nz);
        real* T = pslot(qc);
        if (fix_x || fix_y) {                      // mirror planes x = 0 / y = 0 (W:176-200)
            if (fix_x)
                for (int e = tid; e < L::PH * 3; e += NT) {
                    const int row = e / 3, k = e % 3 + 1;
                    T[row * L::PW + 4 - k] = T[row * L::PW + 4 + k];
                }
            __syncthreads();
            if (fix_y)
                for (int e = tid; e < L::PW * 3; e += NT) {
                    const int cc = e % L::PW, k = e / L::PW + 1;
                    T[(3 - k) * L::PW + cc] = T[(3 + k) * L::PW + cc];
                }
            // TMA refills this slot later: order these ordinary stores before that copy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
        }
        waitQ(r);
        const unsigned char* Qs = qslot(r);
        const real* q1t = reinterpret_cast<const real*>(Qs);
        const real* q2t = q1t + L::QT;
        const real* q3t = q2t + L::QT;
        const real* q4t = q3t + L::QT;
        const real* pkt = reinterpret_cast<const real*>(Qs + L::K_PEAK * L::QTB);
        const real* ent = reinterpret_cast<const real*>(Qs + L::K_ENERGY * L::QTB);
        const float* ct = reinterpret_cast<const float*>(Qs + L::NQR * L::QTB);
        const uint8_t* mtl = reinterpret_cast<const uint8_t*>(Qs + L::NQR * L::QTB + L::QTF);
        const bool src_plane = iz == a.src_iz;
        const bool zin = iz >= a.zlo && iz <= a.zhi && !src_plane;
        const bool murz = (a.mur_zp && iz >= a.nz - a.L) || (a.mur_zm && iz < a.Lzm);
        const real wzi = a.wz ? a.wz[iz] : real(1);
        const int mplane = single_mat ? 0 : (a.plane_mat ? __ldg(a.plane_mat + iz) : 0);
        const long long zoff = (long long)iz * a.plane;
        real* const p4z = a.p4 + zoff;
        real* const pkz = a.peak + zoff;
        real* const enz = a.energy + zoff;
        real* rolz[NRMAX > 0 ? NRMAX : 1];
#pragma unroll
        for (int v = 0; v < NRMAX; ++v) rolz[v] = a.rold[v] + zoff;
        // FAST: every cell of the tile is updated and accumulates on this plane
        auto cells = [&](auto fast_tag) {
        constexpr bool FAST = decltype(fast_tag)::value;
        {
            if (!FAST && !active[0]) return;       // a thread's first cell is the last to leave the grid
            const F2 q1p = ld2(q1t + k);
            F2 pnp, ro[NRMAX > 0 ? NRMAX : 1];
            const F2 q2 = ld2(q2t + k), q3 = ld2(q3t + k), q4 = ld2(q4t + k);
            bool have[CX] = {FAST, FAST};
            int nrx[CX] = {0, 0};                  // relaxation processes of the cells' materials
            if (!FAST && src_plane) {
                pnp = f2(source_value<real>(a, step, col), source_value<real>(a, step, col + 1));
                have[0] = have[1] = true;
            } else if (FAST || zin) {
                // x and y neighbours from the plane tile
                const real* cp = T + own;
                constexpr int W = L::PW;
                float e[10];                       // x offsets -4 .. +5 from the first cell
                const F2 xm = ld2(cp - 2), xp = ld2(cp + 2);
                f2_split(ld2(cp - 4), e[0], e[1]);
                f2_split(xm, e[2], e[3]);
                f2_split(w[3], e[4], e[5]);
                f2_split(xp, e[6], e[7]);
                f2_split(ld2(cp + 4), e[8], e[9]);
                const F2 sx1 = f2(add_(e[5], e[3]), add_(e[6], e[4])), sx2 = f2_add(xp, xm),
                         sx3 = f2(add_(e[7], e[1]), add_(e[8], e[2]));
                const F2 sy1 = f2_add(ld2(cp + W), ld2(cp - W)), sy2 = f2_add(ld2(cp + 2 * W), ld2(cp - 2 * W)),
                         sy3 = f2_add(ld2(cp + 3 * W), ld2(cp - 3 * W));
                F2 rc[NRMAX > 0 ? NRMAX : 1];
#pragma unroll
                for (int v = 0; v < NRMAX; ++v) {
                    rc[v] = ld2(reinterpret_cast<const real*>(Qs + (4 + v) * L::QTB) + k);
                    ro[v] = ld2(reinterpret_cast<const real*>(Qs + (4 + NRMAX + v) * L::QTB) + k);
                }
                int m0 = 0, m1 = 0;
                if constexpr (!(FL >= 0 && (FL & 1))) {
                    m0 = m1 = mplane;
                    if (a.matmap) {
                        m0 = a.mat_tile ? (int)mtl[k] : (int)__ldg(a.matmap + zoff + col);
                        m1 = a.mat_tile ? (int)mtl[k + 1] : active[1] ? (int)__ldg(a.matmap + zoff + col + 1) : m0;
                    }
                }
                const MatConst<float>&A = sK[m0], &B = sK[m1];
                const int nr0 = A.n_relax, nr1 = B.n_relax;
                const Coef2<NRMAX> cf = has_c ? coef2_c<NRMAX>(a, A, B, ld2(ct + k)) : coef2<NRMAX>(A, B);
                pnp = cell_update2<NRMAX>(a, cf, NRMAX > 0 && (nr0 > 0 || nr1 > 0), sx1, sx2, sx3, sy1, sy2, sy3, w, q1p, q2,
                                          q3, q4, rc, ro);
                if (a.wz) pnp = f2_mul(pnp, f2_mul(swxy, f2(wzi)));
                if (!FAST) { have[0] = inbox[0]; have[1] = inbox[1]; }
                nrx[0] = have[0] ? nr0 : 0;
                nrx[1] = have[1] ? nr1 : 0;
            }
            float pn[CX];
            f2_split(pnp, pn[0], pn[1]);
            // stores: a pair access where both cells take part, else per cell
            if (FAST || (have[0] && have[1])) st2(p4z + col, pnp);
            else
#pragma unroll
                for (int c = 0; c < CX; ++c)
                    if (have[c]) p4z[col + c] = pn[c];
            // relaxation variables of the processes of each cell's material (as in cell_update)
#pragma unroll
            for (int v = 0; v < NRMAX; ++v) {
                if (v < nrx[0] && v < nrx[1]) st2(rolz[v] + col, ro[v]);
                else if (v < nrx[0] || v < nrx[1]) {
                    float r0, r1;
                    f2_split(ro[v], r0, r1);
                    if (v < nrx[0]) rolz[v][col] = r0;
                    if (v < nrx[1]) rolz[v][col + 1] = r1;
                }
            }
            bool acc[CX];
#pragma unroll
            for (int c = 0; c < CX; ++c) acc[c] = FAST || (have[c] && !(murz || murxy[c]));
            const bool acc_pair = acc[0] && acc[1];
            if constexpr (ACC != ACC_NONE) {
            // pressures of the steps to accumulate, newest first, and what precedes the oldest
            const F2 lev[ACC_STEPS + 1] = {pnp, w[3], q1p, q2, q3, q4};
            if (do_peak) {
                float pk[CX];
                f2_split(ld2(pkt + k), pk[0], pk[1]);
#pragma unroll
                for (int m = ACC_STEPS - 1; m >= 0; --m) {
                    if (!(peak_m >> m & 1u)) continue;
                    float v[CX];
                    f2_split(lev[m], v[0], v[1]);
#pragma unroll
                    for (int c = 0; c < CX; ++c) {
                        const real av = fabs(v[c]);
                        pk[c] = av > pk[c] ? av : pk[c];
                    }
                }
                if (acc_pair) st2(pkz + col, f2(pk[0], pk[1]));
                else
#pragma unroll
                    for (int c = 0; c < CX; ++c)
                        if (acc[c]) pkz[col + c] = pk[c];
            }
            if (do_energy) {
                F2 ev = ld2(ent + k);
                const real h = mul_(real(2.0), a.dt);
#pragma unroll
                for (int m = ACC_STEPS - 1; m >= 0; --m) {
                    if (!(energy_m >> m & 1u)) continue;
                    F2 d = lev[m];
                    if (dpdt) {                    // p^{t+1} - p^{t-1} (at most ACC_DPDT steps, so lev[m + 2] exists)
                        float v0, v1, u0, u1;
                        f2_split(lev[m], v0, v1);
                        f2_split(lev[m + 2 <= ACC_STEPS ? m + 2 : ACC_STEPS], u0, u1);
                        d = f2(div_(add_(v0, -u0), h), div_(add_(v1, -u1), h));
                    }
                    ev = f2_add(ev, f2_mul1(f2_mul(d, d), f2(a.dt)));
                }
                if (acc_pair) st2(enz + col, ev);
                else {
                    float e0, e1;
                    f2_split(ev, e0, e1);
                    if (acc[0]) enz[col] = e0;
                    if (acc[1]) enz[col + 1] = e1;
                }
            }
            }
        }
        };
        if (tile_fast && zin && !murz) cells(std::true_type{});
        else cells(std::false_type{});
#pragma unroll
        for (int j = 0; j < 6; ++j) w[j] = w[j + 1];
    }
        __syncthreads();                           // everyone is done with this round's planes and their tiles
        if (tid == 0) {
#pragma unroll
            for (int u = 0; u < ZU; ++u) {
                issueP(rg + u + 3 + TMA_NP);
                issueQ(rg + u + NQ);
            }
        }
    }
}

}  // namespace bd
