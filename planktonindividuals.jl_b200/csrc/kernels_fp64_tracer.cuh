// FP64 plain form: the tracer update (Biogeochemistry/tracer_update.jl:22-43) in two kernels and the
// halo fill.
//
//   k64_plk     particle terms of the occupied cells, in the order of a sequential reference run
//   k64_xy      x and y sweeps of DST3FL: a warp walks rows of one tracer
//   k64_ztail   z sweep walking down columns, then diffusion, sinking, forcing, boundary fluxes,
//               particle terms and apply_tendency!
//   k64_halo    fill_halo_tracer! in one pass
//
// Every value is the IEEE expression of the reference in its operation order, so the results are the
// oracle's bits. What is saved is work that cannot change a value:
//  - of the two one-sided terms of adv_flux (Advection/DST3FL.jl), ½(tr + |tr|)·(upwind) +
//    ½(tr − |tr|)·(downwind), one has a zero factor: it is left out unless a non-finite tracer value
//    reaches only that term;
//  - the limiter's third argument θ(1 − cfl)/(cfl + 1e-20) is only divided out when a product does
//    not already show it to be negative or above the other two;
//  - what does not depend on the tracer (Courant number, d₀, d₁, transports, ΔT/volume) is formed
//    once per face in shared memory for the 14 tracer warps of a block.
#pragma once

#include "kernels_fp64.cuh"

namespace pib {

// per-face coefficients as planes of a shared array [plane][row][lane]
enum { FC_D0 = 0, FC_D1, FC_OMC, FC_CPE, FC_H, FC_FTR, FC_DTV, FC_N };
#define FB_ZERO 16u      // mask byte: bits 0-3 the landmask of the four stencil points, 4: no flux

__device__ __forceinline__ double side_factor(const FaceCoef& f) {
    // the factor of the upwind side; NaN where the other factor would not be a zero
    const double h = f.hp > 0.0 ? f.hp : f.hm;
    return h - h == 0.0 ? h : h - h;
}
__device__ __forceinline__ void put_face(double* s, int stride, const FaceCoef& f) {
    s[FC_D0 * stride] = f.d0c; s[FC_D1 * stride] = f.d1c; s[FC_OMC * stride] = f.omc; s[FC_CPE * stride] = f.cpe;
    s[FC_H * stride] = side_factor(f);
}
// psi_c with the quotient left out where it decides nothing: a quotient of p = θ(1 − cfl) that is
// negative gives zero, one above 1.0000001·m (a margin far above the rounding of the product) leaves m
__device__ __forceinline__ double psi_s(const double* s, int stride, double dnum, double d0) {
    const double th = theta(dnum, d0);
    const double m = jl_min(1.0, s[FC_D0 * stride] + s[FC_D1 * stride] * th);
    const double p = th * s[FC_OMC * stride], cpe = s[FC_CPE * stride];
    if (p < 0.0) return 0.0;
    if (p > 1.0000001 * (m * cpe)) return jl_max(0.0, m);
    return jl_max(0.0, jl_min(m, p / cpe));
}
__device__ __forceinline__ bool finite64(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// flux_xy_c from c[f-2], c[f-1], c[f], c[f+1] (flux_z_c is the same with the four points in reverse)
template <bool LM>
__device__ __forceinline__ double flux_s(const double* s, int stride, double cm2, double cm1, double c0, double cp1, unsigned mb) {
    const int lm2 = mb & 1u, lm1 = mb >> 1 & 1u, l0 = mb >> 2 & 1u, lp1 = mb >> 3 & 1u;
    auto mk = [](double x, int a, int b) { return LM ? jl_mulb(jl_mulb(x, a), b) : x; };
    const double h = s[FC_H * stride];
    const bool pos = h > 0.0;
    const double d0 = mk(c0 - cm1, l0, lm1);
    const double dn = pos ? mk(cm1 - cm2, lm1, lm2) : mk(cp1 - c0, lp1, l0);
    const double ps = psi_s(s, stride, dn, d0);
    const double F = h * (pos ? cm1 + ps * d0 : c0 - ps * d0);
    // (a water cell beyond makes d0, and with it F, not finite; one on land is masked out of d0)
    if (!finite64(pos ? cp1 : cm2) || (LM && !finite64(pos ? c0 : cm1))) {
        const double dx = pos ? mk(cp1 - c0, lp1, l0) : mk(cm1 - cm2, lm1, lm2);
        const double px = psi_s(s, stride, dx, d0);
        return F + 0.0 * (pos ? c0 - px * d0 : cm1 + px * d0);
    }
    return F;
}

// ------------------------------------------------------------------------------------------
// particle terms (plk) of every occupied interior cell, by tracer in `plk` (14 × G); cells without
// individuals are not written and not read
// ------------------------------------------------------------------------------------------
struct PlkArgs {
    DGrid g;
    long long C;
    const uint32_t* off;
    const uint32_t* gid_sorted;
    const uint8_t* evk;
    const double* loss;
    const double* contrib;
    double* plk;
    const uint32_t* ncrowd;  // cells of more than CROWD_CELL individuals, listed in crowd
    const uint32_t* crowd;
    unsigned cell_blocks;    // blocks of a thread per cell; those after them take the listed cells
    const uint32_t* err;
};
// A crowded cell by a warp: the entries' contributions are loaded 32 entries at a time, and lane q adds its
// tracer's in the order of the entries (the sums of a sequential run), the five of calc_consume! from
// shared memory. A thread alone waited for the loads of each entry: 1.6 million individuals in 16,384 cells
// 186 µs, in 4,096 717, in 256 10,669; so 37, 35 and 327. A cell of up to CROWD_CELL keeps its thread: many
// cells hide the waits of one another.
template <bool IRON>
__device__ __forceinline__ void plk_crowded(const PlkArgs& a, uint32_t c, double* sh) {
    const int lane = threadIdx.x & 31;
    // lane q: tracer, and column of its loss (-1: none); lanes 0-4 are the columns of contrib
    const int NT = IRON ? 12 : 10, LW = IRON ? 10 : 6;
    const int tq[10] = { PI_DIC, PI_DOC, PI_NH4, PI_NO3, PI_PO4, PI_DON, PI_DOP, PI_POC, PI_PON, PI_POP };
    const int lq[10] = { -1, 0, -1, -1, -1, 1, 2, 3, 4, 5 };
    const int ti[12] = { PI_DIC, PI_NH4, PI_NO3, PI_PO4, PI_DFe, PI_DOC, PI_DON, PI_DOP, PI_POC, PI_PON, PI_POP, PI_PFe_bio };
    const int li[12] = { -1, 0, 1, -1, 5, 2, 3, 4, 6, 7, 8, 9 };
    int tr = 0, lc = -1;
#pragma unroll
    for (int q = 0; q < NT; ++q)
        if (lane == q) { tr = IRON ? ti[q] : tq[q % 10]; lc = IRON ? li[q] : lq[q % 10]; }
    double acc = 0.0;
    const uint32_t p0 = a.off[c], p1 = a.off[c + 1];
    for (uint32_t p = p0; p < p1;) {
        const uint32_t s = a.gid_sorted[p] / (uint32_t)a.C;
        // the species' run, and whether any of it was lost
        uint32_t e = p, any = 0u;
        for (;;) {
            const bool in = e + lane < p1 && a.gid_sorted[e + lane] / (uint32_t)a.C == s;
            any |= __reduce_or_sync(0xffffffffu, in ? (unsigned)a.evk[e + lane] : 0u);
            const unsigned mk = __ballot_sync(0xffffffffu, in);
            if (mk != 0xffffffffu) { e += __ffs(~mk) - 1; break; }
            e += 32;
        }
        for (uint32_t pass = 1; pass <= 2; ++pass) {
            if (!(any & pass)) continue;
            for (uint32_t x = p; x < e; x += 32)
                for (unsigned mk = __ballot_sync(0xffffffffu, x + lane < e && a.evk[x + lane] == pass); mk; mk &= mk - 1u)
                    if (lc >= 0) acc += a.loss[(long long)(x + __ffs(mk) - 1) * LW + lc];
        }
        double r[5];
        auto load = [&](uint32_t x) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const long long at = (long long)x * 5 + q * 32 + lane;
                r[q] = at < (long long)e * 5 ? a.contrib[at] : 0.0;
            }
        };
        load(p);
        for (uint32_t x = p; x < e; x += 32) {
#pragma unroll
            for (int q = 0; q < 5; ++q) sh[q * 32 + lane] = r[q];
            __syncwarp();
            if (x + 32 < e) load(x + 32);
            const int n = min(32u, e - x);
            if (lane < 5) {
#pragma unroll 8
                for (int y = 0; y < n; ++y) acc += sh[y * 5 + lane];
            }
            __syncwarp();
        }
        p = e;
    }
    if (lane < NT) a.plk[tr * a.g.G + c] = acc;
}
template <bool IRON>
__global__ void __launch_bounds__(128) k64_plk(PlkArgs a) {
    __shared__ double sh[4][160];
    const DGrid& g = a.g;
    if (blockIdx.x >= a.cell_blocks) {
        const int wid = threadIdx.x >> 5;
        const uint32_t n = *a.ncrowd;                     // (beside the error word: both loads are on the way)
        if (*a.err & PI_DEVERR_CAPACITY) return;
        for (uint32_t t = (blockIdx.x - a.cell_blocks) * 4 + wid; t < n; t += (gridDim.x - a.cell_blocks) * 4)
            plk_crowded<IRON>(a, a.crowd[t], sh[wid]);
        return;
    }
    if (*a.err & PI_DEVERR_CAPACITY) return;
    const long long V = (long long)g.Nx * g.Ny * g.Nz, t = (long long)blockIdx.x * 128 + threadIdx.x;
    if (t >= V) return;
    const int i = (int)(t % g.Nx), r = (int)(t / g.Nx);
    const int q = gidx(g, i + 1 + g.Hx, r % g.Ny + 1 + g.Hy, r / g.Ny + 1 + g.Hz);
    const uint32_t p0 = a.off[q], p1 = a.off[q + 1];
    if (p0 == p1 || p1 - p0 > CROWD_CELL) return;
    double DIC = 0.0, NH4 = 0.0, NO3 = 0.0, PO4 = 0.0, DOC = 0.0, DON = 0.0, DOP = 0.0, POC = 0.0, PON = 0.0, POP = 0.0;
    double DFe = 0.0, PFe = 0.0;                 // IronEnergyMode only
    uint32_t p = p0;
    while (p < p1) {
        const uint32_t s = a.gid_sorted[p] / (uint32_t)a.C;
        // the species' run, and whether any of it was lost
        uint32_t e = p;
        unsigned any = 0;
        while (e < p1 && a.gid_sorted[e] / (uint32_t)a.C == s) any |= a.evk[e++];
        for (int pass = 1; pass <= 2 && any; ++pass)
            for (uint32_t x = p; x < e; ++x)
                if (a.evk[x] == pass) {
                    if (IRON) {                  // NH4, NO3, DOC, DON, DOP, DFe, POC, PON, POP, PFe_bio
                        const double* L = a.loss + (long long)x * 10;
                        NH4 += L[0]; NO3 += L[1]; DOC += L[2]; DON += L[3]; DOP += L[4];
                        DFe += L[5]; POC += L[6]; PON += L[7]; POP += L[8]; PFe += L[9];
                    } else {
                        const double* L = a.loss + (long long)x * 6;
                        DOC += L[0]; DON += L[1]; DOP += L[2];
                        POC += L[3]; PON += L[4]; POP += L[5];
                    }
                }
        for (uint32_t x = p; x < e; ++x) {
            const double* K = a.contrib + (long long)x * 5;
            if (IRON) { DIC += K[0]; NH4 += K[1]; NO3 += K[2]; PO4 += K[3]; DFe += K[4]; }
            else { DIC += K[0]; DOC += K[1]; NH4 += K[2]; NO3 += K[3]; PO4 += K[4]; }
        }
        p = e;
    }
    double* o = a.plk + q;
    const long long G = g.G;
    o[PI_DIC * G] = DIC; o[PI_NH4 * G] = NH4; o[PI_NO3 * G] = NO3; o[PI_PO4 * G] = PO4; o[PI_DOC * G] = DOC;
    o[PI_DON * G] = DON; o[PI_DOP * G] = DOP; o[PI_POC * G] = POC; o[PI_PON * G] = PON; o[PI_POP * G] = POP;
    if (IRON) { o[PI_DFe * G] = DFe; o[PI_PFe_bio * G] = PFe; }
}

// ------------------------------------------------------------------------------------------
// x and y sweeps
// ------------------------------------------------------------------------------------------
// A block takes 31 columns (32 x faces, one per lane) and `rows` rows of one level; warp n walks
// the rows of tracer n from two above to two below. Each row's x sweep gives the tracer_temp row
// that the y sweep keeps in a window of four; the flux of a y face is formed once and serves the
// rows on both sides. The x sweep's result is never stored: the two kernels that did stored and
// read 14 fields in between, and the one of the y sweep walked its 14 tracers one after another (16
// blocks and 248 µs on 128×128×1, 391 µs on 128×128×64).
// Rows outside the domain are the interior rows that the halo fill of tracer_temp maps them to.
#define XY64_MAXROWS 16
inline size_t xy64_smem(int rows) {
    return (size_t)(rows + 4) * 32 * FC_N * 8 + (size_t)(rows + 1) * 32 * FC_N * 8 + (size_t)(rows + 4) * 4 + (size_t)(2 * rows + 5) * 32;
}
template <bool LL, bool LM>
__global__ void __launch_bounds__(32 * PI_NTRACERS, 2) k64_xy(DGrid g, const double* __restrict__ tr, double* __restrict__ ttb,
                                                              const double* __restrict__ u, const double* __restrict__ v,
                                                              double dT, int rows, const uint32_t* err) {
    if (*err & PI_DEVERR_CAPACITY) return;
    extern __shared__ double sm64[];
    const int lane = threadIdx.x, n = threadIdx.y, tid = n * 32 + lane;
    const int i0 = blockIdx.x * 31 + 1 + g.Hx, j0 = blockIdx.y * rows + 1 + g.Hy, k = blockIdx.z + 1 + g.Hz;
    const int lastx = g.Nx + g.Hx, lasty = g.Ny + g.Hy;
    const int nr = min(rows, lasty - j0 + 1);                  // rows of this block
    const int xst = (rows + 4) * 32, yst = (rows + 1) * 32;     // plane strides
    double* sX = sm64;                                          // [FC_N][rows + 4][32]
    double* sY = sX + FC_N * xst;                               // [FC_N][rows + 1][32]
    int* sRow = reinterpret_cast<int*>(sY + FC_N * yst);        // first cell of each row read
    uint8_t* sXm = reinterpret_cast<uint8_t*>(sRow + rows + 4);
    uint8_t* sYm = sXm + xst;
    const double ax = g.dy * dzF1(g, k), ay = g.dx * dzF1(g, k);   // Ax, Ay of a RectilinearGrid
    const double dtv0 = LL ? 0.0 : dT / vol<false>(g, 1, 1, k);
    for (int e = tid; e < (nr + 4) * 32; e += 32 * PI_NTRACERS) {
        const int r = e >> 5, f = i0 + (e & 31);
        const int j = wrap_axis(j0 - 2 + r, g.Ny, g.Hy, g.ty);
        if ((e & 31) == 0) sRow[r] = gidx(g, 1, j, k);
        const bool special = f == lastx + 1;
        const bool zero = f > lastx + 1 || (special && g.tx != PI_PERIODIC);   // fill_halo_east_Gc! (Bounded)
        const int fs = special ? g.Hx + 1 : f;                  // face whose stencil gives the flux
        unsigned mb = zero ? FB_ZERO : 0u;
        double ftr = 0.0, dtv = 0.0;
        if (!zero) {
            put_face(sX + e, xst, face_coef(u[gidx(g, fs, j, k)], LL ? Axm<LL>(g, fs, j, k) : ax, dxCm<LL>(g, fs, j), dT));
            if (LM) mb |= lmask(g, fs - 2, j, k) | lmask(g, fs - 1, j, k) << 1 | lmask(g, fs, j, k) << 2 | lmask(g, fs + 1, j, k) << 3;
        }
        if (f <= lastx) {
            const int qc = gidx(g, f, j, k);
            const int cl0 = LM ? lmask(g, f, j, k) : 1, clp = LM ? lmask(g, f + 1, j, k) : 1;
            ftr = jl_mulb(jl_mulb((LL ? Axm<LL>(g, f + 1, j, k) : ax) * u[qc + 1] - (LL ? Axm<LL>(g, f, j, k) : ax) * u[qc], clp), cl0);
            if (LL) dtv = dT / vol<LL>(g, f, j, k);
            mb |= cl0 << 5 | clp << 6;
        }
        sX[FC_FTR * xst + e] = ftr;
        if (LL) sX[FC_DTV * xst + e] = dtv;
        sXm[e] = (uint8_t)mb;
    }
    for (int e = tid; e < (nr + 1) * 32; e += 32 * PI_NTRACERS) {
        const int f = j0 + (e >> 5), i = i0 + (e & 31);
        const bool special = f == lasty + 1;
        const bool zero = i > lastx || (special && g.ty != PI_PERIODIC);       // fill_halo_north_Gc! (Bounded)
        const int fs = special ? g.Hy + 1 : f;
        unsigned mb = zero ? FB_ZERO : 0u;
        if (!zero) {
            put_face(sY + e, yst, face_coef(v[gidx(g, i, fs, k)], LL ? Aym<LL>(g, i, fs, k) : ay, dyCm<LL>(g, i, fs), dT));
            if (LM) mb |= lmask(g, i, fs - 2, k) | lmask(g, i, fs - 1, k) << 1 | lmask(g, i, fs, k) << 2 | lmask(g, i, fs + 1, k) << 3;
        }
        double ftr = 0.0;
        if (i <= lastx && f <= lasty) {
            const int q = gidx(g, i, f, k);
            const int cl0 = LM ? lmask(g, i, f, k) : 1, clp = LM ? lmask(g, i, f + 1, k) : 1;
            ftr = jl_mulb(jl_mulb((LL ? Aym<LL>(g, i, f + 1, k) : ay) * v[q + g.Gx] - (LL ? Aym<LL>(g, i, f, k) : ay) * v[q], clp), cl0);
            mb |= cl0 << 5 | clp << 6;
        }
        sY[FC_FTR * yst + e] = ftr;
        sYm[e] = (uint8_t)mb;
    }
    __syncthreads();
    auto mkc = [](double x, unsigned mb) { return LM ? jl_mulb(jl_mulb(x, mb >> 6 & 1), mb >> 5 & 1) : x; };
    const int f = i0 + lane;
    const bool face = f <= lastx + 1, cell = lane < 31 && f <= lastx;
    const int fx = (face ? (f == lastx + 1 ? g.Hx + 1 : f) : i0) - 1;          // offset of the face's cell in a row
    const double* __restrict__ c = tr + n * g.G;
    double* __restrict__ out = ttb + n * g.G;
    double T0 = 0.0, T1 = 0.0, T2 = 0.0, T3 = 0.0, o1 = 0.0, o2 = 0.0, o3 = 0.0, Fy = 0.0;
    const double* p = c + sRow[0] + fx;
    double a0 = p[-2], a1 = p[-1], a2 = p[0], a3 = p[1];
    for (int r = 0; r < nr + 4; ++r) {
        const double cm2 = a0, cm1 = a1, c0 = a2, cp1 = a3;
        if (r + 1 < nr + 4) { p = c + sRow[r + 1] + fx; a0 = p[-2]; a1 = p[-1]; a2 = p[0]; a3 = p[1]; }
        const int ex = r * 32 + lane;
        const unsigned mx = sXm[ex];
        const double F = mx & FB_ZERO ? 0.0 : flux_s<LM>(sX + ex, xst, cm2, cm1, c0, cp1, mx);
        const double Fe = __shfl_down_sync(0xffffffffu, F, 1);
        T0 = T1; T1 = T2; T2 = T3;
        o1 = o2; o2 = o3; o3 = c0;
        const double dtvx = LL ? sX[FC_DTV * xst + ex] : dtv0;
        T3 = c0 - dtvx * (mkc(Fe - F, mx) - c0 * sX[FC_FTR * xst + ex]);
        if (r < 3) continue;
        // y face j0 + r - 3 from rows r - 3 .. r, and the row between it and the face before
        const int ey = (r - 3) * 32 + lane;
        const unsigned my = sYm[ey];
        const double Fn = my & FB_ZERO ? 0.0 : flux_s<LM>(sY + ey, yst, T0, T1, T2, T3, my);
        if (r > 3 && cell) {
            // row j0 + r - 4 is row r - 2 of the walk: window entry T1, original tracer o1
            const int ec = ey - 32, exc = ex - 2 * 32;
            const double dtv = LL ? sX[FC_DTV * xst + exc] : dtv0;
            out[sRow[r - 2] + f - 1] = T1 - dtv * (mkc(Fn - Fy, sYm[ec]) - o1 * sY[FC_FTR * yst + ec]);
        }
        Fy = Fn;
    }
}

// ------------------------------------------------------------------------------------------
// z sweep and the rest of tracer_update!
// ------------------------------------------------------------------------------------------
struct Z64Args {
    DGrid g;
    const double* tr;        // 14 × G, current tracers
    const double* ttb;       // 14 × G, tracer_temp after x and y
    double* tr_next;         // 14 × G
    const double* plk;       // 14 × G, particle terms of the occupied cells
    const uint32_t* off;     // G + 1, the cell's individuals
    const double* w;
    double dT;
    pi_bgc_params b;
    int diffuse;             // κh or κv nonzero
    int any_bc;
    const FluxBCDev* bcs;    // [14][6]
    int64_t iter;
    int levels;              // levels walked by a block
    const uint32_t* err;
};

// The rest of tracer_update! of one tracer of one cell, given its advective tendency: diffusion on the
// original tracer, sinking, forcing on max(0, tracer), boundary fluxes (the operation order of
// tracer_update.jl:22-43)
template <bool LL>
__device__ __forceinline__ double diffuse64(const Z64Args& a, const double* c, int i, int j, int k, double volk) {
    const DGrid& g = a.g;
    const double kx = a.b.kappa_h, kz = a.b.kappa_v, az = Azm<LL>(g, i, j);
    const int li = lmask(g, i, j, k);
    auto dx0 = [&](int ii) { return jl_mulb(jl_mulb(c[gidx(g, ii, j, k)] - c[gidx(g, ii - 1, j, k)], lmask(g, ii, j, k)), lmask(g, ii - 1, j, k)); };
    auto dy0 = [&](int jj) { return jl_mulb(jl_mulb(c[gidx(g, i, jj, k)] - c[gidx(g, i, jj - 1, k)], lmask(g, i, jj, k)), lmask(g, i, jj - 1, k)); };
    auto dz0 = [&](int kk) { return jl_mulb(jl_mulb(c[gidx(g, i, j, kk - 1)] - c[gidx(g, i, j, kk)], lmask(g, i, j, kk)), lmask(g, i, j, kk - 1)); };
    const double fx1 = kx * Axm<LL>(g, i + 1, j, k) * (dx0(i + 1) / dxFm<LL>(g, i + 1, j)), fx0 = kx * Axm<LL>(g, i, j, k) * (dx0(i) / dxFm<LL>(g, i, j));
    const double fy1 = kx * Aym<LL>(g, i, j + 1, k) * (dy0(j + 1) / dyFm<LL>(g, i, j + 1)), fy0 = kx * Aym<LL>(g, i, j, k) * (dy0(j) / dyFm<LL>(g, i, j));
    const double fz0 = kz * az * (dz0(k) / dzF1(g, k)), fz1 = kz * az * (dz0(k + 1) / dzF1(g, k + 1));
    const double ax_ = jl_mulb(jl_mulb(fx1 - fx0, lmask(g, i + 1, j, k)), li);
    const double ay_ = jl_mulb(jl_mulb(fy1 - fy0, lmask(g, i, j + 1, k)), li);
    const double az_ = jl_mulb(jl_mulb(fz0 - fz1, lmask(g, i, j, k + 1)), li);
    const double lap = 1.0 / volk * (ax_ + ay_ + az_);
    return lap * a.dT;
}
// tracer_forcing! of tracer n (tracer_forcings.jl:2-50); T(m) = max(0, tracer m) at the cell
template <class TF>
__device__ __forceinline__ double forcing64(int n, double G, const pi_bgc_params& b, double dT, TF T) {
    switch (n) {
        case PI_DIC: return G + T(PI_DOC) * b.kDOC * dT;
        case PI_DOC: return G - T(PI_DOC) * b.kDOC * dT + T(PI_POC) * b.kPOC * dT;
        case PI_POC: return G - T(PI_POC) * b.kPOC * dT;
        case PI_NH4: return G + T(PI_DON) * b.kDON * dT - T(PI_NH4) * b.Nit * dT;
        case PI_NO3: return G + T(PI_NH4) * b.Nit * dT;
        case PI_DON: return G - T(PI_DON) * b.kDON * dT + T(PI_PON) * b.kPON * dT;
        case PI_PON: return G - T(PI_PON) * b.kPON * dT;
        case PI_PO4: return G + T(PI_DOP) * b.kDOP * dT;
        case PI_DOP: return G - T(PI_DOP) * b.kDOP * dT + T(PI_POP) * b.kPOP * dT;
        case PI_POP: return G - T(PI_POP) * b.kPOP * dT;
        case PI_DFe:
            return G + T(PI_PFe_bio) * b.kPOC * dT
                   - (b.lambda_POC * T(PI_POC) + b.lambda_min + b.lambda_dust * T(PI_Dust)) * T(PI_DFe) * b.DFeFrac * dT
                   + T(PI_PFe_inorg) * b.kdiss * dT
                   - jl_max((T(PI_DFe) - b.ligand), 0.0) * T(PI_DFe) * b.DFeFrac * b.lambda_Fe * dT;
        case PI_PFe_bio:
            return G + T(PI_POC) * T(PI_DFe) * b.DFeFrac * b.lambda_POC * dT
                   - b.kPOC * T(PI_PFe_bio) * dT;
        case PI_PFe_inorg:
            return G - T(PI_PFe_inorg) * b.kdiss * dT
                   + (b.lambda_min + b.lambda_dust * T(PI_Dust)) * T(PI_DFe) * b.DFeFrac * dT
                   + jl_max((T(PI_DFe) - b.ligand), 0.0) * T(PI_DFe) * b.DFeFrac * b.lambda_Fe * dT;
        default: return G;
    }
}

// A block takes 32 columns of one row and `levels` levels; warp n walks tracer n down the levels with
// the four levels of tracer_temp around a face in registers and the flux of the face above kept.
// Separately, the z sweep stored its tendency for a per-cell kernel that read the tracers again
// (312 + 135 µs on 128×128×64, each tracer after the other in the first).
#define Z64_MAXLEV 16
inline size_t z64_smem(int levels) { return (size_t)(levels + 1) * 32 * (FC_N * 8 + 1) + (size_t)levels * 32 * 9; }
template <bool LL, bool LM, bool IRON>
__global__ void __launch_bounds__(32 * PI_NTRACERS, 2) k64_ztail(Z64Args a) {
    const DGrid& g = a.g;
    if (*a.err & PI_DEVERR_CAPACITY) return;
    extern __shared__ double sm64[];
    const int lane = threadIdx.x, n = threadIdx.y, tid = n * 32 + lane, LZ = a.levels;
    const int i = blockIdx.x * 32 + lane + 1 + g.Hx, j = blockIdx.y + 1 + g.Hy, k0 = blockIdx.z * LZ + 1 + g.Hz;
    const int bot = g.Nz + g.Hz, nl = min(LZ, bot - k0 + 1), st = (LZ + 1) * 32, slab = g.Gx * g.Gy;
    double* sZ = sm64;                                          // [FC_N][LZ + 1][32]
    double* sVol = sZ + FC_N * st;                              // [LZ][32]
    uint8_t* sM = reinterpret_cast<uint8_t*>(sVol + LZ * 32);   // [LZ + 1][32]
    uint8_t* sOcc = sM + st;                                    // [LZ][32] the cell holds individuals
    const double dT = a.dT;
    for (int e = tid; e < (nl + 1) * 32; e += 32 * PI_NTRACERS) {
        const int f = k0 + (e >> 5), ii = blockIdx.x * 32 + (e & 31) + 1 + g.Hx;
        unsigned mb = f > bot || ii > g.Nx + g.Hx ? FB_ZERO : 0u;              // fill_halo_bottom_Gc! (Bounded)
        if (!mb) {
            const int q = gidx(g, ii, j, f);
            const double az = Azm<LL>(g, ii, j);
            put_face(sZ + e, st, face_coef(a.w[q], az, dzC1(g, f), dT));
            const int cl0 = LM ? lmask(g, ii, j, f) : 1, clp = LM ? lmask(g, ii, j, f + 1) : 1;
            if (LM) mb |= clp | cl0 << 1 | lmask(g, ii, j, f - 1) << 2 | lmask(g, ii, j, f - 2) << 3;
            mb |= cl0 << 5 | clp << 6;
            if (f - k0 < nl) {
                const double vk = vol<LL>(g, ii, j, f);
                sZ[FC_FTR * st + e] = jl_mulb(jl_mulb(az * a.w[q] - az * a.w[q + slab], clp), cl0);
                sZ[FC_DTV * st + e] = dT / vk;
                sVol[e] = vk;
                sOcc[e] = a.off[q] != a.off[q + 1];
            }
        }
        sM[e] = (uint8_t)mb;
    }
    __syncthreads();
    if (i > g.Nx + g.Hx) return;
    auto mkc = [](double x, unsigned mb) { return LM ? jl_mulb(jl_mulb(x, mb >> 6 & 1), mb >> 5 & 1) : x; };
    const long long G = g.G;
    const int qcol = gidx(g, i, j, 1);
    const double* __restrict__ c = a.tr + n * G;
    const double* __restrict__ t = a.ttb + n * G;
    const pi_bgc_params& b = a.b;
    const bool sinks = n == PI_PFe_inorg || n == PI_Dust || n == PI_PFe_bio;
    const bool plks = !(n == PI_PFe_inorg || n == PI_Dust || ((n == PI_DFe || n == PI_PFe_bio) && !IRON));
    const double ws = n == PI_PFe_bio ? b.w_sink_org : b.w_sink_inorg;
    // levels outside the interior are read through the clamped map of the Bounded halo fill
    auto lev = [&](int kk) { return qcol + (min(max(kk, g.Hz + 1), bot) - 1) * slab; };
    double w0 = t[lev(k0 - 2)], w1 = t[lev(k0 - 1)], w2 = t[lev(k0)], w3 = t[lev(k0 + 1)];
    double tn = t[lev(k0 + 2)], cn = c[lev(k0)];
    double cup = sinks && k0 - 1 > g.Hz ? c[lev(k0 - 1)] : 0.0;
    // the four points of a z face in reverse are those of an x or y face
    double Ft = flux_s<LM>(sZ + lane, st, w3, w2, w1, w0, sM[lane]);
    for (int l = 0; l < nl; ++l) {
        const int k = k0 + l, q = qcol + (k - 1) * slab, e = l * 32 + lane;
        const double cc = cn;
        w0 = w1; w1 = w2; w2 = w3; w3 = tn;
        if (l + 1 < nl) { tn = t[lev(k + 3)]; cn = c[lev(k + 1)]; }
        const unsigned mf = sM[e + 32];
        const double Fb = mf & FB_ZERO ? 0.0 : flux_s<LM>(sZ + e + 32, st, w3, w2, w1, w0, mf);
        const double dG = mkc(Ft - Fb, sM[e]);
        const double ct = w1 - sZ[FC_DTV * st + e] * (dG - cc * sZ[FC_FTR * st + e]);
        Ft = Fb;
        double Gc = ct - cc;                                    // calc_tracer_tendency!
        const double volk = sVol[e];
        if (a.diffuse) Gc = Gc + diffuse64<LL>(a, c, i, j, k, volk);
        if (sinks) {
            // tracer_sinking! (tracer_sinking.jl:1-42); flux_sink is zero on k <= Hz and k >= Nz+Hz
            const double fup = (k - 1 <= g.Hz || k - 1 >= bot) ? 0.0 : ws * cup;
            const double fdn = (k >= bot) ? 0.0 : ws * cc;
            Gc = Gc + (fup - fdn) / dzC1(g, k - g.Hz) * dT;
            cup = cc;
        }
        Gc = forcing64(n, Gc, b, dT, [&](int m) { return jl_max(0.0, m == n ? cc : __ldg(a.tr + m * G + q)); });
        if (a.any_bc) {
            // apply_bcs! (apply_bcs.jl:4-98), faces in the reference's order
            const FluxBCDev* B = a.bcs + n * 6;
            const int ii = i - g.Hx, jj = j - g.Hy, kk = k - g.Hz;
            const double axk = Axm<LL>(g, i, j, k), ayk = Aym<LL>(g, i, j, k), az = Azm<LL>(g, i, j);
            if (B[PI_WEST].kind && i == 1 + g.Hx) Gc += getbc_dev(B[PI_WEST], jj, kk, a.iter) * dT * axk / volk;
            if (B[PI_EAST].kind && i == g.Nx + g.Hx) Gc -= getbc_dev(B[PI_EAST], jj, kk, a.iter) * dT * axk / volk;
            if (B[PI_SOUTH].kind && j == 1 + g.Hy) Gc += getbc_dev(B[PI_SOUTH], ii, kk, a.iter) * dT * ayk / volk;
            if (B[PI_NORTH].kind && j == g.Ny + g.Hy) Gc -= getbc_dev(B[PI_NORTH], ii, kk, a.iter) * dT * ayk / volk;
            if (B[PI_BOTTOM].kind && k == bot) Gc += getbc_dev(B[PI_BOTTOM], ii, jj, a.iter) * dT * az / volk;
            if (B[PI_TOP].kind && k == 1 + g.Hz) Gc -= getbc_dev(B[PI_TOP], ii, jj, a.iter) * dT * az / volk;
        }
        // apply_tendency!: tracer += Gc + plk / volume
        const double pk = plks && sOcc[e] ? a.plk[n * G + q] / volk : 0.0;
        a.tr_next[n * G + q] = cc + (Gc + pk);
    }
}

// fill_halo_tracer! (halo_regions.jl:2-62) in one pass, where every halo cell's source is interior (no
// periodic axis with N < H): the rule of each axis applied in turn is what the three sequential
// passes produce. Grid: (x blocks, tracers). After a capacity error the step stops where the
// reference throws: the buffer that becomes current is a copy of the old one.
__device__ __forceinline__ int halo_src64(int a, int N, int H, int topo) {
    if (a > H && a <= N + H) return a;
    if (topo == PI_PERIODIC) return a <= H ? a + N : a - N;
    return a <= H ? H + 1 : N + H;
}
__global__ void k64_halo(DGrid g, double* __restrict__ f, const double* __restrict__ src, const uint32_t* err) {
    double* __restrict__ c = f + blockIdx.y * g.G;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    if (*err & PI_DEVERR_CAPACITY) {
        for (long long q = t0; q < g.G; q += nt) c[q] = src[blockIdx.y * g.G + q];
        return;
    }
    const long long nz = 2LL * g.Hz * g.Gx * g.Gy, ny = 2LL * g.Nz * g.Hy * g.Gx, n = nz + ny + 2LL * g.Nz * g.Ny * g.Hx;
    for (long long t = t0; t < n; t += nt) {
        int i, j, k;
        if (t < nz) {
            const int kk = (int)(t / (g.Gx * g.Gy)), r = (int)(t - (long long)kk * (g.Gx * g.Gy));
            k = kk < g.Hz ? kk + 1 : g.Nz + kk + 1;
            j = r / g.Gx + 1; i = r - (j - 1) * g.Gx + 1;
        } else if (t < nz + ny) {
            const int u = (int)(t - nz), kk = u / (2 * g.Hy * g.Gx), r = u - kk * (2 * g.Hy * g.Gx), jj = r / g.Gx;
            k = g.Hz + 1 + kk;
            j = jj < g.Hy ? jj + 1 : g.Ny + jj + 1;
            i = r - jj * g.Gx + 1;
        } else {
            const int u = (int)(t - nz - ny), kk = u / (2 * g.Hx * g.Ny), r = u - kk * (2 * g.Hx * g.Ny), jj = r / (2 * g.Hx);
            const int ii = r - jj * 2 * g.Hx;
            k = g.Hz + 1 + kk; j = g.Hy + 1 + jj;
            i = ii < g.Hx ? ii + 1 : g.Nx + ii + 1;
        }
        c[gidx(g, i, j, k)] = c[gidx(g, halo_src64(i, g.Nx, g.Hx, g.tx), halo_src64(j, g.Ny, g.Hy, g.ty),
                                     halo_src64(k, g.Nz, g.Hz, PI_BOUNDED))];
    }
}

}  // namespace pib
