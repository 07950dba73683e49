// FP64 plain-form kernels of the model time step (the abiotic particles' own kernels are in
// kernels_abiotic.cuh).
//
// Every arithmetic expression below is written in the operation order of the reference Julia
// code it cites, and the library is compiled with -fmad=false, so each result is the same IEEE
// double the CPU oracle produces. Scatters that the reference does with float atomics are done
// here by binning individuals per cell (sorted by species then slot, the order of a sequential
// reference run) and summing each cell's contributions in that order.
#pragma once

#include "pib200_internal.h"

namespace pib {

__device__ __forceinline__ void set_err(uint32_t* err, uint32_t bit) { atomicOr(err, bit); }

__device__ __forceinline__ int clamp_idx(long long v, int lo, int hi, uint32_t* err) {
    if (v < lo) { set_err(err, PI_DEVERR_DOMAIN); return lo; }
    if (v > hi) { set_err(err, PI_DEVERR_DOMAIN); return hi; }
    return (int)v;
}

__device__ __forceinline__ double dzF1(const DGrid& g, int k) { return g.dzF[k - 1]; }
__device__ __forceinline__ double dzC1(const DGrid& g, int k) { return g.dzC[k - 1]; }
// Grids/areas_volumes_spacings.jl:9-38 with 1-based halo-inclusive indices. LL = false: a
// RectilinearGrid, whose metrics are formed from Δx, Δy and dzF in the reference's operation order;
// LL = true: a LatLonGrid, whose arrays are read. The kernels that use them are instantiated for
// both, so the RectilinearGrid code reads no metric array.
__device__ __forceinline__ int gidx2(const DGrid& g, int i, int j) { return (i - 1) + g.Gx * (j - 1); }
__device__ __forceinline__ long long gidx3l(const DGrid& g, int i, int j, int k) {
    return (i - 1) + (long long)g.Gx * ((j - 1) + (long long)g.Gy * (k - 1));
}
template <bool LL> __device__ __forceinline__ double vol(const DGrid& g, int i, int j, int k) {
    return LL ? g.mVol[gidx3l(g, i, j, k)] : g.dx * g.dy * dzF1(g, k);
}
template <bool LL> __device__ __forceinline__ double Axm(const DGrid& g, int i, int j, int k) {
    return LL ? g.mAx[gidx3l(g, i, j, k)] : g.dy * dzF1(g, k);
}
template <bool LL> __device__ __forceinline__ double Aym(const DGrid& g, int i, int j, int k) {
    return LL ? g.mAy[gidx3l(g, i, j, k)] : g.dx * dzF1(g, k);
}
template <bool LL> __device__ __forceinline__ double Azm(const DGrid& g, int i, int j) { return LL ? g.mAz[gidx2(g, i, j)] : g.dx * g.dy; }
template <bool LL> __device__ __forceinline__ double dxCm(const DGrid& g, int i, int j) { return LL ? g.mdxC[gidx2(g, i, j)] : g.dx; }
template <bool LL> __device__ __forceinline__ double dyCm(const DGrid& g, int i, int j) { return LL ? g.mdyC[gidx2(g, i, j)] : g.dy; }
template <bool LL> __device__ __forceinline__ double dxFm(const DGrid& g, int i, int j) { return LL ? g.mdxF[gidx2(g, i, j)] : g.dx; }
template <bool LL> __device__ __forceinline__ double dyFm(const DGrid& g, int i, int j) { return LL ? g.mdyF[gidx2(g, i, j)] : g.dy; }
// volume of a RectilinearGrid cell at level k (pi_tracer_advection_noalloc takes only these)
__device__ __forceinline__ double vol(const DGrid& g, int k) { return g.dx * g.dy * dzF1(g, k); }
__device__ __forceinline__ int lmask(const DGrid& g, int i, int j, int k) {
    return g.all_water ? 1 : (int)g.lm[gidx(g, i, j, k)];
}

// ------------------------------------------------------------------------------------------
// (a) RK4 advection + random-walk diffusion + cell lookup
//     particle_advection.jl:2-56, particle_advection_kernels.jl:2-50, interpolation.jl:3-83,
//     particle_diffusion.jl:2-33, Individuals/utils.jl:2-7
// ------------------------------------------------------------------------------------------

// particle_boundary_condition, particle_advection_kernels.jl:2-11
__device__ __forceinline__ double bc_pos(double x, double xr, int topo) {
    const double xl = 0.0;
    if (topo == PI_PERIODIC) {
        if (x > xr) return xl + (x - xr);
        if (x < xl) return xr - (xl - x);
        return x;
    }
    if (x > xr) return xr - (x - xr) * 1.0;
    if (x < xl) return xl + (xl - x) * 1.0;
    return x;
}

// Index (base corner) and offset of one axis of the interpolation from f = x + 1 or x + ½: trunc(f) + H
// clamped into 1 .. G - 1, and mod(f, 1). Out of line: NaN and positions outside the grid.
__device__ __noinline__ double index_axis_any(double f, int H, int G, int* idx, uint32_t* err) {
    *idx = clamp_idx(jl_trunc(f) + H, 1, G - 1, err);
    return jl_mod1(f);
}
__device__ __forceinline__ double index_axis(double f, int H, int G, int& idx, uint32_t* err) {
    if (f >= 0.0 && f < (double)(G - H)) {            // 0 <= trunc(f) <= G - 1 - H: nothing to clamp
        const double t = trunc(f);
        idx = (int)t + H;
        return f - t;
    }
    int i;
    const double r = index_axis_any(f, H, G, &i, err);
    idx = i;
    return r;
}

// Trilinear interpolation in grid-index units (u_itpl/v_itpl/w_itpl).
template <int COMP, bool LL>
__device__ __forceinline__ double itpl(const DGrid& g, const double* __restrict__ f0, double x, double y, double z, uint32_t* err) {
    int i, j, k;
    const double xd = index_axis(COMP == 0 ? x + 1.0 : x + 0.5, g.Hx, g.Gx, i, err);
    const double yd = index_axis(COMP == 1 ? y + 1.0 : y + 0.5, g.Hy, g.Gy, j, err);
    const double zd = index_axis(COMP == 2 ? z + 1.0 : z + 0.5, g.Hz, g.Gz, k, err);
    const double* __restrict__ p = f0 + gidx(g, i, j, k);
    const int sy = g.Gx, sz = g.Gx * g.Gy;
    double c000 = p[0], c001 = p[sz], c010 = p[sy], c011 = p[sy + sz];
    double c100 = p[1], c101 = p[1 + sz], c110 = p[1 + sy], c111 = p[1 + sy + sz];
    double w000 = (1.0 - xd) * (1.0 - yd) * (1.0 - zd);
    double w001 = (1.0 - xd) * (1.0 - yd) * zd;
    double w010 = (1.0 - xd) * yd * (1.0 - zd);
    double w011 = (1.0 - xd) * yd * zd;
    double w100 = xd * (1.0 - yd) * (1.0 - zd);
    double w101 = xd * (1.0 - yd) * zd;
    double w110 = xd * yd * (1.0 - zd);
    double w111 = xd * yd * zd;
    // each corner divided by ΔxC, ΔyC or ΔzC at that corner (interpolation.jl:23-50)
    auto D = [&](int a, int b, int c) -> double {
        return COMP == 0 ? dxCm<LL>(g, i + a, j + b) : COMP == 1 ? dyCm<LL>(g, i + a, j + b) : dzC1(g, k + c);
    };
    return w000 * c000 / D(0, 0, 0) + w001 * c001 / D(0, 0, 1) + w010 * c010 / D(0, 1, 0) + w011 * c011 / D(0, 1, 1)
         + w100 * c100 / D(1, 0, 0) + w101 * c101 / D(1, 0, 1) + w110 * c110 / D(1, 1, 0) + w111 * c111 / D(1, 1, 1);
}


// vel½ = (vel₀ + vel₁) * 0.5 (time_step.jl:17-19), once per step for the three components.
__global__ void k_velhalf(long long G, const double* __restrict__ u0, const double* __restrict__ v0,
                          const double* __restrict__ w0, const double* __restrict__ u1,
                          const double* __restrict__ v1, const double* __restrict__ w1,
                          double* __restrict__ uh, double* __restrict__ vh, double* __restrict__ wh,
                          const uint32_t* err) {
    if (*err & PI_DEVERR_CAPACITY) return;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < G; q += (long long)gridDim.x * blockDim.x) {
        uh[q] = (u0[q] + u1[q]) * 0.5;
        vh[q] = (v0[q] + v1[q]) * 0.5;
        wh[q] = (w0[q] + w1[q]) * 0.5;
    }
}

struct VelPtrs { const double *u0, *v0, *w0, *uh, *vh, *wh, *u1, *v1, *w1; };

// RK4 + diffusion + find_inds! of one active particle at `slot` of the columns x, y, z, cell of P
// (a phytoplankton species, SpcDev, or an abiotic species, AbioDev, whose steps are the same
// kernels, time_step.jl:29-38); the diffusion draw is keyed by (dsp, purpose). BIN: writes the
// binning key of a phytoplankton individual and its number among those of its cell (in the order
// of the atomics).
template <bool LL, bool BIN = true, class PV>
__device__ __forceinline__ void particle_step(const DGrid& g, const PV& P, uint32_t dsp, uint32_t purpose, long long slot,
                                              long long gid, double dT, uint64_t seed, uint32_t iter,
                                              const VelPtrs& vel, double kappa_h, double kappa_v,
                                              uint32_t* __restrict__ cnt, uint32_t* __restrict__ key,
                                              int32_t* __restrict__ pos, uint32_t* err) {
    int oxi, oyi, ozi;
    unpack_cell(g, P.cell[slot], oxi, oyi, ozi);
    int kdz = clamp_idx((long long)ozi + g.Hz, 1, g.Gz, err);   // ΔzC at the stored zi + Hz
    const double X = P.x[slot], Y = P.y[slot], Z = P.z[slot];
    const double NX = (double)g.Nx, NY = (double)g.Ny, NZ = (double)g.Nz;
    // the four stages at vel₀, vel½, vel½, vel₁: one body, a quarter of the instructions of four
    // (products by 1.0 are exact)
    double u2 = 0.0, v2 = 0.0, w2 = 0.0, vx = X, vy = Y, vz = Z;
#pragma unroll 1
    for (int st = 0; st < 4; ++st) {
        const double* __restrict__ fu = st == 0 ? vel.u0 : st == 3 ? vel.u1 : vel.uh;
        const double* __restrict__ fv = st == 0 ? vel.v0 : st == 3 ? vel.v1 : vel.vh;
        const double* __restrict__ fw = st == 0 ? vel.w0 : st == 3 ? vel.w1 : vel.wh;
        const double u1 = itpl<0, LL>(g, fu, vx, vy, vz, err);
        const double v1 = itpl<1, LL>(g, fv, vx, vy, vz, err);
        const double w1 = itpl<2, LL>(g, fw, vx, vy, vz, err);
        const double wt = st == 1 || st == 2 ? 2.0 : 1.0, hs = st < 2 ? 0.5 : 1.0;
        if (st == 0) { u2 = u1; v2 = v1; w2 = w1; }
        else { u2 = u2 + u1 * wt; v2 = v2 + v1 * wt; w2 = w2 + w1 * wt; }
        vx = bc_pos(X + hs * u1 * dT, NX, g.tx); vy = bc_pos(Y + hs * v1 * dT, NY, g.ty); vz = bc_pos(Z - hs * w1 * dT, NZ, g.tz);
    }
    u2 = u2 / 6.0; v2 = v2 / 6.0; w2 = w2 / 6.0;
    double x = bc_pos(X + 1.0 * u2 * dT, NX, g.tx);
    double y = bc_pos(Y + 1.0 * v2 * dT, NY, g.ty);
    double z = bc_pos(Z - 1.0 * w2 * dT, NZ, g.tz);
    // diffusion: rnd ∈ [0,1) → (rnd - 0.5) * 2 → · √(κΔT) / Δ
    double r0, r1, r2;
    pi_draw3(seed, iter, dsp, purpose, (uint32_t)slot, &r0, &r1, &r2);
    r0 = (r0 - 0.5) * 2.0; r1 = (r1 - 0.5) * 2.0; r2 = (r2 - 0.5) * 2.0;
    // ΔxC/ΔyC at (xi+Hx, yi+Hy) of the stored indices (particle_diffusion.jl:4-5); the reference
    // reads past the metric array there when x = Nx exactly, which is held at the last column here
    const int dxi = min(max(oxi + g.Hx, 1), g.Gx), dyi = min(max(oyi + g.Hy, 1), g.Gy);
    r0 = r0 * sqrt(kappa_h * dT) / dxCm<LL>(g, dxi, dyi);
    r1 = r1 * sqrt(kappa_h * dT) / dyCm<LL>(g, dxi, dyi);
    r2 = r2 * sqrt(kappa_v * dT) / dzC1(g, kdz);
    x = bc_pos(x + r0, NX, g.tx); y = bc_pos(y + r1, NY, g.ty); z = bc_pos(z + r2, NZ, g.tz);
    P.x[slot] = x; P.y[slot] = y; P.z[slot] = z;
    // find_inds!
    int xi = clamp_idx(jl_trunc(x + 1.0) + g.Hx, 1, g.Gx, err);
    int yi = clamp_idx(jl_trunc(y + 1.0) + g.Hy, 1, g.Gy, err);
    int zi = clamp_idx(jl_trunc(z + 1.0) + g.Hz, 1, g.Gz, err);
    P.cell[slot] = pack_cell(g, xi, yi, zi);
    if (BIN) {
        int c = gidx(g, xi, yi, zi);
        key[gid] = (uint32_t)c;
        pos[gid] = (int32_t)atomicAdd(&cnt[c], 1u);
    }
}

// Slot-order pass over every (species, slot): inactive slots (every stage multiplies by ac, so
// their positions end as zeros and their cell is (Hx, Hy, Hz)), and active individuals that were
// not binned in the previous step (new daughters, uploaded state). The others are moved by
// k_particles_sorted in cell order.
template <bool LL>
__global__ void k_particles(DGrid g, const SpcDev* __restrict__ spc, int nsp, long long C,
                            double dT, uint64_t seed, uint32_t iter, VelPtrs vel,
                            double kappa_h, double kappa_v, uint32_t* __restrict__ cnt,
                            uint32_t* __restrict__ key, int32_t* __restrict__ pos, uint32_t sentinel, uint32_t* err) {
    long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)nsp * C) return;
    if (*err & PI_DEVERR_CAPACITY) return;
    int s = (int)(gid / C);
    long long slot = gid - (long long)s * C;
    const SpcDev& P = spc[s];
    const uint8_t stt = P.stat[slot];
    if (!(P.flags[slot] & FL_AC)) {
        if (stt & ST_HOME) return;                    // as this pass left it
        P.stat[slot] = ST_HOME;
        int oxi, oyi, ozi;
        unpack_cell(g, P.cell[slot], oxi, oyi, ozi);
        clamp_idx((long long)ozi + g.Hz, 1, g.Gz, err);
        if (P.x[slot] != 0.0) P.x[slot] = 0.0;
        if (P.y[slot] != 0.0) P.y[slot] = 0.0;
        if (P.z[slot] != 0.0) P.z[slot] = 0.0;
        P.cell[slot] = pack_cell(g, g.Hx, g.Hy, g.Hz);
        key[gid] = sentinel;
        return;
    }
    if (stt & ST_AC0) return;                         // moved by k_particles_sorted
    particle_step<LL>(g, P, (uint32_t)s, PI_DRAW_DIFFUSION, slot, gid, dT, seed, iter, vel, kappa_h, kappa_v, cnt, key,
                      pos, err);
}

// Cell-order pass: the individuals binned in the previous step (prev_sorted[0 .. off[G]), which
// were active then) that are still active. Neighbouring threads interpolate in neighbouring cells.
// Bound by the latency of FP64 chains (96 quotients and as many loads per individual), so warps count
// more than registers: 110 registers 275 µs, 80 registers 227 µs for 1,048,576 individuals. Dividing
// by reciprocals with exact remainders was slower than the division (301 µs): the compiler already
// shares the reciprocal of a divisor.
template <bool LL>
__global__ void __launch_bounds__(128, 6) k_particles_sorted(DGrid g, const SpcDev* __restrict__ spc, long long C,
                                   const uint32_t* __restrict__ prev_sorted,
                                   const uint32_t* __restrict__ prev_off, long long Gcells,
                                   double dT, uint64_t seed, uint32_t iter, VelPtrs vel,
                                   double kappa_h, double kappa_v, uint32_t* __restrict__ cnt,
                                   uint32_t* __restrict__ key, int32_t* __restrict__ pos, uint32_t* err) {
    long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (*err & PI_DEVERR_CAPACITY) return;
    if (p >= (long long)prev_off[Gcells]) return;
    uint32_t gd = prev_sorted[p];
    int s = (int)(gd / C);
    long long slot = gd - (long long)s * C;
    const SpcDev& P = spc[s];
    if (!(P.flags[slot] & FL_AC) || !(P.stat[slot] & ST_AC0)) return;
    particle_step<LL>(g, P, (uint32_t)s, PI_DRAW_DIFFUSION, slot, gd, dT, seed, iter, vel, kappa_h, kappa_v, cnt, key,
                      pos, err);
}

// The cell-sorted entry list (cells in order, gid = species·C + slot ascending within a cell, the
// order of a sequential reference run) from the counting sort that k_particles began: k64_place puts
// the individuals of a cell together in the order of the atomics, k64_order gives each its rank by
// gid among them, by comparing it with all of them (98 per cell: 84 µs, 125 by a block each); cells of more
// than ORDER_CELL are left to k64_order_big. Cells of more than CROWD_CELL are listed for the particle terms
// (k64_plk). The radix sort of all keys took six launches: 35 µs for 32,768 slots, 80 µs for 2,097,152.
#define ORDER_CELL 128
#define CROWD_CELL 64
__global__ void k64_place(const uint32_t* __restrict__ off, uint32_t Gcells, const uint32_t* __restrict__ key,
                          const int32_t* __restrict__ pos, uint32_t* __restrict__ list, long long n, const uint32_t* err) {
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= n || (*err & PI_DEVERR_CAPACITY)) return;
    const uint32_t c = key[gid];
    if (c < Gcells) list[off[c] + (uint32_t)pos[gid]] = (uint32_t)gid;
}
__global__ void k64_order(const uint32_t* __restrict__ off, long long G, const uint32_t* __restrict__ key,
                          const uint32_t* __restrict__ list, uint32_t* __restrict__ gid_sorted, int32_t* __restrict__ pos,
                          long long n, uint32_t* __restrict__ ncell, uint32_t* __restrict__ big, uint32_t* __restrict__ crowd,
                          const uint32_t* err) {
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n || (*err & PI_DEVERR_CAPACITY) || p >= (long long)off[G]) return;
    const uint32_t gid = list[p], c = key[gid], p0 = off[c], m = off[c + 1] - p0;
    if (m > CROWD_CELL && p == (long long)p0) {
        crowd[atomicAdd(&ncell[1], 1u)] = c;
        if (m > ORDER_CELL) big[atomicAdd(&ncell[0], 1u)] = c;
    }
    if (m > ORDER_CELL) return;
    uint32_t r = 0;
#pragma unroll 4
    for (uint32_t x = 0; x < m; ++x) r += list[p0 + x] < gid;
    gid_sorted[p0 + r] = gid;
    pos[gid] = (int32_t)(p0 + r);
}
// A block per crowded cell, from the cell's own entries: up to ORDER_SORT of them are sorted in shared
// memory (bitonic), more are set as bits of a window of the gids at a time and read back in order
// (0D models: one cell holds every individual). The work grows with the entries, not with the slots. A step
// with 1.6 million individuals in 2,097,152 slots, k64_place to here (radix sort of all keys; looking for each
// crowded cell's key among all slots): 16 cells 422 µs (75; 614), 256 161 (82; 1,129), 1,024 102 (87; 813),
// 4,096 90 (88; 230). Blocks of 256: with 1,024 threads 236, 123, 114 and 179.
#define ORDER_SORT 8192
#define ORDER_THREADS 256
__global__ void __launch_bounds__(ORDER_THREADS) k64_order_big(const uint32_t* __restrict__ off, const uint32_t* __restrict__ list,
                                                               long long n, const uint32_t* __restrict__ ncell,
                                                               const uint32_t* __restrict__ big, uint32_t* __restrict__ gid_sorted,
                                                               int32_t* __restrict__ pos, const uint32_t* err) {
    // the entries, or a bit per gid of the window (32 words per thread, padded by one against bank conflicts)
    __shared__ uint32_t s[ORDER_SORT + ORDER_SORT / 32], sums[ORDER_THREADS / 32];
    if (*err & PI_DEVERR_CAPACITY) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    auto pad = [](uint32_t w) { return w + (w >> 5); };
    for (uint32_t t = blockIdx.x; t < ncell[0]; t += gridDim.x) {
        const uint32_t c = big[t], p0 = off[c], m = off[c + 1] - p0;
        if (m <= ORDER_SORT) {
            uint32_t P = 2 * ORDER_CELL;
            while (P < m) P *= 2;
            for (uint32_t q = tid; q < P; q += ORDER_THREADS) s[q] = q < m ? list[p0 + q] : 0xffffffffu;
            __syncthreads();
            for (uint32_t k = 2; k <= P; k *= 2)
                for (uint32_t j = k / 2; j; j /= 2) {
                    for (uint32_t q = tid; q < P / 2; q += ORDER_THREADS) {
                        const uint32_t i0 = 2 * q - (q & (j - 1)), i1 = i0 + j, x = s[i0], y = s[i1];
                        if ((x > y) == ((i0 & k) == 0)) { s[i0] = y; s[i1] = x; }
                    }
                    __syncthreads();
                }
            for (uint32_t q = tid; q < m; q += ORDER_THREADS) {
                gid_sorted[p0 + q] = s[q];
                pos[s[q]] = (int32_t)(p0 + q);
            }
            __syncthreads();
            continue;
        }
        uint32_t at = p0;
        for (long long base = 0; base < n; base += 32LL * ORDER_SORT) {
            for (int q = tid; q < ORDER_SORT + ORDER_SORT / 32; q += ORDER_THREADS) s[q] = 0u;
            __syncthreads();
#pragma unroll 4
            for (uint32_t q = tid; q < m; q += ORDER_THREADS) {
                const long long g = (long long)list[p0 + q] - base;
                if (g >= 0 && g < 32LL * ORDER_SORT) atomicOr(&s[pad((uint32_t)g >> 5)], 1u << ((uint32_t)g & 31u));
            }
            __syncthreads();
            // each thread its run of words, behind the counts of the threads before it
            const uint32_t w0 = tid * (ORDER_SORT / ORDER_THREADS);
            uint32_t cnt = 0;
            for (uint32_t w = w0; w < w0 + ORDER_SORT / ORDER_THREADS; ++w) cnt += __popc(s[pad(w)]);
            uint32_t inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) sums[wid] = inc;
            __syncthreads();
            uint32_t e = at + inc - cnt;
            for (int w = 0; w < ORDER_THREADS / 32; ++w) {
                if (w < wid) e += sums[w];
                at += sums[w];
            }
            for (uint32_t w = w0; cnt && w < w0 + ORDER_SORT / ORDER_THREADS; ++w)
                for (uint32_t b = s[pad(w)]; b; b &= b - 1u, ++e) {
                    const uint32_t gid = (uint32_t)base + w * 32u + __ffs(b) - 1u;
                    gid_sorted[e] = gid;
                    pos[gid] = (int32_t)e;
                }
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------------------------------
// PAR: calc_par! down each column (Individuals/utils.jl:55-63, time_step.jl:63-67) with the Chl
// of acc_chl! (utils.jl:33-36) summed per cell in species-then-slot order, and
// diags.tracer.PAR .+= par (time_step.jl:167).
//
// `lw` warps (a power of two) share 32 columns: each sums the Chl of PAR64_CH levels and forms their
// attenuation, the first carries the light down through shared memory, all write their levels. One
// thread per column waited for the gathered Chl cell by cell: 207 µs on 128×128×64 with 6 % of the
// warps resident.
// ------------------------------------------------------------------------------------------
#define PAR64_CH 4
#define PAR64_WARPS 16
template <bool LL>
__global__ void __launch_bounds__(32 * PAR64_WARPS, 2) k64_par(DGrid g, const SpcDev* __restrict__ spc, long long C,
                      const uint32_t* __restrict__ off, const uint32_t* __restrict__ gid_sorted,
                      double* __restrict__ PARF, double* __restrict__ par, double* __restrict__ diag_par, double kc, double kw,
                      int lw, const uint32_t* err) {
    __shared__ double sEx[PAR64_WARPS * PAR64_CH][32], sIn[PAR64_WARPS * PAR64_CH][32];
    if (*err & PI_DEVERR_CAPACITY) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, part = wid & (lw - 1), row0 = wid * PAR64_CH;
    const int nx32 = (g.Nx + 31) / 32, w = blockIdx.x * ((blockDim.x >> 5) / lw) + wid / lw;
    const int i = (w % nx32) * 32 + lane + 1, j = w / nx32 + 1;
    const bool col = j <= g.Ny && i <= g.Nx;
    const int ii = i + g.Hx, jj = j + g.Hy, slab = g.Gx * g.Gy;
    const int f = (i - 1) + g.Nx * (j - 1);
    const int q1 = col ? gidx(g, ii, jj, 1 + g.Hz) : 0;
    double parf = col && part == 0 ? PARF[f] : 0.0;
    for (int kc0 = 0; kc0 < g.Nz; kc0 += PAR64_CH * lw) {
        const int k0 = kc0 + part * PAR64_CH;                   // 0-based levels k0 .. k0 + PAR64_CH - 1
        double ex[PAR64_CH], at[PAR64_CH];
        if (col) {
            uint32_t p0[PAR64_CH], p1[PAR64_CH];
#pragma unroll
            for (int e = 0; e < PAR64_CH; ++e) {
                const bool in = k0 + e < g.Nz;
                const int c = q1 + (k0 + e) * slab;
                p0[e] = in ? off[c] : 0u; p1[e] = in ? off[c + 1] : 0u;
            }
#pragma unroll
            for (int e = 0; e < PAR64_CH; ++e) {
                if (k0 + e >= g.Nz) continue;
                double chl = 0.0;
                for (uint32_t p = p0[e]; p < p1[e]; ++p) {
                    const uint32_t gd = gid_sorted[p];
                    const int s = (int)(gd / (uint32_t)C);
                    chl += spc[s].Chl[gd - (uint32_t)s * (uint32_t)C];
                }
                const int kk = k0 + e + 1 + g.Hz;
                at[e] = (chl / vol<LL>(g, ii, jj, kk) * kc + kw) * dzF1(g, kk);
                ex[e] = pi_exp(-at[e]);
                sEx[row0 + e][lane] = ex[e];
            }
        }
        __syncthreads();
        if (part == 0 && col) {
            const int n = min(PAR64_CH * lw, g.Nz - kc0);
            for (int e = 0; e < n; ++e) {
                sIn[row0 + e][lane] = parf;
                parf = parf * sEx[row0 + e][lane];
            }
        }
        __syncthreads();
        if (col) {
#pragma unroll
            for (int e = 0; e < PAR64_CH; ++e) {
                if (k0 + e >= g.Nz) continue;
                const int c = q1 + (k0 + e) * slab;
                const double pv = sIn[row0 + e][lane] * (1.0 - ex[e]) / at[e];
                par[c] = pv;
                diag_par[c] = diag_par[c] + pv;
            }
        }
        __syncthreads();
    }
    if (col && part == 0) PARF[f] = parf;
}

// ------------------------------------------------------------------------------------------
// (e) grazing, mortality, division — plankton_update.jl:5-24, division_death.jl:2-77,
//     consume_loss.jl:17-26, Diagnostics/diagnostics_kernels.jl:4-7
// ------------------------------------------------------------------------------------------

// total_C/N/P_biomass (MacroMolecularMode/plankton_generation.jl:82-93)
__host__ __device__ __forceinline__ double m_totC(double PRO, double DNA, double RNA, double CH, double Chl) {
    return PRO + DNA + RNA + CH + Chl / F_CHL * 55.0;
}
__host__ __device__ __forceinline__ double m_totN(double PRO, double DNA, double RNA, double NST, double Chl,
                                                  const pi_macro_params& p) {
    return PRO * p.R_NC_PRO + DNA * p.R_NC_DNA + RNA * p.R_NC_RNA + NST + Chl / F_CHL * 4.0;
}
__host__ __device__ __forceinline__ double m_totP(double DNA, double RNA, double PST, const pi_macro_params& p) {
    return DNA * p.R_PC_DNA + RNA * p.R_PC_RNA + PST;
}

// Applies last step's grazing/mortality decisions, writes the loss contributions of the
// individuals lost, the divider and free-slot bits of 32 slots per word and the graz/mort/dvid diags.
// mode MODE_CARBON: CarbonMode losses (CarbonMode/consume_loss.jl:12-16), DOC and POC from Bm only;
// MODE_MACRO: MacroMolecularMode losses (MacroMolecularMode/consume_loss.jl:14-24) from the total
// C, N and P biomass (mp holds its R_NC_* and R_PC_* ratios).
__global__ void k_decide(DGrid g, SpcDev P, pi_quota_params p, pi_macro_params mp, pi_iron_params ip, long long C, int s,
                         const int32_t* __restrict__ pos, double* __restrict__ loss,
                         uint8_t* __restrict__ evk, uint32_t* __restrict__ dvw, uint32_t* __restrict__ frw,
                         double* __restrict__ d_graz, double* __restrict__ d_mort,
                         double* __restrict__ d_dvid, uint32_t* err, int mode) {
    long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (*err & PI_DEVERR_CAPACITY) return;
    const bool in = slot < C;
    uint8_t f = in ? P.flags[slot] : 0;
    int ac0 = f & FL_AC, gz = (f & FL_GRAZ) != 0, mt = (f & FL_MORT) != 0, dv = (f & FL_DVID) != 0;
    if (in) P.stat[slot] = ac0 ? ST_AC0 : (uint8_t)(P.stat[slot] & ST_HOME);
    int ac1 = ac0 && !gz;          // inactivate!(plank, graz): ac &= isless(graz, 1)
    int ac2 = ac1 && !mt;          // inactivate!(plank, mort)
    int dv2 = dv && ac2;           // plank.dvid .*= plank.ac
    if (ac0) {
        int xi, yi, zi;
        unpack_cell(g, P.cell[slot], xi, yi, zi);
        int c = gidx(g, xi, yi, zi);
        if (gz) atomicAdd(&d_graz[c], 1.0);
        if (ac1 && mt) atomicAdd(&d_mort[c], 1.0);
        if (dv2) atomicAdd(&d_dvid[c], 1.0);
        long long e = pos[(long long)s * C + slot];
        uint8_t kind = gz ? 1 : (ac1 && mt) ? 2 : 0;
        evk[e] = kind;
        if (kind) {
            double fC = kind == 1 ? p.grazFracC : p.mortFracC;
            double fN = kind == 1 ? p.grazFracN : p.mortFracN;
            double fP = kind == 1 ? p.grazFracP : p.mortFracP;
            if (mode == MODE_IRON) {
                // IronEnergyMode/consume_loss.jl:17-32: NH4, NO3, DOC, DON, DOP, DFe, POC, PON, POP, PFe_bio
                double* L = loss + e * 10;
                const double fFe = kind == 1 ? ip.grazFracFe : ip.mortFracFe;
                const double Bm = P.Bm[slot], CH = P.CH[slot], qP = P.qP[slot];
                const double fe = P.qFe[slot] + P.qFePS[slot] + P.qFeNF[slot] + P.qFeNR[slot];
                L[0] = jl_mulb(P.qNH4[slot], 1) * 1.0;
                L[1] = jl_mulb(P.qNO3[slot], 1) * 1.0;
                L[2] = jl_mulb((Bm + CH) * fC, 1) * 1.0;
                L[3] = jl_mulb(Bm * ip.R_NC * fN, 1) * 1.0;
                L[4] = jl_mulb((Bm * ip.R_PC + qP) * fP, 1) * 1.0;
                L[5] = jl_mulb(fe * fFe, 1) * 1.0;
                L[6] = jl_mulb((Bm + CH) * (1.0 - fC), 1) * 1.0;
                L[7] = jl_mulb(Bm * ip.R_NC * (1.0 - fN), 1) * 1.0;
                L[8] = jl_mulb((Bm * ip.R_PC + qP) * (1.0 - fP), 1) * 1.0;
                L[9] = jl_mulb(fe * (1.0 - fFe), 1) * 1.0;
            } else {
            double* L = loss + e * 6;
            if (mode == MODE_CARBON) {
                const double Bm = P.Bm[slot];
                L[0] = jl_mulb(Bm * fC, 1) * 1.0;                     // DOC
                L[3] = jl_mulb(Bm * (1.0 - fC), 1) * 1.0;             // POC
                L[1] = 0.0; L[2] = 0.0; L[4] = 0.0; L[5] = 0.0;
            } else if (mode == MODE_MACRO) {
                const double tC = m_totC(P.PRO[slot], P.DNA[slot], P.RNA[slot], P.CH[slot], P.Chl[slot]);
                const double tN = m_totN(P.PRO[slot], P.DNA[slot], P.RNA[slot], P.NST[slot], P.Chl[slot], mp);
                const double tP = m_totP(P.DNA[slot], P.RNA[slot], P.PST[slot], mp);
                L[0] = jl_mulb(tC * fC, 1) * 1.0;                     // DOC
                L[1] = jl_mulb(tN * fN, 1) * 1.0;                     // DON
                L[2] = jl_mulb(tP * fP, 1) * 1.0;                     // DOP
                L[3] = jl_mulb(tC * (1.0 - fC), 1) * 1.0;             // POC
                L[4] = jl_mulb(tN * (1.0 - fN), 1) * 1.0;             // PON
                L[5] = jl_mulb(tP * (1.0 - fP), 1) * 1.0;             // POP
            } else {
            double Bm = P.Bm[slot], Cq = P.Cq[slot], Nq = P.Nq[slot], Pq = P.Pq[slot];
            L[0] = jl_mulb((Bm + Cq) * fC, 1) * 1.0;                  // DOC
            L[1] = jl_mulb((Bm * p.R_NC + Nq) * fN, 1) * 1.0;         // DON
            L[2] = jl_mulb((Bm * p.R_PC + Pq) * fP, 1) * 1.0;         // DOP
            L[3] = jl_mulb((Bm + Cq) * (1.0 - fC), 1) * 1.0;          // POC
            L[4] = jl_mulb((Bm * p.R_NC + Nq) * (1.0 - fN), 1) * 1.0; // PON
            L[5] = jl_mulb((Bm * p.R_PC + Pq) * (1.0 - fP), 1) * 1.0; // POP
            }
            }
        }
    }
    if (in) P.flags[slot] = (uint8_t)((ac2 ? FL_AC : 0) | (dv2 ? FL_DVID : 0));
    // dividers and free slots, one bit per slot
    const uint32_t wd = __ballot_sync(0xffffffffu, dv2), wf = __ballot_sync(0xffffffffu, in && !ac2);
    if ((threadIdx.x & 31) == 0 && in) { dvw[slot >> 5] = wd; frw[slot >> 5] = wf; }
}

// After the exclusive scan of flag64 (abiotic release): the k-th releaser (slot order) and the k-th
// free slot (findall(!ac), ascending) — get_tind!, Individuals/utils.jl:76-86. Checks capacity.
__global__ void k_lists(const unsigned long long* __restrict__ flag64,
                        const unsigned long long* __restrict__ rank64, long long C,
                        int32_t* __restrict__ divlist, int32_t* __restrict__ freelist,
                        uint32_t* ndiv, uint32_t* err, int64_t* err_iter, int64_t iter,
                        uint32_t errbits = PI_DEVERR_CAPACITY) {
    long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C) return;
    if (*err & PI_DEVERR_CAPACITY) return;
    unsigned long long tot = rank64[C - 1] + flag64[C - 1];
    unsigned long long tdiv = tot >> 32, tfree = tot & 0xffffffffull;
    if (tdiv > tfree) {
        if (slot == 0) { *ndiv = 0; *err_iter = iter; }
        __threadfence();
        // every thread sees the same totals; one flag write is enough but all are harmless
        if (slot == 0) set_err(err, errbits);
        return;
    }
    if (slot == 0) *ndiv = (uint32_t)tdiv;
    unsigned long long f = flag64[slot], r = rank64[slot];
    if (f >> 32) divlist[r >> 32] = (int32_t)slot;
    if (f & 1ull) {
        unsigned long long fr = r & 0xffffffffull;
        if (fr < tdiv) freelist[fr] = (int32_t)slot;
    }
}

// copy_daughter_individuals! then divide_to_half! for the dividers and their daughters
// (division_death.jl:28-63). Other slots are unchanged by divide_to_half (factor 1, +0, ×1).
// CarbonMode (CarbonMode/division_death.jl:28-57): x, y, z, Sz, Bm, Chl and gen are copied, Bd is
// not — the daughter halves the damaged biomass its slot held before.
// the pools of a mode, copied and halved in both
template <int N>
__device__ __forceinline__ void halve_pools(double* const (&pools)[N], long long p, long long d) {
    const double h = (2.0 - 1.0) / 2.0;
    double v[N];
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = pools[q][p] * h;
#pragma unroll
    for (int q = 0; q < N; ++q) { pools[q][d] = v[q]; pools[q][p] = v[q]; }
}
// divider p and its daughter's slot d; every mode reads before it writes (the slots are different)
__device__ __forceinline__ void daughter_pair(const SpcDev& P, long long p, long long d, int mode) {
    const double h = (2.0 - 1.0) / 2.0;
    const double x = P.x[p], y = P.y[p], z = P.z[p], gen = P.gen[p];
    const double aged = P.age[d] * (1.0 - 1.0), agep = P.age[p] * (1.0 - 1.0);
    P.x[d] = x; P.y[d] = y; P.z[d] = z;
    P.gen[d] = gen + 1.0; P.age[d] = aged;
    P.flags[d] = FL_AC | FL_DVID;
    P.gen[p] = gen + 1.0; P.age[p] = agep;
    if (mode == MODE_IRON) {
        // IronEnergyMode/division_death.jl:44-82: x, y, z, tdark and gen copied; Sz, Bm, CH, the
        // quotas, exEn and Chl copied and halved in both; age not copied
        P.tdark[d] = P.tdark[p];
        double* const pools[12] = { P.Sz, P.Bm, P.CH, P.qNO3, P.qNH4, P.qP, P.qFe, P.qFePS, P.qFeNR, P.qFeNF, P.exEn, P.Chl };
        halve_pools(pools, p, d);
    } else if (mode == MODE_MACRO) {
        // MacroMolecularMode/division_death.jl:28-62: the seven pools, x, y, z and gen are
        // copied and halved in both (not age)
        double* const pools[7] = { P.PRO, P.DNA, P.RNA, P.CH, P.NST, P.PST, P.Chl };
        halve_pools(pools, p, d);
    } else if (mode == MODE_CARBON) {
        const double bd = P.Bd[d] * h, bp = P.Bd[p] * h;
        P.Bd[d] = bd; P.Bd[p] = bp;
        double* const pools[3] = { P.Sz, P.Bm, P.Chl };
        halve_pools(pools, p, d);
    } else {
        double* const pools[6] = { P.Sz, P.Bm, P.Cq, P.Nq, P.Pq, P.Chl };
        halve_pools(pools, p, d);
    }
}
__global__ void k_daughters(SpcDev P, const int32_t* __restrict__ divlist,
                            const int32_t* __restrict__ freelist, const uint32_t* ndiv,
                            const uint32_t* err, int mode) {
    if (*err & PI_DEVERR_CAPACITY) return;
    uint32_t n = *ndiv;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        daughter_pair(P, divlist[k], freelist[k], mode);
}

// The k-th divider (slot order) and the k-th free slot (findall(!ac), ascending) — get_tind!,
// Individuals/utils.jl:76-86 — from k_decide's bits, with the capacity check (plankton_update.jl:18-22). A block
// takes DIVIDE_WORDS words: each warp counts a run of them, then lists behind the warps and blocks before
// it. One block serves a species of up to DIVIDE_INBLOCK slots, and with `daughters` copies and halves them
// too; above, k64_divide_count leaves every block's counts first, and k_daughters follows. With 1, 2, 4 and 8
// times 1,048,576 slots: a scan of one 64-bit flag per slot and a list kernel 23, 31, 43 and 83 µs, one block for
// all of them 24, 43, 75 and 139, these two 15, 15, 16 and 16.
#define DIVIDE_WORDS 2048
__device__ __forceinline__ uint2 divide_count(const uint32_t* __restrict__ dvw, const uint32_t* __restrict__ frw, long long w0, long long w1) {
    uint32_t nd = 0, nf = 0;
#pragma unroll 4
    for (long long w = w0 + (threadIdx.x & 31); w < w1; w += 32) { nd += __popc(dvw[w]); nf += __popc(frw[w]); }
    return make_uint2(__reduce_add_sync(0xffffffffu, nd), __reduce_add_sync(0xffffffffu, nf));
}
__global__ void __launch_bounds__(1024) k64_divide_count(long long words, const uint32_t* __restrict__ dvw, const uint32_t* __restrict__ frw,
                                                         uint2* __restrict__ counts, const uint32_t* err) {
    __shared__ uint32_t shd[32], shf[32];
    if (*err & PI_DEVERR_CAPACITY) return;
    const int wid = threadIdx.x >> 5;
    const long long b0 = (long long)blockIdx.x * DIVIDE_WORDS, w0 = min(words, b0 + wid * (DIVIDE_WORDS / 32)), w1 = min(words, w0 + DIVIDE_WORDS / 32);
    const uint2 n = divide_count(dvw, frw, w0, w1);
    if ((threadIdx.x & 31) == 0) { shd[wid] = n.x; shf[wid] = n.y; }
    __syncthreads();
    if (wid) return;
    const uint32_t nd = __reduce_add_sync(0xffffffffu, shd[threadIdx.x]), nf = __reduce_add_sync(0xffffffffu, shf[threadIdx.x]);
    if (threadIdx.x == 0) counts[blockIdx.x] = make_uint2(nd, nf);
}
// words of a block: DIVIDE_WORDS, or all of them when it is the only one
__global__ void __launch_bounds__(1024) k64_divide(SpcDev P, long long C, const uint32_t* __restrict__ dvw,
                                                   const uint32_t* __restrict__ frw, const uint2* __restrict__ counts,
                                                   int32_t* divlist, int32_t* freelist,
                                                   uint32_t* ndiv, uint32_t* err, int64_t* err_iter, int64_t iter,
                                                   int daughters, int mode) {
    __shared__ uint32_t shd[32], shf[32], blk[4];
    if (*err & PI_DEVERR_CAPACITY) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long words = (C + 31) / 32, b0 = (long long)blockIdx.x * DIVIDE_WORDS, b1 = gridDim.x == 1 ? words : min(words, b0 + DIVIDE_WORDS);
    const long long run = (b1 - b0 + 1023) / 1024 * 32, w0 = min(b1, b0 + wid * run), w1 = min(b1, w0 + run);
    const uint2 own = divide_count(dvw, frw, w0, w1);
    const uint32_t nd = own.x, nf = own.y;
    if (lane == 0) { shd[wid] = nd; shf[wid] = nf; }
    if (threadIdx.x < 4) blk[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t tdiv = 0, tfree = 0, db = 0, fb = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < wid) { db += shd[w]; fb += shf[w]; }
        tdiv += shd[w]; tfree += shf[w];
    }
    if (gridDim.x > 1) {
        // all blocks' counts: the blocks before this one, and the totals
        uint32_t v[4] = { 0u, 0u, 0u, 0u };
        for (unsigned q = threadIdx.x; q < gridDim.x; q += blockDim.x) {
            const uint2 n = counts[q];
            if (q < blockIdx.x) { v[0] += n.x; v[1] += n.y; }
            v[2] += n.x; v[3] += n.y;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = __reduce_add_sync(0xffffffffu, v[q]);
            if (lane == 0 && v[q]) atomicAdd(&blk[q], v[q]);
        }
        __syncthreads();
        db += blk[0]; fb += blk[1]; tdiv = blk[2]; tfree = blk[3];
    }
    if (tdiv > tfree) {
        if (threadIdx.x == 0 && blockIdx.x == 0) { *ndiv = 0; *err_iter = iter; __threadfence(); set_err(err, PI_DEVERR_CAPACITY); }
        return;
    }
    if (threadIdx.x == 0 && blockIdx.x == 0) *ndiv = tdiv;
    if (tdiv == 0) return;
    for (long long w = w0; w < w1 && (nd || fb < tdiv); w += 32) {          // uniform over the warp
        uint32_t dw = nd && w + lane < w1 ? dvw[w + lane] : 0u, fw = fb < tdiv && w + lane < w1 ? frw[w + lane] : 0u;
        uint32_t cd = __popc(dw), cf = __popc(fw), xd = cd, xf = cf;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t yd = __shfl_up_sync(0xffffffffu, xd, o), yf = __shfl_up_sync(0xffffffffu, xf, o);
            if (lane >= o) { xd += yd; xf += yf; }
        }
        uint32_t rd = db + xd - cd, rf = fb + xf - cf;
        const int32_t s0 = (int32_t)((w + lane) * 32);
        while (dw) { divlist[rd++] = s0 + __ffs(dw) - 1; dw &= dw - 1u; }
        while (fw && rf < tdiv) { freelist[rf++] = s0 + __ffs(fw) - 1; fw &= fw - 1u; }
        db += __shfl_sync(0xffffffffu, xd, 31);
        fb += __shfl_sync(0xffffffffu, xf, 31);
    }
    if (!daughters) return;
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < tdiv; k += blockDim.x) daughter_pair(P, divlist[k], freelist[k], mode);
}

// ------------------------------------------------------------------------------------------
// (b) physiology — QuotaMode/plankton_growth.jl:2-24, growth_kernels.jl:2-166,
//     division_death_probability.jl:7-107, find_NPT! (utils.jl:14-25), calc_consume!
//     (consume_loss.jl:2-9), diags_proc!(num) (plankton_update.jl:33)
// ------------------------------------------------------------------------------------------

__device__ __forceinline__ double shape_dec(double x, double xmax, double k, int pw) {
    double fx = jl_max(0.0, jl_min(1.0, 1.0 - x / xmax));
    return pi_pow_int(fx, pw) / (k + pi_pow_int(fx, pw));
}
__device__ __forceinline__ double shape_inc(double x, double xmax, double k, int pw) {
    double fx = jl_max(0.0, jl_min(1.0, 1.0 - x / xmax));
    double reg = pi_pow_int(fx, pw) / (k + pi_pow_int(fx, pw));
    return 1.0 - reg;
}
// tempFunc's normaliser exp(-Ea / (R (Topt + 273.15))), a constant of the species formed on the host
// (pi_exp has the same bits there) and passed as OGT_rate
template <class P>
inline double ogt_rate(const P& p) { return pi_exp(-p.Ea / (F_RGAS * (p.Topt + F_T0))); }
__device__ __forceinline__ double tempFunc_PS(double T, const pi_quota_params& p, double OGT_rate) {
    double x = T - p.Topt, xmax = p.Tmax - p.Topt;
    double regT = shape_dec(x, xmax, F_4em2, 4);
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0))) * regT;
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}
__device__ __forceinline__ double tempFunc(double T, const pi_quota_params& p, double OGT_rate) {
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0)));
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}

struct TracerPtrs { const double* c[PI_NTRACERS]; };

__global__ void k_physiology(DGrid g, SpcDev P, pi_quota_params p, double ogt, long long C, int s,
                             double dT, double t, uint64_t seed, uint32_t iter, int shared_graz,
                             const double* __restrict__ NH4f, const double* __restrict__ NO3f,
                             const double* __restrict__ PO4f, const double* __restrict__ DOCf,
                             const double* __restrict__ par, const double* __restrict__ temp,
                             const uint32_t* __restrict__ off, const uint32_t* __restrict__ gid_sorted,
                             const int32_t* __restrict__ pos, double* __restrict__ contrib,
                             double* __restrict__ d_num, double* __restrict__ procv, const uint32_t* err) {
    long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C) return;
    if (*err & PI_DEVERR_CAPACITY) return;
    uint8_t f = P.flags[slot];
    int ac = f & FL_AC;
    int ac0 = P.stat[slot] & ST_AC0;
    long long e = ac0 ? pos[(long long)s * C + slot] : -1;
    if (!ac) {
        // Inactive after this step's deaths: every rate is multiplied by ac, the state is left
        // as it is (quotas of a lost individual are non-negative) and its decisions are 0.
        if (ac0) {
            double* K = contrib + e * 5;
            K[0] = 0.0; K[1] = 0.0; K[2] = 0.0; K[3] = 0.0; K[4] = 0.0;
        }
        return;
    }
    int xi, yi, zi;
    unpack_cell(g, P.cell[slot], xi, yi, zi);
    int c = gidx(g, xi, yi, zi);
    // find_NPT!: environment at the cell, times ac at gather time
    double NH4 = 0.0, NO3 = 0.0, PO4 = 0.0, DOC = 0.0, parv = 0.0, T = 0.0, pop = 0.0;
    if (ac0) {
        NH4 = jl_max(0.0, NH4f[c]); NO3 = jl_max(0.0, NO3f[c]); PO4 = jl_max(0.0, PO4f[c]);
        DOC = jl_max(0.0, DOCf[c]); parv = par[c]; T = temp[c];
        if (shared_graz) {
            pop = (double)(off[c + 1] - off[c]);
        } else {
            uint32_t n = 0;
            for (uint32_t q = off[c]; q < off[c + 1]; ++q) n += (gid_sorted[q] / (uint32_t)C) == (uint32_t)s;
            pop = (double)n;
        }
    }
    double Bm = P.Bm[slot], Cq = P.Cq[slot], Nq = P.Nq[slot], Pq = P.Pq[slot], Chl = P.Chl[slot];
    double age = P.age[slot];
    const double tf = tempFunc(T, p, ogt);
    // calc_inorganic_uptake_kernel! (growth_kernels.jl:48-56)
    double aI = parv * p.alpha * p.Phi;
    double PCm = p.PCmax * tempFunc_PS(T, p, ogt);
    double PS = PCm * (1.0 - pi_exp(-aI / jl_max(F_1em30, PCm) * Chl / jl_max(F_1em30, Bm))) * Bm;
    PS = jl_mulb(PS, ac);
    double VNH4, VNO3, VPO4;
    {
        double Qn = (Nq + Bm * p.R_NC) / jl_max(F_1em30, Bm + Cq);
        double Qp = (Pq + Bm * p.R_PC) / jl_max(F_1em30, Bm + Cq);
        double regQN = shape_dec(Qn, p.Nqmax, F_1em4, 4);
        double regQP = shape_dec(Qp, p.Pqmax, F_1em4, 4);
        double a = jl_mulb(p.VNH4max * regQN * NH4 / jl_max(F_1em30, NH4 + p.KsatNH4) * tf * Bm, ac);
        double b = jl_mulb(p.VNO3max * regQN * NO3 / jl_max(F_1em30, NO3 + p.KsatNO3) * tf * Bm, ac);
        double cc = jl_mulb(p.VPO4max * regQP * PO4 / jl_max(F_1em30, PO4 + p.KsatPO4) * tf * Bm, ac);
        VNH4 = jl_min(a, NH4 / dT / jl_max(1.0, pop));
        VNO3 = jl_min(b, NO3 / dT / jl_max(1.0, pop));
        VPO4 = jl_min(cc, PO4 / dT / jl_max(1.0, pop));
    }
    // update_quotas_1_kernel! (:64-69)
    Cq += PS * dT;
    Pq += VPO4 * dT;
    Nq += (VNH4 + VNO3) * dT;
    // calc_organic_uptake_kernel! (:78-84)
    double VDOC;
    {
        double Qc = Cq / jl_max(F_1em30, Bm + Cq);
        double regQ = shape_dec(Qc, p.Cqmax, F_1em4, 4);
        double VN = p.VDOCmax * regQ * DOC / jl_max(F_1em30, DOC + p.KsatDOC) * tf * Bm;
        VDOC = jl_mulb(jl_min(VN, DOC / dT / jl_max(1.0, pop)), ac);
        VDOC = jl_mulb(VDOC, jl_isless(F_1em2, PS / (VDOC + PS)));
    }
    // calc_ρChl_kernel! (:92-97)
    double rChl = jl_mulb(jl_mulb(PS / jl_max(F_1em30, Bm) * p.Chl2N /
                                  jl_max(F_1em30, parv * p.alpha * p.Phi * Chl / Bm),
                                  jl_isless(F_1em1, parv)), ac);
    // calc_respir_kernel! (:105-108)
    double resp = jl_mulb(p.respir * Bm * tf, ac);
    // update_quotas_2_kernel! (:117-124)
    Cq = Cq + (VDOC - resp) * dT;
    Bm = Bm - jl_max(0.0, (0.0 - Cq));
    Nq = Nq + jl_max(0.0, (0.0 - Cq)) * p.R_NC;
    Pq = Pq + jl_max(0.0, (0.0 - Cq)) * p.R_PC;
    Cq = Cq + jl_max(0.0, (0.0 - Cq));
    // calc_BS_kernel! (:132-138)
    double mn = jl_min(jl_min(Cq, Nq / p.R_NC), Pq / p.R_PC);
    double BS = jl_mulb(mn * p.k_mtb, ac);
    double exu = jl_mulb(jl_max(0.0, Cq - mn) * p.k_mtb, ac);
    // update_biomass_kernel! (:146-154)
    Bm += dT * BS;
    Cq -= dT * (BS + exu);
    Nq -= dT * BS * p.R_NC;
    Pq -= dT * BS * p.R_PC;
    Chl += dT * BS * p.R_NC * rChl;
    age += jl_mulb(dT / 3600.0, ac);
    // update_cellsize_kernel! (:163-166)
    double Sz = Bm / (p.Cquota * p.Nsuper);
    // probabilities (division_death_probability.jl:49-68, 26-30)
    double graz = jl_mulb(pop * p.grz_P, ac);
    double mort = jl_mulb(p.mort_P * shape_dec(Sz, p.mort_reg, F_1em5, 4), ac);
    double dv;
    int ty = (int)p.dvid_type;
    if (ty == 1) dv = p.dvid_P * shape_inc(Sz, p.dvid_reg, F_2em3, 2);
    else if (ty == 2) dv = p.dvid_P * shape_inc(fmod(t, 86400.0) / 3600.0, p.dvid_reg, F_1em5, 4);
    else dv = p.dvid_P * shape_inc(Sz, p.dvid_reg, F_1em3, 4) * shape_inc(fmod(t, 86400.0) / 3600.0, p.dvid_reg2, F_1em5, 4);
    double dvid = jl_mulb(dv, ac);
    // get_probability! (:95-107)
    double r0, r1, r2;
    pi_draw3(seed, iter, (uint32_t)s, PI_DRAW_DECISION, (uint32_t)slot, &r0, &r1, &r2);
    int dg = jl_isless(r0, graz * dT) && ac;
    int dm = jl_isless(r1, mort * dT) && ac;
    int dd = jl_isless(r2, dvid * dT) && ac;
    P.Bm[slot] = Bm; P.Cq[slot] = Cq; P.Nq[slot] = Nq; P.Pq[slot] = Pq; P.Chl[slot] = Chl;
    P.age[slot] = age; P.Sz[slot] = Sz;
    P.flags[slot] = (uint8_t)(FL_AC | (dg ? FL_GRAZ : 0) | (dm ? FL_MORT : 0) | (dd ? FL_DVID : 0));
    // calc_consume_kernel!: contributions kept per cell entry, summed in order later
    if (ac0) {
        double* K = contrib + e * 5;
        K[0] = jl_mulb((resp - PS) * dT, ac);
        K[1] = jl_mulb((exu - VDOC) * dT, ac);
        K[2] = jl_mulb(-VNH4 * dT, ac);
        K[3] = jl_mulb(-VNO3 * dT, ac);
        K[4] = jl_mulb(-VPO4 * dT, ac);
    }
    // diags_spcs! values of the slot (PI_PROC_* order), summed per cell in slot order later
    if (procv) {
        const double v[PI_NPROC] = { PS, BS, VDOC, VNH4, VNO3, VPO4, resp, exu, Bm, Cq, Nq, Pq, Chl };
        for (int q = 0; q < PI_NPROC; ++q) procv[(long long)q * C + slot] = v[q];
    }
    // diags_proc!(num, ac, ac) at the slot's (possibly stale) cell
    atomicAdd(&d_num[c], 1.0);
}

// ------------------------------------------------------------------------------------------
// CarbonMode physiology — CarbonMode/plankton_growth.jl:2-29, growth_kernels.jl:2-120,
// division_death_probability.jl:7-107, calc_consume! (consume_loss.jl:2-5)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double c_tempFunc_PS(double T, const pi_carbon_params& p, double OGT_rate) {
    double x = T - p.Topt, xmax = p.Tmax - p.Topt;
    double regT = shape_dec(x, xmax, F_1em1, 4);
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0))) * regT;
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}
__device__ __forceinline__ double c_tempFunc(double T, const pi_carbon_params& p, double OGT_rate) {
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0)));
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}
// gamma_alloc (growth_kernels.jl:22-26)
__device__ __forceinline__ double c_gamma(double Bm, double Bd, const pi_carbon_params& p) {
    double gm = jl_mulb(Bd / jl_max(F_1em30, Bm), jl_isless(0.0, Bd));
    return jl_mulb(jl_min(1.0, gm), p.thermal == 1.0);
}

__global__ void k_physiology_carbon(DGrid g, SpcDev P, pi_carbon_params p, double ogt, long long C, int s,
                                    double dT, double t, uint64_t seed, uint32_t iter, int shared_graz,
                                    const double* __restrict__ par, const double* __restrict__ temp,
                                    const uint32_t* __restrict__ off, const uint32_t* __restrict__ gid_sorted,
                                    const int32_t* __restrict__ pos, double* __restrict__ contrib,
                                    double* __restrict__ d_num, double* __restrict__ procv, const uint32_t* err) {
    long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C) return;
    if (*err & PI_DEVERR_CAPACITY) return;
    uint8_t f = P.flags[slot];
    int ac = f & FL_AC;
    int ac0 = P.stat[slot] & ST_AC0;
    long long e = ac0 ? pos[(long long)s * C + slot] : -1;
    if (!ac) {
        // inactive after this step's deaths: every rate that carries ac is 0. Thermal damage does
        // not (growth_kernels.jl:69-75), and an individual killed in this step gathered its
        // temperature while it was active, so its damaged biomass still grows by TD·ΔT; the
        // state of a slot inactive before the step keeps its values (T = 0 gives TD = 0).
        if (ac0) {
            double* K = contrib + e * 5;
            K[0] = 0.0; K[1] = 0.0; K[2] = 0.0; K[3] = 0.0; K[4] = 0.0;
            int xi, yi, zi;
            unpack_cell(g, P.cell[slot], xi, yi, zi);
            const double T = temp[gidx(g, xi, yi, zi)];
            const double Bm = P.Bm[slot], Bd = P.Bd[slot];
            double TD = jl_mulb(jl_mulb(jl_mulb((T - p.Topt) * p.f_T2B * (Bm - Bd), jl_isless(p.Topt, T)),
                                        jl_isless(Bd, Bm)), p.thermal == 1.0);
            TD = jl_max(0.0, jl_min(TD, (Bm - Bd) / dT));
            P.Bd[slot] = Bd + (TD - 0.0) * dT;           // RP = PS·γ = 0 (PS carries ac)
        }
        return;
    }
    int xi, yi, zi;
    unpack_cell(g, P.cell[slot], xi, yi, zi);
    int c = gidx(g, xi, yi, zi);
    double parv = 0.0, T = 0.0, pop = 0.0;
    if (ac0) {
        parv = par[c]; T = temp[c];
        if (shared_graz) {
            pop = (double)(off[c + 1] - off[c]);
        } else {
            uint32_t n = 0;
            for (uint32_t q = off[c]; q < off[c + 1]; ++q) n += (gid_sorted[q] / (uint32_t)C) == (uint32_t)s;
            pop = (double)n;
        }
    }
    double Bm = P.Bm[slot], Bd = P.Bd[slot], Chl = P.Chl[slot], age = P.age[slot];
    const double tf = c_tempFunc(T, p, ogt);
    // calc_PS! (calc_photosynthesis, growth_kernels.jl:29-36)
    double aI = parv * p.alpha * p.Phi;
    double PCm = p.PCmax * (tf * p.thermal + c_tempFunc_PS(T, p, ogt) * (1.0 - p.thermal));
    double light = 1.0 - pi_exp(-aI / jl_max(F_1em30, PCm) * Chl / jl_max(F_1em30, Bm));
    double PS = jl_mulb(PCm * jl_max(0.0, Bm - Bd) * (light * (1.0 - p.is_bact) + p.is_bact), ac);
    // calc_BS!, calc_repair! (:55-64), calc_thermal_damage! (:69-75), calc_respir! (:82-85)
    double BS = PS * (1.0 - c_gamma(Bm, Bd, p));
    double RP = PS * c_gamma(Bm, Bd, p);
    double TD = jl_mulb(jl_mulb(jl_mulb((T - p.Topt) * p.f_T2B * (Bm - Bd), jl_isless(p.Topt, T)),
                                jl_isless(Bd, Bm)), p.thermal == 1.0);
    TD = jl_max(0.0, jl_min(TD, (Bm - Bd) / dT));
    double RS = jl_mulb(p.respir * Bm * tf, ac);
    // update_quotas! (:92-97), update_cellsize! (:104-108)
    Bm += (BS - RS) * dT;
    Bd += (TD - RP) * dT;
    age += jl_mulb(dT / 3600.0, ac);
    double Sz = Bm / (p.Cquota * p.Nsuper);
    Chl = Bm * p.Chl2C;
    // probabilities (division_death_probability.jl:26-30, 49-52, 60-77)
    double graz = jl_mulb(pop * p.grz_P, ac);
    double dv;
    int ty = (int)p.dvid_type;
    if (ty == 1) dv = p.dvid_P * shape_inc(Sz, p.dvid_reg, F_2em3, 2);
    else if (ty == 2) dv = p.dvid_P * shape_inc(fmod(t, 86400.0) / 3600.0, p.dvid_reg, F_1em5, 4);
    else dv = p.dvid_P * shape_inc(Sz, p.dvid_reg, F_1em3, 4) * shape_inc(fmod(t, 86400.0) / 3600.0, p.dvid_reg2, F_1em5, 4);
    double dvid = jl_mulb(dv, ac);
    double mort = p.thermal == 1.0 ? jl_mulb(p.mort_P * shape_inc(Bd / jl_max(F_1em30, Bm), F_0p99, F_1em6, 4), ac)
                                   : jl_mulb(p.mort_P * shape_dec(Sz, p.mort_reg, F_1em5, 4), ac);
    // get_probability! (:95-107)
    double r0, r1, r2;
    pi_draw3(seed, iter, (uint32_t)s, PI_DRAW_DECISION, (uint32_t)slot, &r0, &r1, &r2);
    int dg = jl_isless(r0, graz * dT) && ac;
    int dm = jl_isless(r1, mort * dT) && ac;
    int dd = jl_isless(r2, dvid * dT) && ac;
    P.Bm[slot] = Bm; P.Bd[slot] = Bd; P.Chl[slot] = Chl; P.age[slot] = age; P.Sz[slot] = Sz;
    P.flags[slot] = (uint8_t)(FL_AC | (dg ? FL_GRAZ : 0) | (dm ? FL_MORT : 0) | (dd ? FL_DVID : 0));
    // calc_consume_kernel!: DIC only
    if (ac0) {
        double* K = contrib + e * 5;
        K[0] = jl_mulb((RS - PS) * dT, ac);
        K[1] = 0.0; K[2] = 0.0; K[3] = 0.0; K[4] = 0.0;
    }
    // diags_spcs! values of the slot (PI_CPROC_* order)
    if (procv) {
        const double v[PI_NCPROC] = { PS, BS, RP, RS, TD, Bm, Bd, Chl };
        for (int q = 0; q < PI_NCPROC; ++q) procv[(long long)q * C + slot] = v[q];
    }
    atomicAdd(&d_num[c], 1.0);
}

// ------------------------------------------------------------------------------------------
// MacroMolecularMode physiology — MacroMolecularMode/plankton_growth.jl:2-28, growth_kernels.jl:1-200,
// division_death_probability.jl:37-40, 49-52, 84-107, calc_consume! (consume_loss.jl:2-9)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double m_tempFunc_PS(double T, const pi_macro_params& p, double OGT_rate) {
    double x = T - p.Topt, xmax = p.Tmax - p.Topt;
    double regT = shape_dec(x, xmax, F_4em2, 4);
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0))) * regT;
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}
__device__ __forceinline__ double m_tempFunc(double T, const pi_macro_params& p, double OGT_rate) {
    double k = pi_exp(-p.Ea / (F_RGAS * (T + F_T0)));
    k = jl_max(0.0, k);
    return jl_min(1.0, k / OGT_rate);
}
// Every slot is updated: the synthesis and exudation terms carry no ac, so the state of an
// inactive slot keeps changing as in the reference, from zero light, temperature and nutrients
// unless it was active when they were gathered (an individual grazed or dead in this step).
__global__ void k_physiology_macro(DGrid g, SpcDev P, pi_macro_params p, double ogt, long long C, int s,
                                   double dT, uint64_t seed, uint32_t iter, int shared_graz,
                                   const double* __restrict__ NH4f, const double* __restrict__ NO3f,
                                   const double* __restrict__ PO4f, const double* __restrict__ DOCf,
                                   const double* __restrict__ par, const double* __restrict__ temp,
                                   const uint32_t* __restrict__ off, const uint32_t* __restrict__ gid_sorted,
                                   const int32_t* __restrict__ pos, double* __restrict__ contrib,
                                   double* __restrict__ d_num, double* __restrict__ procv, const uint32_t* err) {
    long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C) return;
    if (*err & PI_DEVERR_CAPACITY) return;
    const int ac = P.flags[slot] & FL_AC;
    const int ac0 = P.stat[slot] & ST_AC0;
    int c = -1;
    double NH4 = 0.0, NO3 = 0.0, PO4 = 0.0, DOC = 0.0, parv = 0.0, T = 0.0, pop = 0.0;
    if (ac0) {                                         // find_NPT! (utils.jl:14-25), × ac at gathering
        int xi, yi, zi;
        unpack_cell(g, P.cell[slot], xi, yi, zi);
        c = gidx(g, xi, yi, zi);
        NH4 = jl_max(0.0, NH4f[c]); NO3 = jl_max(0.0, NO3f[c]); PO4 = jl_max(0.0, PO4f[c]); DOC = jl_max(0.0, DOCf[c]);
        parv = par[c]; T = temp[c];
        if (shared_graz) {
            pop = (double)(off[c + 1] - off[c]);
        } else {
            uint32_t n = 0;
            for (uint32_t q = off[c]; q < off[c + 1]; ++q) n += (gid_sorted[q] / (uint32_t)C) == (uint32_t)s;
            pop = (double)n;
        }
    }
    double PRO = P.PRO[slot], DNA = P.DNA[slot], RNA = P.RNA[slot], CH = P.CH[slot];
    double NST = P.NST[slot], PST = P.PST[slot], Chl = P.Chl[slot], age = P.age[slot];
    const double tf = m_tempFunc(T, p, ogt);
    // calc_inorganic_uptake_kernel! (growth_kernels.jl:45-54): calc_PS (:20-25), calc_NP_uptake (:28-42)
    double aI = parv * p.alpha * p.Phi;
    double PCm = p.PCmax * m_tempFunc_PS(T, p, ogt);
    double PS = jl_mulb(PCm * (1.0 - pi_exp(-aI / jl_max(F_1em30, PCm) * Chl / jl_max(F_1em30, PRO))) * PRO, ac);
    double R_NST = NST / jl_max(F_1em30, m_totN(PRO, DNA, RNA, NST, Chl, p));
    double R_PST = PST / jl_max(F_1em30, m_totP(DNA, RNA, PST, p));
    double regQN = shape_dec(R_NST, p.NSTmax, F_1em4, 4), regQP = shape_dec(R_PST, p.PSTmax, F_1em4, 4);
    double VNH4 = jl_mulb(p.VNH4max * regQN * NH4 / jl_max(F_1em30, NH4 + p.KsatNH4) * tf * PRO, ac);
    double VNO3 = jl_mulb(p.VNO3max * regQN * NO3 / jl_max(F_1em30, NO3 + p.KsatNO3) * tf * PRO, ac);
    double VPO4 = jl_mulb(p.VPO4max * regQP * PO4 / jl_max(F_1em30, PO4 + p.KsatPO4) * tf * PRO, ac);
    VNH4 = jl_min(VNH4, NH4 / dT / jl_max(1.0, pop));
    VNO3 = jl_min(VNO3, NO3 / dT / jl_max(1.0, pop));
    VPO4 = jl_min(VPO4, PO4 / dT / jl_max(1.0, pop));
    // update_quotas_1_kernel! (:63-67)
    CH += PS * dT; PST += VPO4 * dT; NST += (VNH4 + VNO3) * dT;
    // calc_organic_uptake_kernel! (:82-90), calc_DOC_uptake (:73-80)
    double R_CH = CH / jl_max(F_1em30, m_totC(PRO, DNA, RNA, CH, Chl));
    double regQ = shape_dec(R_CH, p.CHmax, F_1em4, 4);
    double VN = p.VDOCmax * regQ * DOC / jl_max(F_1em30, DOC + p.KsatDOC) * tf * PRO;
    double VDOC = jl_mulb(jl_min(VN, DOC / dT / jl_max(1.0, pop)), ac);
    VDOC = jl_mulb(VDOC, jl_isless(F_5em2, PS / (VDOC + PS)));
    // calc_ρChl_kernel! (:98-103), calc_respir_kernel! (:111-114)
    double rChl = jl_mulb(jl_mulb(PS / jl_max(F_1em30, PRO) / jl_max(F_1em30, parv * p.alpha * p.Phi * Chl / jl_max(F_1em30, PRO)),
                                  jl_isless(F_1em1, parv)), ac);
    double resp = jl_mulb(p.respir * PRO * tf, ac);
    // update_quotas_2_kernel! (:124-130)
    CH = CH + (VDOC - resp) * dT;
    PRO = PRO - jl_max(0.0, 0.0 - CH);
    NST = NST + jl_max(0.0, 0.0 - CH) * p.R_NC_PRO;
    CH = CH + jl_max(0.0, 0.0 - CH);
    // calc_BS_kernel! (:136-152)
    double limit_PRO = jl_min(CH / (CH + p.k_sat_pro * p.Nsuper), NST / (NST + p.k_sat_pro * p.Nsuper * p.R_NC_PRO));
    double limit_DNA = jl_min(jl_min(CH / (CH + p.k_sat_dna * p.Nsuper), NST / (NST + p.k_sat_dna * p.Nsuper * p.R_NC_DNA)),
                              PST / (PST + p.k_sat_dna * p.Nsuper * p.R_PC_DNA));
    double limit_RNA = jl_min(jl_min(CH / (CH + p.k_sat_rna * p.Nsuper), NST / (NST + p.k_sat_rna * p.Nsuper * p.R_NC_RNA)),
                              PST / (PST + p.k_sat_rna * p.Nsuper * p.R_PC_RNA));
    double S_PRO = p.k_pro * RNA * limit_PRO * tf;
    double S_DNA = jl_mulb(p.k_dna * PRO * limit_DNA * tf, jl_isless(DNA / (p.C_DNA * p.Nsuper), 2.0));
    double S_RNA = p.k_rna * PRO * limit_RNA * tf;
    // update_biomass_kernel! (:159-171)
    PRO += dT * S_PRO;
    DNA += dT * S_DNA;
    RNA += dT * S_RNA;
    CH -= dT * (S_PRO + S_DNA + S_RNA + S_PRO * rChl);
    NST -= dT * (S_PRO * p.R_NC_PRO + S_DNA * p.R_NC_DNA + S_RNA * p.R_NC_RNA + S_PRO * rChl * 4.0 / 55.0);
    PST -= dT * (S_DNA * p.R_PC_DNA + S_RNA * p.R_PC_RNA);
    Chl += dT * S_PRO * rChl * F_CHL / 55.0;
    age += jl_mulb(dT / 3600.0, ac);
    // calc_exudation_kernel! (:179-183), update_CH_kernel! (:190-193)
    double exu = jl_max(0.0, CH - p.CHmax * m_totC(PRO, DNA, RNA, CH, Chl));
    CH -= exu;
    // calc_graz_quadratic!, calc_MM_mort!, calc_MM_dvid!, get_probability!
    double graz = jl_mulb(pop * p.grz_P, ac);
    double mort = jl_mulb(p.mort_P * shape_inc(age, p.mort_reg, F_1em4, 4), ac);
    double dvid = jl_mulb(p.dvid_P, jl_isless(2.0, DNA / (p.C_DNA * p.Nsuper)));
    double r0, r1, r2;
    pi_draw3(seed, iter, (uint32_t)s, PI_DRAW_DECISION, (uint32_t)slot, &r0, &r1, &r2);
    int dg = jl_isless(r0, graz * dT) && ac;
    int dm = jl_isless(r1, mort * dT) && ac;
    int dd = jl_isless(r2, dvid * dT) && ac;
    P.PRO[slot] = PRO; P.DNA[slot] = DNA; P.RNA[slot] = RNA; P.CH[slot] = CH;
    P.NST[slot] = NST; P.PST[slot] = PST; P.Chl[slot] = Chl; P.age[slot] = age;
    P.flags[slot] = (uint8_t)((ac ? FL_AC : 0) | (dg ? FL_GRAZ : 0) | (dm ? FL_MORT : 0) | (dd ? FL_DVID : 0));
    // calc_consume_kernel! (consume_loss.jl:2-9) for the individuals binned this step
    if (ac0) {
        double* K = contrib + (long long)pos[(long long)s * C + slot] * 5;
        K[0] = jl_mulb((resp - PS) * dT, ac);
        K[1] = jl_mulb((exu - VDOC) * dT, ac);
        K[2] = jl_mulb(-VNH4 * dT, ac);
        K[3] = jl_mulb(-VNO3 * dT, ac);
        K[4] = jl_mulb(-VPO4 * dT, ac);
    }
    // diags_spcs! (Diagnostics/diagnostics_kernels.jl:20-21) in PI_MPROC_* order: VNH4 (listed
    // there as :VHN4) and exu are never accumulated
    if (procv) {
        const double v[PI_NMPROC] = { PS, VDOC, 0.0, VNO3, VPO4, resp, rChl, S_PRO, S_DNA, S_RNA, 0.0,
                                      CH, NST, PST, PRO, DNA, RNA, Chl };
        for (int q = 0; q < PI_NMPROC; ++q) procv[(long long)q * C + slot] = v[q];
    }
    if (ac) {
        int xi, yi, zi;
        unpack_cell(g, P.cell[slot], xi, yi, zi);
        atomicAdd(&d_num[gidx(g, xi, yi, zi)], 1.0);
    }
}

// diags_spcs! (Diagnostics/diagnostics_kernels.jl:14-33): the cell of every slot active after the
// species' update (its find_inds! cell), G for the others, for a stable sort by cell.
__global__ void k_diag_keys(DGrid g, SpcDev P, long long C, uint32_t* __restrict__ key, uint32_t* __restrict__ val,
                            const uint32_t* err) {
    const long long slot = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C) return;
    uint32_t k = (uint32_t)g.G;
    if (!(*err & PI_DEVERR_CAPACITY) && (P.flags[slot] & FL_AC)) {
        int xi, yi, zi;
        unpack_cell(g, P.cell[slot], xi, yi, zi);
        k = (uint32_t)gidx(g, xi, yi, zi);
    }
    key[slot] = k;
    val[slot] = (uint32_t)slot;
}

// d[cell] += value of each of the cell's slots in ascending slot order (the sorted run of the
// cell), for the enabled processes; one thread per run.
__global__ void k_diag_sum(long long C, long long G, const uint32_t* __restrict__ key, const uint32_t* __restrict__ val,
                           const double* __restrict__ procv, uint32_t mask, double* __restrict__ d) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C) return;
    const uint32_t c = key[i];
    if (c >= (uint32_t)G || (i > 0 && key[i - 1] == c)) return;
    for (int q = 0; q < PI_MAXPROC; ++q) {
        if (!(mask >> q & 1u)) continue;
        double x = d[(long long)q * G + c];
        for (long long j = i; j < C && key[j] == c; ++j) x = x + procv[(long long)q * C + val[j]];
        d[(long long)q * G + c] = x;
    }
}

// diags.tracer[name] .+= tracer (time_step.jl:168-172) for the enabled tracers, halos included.
__global__ void k_diag_tracers(double* __restrict__ d, const double* __restrict__ tr, uint32_t mask, long long G,
                               const uint32_t* err) {
    if (*err & PI_DEVERR_CAPACITY) return;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < (long long)PI_NTRACERS * G;
         q += (long long)gridDim.x * blockDim.x)
        if (mask >> (q / G) & 1u) d[q] = d[q] + tr[q];
}

// ------------------------------------------------------------------------------------------
// (d) tracer update — Biogeochemistry/tracer_update.jl:22-43, Advection/DST3FL.jl:1-73,
//     Advection/multi_dim_adv.jl:1-135, operaters.jl:1-27, tracer_diffusion.jl, tracer_sinking.jl,
//     tracer_forcings.jl, HaloRegions/apply_bcs.jl
// ------------------------------------------------------------------------------------------

__device__ __forceinline__ double theta(double dnum, double d0) {
    return fabs(d0) * F_THMAX <= fabs(dnum) ? copysign(F_THMAX, dnum * d0) : dnum / d0;
}
__device__ __forceinline__ double psi_lim(double cfl, double th) {
    double d0 = (2.0 - cfl) * (1.0 - cfl) / 6.0;
    double d1 = (1.0 - cfl * cfl) / 6.0;
    return jl_max(0.0, jl_min(jl_min(1.0, d0 + d1 * th), th * (1.0 - cfl) / (cfl + F_1em20)));
}
// DST3FL face flux on one axis from the 4 values around the face (cm2 = c[i-2], cm1 = c[i-1],
// c0 = c[i], cp1 = c[i+1]) and the landmask at those points. UP = 1 for x/y (upwind cell i-1),
// UP = 0 for z (index grows downward: upwind cell is k for upward flow), adv_flux_x/y/z.
__device__ __forceinline__ double dst3_flux_xy(double cm2, double cm1, double c0, double cp1,
                                               int lm2, int lm1, int l0, int lp1,
                                               double vel, double area, double dxc, double dT) {
    double cfl = fabs(vel * dT / dxc);
    double tr = area * vel;
    double d0 = jl_mulb(jl_mulb(c0 - cm1, l0), lm1);     // δ⁰ = (c[i] - c[i-1])
    double dm = jl_mulb(jl_mulb(cm1 - cm2, lm1), lm2);   // δ⁻ = (c[i-1] - c[i-2])
    double dp = jl_mulb(jl_mulb(cp1 - c0, lp1), l0);     // δ⁺ = (c[i+1] - c[i])
    double psp = psi_lim(cfl, theta(dm, d0));
    double psm = psi_lim(cfl, theta(dp, d0));
    return 0.5 * (tr + fabs(tr)) * (cm1 + psp * d0) + 0.5 * (tr - fabs(tr)) * (c0 - psm * d0);
}
// z: cm2 = c[k-2], cm1 = c[k-1], c0 = c[k], cp1 = c[k+1]
__device__ __forceinline__ double dst3_flux_z(double cm2, double cm1, double c0, double cp1,
                                              int lm2, int lm1, int l0, int lp1,
                                              double w, double area, double dzc, double dT) {
    double cfl = fabs(w * dT / dzc);
    double tr = area * w;
    double d0 = jl_mulb(jl_mulb(cm1 - c0, l0), lm1);     // δz⁰ = c[k-1] - c[k]
    double dm = jl_mulb(jl_mulb(cm2 - cm1, lm1), lm2);   // δz⁻ = c[k-2] - c[k-1]
    double dp = jl_mulb(jl_mulb(c0 - cp1, lp1), l0);     // δz⁺ = c[k] - c[k+1]
    double psp = psi_lim(cfl, theta(dm, d0));            // Ψz⁺
    double psm = psi_lim(cfl, theta(dp, d0));            // Ψz⁻
    return 0.5 * (tr + fabs(tr)) * (c0 + psm * d0) + 0.5 * (tr - fabs(tr)) * (cm1 - psp * d0);
}

// Index maps that stand in for the halo fill of tracer_temp between sweeps.
__device__ __forceinline__ int wrap_axis(int a, int N, int H, int topo) {
    if (topo == PI_PERIODIC) {
        while (a < H + 1) a += N;
        while (a > N + H) a -= N;
        return a;
    }
    return a < H + 1 ? H + 1 : (a > N + H ? N + H : a);
}

// Per-face quantities of DST3FL that do not depend on the tracer (CFL, transport, d₀ and d₁ of
// DST3FL.jl:5-11, the factors of adv_flux): computed once per face and shared by the 14 tracers.
// Each is the same IEEE expression the per-tracer formula evaluates, so results are unchanged.
struct FaceCoef { double d0c, d1c, omc, cpe, hp, hm; };

__device__ __forceinline__ FaceCoef face_coef(double vel, double area, double dxc, double dT) {
    FaceCoef f;
    double cfl = fabs(vel * dT / dxc);
    double tr = area * vel;
    f.d0c = (2.0 - cfl) * (1.0 - cfl) / 6.0;
    f.d1c = (1.0 - cfl * cfl) / 6.0;
    f.omc = 1.0 - cfl;
    f.cpe = cfl + F_1em20;
    f.hp = 0.5 * (tr + fabs(tr));
    f.hm = 0.5 * (tr - fabs(tr));
    return f;
}
__device__ __forceinline__ double getbc_dev(const FluxBCDev& b, int a, int c, int64_t it) {
    if (b.kind == PI_BC_CONST) return b.v[0];
    if (b.kind == PI_BC_ARRAY2D) return b.v[(a - 1) + (long long)b.n1 * (c - 1)];
    const int64_t t = it < 1 ? 1 : (it > b.nt ? b.nt : it);   // the host rejects steps past nt
    return b.v[(a - 1) + (long long)b.n1 * ((c - 1) + (long long)b.n2 * (t - 1))];
}

// fill_halo_tracer! in three passes (x, y, z), where a periodic axis has fewer cells than halo points
// (k64_halo otherwise). Each thread owns one line along the axis and
// reads all its source values before writing, as Julia's broadcast unaliases views.
template <int AXIS>
__global__ void k_halo(DGrid g, double* __restrict__ f, int nfields, const uint32_t* err) {
    int a = blockIdx.x * blockDim.x + threadIdx.x + 1;   // first transverse index
    int b = blockIdx.y + 1;                              // second transverse index
    int n = blockIdx.z;
    int na = AXIS == 0 ? g.Gy : g.Gx;
    if (a > na || n >= nfields) return;
    if (err && (*err & PI_DEVERR_CAPACITY)) return;
    int N = AXIS == 0 ? g.Nx : AXIS == 1 ? g.Ny : g.Nz;
    int H = AXIS == 0 ? g.Hx : AXIS == 1 ? g.Hy : g.Hz;
    int topo = AXIS == 0 ? g.tx : AXIS == 1 ? g.ty : g.tz;
    double* c = f + (long long)n * g.G;
    auto at = [&](int t) -> double& {
        if (AXIS == 0) return c[gidx(g, t, a, b)];
        if (AXIS == 1) return c[gidx(g, a, t, b)];
        return c[gidx(g, a, b, t)];
    };
    double wv[8], ev[8];
    for (int h = 1; h <= H; ++h) {
        wv[h - 1] = topo == PI_PERIODIC ? at(N + h) : at(H + 1);
        ev[h - 1] = topo == PI_PERIODIC ? at(H + h) : at(N + H);
    }
    for (int h = 1; h <= H; ++h) {
        at(h) = wv[h - 1];
        at(N + H + h) = ev[h - 1];
    }
}

// Interior array (reference layout nx×ny×nz, x fastest) into a halo-padded field at offset
// (Hx, Hy, Hz): copy_interior! / copy_interior_u! (Simulation/utils.jl:13-34).
__global__ void k_scatter_interior(DGrid g, double* __restrict__ dst, const double* __restrict__ src,
                                   int nx, int ny, int nz) {
    long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long n = (long long)nx * ny * nz;
    if (q >= n) return;
    int i = (int)(q % nx);
    long long r = q / nx;
    int j = (int)(r % ny);
    int k = (int)(r / ny);
    dst[gidx(g, i + 1 + g.Hx, j + 1 + g.Hy, k + 1 + g.Hz)] = src[q];
}

// Velocity halo rule along one axis (fill_halo_u/v/w!, halo_regions.jl:64-99) when the field is a
// face field on that axis and the axis is Bounded: the high halo copies the extra face N+H+1.
// Otherwise the tracer rule. One thread per line; sources are read before writes.
template <int AXIS>
__global__ void k_halo_vel(DGrid g, double* __restrict__ c, int face_axis) {
    int a = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int b = blockIdx.y + 1;
    int na = AXIS == 0 ? g.Gy : g.Gx;
    if (a > na) return;
    int N = AXIS == 0 ? g.Nx : AXIS == 1 ? g.Ny : g.Nz;
    int H = AXIS == 0 ? g.Hx : AXIS == 1 ? g.Hy : g.Hz;
    int topo = AXIS == 0 ? g.tx : AXIS == 1 ? g.ty : g.tz;
    auto at = [&](int t) -> double& {
        if (AXIS == 0) return c[gidx(g, t, a, b)];
        if (AXIS == 1) return c[gidx(g, a, t, b)];
        return c[gidx(g, a, b, t)];
    };
    double wv[8], ev[8];
    int velrule = (face_axis == AXIS) && topo == PI_BOUNDED;
    for (int h = 1; h <= H; ++h) {
        wv[h - 1] = topo == PI_PERIODIC ? at(N + h) : at(H + 1);
        ev[h - 1] = topo == PI_PERIODIC ? at(H + h) : at(N + H);
    }
    double face = velrule ? at(N + H + 1) : 0.0;
    for (int h = 1; h <= H; ++h) at(h) = wv[h - 1];
    if (velrule) {
        for (int h = N + H + 2; h <= N + 2 * H; ++h) at(h) = face;
    } else {
        for (int h = 1; h <= H; ++h) at(N + H + h) = ev[h - 1];
    }
}

// Slots s0 .. s0 + n - 1 of the boundary's columns that are not stored as such: graz, mort and dvid as
// Float64 and xi, yi and zi as int64 (bits 0-5 of mask), 8-byte columns of n one after another in
// `out`, then ac as bytes (bit 6).
__global__ void k64_export(DGrid g, SpcDev P, long long s0, long long n, uint32_t mask, unsigned long long* __restrict__ out) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const uint8_t f = P.flags[s0 + t];
    int x[3];
    unpack_cell(g, P.cell[s0 + t], x[0], x[1], x[2]);
    const uint8_t bits[3] = { FL_GRAZ, FL_MORT, FL_DVID };
    long long at = 0;
    for (int q = 0; q < 6; ++q) {
        if (!(mask >> q & 1u)) continue;
        out[at * n + t] = q < 3 ? (unsigned long long)__double_as_longlong(f & bits[q] ? 1.0 : 0.0) : (unsigned long long)x[q - 3];
        ++at;
    }
    if (mask >> 6 & 1u) reinterpret_cast<uint8_t*>(out + at * n)[t] = f & FL_AC ? 1 : 0;
}

// Index of the first non-finite value of a[0, n) (atomicMin into *first, which starts at ~0).
__global__ void k_first_nonfinite(const double* __restrict__ a, long long n, unsigned long long* first) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        if (!isfinite(a[q])) atomicMin(first, (unsigned long long)q);
}

// First active slot of a species with a non-finite Float64 attribute.
__global__ void k_first_nonfinite_inds(SpcDev s, long long C, unsigned long long* first) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x) {
        if (!(s.flags[q] & FL_AC)) continue;
        const double v[11] = { s.x[q], s.y[q], s.z[q], s.Sz[q], s.Bm[q], s.Cq[q], s.Nq[q], s.Pq[q], s.Chl[q], s.gen[q], s.age[q] };
        bool bad = false;
        for (int k = 0; k < 11; ++k) bad |= !isfinite(v[k]);
        if (s.PRO) {                                  // MacroMolecularMode pools
            const double w[6] = { s.PRO[q], s.DNA[q], s.RNA[q], s.CH[q], s.NST[q], s.PST[q] };
            for (int k = 0; k < 6; ++k) bad |= !isfinite(w[k]);
        }
        if (bad) atomicMin(first, (unsigned long long)q);
    }
}

// Mass budgets (no counterpart in the reference): block partials of the interior Σ vol·c of the
// carbon (DIC+DOC+POC), nitrogen (NH4+NO3+DON+PON) and phosphorus (PO4+DOP+POP) tracers, and of the
// active individuals' C (Bm+Cq), N (Bm·R_NC+Nq) and P (Bm·R_PC+Pq). Each block sums a fixed set of
// cells (slots) in a fixed order, so the result does not depend on the run.
__device__ __forceinline__ void block_sum3(double c, double n, double p, double* partial) {
    __shared__ double sh[3][256];
    sh[0][threadIdx.x] = c; sh[1][threadIdx.x] = n; sh[2][threadIdx.x] = p;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) for (int r = 0; r < 3; ++r) sh[r][threadIdx.x] += sh[r][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) for (int r = 0; r < 3; ++r) partial[blockIdx.x * 3 + r] = sh[r][0];
}
__global__ void __launch_bounds__(256) k_budget_cells(DGrid g, const double* __restrict__ tr, double* __restrict__ partial) {
    double c = 0.0, n = 0.0, p = 0.0;
    const long long V = (long long)g.Nx * g.Ny * g.Nz, G = g.G;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < V; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % g.Nx) + 1 + g.Hx;
        const long long r = q / g.Nx;
        const int j = (int)(r % g.Ny) + 1 + g.Hy, k = (int)(r / g.Ny) + 1 + g.Hz;
        const long long cq = gidx(g, i, j, k);
        const double vol = g.mVol ? pib::vol<true>(g, i, j, k) : pib::vol<false>(g, i, j, k);
        c += vol * (tr[PI_DIC * G + cq] + tr[PI_DOC * G + cq] + tr[PI_POC * G + cq]);
        n += vol * (tr[PI_NH4 * G + cq] + tr[PI_NO3 * G + cq] + tr[PI_DON * G + cq] + tr[PI_PON * G + cq]);
        p += vol * (tr[PI_PO4 * G + cq] + tr[PI_DOP * G + cq] + tr[PI_POP * G + cq]);
    }
    block_sum3(c, n, p, partial);
}
__global__ void __launch_bounds__(256) k_budget_inds(SpcDev s, long long C, double R_NC, double R_PC, double* __restrict__ partial) {
    double c = 0.0, n = 0.0, p = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x) {
        if (!(s.flags[q] & FL_AC)) continue;
        const double Bm = s.Bm[q];
        c += Bm + s.Cq[q];
        n += Bm * R_NC + s.Nq[q];
        p += Bm * R_PC + s.Pq[q];
    }
    block_sum3(c, n, p, partial);
}

// MacroMolecularMode individuals: total_C/N/P_biomass (plankton_generation.jl:82-93) of the active ones
__global__ void __launch_bounds__(256) k_budget_inds_macro(SpcDev s, long long C, pi_macro_params mp, double* __restrict__ partial) {
    double c = 0.0, n = 0.0, p = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x) {
        if (!(s.flags[q] & FL_AC)) continue;
        c += m_totC(s.PRO[q], s.DNA[q], s.RNA[q], s.CH[q], s.Chl[q]);
        n += m_totN(s.PRO[q], s.DNA[q], s.RNA[q], s.NST[q], s.Chl[q], mp);
        p += m_totP(s.DNA[q], s.RNA[q], s.PST[q], mp);
    }
    block_sum3(c, n, p, partial);
}

// Active individuals of one species (calc_active_individuals, models.jl:157-164).
__global__ void k_count_active(const uint8_t* __restrict__ flags, long long C, unsigned long long* out) {
    unsigned long long n = 0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x)
        n += (flags[q] & FL_AC) ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(out, n);
}

// After a capacity error the step stops where the reference throws: the tracers keep their
// values, so the buffer that becomes current is a copy of the old one.
__global__ void k_copy_if_err(double* __restrict__ dst, const double* __restrict__ src, long long n,
                              const uint32_t* err) {
    if (!(*err & PI_DEVERR_CAPACITY)) return;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = src[q];
}

}  // namespace pib
