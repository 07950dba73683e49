// FP32 form: kernels. Every launch covers all members of a batch; blocks and warps find their
// member through work tables built when the batch is created.
//
// The formulas are those of the FP64 kernels (and of the reference lines they cite) evaluated in
// Float32, with three changes of representation:
//  - a position is an interior cell (ci, cj, ck) plus an in-cell offset in [0, 1): find_inds! is
//    the cell itself, interpolation weights come straight from the offsets, and the precision of a
//    position does not degrade with the size of the grid;
//  - particle→grid sums (Chl for light, consumption, grazing and mortality losses) are 64-bit
//    fixed-point integers added with atomics; integer addition commutes, so the sums do not depend
//    on the order in which individuals are visited and no sort is needed for determinism; pop and
//    the diagnostic counts are exact integer counts;
//  - Sz is not stored: it is Bm / (Cquota Nsuper), as update_cellsize_kernel! sets it;
//  - individuals are stored in a physical order grouped by cell (kept by a periodic counting sort)
//    behind their logical slot numbers: draws are keyed by the logical slot and the division
//    bookkeeping runs on bitmaps over logical slots, so the order changes no result.
// FP64 is used for the fixed-point conversions, the mass budgets and the DST3FL limiter ratio
// where the centred gradient is within a few FP32 ulps of zero.
#pragma once

#include <cstddef>

#include "fp32_internal.h"

namespace p32 {

#define THMAX_F 1.0e20f
#define EPS20_F 1.0e-20f

struct Tab32 {
    const MemberDev* md;
    int nsp;
    const int2* tiles;        // {segment = member*nsp + species, first slot}, F32_TILE slots each
    int ntiles;
    const int* seg_tile0;     // first tile of each segment (nseg + 1 entries)
    const int4* icol; int nicol;  // column warps {m, i0, j, 0}
};

__device__ __forceinline__ int gid3(const MemberDev& m, int i, int j, int k) {   // 1-based, member-local
    return (i - 1) + m.Gx * ((j - 1) + m.Gy * (k - 1));
}
__device__ __forceinline__ int lm32(const MemberDev& m, const uint8_t* __restrict__ lm, int i, int j, int k) {
    return m.all_water ? 1 : (int)lm[m.cell_off + gid3(m, i, j, k)];
}
__device__ __forceinline__ float mulbf(float x, int b) { return b ? x : copysignf(0.0f, x); }
__device__ __forceinline__ void seterr(uint32_t* err, uint32_t bit) { atomicOr(err, bit); }
__device__ __forceinline__ bool stopped(const uint32_t* err) {
    return (*(volatile const uint32_t*)err & F32_ERR_CAPACITY) != 0;
}
__device__ __forceinline__ void seg_of(const Tab32& T, int seg, int& m, int& s) { m = seg / T.nsp; s = seg - m * T.nsp; }

// ------------------------------------------------------------------------------------------
// cells and positions
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void unpack_int(const MemberDev& m, int32_t code, int& ci, int& cj, int& ck) {
    f32_unpack(code, m.cbx, m.cby, ci, cj, ck);
}
__device__ __forceinline__ int32_t pack_int(const MemberDev& m, int ci, int cj, int ck) {
    return f32_pack(ci, cj, ck, m.cbx, m.cby);
}
__device__ __forceinline__ int32_t pack_halo(const MemberDev& m, int xi, int yi, int zi) {
    return f32_pack(xi, yi, zi, m.hbx, m.hby);
}
__device__ __forceinline__ void unpack_halo(const MemberDev& m, int32_t c, int& xi, int& yi, int& zi) {
    f32_unpack(c, m.hbx, m.hby, xi, yi, zi);
}
// halo-inclusive member-local cell of an interior position cell (find_inds!, Individuals/utils.jl:2-7)
__device__ __forceinline__ int q_of(const MemberDev& m, int ci, int cj, int ck) {
    return gid3(m, ci + 1 + m.Hx, cj + 1 + m.Hy, ck + 1 + m.Hz);
}
__device__ __forceinline__ bool interior_q(const MemberDev& m, int q) {
    const int i = q % m.Gx + 1, r = q / m.Gx, j = r % m.Gy + 1, k = r / m.Gy + 1;
    return i > m.Hx && i <= m.Nx + m.Hx && j > m.Hy && j <= m.Ny + m.Hy && k > m.Hz && k <= m.Nz + m.Hz;
}

struct Ax1 { int c; float o; };

// particle_boundary_condition (particle_advection_kernels.jl:2-11) on x = c + o
__device__ __forceinline__ void bc_axis(Ax1& a, int N, int topo) {
    const bool above = a.c > N || (a.c == N && a.o > 0.0f);
    const bool below = a.c < 0;
    if (topo == PI_PERIODIC) {
        if (above) a.c -= N;
        else if (below) a.c += N;
    } else if (above || below) {              // x → 2N − x or x → −x
        const int pivot = above ? 2 * N : 0;
        if (a.o > 0.0f) { a.c = pivot - a.c - 1; a.o = 1.0f - a.o; } else { a.c = pivot - a.c; }
        if (a.o >= 1.0f) { a.c += 1; a.o = 0.0f; }
    }
}
__device__ __forceinline__ void move(Ax1& a, float d, int N, int topo) {
    const float o = a.o + d;
    const float n = floorf(o);
    a.c += (int)n;
    a.o = o - n;
    if (a.o >= 1.0f) { a.c += 1; a.o = 0.0f; }
    bc_axis(a, N, topo);
}
// move() to an RK stage position, which is only sampled: a position left outside [0, N] by a
// displacement above one domain length (CFL far above 1) is noted in `bad` and held at the edge,
// so every corner index of the interpolation stays inside the halo-padded grid (H >= 2)
__device__ __forceinline__ void move_stage(Ax1& a, float d, int N, int topo, bool& bad) {
    move(a, d, N, topo);
    if (a.c < 0 || a.c > N) { bad = true; a.c = a.c < 0 ? 0 : N; a.o = 0.0f; }
}

// index and weight along one axis for a face-centred (own axis) or cell-centred field
// (interpolation.jl:3-83: x + 1 or x + 0.5 split into trunc and mod)
__device__ __forceinline__ void axis_iw(const Ax1& a, int H, bool face, int& idx, float& w) {
    if (face) { idx = a.c + 1 + H; w = a.o; return; }
    const bool lo = a.o < 0.5f;
    idx = a.c + H + (lo ? 0 : 1);
    w = lo ? a.o + 0.5f : a.o - 0.5f;
}
// clamp into [lo, hi], noting an index outside in `bad` (reported once per individual)
__device__ __forceinline__ int clampb(int v, int lo, int hi, bool& bad) {
    const int c = min(max(v, lo), hi);
    bad |= c != v;
    return c;
}

// The 8 corner values of each velocity component around a position, at (i + a, j + b, k + c) of the
// component's base corner q (the vertical component in levels per second, its ΔzC differing between the
// two). The four RK stages of a step sample points a small fraction of a cell apart, usually from the
// same field (vel₀ = vel½ = vel₁ between velocity refreshes), so a stage reuses the corners of the
// previous one when the field and the base corners are the same.
struct Corners { int fid; int q[3]; float v[3][8]; };      // fid: 0 vel₀, 1 vel½, 2 vel₁

// Member constants of the particle kernels, held in registers.
struct PGeom {
    int Nx, Ny, Nz, Hx, Hy, Hz, Gx, Gy, Gz, tx, ty, tz, dz_off;
    float rdx, rdy;
    int fh, f1;     // field ids of vel½ and vel₁ (fields that are the same arrays share an id)
};
__device__ __forceinline__ bool same3(const float* const* a, const float* const* b) {
    return a[0] == b[0] && a[1] == b[1] && a[2] == b[2];
}
__device__ __forceinline__ PGeom pgeom(const MemberDev& m, const MemberForcing& f) {
    PGeom g;
    g.fh = same3(f.velh, f.vel0) ? 0 : 1;
    g.f1 = same3(f.vel1, f.velh) ? g.fh : same3(f.vel1, f.vel0) ? 0 : 2;
    g.Nx = m.Nx; g.Ny = m.Ny; g.Nz = m.Nz; g.Hx = m.Hx; g.Hy = m.Hy; g.Hz = m.Hz;
    g.Gx = m.Gx; g.Gy = m.Gy; g.Gz = m.Gz; g.tx = m.tx; g.ty = m.ty; g.tz = m.tz; g.dz_off = m.dz_off;
    g.rdx = m.rdx; g.rdy = m.rdy;
    return g;
}

// trilinear interpolation of the three velocity components (member-local fields), in grid cells per second
// The 8 corner values come from the component's own halo-padded field: in the cell-sorted
// storage order the lanes of a warp sit in neighbouring cells, so the corner loads of a warp
// share sectors and the fields (12 bytes per cell) stay in L2. In a warp some lane nearly always needs
// other corners, of any component: one branch loads those of all three, so that a stage waits for memory
// once, not three times.
// Every position passed here lies in [0, N] on each axis (uploads are validated, stored positions
// are clamped, stage positions pass through move_stage), so with H >= 2 the base corner (i, j, k)
// satisfies 1 <= i <= Gx - 1 (likewise j, k) and needs no clamp.
__device__ __forceinline__ void itpl32(const PGeom& m, const float* const* fld, int fid, const float* __restrict__ rdzC,
                                       const Ax1& X, const Ax1& Y, const Ax1& Z, Corners& cc, float& u, float& v, float& w) {
    // own axis: on the faces; the other two: between the cell centres
    int iF, jF, kF, iC, jC, kC;
    float wx[2], wy[2], wz[2];
    axis_iw(X, m.Hx, true, iF, wx[1]); axis_iw(Y, m.Hy, true, jF, wy[1]); axis_iw(Z, m.Hz, true, kF, wz[1]);
    axis_iw(X, m.Hx, false, iC, wx[0]); axis_iw(Y, m.Hy, false, jC, wy[0]); axis_iw(Z, m.Hz, false, kC, wz[0]);
    const int sy = m.Gx, sz = m.Gx * m.Gy;
    const int q[3] = { (iF - 1) + sy * (jC - 1) + sz * (kC - 1), (iC - 1) + sy * (jF - 1) + sz * (kC - 1),
                       (iC - 1) + sy * (jC - 1) + sz * (kF - 1) };
    if (cc.fid != fid || cc.q[0] != q[0] || cc.q[1] != q[1] || cc.q[2] != q[2]) {
        cc.fid = fid;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float* __restrict__ p = fld[c] + q[c];
            float* x = cc.v[c];
            cc.q[c] = q[c];
            x[0] = __ldg(p); x[1] = __ldg(p + 1); x[2] = __ldg(p + sy); x[3] = __ldg(p + sy + 1);
            p += sz;
            x[4] = __ldg(p); x[5] = __ldg(p + 1); x[6] = __ldg(p + sy); x[7] = __ldg(p + sy + 1);
        }
        const float s0 = __ldg(rdzC + m.dz_off + kF - 1), s1 = __ldg(rdzC + m.dz_off + kF);
#pragma unroll
        for (int e = 0; e < 8; ++e) cc.v[2][e] *= e < 4 ? s0 : s1;
    }
    auto lerp = [](float t, float x, float y) { return fmaf(t, y - x, x); };
    float r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float tx = wx[c == 0], ty = wy[c == 1], tz = wz[c == 2];
        const float* x = cc.v[c];
        r[c] = lerp(tz, lerp(ty, lerp(tx, x[0], x[1]), lerp(tx, x[2], x[3])), lerp(ty, lerp(tx, x[4], x[5]), lerp(tx, x[6], x[7])));
    }
    u = r[0] * m.rdx; v = r[1] * m.rdy; w = r[2];
}

// the draws of the FP64 form (same keys, same numbers; lattice values are exact in float)
__device__ __forceinline__ void draw3f(uint64_t seed, uint32_t iter, uint32_t sp, uint32_t purpose,
                                       uint32_t slot, float& r0, float& r1, float& r2) {
    uint32_t ctr[4] = { slot, iter, (sp & 0xFFFFu) | (purpose << 16), 0x706c6b74u };
    uint32_t key[2] = { (uint32_t)seed, (uint32_t)(seed >> 32) };
    uint32_t o[4];
    pi_philox4x32_10(ctr, key, o);
    r0 = (float)(o[0] >> 8) * 0x1p-24f;
    r1 = (float)(o[1] >> 8) * 0x1p-24f;
    r2 = (float)(o[2] >> 8) * 0x1p-24f;
}

__device__ __forceinline__ unsigned long long to_fixed(float v, double inv_unit) {
    return (unsigned long long)__double2ll_rn((double)v * inv_unit);
}
__device__ __forceinline__ void add_fixed(unsigned long long* a, float v, double inv_unit) {
    const unsigned long long x = to_fixed(v, inv_unit);
    if (x) atomicAdd(a, x);
}

// Warp-segmented sums for the particle → grid scatters. In the cell-sorted storage order the
// individuals of one cell sit in adjacent slots, so the lanes of a warp form runs of equal cell
// keys; each run's first lane adds the run's total with one integer atomic instead of one atomic
// per individual. A warp whose runs are short (more than 16 runs in 32 lanes) adds per lane: the
// shuffles of the segmented sums would cost more than the atomics they save. Sums are integers
// (counts, fixed-point masses), so the result is the same either way. All 32 lanes call these
// with converged control flow; a key of -1 takes no part.
struct WarpRuns {
    bool head;      // this lane adds: the first lane of its run, or every lane when not aggregating
    bool agg;       // the warp adds per run (warp-uniform)
    int end;        // last lane of this lane's run
};
__device__ __forceinline__ WarpRuns warp_runs(long long key) {
    const int lane = threadIdx.x & 31;
    const long long prev = __shfl_up_sync(0xffffffffu, key, 1);
    WarpRuns R;
    const bool head = lane == 0 || prev != key;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const unsigned after = lane == 31 ? 0u : heads & ~((2u << lane) - 1u);
    R.end = after ? __ffs(after) - 2 : 31;
    R.agg = __popc(heads) <= 16;
    R.head = R.agg ? head : true;
    return R;
}
// the total of v over the lanes from this lane to the end of its run (the run's total at its head)
template <typename T>
__device__ __forceinline__ T run_sum(T v, const WarpRuns& R) {
    if (!R.agg) return v;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_down_sync(0xffffffffu, v, o);
        if (lane + o <= R.end) v += y;
    }
    return v;
}

// ------------------------------------------------------------------------------------------
// step prologue: forcing of the step, vel½
// ------------------------------------------------------------------------------------------

__device__ __forceinline__ long long snap_index(double tm, double tc, int use_call, double dT_s, long long n,
                                                uint32_t* err, bool flag) {
    long long t = (long long)floor((use_call ? tc : tm) / dT_s);
    if (t < 0 || t >= n) { if (flag) seterr(err, F32_ERR_FORCING); t = t < 0 ? 0 : n - 1; }
    return t;
}

// The step's prologue in one launch (grid: x blocks, members), each block its share of a member:
//  - update!'s forcing selection (Simulation/update.jl:14-26) for members with device-resident
//    series, from model.t before the step (or the step index of the call with time_offset). Every
//    block works it out from the tables; the first thread of block x = 0 writes it down, and only
//    the entries that no other block reads here;
//  - the surface PAR snapshot;
//  - vel½ = (vel₀ + vel₁) * 0.5 (time_step.jl:17-19) when the two are different fields;
//  - zeros in the per-cell counts (a memset and two kernels were three launches: 12 µs of a small
//    model's step).
struct BeginArgs {
    const MemberDev* md;
    const MemberSeries* S;
    MemberForcing* F;
    StepState* st;
    double dT;
    float* PARF;
    int* pop;
    int* pop_sp;               // nsp × Gtot or null
    uint32_t *segdiv, *segfree;
    int nsp;
    long long Gtot;
    uint32_t* err;
};
__global__ void k32_begin(BeginArgs a) {
    const int mi = blockIdx.y;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const bool live = !stopped(a.err);
    if (lead && mi == 0) a.st->live = live;
    if (!live) return;
    if (blockIdx.x == 0)
        for (int q = mi * a.nsp + threadIdx.x; q < (mi + 1) * a.nsp; q += blockDim.x) {
            a.segfree[q] -= a.segdiv[q];        // the slots taken in the step before
            a.segdiv[q] = 0u;
        }
    const MemberSeries& s = a.S[mi];
    const MemberDev& M = a.md[mi];
    const MemberForcing& F = a.F[mi];
    const double tm = a.st->t, tc = (double)a.st->call_step * a.dT;
    const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, nt = (long long)gridDim.x * blockDim.x;
    const float *v0[3], *v1[3], *temp = nullptr;
    for (int c = 0; c < 3; ++c) v0[c] = F.vel0[c];
    if (s.has_series && s.has_vel) {
        const long long tv = snap_index(tm, tc, s.time_offset & 1, s.dT_vel, s.nvel, a.err, lead);
        for (int c = 0; c < 3; ++c) v1[c] = s.vel + (tv * 3 + c) * M.G;
    } else {
        for (int c = 0; c < 3; ++c) v1[c] = F.vel1[c];
    }
    if (s.has_series) temp = s.temp + snap_index(tm, tc, s.time_offset & 4, s.dT_temp, s.ntemp, a.err, lead) * M.G;
    if (lead) {
        MemberForcing& W = a.F[mi];
        if (s.has_series && s.has_vel) for (int c = 0; c < 3; ++c) W.vel1[c] = v1[c];
        if (s.has_series) W.temp = temp;
        for (int c = 0; c < 3; ++c) W.velh[c] = v0[c] == v1[c] ? v1[c] : s.velh_buf[c];
    }
    // members start on multiples of 64 cells, so the counts are cleared 16 bytes at a time
    const long long n4 = (M.G + 3) >> 2;
    for (int p = -1; p < (a.pop_sp ? a.nsp : 0); ++p) {
        int4* z = reinterpret_cast<int4*>((p < 0 ? a.pop : a.pop_sp + p * a.Gtot) + M.cell_off);
        for (long long q = t0; q < n4; q += nt) z[q] = make_int4(0, 0, 0, 0);
    }
    if (v0[0] != v1[0]) {
        float *h0 = s.velh_buf[0], *h1 = s.velh_buf[1], *h2 = s.velh_buf[2];
        for (long long q = t0; q < M.G; q += nt) {
            h0[q] = (v0[0][q] + v1[0][q]) * 0.5f;
            h1[q] = (v0[1][q] + v1[1][q]) * 0.5f;
            h2[q] = (v0[2][q] + v1[2][q]) * 0.5f;
        }
    }
    if (!s.has_series) return;
    const long long tp = snap_index(tm, tc, s.time_offset & 2, s.dT_PAR, s.npar, a.err, lead);
    const long long n = (long long)M.Nx * M.Ny;
    const float* src = s.parf + tp * n;
    for (long long q = t0; q < n; q += nt) a.PARF[M.col_off + q] = src[q];
}

// ------------------------------------------------------------------------------------------
// (a)+(e) particles: RK4 + diffusion + find_inds!, pop and Chl into the per-cell sums, then the
// grazing/mortality decisions of the previous step (inactivate!, calc_loss!, diagnostics) and the
// division/free counts of each tile of slots for the compaction.
// ------------------------------------------------------------------------------------------
struct MoveArgs {
    Tab32 T;
    IndDev32 P;
    const SpeciesDev32* sp;        // [member * nsp + species]
    const BgcDev32* bgc;           // [member]
    const MemberForcing* F;
    const float* rdzC;             // 1 / ΔzC
    const StepState* st;
    float dT;
    long long Gtot;
    int* pop;                      // Gtot: all species
    int* pop_sp;                   // nsp × Gtot when grazing is not shared, else null
    unsigned long long* chl_acc;   // Gtot
    unsigned long long* acc;       // ACC_N × Gtot
    uint32_t* dcnt;                // nsp × 4 × Gtot: num, graz, mort, dvid
    uint32_t* err;
    int sub;                       // work units per tile (see unit_tile)
};

// A work unit of the particle kernels is 1/sub of a tile: F32_TILE / sub consecutive slots. With
// sub = 1 a thread walks F32_TILE / blockDim.x slots and loads the next while it works on the
// current one, which is best when the tiles fill the chip. A model of few tiles leaves most SMs
// idle that way (1024 individuals are one tile, that is one block walking 8 slots deep: 34 µs of
// k32_physiology); there sub = F32_TILE / blockDim.x gives every slot its own thread.
__device__ __forceinline__ int unit_tile(int u, int sub, int& first) {
    const int t = sub == 1 ? u : u / sub;
    first = (u - t * sub) * (F32_TILE / sub);
    return t;
}

// bit of logical slot L of species s of member m in a logical-slot bitmap
__device__ __forceinline__ void slot_bit(const MemberDev& m, int s, int L, long long& w, uint32_t& bit) {
    w = m.woff + (long long)s * m.wps + (L >> 5);
    bit = 1u << (L & 31);
}

// The slot state k32_move reads first, loaded one slot ahead of its use (the offsets and Chl of an
// inactive slot are read and unused).
struct MState { int32_t code; float ox, oy, oz, chl; uint8_t fl, stt; };
__device__ __forceinline__ MState move_state(const IndDev32& P, long long g, bool valid) {
    MState S{-1, 0.0f, 0.0f, 0.0f, 0.0f, 0, 0};
    if (valid) {
        S.fl = P.flags[g]; S.stt = P.stat[g]; S.code = P.cell[g];
        S.ox = P.ox[g]; S.oy = P.oy[g]; S.oz = P.oz[g]; S.chl = P.Chl[g];
    }
    return S;
}

// What k32_move adds to the grid for one slot: the cell (-1: nothing), a packed count
// (pop | grazed << 8 | dead << 16 | dividing << 24; a warp's run sums stay below 256 per field) and
// the Chl sum in fixed point (interior cells only).
struct MoveOut { long long cq; uint32_t cnt; unsigned long long chl; };

__device__ __forceinline__ MoveOut move_one(const MoveArgs& a, const MemberDev& m, const PGeom& pg, int mi, int s,
                                            long long g, uint32_t iter, const MState& S) {
    const IndDev32& P = a.P;
    MoveOut out{-1, 0u, 0ull};
    const uint8_t fl = S.fl, stt = S.stt;
    const int32_t code = S.code;
    const float ox = S.ox, oy = S.oy, oz = S.oz;
    const float chl = S.chl;
    if (!(fl & F32_AC)) {
        // every stage multiplies by ac: the position becomes (0, 0, 0) and the cell (Hx, Hy, Hz)
        if (code != -1) {
            P.cell[g] = -1;
            P.ox[g] = 0.0f; P.oy[g] = 0.0f; P.oz[g] = 0.0f;
        }
        if (stt) P.stat[g] = 0;
        return out;
    }
    uint32_t* err = a.err;
    int ci, cj, ck;
    unpack_int(m, code, ci, cj, ck);
    // ΔzC at the find_inds! zi of the previous step, plus Hz (particle_diffusion.jl:26-28)
    int zi = ck + 1 + pg.Hz;
    if (stt & F32_ST_STALE) { int a0, a1; unpack_halo(m, P.scell[g], a0, a1, zi); }
    bool bad = false;
    const int kdz = clampb(zi + pg.Hz, 1, pg.Gz, bad);
    const MemberForcing& f = a.F[mi];
    const Ax1 X0{ci, ox}, Y0{cj, oy}, Z0{ck, oz};
    const float dT = a.dT, hdT = 0.5f * dT;
    const float* __restrict__ rdzC = a.rdzC;
    // RK4: stages at X0, X0 + k1·ΔT/2, X0 + k2·ΔT/2, X0 + k3·ΔT, weights 1, 2, 2, 1
    Corners cc;
    cc.fid = -1;
    Ax1 X = X0, Y = Y0, Z = Z0;
    float u2 = 0.0f, v2 = 0.0f, w2 = 0.0f;
#pragma unroll
    for (int st = 0; st < 4; ++st) {
        float u, v, w;
        itpl32(pg, st == 0 ? f.vel0 : st == 3 ? f.vel1 : f.velh, st == 0 ? 0 : st == 3 ? pg.f1 : pg.fh, rdzC, X, Y, Z, cc, u, v, w);
        const float wt = st == 0 || st == 3 ? 1.0f : 2.0f, h = st == 2 ? dT : hdT;
        u2 += u * wt; v2 += v * wt; w2 += w * wt;
        X = X0; Y = Y0; Z = Z0;
        if (st == 3) break;
        move_stage(X, u * h, pg.Nx, pg.tx, bad); move_stage(Y, v * h, pg.Ny, pg.ty, bad); move_stage(Z, -(w * h), pg.Nz, pg.tz, bad);
    }
    const float sixth = 1.0f / 6.0f;
    u2 *= sixth; v2 *= sixth; w2 *= sixth;
    move(X, u2 * dT, pg.Nx, pg.tx); move(Y, v2 * dT, pg.Ny, pg.ty); move(Z, -(w2 * dT), pg.Nz, pg.tz);
    // random-walk diffusion (particle_diffusion.jl:16-33); a zero κ moves nothing
    const BgcDev32& b = a.bgc[mi];
    if (b.kappa_hP != 0.0f || b.kappa_vP != 0.0f) {
        float r0, r1, r2;
        draw3f(m.seed, iter, (uint32_t)s, PI_DRAW_DIFFUSION, (uint32_t)P.lslot[g], r0, r1, r2);
        move(X, (r0 - 0.5f) * 2.0f * sqrtf(b.kappa_hP * dT) * pg.rdx, pg.Nx, pg.tx);
        move(Y, (r1 - 0.5f) * 2.0f * sqrtf(b.kappa_hP * dT) * pg.rdy, pg.Ny, pg.ty);
        move(Z, (r2 - 0.5f) * 2.0f * sqrtf(b.kappa_vP * dT) * __ldg(rdzC + pg.dz_off + kdz - 1), pg.Nz, pg.tz);
    }
    if (X.c < 0 || X.c > pg.Nx) { bad = true; X.c = X.c < 0 ? 0 : pg.Nx; X.o = 0.0f; }
    if (Y.c < 0 || Y.c > pg.Ny) { bad = true; Y.c = Y.c < 0 ? 0 : pg.Ny; Y.o = 0.0f; }
    if (Z.c < 0 || Z.c > pg.Nz) { bad = true; Z.c = Z.c < 0 ? 0 : pg.Nz; Z.o = 0.0f; }
    if (bad) seterr(err, F32_ERR_DOMAIN);
    // everything that reads the member record is formed before the stores below
    const int32_t code_new = pack_int(m, X.c, Y.c, Z.c);
    const long long cq = m.cell_off + q_of(m, X.c, Y.c, Z.c);
    const bool inside = X.c < pg.Nx && Y.c < pg.Ny && Z.c < pg.Nz;
    const double chl_inv = m.chl_inv, fx_inv = m.fx_inv;
    P.ox[g] = X.o; P.oy[g] = Y.o; P.oz[g] = Z.o;
    P.cell[g] = code_new;
    const long long G = a.Gtot;
    // previous step's decisions (plankton_update.jl:5-16, division_death.jl:2-25)
    const int gz = (fl & F32_GRAZ) != 0, mt = (fl & F32_MORT) != 0, dv = (fl & F32_DVID) != 0;
    const int ac1 = !gz, ac2 = ac1 && !mt, dv2 = dv && ac2;
    // pop, the Chl sum and the graz/mort/dvid diagnostics counts, added by scatter_move
    out.cq = cq;
    out.cnt = 1u | (gz ? 1u << 8 : 0u) | (ac1 && mt ? 1u << 16 : 0u) | (dv2 ? 1u << 24 : 0u);
    out.chl = inside ? to_fixed(chl, chl_inv) : 0ull;
    const int kind = gz ? 1 : (ac1 && mt) ? 2 : 0;
    if (kind && inside) {
        const SpeciesDev32& p = a.sp[mi * a.T.nsp + s];
        const float fC = kind == 1 ? p.grazFracC : p.mortFracC;
        const float fN = kind == 1 ? p.grazFracN : p.mortFracN;
        const float fP = kind == 1 ? p.grazFracP : p.mortFracP;
        const float Bm = P.Bm[g], Cq = P.Cq[g], Nq = P.Nq[g], Pq = P.Pq[g];
        const double u = fx_inv;
        add_fixed(&a.acc[ACC_DOC * G + cq], (Bm + Cq) * fC, u);
        add_fixed(&a.acc[ACC_DON * G + cq], (Bm * p.R_NC + Nq) * fN, u);
        add_fixed(&a.acc[ACC_DOP * G + cq], (Bm * p.R_PC + Pq) * fP, u);
        add_fixed(&a.acc[ACC_POC * G + cq], (Bm + Cq) * (1.0f - fC), u);
        add_fixed(&a.acc[ACC_PON * G + cq], (Bm * p.R_NC + Nq) * (1.0f - fN), u);
        add_fixed(&a.acc[ACC_POP * G + cq], (Bm * p.R_PC + Pq) * (1.0f - fP), u);
    }
    P.flags[g] = (uint8_t)((ac2 ? F32_AC : 0) | (dv2 ? F32_DVID : 0));
    P.stat[g] = F32_ST_AC0;
    // division bookkeeping on logical slots: dividers of this step, slots freed by this step's
    // grazing and mortality (free slots stay marked until a daughter takes them)
    if (dv2 || !ac2) {
        long long w;
        uint32_t bit;
        slot_bit(m, s, P.lslot[g], w, bit);
        atomicOr(dv2 ? &P.dvbits[w] : &P.freebits[w], bit);
    }
    return out;
}

// k32_move's grid sums of one warp (segment s of one member): one atomic per run of a cell; and the
// segment's dividers and newly freed slots
__device__ __forceinline__ void scatter_move(const MoveArgs& a, int s, int seg, const MoveOut& o) {
    if (__all_sync(0xffffffffu, o.cq < 0)) return;      // a warp of inactive slots adds nothing
    const unsigned dv = __ballot_sync(0xffffffffu, o.cnt >> 24 != 0), fr = __ballot_sync(0xffffffffu, (o.cnt & 0xffff00u) != 0);
    if ((threadIdx.x & 31) == 0) {
        if (dv) atomicAdd(&a.P.segdiv[seg], __popc(dv));
        if (fr) atomicAdd(&a.P.segfree[seg], __popc(fr));
    }
    const WarpRuns R = warp_runs(o.cq);
    const uint32_t c = run_sum(o.cnt, R);
    const unsigned long long chl = run_sum(o.chl, R);
    if (R.head && o.cq >= 0) {
        const long long G = a.Gtot, cq = o.cq;
        const int np = (int)(c & 0xffu);
        atomicAdd(&a.pop[cq], np);
        if (a.pop_sp) atomicAdd(&a.pop_sp[(long long)s * G + cq], np);
        if (chl) atomicAdd(&a.chl_acc[cq], chl);
        uint32_t* dc = a.dcnt + (long long)s * 4 * G + cq;
        if (c >> 8 & 0xffu) atomicAdd(dc + 1 * G, c >> 8 & 0xffu);
        if (c >> 16 & 0xffu) atomicAdd(dc + 2 * G, c >> 16 & 0xffu);
        if (c >> 24) atomicAdd(dc + 3 * G, c >> 24);
    }
}

// MINB: blocks per SM the registers are fitted for, of 256 threads (2: 128 registers, 3: 80, 4: 64) or, as
// 5, of 128 (96 registers). The stages' loads wait for L2, so what bounds the kernel is how many warps wait
// beside them: on 256×256×64 with 4 M individuals 318 µs with 16 warps per SM, 262 with 20 at 96 registers,
// 295 with 24 at 80 (which spill). The autotuner picks the variant.
template <int MINB>
__global__ void __launch_bounds__(MINB == 5 ? 128 : 256, MINB) k32_move(MoveArgs a) {
    if (stopped(a.err)) return;
    __shared__ PGeom sg;
    const int bs = blockDim.x, ppt = F32_TILE / (bs * a.sub);
    const uint32_t iter = (uint32_t)(a.st->iteration + 1);
    for (int u = blockIdx.x; u < a.T.ntiles * a.sub; u += gridDim.x) {
        int first;
        const int2 tl = a.T.tiles[unit_tile(u, a.sub, first)];
        int mi, s;
        seg_of(a.T, tl.x, mi, s);
        const MemberDev& m = a.T.md[mi];
        if (threadIdx.x == 0) sg = pgeom(m, a.F[mi]);
        __syncthreads();
        const long long base = m.slot_off + (long long)s * m.C;
        long long slot = (long long)tl.y + first + threadIdx.x;
        MState nx = move_state(a.P, base + slot, slot < m.C);
        for (int p = 0; p < ppt; ++p, slot += bs) {
            const MState cur = nx;
            if (p + 1 < ppt) nx = move_state(a.P, base + slot + bs, slot + bs < m.C);
            MoveOut o{-1, 0u, 0ull};
            if (slot < m.C) o = move_one(a, m, sg, mi, s, base + slot, iter, cur);
            scatter_move(a, s, tl.x, o);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------
// PAR down each column (calc_par!, Individuals/utils.jl:55-63); consumes the Chl sums
// ------------------------------------------------------------------------------------------
//
// For every interior cell holding individuals it also packs the environment physiology gathers
// (find_NPT!, utils.jl:14-25: NH4, NO3, PO4, DOC, par, temperature, pop) into one 32-byte record,
// so an individual reads one sector instead of seven.
//
// One thread walking a column waits for memory level by level, and 32 columns are one warp (ncu on
// 128×128×64: 5 % of the warps resident, 34 µs at 9 % of DRAM). So 1, 2, 4 or 8 warps take the same 32
// columns: each forms the attenuation of PAR_CH levels, the first carries the light down through
// shared memory (one product per level), and all write their levels. Two blocks per SM, so that no register of
// the loads in flight spills: three, which spilled, took 58 µs on 256×256×64 and 23 on 128×128×64, two 53
// and 21 (one thread per column there 48 and 37, and 75 and 62 once the individuals had spread over more levels,
// where two blocks take 60 and 23).
#define PAR_CH 8
#define PAR_WARPS 8
#define PAR_BLOCKS 2
struct ParArgs {
    Tab32 T;
    const float* dzF;
    const BgcDev32* bgc;
    unsigned long long* chl_acc;
    float* PARF;
    float* par;
    float* diag_par;
    const float* tr;
    long long Gtot;
    const MemberForcing* F;
    const int* pop;
    float4* env;
    const StepState* st;
    int lw;                    // warps per 32 columns: 1, 2, 4 or 8
    int maxNz;
};
// the 32-column items of one block of PAR_WARPS warps
__device__ __forceinline__ void par_columns(const ParArgs& a, int block) {
    __shared__ float sEx[PAR_WARPS * PAR_CH][32], sIn[PAR_WARPS * PAR_CH][32];
    if (!a.st->live) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, lw = a.lw;
    const int part = wid & (lw - 1), row0 = wid * PAR_CH;           // rows of this warp in shared memory
    const int w = block * (PAR_WARPS / lw) + wid / lw;
    const bool has = w < a.T.nicol;
    const int4 it = a.T.icol[has ? w : 0];
    const MemberDev& m = a.T.md[it.x];
    const int Nz = m.Nz, Hz = m.Hz;
    const int i = it.y + lane, j = it.z;                            // 1-based interior column
    const bool col = has && i <= m.Nx;
    const float kc = a.bgc[it.x].kc, kw = a.bgc[it.x].kw;
    const long long fcol = m.col_off + (i - 1) + (long long)m.Nx * (j - 1);
    const int q1 = gid3(m, i + m.Hx, j + m.Hy, 1 + Hz), slab = m.Gx * m.Gy;
    const long long off = m.cell_off;
    const double chl_unit = m.chl_unit;
    const float areaf = m.dx * m.dy;
    const float* dzp = a.dzF + m.dz_off + Hz;
    const float* temp = a.F[it.x].temp;
    const int* pop = a.pop + off;
    const float* tr = a.tr + off;
    unsigned long long* chl_acc = a.chl_acc + off;
    float *par = a.par + off, *diag = a.diag_par + off;
    float4* env = a.env + 2 * off;
    float parf = col && part == 0 ? a.PARF[fcol] : 0.0f;
    for (int kc0 = 0; kc0 < a.maxNz; kc0 += PAR_CH * lw) {          // same trip count for every warp
        const int k0 = kc0 + part * PAR_CH;                         // 0-based levels k0 .. k0 + PAR_CH - 1
        float ex[PAR_CH], at[PAR_CH], dg[PAR_CH];
        int pp[PAR_CH];
        if (col) {
            long long v[PAR_CH];
#pragma unroll
            for (int e = 0; e < PAR_CH; ++e) {
                const bool in = k0 + e < Nz;
                const int q = q1 + (k0 + e) * slab;
                v[e] = in ? (long long)chl_acc[q] : 0;
                pp[e] = in ? __ldg(pop + q) : 0;
                dg[e] = in ? diag[q] : 0.0f;
            }
#pragma unroll
            for (int e = 0; e < PAR_CH; ++e) {
                if (k0 + e >= Nz) continue;
                if (v[e]) chl_acc[q1 + (k0 + e) * slab] = 0ull;
                const float dz = __ldg(dzp + k0 + e);
                const float chl = (float)((double)v[e] * chl_unit);
                at[e] = (chl / (areaf * dz) * kc + kw) * dz;
                ex[e] = expf(-at[e]);
                sEx[row0 + e][lane] = ex[e];
            }
        }
        __syncthreads();
        if (part == 0 && col) {
            const int n = min(PAR_CH * lw, Nz - kc0);
            for (int e = 0; e < n; ++e) {
                sIn[row0 + e][lane] = parf;
                parf = parf * sEx[row0 + e][lane];
            }
        }
        __syncthreads();
        if (col) {
            // four levels' loads of the environment of occupied cells at a time
#pragma unroll
            for (int g = 0; g < PAR_CH; g += 4) {
                float4 nv[4];
                float tv[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int q = q1 + (k0 + g + e) * slab;
                    if (pp[g + e] > 0) {
                        nv[e] = make_float4(__ldg(tr + PI_NH4 * a.Gtot + q), __ldg(tr + PI_NO3 * a.Gtot + q),
                                            __ldg(tr + PI_PO4 * a.Gtot + q), __ldg(tr + PI_DOC * a.Gtot + q));
                        tv[e] = __ldg(temp + q);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (k0 + g + e >= Nz) continue;
                    const int q = q1 + (k0 + g + e) * slab;
                    const float pv = sIn[row0 + g + e][lane] * (1.0f - ex[g + e]) / at[g + e];
                    par[q] = pv;
                    diag[q] = dg[g + e] + pv;
                    if (pp[g + e] > 0) {
                        env[2 * q] = nv[e];
                        env[2 * q + 1] = make_float4(pv, tv[e], (float)pp[g + e], 0.0f);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (col && part == 0) a.PARF[fcol] = parf;
}

__global__ void __launch_bounds__(32 * PAR_WARPS, PAR_BLOCKS) k32_par(ParArgs a) { par_columns(a, blockIdx.x); }

// ------------------------------------------------------------------------------------------
// (e) division: k-th divider (logical slot order) → k-th free logical slot (findall(!ac),
// ascending), per segment (get_tind!, Individuals/utils.jl:76-86), with the capacity check
// (plankton_update.jl:18-22). Dividers and free slots are bits of two bitmaps over logical slots;
// a tile of F32_TILE logical slots is 32 words, one per lane of a warp.
// ------------------------------------------------------------------------------------------

// (dividers << 32) | free slots of every tile, from the bitmaps. One warp per tile.
__global__ void k32_count_tiles(Tab32 T, IndDev32 P, unsigned long long* __restrict__ tile_cnt, const uint32_t* err) {
    if (stopped(err)) return;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < T.ntiles; t += nw) {
        const int2 tl = T.tiles[t];
        int mi, s;
        seg_of(T, tl.x, mi, s);
        const MemberDev& m = T.md[mi];
        const long long w = m.woff + (long long)s * m.wps + (tl.y >> 5) + lane;
        const unsigned nd = __reduce_add_sync(0xffffffffu, (unsigned)__popc(P.dvbits[w]));
        const unsigned nf = __reduce_add_sync(0xffffffffu, (unsigned)__popc(P.freebits[w]));
        if (lane == 0) tile_cnt[t] = ((unsigned long long)nd << 32) | nf;
    }
}

// ---- exclusive prefix sums of 64-bit counts (block-wide, 1024 threads) ----------------------
// inclusive scan over the lanes of a warp
__device__ __forceinline__ unsigned long long warp_inscan64(unsigned long long x) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}
// Exclusive scan of v over the block (blockDim.x == 1024); returns the thread's prefix and the
// block total in *total. sh holds 33 values.
__device__ __forceinline__ unsigned long long block_exscan64(unsigned long long v, unsigned long long* sh,
                                                             unsigned long long* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned long long inc = warp_inscan64(v);
    if (lane == 31) sh[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        const unsigned long long w = sh[lane];
        const unsigned long long wi = warp_inscan64(w);
        sh[lane] = wi - w;
        if (lane == 31) sh[32] = wi;
    }
    __syncthreads();
    const unsigned long long out = sh[wid] + inc - v;
    *total = sh[32];
    __syncthreads();
    return out;
}

// Exclusive scan of the tile counts within each (member, species) segment: one block of 1024
// threads per segment.
__global__ void __launch_bounds__(1024) k32_scan_tiles(Tab32 T, const unsigned long long* __restrict__ tile_cnt,
                                                       unsigned long long* __restrict__ tile_off, int nseg,
                                                       const uint32_t* err) {
    if (stopped(err)) return;
    __shared__ unsigned long long sh[33];
    for (int seg = blockIdx.x; seg < nseg; seg += gridDim.x) {
        const int t0 = T.seg_tile0[seg], t1 = T.seg_tile0[seg + 1];
        unsigned long long run = 0;
        for (int base = t0; base < t1; base += 1024) {
            const int t = base + threadIdx.x;
            const unsigned long long v = t < t1 ? tile_cnt[t] : 0ull;
            unsigned long long tot;
            const unsigned long long ex = block_exscan64(v, sh, &tot);
            if (t < t1) tile_off[t] = run + ex;
            run += tot;
        }
    }
}

// Exclusive scan of n 64-bit values in three passes (chunks of 1024 × PER values): chunk sums,
// a scan of the chunk sums in one block, then each chunk's scan from its offset.
#define SCAN_PER 8
__global__ void __launch_bounds__(1024) k32_scan_sums(const unsigned long long* __restrict__ in, long long n,
                                                      unsigned long long* __restrict__ sums) {
    __shared__ unsigned long long sh[33];
    const long long base = (long long)blockIdx.x * 1024 * SCAN_PER;
    unsigned long long v = 0;
    for (int e = 0; e < SCAN_PER; ++e) {
        const long long q = base + (long long)e * 1024 + threadIdx.x;
        if (q < n) v += in[q];
    }
    unsigned long long tot;
    block_exscan64(v, sh, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}
__global__ void __launch_bounds__(1024) k32_scan_chunks(unsigned long long* __restrict__ sums, long long nchunks) {
    __shared__ unsigned long long sh[33];
    unsigned long long run = 0;
    for (long long b = 0; b < nchunks; b += 1024) {
        const long long q = b + threadIdx.x;
        const unsigned long long v = q < nchunks ? sums[q] : 0ull;
        unsigned long long tot;
        const unsigned long long ex = block_exscan64(v, sh, &tot);
        if (q < nchunks) sums[q] = run + ex;
        run += tot;
    }
}
__global__ void __launch_bounds__(1024) k32_scan_apply(const unsigned long long* __restrict__ in, long long n,
                                                       const unsigned long long* __restrict__ sums,
                                                       unsigned long long* __restrict__ out) {
    __shared__ unsigned long long sh[33];
    const long long base = (long long)blockIdx.x * 1024 * SCAN_PER;
    // each thread takes PER consecutive values so that the chunk is scanned in order
    const long long q0 = base + (long long)threadIdx.x * SCAN_PER;
    unsigned long long loc[SCAN_PER], v = 0;
#pragma unroll
    for (int e = 0; e < SCAN_PER; ++e) { loc[e] = q0 + e < n ? in[q0 + e] : 0ull; v += loc[e]; }
    unsigned long long tot;
    unsigned long long run = sums[blockIdx.x] + block_exscan64(v, sh, &tot);
#pragma unroll
    for (int e = 0; e < SCAN_PER; ++e) {
        if (q0 + e < n) out[q0 + e] = run;
        run += loc[e];
    }
}

// exclusive prefix sum over the lanes of a warp
__device__ __forceinline__ unsigned warp_exscan(unsigned v) {
    const int lane = threadIdx.x & 31;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x - v;
}

// Lists of the dividers and of the free slots they take, in logical order. One warp per tile;
// tiles with neither dividers nor needed free slots do nothing. The divider bits are cleared once
// listed.
__global__ void k32_assign(Tab32 T, IndDev32 P, const unsigned long long* __restrict__ tile_cnt,
                           const unsigned long long* __restrict__ tile_off, int* __restrict__ divlist,
                           int* __restrict__ freelist, uint32_t* __restrict__ ndiv, StepState* st,
                           uint32_t* err) {
    if (stopped(err)) return;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < T.ntiles; t += nw) {
        const int2 tl = T.tiles[t];
        const int seg = tl.x;
        int mi, s;
        seg_of(T, seg, mi, s);
        const MemberDev& m = T.md[mi];
        const long long base = m.slot_off + (long long)s * m.C;
        const int t0 = T.seg_tile0[seg], t1 = T.seg_tile0[seg + 1];
        const unsigned long long b0 = tile_off[t0];
        const unsigned long long tot = tile_off[t1 - 1] + tile_cnt[t1 - 1] - b0;
        const unsigned int tdiv = (unsigned int)(tot >> 32), tfree = (unsigned int)(tot & 0xffffffffull);
        if (tdiv > tfree) {
            if (t == t0 && lane == 0) {
                ndiv[seg] = 0;
                if (!(atomicOr(err, F32_ERR_CAPACITY) & F32_ERR_CAPACITY)) {
                    st->err_iter = st->iteration + 1;
                    st->err_member = mi;
                }
            }
            continue;
        }
        if (t == t0 && lane == 0) ndiv[seg] = tdiv;
        const unsigned long long before = tile_off[t] - b0;
        const unsigned int dbefore = (unsigned int)(before >> 32), fbefore = (unsigned int)(before & 0xffffffffull);
        const unsigned long long c = tile_cnt[t];
        const bool wd = (c >> 32) != 0, wf = (c & 0xffffffffull) != 0 && fbefore < tdiv;
        if (!wd && !wf) continue;                                   // uniform over the warp
        const long long w = m.woff + (long long)s * m.wps + (tl.y >> 5) + lane;
        uint32_t dw = wd ? P.dvbits[w] : 0u, fw = wf ? P.freebits[w] : 0u;
        unsigned rd = dbefore + warp_exscan((unsigned)__popc(dw));
        unsigned rf = fbefore + warp_exscan((unsigned)__popc(fw));
        const int L0 = tl.y + lane * 32;
        while (dw) {
            const int bpos = __ffs(dw) - 1;
            dw &= dw - 1u;
            divlist[base + rd++] = L0 + bpos;
        }
        while (fw && rf < tdiv) {
            const int bpos = __ffs(fw) - 1;
            fw &= fw - 1u;
            freelist[base + rf++] = L0 + bpos;
        }
        if (wd) P.dvbits[w] = 0u;
    }
}

// copy_daughter_individuals! and divide_to_half! (division_death.jl:28-63) of one divider and its
// daughter's slot (logical slots of segment base; phys gives where each is stored).
__device__ __forceinline__ void daughter_one(const IndDev32& P, const MemberDev& m, int s, long long base, int pl, int dl,
                                             uint32_t* err) {
    if (pl < 0 || pl >= m.C || dl < 0 || dl >= m.C) { seterr(err, F32_ERR_LISTS); return; }
    const int pp = P.phys[base + pl], dp = P.phys[base + dl];
    if (pp < 0 || pp >= m.C || dp < 0 || dp >= m.C) { seterr(err, F32_ERR_LISTS); return; }
    const long long p = base + pp, d = base + dp;
    // all reads first: the mother's and the daughter's slots are different
    const int32_t cd = P.cell[d], cp = P.cell[p];
    const float ox = P.ox[p], oy = P.oy[p], oz = P.oz[p];
    const float Bm = P.Bm[p] * 0.5f, Cq = P.Cq[p] * 0.5f, Nq = P.Nq[p] * 0.5f, Pq = P.Pq[p] * 0.5f;
    const float Chl = P.Chl[p] * 0.5f, gen = P.gen[p] + 1.0f;
    const float aged = P.age[d] * 0.0f, agep = P.age[p] * 0.0f;
    const uint8_t std_ = P.stat[d];
    // the daughter's slot keeps the cell find_inds! gave it this step
    int32_t sc;
    if (cd < 0) sc = pack_halo(m, m.Hx, m.Hy, m.Hz);
    else { int a0, a1, a2; unpack_int(m, cd, a0, a1, a2); sc = pack_halo(m, a0 + 1 + m.Hx, a1 + 1 + m.Hy, a2 + 1 + m.Hz); }
    P.scell[d] = sc;
    P.cell[d] = cp;
    P.ox[d] = ox; P.oy[d] = oy; P.oz[d] = oz;
    P.Bm[d] = Bm; P.Cq[d] = Cq; P.Nq[d] = Nq; P.Pq[d] = Pq; P.Chl[d] = Chl; P.gen[d] = gen;
    P.age[d] = aged;
    P.Bm[p] = Bm; P.Cq[p] = Cq; P.Nq[p] = Nq; P.Pq[p] = Pq; P.Chl[p] = Chl; P.gen[p] = gen;
    P.age[p] = agep;
    P.flags[d] = F32_AC | F32_DVID;
    P.stat[d] = (uint8_t)((std_ & F32_ST_AC0) | F32_ST_STALE);
    long long w;
    uint32_t bit;
    slot_bit(m, s, dl, w, bit);
    atomicAnd(&P.freebits[w], ~bit);
}

// Grid: (x, segments).
__global__ void k32_daughters(Tab32 T, IndDev32 P, const int* __restrict__ divlist,
                              const int* __restrict__ freelist, const uint32_t* __restrict__ ndiv,
                              uint32_t* err) {
    if (stopped(err)) return;
    const int seg = blockIdx.y;
    int mi, s;
    seg_of(T, seg, mi, s);
    const MemberDev& m = T.md[mi];
    const long long base = m.slot_off + (long long)s * m.C;
    const uint32_t n = ndiv[seg];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        if (k >= (uint32_t)m.C) { seterr(err, F32_ERR_LISTS); continue; }
        daughter_one(P, m, s, base, divlist[base + k], freelist[base + k], err);
    }
}

// Division of a whole segment by one block (DIV_WARPS warps): k32_count_tiles, k32_scan_tiles,
// k32_assign and k32_daughters in one, for segments of at most DIV_WORDS bitmap words. Each warp
// counts a run of words, the warps' counts are added up in shared memory, and each warp walks its
// run again to list its dividers and the free slots they take.
#define DIV_WARPS 8
#define DIV_WORDS 8192
struct DivArgs {
    Tab32 T;
    IndDev32 P;
    int* divlist;
    int* freelist;
    int nseg;
    StepState* st;
    uint32_t* err;
};
__device__ __forceinline__ void divide_segment(const DivArgs& a, int seg) {
    __shared__ uint32_t shd[DIV_WARPS], shf[DIV_WARPS];
    const IndDev32& P = a.P;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int mi, s;
    seg_of(a.T, seg, mi, s);
    const MemberDev& m = a.T.md[mi];
    const long long base = m.slot_off + (long long)s * m.C, wbase = m.woff + (long long)s * m.wps;
    const uint32_t tdiv = P.segdiv[seg];
    // the capacity check (plankton_update.jl:18-22): the step divides in every segment or in none,
    // so every block looks at all of them (k32_move's counts, which nothing changes here)
    bool over = false;
    for (int q = threadIdx.x; q < a.nseg; q += blockDim.x) over |= P.segdiv[q] > P.segfree[q];
    if (__syncthreads_or(over)) {
        if (threadIdx.x == 0 && tdiv > P.segfree[seg] && !(atomicOr(a.err, F32_ERR_CAPACITY) & F32_ERR_CAPACITY)) {
            a.st->err_iter = a.st->iteration + 1;
            a.st->err_member = mi;
        }
        return;
    }
    if (tdiv == 0) return;
    const int words = (int)m.wps, run = (words / 32 + DIV_WARPS - 1) / DIV_WARPS * 32;
    const int w0 = min(wid * run, words), w1 = min(w0 + run, words);
    unsigned nd = 0, nf = 0;
#pragma unroll 4
    for (int w = w0; w < w1; w += 32) {
        nd += (unsigned)__popc(P.dvbits[wbase + w + lane]);
        nf += (unsigned)__popc(P.freebits[wbase + w + lane]);
    }
    nd = __reduce_add_sync(0xffffffffu, nd);
    nf = __reduce_add_sync(0xffffffffu, nf);
    if (lane == 0) { shd[wid] = nd; shf[wid] = nf; }
    __syncthreads();
    unsigned cdiv = 0, cfree = 0, dbefore = 0, fbefore = 0;
#pragma unroll
    for (int q = 0; q < DIV_WARPS; ++q) {
        if (q < wid) { dbefore += shd[q]; fbefore += shf[q]; }
        cdiv += shd[q]; cfree += shf[q];
    }
    if (cdiv != tdiv || tdiv > cfree) {           // the bitmaps hold what k32_move counted
        if (threadIdx.x == 0) seterr(a.err, F32_ERR_LISTS);
        return;
    }
    for (int w = w0; w < w1 && (nd || fbefore < tdiv); w += 32) {
        uint32_t dw = nd ? P.dvbits[wbase + w + lane] : 0u, fw = fbefore < tdiv ? P.freebits[wbase + w + lane] : 0u;
        if (dw) P.dvbits[wbase + w + lane] = 0u;
        const unsigned cd = (unsigned)__popc(dw), cf = (unsigned)__popc(fw);
        unsigned rd = dbefore + warp_exscan(cd), rf = fbefore + warp_exscan(cf);
        dbefore += __reduce_add_sync(0xffffffffu, cd);
        fbefore += __reduce_add_sync(0xffffffffu, cf);
        const int L0 = (w + lane) * 32;
        while (dw) {
            a.divlist[base + rd++] = L0 + __ffs(dw) - 1;
            dw &= dw - 1u;
        }
        while (fw && rf < tdiv) {
            a.freelist[base + rf++] = L0 + __ffs(fw) - 1;
            fw &= fw - 1u;
        }
    }
    __syncthreads();
    for (unsigned k = threadIdx.x; k < tdiv; k += blockDim.x)
        daughter_one(P, m, s, base, a.divlist[base + k], a.freelist[base + k], a.err);
}

// Division and light depend on k32_move only and touch different arrays, so small models run both
// in one launch: blocks 0 .. nseg - 1 divide a segment each, the others take the columns. Both go by
// the step's `live` mark: a step that a dividing block stops still has its light.
__global__ void __launch_bounds__(32 * DIV_WARPS, PAR_BLOCKS) k32_par_divide(ParArgs pa, DivArgs da) {
    if ((int)blockIdx.x < da.nseg) {
        if (da.st->live) divide_segment(da, blockIdx.x);
    } else {
        par_columns(pa, blockIdx.x - da.nseg);
    }
}

// ------------------------------------------------------------------------------------------
// (b) QuotaMode physiology in Float32 (plankton_growth.jl:2-24, growth_kernels.jl:2-166,
//     division_death_probability.jl:7-107, find_NPT!, calc_consume!, diags num)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float shape_dec_f(float x, float xmax, float k, int pw) {
    const float fx = fmaxf(0.0f, fminf(1.0f, 1.0f - x / xmax));
    const float p = pw == 2 ? fx * fx : (fx * fx) * (fx * fx);
    return p / (k + p);
}
__device__ __forceinline__ float shape_inc_f(float x, float xmax, float k, int pw) {
    return 1.0f - shape_dec_f(x, xmax, k, pw);
}
__device__ __forceinline__ float tempFunc_f(float T, const SpeciesDev32& p) {
    const float k = fmaxf(0.0f, expf(-p.Ea / (8.3145f * (T + 273.15f))));
    return fminf(1.0f, k / p.OGT_rate);
}
__device__ __forceinline__ float tempFunc_PS_f(float T, const SpeciesDev32& p) {
    const float regT = shape_dec_f(T - p.Topt, p.Tmax - p.Topt, 4.0e-2f, 4);
    const float k = fmaxf(0.0f, expf(-p.Ea / (8.3145f * (T + 273.15f))) * regT);
    return fminf(1.0f, k / p.OGT_rate);
}
// Julia isless on floats without signed zeros: NaN orders last
__device__ __forceinline__ bool jl_lessf(float x, float y) { return x < y || (y != y && x == x); }

struct PhysArgs {
    Tab32 T;
    IndDev32 P;
    const SpeciesDev32* sp;
    const MemberForcing* F;
    const StepState* st;
    float dT;
    long long Gtot;
    const float* tr;
    const float* par;
    const int* pop;
    const int* pop_sp;
    const float4* env;          // packed environment of occupied interior cells
    unsigned long long* acc;
    uint32_t* dcnt;
    const uint32_t* err;
    const SpeciesDec64* dec64;  // [member * nsp + species]
    unsigned long long* guard;  // [0] decisions recomputed in Float64, [1] of those, decisions changed
    unsigned long long* dproc;  // optional process diagnostics, fixed point: (species * PI_NPROC + q) * Gtot
    uint32_t pmask;             // enabled processes (PI_PROC_* bits)
    int sub;                    // work units per tile (see unit_tile)
};

// Fixed-point units of the process diagnostics: rates (mmol s⁻¹) in the mass unit per minute,
// Bm, Cq, Nq and Pq in the mass unit, Chl in the Chl unit (so a sum over any set of individuals is
// exact in 64 bits and independent of the order).
__host__ __device__ inline double proc_unit(const MemberDev& m, int q) {
    return q < PI_PROC_Bm ? m.fx_unit / 60.0 : q < PI_PROC_Chl ? m.fx_unit : m.chl_unit;
}

// Guard band of the decisions (get_probability!, division_death_probability.jl:95-107): a draw
// within this relative distance of p·ΔT in Float32 takes the decision from p recomputed in Float64
// from the individual's Float32 state, which removes the rounding of the probability formulas
// (a few Float32 ulps) from the comparison.
#define F32_GUARD_REL 1.0e-5f

__device__ __forceinline__ double shape_dec_d(double x, double xmax, double k, int pw) {
    const double fx = fmax(0.0, fmin(1.0, 1.0 - x / xmax));
    const double p = pw == 2 ? fx * fx : (fx * fx) * (fx * fx);
    return p / (k + p);
}
__device__ __forceinline__ bool near_threshold(float r, float t) {
    return fabsf(r - t) <= F32_GUARD_REL * fabsf(t);
}

// flags, status, cell and logical slot of a slot, loaded one slot ahead of its physiology, and,
// for an active slot, its quotas and age and, when it was binned this step into an interior cell
// (not a stale cell), the environment record of that cell: phys_one then waits on no load.
struct PHead {
    int32_t code, ls;
    uint8_t fl, stt;
    int env;                    // e0, e1 hold the environment record
    float Bm, Cq, Nq, Pq, Chl, age;
    float4 e0, e1;
};
// The first level of a slot's loads (flags, status, cell, logical slot): the loads of phys_head
// depend on them, so k32_physiology issues these two slots ahead and phys_head one slot ahead.
struct PPre { int32_t code, ls; uint8_t fl, stt; };
__device__ __forceinline__ PPre phys_pre(const IndDev32& P, long long g, bool valid) {
    PPre r{-1, 0, 0, 0};
    if (valid) { r.fl = P.flags[g]; r.stt = P.stat[g]; r.code = P.cell[g]; r.ls = P.lslot[g]; }
    return r;
}
__device__ __forceinline__ PHead phys_head(const IndDev32& P, long long g, const PPre& pre, const MemberDev& m,
                                           const float4* __restrict__ envr) {
    PHead h{-1, 0, 0, 0, 0, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, {}, {}};
    {
        h.fl = pre.fl; h.stt = pre.stt; h.code = pre.code; h.ls = pre.ls;
        if (h.fl & F32_AC) {
            h.Bm = P.Bm[g]; h.Cq = P.Cq[g]; h.Nq = P.Nq[g]; h.Pq = P.Pq[g]; h.Chl = P.Chl[g]; h.age = P.age[g];
            if ((h.stt & F32_ST_AC0) && !(h.stt & F32_ST_STALE)) {
                int ci, cj, ck;
                unpack_int(m, h.code, ci, cj, ck);
                if (ci < m.Nx && cj < m.Ny && ck < m.Nz) {
                    const long long cq = m.cell_off + q_of(m, ci, cj, ck);
                    h.e0 = envr[2 * cq]; h.e1 = envr[2 * cq + 1];
                    h.env = 1;
                }
            }
        }
    }
    return h;
}

// What k32_physiology adds to the grid for one slot: the cell (-1: nothing; the diagnostics count
// num is added there) and the consumption of DIC, DOC, NH4, NO3, PO4 in fixed point (zero unless
// the individual was binned this step into an interior cell).
struct PhysOut { long long cq; unsigned long long v[5]; };

__device__ __forceinline__ PhysOut phys_one(const PhysArgs& a, const MemberDev& m, int mi, int s,
                                            long long g, uint32_t iter, double tnow, const PHead& hd) {
    const IndDev32& P = a.P;
    PhysOut out{-1, {0ull, 0ull, 0ull, 0ull, 0ull}};
    // the quotas are loaded with the environment
    const uint8_t fl = hd.fl, stt = hd.stt;
    const int32_t code = hd.code;
    if (!(fl & F32_AC)) return out;
    const int ac0 = stt & F32_ST_AC0;
    int q;
    bool inside;
    if (stt & F32_ST_STALE) {
        int xi, yi, zi;
        unpack_halo(m, P.scell[g], xi, yi, zi);
        q = gid3(m, xi, yi, zi);
        inside = interior_q(m, q);
    } else {
        int ci, cj, ck;
        unpack_int(m, code, ci, cj, ck);
        q = q_of(m, ci, cj, ck);
        inside = ci < m.Nx && cj < m.Ny && ck < m.Nz;
    }
    const long long cq = m.cell_off + q;
    const long long G = a.Gtot;
    const SpeciesDev32& p = a.sp[mi * a.T.nsp + s];
    const float dT = a.dT;
    float NH4 = 0.0f, NO3 = 0.0f, PO4 = 0.0f, DOC = 0.0f, parv = 0.0f, Tm = 0.0f, popv = 0.0f;
    if (ac0 && inside) {
        const float4 e0 = hd.env ? hd.e0 : a.env[2 * cq], e1 = hd.env ? hd.e1 : a.env[2 * cq + 1];
        NH4 = fmaxf(0.0f, e0.x); NO3 = fmaxf(0.0f, e0.y); PO4 = fmaxf(0.0f, e0.z); DOC = fmaxf(0.0f, e0.w);
        parv = e1.x; Tm = e1.y;
        popv = a.pop_sp ? (float)a.pop_sp[(long long)s * G + cq] : e1.z;
    } else if (ac0) {
        // a cell on the halo face (a position exactly at x = Nx): read the fields themselves
        NH4 = fmaxf(0.0f, a.tr[PI_NH4 * G + cq]); NO3 = fmaxf(0.0f, a.tr[PI_NO3 * G + cq]);
        PO4 = fmaxf(0.0f, a.tr[PI_PO4 * G + cq]); DOC = fmaxf(0.0f, a.tr[PI_DOC * G + cq]);
        parv = a.par[cq];
        Tm = a.F[mi].temp[q];
        popv = (float)(a.pop_sp ? a.pop_sp[(long long)s * G + cq] : a.pop[cq]);
    }
    float Bm = hd.Bm, Cq = hd.Cq, Nq = hd.Nq, Pq = hd.Pq, Chl = hd.Chl;
    const double fx_inv = m.fx_inv;         // read before the stores below
    const float tf = tempFunc_f(Tm, p);
    // calc_inorganic_uptake_kernel! (:48-56)
    const float aI = parv * p.alpha * p.Phi;
    const float PCm = p.PCmax * tempFunc_PS_f(Tm, p);
    const float PS = PCm * (1.0f - expf(-aI / fmaxf(1.0e-30f, PCm) * Chl / fmaxf(1.0e-30f, Bm))) * Bm;
    const float Qn = (Nq + Bm * p.R_NC) / fmaxf(1.0e-30f, Bm + Cq);
    const float Qp = (Pq + Bm * p.R_PC) / fmaxf(1.0e-30f, Bm + Cq);
    const float regQN = shape_dec_f(Qn, p.Nqmax, 1.0e-4f, 4), regQP = shape_dec_f(Qp, p.Pqmax, 1.0e-4f, 4);
    const float ipop = fmaxf(1.0f, popv);
    const float VNH4 = fminf(p.VNH4max * regQN * NH4 / fmaxf(1.0e-30f, NH4 + p.KsatNH4) * tf * Bm, NH4 / dT / ipop);
    const float VNO3 = fminf(p.VNO3max * regQN * NO3 / fmaxf(1.0e-30f, NO3 + p.KsatNO3) * tf * Bm, NO3 / dT / ipop);
    const float VPO4 = fminf(p.VPO4max * regQP * PO4 / fmaxf(1.0e-30f, PO4 + p.KsatPO4) * tf * Bm, PO4 / dT / ipop);
    // update_quotas_1_kernel! (:64-69)
    Cq += PS * dT; Pq += VPO4 * dT; Nq += (VNH4 + VNO3) * dT;
    // calc_organic_uptake_kernel! (:78-84)
    const float Qc = Cq / fmaxf(1.0e-30f, Bm + Cq);
    const float regQ = shape_dec_f(Qc, p.Cqmax, 1.0e-4f, 4);
    float VDOC = fminf(p.VDOCmax * regQ * DOC / fmaxf(1.0e-30f, DOC + p.KsatDOC) * tf * Bm, DOC / dT / ipop);
    VDOC = mulbf(VDOC, jl_lessf(1.0e-2f, PS / (VDOC + PS)));
    // calc_ρChl_kernel! (:92-97)
    const float rChl = mulbf(PS / fmaxf(1.0e-30f, Bm) * p.Chl2N / fmaxf(1.0e-30f, parv * p.alpha * p.Phi * Chl / Bm),
                             jl_lessf(1.0e-1f, parv));
    // calc_respir_kernel! (:105-108)
    const float resp = p.respir * Bm * tf;
    // update_quotas_2_kernel! (:117-124)
    Cq = Cq + (VDOC - resp) * dT;
    const float def = fmaxf(0.0f, 0.0f - Cq);
    Bm = Bm - def; Nq = Nq + def * p.R_NC; Pq = Pq + def * p.R_PC; Cq = Cq + def;
    // calc_BS_kernel! (:132-138)
    const float mn = fminf(fminf(Cq, Nq / p.R_NC), Pq / p.R_PC);
    const float BS = mn * p.k_mtb, exu = fmaxf(0.0f, Cq - mn) * p.k_mtb;
    // update_biomass_kernel! (:146-154)
    Bm += dT * BS; Cq -= dT * (BS + exu); Nq -= dT * BS * p.R_NC; Pq -= dT * BS * p.R_PC;
    Chl += dT * BS * p.R_NC * rChl;
    const float age = hd.age + dT / 3600.0f;
    // update_cellsize_kernel! (:163-166) and the probabilities (division_death_probability.jl:7-68)
    const float Sz = Bm / (p.Cquota * p.Nsuper);
    const float graz = popv * p.grz_P;
    const float mort = p.mort_P * shape_dec_f(Sz, p.mort_reg, 1.0e-5f, 4);
    float dv;
    if (p.dvid_type == 1) dv = p.dvid_P * shape_inc_f(Sz, p.dvid_reg, 2.0e-3f, 2);
    else {
        const float h = (float)(fmod(tnow, 86400.0) / 3600.0);
        if (p.dvid_type == 2) dv = p.dvid_P * shape_inc_f(h, p.dvid_reg, 1.0e-5f, 4);
        else dv = p.dvid_P * shape_inc_f(Sz, p.dvid_reg, 1.0e-3f, 4) * shape_inc_f(h, p.dvid_reg2, 1.0e-5f, 4);
    }
    // get_probability! (:95-107)
    float r0, r1, r2;
    draw3f(m.seed, iter, (uint32_t)s, PI_DRAW_DECISION, (uint32_t)hd.ls, r0, r1, r2);
    int dg = jl_lessf(r0, graz * dT), dm = jl_lessf(r1, mort * dT), dd = jl_lessf(r2, dv * dT);
    if (near_threshold(r0, graz * dT) || near_threshold(r1, mort * dT) || near_threshold(r2, dv * dT)) {
        // the same probabilities in Float64 from the Float32 state (the constants are the Float32
        // literals of the reference's formulas)
        const SpeciesDec64& q = a.dec64[mi * a.T.nsp + s];
        const double dTd = (double)dT, Sz64 = (double)Bm / q.CqNs;
        const double g64 = (double)popv * q.grz_P;
        const double m64 = q.mort_P * shape_dec_d(Sz64, q.mort_reg, (double)1.0e-5f, 4);
        double d64;
        if (q.dvid_type == 1) d64 = q.dvid_P * (1.0 - shape_dec_d(Sz64, q.dvid_reg, (double)2.0e-3f, 2));
        else {
            const double h = fmod(tnow, 86400.0) / 3600.0;
            if (q.dvid_type == 2) d64 = q.dvid_P * (1.0 - shape_dec_d(h, q.dvid_reg, (double)1.0e-5f, 4));
            else d64 = q.dvid_P * (1.0 - shape_dec_d(Sz64, q.dvid_reg, (double)1.0e-3f, 4)) *
                       (1.0 - shape_dec_d(h, q.dvid_reg2, (double)1.0e-5f, 4));
        }
        const int dg2 = (double)r0 < g64 * dTd, dm2 = (double)r1 < m64 * dTd, dd2 = (double)r2 < d64 * dTd;
        atomicAdd(&a.guard[0], 1ull);
        if (dg2 != dg || dm2 != dm || dd2 != dd) atomicAdd(&a.guard[1], 1ull);
        dg = dg2; dm = dm2; dd = dd2;
    }
    P.Bm[g] = Bm; P.Cq[g] = Cq; P.Nq[g] = Nq; P.Pq[g] = Pq; P.Chl[g] = Chl; P.age[g] = age;
    P.flags[g] = (uint8_t)(F32_AC | (dg ? F32_GRAZ : 0) | (dm ? F32_MORT : 0) | (dd ? F32_DVID : 0));
    // calc_consume_kernel! (consume_loss.jl:2-9): only individuals binned this step reach the grid
    out.cq = cq;                // diags num at the (possibly stale) cell
    if (ac0 && inside) {
        const double u = fx_inv;
        out.v[0] = to_fixed((resp - PS) * dT, u);
        out.v[1] = to_fixed((exu - VDOC) * dT, u);
        out.v[2] = to_fixed(-VNH4 * dT, u);
        out.v[3] = to_fixed(-VNO3 * dT, u);
        out.v[4] = to_fixed(-VPO4 * dT, u);
    }
    // diags_spcs! (Diagnostics/diagnostics_kernels.jl:14-33) at the same cell
    if (a.pmask) {
        const float v[PI_NPROC] = { PS, BS, VDOC, VNH4, VNO3, VPO4, resp, exu, Bm, Cq, Nq, Pq, Chl };
        for (int q = 0; q < PI_NPROC; ++q)
            if (a.pmask >> q & 1u) add_fixed(&a.dproc[((long long)s * PI_NPROC + q) * G + cq], v[q], 1.0 / proc_unit(m, q));
    }
    return out;
}

// k32_physiology's grid sums of one warp (segment s of one member): one atomic per run of a cell
__device__ __forceinline__ void scatter_phys(const PhysArgs& a, int s, const PhysOut& o) {
    if (__all_sync(0xffffffffu, o.cq < 0)) return;      // a warp of inactive slots adds nothing
    const WarpRuns R = warp_runs(o.cq);
    const int n = (int)run_sum(o.cq >= 0 ? 1u : 0u, R);
    unsigned long long v[5];
#pragma unroll
    for (int e = 0; e < 5; ++e) v[e] = run_sum(o.v[e], R);
    if (R.head && o.cq >= 0) {
        const long long G = a.Gtot, cq = o.cq;
        atomicAdd(&a.dcnt[(long long)s * 4 * G + cq], (uint32_t)n);
        const int slot_of[5] = { ACC_DIC, ACC_DOC, ACC_NH4, ACC_NO3, ACC_PO4 };
#pragma unroll
        for (int e = 0; e < 5; ++e)
            if (v[e]) atomicAdd(&a.acc[(long long)slot_of[e] * G + cq], v[e]);
    }
}

// MINB: blocks of 256 threads per SM the registers are fitted for. On 256×256×64 with 4 M individuals in
// blocks of 128: 264 µs with 4 (64 registers, which spill), 257 at 72 registers, 237 with 3 (80).
template <int MINB>
__global__ void __launch_bounds__(256, MINB) k32_physiology(PhysArgs a) {
    if (stopped(a.err)) return;
    const int bs = blockDim.x, ppt = F32_TILE / (bs * a.sub);
    const uint32_t iter = (uint32_t)(a.st->iteration + 1);
    const double tnow = (double)(a.st->iteration + 1) * (double)a.dT;
    for (int u = blockIdx.x; u < a.T.ntiles * a.sub; u += gridDim.x) {
        int first;
        const int2 tl = a.T.tiles[unit_tile(u, a.sub, first)];
        int mi, s;
        seg_of(a.T, tl.x, mi, s);
        const MemberDev& m = a.T.md[mi];
        const long long base = m.slot_off + (long long)s * m.C;
        long long slot = (long long)tl.y + first + threadIdx.x;
        PHead hd = phys_head(a.P, base + slot, phys_pre(a.P, base + slot, slot < m.C), m, a.env);
        PPre pre = phys_pre(a.P, base + slot + bs, 1 < ppt && slot + bs < m.C);
        for (int p = 0; p < ppt; ++p, slot += bs) {
            const PHead cur = hd;
            if (p + 1 < ppt) {
                hd = phys_head(a.P, base + slot + bs, pre, m, a.env);
                pre = phys_pre(a.P, base + slot + 2 * bs, p + 2 < ppt && slot + 2 * bs < m.C);
            }
            PhysOut o{-1, {0ull, 0ull, 0ull, 0ull, 0ull}};
            if (slot < m.C) o = phys_one(a, m, mi, s, base + slot, iter, tnow, cur);
            scatter_phys(a, s, o);
        }
    }
}

// ------------------------------------------------------------------------------------------
// (d) tracer update in Float32: the three DST3FL sweeps (DST3FL.jl:1-73, multi_dim_adv.jl:1-135)
//     and the rest of tracer_update! (tracer_update.jl:22-43) in two kernels: k32_xy (x and y sweeps
//     of a level tile, walked row by row) and k32_ztail (z sweep walking columns, then diffusion, sinking,
//     forcing, particle terms and apply_tendency!), and k32_close for the cells with a flux condition.
//     A warp walks one pair of tracers with its stencil window in registers; the coefficients of a face
//     are formed once, in shared memory, for the seven pairs of a block.
//
// The flux limiter is evaluated without forming θ: for the upwind side,
//   ψ(δ/δ⁰)·δ⁰ = max(0, min(δ⁰, d₀δ⁰ + d₁δ, Rδ)) for δ⁰ ≥ 0 and min(0, max(δ⁰, d₀δ⁰ + d₁δ, Rδ))
//   for δ⁰ < 0, R = (1 − cfl)/(cfl + 1e-20),
// which equals ψ(θ)·δ⁰ (the θmax cap never changes ψ) and needs no division by δ⁰, so gradients
// near zero are exact. The downwind term of the reference multiplies a zero transport and is
// dropped.
// ------------------------------------------------------------------------------------------
//
// Every product and sum of the tracer update is written with an explicit rounding intrinsic
// (__fmul_rn, __fadd_rn, __fsub_rn, and __fmaf_rn where a fused multiply-add is chosen), so the
// compiler contracts nothing on its own: the kernels that evaluate these formulas (k32_xy and
// k32_ztail, and the fused k32_tracer) give the same bits in whatever code they are inlined into.
struct FCu { float tr, d0c, d1c, R; };

__device__ __forceinline__ FCu fcu(float vel, float area, float rdxc, float dT) {
    FCu f;
    const float cfl = fabsf(__fmul_rn(__fmul_rn(vel, dT), rdxc));
    f.tr = __fmul_rn(area, vel);
    f.d0c = __fmul_rn(__fmul_rn(__fsub_rn(2.0f, cfl), __fsub_rn(1.0f, cfl)), 1.0f / 6.0f);
    f.d1c = __fmul_rn(__fmaf_rn(-cfl, cfl, 1.0f), 1.0f / 6.0f);
    f.R = __fdividef(__fsub_rn(1.0f, cfl), __fadd_rn(cfl, EPS20_F));
    return f;
}
// max(0, min(|d|, a, b)) with the sign of d on d, a and b: the two cases of δ⁰ in one, five or six
// operations instead of eight
__device__ __forceinline__ float limited(float d, float a, float b) {
    const unsigned sg = __float_as_uint(d) & 0x80000000u;
    const float as = __uint_as_float(__float_as_uint(a) ^ sg), bs = __uint_as_float(__float_as_uint(b) ^ sg);
    return __uint_as_float(__float_as_uint(fmaxf(0.0f, fminf(fminf(fabsf(d), as), bs))) | sg);
}
__device__ __forceinline__ float psid0(float d0, float dn, const FCu& f) {
    return limited(d0, __fmaf_rn(f.d0c, d0, __fmul_rn(f.d1c, dn)), __fmul_rn(f.R, dn));
}
// one sweep's update v − dtv·(ΔF − c·ftr) (multi_dim_adv.jl:111-135)
__device__ __forceinline__ float upd_sweep(float v, float dtv, float dF, float c, float ftr) {
    return __fmaf_rn(-dtv, __fmaf_rn(-c, ftr, dF), v);
}
// a·x1 − a·x0: the transport difference of a cell's two faces
__device__ __forceinline__ float tdiff(float a, float x1, float x0) { return __fmaf_rn(a, x1, -__fmul_rn(a, x0)); }
// tracer_forcing! of a nutrient tracer on max(0, ·): G + (aS·T + aO·T_partner)
__device__ __forceinline__ float add_forcing(float G, float aS, float own, float aO, float partner) {
    return __fadd_rn(G, __fmaf_rn(aS, fmaxf(0.0f, own), __fmul_rn(aO, fmaxf(0.0f, partner))));
}
// tracer_sinking!: G + (ws·T_above − ws·T)·ΔT/ΔzC
__device__ __forceinline__ float add_sinking(float G, float fup, float fdn, float sk) {
    return __fmaf_rn(__fsub_rn(fup, fdn), sk, G);
}
// the new tracer value T + (G + particle term) (apply_tendency!)
__device__ __forceinline__ float tendency(float c, float G, float plk) { return __fadd_rn(c, __fadd_rn(G, plk)); }
// landmask product of a difference (δ·mask_a·mask_b); LM = false: every cell is water
template <bool LM>
__device__ __forceinline__ float mk(float x, int ma, int mb) { return LM ? mulbf(mulbf(x, ma), mb) : x; }

// adv_flux_x / adv_flux_y at a face from c[f-2], c[f-1], c[f], c[f+1] and the landmask there; the
// upwind side is selected, not branched on (a zero transport gives a zero flux either way)
template <bool LM>
__device__ __forceinline__ float flux_h(const FCu& f, float cm2, float cm1, float c0, float cp1,
                                        int lm2, int lm1, int l0, int lp1) {
    const float d0 = mk<LM>(__fsub_rn(c0, cm1), l0, lm1);
    const bool pos = f.tr > 0.0f;
    const float dn = pos ? mk<LM>(__fsub_rn(cm1, cm2), lm1, lm2) : mk<LM>(__fsub_rn(cp1, c0), lp1, l0);
    const float ps = psid0(d0, dn, f);
    return __fmul_rn(f.tr, pos ? __fadd_rn(cm1, ps) : __fsub_rn(c0, ps));
}
// adv_flux_z at face k from c[k-2], c[k-1], c[k], c[k+1] (the index grows downward)
template <bool LM>
__device__ __forceinline__ float flux_v(const FCu& f, float cm2, float cm1, float c0, float cp1,
                                        int lm2, int lm1, int l0, int lp1) {
    const float d0 = mk<LM>(__fsub_rn(cm1, c0), l0, lm1);
    const bool pos = f.tr > 0.0f;
    const float dn = pos ? mk<LM>(__fsub_rn(c0, cp1), lp1, l0) : mk<LM>(__fsub_rn(cm2, cm1), lm1, lm2);
    const float ps = psid0(d0, dn, f);
    return __fmul_rn(f.tr, pos ? __fadd_rn(c0, ps) : __fsub_rn(cm1, ps));
}
__device__ __forceinline__ int wrap_ax(int a, int N, int H, int topo) {
    if (topo == PI_PERIODIC) { while (a < H + 1) a += N; while (a > N + H) a -= N; return a; }
    return a < H + 1 ? H + 1 : (a > N + H ? N + H : a);
}

__device__ __forceinline__ int acc_slot(int n) {
    switch (n) {
        case PI_DIC: return ACC_DIC; case PI_NH4: return ACC_NH4; case PI_NO3: return ACC_NO3;
        case PI_PO4: return ACC_PO4; case PI_DOC: return ACC_DOC; case PI_DON: return ACC_DON;
        case PI_DOP: return ACC_DOP; case PI_POC: return ACC_POC; case PI_PON: return ACC_PON;
        case PI_POP: return ACC_POP; default: return -1;
    }
}

__device__ __forceinline__ float getbc32(const FluxBC32& b, int a, int c, int64_t it) {
    if (b.kind == PI_BC_CONST) return b.v[0];
    if (b.kind == PI_BC_ARRAY2D) return b.v[(a - 1) + (long long)b.n1 * (c - 1)];
    const int64_t t = it < 1 ? 1 : (it > b.nt ? b.nt : it);   // the host rejects steps past nt
    return b.v[(a - 1) + (long long)b.n1 * ((c - 1) + (long long)b.n2 * (t - 1))];
}

// Pairs of FP32 values — the same cell of tracers 2p and 2p+1 — in one 64-bit register, for the
// packed FP32 instructions of sm_100 (add/sub/mul/fma .rn.f32x2). Each half is rounded exactly as the
// scalar __fadd_rn, __fsub_rn, __fmul_rn and __fmaf_rn, so the kernels that use them give the same bits
// as k32_tracer's scalar formulas with one instruction for two tracers.
typedef unsigned long long fx2;
__device__ __forceinline__ fx2 fx2_of(float lo, float hi) {
    fx2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fx2_split(fx2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ fx2 fx2_add(fx2 a, fx2 b) { fx2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ fx2 fx2_sub(fx2 a, fx2 b) { fx2 d; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ fx2 fx2_mul(fx2 a, fx2 b) { fx2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ fx2 fx2_fma(fx2 a, fx2 b, fx2 c) {
    fx2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// the face coefficients of one face for both halves
struct FCu2 { fx2 tr, d0c, d1c, R; };
// adv_flux at a face for two tracers from the upwind cell B, the cell A behind it and the downwind cell
// C: flux_h and flux_v select their operands by the sign of the transport; here the caller has, and as
// the limiter is odd, both signs are the one formula tr·(B + ψ). mAB, mBC: landmask products of the
// two differences as AND masks (δ·mask = copysign(0, δ) on land), all ones for water.
__device__ __forceinline__ fx2 flux3(const FCu2& f, fx2 A, fx2 B, fx2 C, bool lm, unsigned mAB, unsigned mBC) {
    fx2 d = fx2_sub(C, B), dn = fx2_sub(B, A);
    if (lm) {
        d &= ((fx2)mBC << 32) | mBC;
        dn &= ((fx2)mAB << 32) | mAB;
    }
    const fx2 a = fx2_fma(f.d0c, d, fx2_mul(f.d1c, dn)), b = fx2_mul(f.R, dn);
    float dl, dh, al, ah, bl, bh;
    fx2_split(d, dl, dh); fx2_split(a, al, ah); fx2_split(b, bl, bh);
    return fx2_mul(f.tr, fx2_add(B, fx2_of(limited(dl, al, bl), limited(dh, ah, bh))));
}
// upd_sweep for two tracers: v − dtv·(ΔF − c·ftr), with −dtv and −ftr given
__device__ __forceinline__ fx2 upd_sweep2(fx2 v, fx2 ndtv, fx2 dF, fx2 c, fx2 nftr) {
    return fx2_fma(ndtv, fx2_fma(c, nftr, dF), v);
}

struct TrArgs {
    Tab32 T;
    const int4* items;          // k32_xy: {member, i0, j0, level}; k32_ztail: {member, i0, j, k0}
    int nitems;
    const uint8_t* lm;
    const float* dzF;
    const float* dzC;
    const float* rdzC;          // 1 / dzC
    const BgcDev32* bgc;
    const FluxBC32* bcs;
    const StepState* st;
    const MemberForcing* F;
    long long Gtot;
    const float* tr;            // tracers at the start of the step
    float* tb;                  // tracer_temp after the x and y sweeps
    float* tr_next;
    unsigned long long* acc;
    const int* pop;
    float dT;
    const uint32_t* err;
};

// The coefficients of a face as the walking kernels keep them in shared memory, doubled on their way to
// the packed instructions: the copies would halve the accesses' moves, but take shared memory that is
// then missing as L1 (see k32_ztail).
__device__ __forceinline__ FCu2 get_fcu(const float4* s, int e, bool& pos) {
    const float4 a = s[e];
    pos = a.x > 0.0f;
    FCu2 f;
    f.tr = fx2_of(a.x, a.x); f.d0c = fx2_of(a.y, a.y); f.d1c = fx2_of(a.z, a.z); f.R = fx2_of(a.w, a.w);
    return f;
}
// Mask byte of a face and of the cell after it: water on both sides of B-C and of A-B (by the sign of the
// transport), no flux through the face, water in the cell and beyond its far face, and that sign
#define MB_BC 1u
#define MB_AB 2u
#define MB_ZERO 4u
#define MB_CELL 8u
#define MB_POS 16u                    // the transport is positive
__device__ __forceinline__ unsigned mask_byte(float tr, int lm2, int lm1, int l0, int lp1) {
    return (l0 & lm1 ? MB_BC : 0u) | ((tr > 0.0f ? lm1 & lm2 : lp1 & l0) ? MB_AB : 0u);
}
__device__ __forceinline__ unsigned and_mask(unsigned mb, unsigned bit) { return mb & bit ? 0xffffffffu : 0x80000000u; }
__device__ __forceinline__ fx2 fx2_and(fx2 v, unsigned m) { return v & (((fx2)m << 32) | m); }
__device__ __forceinline__ fx2 cell_mask(fx2 v, unsigned mb) { return fx2_and(v, and_mask(mb, MB_CELL)); }
// The two tracers of a pair: nutrients in the first five pairs, the iron tracers and dust in the last two
__host__ __device__ constexpr int pair_tracer(int p, int h) {
    return p == 0 ? (h ? PI_NH4 : PI_DIC) : p == 1 ? (h ? PI_PO4 : PI_NO3) : p == 2 ? (h ? PI_DON : PI_DOC)
         : p == 3 ? (h ? PI_POC : PI_DOP) : p == 4 ? (h ? PI_POP : PI_PON) : p == 5 ? (h ? PI_PFe_inorg : PI_DFe)
         : (h ? PI_Dust : PI_PFe_bio);
}
#define TR_PAIRS (PI_NTRACERS / 2)
// threadIdx.y as a value the compiler knows to be the same for the warp, so that what follows from it (the
// bases of the pair's arrays) can stay in uniform registers
__device__ __forceinline__ int warp_row() { return __shfl_sync(0xffffffffu, (int)threadIdx.y, 0); }
// element at a byte offset below 4 GB from a uniform base (a member's field: 14 of them, twice, and the
// particle sums would not fit the memory beyond that), which needs no 64-bit address arithmetic per access
__device__ __forceinline__ float ldg_at(const float* base, unsigned byte) {
    return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(base) + byte));
}
__device__ __forceinline__ void st_at(float* base, unsigned byte, float v) {
    *reinterpret_cast<float*>(reinterpret_cast<char*>(base) + byte) = v;
}

// x and y sweeps on one level of 31 columns (32 x faces, one per lane) × TY rows: warp p of the block walks
// the rows of tracer pair p from two above to two below (outside the domain through the halo-fill
// map). Each row's x sweep gives the tracer_temp row that the y sweep keeps in a window of four
// registers; a y face's flux is formed once and serves the rows on both sides, so nothing but the
// face coefficients, formed once for the 14 tracers, goes through shared memory. The x sweep loads a
// face's three cells in upwind order (no selects), two rows ahead. What bounds it is the latency of
// those loads and of the limiter's chain, so warps count more than registers: on 256×256×64 309 µs with
// two pairs per warp (16 warps per SM), 256 µs with one (28 warps), 231 µs at five blocks (35 warps, 56
// registers); 326 µs when every tile staged its rows, fluxes and intermediate rows in shared memory.
// Rows per tile (the walk costs TY + 4): 16 and 28 take 231 and 221 µs on 256×256×64, 74 and 75 on 128×128×64,
// 20 and 23 on 88×88×24, which 28 leaves short of blocks.
struct XYRows { float4 *fx, *fy; float *tx, *ty; int* row; uint8_t *mx, *my; };
__host__ __device__ inline size_t xy_smem(int ty) {
    return (size_t)(2 * ty + 5) * 32 * (sizeof(float4) + sizeof(float) + 1) + (size_t)(ty + 4) * sizeof(int);
}
template <bool LM>
__device__ __forceinline__ void xy_walk(const TrArgs& a, const MemberDev& m, const int4 it, const XYRows& S, int nr, int p) {
    const int lane = threadIdx.x;
    const int i0 = it.y, L = it.w, lastx = m.Nx + m.Hx;
    const float dz = a.dzF[m.dz_off + L - 1];
    const float az = __fmul_rn(m.dx, m.dy), dtv = __fdiv_rn(a.dT, __fmul_rn(az, dz));
    const fx2 ndtv = fx2_of(-dtv, -dtv);
    const int f = i0 + lane;
    const bool cell = lane < 31 && f <= lastx;
    const bool nox = f == lastx + 1 && m.tx != PI_PERIODIC;            // fill_halo_east_Gc! (Bounded)
    const unsigned fx4 = 4u * (unsigned)(min(f, lastx + 1) - 1);       // byte offset of the face's cell in a row
    const long long oa = pair_tracer(p, 0) * a.Gtot + m.cell_off, ob = pair_tracer(p, 1) * a.Gtot + m.cell_off;
    const float *ca = a.tr + oa, *cb = a.tr + ob;
    float *ta = a.tb + oa, *tb = a.tb + ob;
    // a row's cells in upwind order: behind, upwind and downwind of the face; two rows ahead of the sweep
    struct In { float a[2], b[2], c[2]; };
    In I0, I1;
    auto load = [&](In& I, int r) {
        if (r >= nr + 4) return;
        const bool pos = S.mx[r * 32 + lane] & MB_POS;
        const unsigned qb = 4u * (unsigned)S.row[r] + fx4 - (pos ? 4u : 0u), st = pos ? 0u - 4u : 4u;
        I.a[0] = ldg_at(ca, qb + st); I.a[1] = ldg_at(cb, qb + st);
        I.b[0] = ldg_at(ca, qb); I.b[1] = ldg_at(cb, qb);
        I.c[0] = ldg_at(ca, qb - st); I.c[1] = ldg_at(cb, qb - st);
    };
    fx2 T0 = 0ull, T1 = 0ull, T2 = 0ull, T3 = 0ull, g0 = 0ull, g1 = 0ull, g2 = 0ull, Fy = 0ull;
    auto row = [&](In& I, int r, bool face, bool store) {
        const int ex = r * 32 + lane;
        bool pos;
        const FCu2 fc = get_fcu(S.fx, ex, pos);
        const float tx = S.tx[ex];
        const unsigned mx = LM ? S.mx[ex] : 0u;
        const fx2 A = fx2_of(I.a[0], I.a[1]), B = fx2_of(I.b[0], I.b[1]), C = fx2_of(I.c[0], I.c[1]);
        load(I, r + 2);
        fx2 F = flux3(fc, A, B, C, LM, and_mask(mx, MB_AB), and_mask(mx, MB_BC));
        if (nox) F = 0ull;
        T0 = T1; T1 = T2; T2 = T3;
        g0 = g1; g1 = g2; g2 = pos ? C : B;
        float Fl, Fh;
        fx2_split(F, Fl, Fh);
        fx2 dF = fx2_sub(fx2_of(__shfl_down_sync(0xffffffffu, Fl, 1), __shfl_down_sync(0xffffffffu, Fh, 1)), F);
        if (LM) dF = cell_mask(dF, mx);
        T3 = upd_sweep2(g2, ndtv, dF, g2, fx2_of(tx, tx));
        if (!face) return;
        // y face j0 + r - 3 from rows r - 3 .. r, and the row between it and the face before
        const int ey = ex - 3 * 32;
        const FCu2 fy = get_fcu(S.fy, ey, pos);
        const unsigned my = S.my[ey];
        fx2 Fn = flux3(fy, pos ? T0 : T3, pos ? T1 : T2, pos ? T2 : T1, LM, and_mask(my, MB_AB), and_mask(my, MB_BC));
        if (my & MB_ZERO) Fn = 0ull;
        if (store && cell) {
            // row j0 + r - 4 is row r - 2 of the walk: window entry 1, its original tracer g0
            const float ty = S.ty[ey - 32];
            fx2 dG = fx2_sub(Fn, Fy);
            if (LM) dG = cell_mask(dG, S.my[ey - 32]);
            const unsigned q = 4u * (unsigned)S.row[r - 2] + fx4;
            float lo, hi;
            fx2_split(upd_sweep2(T1, ndtv, dG, g0, fx2_of(ty, ty)), lo, hi);
            st_at(ta, q, lo);
            st_at(tb, q, hi);
        }
        Fy = Fn;
    };
    load(I0, 0);
    load(I1, 1);
    row(I0, 0, false, false);
    row(I1, 1, false, false);
    row(I0, 2, false, false);
    row(I1, 3, true, false);
    int r = 4;
#pragma unroll 2
    for (; r + 1 < nr + 4; r += 2) {
        row(I0, r, true, true);
        row(I1, r + 1, true, true);
    }
    if (r < nr + 4) row(I0, r, true, true);
}

template <int TY>
__global__ void __launch_bounds__(32 * TR_PAIRS, 5) k32_xy(TrArgs a) {
    if (stopped(a.err)) return;
    extern __shared__ __align__(16) unsigned char xsm[];
    const int4 it = a.items[blockIdx.x];
    const MemberDev& m = a.T.md[it.x];
    XYRows S;
    S.fx = reinterpret_cast<float4*>(xsm);
    S.fy = S.fx + (TY + 4) * 32;
    S.tx = reinterpret_cast<float*>(S.fy + (TY + 1) * 32);
    S.ty = S.tx + (TY + 4) * 32;
    S.row = reinterpret_cast<int*>(S.ty + (TY + 1) * 32);
    S.mx = reinterpret_cast<uint8_t*>(S.row + TY + 4);
    S.my = S.mx + (TY + 4) * 32;
    const int lane = threadIdx.x, i0 = it.y, j0 = it.z, L = it.w, lastx = m.Nx + m.Hx, lasty = m.Ny + m.Hy;
    const int nr = min(TY, lasty - j0 + 1);
    const MemberForcing& F = a.F[it.x];
    const float *uu = F.vel1[0], *vv = F.vel1[1];
    const float dz = a.dzF[m.dz_off + L - 1], ax = __fmul_rn(m.dy, dz), ay = __fmul_rn(m.dx, dz);
    const float rdx = __frcp_rn(m.dx), rdy = __frcp_rn(m.dy);
    const bool land = !m.all_water;
    const int f = i0 + lane, fi = min(f, lastx + 1);             // lanes past the last face repeat it
    // (the velocities are loaded through the read-only path, so that several rows' loads are in flight)
#pragma unroll 5
    for (int r = threadIdx.y; r < nr + 4; r += TR_PAIRS) {
        const int e = r * 32 + lane, j = wrap_ax(j0 - 2 + r, m.Ny, m.Hy, m.ty);
        const int q = gid3(m, fi, j, L);
        const float uw = __ldg(uu + q), ue = __ldg(uu + q + 1);
        const FCu fc = fcu(uw, ax, rdx, a.dT);
        S.fx[e] = make_float4(fc.tr, fc.d0c, fc.d1c, fc.R);
        float ftr = tdiff(ax, ue, uw);
        unsigned mb = fc.tr > 0.0f ? MB_POS : 0u;
        if (land) {
            const int l0 = lm32(m, a.lm, fi, j, L), lp1 = lm32(m, a.lm, fi + 1, j, L);
            mb |= mask_byte(fc.tr, lm32(m, a.lm, fi - 2, j, L), lm32(m, a.lm, fi - 1, j, L), l0, lp1) | (l0 & lp1 ? MB_CELL : 0u);
            ftr = mk<true>(ftr, lp1, l0);
        }
        S.tx[e] = -ftr;
        S.mx[e] = (uint8_t)mb;
        if (lane == 0) S.row[r] = gid3(m, 1, j, L);
    }
#pragma unroll 5
    for (int r = threadIdx.y; r < nr + 1; r += TR_PAIRS) {
        const int e = r * 32 + lane, fj = j0 + r, ic = min(f, m.Gx);
        const bool special = fj == lasty + 1;
        const bool zero = f > lastx || (special && m.ty != PI_PERIODIC);       // fill_halo_north_Gc! (Bounded)
        const int fs = special ? m.Hy + 1 : fj;
        const FCu fc = fcu(zero ? 0.0f : __ldg(vv + gid3(m, ic, fs, L)), ay, rdy, a.dT);
        S.fy[e] = make_float4(fc.tr, fc.d0c, fc.d1c, fc.R);
        unsigned mb = zero ? MB_ZERO : 0u;
        const int jr = min(fj, m.Gy - 1), qr = gid3(m, ic, jr, L);
        float ftr = tdiff(ay, __ldg(vv + qr + m.Gx), __ldg(vv + qr));
        if (land) {
            mb |= mask_byte(fc.tr, lm32(m, a.lm, ic, fs - 2, L), lm32(m, a.lm, ic, fs - 1, L), lm32(m, a.lm, ic, fs, L),
                            lm32(m, a.lm, ic, fs + 1, L));
            const int c0 = lm32(m, a.lm, ic, jr, L), cp = lm32(m, a.lm, ic, jr + 1, L);
            mb |= c0 & cp ? MB_CELL : 0u;
            ftr = mk<true>(ftr, cp, c0);
        }
        S.ty[e] = -ftr;
        S.my[e] = (uint8_t)mb;
    }
    __syncthreads();
    if (land) xy_walk<true>(a, m, it, S, nr, warp_row());
    else xy_walk<false>(a, m, it, S, nr, warp_row());
}

// z sweep and the rest of tracer_update! for LZ levels of 32 columns: warp p of the block walks tracer
// pair p down the columns (packed instructions for both tracers) with the 4-level stencil window of
// tracer_temp and the flux of the face above the current cell in registers, and the inputs of the
// next two levels on their way. What does not depend on the tracer is formed once per item in
// shared memory for the 7 warps: the face coefficients, the vertical transport term of each cell, a bit
// per cell with individuals and the per-level constants (ΔT/vol, ΔT/ΔzC and the fixed-point unit per
// volume). As the warps walk the same cells, the forcing terms' reads of the other tracers at a cell hit
// lines already loaded: while they are in L1, which is what shared memory leaves of it. On 256×256×64 the
// kernel took 368 µs with 49 KB per block (which rounds to all of L1 at four blocks), 284 µs at 48 KB and
// 260 µs at 23 KB; 337 µs with a warp per pair whose inputs were not fetched ahead. Five blocks (56
// registers) spill: 309 µs. Levels per walk: 358 µs with 16, 260 with 32, 278 with 64 (each walk reads
// three levels of tracer_temp more than it writes). Latency bounds what is left.
struct ZLev {
    float dtv;      // ΔT / (Δx Δy ΔzF[k])
    float sk;       // ΔT / ΔzC (tracer_sinking!)
    float dz;       // ΔzF[k]
    float kzu, kzd; // tracer_diffusion!: κv·ΔT / ΔzF[k]², κv·ΔT / (ΔzF[k]·ΔzF[k+1])
    double fxv;     // mmol per fixed-point unit / (Δx Δy ΔzF[k])
};

// tracer_forcing! (tracer_forcings.jl:2-50) of the three iron tracers on max(0, tracer), with the
// products of rate constants and ΔT formed once per walk
struct FeCoef { float kpoc, frac, kdiss, fefe, frac_poc, lig, lpoc, lmin, ldust; };
__device__ __forceinline__ FeCoef fe_coef(const BgcDev32& b, float dT) {
    FeCoef c;
    c.kpoc = b.kPOC * dT; c.frac = b.DFeFrac * dT; c.kdiss = b.kdiss * dT;
    c.fefe = b.DFeFrac * b.lambda_Fe * dT; c.frac_poc = b.DFeFrac * b.lambda_POC * dT;
    c.lig = b.ligand; c.lpoc = b.lambda_POC; c.lmin = b.lambda_min; c.ldust = b.lambda_dust;
    return c;
}
__device__ __forceinline__ float fe_forcing(int n, const FeCoef& c, float dfe, float poc, float dust, float pfeb, float pfei) {
    const float fe = __fmul_rn(__fmul_rn(fmaxf(__fsub_rn(dfe, c.lig), 0.0f), dfe), c.fefe);
    const float bio = __fmul_rn(pfeb, c.kpoc), diss = __fmul_rn(pfei, c.kdiss);
    if (n == PI_DFe) {
        const float scav = __fadd_rn(__fadd_rn(__fmul_rn(c.lpoc, poc), c.lmin), __fmul_rn(c.ldust, dust));
        return __fsub_rn(__fadd_rn(__fsub_rn(bio, __fmul_rn(__fmul_rn(scav, dfe), c.frac)), diss), fe);
    }
    if (n == PI_PFe_bio) return __fsub_rn(__fmul_rn(__fmul_rn(poc, dfe), c.frac_poc), bio);
    const float scav = __fadd_rn(c.lmin, __fmul_rn(c.ldust, dust));
    return __fadd_rn(__fadd_rn(-diss, __fmul_rn(__fmul_rn(scav, dfe), c.frac)), fe);
}

// tracer_diffusion! (tracer_diffusion.jl:1-21) of one cell for two tracers, with the face areas, widths
// and ΔT of each axis folded into one coefficient (κh·ΔT/Δx², κh·ΔT/Δy², and per level κv·ΔT/ΔzF[k]² and
// κv·ΔT/(ΔzF[k]·ΔzF[k+1])): per tracer and cell six differences and as many multiply-adds, where the terms
// as the reference groups them take seven divisions.
#define DB_E 1u                       // water in the cell and its eastern neighbour
#define DB_W 2u                       // … and the western one as well (the x term is masked as a whole by DB_E)
#define DB_N 4u
#define DB_S 8u
#define DB_DN 16u                     // the z term as a whole is masked by the cell below
#define DB_UP 32u
struct DifNb { fx2 e, w, n, s, up, dn; };
__device__ __forceinline__ unsigned dif_bits(const MemberDev& m, const uint8_t* lm, int i, int j, int k) {
    const int c = lm32(m, lm, i, j, k), e = c & lm32(m, lm, i + 1, j, k), n = c & lm32(m, lm, i, j + 1, k), d = c & lm32(m, lm, i, j, k + 1);
    return (e ? DB_E : 0u) | (e & lm32(m, lm, i - 1, j, k) ? DB_W : 0u) | (n ? DB_N : 0u) | (n & lm32(m, lm, i, j - 1, k) ? DB_S : 0u)
         | (d ? DB_DN : 0u) | (d & lm32(m, lm, i, j, k - 1) ? DB_UP : 0u);
}
template <bool LM>
__device__ __forceinline__ fx2 z_diffusion(const DifNb& v, fx2 c, unsigned bits, fx2 kx, fx2 ky, float kzu, float kzd) {
    auto dif = [&](fx2 x, unsigned b) { const fx2 d = fx2_sub(x, c); return LM ? fx2_and(d, and_mask(bits, b)) : d; };
    const fx2 x = fx2_add(dif(v.e, DB_E), dif(v.w, DB_W)), y = fx2_add(dif(v.n, DB_N), dif(v.s, DB_S));
    const fx2 z = fx2_fma(fx2_of(kzu, kzu), dif(v.up, DB_UP), fx2_mul(fx2_of(kzd, kzd), dif(v.dn, DB_DN)));
    return fx2_fma(kx, x, fx2_fma(ky, y, z));
}
// apply_bcs! (apply_bcs.jl:4-98) of a tracer (conditions B of its six faces) in a cell on the boundary faces
// that are set in `on`
__device__ __forceinline__ float z_fluxes(const MemberDev& md, const FluxBC32* B, unsigned on, int i, int j, int k, float dz, float dT, int64_t itn) {
    float Gc = 0.0f;
    const int ii = i - md.Hx, jj = j - md.Hy, kk = k - md.Hz;
    const float az = md.dx * md.dy, volk = az * dz;
    const float axk = md.dy * dz, ayk = md.dx * dz;
    if (on >> PI_WEST & 1u) Gc += getbc32(B[PI_WEST], jj, kk, itn) * dT * axk / volk;
    if (on >> PI_EAST & 1u) Gc -= getbc32(B[PI_EAST], jj, kk, itn) * dT * axk / volk;
    if (on >> PI_SOUTH & 1u) Gc += getbc32(B[PI_SOUTH], ii, kk, itn) * dT * ayk / volk;
    if (on >> PI_NORTH & 1u) Gc -= getbc32(B[PI_NORTH], ii, kk, itn) * dT * ayk / volk;
    if (on >> PI_BOTTOM & 1u) Gc += getbc32(B[PI_BOTTOM], ii, jj, itn) * dT * az / volk;
    if (on >> PI_TOP & 1u) Gc -= getbc32(B[PI_TOP], ii, jj, itn) * dT * az / volk;
    return Gc;
}

// the x and y boundary faces of a cell in column (i, j)
__device__ __forceinline__ unsigned side_faces(const MemberDev& md, int i, int j) {
    return (i == 1 + md.Hx ? 1u << PI_WEST : 0u) | (i == md.Nx + md.Hx ? 1u << PI_EAST : 0u)
         | (j == 1 + md.Hy ? 1u << PI_SOUTH : 0u) | (j == md.Ny + md.Hy ? 1u << PI_NORTH : 0u);
}
// Shared memory of an item: coefficients of the faces k0 .. k0 + LZ of the 32 columns, vertical transport
// terms and populations of the cells, per-level constants, and with land the mask bits of face and cell
// and of the cell's diffusion.
struct ZItem { float4* f; float* tr; unsigned* pop; ZLev* lev; uint8_t *m, *d; };
__host__ __device__ inline size_t ztail_smem(int lz, bool gen) {
    return (size_t)(lz + 1) * 32 * sizeof(float4) + (size_t)lz * (32 * sizeof(float) + sizeof(unsigned) + sizeof(ZLev))
         + (size_t)((gen ? 2 : 1) * lz + 1) * 32;
}
// add_forcing's coefficients of nutrient tracer n (tracer_forcings.jl:2-50): aS·T(n) + aO·T(other),
// aO = 0 and other = n where there is no second tracer
__device__ __forceinline__ int nutrient_forcing(int n, const BgcDev32& b, float dT, float& aS, float& aO) {
    aS = 0.0f; aO = 0.0f;
    switch (n) {
        case PI_DIC: aO = b.kDOC * dT; return PI_DOC;
        case PI_DOC: aS = -b.kDOC * dT; aO = b.kPOC * dT; return PI_POC;
        case PI_POC: aS = -b.kPOC * dT; return n;
        case PI_NH4: aS = -b.Nit * dT; aO = b.kDON * dT; return PI_DON;
        case PI_NO3: aO = b.Nit * dT; return PI_NH4;
        case PI_DON: aS = -b.kDON * dT; aO = b.kPON * dT; return PI_PON;
        case PI_PON: aS = -b.kPON * dT; return n;
        case PI_PO4: aO = b.kDOP * dT; return PI_DOP;
        case PI_DOP: aS = -b.kDOP * dT; aO = b.kPOP * dT; return PI_POP;
        default: aS = -b.kPOP * dT; return n;                     // POP
    }
}
__device__ __forceinline__ fx2 fx2_max0(fx2 v) {
    float l, h;
    fx2_split(v, l, h);
    return fx2_of(fmaxf(0.0f, l), fmaxf(0.0f, h));
}

// KIND 0: a nutrient pair (linear forcing, particle sums); 1: DFe and PFe_inorg; 2: PFe_bio and Dust (iron
// forcing, sinking). GEN: diffusion or flux boundary conditions are switched on. CLOSE: the cells with a flux
// condition are finished here, not in k32_close.
template <int LZ, bool LM, int KIND, bool GEN, bool CLOSE>
__device__ __forceinline__ void z_walk(const TrArgs& a, const MemberDev& md, const int4 it, const ZItem& S) {
    const int lane = threadIdx.x, p = warp_row();
    const int na = pair_tracer(p, 0), nb = pair_tracer(p, 1);
    // member constants in registers: the stores of the walk could otherwise alias them
    const int Nx = md.Nx, Hx = md.Hx, Hz = md.Hz, Gx = md.Gx, Gy = md.Gy;
    const int i = it.y + lane, j = it.z, k0 = it.w;
    const int top = Hz + 1, bot = md.Nz + Hz, nl = min(LZ, bot - k0 + 1);
    // levels of the walk where any of the 32 columns holds an individual: only those have
    // particle sums to read and zero (a warp-uniform test)
    uint64_t occm = 0;
    if (KIND == 0) {
        for (int l = 0; l < nl; l += 32) occm |= (uint64_t)__ballot_sync(0xffffffffu, l + lane < nl && S.pop[l + lane]) << l;
    }
    if (i > Nx + Hx) return;
    const long long G = a.Gtot, off = md.cell_off;
    const float dT = a.dT;
    const int slab = Gx * Gy;
    const int qcol = (i - 1) + Gx * (j - 1);             // level 1 of the column, member-local
    const BgcDev32& b = a.bgc[it.x];
    const float* trm = a.tr + off;                        // all tracers of the member
    const float* ca = trm + na * G;
    const float* cb = trm + nb * G;
    const float* ta = a.tb + na * G + off;
    const float* tb = a.tb + nb * G + off;
    float* oa = a.tr_next + na * G + off;
    float* ob = a.tr_next + nb * G + off;
    unsigned long long* accA = nullptr;
    unsigned long long* accB = nullptr;
    // forcing: two other tracers of a nutrient pair (its own where there is none), or POC, DFe and Dust,
    // PFe_bio for the iron tracers
    const float *x0 = nullptr, *x1 = nullptr, *x2 = nullptr;
    bool has0 = true, has1 = true;
    fx2 aS = 0ull, aO = 0ull;
    if (KIND == 0) {
        float sa, oa_, sb, ob_;
        const int pa = nutrient_forcing(na, b, dT, sa, oa_), pb = nutrient_forcing(nb, b, dT, sb, ob_);
        aS = fx2_of(sa, sb); aO = fx2_of(oa_, ob_);
        has0 = pa != na; has1 = pb != nb;
        x0 = trm + pa * G; x1 = trm + pb * G;
        accA = a.acc + acc_slot(na) * G + off;
        accB = a.acc + acc_slot(nb) * G + off;
    } else if (KIND == 1) {
        x0 = trm + PI_POC * G; x1 = trm + PI_Dust * G; x2 = trm + PI_PFe_bio * G;
    } else {
        x0 = trm + PI_POC * G; x1 = trm + PI_DFe * G;
    }
    const FeCoef fc = fe_coef(b, dT);
    const float wsa = b.w_sink_org, wsb = b.w_sink_inorg;        // PFe_bio; Dust and PFe_inorg
    const bool dif = GEN && (b.kappa_h != 0.0f || b.kappa_v != 0.0f);
    const unsigned slab4 = 4u * (unsigned)slab, q40 = 4u * (unsigned)(qcol + (k0 - 1) * slab);
    auto tl = [&](int kk) { return 4u * (unsigned)(qcol + (min(max(kk, top), bot) - 1) * slab); };
    auto ld2 = [](const float* x, const float* y, unsigned q) { return fx2_of(ldg_at(x, q), ldg_at(y, q)); };
    // apply_bcs! touches boundary cells only. Where a tracer of the pair has a condition on a face of the cell,
    // the walk leaves the tendency in tr_next and the fluxes join it after the walk (CLOSE) or in k32_close; added
    // to the new tracer, a flux below half an ulp of it would be lost.
    // `open`: such cells are 1 all levels of the column, 2 the top one, 4 the bottom one.
    unsigned open = 0u;
    if (GEN) {
        const unsigned any = md.bcf[na] | md.bcf[nb];
        open = (any & side_faces(md, i, j) ? 1u : 0u) | (any >> PI_TOP & 1u ? 2u : 0u) | (any >> PI_BOTTOM & 1u ? 4u : 0u);
    }
    // inputs of a level: own tracers, tracer_temp two levels below, the others, the particle sums
    struct In { fx2 c, t; float e0, e1, e2; long long sa, sb; };
    unsigned qf = q40, qt = tl(k0 + 2);                   // byte offsets of the next level to fetch
    auto fetch = [&](In& I, int l) {
        if (l >= nl) {
            if (GEN && l == nl) I.c = ld2(ca, cb, qf);    // the cell below the last one, for the diffusion
            return;
        }
        I.c = ld2(ca, cb, qf);
        I.t = ld2(ta, tb, qt);
        if (KIND == 0) {
            if (has0) I.e0 = ldg_at(x0, qf);
            if (has1) I.e1 = ldg_at(x1, qf);
            if (occm >> l & 1ull) {
                const bool on = S.pop[l] >> lane & 1u;
                I.sa = on ? (long long)accA[qf >> 2] : 0;
                I.sb = on ? (long long)accB[qf >> 2] : 0;
            }
        } else {
            I.e0 = ldg_at(x0, qf);
            I.e1 = ldg_at(x1, qf);
            if (KIND == 1) I.e2 = ldg_at(x2, qf);
        }
        qf += slab4;
        if (k0 + l + 2 < bot) qt += slab4;                // the clamped map of the Bounded halo fill
    };
    In I0{}, I1{};
    fetch(I0, 0);
    fetch(I1, 1);
    // flux of a face between the cells w1 (above) and w2 (below) of the window: the upwind cell of a
    // positive (upward) transport is the one below
    auto zflux = [&](int e, fx2 w0, fx2 w1, fx2 w2, fx2 w3) {
        bool pos;
        const FCu2 fcz = get_fcu(S.f, e, pos);
        const unsigned mb = LM ? S.m[e] : 0u;
        return flux3(fcz, pos ? w3 : w0, pos ? w2 : w1, pos ? w1 : w2, LM, and_mask(mb, MB_AB), and_mask(mb, MB_BC));
    };
    // window of tracer_temp at levels k - 1 .. k + 2 of the current cell k
    fx2 w0 = ld2(ta, tb, tl(k0 - 2)), w1 = ld2(ta, tb, tl(k0 - 1)), w2 = ld2(ta, tb, tl(k0)), w3 = ld2(ta, tb, tl(k0 + 1));
    fx2 Ft = zflux(lane, w0, w1, w2, w3);
    // sinking tracers of the level above: PFe_inorg, or PFe_bio and Dust
    fx2 above = KIND != 0 && k0 - 1 > Hz ? ld2(ca, cb, tl(k0 - 1)) : 0ull;
    unsigned q4 = q40;
    const float khx = GEN ? b.kappa_h * dT / (md.dx * md.dx) : 0.0f, khy = GEN ? b.kappa_h * dT / (md.dy * md.dy) : 0.0f;
    DifNb nb4;
    if (GEN) nb4.up = ld2(ca, cb, q40 - slab4);
    auto level = [&](In& I, const In& next, int l) {
        const int k = k0 + l, e = l * 32 + lane;
        const fx2 c = I.c;
        w0 = w1; w1 = w2; w2 = w3; w3 = I.t;
        const float e0 = I.e0, e1 = I.e1, e2 = I.e2;
        const long long sa = I.sa, sb = I.sb;
        if (GEN && dif) {
            nb4.e = ld2(ca, cb, q4 + 4u); nb4.w = ld2(ca, cb, q4 - 4u);
            nb4.n = ld2(ca, cb, q4 + 4u * (unsigned)Gx); nb4.s = ld2(ca, cb, q4 - 4u * (unsigned)Gx);
            nb4.dn = next.c;
        }
        fetch(I, l + 2);
        const fx2 Fb = zflux(e + 32, w0, w1, w2, w3);                  // zero at the bottom
        const ZLev& L = S.lev[l];
        const float tr = S.tr[e], ndtv = -L.dtv;
        fx2 dF = fx2_sub(Ft, Fb);
        if (LM) dF = cell_mask(dF, S.m[e]);
        fx2 Gc = fx2_sub(upd_sweep2(w1, fx2_of(ndtv, ndtv), dF, c, fx2_of(tr, tr)), c);
        Ft = Fb;
        float cl, ch, gl, gh;
        fx2_split(c, cl, ch);
        if (GEN && dif) {
            Gc = fx2_add(Gc, z_diffusion<LM>(nb4, c, LM ? S.d[e] : 0u, fx2_of(khx, khx), fx2_of(khy, khy), L.kzu, L.kzd));
            nb4.up = c;
        }
        if (KIND == 0) {
            // tracer_forcing! on max(0, tracer): G + (aS·T + aO·T_other)
            Gc = fx2_add(Gc, fx2_fma(aS, fx2_max0(c), fx2_mul(aO, fx2_max0(fx2_of(has0 ? e0 : cl, has1 ? e1 : ch)))));
        } else {
            // tracer_sinking! (tracer_sinking.jl:1-42), then the iron forcing
            float al, ah;
            fx2_split(above, al, ah);
            fx2_split(Gc, gl, gh);
            auto sink = [&](float G0, float ws, float up, float own) {
                const float fup = (k - 1 <= Hz) ? 0.0f : __fmul_rn(ws, up);
                const float fdn = (k >= bot) ? 0.0f : __fmul_rn(ws, own);
                return add_sinking(G0, fup, fdn, L.sk);
            };
            if (KIND == 2) gl = sink(gl, wsa, al, cl);
            gh = sink(gh, wsb, ah, ch);
            above = c;
            const float poc = fmaxf(0.0f, e0);
            if (KIND == 1) {
                const float dfe = fmaxf(0.0f, cl), pfei = fmaxf(0.0f, ch), dust = fmaxf(0.0f, e1), pfeb = fmaxf(0.0f, e2);
                gl = __fadd_rn(gl, fe_forcing(PI_DFe, fc, dfe, poc, dust, pfeb, pfei));
                gh = __fadd_rn(gh, fe_forcing(PI_PFe_inorg, fc, dfe, poc, dust, pfeb, pfei));
            } else {
                const float dfe = fmaxf(0.0f, e1), pfeb = fmaxf(0.0f, cl);
                gl = __fadd_rn(gl, fe_forcing(PI_PFe_bio, fc, dfe, poc, 0.0f, pfeb, 0.0f));
            }
            Gc = fx2_of(gl, gh);
        }
        // particle terms from the fixed-point sums (zeroed as they are consumed), apply_tendency!
        // (tracer_update.jl:6-13)
        fx2 plk = 0ull;
        if (KIND == 0 && (occm >> l & 1ull)) {
            float pl = 0.0f, ph = 0.0f;
            if (sa) { accA[q4 >> 2] = 0ull; pl = (float)((double)sa * L.fxv); }
            if (sb) { accB[q4 >> 2] = 0ull; ph = (float)((double)sb * L.fxv); }
            plk = fx2_of(pl, ph);
        }
        float lo, hi;
        Gc = fx2_add(Gc, plk);
        fx2_split(GEN && (open & (1u | (k == top ? 2u : 0u) | (k == bot ? 4u : 0u))) ? Gc : fx2_add(c, Gc), lo, hi);
        st_at(oa, q4, lo);
        st_at(ob, q4, hi);
        q4 += slab4;
    };
    int l = 0;
#pragma unroll 2
    for (; l + 1 < nl; l += 2) {
        level(I0, I1, l);
        level(I1, I0, l + 1);
    }
    if (l < nl) level(I0, I1, l);
    if (CLOSE && open) {
        const FluxBC32 *Ba = a.bcs + md.bc_off + na * 6, *Bb = a.bcs + md.bc_off + nb * 6;
        const unsigned fa = md.bcf[na], fb = md.bcf[nb], side = side_faces(md, i, j);
        const int64_t itn = a.st->iteration + 1;
        for (l = 0; l < nl; ++l) {
            const int k = k0 + l, q = (int)(q40 >> 2) + l * slab;
            const unsigned on = side | (k == top ? 1u << PI_TOP : 0u) | (k == bot ? 1u << PI_BOTTOM : 0u);
            if (!((fa | fb) & on)) continue;
            const float ga = oa[q], gb = ob[q], va = __ldg(ca + q), vb = __ldg(cb + q), dz = S.lev[l].dz;
            oa[q] = __fadd_rn(va, __fadd_rn(ga, z_fluxes(md, Ba, fa & on, i, j, k, dz, dT, itn)));
            ob[q] = __fadd_rn(vb, __fadd_rn(gb, z_fluxes(md, Bb, fb & on, i, j, k, dz, dT, itn)));
        }
    }
}

template <int LZ, bool LM, bool GEN, bool CLOSE>
__device__ __forceinline__ void z_walk_any(const TrArgs& a, const MemberDev& m, const int4 it, const ZItem& S) {
    const int p = warp_row();
    if (p < 5) z_walk<LZ, LM, 0, GEN, CLOSE>(a, m, it, S);
    else if (p == 5) z_walk<LZ, LM, 1, GEN, CLOSE>(a, m, it, S);
    else z_walk<LZ, LM, 2, GEN, CLOSE>(a, m, it, S);
}

template <int LZ, bool GEN, bool CLOSE = false>
__global__ void __launch_bounds__(32 * TR_PAIRS, GEN ? 3 : 4) k32_ztail(TrArgs a) {
    if (stopped(a.err)) return;
    extern __shared__ __align__(16) unsigned char zsm[];
    ZItem S;
    S.f = reinterpret_cast<float4*>(zsm);                               // faces k0 .. k0 + LZ of the 32 columns
    S.lev = reinterpret_cast<ZLev*>(S.f + (LZ + 1) * 32);               // per-level constants
    S.tr = reinterpret_cast<float*>(S.lev + LZ);                        // vertical transport term of the cells k0 .. k0 + LZ - 1
    S.pop = reinterpret_cast<unsigned*>(S.tr + LZ * 32);                // a bit per cell of a level with individuals
    S.m = reinterpret_cast<uint8_t*>(S.pop + LZ);
    S.d = S.m + (LZ + 1) * 32;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int4 it = a.items[blockIdx.x];
    const MemberDev& m = a.T.md[it.x];
    const int k0 = it.w, bot = m.Nz + m.Hz, nl = min(LZ, bot - k0 + 1);
    const float* wv = a.F[it.x].vel1[2];
    const float az = __fmul_rn(m.dx, m.dy);
    const bool land = !m.all_water;
#pragma unroll 4
    for (int e = tid; e < (nl + 1) * 32; e += 32 * TR_PAIRS) {
        const int f = k0 + e / 32, i = it.y + (e & 31), j = it.z;
        FCu fc = {0.0f, 0.0f, 0.0f, 0.0f};
        unsigned mb = 0u;
        float ftr = 0.0f;
        int pop = 0;
        if (i <= m.Nx + m.Hx && f <= bot) {                   // fill_halo_bottom_Gc!: zero flux at the bottom
            const int q = gid3(m, i, j, f);
            const float wt = __ldg(wv + q);
            fc = fcu(wt, az, __ldg(a.rdzC + m.dz_off + f - 1), a.dT);
            ftr = tdiff(az, wt, __ldg(wv + q + m.Gx * m.Gy));  // cell f: w at its top and bottom faces
            if (land) {
                // the four points of the face from below, as those of an x or y face
                const int c0 = lm32(m, a.lm, i, j, f), cp = lm32(m, a.lm, i, j, f + 1);
                mb = mask_byte(fc.tr, cp, c0, lm32(m, a.lm, i, j, f - 1), lm32(m, a.lm, i, j, f - 2)) | (c0 & cp ? MB_CELL : 0u);
                ftr = mulbf(mulbf(ftr, cp), c0);
            }
            pop = __ldg(a.pop + m.cell_off + q);
        }
        S.f[e] = make_float4(fc.tr, fc.d0c, fc.d1c, fc.R);
        S.m[e] = (uint8_t)mb;
        if (GEN && land && e < nl * 32) S.d[e] = (uint8_t)(i <= m.Nx + m.Hx ? dif_bits(m, a.lm, i, j, f) : 0u);
        const unsigned occ = __ballot_sync(0xffffffffu, pop > 0);
        if (e < nl * 32) {
            S.tr[e] = -ftr;
            if (threadIdx.x == 0) S.pop[e / 32] = occ;
        }
    }
    if (tid < nl) {
        const int k = k0 + tid;
        ZLev L;
        const float dz = a.dzF[m.dz_off + k - 1], volk = __fmul_rn(az, dz);
        L.dtv = __fdiv_rn(a.dT, volk);
        L.sk = __fdiv_rn(a.dT, a.dzC[m.dz_off + k - m.Hz - 1]);
        L.dz = dz;
        const float kv = a.bgc[it.x].kappa_v * a.dT / dz;
        L.kzu = kv / dz;
        L.kzd = kv / a.dzF[m.dz_off + k];
        L.fxv = m.fx_unit / (double)volk;
        S.lev[tid] = L;
    }
    __syncthreads();
    if (land) z_walk_any<LZ, true, GEN, CLOSE>(a, m, it, S);
    else z_walk_any<LZ, false, GEN, CLOSE>(a, m, it, S);
}

// Closes the cells that the walks of an item of k32_ztail left open (a tracer of the pair has a condition on
// one of their faces): the fluxes join the tendency that waits in tr_next, and the tracer before the step is
// added. A kernel of its own, launched when a member has a flux condition: at the end of k32_ztail a warp had
// 31 levels of a boundary column one after the other, and the code cost the walk registers (117×93×31 with a
// western, a bottom and a top condition: 75.5 µs there, 72 µs for the two kernels; 81 to 93 µs with the
// tendency in k32_ztail in several forms). A launch more costs 4 µs of a small step, so batches of at most
// CLOSE_LEVELS levels have their walks finish the cells themselves (CLOSE): 22×33×5 44.2 µs per step against 47.4,
// 22×33×9 50.5 and 53.5, 60×50×12 59.0 and 57.8, 117×93×16 80.4 and 75.8.
#define CLOSE_LEVELS 10
__global__ void __launch_bounds__(256) k32_close(TrArgs a, int lz) {
    if (stopped(a.err)) return;
    const int4 it = a.items[blockIdx.x];
    const MemberDev& md = a.T.md[it.x];
    if (!md.any_bc) return;
    const FluxBC32* B = a.bcs + md.bc_off;
    const int j = it.z, k0 = it.w, bot = md.Nz + md.Hz, nl = min(lz, bot - k0 + 1);
    const int64_t itn = a.st->iteration + 1;
    for (int p = 0; p < TR_PAIRS; ++p) {
        const int na = pair_tracer(p, 0), nb = pair_tracer(p, 1);
        const unsigned fa = md.bcf[na], fb = md.bcf[nb];
        if (!(fa | fb)) continue;
        const float *ca = a.tr + na * a.Gtot + md.cell_off, *cb = a.tr + nb * a.Gtot + md.cell_off;
        float *oa = a.tr_next + na * a.Gtot + md.cell_off, *ob = a.tr_next + nb * a.Gtot + md.cell_off;
        for (int e = threadIdx.x; e < nl * 32; e += 256) {
            const int i = it.y + (e & 31), k = k0 + (e >> 5);
            const unsigned on = side_faces(md, i, j) | (k == 1 + md.Hz ? 1u << PI_TOP : 0u) | (k == bot ? 1u << PI_BOTTOM : 0u);
            if (i > md.Nx + md.Hx || !((fa | fb) & on)) continue;
            const int q = gid3(md, i, j, k);
            const float ga = oa[q], gb = ob[q], va = __ldg(ca + q), vb = __ldg(cb + q), dz = a.dzF[md.dz_off + k - 1];
            oa[q] = __fadd_rn(va, __fadd_rn(ga, z_fluxes(md, B + na * 6, fa & on, i, j, k, dz, a.dT, itn)));
            ob[q] = __fadd_rn(vb, __fadd_rn(gb, z_fluxes(md, B + nb * 6, fb & on, i, j, k, dz, a.dT, itn)));
        }
    }
}

// What the last kernel of a step does besides its own work: vel₀ .= vel₁ (time_step.jl:174-176),
// model.iteration += 1, model.t = iteration·ΔT. After a capacity error nothing advances and the
// tracers keep their values: the buffer that becomes current is a copy (every block copies its
// share). Nothing else in that kernel reads the forcing table or the counters.
struct StepEnd {
    int nm;
    MemberForcing* F;
    StepState* st;
    double dT;
    float* dst;                // tr_next
    const float* src;          // tracers at the start of the step
    long long n;               // PI_NTRACERS × Gtot
};
__device__ __forceinline__ void end_step(const StepEnd& e, int t, int nt) {
    for (int m = t; m < e.nm; m += nt)
        for (int c = 0; c < 3; ++c) e.F[m].vel0[c] = e.F[m].vel1[c];
    if (t == 0) { e.st->iteration += 1; e.st->t = (double)e.st->iteration * e.dT; e.st->call_step += 1; }
}
// true when the step stopped (a capacity error): copied, nothing more to do; otherwise the block
// `lead` advances the counters. t of nt threads over the grid, b of the block.
__device__ __forceinline__ bool close_step(const StepEnd& e, const uint32_t* err, long long t, long long nt, bool lead) {
    if (stopped(err)) {
        for (long long q = t; q < e.n; q += nt) e.dst[q] = e.src[q];
        return true;
    }
    if (lead) end_step(e, threadIdx.x, blockDim.x);
    return false;
}

// The source of halo index a along one axis of fill_halo_tracer! (halo_regions.jl:2-62): periodic
// ±N; Bounded the nearest interior cell; an interior index is its own.
__device__ __forceinline__ int halo_src(int a, int N, int H, int topo) {
    if (a > H && a <= N + H) return a;
    if (topo == PI_PERIODIC) return a <= H ? a + N : a - N;
    return a <= H ? H + 1 : N + H;
}

// fill_halo_tracer! in three passes (x, y, z), for members with a periodic axis of fewer cells than
// halo points, whose halo takes values of the halo itself as they were before the pass: one thread
// per line and field over all members' lines (grid y: fields); sources are read before writes.
// line_off[m] = first line of member m. The last pass (AXIS 2) closes the step.
template <int AXIS>
__global__ void k32_halo(const MemberDev* __restrict__ md, const long long* __restrict__ line_off, int nm,
                         long long Gtot, float* __restrict__ f, StepEnd end, const uint32_t* err) {
    if (AXIS == 2) {
        const long long nx = (long long)gridDim.x * blockDim.x;
        if (close_step(end, err, blockIdx.y * nx + (long long)blockIdx.x * blockDim.x + threadIdx.x, nx * gridDim.y,
                       blockIdx.x == 0 && blockIdx.y == 0)) return;
    } else if (stopped(err)) return;
    const long long nlines = line_off[nm];
    for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < nlines; l += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = nm - 1;
        while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (line_off[mid] <= l) lo = mid; else hi = mid - 1; }
        const MemberDev& m = md[lo];
        const long long ll = l - line_off[lo];
        const int na = AXIS == 0 ? m.Gy : m.Gx;
        const int a1 = (int)(ll % na) + 1, b1 = (int)(ll / na) + 1;
        const int N = AXIS == 0 ? m.Nx : AXIS == 1 ? m.Ny : m.Nz;
        const int H = AXIS == 0 ? m.Hx : AXIS == 1 ? m.Hy : m.Hz;
        const int topo = AXIS == 0 ? m.tx : AXIS == 1 ? m.ty : m.tz;
        float* c = f + blockIdx.y * Gtot + m.cell_off;
        auto at = [&](int t) -> float& {
            if (AXIS == 0) return c[gid3(m, t, a1, b1)];
            if (AXIS == 1) return c[gid3(m, a1, t, b1)];
            return c[gid3(m, a1, b1, t)];
        };
        float wv[8], ev[8];
        for (int h = 1; h <= H; ++h) {
            wv[h - 1] = at(halo_src(h, N, H, topo));
            ev[h - 1] = at(halo_src(N + H + h, N, H, topo));
        }
        for (int h = 1; h <= H; ++h) { at(h) = wv[h - 1]; at(N + H + h) = ev[h - 1]; }
    }
}

// The three passes above in one for small members (at most HALO_SMALL halo-padded cells: 0D boxes
// and short columns): composed, they give every cell the value that the cell reached by halo_src on
// each axis held before the first pass, so a block per member and field reads all its sources
// before it writes. A 0D box is 125 cells: the passes took 13 + 13 + 12 µs for their 14 dependent
// fields, this takes about 3.
#define HALO_SMALL 1024
__global__ void __launch_bounds__(256) k32_halo_small(const MemberDev* __restrict__ md, long long Gtot, float* __restrict__ f,
                                                      StepEnd end, const uint32_t* err) {
    const long long nb = gridDim.x * (long long)blockDim.x;
    if (close_step(end, err, blockIdx.y * nb + (long long)blockIdx.x * blockDim.x + threadIdx.x, nb * gridDim.y,
                   blockIdx.x == 0 && blockIdx.y == 0)) return;
    const MemberDev& m = md[blockIdx.x];
    const int G = (int)m.G;
    float* __restrict__ c = f + blockIdx.y * Gtot + m.cell_off;
    float v[HALO_SMALL / 256];
#pragma unroll
    for (int e = 0; e < HALO_SMALL / 256; ++e) {
        const int q = e * 256 + threadIdx.x;
        if (q >= G) continue;
        const int i = q % m.Gx + 1, r = q / m.Gx, j = r % m.Gy + 1, k = r / m.Gy + 1;
        v[e] = c[gid3(m, halo_src(i, m.Nx, m.Hx, m.tx), halo_src(j, m.Ny, m.Hy, m.ty), halo_src(k, m.Nz, m.Hz, m.tz))];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < HALO_SMALL / 256; ++e) {
        const int q = e * 256 + threadIdx.x;
        if (q < G) c[q] = v[e];
    }
}

// fill_halo_tracer! in one pass when every source cell is interior (no periodic axis has N < H): each
// halo cell takes the value of the cell reached by halo_src on each axis, which is what the three
// sequential passes produce. Grid: (x blocks, members); every thread walks halo cells of its
// member, all fields.
// halo cells of a member: the 2Hz halo levels, then the 2Hy halo rows of the interior levels,
// then the 2Hx halo columns of the interior rows
__global__ void k32_halo_direct(const MemberDev* __restrict__ md, long long Gtot, float* __restrict__ f,
                                StepEnd end, const uint32_t* err) {
    const long long nb = gridDim.x * (long long)blockDim.x;
    if (close_step(end, err, blockIdx.y * nb + (long long)blockIdx.x * blockDim.x + threadIdx.x, nb * gridDim.y,
                   blockIdx.x == 0 && blockIdx.y == 0)) return;
    const MemberDev& m = md[blockIdx.y];
    const int Gx = m.Gx, Gy = m.Gy, Nx = m.Nx, Ny = m.Ny, Nz = m.Nz, Hx = m.Hx, Hy = m.Hy, Hz = m.Hz;
    const int tx = m.tx, ty = m.ty;
    const int nz = 2 * Hz * Gx * Gy, ny = 2 * Nz * Hy * Gx, n = nz + ny + 2 * Nz * Ny * Hx;   // below 2^31
    float* __restrict__ c = f + m.cell_off;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        int i, j, k;
        if (t < nz) {
            const int kk = t / (Gx * Gy), r = t - kk * (Gx * Gy);
            k = kk < Hz ? kk + 1 : Nz + kk + 1;
            j = r / Gx + 1; i = r - (j - 1) * Gx + 1;
        } else if (t < nz + ny) {
            const int u = t - nz, kk = u / (2 * Hy * Gx), r = u - kk * (2 * Hy * Gx), jj = r / Gx;
            k = Hz + 1 + kk;
            j = jj < Hy ? jj + 1 : Ny + jj + 1;
            i = r - jj * Gx + 1;
        } else {
            const int u = t - nz - ny, kk = u / (2 * Hx * Ny), r = u - kk * (2 * Hx * Ny), jj = r / (2 * Hx);
            const int ii = r - jj * 2 * Hx;
            k = Hz + 1 + kk; j = Hy + 1 + jj;
            i = ii < Hx ? ii + 1 : Nx + ii + 1;
        }
        const int q = (i - 1) + Gx * ((j - 1) + Gy * (k - 1));
        const int si = halo_src(i, Nx, Hx, tx), sj = halo_src(j, Ny, Hy, ty), sk = halo_src(k, Nz, Hz, PI_BOUNDED);
        const int src = (si - 1) + Gx * ((sj - 1) + Gy * (sk - 1));
        // all reads before the writes, so that the fields' loads are in flight together
        float v[PI_NTRACERS];
#pragma unroll
        for (int n2 = 0; n2 < PI_NTRACERS; ++n2) v[n2] = c[n2 * Gtot + src];
#pragma unroll
        for (int n2 = 0; n2 < PI_NTRACERS; ++n2) c[n2 * Gtot + q] = v[n2];
    }
}

// Closes a step whose halo was written by the fused tracer kernel.
__global__ void k32_end_step(StepEnd end, const uint32_t* err) {
    close_step(end, err, (long long)blockIdx.x * blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x, blockIdx.x == 0);
}

// ------------------------------------------------------------------------------------------
// uploads, counts, budgets
// ------------------------------------------------------------------------------------------

// Interior array (reference layout, x fastest, Float64 or Float32) into a member's halo-padded
// FP32 field.
template <typename S>
__global__ void k32_scatter_interior(MemberDev m, float* __restrict__ dst, const S* __restrict__ src,
                                     int nx, int ny, int nz) {
    const long long n = (long long)nx * ny * nz;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % nx);
        const long long r = q / nx;
        const int j = (int)(r % ny), k = (int)(r / ny);
        dst[gid3(m, i + 1 + m.Hx, j + 1 + m.Hy, k + 1 + m.Hz)] = (float)src[q];
    }
}

// Velocity halo rule along one axis (halo_regions.jl:64-99) on one member-local field.
template <int AXIS>
__global__ void k32_halo_vel(MemberDev m, float* __restrict__ c, int face_axis) {
    const int na = AXIS == 0 ? m.Gy : m.Gx, nb = AXIS == 2 ? m.Gy : m.Gz;
    const long long nl = (long long)na * nb;
    for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < nl; l += (long long)gridDim.x * blockDim.x) {
        const int a1 = (int)(l % na) + 1, b1 = (int)(l / na) + 1;
        const int N = AXIS == 0 ? m.Nx : AXIS == 1 ? m.Ny : m.Nz;
        const int H = AXIS == 0 ? m.Hx : AXIS == 1 ? m.Hy : m.Hz;
        const int topo = AXIS == 0 ? m.tx : AXIS == 1 ? m.ty : m.tz;
        auto at = [&](int t) -> float& {
            if (AXIS == 0) return c[gid3(m, t, a1, b1)];
            if (AXIS == 1) return c[gid3(m, a1, t, b1)];
            return c[gid3(m, a1, b1, t)];
        };
        float wv[8], ev[8];
        const int velrule = (face_axis == AXIS) && topo == PI_BOUNDED;
        for (int h = 1; h <= H; ++h) {
            wv[h - 1] = topo == PI_PERIODIC ? at(N + h) : at(H + 1);
            ev[h - 1] = topo == PI_PERIODIC ? at(H + h) : at(N + H);
        }
        const float face = velrule ? at(N + H + 1) : 0.0f;
        for (int h = 1; h <= H; ++h) at(h) = wv[h - 1];
        if (velrule) { for (int h = N + H + 2; h <= N + 2 * H; ++h) at(h) = face; }
        else { for (int h = 1; h <= H; ++h) at(N + H + h) = ev[h - 1]; }
    }
}

// A setter's new own velocity (vel₁) and/or temperature of a member, bound on the device in
// stream order (after the steps already queued).
__global__ void k32_bind_own(MemberForcing* __restrict__ F, int m, const float* u, const float* v, const float* w,
                             const float* temp) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    MemberForcing& f = F[m];
    if (u) { f.vel1[0] = u; f.vel1[1] = v; f.vel1[2] = w; }
    if (temp) f.temp = temp;
}

template <typename S>
__global__ void k32_to_f32(float* __restrict__ dst, const S* __restrict__ src, long long n) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (float)src[q];
}

__global__ void k32_d2f(float* __restrict__ dst, const double* __restrict__ src, long long n) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (float)src[q];
}
__global__ void k32_f2d(double* __restrict__ dst, const float* __restrict__ src, long long n) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (double)src[q];
}
__global__ void k32_u2d(double* __restrict__ dst, const uint32_t* __restrict__ src, long long n) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (double)src[q];
}

// Index of the first non-finite value of a[0, n) (atomicMin into *first, which starts at ~0).
__global__ void k32_first_nonfinite(const float* __restrict__ a, long long n, unsigned long long* first) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        if (!isfinite(a[q])) atomicMin(first, (unsigned long long)q);
}

// First logical slot of a segment whose active individual has a non-finite attribute.
__global__ void k32_first_nonfinite_inds(IndDev32 P, long long base, long long C, unsigned long long* first) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x) {
        const long long g = base + q;
        if (!(P.flags[g] & F32_AC)) continue;
        const float v[10] = { P.ox[g], P.oy[g], P.oz[g], P.Bm[g], P.Cq[g], P.Nq[g], P.Pq[g], P.Chl[g], P.age[g], P.gen[g] };
        bool bad = false;
        for (int k = 0; k < 10; ++k) bad |= !isfinite(v[k]);
        if (bad) atomicMin(first, (unsigned long long)P.lslot[g]);
    }
}

// diags.tracer[name] .+= tracer (time_step.jl:168-172) for the enabled tracers, halos included.
__global__ void k32_diag_tracers(float* __restrict__ d, const float* __restrict__ tr, uint32_t mask, long long Gtot,
                                 const uint32_t* err) {
    if (stopped(err)) return;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < (long long)PI_NTRACERS * Gtot;
         q += (long long)gridDim.x * blockDim.x)
        if (mask >> (q / Gtot) & 1u) d[q] = d[q] + tr[q];
}

// fixed-point sums to Float64 values
__global__ void k32_fx2d(double* __restrict__ dst, const unsigned long long* __restrict__ src, long long n, double unit) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = (double)(long long)src[q] * unit;
}

// Active individuals of a slot range (calc_active_individuals, models.jl:157-164).
__global__ void k32_count_active(const uint8_t* __restrict__ flags, long long n, unsigned long long* out) {
    unsigned long long c = 0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        c += (flags[q] & F32_AC) ? 1 : 0;
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// FP64 mass budgets of one member: interior Σ c·vol of the C, N and P tracers (DIC+DOC+POC,
// NH4+NO3+DON+PON, PO4+DOP+POP) and the individuals' C, N, P. Block partials (fixed order).
__global__ void k32_budget_cells(MemberDev m, const float* __restrict__ tr, const float* __restrict__ dzF,
                                 long long Gtot, double* __restrict__ partial) {
    __shared__ double sh[3][256];
    double c = 0.0, n = 0.0, p = 0.0;
    const long long V = (long long)m.Nx * m.Ny * m.Nz;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < V; q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % m.Nx) + 1 + m.Hx;
        const long long r = q / m.Nx;
        const int j = (int)(r % m.Ny) + 1 + m.Hy, k = (int)(r / m.Ny) + 1 + m.Hz;
        const long long cq = m.cell_off + gid3(m, i, j, k);
        const double vol = (double)m.dx * (double)m.dy * (double)dzF[m.dz_off + k - 1];
        c += vol * ((double)tr[PI_DIC * Gtot + cq] + (double)tr[PI_DOC * Gtot + cq] + (double)tr[PI_POC * Gtot + cq]);
        n += vol * ((double)tr[PI_NH4 * Gtot + cq] + (double)tr[PI_NO3 * Gtot + cq] + (double)tr[PI_DON * Gtot + cq] + (double)tr[PI_PON * Gtot + cq]);
        p += vol * ((double)tr[PI_PO4 * Gtot + cq] + (double)tr[PI_DOP * Gtot + cq] + (double)tr[PI_POP * Gtot + cq]);
    }
    sh[0][threadIdx.x] = c; sh[1][threadIdx.x] = n; sh[2][threadIdx.x] = p;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) for (int r = 0; r < 3; ++r) sh[r][threadIdx.x] += sh[r][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) for (int r = 0; r < 3; ++r) partial[blockIdx.x * 3 + r] = sh[r][0];
}

__global__ void k32_budget_inds(MemberDev m, int nsp, const SpeciesDev32* __restrict__ sp, IndDev32 P,
                                double* __restrict__ partial) {
    __shared__ double sh[3][256];
    double c = 0.0, n = 0.0, p = 0.0;
    const long long S = (long long)nsp * m.C;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < S; q += (long long)gridDim.x * blockDim.x) {
        // logical slot order, so the sum does not depend on the storage order
        const long long g = m.slot_off + (q / m.C) * m.C + P.phys[m.slot_off + q];
        if (!(P.flags[g] & F32_AC)) continue;
        const SpeciesDev32& s = sp[q / m.C];
        const double Bm = P.Bm[g];
        c += Bm + (double)P.Cq[g];
        n += Bm * (double)s.R_NC + (double)P.Nq[g];
        p += Bm * (double)s.R_PC + (double)P.Pq[g];
    }
    sh[0][threadIdx.x] = c; sh[1][threadIdx.x] = n; sh[2][threadIdx.x] = p;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) for (int r = 0; r < 3; ++r) sh[r][threadIdx.x] += sh[r][threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) for (int r = 0; r < 3; ++r) partial[blockIdx.x * 3 + r] = sh[r][0];
}

// ------------------------------------------------------------------------------------------
// storage order: counting sort of every segment by cell (a periodic pass between steps)
// ------------------------------------------------------------------------------------------

// Sort bin of a stored slot: its interior cell in x-fastest order; an inactive slot goes to one of
// the bins after the cells, one per tile of F32_TILE stored positions (so inactive slots keep
// their relative order and no bin collects a whole segment).
__device__ __forceinline__ long long sort_bin(const MemberDev& m, int s, uint8_t fl, int32_t code, long long slot) {
    const long long V = (long long)m.Nx * m.Ny * m.Nz;
    const long long per = V + (m.wps >> 5);
    long long b;
    if ((fl & F32_AC) && code >= 0) {
        int ci, cj, ck;
        unpack_int(m, code, ci, cj, ck);
        b = min(ci, m.Nx - 1) + (long long)m.Nx * (min(cj, m.Ny - 1) + (long long)m.Ny * min(ck, m.Nz - 1));
    } else {
        b = V + slot / F32_TILE;
    }
    return m.bin_off + (long long)s * per + b;
}

// Warp-aggregated increment of bin counters: lanes with the same bin add once; each lane gets the
// counter value before its own increment (the lanes of a bin take consecutive values). All 32
// lanes call it; lanes with valid = false take no part.
__device__ __forceinline__ unsigned long long bin_claim(unsigned long long* ctr, long long bin, bool valid) {
    const int lane = threadIdx.x & 31;
    const unsigned vmask = __ballot_sync(0xffffffffu, valid);
    const unsigned long long key = valid ? (unsigned long long)bin : ~0ull;
    const unsigned peers = __match_any_sync(0xffffffffu, key) & vmask;
    const int leader = valid ? __ffs(peers) - 1 : lane;
    unsigned long long base = 0;
    if (valid && lane == leader) base = atomicAdd(&ctr[bin], (unsigned long long)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    return base + (unsigned long long)__popc(peers & ((1u << lane) - 1u));
}

// population of every bin (bins zeroed beforehand); blockDim.x divides F32_TILE
__global__ void k32_sort_count(Tab32 T, IndDev32 P, unsigned long long* __restrict__ bins) {
    for (int t = blockIdx.x; t < T.ntiles; t += gridDim.x) {
        const int2 tl = T.tiles[t];
        int mi, s;
        seg_of(T, tl.x, mi, s);
        const MemberDev& m = T.md[mi];
        const long long base = m.slot_off + (long long)s * m.C;
        for (int p = 0; p < F32_TILE / (int)blockDim.x; ++p) {
            const long long slot = (long long)tl.y + p * blockDim.x + threadIdx.x;
            const bool valid = slot < m.C;
            const long long g = base + (valid ? slot : 0);
            const long long bin = valid ? sort_bin(m, s, P.flags[g], P.cell[g], slot) : 0;
            bin_claim(bins, bin, valid);
        }
    }
}

// Moves every slot from P to Q at the next position of its bin (offs: the exclusive scan of the
// bin populations over the whole batch, which starts each segment's bins at the segment's first
// slot) and records where each logical slot went. The order inside a bin is that of the atomics;
// nothing computed from the individuals depends on it.
__global__ void k32_sort_scatter(Tab32 T, IndDev32 P, IndDev32 Q, unsigned long long* __restrict__ offs) {
    for (int t = blockIdx.x; t < T.ntiles; t += gridDim.x) {
        const int2 tl = T.tiles[t];
        int mi, s;
        seg_of(T, tl.x, mi, s);
        const MemberDev& m = T.md[mi];
        const long long base = m.slot_off + (long long)s * m.C;
        for (int p = 0; p < F32_TILE / (int)blockDim.x; ++p) {
            const long long slot = (long long)tl.y + p * blockDim.x + threadIdx.x;
            const bool valid = slot < m.C;
            const long long g = base + (valid ? slot : 0);
            const uint8_t fl = P.flags[g];
            const int32_t code = P.cell[g];
            const long long np = (long long)bin_claim(offs, valid ? sort_bin(m, s, fl, code, slot) : 0, valid);
            if (!valid) continue;
            Q.cell[np] = code; Q.scell[np] = P.scell[g];
            Q.ox[np] = P.ox[g]; Q.oy[np] = P.oy[g]; Q.oz[np] = P.oz[g];
            Q.Bm[np] = P.Bm[g]; Q.Cq[np] = P.Cq[g]; Q.Nq[np] = P.Nq[g]; Q.Pq[np] = P.Pq[g];
            Q.Chl[np] = P.Chl[g]; Q.age[np] = P.age[g]; Q.gen[np] = P.gen[g];
            Q.flags[np] = fl; Q.stat[np] = P.stat[g];
            const int L = P.lslot[g];
            Q.lslot[np] = L;
            P.phys[base + L] = (int)(np - base);
        }
    }
}

// Slots L0 .. L0 + n - 1 of one segment (logical order) as the boundary's columns: 8-byte columns of n
// values one after another in `out` (bit q of mask: column q of ECOL_*; xi, yi, zi as int64), then ac
// as bytes when bit ECOL_AC is set.
enum { ECOL_X = 0, ECOL_Y, ECOL_Z, ECOL_SZ, ECOL_BM, ECOL_CQ, ECOL_NQ, ECOL_PQ, ECOL_CHL, ECOL_GEN, ECOL_AGE, ECOL_GRAZ,
       ECOL_MORT, ECOL_DVID, ECOL_XI, ECOL_YI, ECOL_ZI, ECOL_AC };
__global__ void __launch_bounds__(256) k32_export(IndDev32 P, MemberDev m, long long base, long long L0, long long n, uint32_t mask,
                                                  float cq_ns, unsigned long long* __restrict__ out, uint32_t* __restrict__ bad) {
    const long long t = (long long)blockIdx.x * 256 + threadIdx.x;
    if (t >= n) return;
    const long long L = L0 + t;
    const int ph = P.phys[base + L];
    if (ph < 0 || ph >= m.C || P.lslot[base + ph] != (int)L) { *bad = 1u; return; }
    const long long g = base + ph;
    const int32_t code = P.cell[g];
    const uint8_t fl = P.flags[g];
    int c[3] = { 0, 0, 0 };
    if (code >= 0) unpack_int(m, code, c[0], c[1], c[2]);
    long long at = 0;
    auto put = [&](int q, double v) { if (mask >> q & 1u) { out[at * n + t] = (unsigned long long)__double_as_longlong(v); ++at; } };
    const float off[3] = { P.ox[g], P.oy[g], P.oz[g] };
    for (int a = 0; a < 3; ++a) put(ECOL_X + a, code < 0 ? 0.0 : c[a] + (double)off[a]);
    const float Bm = P.Bm[g];
    put(ECOL_SZ, (double)__fdiv_rn(Bm, cq_ns));
    put(ECOL_BM, (double)Bm);
    if (mask >> ECOL_CQ & 1u) put(ECOL_CQ, (double)P.Cq[g]);
    if (mask >> ECOL_NQ & 1u) put(ECOL_NQ, (double)P.Nq[g]);
    if (mask >> ECOL_PQ & 1u) put(ECOL_PQ, (double)P.Pq[g]);
    if (mask >> ECOL_CHL & 1u) put(ECOL_CHL, (double)P.Chl[g]);
    if (mask >> ECOL_GEN & 1u) put(ECOL_GEN, (double)P.gen[g]);
    if (mask >> ECOL_AGE & 1u) put(ECOL_AGE, (double)P.age[g]);
    put(ECOL_GRAZ, fl & F32_GRAZ ? 1.0 : 0.0);
    put(ECOL_MORT, fl & F32_MORT ? 1.0 : 0.0);
    put(ECOL_DVID, fl & F32_DVID ? 1.0 : 0.0);
    if (mask >> ECOL_XI & 7u) {
        const int H[3] = { m.Hx, m.Hy, m.Hz };
        int x[3];
        if (P.stat[g] & F32_ST_STALE) unpack_halo(m, P.scell[g], x[0], x[1], x[2]);
        else for (int a = 0; a < 3; ++a) x[a] = code < 0 ? H[a] : c[a] + 1 + H[a];
        for (int a = 0; a < 3; ++a)
            if (mask >> (ECOL_XI + a) & 1u) { out[at * n + t] = (unsigned long long)x[a]; ++at; }
    }
    if (mask >> ECOL_AC & 1u) reinterpret_cast<uint8_t*>(out + at * n)[t] = fl & F32_AC ? 1 : 0;
}

// Storage order equal to the logical order over a slot range (after an upload): lslot and phys
// are the identity, relative to the segment's first slot.
__global__ void k32_identity_order(IndDev32 P, long long base, long long C) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < C; q += (long long)gridDim.x * blockDim.x) {
        P.lslot[base + q] = (int)q;
        P.phys[base + q] = (int)q;
    }
}

}  // namespace p32
