// fx_plan.h — index maps and launch plans that need no CUDA: included by the kernels and the engine,
// and compiled by the host compiler alone in the CPU tests.
#pragma once

#include <algorithm>
#include <array>
#include <cmath>
#include <vector>

#include "../../include/firex.h"

#ifdef __CUDACC__
#define FX_HOST_DEVICE __host__ __device__ inline
#else
#define FX_HOST_DEVICE inline
#endif

// ---- the two-sweep pass by strips (fx_jacobi_zs.cuh) ---------------------------------------------
#define FX_ZS_THREADS 64
#define FX_ZS_ROWS 2  // rows of a thread's strip
#define FX_ZS_TXG 8   // 4-cell groups of a tile row

// Index of a plane or row outside 0 .. n - 1 reflected into it (-1 is 0, n is n - 1), for an index
// less than n outside.
FX_HOST_DEVICE int fx_zs_reflect(int q, int n) { return q < 0 ? -1 - q : (q >= n ? 2 * n - 1 - q : q); }

// Row of the grid that a strip tile's input row q is copied from (fx_jacobi_zs.cuh): rows below the
// floor are reflected, rows above the open top (q >= Y, whose values reach no stored cell) are
// the top row. q is -2 or more; a tile of few rows reaches far above the top of a flat grid.
FX_HOST_DEVICE int fx_zs_input_row(int q, int Y) { return q < 0 ? -1 - q : (q < Y ? q : Y - 1); }

FX_HOST_DEVICE int fx_zs_bricks(int X, int Y, int Z, int zc, int txg) {
    const int tx = 4 * txg, ty = FX_ZS_ROWS * (FX_ZS_THREADS / txg) - 2;
    return ((X + tx - 1) / tx) * ((Y + ty - 1) / ty) * ((Z + zc - 1) / zc);
}

// ---- the resident Jacobi (fx_jacobi_res.cuh, fx_jacobi_reg.cuh) -----------------------------------
#define FX_RES_THREADS 512
#define FX_RES_COPY_TC (FX_RES_THREADS - 32)  // compute threads of variant 4 (the last warp copies)
#define FX_RES_MAXG 12                // groups of 4 cells per thread, column variant
#define FX_RES_MAXF 4                 // face groups per thread, faces-first variant
#define FX_RES_MAXI 11                // interior groups per thread, faces-first variant
#define FX_RES_MAXI_SMALL 7           // ... its instance for small boxes (fewer registers)
#define FX_RES_MAXZ 10                // interior planes per thread column, faces-first column variant
#define FX_RES_SMEM_MAX (226 * 1024)  // dynamic shared memory per CTA (227 KB opt-in less static)
#define FX_RES_MAX_CTAS 1024          // boxes per simulation and phase (flag slots)

#define FX_REG_THREADS 384
#define FX_REG_MAXZ 4  // planes of a thread's column part
#define FX_REG_MAXH 4  // halo quads a thread receives per sweep

// Box decomposition of one simulation for the resident Jacobi: boxes of by x bz rows of
// full x rows, nby x nbz of them (CTA b owns box (b % nby, b / nby)).
struct FxResBox {
    int by, bz, nby, nbz;
    int exOff;  // FX_RES_REGISTERS: the member's first packet (16 bytes) in the exchange buffer
    int pad[3];
};

// Shared-memory bytes of a box: pressure with halo rows + divergence.
FX_HOST_DEVICE long long fx_res_smem_bytes(int X, int by, int bz) {
    return ((long long)(by + 2) * (bz + 2) + (long long)by * bz) * X * 4;
}

// Geometry of box b of a plan: rows y0 .. y0 + ny - 1 (strips of two), planes z0 .. z0 + nz - 1 dealt
// evenly over the nbz boxes, each column of strips split into `parts` runs of `len` planes, which
// overlap where nz is not a multiple of len.
struct FxRegGeom {
    int y0, ny, z0, nz, ns, cols, parts, len;
};
FX_HOST_DEVICE FxRegGeom fx_reg_geom(int X, int Y, int Z, const FxResBox& bx, int b) {
    FxRegGeom g;
    const int iy = b % bx.nby, iz = b / bx.nby;
    g.y0 = iy * bx.by;
    g.ny = Y - g.y0 < bx.by ? Y - g.y0 : bx.by;
    g.z0 = (int)((long long)iz * Z / bx.nbz);
    g.nz = (int)((long long)(iz + 1) * Z / bx.nbz) - g.z0;
    g.ns = g.ny / 2;
    g.cols = (X / 4) * g.ns;
    const int most = FX_REG_THREADS / (g.cols > 0 ? g.cols : 1);
    g.len = most > 0 ? (g.nz + most - 1) / most : g.nz;
    g.parts = (g.nz + g.len - 1) / g.len;
    return g;
}
// Shared memory: the box's pressure with a halo row or plane on each side, and each thread's
// divergence.
FX_HOST_DEVICE int fx_reg_pressure_floats(int X, const FxRegGeom& g) { return (g.nz + 2) * (g.ny + 2) * X; }
FX_HOST_DEVICE long long fx_reg_smem_bytes(int X, const FxRegGeom& g) {
    return 4LL * fx_reg_pressure_floats(X, g) + 32LL * g.len * FX_REG_THREADS;
}
// Quads a box sends per sweep: sections y low, y high (bz rows), z low, z high (by rows).
FX_HOST_DEVICE int fx_reg_outbox_quads(int X, const FxResBox& bx) { return 2 * (bx.by + bx.bz) * (X / 4); }
// Exchange buffer of a launch: a head whose first word is the tag its packets start from in this step,
// then each member's packets of 16 bytes, four for a quad that a box sends (two slots of two).
#define FX_REG_EXCHANGE_HEAD 128
inline size_t fx_reg_packets(int X, const FxResBox& bx) { return (size_t)bx.nby * bx.nbz * 4 * fx_reg_outbox_quads(X, bx); }
// ... and the most that a launch of `cap` CTAs takes: a box sends no more than it may receive.
inline size_t fx_reg_exchange_most(int cap) {
    return FX_REG_EXCHANGE_HEAD + (size_t)cap * 4 * FX_REG_MAXH * FX_REG_THREADS * 16;
}

// ---- division by a constant in two operations (fx_div_two, fx_step_math.cuh) ------------------------
// The reciprocal 1/d = rh + rl, rh rounded down so that rl > 0 (zeros keep their signs, infinities and
// NaN pass), with rl rounded to nearest or one or two steps beside it: that rounding decides the few
// quotients next to a midpoint. From lo, the smallest power of two for which x rl and x / d are
// normal, a power of two on x scales both products and the quotient exactly, so one binade of x
// decides.
struct FxTwoOp {
    float rh, rl[5], lo;
};
inline FxTwoOp fx_two_op_candidates(float d) {
    FxTwoOp t;
    const double rcp = 1.0 / (double)d;
    t.rh = (float)rcp;
    if ((double)t.rh > rcp) t.rh = std::nextafter(t.rh, 0.0f);
    float rl = (float)(rcp - (double)t.rh);
    if (rl == 0.0f) rl = std::ldexp(t.rh, -60);  // a power of two: any tiny positive term rounds away
    t.rl[0] = rl;
    t.rl[1] = std::nextafter(rl, INFINITY);
    t.rl[2] = std::nextafter(rl, 0.0f);
    t.rl[3] = std::nextafter(t.rl[1], INFINITY);
    t.rl[4] = std::nextafter(t.rl[2], 0.0f);
    t.lo = std::ldexp(1.0f, std::max(-126 - std::ilogb(t.rl[4]), -125 + std::ilogb(d)));
    return t;
}

// The fixed divisors of simulate, by their slot (FxDivSlot): d and a reciprocal that is right for
// zeros, infinities, NaN and every float x of magnitude 2^-27 and above (slot 0: FX_DIV_TWO_LO).
struct FxDivTwo {
    float d, rh, rl;
};
#define FX_DIV_TWO_LO 7.888609052210118e-31f  // 2^-100
#define FX_DIV_TWO_COUNT 8
FX_HOST_DEVICE FxDivTwo fx_div_two_of(int slot) {
    switch (slot) {
        case 0: return {6.0f, 0x1.555554p-3f, 0x1.555556p-27f};                    // DIVC_SIX
        case 1: return {0.78f - 0.30f, 0x1.0aaaacp+1f, 0x1.238e4ap-26f};           // DIVC_FUELCORE
        case 2: return {1500.0f - 400.0f, 0x1.dca01cp-11f, 0x1.ca01dcp-35f};       // DIVC_ENTRAIN_T
        case 3: return {930.0f - 690.0f, 0x1.11111p-8f, 0x1.111112p-32f};          // DIVC_IGNITION
        case 4: return {1650.0f - 520.0f, 0x1.cff8cp-11f, 0x1.cff8cp-39f};         // DIVC_HOTPLUME
        case 5: return {1040.0f - 335.0f, 0x1.73d5ep-10f, 0x1.8b133ep-35f};        // DIVC_EVAP
        case 6: return {0.48f - (-0.42f), 0x1.1c71c6p+0f, 0x1.9add3cp-24f};        // DIVC_LOBE
        default: return {1500.0f, 0x1.5d867cp-11f, 0x1.f67152p-38f};               // DIVC_BUOYANCY
    }
}

// ---- plans (host) ---------------------------------------------------------------------------------
// Cells of these grids over the cells of the strip tiles that cover them: 1 where 32 x 14 tiles fit.
inline double fx_zs_fill(const std::vector<std::array<int, 3>>& dims) {
    double cells = 0, tiled = 0;
    for (const auto& d : dims) {
        cells += (double)d[0] * d[1] * d[2];
        tiled += (double)fx_zs_bricks(d[0], d[1], 1, 1, FX_ZS_TXG) * (4 * FX_ZS_TXG) * (FX_ZS_ROWS * (FX_ZS_THREADS / FX_ZS_TXG) - 2) * d[2];
    }
    return tiled > 0 ? cells / tiled : 1.0;
}

// Jacobi kernel when the caller did not choose one (measured on B200, 96+96 sweeps): below 2 Mi
// cells per batch the unblocked kernel; from there two sweeps per pass by z-marching strips
// (160x240x160: 2.14 ms of Jacobi per step against 3.95 unblocked; 508^3: 31.6 against 56.5
// for one sweep per pass; near the line, 128x128x132, 6.6 us a sweep against 10.3, with FP16 pressure
// 7.3 against 10.3), in chunks fitted to the device (fx_zs_run; zc, 16 or 64 by size, is what
// firex_diagnostics.jacobi_zchunk reports). fire_b200/autotune.py refines this per workload.
// Narrow and flat grids leave the tiles empty: below a fill of 0.42 the unblocked kernel is the faster
// at any size (us per sweep, strips and unblocked: 4x1024x1024, fill 0.12, 37.9 and 14.8;
// 8x512x1024, 0.25, 21.6 and 15.1; 200 grids of 36x16x36, 0.32, 30.4 and 21.7; 128 of 36x44x28, 0.44,
// 24.5 and 27.9; 16x512x512, 0.49, 13.3 and 15.1). FP16 pressure gains less from strips while it
// stays in L2: below 8 Mi cells the line is at 0.50 (60 grids of 36x60x36, 0.48, 23.6 and 21.6;
// 16x512x512, 0.49, 15.3 and 15.0; 256 of 20x48x24, 0.54, 20.4 and 28.3; 48 of 40x60x40, 0.54, 19.4 and
// 21.0; 36x400x300, 0.55, 16.2 and 15.9; 512x8x1024, 0.57, 13.5 and 14.4).
inline void fx_default_jacobi(long long cells, double fill, bool half, int* kernel, int* k, int* zc) {
    const bool fused = cells >= (2LL << 20) && fill >= (half && cells < (8LL << 20) ? 0.50 : 0.42);
    *kernel = fused ? FIREX_JACOBI_FUSED : FIREX_JACOBI_UNBLOCKED;
    *k = fused ? 2 : 1;
    *zc = cells >= (16LL << 20) ? 64 : 16;
}

// Whether AUTO stages the strips' planes by tensor loads (FP32 pressure): they cost a warp next to nothing
// (160x240x160: 2.14 against 2.56 ms of Jacobi per step with cp.async, 508^3: 31.6 against 34.8). Not for
// several grids one tile across (17 to 32 cells), whose tiles have nothing beside them to skip and
// start with two new tensor maps every few planes (us per sweep, tensor loads and cp.async: 60, 130
// and 200 grids of 32x48x32 10.4 / 9.4, 23.7 / 15.5 and 32.4 / 27.8, 150 of 28x48x32 23.2 / 19.5; on the
// other side 150 of 36x48x32 38.8 / 42.9, 500 of 16x24x16 16.6 / 17.7, 32x512x256 alone 8.4 / 9.4).
inline bool fx_zs_auto_tma(const std::vector<std::array<int, 3>>& dims) {
    double cells = 0, oneTile = 0;
    for (const auto& d : dims) {
        const double n = (double)d[0] * d[1] * d[2];
        cells += n;
        if (d[0] > 2 * FX_ZS_TXG && d[0] <= 4 * FX_ZS_TXG) oneTile += n;
    }
    return dims.size() < 2 || oneTile <= 0.5 * cells;
}

// z planes per CTA of the two-sweep pass when the caller did not ask for a number: the chunk
// length that takes the fewest plane steps, counting a chunk's own planes, the one beside it
// at each end and the time its first planes take to arrive (about two steps more), over the
// waves that its bricks make of the `slots` CTAs the device holds at once.
inline int fx_zs_run(const std::vector<std::array<int, 3>>& dims, bool half, int slots) {
    int best = 16, maxZ = 0;
    double least = 0;
    for (const auto& d : dims) maxZ = std::max(maxZ, d[2]);
    // FP16 rows do not gain from long chunks (412x616x412 10.3 ms at 52 planes, 10.8 at 206; 640x400x320 8.5
    // at 54, 9.4 at 206); of eight grids from 10 to 131 M cells the chunk taken so is within 4 % of the
    // best of eleven
    if (half) maxZ = std::min(maxZ, 64);
    for (int zc = std::min(4, maxZ); zc <= maxZ; ++zc) {
        long long bricks = 0, steps = 0;
        for (const auto& d : dims) {
            const long long n = fx_zs_bricks(d[0], d[1], d[2], zc, FX_ZS_TXG);
            const int chunks = (d[2] + zc - 1) / zc;
            bricks += n;
            steps += n / chunks * (d[2] + 4LL * chunks);
        }
        const double waves = (double)((bricks + slots - 1) / slots);
        // uneven members fill a wave's end with short chunks: never below the mean load
        const double cost = std::max(std::min(waves * (zc + 4.0), steps / (double)slots + zc + 4.0), steps / (double)slots);
        if (least == 0 || cost < least * 0.999) {
            least = cost;
            best = zc;
        }
    }
    return best;
}

// Box decomposition of an X x Y x Z grid over at most m CTAs for the resident Jacobi
// (boxes of by x bz full x rows; G = by * bz * X / 4 groups of 4 cells per box). Cost per
// sweep: the groups a thread computes plus the halo traffic per thread (faces written and
// halo rows read, 2 (by + bz) rows of X / 4 groups, both ways).
//   variants 1, 2 (faces-first): face groups and interior groups dealt out separately,
//     within FX_RES_MAXF and FX_RES_MAXI (variant 2: FX_RES_MAXI_SMALL) per thread;
//   variant 0 (columns): thread columns of (x group, row), by * X / 4 <= T, each split into
//     parts along z; at most FX_RES_MAXG planes per column part.
//   FX_RES_REGISTERS: boxes of strips of two rows, their columns split along z (fx_reg_geom), at
//     most FX_REG_MAXZ planes to a thread.
// False when no box fits one CTA's shared memory and registers.
// Shared memory of the largest box of a plan for FX_RES_REGISTERS, -1 when one does not fit. Boxes
// differ only in their rows (the last of a row of boxes may have fewer) and by one plane (the
// first along z has the fewest, the last the most).
inline long long fx_reg_smem(int X, int Y, int Z, const FxResBox& bx) {
    long long most = 0;
    for (int iz : {0, bx.nbz - 1})
        for (int iy : {0, bx.nby - 1}) {
            const FxRegGeom g = fx_reg_geom(X, Y, Z, bx, iz * bx.nby + iy);
            if (g.cols > FX_REG_THREADS || g.len > FX_REG_MAXZ || g.cols * g.parts > FX_REG_THREADS) return -1;
            if (2 * (g.ny + g.nz) * (X / 4) > FX_REG_MAXH * FX_REG_THREADS) return -1;
            most = std::max(most, fx_reg_smem_bytes(X, g));
        }
    return most;
}
inline bool fx_reg_box(int X, int Y, int Z, int m, FxResBox* out) {
    bool found = false;
    double best = 0;
    for (int by = 2; by <= Y; by += 2) {
        const int nby = (Y + by - 1) / by;
        if (nby > m || nby > FX_RES_MAX_CTAS) continue;
        if ((X / 4) * (by / 2) > FX_REG_THREADS) break;
        const int nbz = std::min(Z, std::min(m, FX_RES_MAX_CTAS) / nby);
        FxResBox bx{by, (Z + nbz - 1) / nbz, nby, nbz, 0, {0, 0, 0}};
        const long long smem = fx_reg_smem(X, Y, Z, bx);
        if (smem < 0 || smem > FX_RES_SMEM_MAX) continue;
        const FxRegGeom g = fx_reg_geom(X, Y, Z, bx, (nbz - 1) * nby);
        // cycles of a sweep, roughly: the warps' issue slots or one warp's chain, and the faces. An estimate
        // that orders plans; fx_reg_crowded has its one miss among the 81 grids measured.
        const double warps = (g.cols * g.parts + 31) / 32;
        const double cost = std::max(warps * g.len * 2 * 25.0, g.len * 2 * 100.0) + 2.0 * (by + bx.bz) * (X / 4) / FX_REG_THREADS * 100.0;
        if (!found || cost < best) {
            found = true;
            best = cost;
            *out = bx;
        }
    }
    return found;
}
// Whether the copy warp is the faster for a plan of the register kernel: rows of 244 cells and more, which
// it brings with few copies, in boxes at the registers' limit (us per sweep, registers and copy warp:
// 256x64x64 4.41 and 4.02, 252x80x44 4.34 and 4.14; of the 78 other grids measured none, nearest
// 240x96x48 3.98 and 4.25, 200x80x72 4.08 and 4.31, 256x64x48 3.79 and 3.91).
inline bool fx_reg_crowded(int X, const FxResBox& bx) { return X >= 244 && (long long)X * bx.by * bx.bz >= 7800; }

// The fewest CTAs, up to cap, whose boxes hold the grid (0: none).
inline int fx_reg_min_ctas(int X, int Y, int Z, int cap) {
    FxResBox bx;
    if (!fx_reg_box(X, Y, Z, cap, &bx)) return 0;
    int lo = 1, hi = cap;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (fx_reg_box(X, Y, Z, mid, &bx)) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}
constexpr int FX_RES_REGISTERS = 5;  // variant 4 with the pressure in registers
inline bool fx_res_box(int X, int Y, int Z, int m, int variant, FxResBox* out) {
    if (variant == FX_RES_REGISTERS) return fx_reg_box(X, Y, Z, m, out);
    const long long gx = X / 4;
    bool found = false;
    double best = 0;
    for (int by = 1; by <= Y && by <= 2047; ++by) {
        const int nby = (Y + by - 1) / by;
        if (nby > m || nby > FX_RES_MAX_CTAS) continue;
        const int maxNbz = m / nby;
        const int bz = (Z + maxNbz - 1) / maxNbz;
        if (bz > 1023) continue;
        if (fx_res_smem_bytes(X, by, bz) > FX_RES_SMEM_MAX) continue;
        const long long G = (long long)by * bz * gx;
        double work;
        if (variant == 3 || variant == 4) {
            // faces dealt out; interior columns (rows off the y faces x groups) one per
            // thread, split along z when there are fewer columns than threads (variant 4:
            // the threads but the copy warp)
            const long long T = variant == 4 ? FX_RES_COPY_TC : FX_RES_THREADS;
            if (2LL * (by + bz) * gx > (long long)FX_RES_MAXF * T) continue;
            // the most interior rows and planes a box can have: a box with a neighbour on
            // one side only keeps all but one row (plane) off its faces
            const int nbzHere = (Z + bz - 1) / bz;
            const long long rowsI = nby == 1 ? by : by - 1, planesI = nbzHere == 1 ? bz : bz - 1;
            const long long Cmax = rowsI * gx;
            if (Cmax > T) continue;
            const long long parts = std::max(1LL, T / std::max(1LL, Cmax));
            const long long zlen = (planesI + parts - 1) / parts;
            if (zlen > FX_RES_MAXZ) continue;
            if (zlen < 4) continue;  // short columns: the faces-first variants do better (measured)
            const long long F = 2LL * (by + bz) * gx;
            work = (double)zlen + (double)((F + T - 1) / T);
        } else if (variant != 0) {
            // faces (at most 2 (by + bz) rows of groups) and interior dealt out separately
            const int maxi = variant == 2 ? FX_RES_MAXI_SMALL : FX_RES_MAXI;
            if (2LL * (by + bz) * gx > (long long)FX_RES_MAXF * FX_RES_THREADS) continue;
            if (G > (long long)maxi * FX_RES_THREADS) continue;
            work = (double)((G + FX_RES_THREADS - 1) / FX_RES_THREADS);
        } else {
            if (by * gx > FX_RES_THREADS) continue;
            const int parts = (int)(FX_RES_THREADS / (by * gx));
            const int zlen = (bz + parts - 1) / parts;
            if (zlen > FX_RES_MAXG) continue;
            work = zlen;
        }
        const double cost = work + 4.0 * (by + bz) * gx / FX_RES_THREADS;
        if (!found || cost < best) {
            found = true;
            best = cost;
            *out = FxResBox{by, bz, nby, (Z + bz - 1) / bz, 0, {0, 0, 0}};
        }
    }
    return found;
}

// CTAs for every simulation of a batch within `cap` (one launch of one variant): each gets
// at least the fewest CTAs its grid fits in, the rest in proportion to cells. False when
// the batch does not fit.
inline bool fx_res_assign(const std::vector<std::array<int, 3>>& dims, int cap, int variant, std::vector<FxResBox>* boxes,
                          int* smem) {
    const size_t n = dims.size();
    if (n == 0 || cap <= 0) return false;
    std::vector<int> mins(n), t(n);
    long long sumMin = 0;
    double cells = 0;
    FxResBox tmp;
    for (size_t i = 0; i < n; ++i) {
        const auto& d = dims[i];
        if (!fx_res_box(d[0], d[1], d[2], cap, variant, &tmp)) return false;
        int lo = 1, hi = cap;
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (fx_res_box(d[0], d[1], d[2], mid, variant, &tmp)) hi = mid;
            else lo = mid + 1;
        }
        mins[i] = lo;
        sumMin += lo;
        cells += (double)d[0] * d[1] * d[2];
    }
    if (sumMin > cap) return false;
    long long sum = 0;
    for (size_t i = 0; i < n; ++i) {
        const double share = (double)dims[i][0] * dims[i][1] * dims[i][2] / cells;
        t[i] = std::max(mins[i], (int)std::floor(share * cap));
        sum += t[i];
    }
    while (sum > cap) {  // give back CTAs from the member with the most to spare
        size_t j = 0;
        for (size_t i = 1; i < n; ++i)
            if (t[i] - mins[i] > t[j] - mins[j]) j = i;
        --t[j];
        --sum;
    }
    boxes->resize(n);
    *smem = 0;
    for (size_t i = 0; i < n; ++i) {
        fx_res_box(dims[i][0], dims[i][1], dims[i][2], t[i], variant, &(*boxes)[i]);
        *smem = std::max(*smem, (int)(variant == FX_RES_REGISTERS ? fx_reg_smem(dims[i][0], dims[i][1], dims[i][2], (*boxes)[i])
                                                        : fx_res_smem_bytes(dims[i][0], (*boxes)[i].by, (*boxes)[i].bz)));
    }
    return true;
}
