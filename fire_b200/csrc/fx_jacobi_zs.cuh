// fx_jacobi_zs.cuh — two Jacobi sweeps (solvePressureGlobal, shaders.ts:375-403) per pass over
// memory, by z-marching strips with the z neighbours in registers.
//
// A CTA of two warps owns an x-y tile of 32 columns and 14 rows and a chunk of z planes. Each
// thread takes a strip of two rows of 4 cells of the tile or of its one-row ring (16 rows) and
// keeps, for its own cells, the input planes z - 1, z, z + 1 and the sweep-1 planes z - 2, z - 1, z
// in registers (register sets that rotate through a three-fold unrolled step): of a cell's six
// neighbours the two in z and one in y never touch shared memory. What other threads need does:
// input and divergence planes stream through 3-slot rings (step z requests input plane z + 2 and
// divergence plane z + 1), sweep-1 planes through another. At step z a thread computes sweep 1 on
// plane z, publishes it, and sweep 2 on plane z - 1, whose x and y neighbours were published at
// step z - 1 and whose plane in front it has just computed: one barrier per step. The ring's two
// columns are kept cell by cell, one on a thread.
//
// The planes are brought by tensor loads that one thread issues (TMA) or by cp.async, one 4-cell
// segment to a thread and turn. Waits on the tensor loads are bounded; a tile whose wait runs out waits
// once more, so that its loads have landed before the CTA ends, and reports it.
//
// The update is fx_jacobi_numerators and the two-operation quotient: each sweep computes the single
// sweep's FP32 operations, rounds to FP16 as a stored sweep where the pressure is stored so, and
// writes 0 on the open top row, so two fused sweeps equal two single ones bit for bit. Boundaries
// follow the reference's clamped addressing: planes and rows outside the grid are reflected into
// it; at the side walls a lane reads its own cell.
//
// Measured on B200: bound by the latency of a step at 16 warps per SM (issue slots 44 % busy,
// shared memory 64 %) and, at 508^3, by the power cap; 508^3 31.4 ms of Jacobi per step of 96 + 96
// sweeps against 45.2 for the former 32 x 30 tiles of one row to a thread, whose every neighbour
// came from shared memory (39 instructions per cell and sweep; 20 here); 160x240x160 2.14 ms
// against 3.95 for single sweeps from L2. Small CTAs because the step barrier is what the warps
// wait for: 508^3 with cp.async 36.0 ms with 8 warps and 64 columns, 33.5 with 4, 35.3 with 2 and 32
// columns; twelve uneven grids 17.2, 14.8 and 13.8. One row to a thread at 80 registers and 24
// warps per SM: 40.0 ms. Row by row bulk copies: 39.9.
#pragma once

#include "fx_async.cuh"
#include "fx_jacobi_res.cuh"  // the words of FxSimDev::sync
#include "fx_jacobi_zm.cuh"   // cp.async helpers
#include "fx_plan.h"
#include "fx_step_math.cuh"
#include "fx_storage.cuh"

#define FX_ZS_MINB 8  // CTAs per SM the registers are budgeted for
#define FX_ZS_SLOTS 3
#define FX_ZS_WAIT_LIMIT (1u << 22)  // polls of a step's copies

template <int TXG>
struct FxZsShape {
    static constexpr int ROWS = FX_ZS_ROWS;      // rows of a thread's strip
    static constexpr int RT = FX_ZS_THREADS / TXG;  // strips along y
    static constexpr int NR = ROWS * RT;         // sweep-1 rows y0 - 1 .. y0 + NR - 2
    static constexpr int TX = 4 * TXG, TY = NR - 2;
    static constexpr int SEGS = TXG + 2, COLS = 4 * SEGS;  // a 4-cell segment, the tile, a segment
    static constexpr int PROWS = NR + 2;         // input rows y0 - 2 .. y0 + NR - 1
    static constexpr int PLANE_P = PROWS * COLS, PLANE_R = NR * COLS;
    static constexpr int KP = (PROWS * SEGS + FX_ZS_THREADS - 1) / FX_ZS_THREADS;
    static constexpr int KD = (NR * SEGS + FX_ZS_THREADS - 1) / FX_ZS_THREADS;
};
template <typename PT, int TXG>
struct FxZsSmem {  // the slots of input and divergence planes start on 128-byte boundaries (tensor loads)
    using H = FxZsShape<TXG>;
    PT p[FX_ZS_SLOTS][(H::PLANE_P + 31) / 32 * 32];
    float d[FX_ZS_SLOTS][(H::PLANE_R + 31) / 32 * 32];
    float s[FX_ZS_SLOTS][H::PLANE_R];
    unsigned long long bar;  // the planes of a step have landed (tensor loads)
};

template <int I>
struct FxZsInt {
    static constexpr int value = I;
};

// Tensor maps of a simulation (FxSimDev::tmap): pressure pair, correction pair, divergence.
enum { FX_TM_P0 = 0, FX_TM_P1 = 1, FX_TM_C0 = 2, FX_TM_C1 = 3, FX_TM_DIV = 4, FX_TM_COUNT = 5 };
FXD const CUtensorMap* fx_zs_map_of(const FxSimDev& S, const void* buf) {
    return &S.tmap[buf == S.p[0] ? FX_TM_P0 : buf == S.p[1] ? FX_TM_P1 : buf == S.corr[0] ? FX_TM_C0 : FX_TM_C1];
}

FXD FxQuad fx_zs_ld(const float* p) { return fx_quad(*reinterpret_cast<const float4*>(p)); }
FXD FxQuad fx_zs_ld(const __half* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return FxQuad{__half22float2(*reinterpret_cast<const __half2*>(&v.x)), __half22float2(*reinterpret_cast<const __half2*>(&v.y))};
}
FXD float4 fx_zs_float4(const FxQuad& q) { return make_float4(q.a.x, q.a.y, q.b.x, q.b.y); }
template <bool ROUND>
FXD FxQuad fx_zs_round(FxQuad q) {
    if (ROUND)
        q = fx_quad(make_float4(PStore<__half>::round(q.a.x), PStore<__half>::round(q.a.y), PStore<__half>::round(q.b.x),
                                PStore<__half>::round(q.b.y)));
    return q;
}
FXD void fx_zs_tensor(void* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
                     fx_smem_u32(dst)),
                 "l"(map), "r"(x), "r"(y), "r"(z), "r"(fx_smem_u32(bar))
                 : "memory");
}
// Makes the tensor map at `map` (written by an earlier launch) visible to the proxy of this
// thread's tensor loads.
FXD void fx_zs_map_acquire(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(reinterpret_cast<unsigned long long>(map)) : "memory");
}
// firex_test_hold_face: whether a test holds this brick, whose first wait then counts as run out. Read while
// the first planes are on their way.
FXD bool fx_zs_held(const FxSimDev& S, int brick, int launch) {
    return S.sync[FX_SYNC_HOLD_BOX] == (unsigned)brick + 1u && (unsigned)launch >= S.sync[FX_SYNC_HOLD_SWEEP];
}
// Planes and rows outside the grid are reflected into it (fx_zs_reflect, fx_zs_input_row). The update
// adds the two neighbours of an axis, so the sweep-1 value of a reflected plane or row is that of its
// image, which is what sweep 2's clamped neighbour is: the walls need no code of their own.

// Two sweeps of planes [z0, z1) of the tile at (x0, y0): pin -> pout. TOP: the tile holds rows at
// or above the open top; brick and launch: its place for a test that holds it (fx_zs_held). False when
// a bounded wait ran out.
template <typename PT, int TXG, bool ZERO_IN, bool ROUND, bool TWO, bool TOP, bool TMA>
FXD bool fx_zs_tile(const FxSimDev& S, const PT* __restrict__ pin, PT* __restrict__ pout, int x0, int y0, int z0, int z1,
                    FxZsSmem<PT, TXG>& sm, const CUtensorMap* mapP, const CUtensorMap* mapD, unsigned& parity, int brick, int launch) {
    using H = FxZsShape<TXG>;
    constexpr int COLS = H::COLS;
    const int X = S.X, Y = S.Y, Z = S.Z, XY = X * Y, t = threadIdx.x;
    const float* __restrict__ div = S.div;
    // ---- this thread's copies of a plane: 4-cell segments in slot order (offset 4 i); segments
    // beside the grid copy its edge (no cell of the grid reads them)
    int gP[H::KP], gD[H::KD];
#pragma unroll
    for (int k = 0; k < H::KP; ++k) {
        const int i = t + k * FX_ZS_THREADS, row = i / H::SEGS, gx = min(max(x0 - 4 + 4 * (i - row * H::SEGS), 0), X - 4);
        gP[k] = fx_zs_input_row(y0 - 2 + row, Y) * X + gx;
    }
#pragma unroll
    for (int k = 0; k < H::KD; ++k) {
        const int i = t + k * FX_ZS_THREADS, row = i / H::SEGS, gx = min(max(x0 - 4 + 4 * (i - row * H::SEGS), 0), X - 4);
        gD[k] = min(max(y0 - 1 + row, 0), Y - 1) * X + gx;
    }
    const bool lastP = t + (H::KP - 1) * FX_ZS_THREADS < H::PROWS * H::SEGS;
    const bool lastD = t + (H::KD - 1) * FX_ZS_THREADS < H::NR * H::SEGS;
    constexpr unsigned BP = H::PLANE_P * 4, BD = H::PLANE_R * 4;
    auto issueP = [&](int q, int slot) {
        if (ZERO_IN) return;
        if (TMA) {
            if (t == 0) fx_zs_tensor(sm.p[slot], mapP, x0 - 4, y0 - 2, fx_zs_reflect(q, Z), &sm.bar);
            return;
        }
        const PT* src = pin + (size_t)fx_zs_reflect(q, Z) * XY;
        PT* dst = sm.p[slot] + 4 * t;
#pragma unroll
        for (int k = 0; k < H::KP; ++k)
            if (k < H::KP - 1 || lastP) fx_cp4(dst + 4 * k * FX_ZS_THREADS, src + gP[k]);
    };
    auto issueD = [&](int q, int slot) {
        if (TMA) {
            if (t == 0) fx_zs_tensor(sm.d[slot], mapD, x0 - 4, y0 - 1, fx_zs_reflect(q, Z), &sm.bar);
            return;
        }
        const float* src = div + (size_t)fx_zs_reflect(q, Z) * XY;
        float* dst = sm.d[slot] + 4 * t;
#pragma unroll
        for (int k = 0; k < H::KD; ++k)
            if (k < H::KD - 1 || lastD) fx_cp_async16(dst + 4 * k * FX_ZS_THREADS, src + gD[k]);
    };
    // nP input planes and one divergence plane complete the next phase of sm.bar
    auto expect = [&](int nP) {
        if (TMA && t == 0) fx_mbar_expect_tx(&sm.bar, (ZERO_IN ? 0 : nP) * BP + BD);
    };
    // the copies requested last have landed, for every thread; false when a bounded wait ran out
    auto landed = [&](bool requested, bool held = false) {
        if (!TMA) {
            fx_cp_wait<0>();
            __syncthreads();
            return true;
        }
        const bool late = requested && (held || !fx_mbar_wait(&sm.bar, parity, FX_ZS_WAIT_LIMIT));
        if (requested) parity ^= 1u;
        return !fx_bar_or(0, FX_ZS_THREADS, late);
    };
    const FxJacobiK<TWO> K = fx_jacobi_k<TWO>(S);
    constexpr int ROWS = H::ROWS;
    const int cg = t % TXG, j = t / TXG, x = x0 + 4 * cg, y = y0 - 1 + ROWS * j;  // the strip's first row
    const bool inX = x < X;
    // tensor loads bring zeros for the rows below the floor: the thread whose strip is the rows
    // y = -1 and 0 takes the row 0 for both, as the reflected row of the other copies is
    const bool floorTile = y0 == 0;
    // numerators of cells outside the grid or on the open top are not checked
    float lo[FX_ZS_ROWS];
    bool st[FX_ZS_ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        lo[i] = inX && (!TOP || y + i < Y - 1) ? K.lo : -1.0f;
        st[i] = inX && (i > 0 || j > 0) && (i < ROWS - 1 || j < H::RT - 1) && y + i < Y;
    }
    const bool isL = cg == 0, isR = cg == TXG - 1 || x + 4 >= X;
    const int oP = (ROWS * j + 1) * COLS + 4 + 4 * cg;  // the strip in an input slot
    const int oR = ROWS * j * COLS + 4 + 4 * cg;        // the strip in a divergence or sweep-1 slot
    const int eL = x == 0 ? 0 : -1, eR = x + 4 >= X ? 3 : 4;  // what a row's end lanes read
    const int oUp = j > 0 ? oR - COLS : oR, oDown = j < H::RT - 1 ? oR + ROWS * COLS : oR;
    auto ldp = [&](int slot, int off) { return ZERO_IN ? fx_quad_zero() : fx_zs_ld(&sm.p[slot][off]); };
    auto ends = [&](const auto* row, const FxQuad& c, float& l, float& r) {
        l = __shfl_up_sync(0xffffffffu, c.b.y, 1);
        r = __shfl_down_sync(0xffffffffu, c.a.x, 1);
        if (isL) l = (float)row[eL];
        if (isR) r = (float)row[eR];
    };
    auto divide = [&](FxQuad (&n)[FX_ZS_ROWS], FxQuad (&q)[FX_ZS_ROWS], bool stored) {
        bool rare = false;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            q[i] = fx_jacobi_quotients<TWO>(K, n[i]);
            rare = rare || fx_jacobi_rare<TWO>(K, !stored || st[i] ? lo[i] : -1.0f, n[i]);
        }
        // numerators too small for the checked quotients, which only the fronts of a spreading
        // solve have: through double precision (zeros, as everywhere in a fluid at rest, are not)
        if (__any_sync(0xffffffffu, rare)) {
            bool tiny = !TWO;
#pragma unroll
            for (int i = 0; i < ROWS; ++i) tiny = tiny || fx_jacobi_tiny(!stored || st[i] ? lo[i] : -1.0f, n[i]);
            if (__any_sync(0xffffffffu, tiny)) {
#pragma unroll
                for (int i = 0; i < ROWS; ++i) q[i] = fx_jacobi_small<TWO>(K, n[i]);
            }
        }
#pragma unroll
        for (int i = 0; i < ROWS; ++i)
            if (TOP && y + i >= Y - 1) q[i] = fx_quad_zero();
    };
    // the ring's columns x0 - 1 and x0 + TX, one cell each on 2 NR threads: of CTAs that share an
    // SM one takes them on its first warps, the other on its next ones (other schedulers)
    const int ri = t - ((blockIdx.x * 2 / gridDim.x) & 1) * 2 * H::NR, rrow = ri >> 1, rx = (ri & 1) ? x0 + H::TX : x0 - 1, ry = y0 - 1 + rrow;
    const bool ring = ri >= 0 && ri < 2 * H::NR && rx >= 0 && rx < X;
    const int ro = rrow * COLS + ((ri & 1) ? 4 + H::TX : 3), rl = rx == 0 ? 0 : -1, rr = rx == X - 1 ? 0 : 1;
    auto ld1 = [&](int slot, int off) { return ZERO_IN ? 0.0f : (float)sm.p[slot][off + COLS]; };
    float rm = 0.0f, rc = 0.0f;
    auto ringStep = [&](int cur, int next) {
        if (!ring) return;
        const float n = ld1(next, ro);
        float v = 0.0f;
        if (!TOP || ry < Y - 1) {
            v = fx_jacobi_cell<TWO>(K, ld1(cur, ro + rl), ld1(cur, ro + rr), ld1(cur, ry == 0 ? ro : ro - COLS), ld1(cur, ro + COLS), rm, n,
                                    sm.d[cur][ro]);
            if (ROUND) v = PStore<__half>::round(v);
        }
        sm.s[cur][ro] = v;
        rm = rc;
        rc = n;
    };
    const int zs = z0 - 1;  // first sweep-1 plane
    // One step: sweep 1 on plane z (slot C) from input planes m, c, n (z - 1, z, z + 1; n is read
    // here), then sweep 2 on plane z - 1 from sweep-1 planes k, s, f (z - 2, z - 1, z; f is made here)
    auto step = [&](auto slot, int z, FxQuad (&m)[FX_ZS_ROWS], FxQuad (&c)[FX_ZS_ROWS], FxQuad (&n)[FX_ZS_ROWS], FxQuad (&k)[FX_ZS_ROWS], FxQuad (&s)[FX_ZS_ROWS],
                    FxQuad (&f)[FX_ZS_ROWS]) {
        constexpr int C = decltype(slot)::value, N = (C + 1) % 3, M = (C + 2) % 3;
        if (!landed(z != zs)) return false;  // planes up to z + 1 are here; plane z - 1's input and z - 2's other slots are free
        if (z < z1) {
            expect(1);
            issueP(z + 2, M);
            issueD(z + 1, N);
            if (!TMA) fx_cp_commit();
        }
        const PT* row = &sm.p[C][oP];
        const float* dr = &sm.d[C][oR];
        FxQuad up = ldp(C, oP - COLS), down = ldp(C, oP + ROWS * COLS), q[FX_ZS_ROWS];
        float l = 0.0f, r = 0.0f;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) n[i] = ldp(N, oP + i * COLS);
        if (TMA && floorTile && j == 0) n[0] = n[1];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            if (!ZERO_IN) ends(row + i * COLS, c[i], l, r);
            q[i] = fx_jacobi_numerators<TWO>(K, l, c[i], r, i > 0 ? c[i - 1] : up, i < ROWS - 1 ? c[i + 1] : down, m[i], n[i],
                                             fx_zs_ld(dr + i * COLS));
        }
        divide(q, f, false);
        if (TMA && floorTile && j == 0) f[0] = f[1];
        float* out1 = &sm.s[C][oR];
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            f[i] = fx_zs_round<ROUND>(f[i]);
            *reinterpret_cast<float4*>(out1 + i * COLS) = fx_zs_float4(f[i]);
        }
        ringStep(C, N);
        if (z > z0) {
            const float* pl = sm.s[M];
            const float* dp = &sm.d[M][oR];
            up = fx_zs_ld(pl + oUp);
            down = fx_zs_ld(pl + oDown);
            FxQuad o[FX_ZS_ROWS];
#pragma unroll
            for (int i = 0; i < ROWS; ++i) {
                ends(pl + oR + i * COLS, s[i], l, r);
                q[i] = fx_jacobi_numerators<TWO>(K, l, s[i], r, i > 0 ? s[i - 1] : up, i < ROWS - 1 ? s[i + 1] : down, k[i], f[i],
                                                 fx_zs_ld(dp + i * COLS));
            }
            divide(q, o, true);
            PT* out = pout + (size_t)(z - 1) * XY + (y * X + x);
#pragma unroll
            for (int i = 0; i < ROWS; ++i)
                if (st[i]) PStore<PT>::st4(out, i * X, fx_zs_float4(o[i]));
        }
        return true;
    };
    // slots: plane z in slot (z - zs) mod 3, plane zs - 1 in slot 2 until step zs
    expect(3);
    issueP(zs - 1, 2);
    issueP(zs, 0);
    issueP(zs + 1, 1);
    issueD(zs, 0);
    if (!TMA) fx_cp_commit();
    bool ok = landed(true, TMA && t == 0 && fx_zs_held(S, brick, launch));
    FxQuad p0[FX_ZS_ROWS], p1[FX_ZS_ROWS], p2[FX_ZS_ROWS], s0[FX_ZS_ROWS], s1[FX_ZS_ROWS], s2[FX_ZS_ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        p0[i] = ldp(2, oP + i * COLS);
        p1[i] = ldp(0, oP + i * COLS);
        s0[i] = s1[i] = fx_quad_zero();
    }
    if (TMA && floorTile && j == 0) {
        p0[0] = p0[1];
        p1[0] = p1[1];
    }
    if (ring) {
        rm = ld1(2, ro);
        rc = ld1(0, ro);
    }
    for (int z = zs; ok && z <= z1; z += 3) {
        if (!(ok = step(FxZsInt<0>(), z, p0, p1, p2, s0, s1, s2)) || z + 1 > z1) break;
        if (!(ok = step(FxZsInt<1>(), z + 1, p1, p2, p0, s1, s2, s0)) || z + 2 > z1) break;
        ok = step(FxZsInt<2>(), z + 2, p2, p0, p1, s2, s0, s1);
    }
    if (!ok) {  // the loads of the phase whose wait ran out, the only ones in flight, land before the CTA ends
        if (TMA && t == 0) fx_mbar_wait(&sm.bar, parity ^ 1u, FX_ZS_WAIT_LIMIT);
        return false;
    }
    __syncthreads();  // the next brick's copies may refill every slot
    return true;
}
