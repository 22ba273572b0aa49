// fx_jacobi_reg.cuh — every sweep of one Jacobi phase (solvePressureGlobal, shaders.ts:375-403) in
// one cooperative launch with the pressure in registers: variant 4 of the resident Jacobi (FP32)
// for boxes of short columns; fx_jacobi_res.cuh holds its copy-warp form for long ones.
//
// Each simulation gets a group of CTAs, CTA b a box of full x rows. A thread owns a run of up to
// FX_REG_MAXZ planes of a strip of two rows of 4 cells and keeps its pressure in registers for the
// whole phase; shared memory holds a copy of the box with a halo row or plane on each side, from
// which a thread reads only what it does not own (one row above, one below, the planes at its
// run's ends), and the divergence. A sweep: every thread computes its new values; face cells leave as
// packets; after a barrier the copy is rewritten and the neighbours' faces are received into the
// halo; a second barrier ends the sweep.
//
// The faces' round trip is what bounds small grids, so it is one store and one load: packets carry
// the sweep's tag in every 64-bit word (relaxed accesses, no fence, no flag; a word is one access, so
// the tag vouches for the value beside it). Two packet slots alternate: a box overwrites a slot two
// sweeps later, after it has received its neighbours' faces of the sweep in between, which they
// send only after they have received the slot. Tags start anew each step and phase from the batch's
// running count (fxk_step_end), so no earlier packet matches. Waits are bounded like those of
// fx_jacobi_res.cuh: on expiry the CTA sets the simulation's error word and returns, its
// neighbours' waits expire in turn.
//
// Arithmetic, boundaries and buffer parity are those of one sweep per launch; the last two sweeps
// store every cell.
//
// Measured on B200, us per sweep against the former choice (faces first with flags and fences, or the
// copy warp): 32x48x32 1.4 (3.0), 64x96x64 1.84 (3.4), 80x120x80 2.5 (3.6), 96x144x96 3.4 (4.2),
// 100x148x92 3.7 (4.75). From columns of five planes on the copy warp is the faster (128x192x128 5.6
// against 9.7 with six planes to a thread, whose registers spill). 12 warps at 168 registers: 16 at
// 128 measured 3.6 at 96x144x96, 8 at 224 4.4.
#pragma once

#include "fx_async.cuh"
#include "fx_jacobi_res.cuh"
#include "fx_step_math.cuh"
#include "fx_storage.cuh"

// Faces travel as packets of {value, tag} in 64-bit words, stored and loaded relaxed: a word is
// one access, so a receiver that sees the sweep's tag has the sweep's value, and needs no flag,
// fence or second round trip.
FXD void fx_ll_store(ulonglong2* p, const FxQuad& v, unsigned tag) {
    auto word = [&](float x) { return ((unsigned long long)tag << 32) | __float_as_uint(x); };
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(word(v.a.x)), "l"(word(v.a.y)) : "memory");
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p + 1), "l"(word(v.b.x)), "l"(word(v.b.y)) : "memory");
}
FXD ulonglong2 fx_ll_load(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
FXD FxQuad fx_reg_ld(const float* p) { return fx_quad(*reinterpret_cast<const float4*>(p)); }
FXD float4 fx_reg_f4(const FxQuad& q) { return make_float4(q.a.x, q.a.y, q.b.x, q.b.y); }
FXD void fx_reg_st(float* p, const FxQuad& q) { *reinterpret_cast<float4*>(p) = fx_reg_f4(q); }

template <int NZ, bool EPI, bool TWO>
FXD void fx_reg_box(const FxSimDev& S, const FxBatchDev* __restrict__ B, const FxResBox& bx, const FxRegGeom& g, int b, int phase,
                    float* sm) {
    const int n = phase == 0 ? S.P : S.R;
    const int X = S.X, Y = S.Y, Z = S.Z, gx = X >> 2, t = threadIdx.x, lane = t & 31;
    const int XY = X * Y;
    const bool loY = g.y0 > 0, hiY = g.y0 + g.ny < Y, loZ = g.z0 > 0, hiZ = g.z0 + g.nz < Z;  // neighbour boxes
    // ---- this thread's column part: strip `strip` of two rows, quad q, planes zs .. zs + NZ - 1 of
    // the box. Threads past the last part repeat it without storing anything.
    const int idx = t % g.cols, slotPart = t / g.cols;
    const bool active = slotPart < g.parts;
    const bool warpOn = (t & ~31) < g.cols * g.parts;
    const int part = active ? slotPart : g.parts - 1, strip = idx / gx, q = idx - strip * gx;
    auto start = [&](int r) { return g.parts > 1 ? r * (g.nz - NZ) / (g.parts - 1) : 0; };
    const int zs = start(part);
    // planes before kOwn are also the part before's, which stores them
    const int kOwn = !active ? NZ : part > 0 ? start(part - 1) + NZ - zs : 0;
    // ---- the box in shared memory: cell (x, row ly, plane lz) of it at ((lz + 1) (ny + 2) + ly + 1) X + x
    const int rows = g.ny + 2, plane = rows * X;
    float* const own = sm + ((zs + 1) * rows + 2 * strip + 1) * X + 4 * q;       // its first cell
    float* const sd = sm + fx_reg_pressure_floats(X, g) + 4 * t;  // its divergence, quads 4 FX_REG_THREADS apart
    const bool top = g.y0 + 2 * strip + 2 == Y;                   // its second row is the open top
    // neighbours that the clamped addressing maps onto the cell itself are read from the cell
    const float* const up = strip == 0 && !loY ? own : own - X;
    const float* const down = top ? own + X : own + 2 * X;
    const float* const behind = zs == 0 && !loZ ? own : own - plane;
    const float* const ahead = zs + NZ == g.nz && !hiZ ? own + (NZ - 1) * plane : own + NZ * plane;
    const bool wallL = q == 0, wallR = q == gx - 1;
    const bool edgeL = lane == 0 && !wallL, edgeR = lane == 31 && !wallR;  // x neighbours in another warp
    const FxJacobiK<TWO> K = fx_jacobi_k<TWO>(S);
    const float lo1 = top ? -1.0f : K.lo;  // the open top row's numerators are not used
    const int gOwn = (g.z0 + zs) * XY + (g.y0 + 2 * strip) * X + 4 * q;

    // ---- packets to and from the neighbour boxes
    const int outQuads = fx_reg_outbox_quads(X, bx);
    ulonglong2* const ex = reinterpret_cast<ulonglong2*>(B->ex + 32) + bx.exOff;
    const unsigned tag0 = B->ex[0] + (phase ? (unsigned)B->exPhase : 0u) + 1u;
    const unsigned limit = S.sync[FX_SYNC_SPIN] ? S.sync[FX_SYNC_SPIN] : FX_RES_SPIN_LIMIT;
    const int holdFrom = S.sync[FX_SYNC_HOLD_BOX] == (unsigned)b + 1u ? (int)S.sync[FX_SYNC_HOLD_SWEEP] : 0x7fffffff;
    const int secYhi = bx.bz * gx, secZlo = 2 * bx.bz * gx, secZhi = secZlo + bx.by * gx;
    const bool faceYlo = strip == 0 && loY && active, faceYhi = strip == g.ns - 1 && hiY && active;
    const bool faceZlo = zs == 0 && loZ && active, faceZhi = zs + NZ == g.nz && hiZ && active;
    const bool face = faceYlo || faceYhi || faceZlo || faceZhi;
    // this thread's share of the halo: quads t, t + T, ... of the four sides
    int from[FX_REG_MAXH], to[FX_REG_MAXH];  // packet pair of sweep parity 0, float offset in sm; -1: none
    {
        const int ny1 = loY ? g.nz * gx : 0, ny2 = ny1 + (hiY ? g.nz * gx : 0), nz1 = ny2 + (loZ ? g.ny * gx : 0);
        const int all = nz1 + (hiZ ? g.ny * gx : 0);
#pragma unroll
        for (int i = 0; i < FX_REG_MAXH; ++i) {
            const int h = t + i * FX_REG_THREADS;
            int box = 0, sec = 0, j = 0, at = 0;
            if (h < ny2) {  // rows of the boxes beside in y: their plane j / gx
                j = h < ny1 ? h : h - ny1;
                box = h < ny1 ? b - 1 : b + 1;
                sec = h < ny1 ? secYhi : 0;
                at = ((j / gx + 1) * rows + (h < ny1 ? 0 : g.ny + 1)) * X;
            } else {  // planes of the boxes beside in z: their row j / gx
                j = h < nz1 ? h - ny2 : h - nz1;
                box = h < nz1 ? b - bx.nby : b + bx.nby;
                sec = h < nz1 ? secZhi : secZlo;
                at = ((h < nz1 ? 0 : g.nz + 1) * rows + j / gx + 1) * X;
            }
            from[i] = h < all ? 2 * (2 * box * outQuads + sec + j) : -1;
            to[i] = at + 4 * (j % gx);
        }
    }

    FxQuad p[NZ][2];
    // x neighbours of p[k][i] (old values)
    auto sides = [&](int k, int i, float& l, float& h) {
        l = __shfl_up_sync(0xffffffffu, p[k][i].b.y, 1);
        h = __shfl_down_sync(0xffffffffu, p[k][i].a.x, 1);
        const float* c = own + k * plane + i * X;
        if (edgeL) l = c[-1];
        if (edgeR) h = c[4];
        l = wallL ? p[k][i].a.x : l;
        h = wallR ? p[k][i].b.y : h;
    };

    // ---- first load: the box with its halo, and this thread's column and divergence
    {
        const FxSolveBufs b0 = fx_solve_bufs(S, phase, 0);
        const float* pin = reinterpret_cast<const float*>(b0.pin);
        for (int i = t; i < (g.nz + 2) * rows * gx; i += FX_REG_THREADS) {
            const int row = i / gx, x = 4 * (i - row * gx), lz = row / rows - 1, ly = row - (lz + 1) * rows - 1;
            const int y = g.y0 + ly, z = g.z0 + lz;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (!b0.zeroIn && y >= 0 && y < Y && z >= 0 && z < Z) v = __ldg(reinterpret_cast<const float4*>(pin + z * XY + y * X + x));
            *reinterpret_cast<float4*>(sm + row * X + x) = v;
        }
#pragma unroll
        for (int k = 0; k < NZ; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                *reinterpret_cast<float4*>(sd + (2 * k + i) * 4 * FX_REG_THREADS) =
                    __ldg(reinterpret_cast<const float4*>(S.div + gOwn + k * XY + i * X));
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NZ; ++k)
#pragma unroll
            for (int i = 0; i < 2; ++i) p[k][i] = fx_reg_ld(own + k * plane + i * X);
    }

    for (int s = 0; s < n; ++s) {
        const bool last = s == n - 1;
        if (warpOn) {
            FxQuad num[NZ][2], back[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) back[i] = fx_reg_ld(behind + i * X);
            // plane k's quotients replace its values once plane k + 1 has used them
            auto divide = [&](int k) {
#pragma unroll
                for (int i = 0; i < 2; ++i) p[k][i] = fx_jacobi_quotients<TWO>(K, num[k][i]);
                // numerators too small for the checked quotients: through double precision (zeros are not)
                if (__any_sync(0xffffffffu, fx_jacobi_rare<TWO>(K, K.lo, num[k][0]) || fx_jacobi_rare<TWO>(K, lo1, num[k][1]))) {
                    if (__any_sync(0xffffffffu, !TWO || fx_jacobi_tiny(K.lo, num[k][0]) || fx_jacobi_tiny(lo1, num[k][1]))) {
                        const FxJacobiK<TWO> again = fx_jacobi_k<TWO>(S);  // (its double is not kept)
                        p[k][0] = fx_jacobi_small<TWO>(again, num[k][0]);
                        p[k][1] = fx_jacobi_small<TWO>(again, num[k][1]);
                    }
                }
                if (top) p[k][1] = fx_quad_zero();
            };
#pragma unroll
            for (int k = 0; k < NZ; ++k) {
                const FxQuad u = fx_reg_ld(up + k * plane), d = fx_reg_ld(down + k * plane);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const FxQuad front = k < NZ - 1 ? p[k < NZ - 1 ? k + 1 : k][i] : fx_reg_ld(ahead + i * X);
                    float l, h;
                    sides(k, i, l, h);
                    num[k][i] = fx_jacobi_numerators<TWO>(K, l, p[k][i], h, i ? p[k][0] : u, i ? d : p[k][1],
                                                          k ? p[k ? k - 1 : 0][i] : back[i], front,
                                                          fx_reg_ld(sd + (2 * k + i) * 4 * FX_REG_THREADS));
                }
                if (k) divide(k ? k - 1 : 0);
            }
            divide(NZ - 1);
            if (face && (!last || EPI) && s < holdFrom) {
                ulonglong2* out = ex + 2 * ((size_t)(2 * b + (s & 1)) * outQuads);
                const unsigned tag = tag0 + s;
                const int oY = zs * gx + q, oZ = 2 * strip * gx + q;  // its quads within a section
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (faceZlo) fx_ll_store(out + 2 * (secZlo + oZ + i * gx), p[0][i], tag);
                    if (faceZhi) fx_ll_store(out + 2 * (secZhi + oZ + i * gx), p[NZ - 1][i], tag);
                }
#pragma unroll
                for (int k = 0; k < NZ; ++k)
                    if (k >= kOwn) {
                        if (faceYlo) fx_ll_store(out + 2 * (oY + k * gx), p[k][0], tag);
                        if (faceYhi) fx_ll_store(out + 2 * (secYhi + oY + k * gx), p[k][1], tag);
                    }
            }
            if (s >= n - 2) {  // the last two sweeps fill both buffers of the pair
                float* pout = reinterpret_cast<float*>(fx_solve_bufs(S, phase, s).pout) + gOwn;
#pragma unroll
                for (int k = 0; k < NZ; ++k)
                    if (k >= kOwn) {
                        *reinterpret_cast<float4*>(pout + k * XY) = fx_reg_f4(p[k][0]);
                        *reinterpret_cast<float4*>(pout + k * XY + X) = fx_reg_f4(p[k][1]);
                    }
            }
        }
        if (last && !EPI) break;
        __syncthreads();  // every read of the old values is done
#pragma unroll
        for (int k = 0; k < NZ; ++k)
            if (k >= kOwn) {
                fx_reg_st(own + k * plane, p[k][0]);
                fx_reg_st(own + k * plane + X, p[k][1]);
            }
        bool ok = true;
        {
            const ulonglong2* in = ex + 2 * ((size_t)(s & 1) * outQuads);
            const unsigned tag = tag0 + s;
            ulonglong2 v[FX_REG_MAXH][2];
            for (unsigned spins = 0;; ++spins) {
                bool here = true;
#pragma unroll
                for (int i = 0; i < FX_REG_MAXH; ++i) {
                    if (from[i] >= 0) {
                        v[i][0] = fx_ll_load(in + from[i]);
                        v[i][1] = fx_ll_load(in + from[i] + 1);
                    }
                }
#pragma unroll
                for (int i = 0; i < FX_REG_MAXH; ++i)
                    if (from[i] >= 0)
                        here = here && (unsigned)(v[i][0].x >> 32) == tag && (unsigned)(v[i][0].y >> 32) == tag &&
                               (unsigned)(v[i][1].x >> 32) == tag && (unsigned)(v[i][1].y >> 32) == tag;
                if (here) break;
                if (spins > limit) {
                    ok = false;
                    break;
                }
                if (spins > 64) __nanosleep(32);
            }
#pragma unroll
            for (int i = 0; i < FX_REG_MAXH; ++i)
                if (from[i] >= 0)
                    *reinterpret_cast<float4*>(sm + to[i]) =
                        make_float4(__uint_as_float((unsigned)v[i][0].x), __uint_as_float((unsigned)v[i][0].y),
                                    __uint_as_float((unsigned)v[i][1].x), __uint_as_float((unsigned)v[i][1].y));
        }
        if (fx_bar_or(0, FX_REG_THREADS, !ok)) {  // a bounded wait ran out: every thread leaves
            if (t == 0) atomicExch(S.sync + 2, 1u);
            return;
        }
    }
    if constexpr (EPI) {
        // projectVelocity with the correction (fxk_project phase 1, with its operations): the last
        // barrier left the final values and the neighbours' in shared memory, quads dealt over the
        // threads so that a warp's flow records are contiguous
        const float4* __restrict__ flowIn = reinterpret_cast<const float4*>(S.flow[S.fi]);
        float4* __restrict__ flowOut = reinterpret_cast<float4*>(S.flow[S.fi ^ 1]);
        const float3 m = fx_metric(S.prm.u);
        for (int i = t; i < g.nz * g.ny * X; i += FX_REG_THREADS) {
            const int row = i / X, x = i - row * X, lz = row / g.ny, ly = row - lz * g.ny;
            const int y = g.y0 + ly, z = g.z0 + lz, c = z * XY + y * X + x;
            const int cs = y == Y - 1 ? c - X : c;  // top row: the projected row below
            const float4 f = __ldg(flowIn + c), sv = cs == c ? f : __ldg(flowIn + cs);
            const float* pr = sm + ((lz + 1) * rows + (y == Y - 1 ? ly : ly + 1)) * X + x;
            const float pc = *pr, px = x + 1 < X ? pr[1] : pc, pt = pr[X], pf = z < Z - 1 ? pr[plane] : pc;
            float4 o = make_float4(sv.x - (px - pc) * m.x, sv.y - (pt - pc) * m.y, sv.z - (pf - pc) * m.z, f.w);
            if (x == 0 || x == X - 1) o.x = 0.0f;
            if (z == 0 || z == Z - 1) o.z = 0.0f;
            if (y == 0) o.y = 0.0f;
            if (y == Y - 1) o.y = fx_max(0.0f, o.y);
            flowOut[c] = o;
        }
    }
}
