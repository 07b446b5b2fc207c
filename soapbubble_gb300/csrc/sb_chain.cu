// The chain kernels: the map, velocity, thickness and accumulation stages of
// bubbles with FP32 storage and up to 512 rows (SbBubbleDesc::chains).  A
// cell's independent chains go to different warps of a block (its backward
// and forward trace, its two faces, its five sample points), so that a small
// grid still fills the chip and a thread holds one chain's state, and a chain
// runs in the form of sb_fastgeo.cuh (*_fast, false where it cannot serve the
// cell) or, called out of line, in the general one.
//
// The one-thread-per-cell kernels of sb_step.cu keep the other bubbles, whose results
// a last bit moves: BF16 storage rounds a value to 2^-9 of its deviation, so
// that cells at a rounding boundary jump by that much, and at 1024 rows the
// velocity beside the poles holds the solve's own error (2e-2 of u_phi,
// gamma's rounding over h sin(theta)), of which another rounding of gamma
// changes a tenth.

#define SB_SHORT_FORMS 0
#include "sb_cells.cuh"
#include "sb_fastgeo.cuh"
#include "sb_internal.h"

namespace sb {

namespace {

// Rows with neighbours on both sides.
__device__ __forceinline__ bool inner_row(const SbGrid& g, int i) { return i >= 1 && i <= g.nT - 2; }

// Backward trace of a cell: the new backward map entry and gamma, or, without
// the maps, thickness and gamma (advectionAllCentered, bubble.cu:937-961).
__device__ __noinline__ void backward_general(const SbBubbleDesc& d, int cur, int idx) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP;
    const float dt = f.step->dt;
    const Frame F = cell_frame(g, i, j);
    const Pos q0 = frame_pos(F, 0.0f, 0.0f);
    float gt, gp;
    velocity_at(g, f.uth, f.uph, q0, gt, gp);
    const Trace Tb = trace_gc(g, f.uth, f.uph, F, gt, gp, dt);
    if (d.ph.plain_adv) {
        const SStencil sb = sstencil_of(g, centred_stencil(g, pos_of(F, Tb, g), 0.0f));
        f.eta_adv[idx] = gather_s<float>(f.eta, sb, d.ph.base_eta);
        f.gam_adv[idx] = gather_s<float>(f.gam, sb, d.ph.base_gam);
    } else {
        const CStencil cb = centred_stencil(g, pos_of(F, Tb, g), 0.0f);
        const f3 db = map_at_stencil(g, f.bwd[cur], F, cb);
        f.bwd[cur ^ 1][idx] = make_float4(db.x, db.y, db.z, 0.0f);  // in the cell's own frame
        f.gam_adv[idx] = gather_s<float>(f.gam, sstencil_of(g, cb), d.ph.base_gam);
    }
}

// Forward trace (negative step): the old forward map there.
__device__ __noinline__ void forward_general(const SbBubbleDesc& d, int cur, int idx) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP;
    const Frame F = cell_frame(g, i, j);
    const Pos q0 = frame_pos(F, 0.0f, 0.0f);
    float gt, gp;
    velocity_at(g, f.uth, f.uph, q0, gt, gp);
    const Trace Tf = trace_gc(g, f.uth, f.uph, F, gt, gp, -f.step->dt);
    const f3 df = sample_map(g, f.fwd[cur], F, pos_of(F, Tf, g));
    f.fwd[cur ^ 1][idx] = make_float4(df.x, df.y, df.z, 0.0f);
}

// A cell's departure point: its stencil and the frame of the cell.
__device__ __forceinline__ bool fast_departure(const SbBubbleDesc& d, int idx, float dt, Frame& F,
                                               FStencil& s) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP;
    F = cell_frame(g, i, j);
    const float gt = 0.5f * f.uth[idx - g.nP] + 0.5f * f.uth[idx];
    const float gp = 0.5f * f.uph[idx] + 0.5f * f.uph[(i << g.logP) + ((j + 1) & g.maskP)];
    FTrace T;
    FPos q;
    bool ok = fast_trace<kAtCell, true>(g, f.uth, f.uph, i, j, F.s0, F.c0, gt, gp, dt, fast_rests(gt, gp),
                                         true, T);
    ok &= fast_pos<true>(g, F.s0, F.c0, T.d, q);
    ok &= fast_stencil(g, i, j + q.flip, q.o, g.nT - 2, s);
    return ok;
}

// The map at a departure point, as a new entry of the cell.
__device__ __forceinline__ bool fast_entry(const SbGrid& g, const float4* map, const Frame& F,
                                           const FStencil& s, float4& out) {
    float far = 0.0f;
    float4 R0;
    const f3 m = fast_map(g, map, s, __ldg(&g.rottab[g.nT + 1]), R0, far);
    const f3 e = fast_to_frame(g, F, m, R0, s.j0);
    out = make_float4(e.x, e.y, e.z, 0.0f);
    return far <= kSlerpFar;
}

// (of an inner row)
__device__ __forceinline__ bool backward_fast(const SbBubbleDesc& d, int cur, int idx) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    Frame F;
    FStencil s;
    bool ok = fast_departure(d, idx, f.step->dt, F, s);
    const float gm = fast_gather_s<float>(f.gam, s, g.nP, 0.0f);
    f.gam_adv[idx] = gm;
    if (d.ph.plain_adv) {
        const float e = fast_gather_s<float>(f.eta, s, g.nP, 0.0f);
        f.eta_adv[idx] = e;
        return ok & !isnan(gm + e);
    }
    float4 m;
    ok &= fast_entry(g, f.bwd[cur], F, s, m);
    f.bwd[cur ^ 1][idx] = m;
    return ok & !isnan(gm);
}

__device__ __forceinline__ bool forward_fast(const SbBubbleDesc& d, int cur, int idx) {
    Frame F;
    FStencil s;
    float4 m;
    bool ok = fast_departure(d, idx, -d.f.step->dt, F, s);
    ok &= fast_entry(d.g, d.f.fwd[cur], F, s, m);
    d.f.fwd[cur ^ 1][idx] = m;
    return ok;
}

// The step's start for one cell: statistics reset, the wind, and what the
// thickness stage samples in 64- and 32-bit words: (init, delta) and
// initLast + deltaLast.
__device__ __forceinline__ void start_chain(const SbBubbleDesc& d, int idx) {
    const SbFields& f = d.f;
    step_start(d.g, f, idx);
    if (d.ph.plain_adv) return;
    f.eta_near[idx] = make_float2(ld_s<float>(f.eta_init, idx, 0.0f), f.eta_delta[idx]);
    f.eta_far[idx] = ld_s<float>(f.eta_initL, idx, 0.0f) + f.eta_deltaL[idx];
}

// One face: u_phi (PHI) at (i + 1/2, j - 1/2), u_theta at (i + 1, j).
template <bool PHI>
__device__ __noinline__ float velocity_general(const SbBubbleDesc& d, int idx) {
    return PHI ? velocity_uphi(d.g, d.ph, d.f, idx) : velocity_utheta(d.g, d.ph, d.f, idx);
}

// (of an inner row for u_phi)
template <bool PHI>
__device__ __forceinline__ bool velocity_fast(const SbBubbleDesc& d, int idx, float& out) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP, nP = g.nP;
    constexpr int KIND = PHI ? kAtUphi : kAtUtheta;
    float s0, c0, gt, gp;
    if (PHI) {
        const int w = (i << g.logP) + ((j - 1) & g.maskP);
        s0 = g.sin_c[i];
        c0 = g.cos_c[i];
        gp = f.uph[idx];
        gt = lerp4(f.uth[w - nP], f.uth[idx - nP], f.uth[w], f.uth[idx], dup(0.5f));
    } else {
        const int e = (i << g.logP) + ((j + 1) & g.maskP);
        s0 = g.sin_e[i + 1];
        c0 = g.cos_e[i + 1];
        gt = f.uth[idx];
        gp = lerp4(f.uph[idx], f.uph[e], f.uph[idx + nP], f.uph[e + nP], dup(0.5f));
    }
    // no trace to run: at rest the face keeps its speed, and beside a torn one
    // (NaN) there is no fast form.  Two tests in this order: one for both and a
    // second behind it took 23.9 us in place of 22.6 at 512 x 1024
    if (fast_rests(gt, gp)) {
        out = 0.0f;
        return true;
    }
    if (!(fmaf(gt, gt, __fmul_rn(gp, gp)) > 1e-30f)) return false;
    FTrace T;
    FPos q;
    float vt, vp, a, n;
    bool ok = fast_trace<KIND, false>(g, f.uth, f.uph, i, j, s0, c0, gt, gp, f.step->dt, false,
                                      !d.ph.single_step, T);
    ok &= fast_pos<false>(g, s0, c0, T.d, q);
    ok &= fast_velocity<KIND>(g, f.uth, f.uph, i, j + q.flip, q.o, vt, vp);
    fast_carry(s0, c0, T.ut, T.up, T.sd, T.cdm1, q, T.d.y, vt, vp, a, n);
    out = PHI ? fmaf(a, T.up, __fmul_rn(n, T.ut)) : fmaf(a, T.ut, -__fmul_rn(n, T.up));
    return ok & !isnan(out);
}

// One of the five sample points of a cell through a map (sample_map_multi5's
// values, one at a time): points 0 .. 3 lie a quarter cell off towards
// (-, -), (+, -), (-, +), (+, +) in (theta, phi), point 4 is the cell's own
// entry.
__device__ __forceinline__ f3 map_point5(const SbGrid& g, const float4* __restrict__ map,
                                         const Frame& F, int k) {
    const int nT = g.nT, nP = g.nP, i = F.bi, j = F.bj;
    if (k == 4) return map_point(g, F, map[i * nP + j], i, j);
    const int rA = (k & 1) ? i : i - 1, cA = k >= 2 ? j : j - 1;
    const float a = (k & 1) ? 0.25f : 0.75f, b = k >= 2 ? 0.25f : 0.75f;
    f3 P[2][2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        int row = rA + r, shift = 0;
        if (row < 0) { row = 0; shift = nT; }
        if (row > nT - 1) { row = nT - 1; shift = nT; }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int col = (cA + c + shift) & g.maskP;
            P[r][c] = map_point(g, F, map[row * nP + col], row, col);
        }
    }
    return slerp_disp_inl(F.s0, F.c0, slerp_disp_inl(F.s0, F.c0, P[0][0], P[0][1], b),
                          slerp_disp_inl(F.s0, F.c0, P[1][0], P[1][1], b), a);
}

// BIMOCQ thickness at sample point k: the reconstruction through the new and
// the previous backward map (t1) and the one through the new map alone (t2).
__device__ __noinline__ float2 bimocq_general(const SbBubbleDesc& d, int cur, int idx, int k) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP;
    const float be = d.ph.base_eta;
    const Frame F = cell_frame(g, i, j);
    const f3 d1 = map_point5(g, f.bwd[cur ^ 1], F, k);
    const CStencil c1 = centred_stencil(g, pos_from_disp_fast(F, d1, g.invh, g.nT), 0.0f);
    const f3 d2 = map_at_stencil(g, f.bwdprev, F, c1);
    const Pos q2 = pos_from_disp_fast(F, d2, g.invh, g.nT);
    const SStencil s1 = sstencil_of(g, c1);
    const SStencil s2 = scalar_stencil(g, q2);
    const float sDelta = gather(f.eta_delta, s1);
    return make_float2(gather_s<float>(f.eta_initL, s2, be) + sDelta + gather(f.eta_deltaL, s2),
                       gather_s<float>(f.eta_init, s1, be) + sDelta);
}

// The same at the point d1 of an inner cell.
__device__ __forceinline__ bool bimocq_fast(const SbBubbleDesc& d, const Frame& F, float2 th, f3 d1,
                                            float& t1, float& t2, float& far) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    FPos q;
    FStencil s;
    bool ok = fast_pos<false>(g, F.s0, F.c0, d1, q);
    ok &= fast_stencil(g, F.bi, F.bj + q.flip, q.o, g.nT - 2, s);
    const float2 near = fast_gather2(f.eta_near, s, g.nP);
    // the composed point stays in the frame of the lookup's base cell: only
    // its position is wanted
    float4 R0;
    const f3 m = fast_map(g, f.bwdprev, s, th, R0, far);
    ok &= fast_pos<false>(g, R0.x, R0.z, m, q);
    ok &= fast_stencil(g, s.lo, s.j0 + q.flip, q.o, g.nT - 2, s);
    t1 = fast_gather(f.eta_far, s, g.nP) + near.y;
    t2 = near.x + near.y;
    return ok;
}

// The accumulation stage (accum_cell) by samples.
//
// Sample k of a cell: the increments and the new fields at its point (v:
// d_eta, d_gam, eta, gam); with sample 4, the cell's own forward-map point,
// the squared chord between the cell and bwd(fwd(x)) (estimateDistortion).
__device__ __noinline__ float4 accum_general(const SbBubbleDesc& d, int cur, int idx, int k,
                                             float* c2) {
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const int i = idx >> g.logP, j = idx & g.maskP;
    const Frame F = cell_frame(g, i, j);
    const f3 ds = map_point5(g, f.fwd[cur ^ 1], F, k);
    const CStencil c = centred_stencil(g, pos_from_disp_fast(F, ds, g.invh, g.nT), 0.0f);
    const SStencil s = sstencil_of(g, c);
    const float4 v00 = f.changes[s.i00], v01 = f.changes[s.i01];
    const float4 v10 = f.changes[s.i10], v11 = f.changes[s.i11];
    if (k == 4) {
        const f3 e = map_at_stencil(g, f.bwd[cur ^ 1], F, c);
        *c2 = dot3(e, e);
    }
    return make_float4(bilerp(v00.x, v01.x, v10.x, v11.x, s.a, s.b),
                       bilerp(v00.y, v01.y, v10.y, v11.y, s.a, s.b),
                       bilerp(v00.z, v01.z, v10.z, v11.z, s.a, s.b),
                       bilerp(v00.w, v01.w, v10.w, v11.w, s.a, s.b));
}

// The squared chord between the cell and fwd(bwd(x)).
__device__ __noinline__ float round_trip_general(const SbBubbleDesc& d, int cur, int idx) {
    const SbGrid& g = d.g;
    const int i = idx >> g.logP, j = idx & g.maskP;
    const Frame F = cell_frame(g, i, j);
    const float4 m = d.f.bwd[cur ^ 1][idx];
    const f3 e = sample_map(g, d.f.fwd[cur ^ 1], F,
                            pos_from_disp_fast(F, f3{m.x, m.y, m.z}, g.invh, g.nT));
    return dot3(e, e);
}

// The same at the point ds of an inner cell; trip: with the round trip.
__device__ __forceinline__ bool accum_fast(const SbBubbleDesc& d, int cur, const Frame& F, float2 th,
                                           f3 ds, bool trip, float4& v, float& c2, float& far) {
    const SbGrid& g = d.g;
    FPos q;
    FStencil s;
    bool ok = fast_pos<false>(g, F.s0, F.c0, ds, q);
    ok &= fast_stencil(g, F.bi, F.bj + q.flip, q.o, g.nT - 2, s);
    v = fast_gather4(d.f.changes, s, g.nP);
    if (trip) {
        float4 R0;
        const f3 m = fast_map(g, d.f.bwd[cur ^ 1], s, th, R0, far);
        const f3 e = fast_to_frame(g, F, m, R0, s.j0);
        c2 = fmaf(e.x, e.x, fmaf(e.y, e.y, __fmul_rn(e.z, e.z)));
    }
    return ok;
}

__device__ __forceinline__ bool round_trip_fast(const SbBubbleDesc& d, int cur, const Frame& F,
                                                float2 th, int idx, float& c2) {
    const SbGrid& g = d.g;
    const float4 m = d.f.bwd[cur ^ 1][idx];
    float far = 0.0f;
    float4 R0;
    FPos q;
    FStencil s;
    bool ok = fast_pos<false>(g, F.s0, F.c0, f3{m.x, m.y, m.z}, q);
    ok &= fast_stencil(g, F.bi, F.bj + q.flip, q.o, g.nT - 2, s);
    const f3 r = fast_map(g, d.f.fwd[cur ^ 1], s, th, R0, far);
    const f3 e = fast_to_frame(g, F, r, R0, s.j0);
    c2 = fmaf(e.x, e.x, fmaf(e.y, e.y, __fmul_rn(e.z, e.z)));
    return ok & (far <= kSlerpFar);
}

// PAR = 1: a thread per cell runs the cell's chains side by side; PAR = 2: a
// thread per cell and chain, chain by chain in whole warps.
template <bool ONE, int PAR>
__global__ void __launch_bounds__(256 * PAR, PAR == 1 ? 5 : 2) k_advect_maps_chains(SB_STEP_ARGS) {
    SB_STEP_BLOCK(tile_cells)
    const int cur = B.cur;
    const int chain = PAR == 1 ? -1 : (int)threadIdx.x / tile_cells;
    const int idx = B.first + (int)threadIdx.x - (PAR == 1 ? 0 : chain * tile_cells);
    if (idx >= d.g.N) return;
    const bool inner = inner_row(d.g, idx >> d.g.logP), maps = !d.ph.plain_adv;
    bool back = false, ahead = false;
    if (PAR == 1) {
        start_chain(d, idx);
        if (inner) {
            back = backward_fast(d, cur, idx);
            if (maps) ahead = forward_fast(d, cur, idx);
        }
    } else if (chain == 0) {
        back = inner && backward_fast(d, cur, idx);
    } else {
        start_chain(d, idx);
        if (maps) ahead = inner && forward_fast(d, cur, idx);
    }
    if (chain <= 0 && !back) backward_general(d, cur, idx);
    if (chain != 0 && maps && !ahead) forward_general(d, cur, idx);
}
template <bool ONE, int PAR>
__global__ void __launch_bounds__(256 * PAR, PAR == 1 ? 5 : 2) k_velocity_chains(SB_STEP_ARGS) {
    SB_STEP_BLOCK(tile_cells)
    const int cur = B.cur;
    (void)cur;
    const int chain = PAR == 1 ? -1 : (int)threadIdx.x / tile_cells;
    const int idx = B.first + (int)threadIdx.x - (PAR == 1 ? 0 : chain * tile_cells);
    if (idx >= d.g.N) return;
    const int i = idx >> d.g.logP;
    const bool south = i < d.g.nT - 1;  // the cell has a u_theta face
    float u = 0.0f, v = 0.0f;
    bool oku = false, okv = false;
    if (chain <= 0 && inner_row(d.g, i)) oku = velocity_fast<true>(d, idx, u);
    if (chain != 0 && south) okv = velocity_fast<false>(d, idx, v);
    if (chain <= 0) d.f.uph_adv[idx] = oku ? u : velocity_general<true>(d, idx);
    if (chain != 0 && south) d.f.uth_adv[idx] = okv ? v : velocity_general<false>(d, idx);
}

constexpr int kSampleCells = 64;  // cells of a block with its samples in parallel
static_assert(kSampleCells == kTileSizes[0], "launched over the smallest tiles");

// PAR = 1: the tile's cells, one per thread; PAR = 5: a pair of warps per
// sample point; the first pair adds the samples up in their order.
template <bool ONE, int PAR>
__global__ void __launch_bounds__(PAR == 1 ? 256 : 5 * kSampleCells, 4) k_bimocq_chains(SB_STEP_ARGS) {
    __shared__ float2 s_t[5][PAR == 1 ? 1 : kSampleCells];
    SB_STEP_BLOCK(tile_cells)
    const int cur = B.cur;
    if (d.ph.plain_adv) return;  // thickness advected by k_advect_maps
    const SbGrid& g = d.g;
    const float blend = d.ph.blend;
    const float2 th = __ldg(&g.rottab[g.nT + 1]);
    if (PAR == 1) {
        const int idx = B.first + threadIdx.x, i = idx >> g.logP;
        if (idx >= g.N) return;
        float attrib = 0.0f;
        if (ld_s<float>(d.f.eta, idx, 0.0f) != 0.0f) {
            float t1[5], t2[5];
            unsigned todo = 31u;  // samples the fast form could not serve
            if (inner_row(g, i)) {
                const Frame F = cell_frame(g, i, idx & g.maskP);
                f3 d1[5];
                float far[5];
                fast_map5_all(g, d.f.bwd[cur ^ 1], F, th, d1, far);
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    bool ok = bimocq_fast(d, F, th, d1[k], t1[k], t2[k], far[k]);
                    ok &= far[k] <= kSlerpFar && !isnan(t1[k] + t2[k]);
                    if (ok) todo &= ~(1u << k);
                }
            }
            if (todo) {
#pragma unroll
                for (int k = 0; k < 5; ++k)
                    if ((todo >> k) & 1u) {
                        const float2 v = bimocq_general(d, cur, idx, k);
                        t1[k] = v.x;
                        t2[k] = v.y;
                    }
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                attrib = fmaf((1.0f - blend) * kW5[k], t1[k], attrib);
                attrib = fmaf(blend * kW5[k], t2[k], attrib);
            }
        }
        d.f.eta_adv[idx] = fmaxf(0.0f, attrib);
        return;
    }
    const int k = threadIdx.x / kSampleCells, c = threadIdx.x % kSampleCells;
    const int idx = B.first + c, i = idx >> g.logP;
    const bool film = idx < g.N && ld_s<float>(d.f.eta, idx, 0.0f) != 0.0f;
    if (film) {
        float2 v;
        bool ok = inner_row(g, i);
        if (ok) {
            const Frame F = cell_frame(g, i, idx & g.maskP);
            float far = 0.0f;
            const f3 d1 = fast_map5(g, d.f.bwd[cur ^ 1], F, th, k, far);
            ok = bimocq_fast(d, F, th, d1, v.x, v.y, far);
            ok &= far <= kSlerpFar && !isnan(v.x + v.y);
        }
        s_t[k][c] = ok ? v : bimocq_general(d, cur, idx, k);
    }
    __syncthreads();
    if (k == 0 && idx < g.N) {
        float attrib = 0.0f;
        if (film) {
#pragma unroll
            for (int u = 0; u < 5; ++u) {
                attrib = fmaf((1.0f - blend) * kW5[u], s_t[u][c].x, attrib);
                attrib = fmaf(blend * kW5[u], s_t[u][c].y, attrib);
            }
        }
        d.f.eta_adv[idx] = fmaxf(0.0f, attrib);
    }
}

// The largest distortion of a block: an arc in grid units from the largest
// squared chord (NaN counted as 0).
__device__ __forceinline__ void block_max_chord(float far, unsigned* s_far, const SbGrid& g,
                                                SbDevStats* st) {
    far = warp_max(far);
    if ((threadIdx.x & 31) == 0) atomicMax(s_far, __float_as_uint(far));
    __syncthreads();
    if (threadIdx.x == 0)
        atomicMax(&st->distortion_bits,
                  __float_as_uint(farc_of_chord(sqrtf(__uint_as_float(*s_far))) * g.invh));
}

// Six chains per cell: the five samples and the second round trip (PAR = 6:
// the first chain's threads add the samples up in their order).
struct AccumSum {
    float ed, gd, th, gm;
};
__device__ __forceinline__ void accum_add(AccumSum& a, float w, float4 v) {
    a.ed = fmaf(w, v.x, a.ed);
    a.gd = fmaf(w, v.y, a.gd);
    a.th = fmaf(w, v.z, a.th);
    a.gm = fmaf(w, v.w, a.gm);
}
__device__ __forceinline__ void accum_store(const SbFields& f, int idx, const AccumSum& a, float ie,
                                            float ig) {
    f.eta_delta[idx] = a.ed;
    f.gam_delta[idx] = a.gd;
    f.err_eta[idx] = (a.th - a.ed - ie) * 0.5f;
    f.err_gam[idx] = (a.gm - a.gd - ig) * 0.5f;
}

template <bool ONE, int PAR>
__global__ void __launch_bounds__(PAR == 1 ? 256 : 6 * kSampleCells, 4) k_accum_chains(SB_STEP_ARGS) {
    __shared__ float4 s_v[5][PAR == 1 ? 1 : kSampleCells];
    __shared__ unsigned s_far;
    if (threadIdx.x == 0) s_far = 0u;
    if (ONE) __syncthreads();
    SB_STEP_BLOCK(tile_cells)
    const int cur = B.cur;
    const SbGrid& g = d.g;
    const SbFields& f = d.f;
    const float2 th = __ldg(&g.rottab[g.nT + 1]);
    float most = 0.0f;  // largest squared chord of this thread's cells (fmaxf skips NaN)
    if (PAR == 1) {
        const int idx = B.first + threadIdx.x, i = idx >> g.logP;
        if (idx < g.N) {
            AccumSum a = {f.eta_delta[idx], f.gam_delta[idx], 0.0f, 0.0f};
            unsigned todo = 63u;  // chains the fast forms could not serve
            float4 v[5];
            float c2 = 0.0f, c2r = 0.0f;
            if (inner_row(g, i)) {
                const Frame F = cell_frame(g, i, idx & g.maskP);
                f3 ds[5];
                float far[5];
                fast_map5_all(g, f.fwd[cur ^ 1], F, th, ds, far);
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    bool ok = accum_fast(d, cur, F, th, ds[k], k == 4, v[k], c2, far[k]);
                    ok &= far[k] <= kSlerpFar && !isnan((v[k].x + v[k].y) + (v[k].z + v[k].w));
                    if (ok) todo &= ~(1u << k);
                }
                if (round_trip_fast(d, cur, F, th, idx, c2r)) todo &= ~32u;
            }
            if (todo) {
#pragma unroll
                for (int k = 0; k < 5; ++k)
                    if ((todo >> k) & 1u) v[k] = accum_general(d, cur, idx, k, &c2);
                if (todo & 32u) c2r = round_trip_general(d, cur, idx);
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) accum_add(a, kW5[k], v[k]);
            most = fmaxf(fmaxf(most, c2), c2r);
            accum_store(f, idx, a, ld_s<float>(f.eta_init, idx, 0.0f), ld_s<float>(f.gam_init, idx, 0.0f));
        }
        block_max_chord(most, &s_far, g, f.stats);
        return;
    }
    const int k = threadIdx.x / kSampleCells, c = threadIdx.x % kSampleCells;
    const int idx = B.first + c, i = idx >> g.logP;
    const bool in = idx < g.N;
    AccumSum a = {0.0f, 0.0f, 0.0f, 0.0f};
    float ie = 0.0f, ig = 0.0f;
    if (k == 0 && in) {  // on their way while the samples are taken
        a.ed = f.eta_delta[idx];
        a.gd = f.gam_delta[idx];
        ie = ld_s<float>(f.eta_init, idx, 0.0f);
        ig = ld_s<float>(f.gam_init, idx, 0.0f);
    }
    if (in) {
        float c2 = 0.0f, far = 0.0f;
        bool ok = inner_row(g, i);
        if (k < 5) {
            float4 v;
            if (ok) {
                const Frame F = cell_frame(g, i, idx & g.maskP);
                const f3 ds = fast_map5(g, f.fwd[cur ^ 1], F, th, k, far);
                ok = accum_fast(d, cur, F, th, ds, k == 4, v, c2, far);
                ok &= far <= kSlerpFar && !isnan((v.x + v.y) + (v.z + v.w));
            }
            if (!ok) v = accum_general(d, cur, idx, k, &c2);
            s_v[k][c] = v;
        } else {
            if (ok) ok = round_trip_fast(d, cur, cell_frame(g, i, idx & g.maskP), th, idx, c2);
            if (!ok) c2 = round_trip_general(d, cur, idx);
        }
        if (k >= 4) most = fmaxf(most, c2);
    }
    __syncthreads();
    if (k == 0 && in) {
#pragma unroll
        for (int u = 0; u < 5; ++u) accum_add(a, kW5[u], s_v[u][c]);
        accum_store(f, idx, a, ie, ig);
    }
    block_max_chord(most, &s_far, g, f.stats);
}

}  // namespace

namespace {

// A set's cells decide the form.  Below one thread per cell of a full chip
// (1024 threads an SM, 155,648 on 152 SMs) the chains run in parallel: there a launch lasts as
// long as its longest thread (64 x 128: 40 us per step against 47; 256 x 512:
// k_bimocq 22 us against 33, k_velocity 14 against 16).  Above it they run in
// one thread, which shares the five-point lookups and needs no exchange
// (512 x 1024: k_bimocq 49 us against 58, k_accum 39 against 53).
bool parallel_chains(const SbStepPlan& P) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return P.nchain[0] * kTileSizes[0] <= sms * 1024;
}

// PAR chains of a cell in parallel over the set's tiles of size tile.
template <class K>
void launch_chains(const SbStepPlan& P, int tile, int par, K* one, K* each, cudaStream_t s) {
    launch_cells(P, 0, P.nchain[tile], tile, kTileSizes[tile] * par, one, each, s);
}

}  // namespace

int stage_tile(const SbStepPlan& P, int stage) {
    const bool fixed = parallel_chains(P) && P.nchain[0] == P.ntiles[0] &&
                       (stage == STAGE_BIMOCQ || stage == STAGE_ACCUM);
    return fixed ? 0 : P.sel[stage];
}

void launch_chain_stage(const SbStepPlan& P, int stage, cudaStream_t s) {
    const int k = P.sel[stage];
    const bool par = parallel_chains(P);
    switch (stage) {
        case STAGE_MAPS:
            if (par) launch_chains(P, k, 2, k_advect_maps_chains<true, 2>, k_advect_maps_chains<false, 2>, s);
            else launch_chains(P, k, 1, k_advect_maps_chains<true, 1>, k_advect_maps_chains<false, 1>, s);
            break;
        case STAGE_VELOCITY:
            if (par) launch_chains(P, k, 2, k_velocity_chains<true, 2>, k_velocity_chains<false, 2>, s);
            else launch_chains(P, k, 1, k_velocity_chains<true, 1>, k_velocity_chains<false, 1>, s);
            break;
        case STAGE_BIMOCQ:
            if (par) launch_chains(P, 0, 5, k_bimocq_chains<true, 5>, k_bimocq_chains<false, 5>, s);
            else launch_chains(P, k, 1, k_bimocq_chains<true, 1>, k_bimocq_chains<false, 1>, s);
            break;
        case STAGE_ACCUM:
            if (par) launch_chains(P, 0, 6, k_accum_chains<true, 6>, k_accum_chains<false, 6>, s);
            else launch_chains(P, k, 1, k_accum_chains<true, 1>, k_accum_chains<false, 1>, s);
            break;
        default: break;
    }
}

}  // namespace sb
