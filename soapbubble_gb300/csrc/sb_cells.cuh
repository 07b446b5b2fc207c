// Cell code shared by the step kernels (sb_step.cu, one thread per cell) and
// the chain kernels (sb_chain.cu).
#pragma once
#include "sb_device.cuh"
#include "sb_internal.h"

namespace sb {

namespace {

// Weights of a cell's five sample points (MULTISAMPLE).
__constant__ float kW5[5] = {0.125f, 0.125f, 0.125f, 0.125f, 0.5f};

__device__ __forceinline__ Frame face_frame_uphi(const SbGrid& g, int i, int j) {
    Frame F;
    F.bi = i; F.bj = j; F.fi = 0.5f; F.fj = -0.5f;
    F.s0 = g.sin_c[i]; F.c0 = g.cos_c[i];
    F.s0lo = 0.0f; F.c0lo = 0.0f;
    return F;
}

__device__ __forceinline__ Frame face_frame_utheta(const SbGrid& g, int i, int j) {
    Frame F;
    F.bi = i + 1; F.bj = j; F.fi = 0.0f; F.fj = 0.0f;
    F.s0 = g.sin_e[i + 1]; F.c0 = g.cos_e[i + 1];
    F.s0lo = 0.0f; F.c0lo = 0.0f;
    return F;
}

__device__ __forceinline__ Pos pos_of(const Frame& F, const Trace& T, const SbGrid& g) {
    return T.moved ? pos_from_disp(F, T.d, g.invh, g.nT) : frame_pos(F, 0.0f, 0.0f);
}

// What a step begins with beside the advection: the statistics reset and the
// wind, initial wind + corridor(t); NaN -> 0.
__device__ __forceinline__ void step_start(const SbGrid& g, const SbFields& f, int idx) {
    if (idx == 0) {
        f.stats->distortion_bits = 0u;
        f.stats->reinit = 0;
        f.stats->broken_cells = 0;
    }
    const float wg = f.step->windg;
    float ua = f.uair_init[idx] + wg * f.corr_u[idx];
    f.uair[idx] = isnan(ua) ? 0.0f : ua;
    if ((idx >> g.logP) < g.nT - 1) {
        float va = f.vair_init[idx] + wg * f.corr_v[idx];
        f.vair[idx] = isnan(va) ? 0.0f : va;
    }
}

// Velocity self-advection with parallel transport (RUNGE_KUTTA path).
__device__ __forceinline__ float advect_velocity(const SbGrid& g, const float* __restrict__ uth,
                                                 const float* __restrict__ uph, const Frame& F,
                                                 float gt, float gp, float dt, bool outPhi,
                                                 bool rk2) {
    const f3 w = {F.s0, 0.0f, F.c0};
    // a zero or NaN speed stops the trace; the reference then writes that
    // speed (bubble.cu:689-692, 727-730)
    const Trace T = trace_gc<true>(g, uth, uph, F, gt, gp, dt, rk2);
    if (!T.moved) return T.fail;
    const f3 P = w + T.d;
    const Pos qp = pos_from_disp_fast(F, T.d, g.invh, g.nT);
    float pt, pp;
    velocity_at(g, uth, uph, qp, pt, pp);
    f3 beth, beph;
    basis_at(P, beth, beph);
    const f3 pu = pt * beth + pp * beph;
    const f3 uCircleP = T.cd * T.u_ - T.sd * w;
    const f3 vCircleP = cross3(P, uCircleP);
    const float a = dot3(pu, vCircleP);
    const float b = dot3(pu, uCircleP);
    const f3 pu2 = b * T.u_ + a * T.v_;
    if (outPhi) return pu2.y;                       // e_phi = (0, 1, 0)
    return pu2.x * F.c0 - pu2.z * F.s0;             // e_theta = (c0, 0, -s0)
}

__device__ __forceinline__ float velocity_uphi(const SbGrid& g, const SbPhys& ph,
                                               const SbFields& f, int idx) {
    const Frame F = face_frame_uphi(g, idx >> g.logP, idx & g.maskP);
    const float gp = f.uph[idx];
    const float gt = sample_utheta(g, f.uth, frame_pos(F, 0.0f, 0.0f));
    return advect_velocity(g, f.uth, f.uph, F, gt, gp, f.step->dt, true, !ph.single_step);
}

__device__ __forceinline__ float velocity_utheta(const SbGrid& g, const SbPhys& ph,
                                                 const SbFields& f, int idx) {
    const Frame F = face_frame_utheta(g, idx >> g.logP, idx & g.maskP);
    const float gt = f.uth[idx];
    const float gp = sample_uphi(g, f.uph, frame_pos(F, 0.0f, 0.0f));
    return advect_velocity(g, f.uth, f.uph, F, gt, gp, f.step->dt, false, !ph.single_step);
}

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// The block's bubble descriptor is copied to shared memory first, so the
// cell code reads grid constants and array pointers from there.
__device__ __forceinline__ const SbBubbleDesc& stage_tile_desc(SbBubbleDesc* const* descs, int b,
                                                               SbBubbleDesc* s_d) {
    constexpr int kWords = (int)(sizeof(SbBubbleDesc) / 4);
    const int* src = reinterpret_cast<const int*>(descs[b]);
    int* dst = reinterpret_cast<int*>(s_d);
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    return *s_d;
}

// The bubble of a block: its descriptor, its first cell, the map parity.  A
// bubble stepped alone comes in the kernel's parameters (ONE: its pointers and
// constants are then uniform operands, and nothing is staged: three dependent
// loads and a barrier per block), the cells in block order; what changes on
// the device is read there (the parity, the halt switch, and the offsets of
// BF16 fields, which an upload moves).  A set's blocks find theirs by tile.
struct StepBlock {
    int first, cur;
    bool halted;
    float base_eta, base_gam;
};
template <bool ONE>
__device__ __forceinline__ const SbBubbleDesc& step_block(const SbBubbleDesc& one,
                                                          SbBubbleDesc* const* descs,
                                                          const int2* tiles, int tile_cells,
                                                          SbBubbleDesc* s_d, StepBlock& B) {
    if (ONE) {
        const SbBubbleDesc* self = one.f.self;
        B.first = blockIdx.x * tile_cells;
        B.cur = self->cur;
        B.halted = self->halted != 0;
        B.base_eta = self->ph.base_eta;
        B.base_gam = self->ph.base_gam;
        return one;
    }
    const int2 t = tiles[blockIdx.x];
    const SbBubbleDesc& d = stage_tile_desc(descs, t.x, s_d);
    B.first = t.y;
    B.cur = d.cur;
    B.halted = d.halted != 0;
    B.base_eta = d.ph.base_eta;
    B.base_gam = d.ph.base_gam;
    return d;
}

#define SB_STEP_ARGS                                                                           \
    const __grid_constant__ SbBubbleDesc one, SbBubbleDesc* const* __restrict__ descs,         \
        const int2* __restrict__ tiles, int tile_cells
#define SB_STEP_BLOCK(cells)                                                                   \
    __shared__ __align__(16) SbBubbleDesc s_d[1];                                              \
    StepBlock B;                                                                               \
    const SbBubbleDesc& d = step_block<ONE>(one, descs, tiles, cells, s_d, B);                 \
    if (B.halted) return; /* the same in every thread of the block */

// One launch over `blocks` tiles of size `tile` from tile `first` on.
template <class K>
void launch_cells(const SbStepPlan& P, int first, int blocks, int tile, int threads, K* one, K* each,
                  cudaStream_t s) {
    static const SbBubbleDesc none{};  // a batch: the kernels find their bubble by tile
    const int2* tiles = P.tiles[tile] + first;
    if (P.one) one<<<blocks, threads, 0, s>>>(*P.one, P.descs, tiles, kTileSizes[tile]);
    else each<<<blocks, threads, 0, s>>>(none, P.descs, tiles, kTileSizes[tile]);
}

}  // namespace

}  // namespace sb
