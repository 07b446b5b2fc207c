// The chain kernels' geometry at single points, for tests/test_gpu_geometry.py.
#include "sb_fastgeo.cuh"

using namespace sb;

namespace {

struct Point {
    float s0, c0, dx, dy, dz;
};

__global__ void k_atan(const float* t, float* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = atan_pair(make_float2(t[i], t[i])).x;
}

// out[4 i ..]: the offsets and whether the form serves the point, flip
template <bool EXACT>
__global__ void k_fast_pos(SbGrid g, const Point* p, float4* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    FPos q;
    const bool ok = fast_pos<EXACT>(g, p[i].s0, p[i].c0, f3{p[i].dx, p[i].dy, p[i].dz}, q);
    out[i] = make_float4(q.o.x, q.o.y, ok ? 1.0f : 0.0f, q.flip ? 1.0f : 0.0f);
}
template <bool EXACT>
__global__ void k_general_pos(SbGrid g, const Point* p, float4* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    Frame F = {0, 0, 0.0f, 0.0f, p[i].s0, p[i].c0, 0.0f, 0.0f};
    const f3 d = {p[i].dx, p[i].dy, p[i].dz};
    const Pos q = EXACT ? pos_from_disp(F, d, g.invh, g.nT) : pos_from_disp_fast(F, d, g.invh, g.nT);
    out[i] = make_float4(q.ox, q.oy, 1.0f, q.bj ? 1.0f : 0.0f);
}

struct Chord {
    float s0, c0, a;
    f3 A, B;
};
// both lanes of the pair and the single form, then the general one
__global__ void k_slerp(const Chord* c, f3* out, float* far, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const Chord k = c[i];
    float2 c2;
    const F3P r = slerp_pair(k.s0, k.c0, pair3(k.A, k.A), pair3(k.B, k.B), slerp_coef(k.a), c2);
    float f = 0.0f;
    out[4 * i] = lane0(r);
    out[4 * i + 1] = lane1(r);
    out[4 * i + 2] = slerp_one(k.s0, k.c0, k.A, k.B, slerp_coef(k.a), f);
    out[4 * i + 3] = slerp_disp(k.s0, k.c0, k.A, k.B, k.a);
    far[i] = f;
}

template <class K, class... A>
int run(K* kernel, int n, A... args) {
    kernel<<<(n + 127) / 128, 128>>>(args..., n);
    const cudaError_t e = cudaGetLastError();
    return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

}  // namespace

extern "C" {

// Host arrays in and out; 0 on success.
int geo_atan(const float* t, float* out, int n) {
    float *dt, *dout;
    if (cudaMalloc(&dt, 4 * n) || cudaMalloc(&dout, 4 * n)) return 1;
    cudaMemcpy(dt, t, 4 * n, cudaMemcpyHostToDevice);
    const int rc = run(k_atan, n, dt, dout);
    cudaMemcpy(out, dout, 4 * n, cudaMemcpyDeviceToHost);
    cudaFree(dt);
    cudaFree(dout);
    return rc;
}

int geo_pos(int nT, const float* points, float* out, int n, int fast, int exact) {
    SbGrid g{};
    g.nT = nT;
    g.invh = (float)(nT / 3.14159265358979323846);
    Point* dp;
    float4* dout;
    if (cudaMalloc(&dp, sizeof(Point) * n) || cudaMalloc(&dout, sizeof(float4) * n)) return 1;
    cudaMemcpy(dp, points, sizeof(Point) * n, cudaMemcpyHostToDevice);
    int rc;
    if (fast) rc = exact ? run(k_fast_pos<true>, n, g, dp, dout) : run(k_fast_pos<false>, n, g, dp, dout);
    else rc = exact ? run(k_general_pos<true>, n, g, dp, dout) : run(k_general_pos<false>, n, g, dp, dout);
    cudaMemcpy(out, dout, sizeof(float4) * n, cudaMemcpyDeviceToHost);
    cudaFree(dp);
    cudaFree(dout);
    return rc;
}

int geo_slerp(const float* chords, float* out, float* far, int n) {
    Chord* dc;
    f3* dout;
    float* df;
    if (cudaMalloc(&dc, sizeof(Chord) * n) || cudaMalloc(&dout, sizeof(f3) * 4 * n) || cudaMalloc(&df, 4 * n))
        return 1;
    cudaMemcpy(dc, chords, sizeof(Chord) * n, cudaMemcpyHostToDevice);
    const int rc = run(k_slerp, n, dc, dout, df);
    cudaMemcpy(out, dout, sizeof(f3) * 4 * n, cudaMemcpyDeviceToHost);
    cudaMemcpy(far, df, 4 * n, cudaMemcpyDeviceToHost);
    cudaFree(dc);
    cudaFree(dout);
    cudaFree(df);
    return rc;
}

}  // extern "C"
