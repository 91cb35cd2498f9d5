// hy_tile.cuh -- the pixel tiles and launch shape of the per-view kernels
// (hy_render.cu) and the film passes (hy_pass.cu).
#pragma once

#include "hy_shade.cuh"

namespace {

using namespace hy;
using namespace hy::dev;

constexpr int kTileW = 16, kTileH = 8, kThreads = 128;

__device__ __forceinline__ void load_shared(const ShadeArgs &A, float4 *tf, float *lut) {
    stage_tf(A.tf, A.ntf, tf);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = float(i) / 255.f;
    __syncthreads();
}

__device__ __forceinline__ void tile_xy(int &x, int &y) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    x = blockIdx.x * kTileW + (warp & 1) * 8 + (lane & 7);
    y = blockIdx.y * kTileH + (warp >> 1) * 4 + (lane >> 3);
}

__device__ __forceinline__ void count_samples(const ShadeArgs &A, long long samples) {
    if (!A.count) return;
    unsigned long long s = (unsigned long long)samples;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(A.counter, s);
}

inline size_t smem_bytes(const ShadeArgs &a) {
    return size_t(a.ntf + kTfPad) * sizeof(float4) + 256 * sizeof(float);
}

inline dim3 grid_of(const ShadeArgs &a) {
    return dim3((a.view.W + kTileW - 1) / kTileW, (a.view.H + kTileH - 1) / kTileH);
}

}  // namespace
