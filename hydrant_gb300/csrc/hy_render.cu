// hy_render.cu -- shading kernels and the rendering entry points.
//
// Two ways in:
//  * hy_render / hy_render_device: one fused kernel per view does ray
//    generation, the march and the write_to quantisation; no film goes
//    through HBM.  A warp shades an 8x4 ray tile, a 128-thread block a 16x8
//    pixel tile; the transfer function and the u8 normalisation table sit in
//    shared memory.
//  * hy_shade_pass: the four passes of the reference (cuda_shading.cu:14-96)
//    over a caller-owned film in the reference's pixel layout, so a renderer
//    can swap its ShaderMeta.devices[Cuda] entry for this one.

#include <algorithm>
#include <cstring>

#include "hy_tile.cuh"

using namespace hy;
using namespace hy::dev;

namespace {

// StdVec4Pixel::write_to (pixel_template.hpp:11-20), RGBA: alpha = saturate(v.a).
__device__ __forceinline__ uchar4 quantise(const ShadeArgs &A, float4 v) {
    if (v.w != 0.f)
        return make_uchar4(saturate_u8(v.x), saturate_u8(v.y), saturate_u8(v.z), saturate_u8(v.w));
    return make_uchar4(A.clear_u8[0], A.clear_u8[1], A.clear_u8[2], 0);
}

// LEAN: Volume shader, Default mode, no compositing and no aux output
// (theta / phi are not computed; see VolumeMarch::step).
template <int SHADER, int PC, int DT, bool PADDED, int COMPOSITE, bool LEAN, int GATHER = 0,
          int LOOP = kLoopOne>
__device__ __forceinline__ void render_body(const ShadeArgs &A) {
    extern __shared__ float4 smem[];
    float4 *tf = smem;
    float *lut = reinterpret_cast<float *>(smem + A.ntf + kTfPad);
    load_shared(A, tf, lut);
    const Shared S = make_shared(tf, A.ntf, lut);
    int x, y;
    tile_xy(x, y);
    unsigned int samples = 0;  // one ray: at most max_steps (+ 6 at a hit) samples
    if (x < A.view.W && y < A.view.H) {
        float ox, oy, oz, dx, dy, dz;
        gen_ray(A.view, x, y, ox, oy, oz, dx, dy, dz);
        float4 v, aux;
        if (COMPOSITE) {
            samples = unsigned(
                composite_ray<SHADER, PC, DT, PADDED, GATHER, LOOP>(A, A.view, S, ox, oy, oz, dx, dy,
                                                                  dz, v, aux));
        } else {
            Px p;
            samples = unsigned(emit<SHADER, PC, DT, PADDED, LEAN, GATHER, LOOP>(
                p, A, A.view, S, ox, oy, oz, dx, dy, dz, 0.f, 0.f, 0.f, A.bbox_max[0],
                A.bbox_max[1], A.bbox_max[2]));
            v = make_float4(p.vx, p.vy, p.vz, p.vw);
            if (SHADER == HY_SHADER_VOLUME)
                aux = make_float4(p.e0, p.e1, p.e2, p.e3);
            else if (SHADER == HY_SHADER_ISOSURFACE)
                aux = make_float4(p.e3, 0.f, 0.f, 0.f);
            else
                aux = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if constexpr (LEAN) {
            // the pixel again from the thread's index, not held through the
            // march (the memory clobber keeps the compiler from carrying it)
            asm volatile("" ::: "memory");
            tile_xy(x, y);
        }
        const size_t idx = size_t(y) * A.view.W + x;
        A.rgba[idx] = quantise(A, v);
        if (A.vout) A.vout[idx] = v;
        if (!LEAN && A.aux) A.aux[idx] = aux;
    }
    count_samples(A, samples);
}

template <int SHADER, int PC, int DT, bool PADDED, int COMPOSITE, int LOOP = kLoopOne>
__global__ void __launch_bounds__(kThreads) render_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, PADDED, COMPOSITE, false, false, LOOP>(A);
}

// The Isosurface march with 2 or 4 samples in flight (80 and 128 registers).
template <int PC, int DT, int LOOP>
__global__ void __launch_bounds__(kThreads, LOOP == kLoopBatch4 ? 4 : 6)
    render_iso_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<HY_SHADER_ISOSURFACE, PC, DT, true, 0, false, false, LOOP>(A);
}

// The lean march of the per-view path by loads (f32 volumes, volumes without
// an apron or gather textures) with its own register budget
// (HY_RENDER_LEAN_REGS, 0: the compiler's choice, 56 registers).  64-view
// step of u8 bricks by loads, one launch per view: 56 registers 199.7 ms, 48
// (8 bytes spilled) 211.7 ms, 40 269.0 ms.
#ifndef HY_RENDER_LEAN_REGS
#define HY_RENDER_LEAN_REGS 0
#endif
#if HY_RENDER_LEAN_REGS > 0
#define HY_RENDER_LEAN_BOUNDS __maxnreg__(HY_RENDER_LEAN_REGS)
#else
#define HY_RENDER_LEAN_BOUNDS __launch_bounds__(kThreads)
#endif
template <int SHADER, int PC, int DT, bool PADDED, int LOOP>
__global__ void HY_RENDER_LEAN_BOUNDS render_lean_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, PADDED, 0, true, false, LOOP>(A);
}
// The same march sampling by texture gathers (u8 bricks with an apron in
// the volume's gather textures), one sample at a time, for large views with
// nothing to pass over and for early termination: 64-view step, one launch per view, 169.6 ms at 48
// registers against 172.4 at 56, 173.1 at 64 and 198.8 for the loads
// (HY_RENDER_GATHER=0 builds the per-view path without gathers).
#ifndef HY_RENDER_GATHER
#define HY_RENDER_GATHER 1
#endif
#ifndef HY_RENDER_GATHER_REGS
#define HY_RENDER_GATHER_REGS 48
#endif
// The paged cache's march with early termination (each brick's own mapping, up
// to 16 textures): 56 registers -- 21.2 ms per out-of-core frame against 24.6
// at 48 (64 bytes spilled) and 22.5 at 64, measured without termination.
#ifndef HY_RENDER_PAGED_GATHER_REGS
#define HY_RENDER_PAGED_GATHER_REGS 56
#endif
template <int SHADER, int PC, int DT, bool PADDED, int GATHER, int LOOP>
__global__ void __maxnreg__(GATHER == kGatherPaged ? HY_RENDER_PAGED_GATHER_REGS
                                                   : HY_RENDER_GATHER_REGS)
    render_lean_gather_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, PADDED, 0, true, GATHER, LOOP>(A);
}


// Lean march with 2 or 4 samples of a ray in flight (volume_batches), 64 or
// 128 registers: with fewer the compiler fetches the samples one after the
// other again.
template <int SHADER, int PC, int DT, int GATHER, int LOOP>
__global__ void __launch_bounds__(kThreads, LOOP == kLoopBatch4 ? 4 : 8)
    render_batches_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, true, 0, true, GATHER, LOOP>(A);
}

// Small launches of the lean march: 8 lanes a ray (volume_group).  A warp
// holds 2x2 rays, a block 4 warps.
constexpr int kGroup = 8, kGroupW = 2, kGroupH = 32 / kGroup / kGroupW;
template <int SHADER, int PC, int DT, bool PADDED, int GATHER>
__global__ void __launch_bounds__(kThreads) render_group_kernel(const __grid_constant__ ShadeArgs A) {
    extern __shared__ float4 smem[];
    float4 *tf = smem;
    float *lut = reinterpret_cast<float *>(smem + A.ntf + kTfPad);
    load_shared(A, tf, lut);
    const Shared S = make_shared(tf, A.ntf, lut);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane / kGroup;
    const int x = (blockIdx.x * 2 + (warp & 1)) * kGroupW + r % kGroupW;
    const int y = (blockIdx.y * 2 + (warp >> 1)) * kGroupH + r / kGroupW;
    const bool on = x < A.view.W && y < A.view.H;
    float ox, oy, oz, dx, dy, dz;
    gen_ray(A.view, x, y, ox, oy, oz, dx, dy, dz);
    Px p;
    const bool hit = emit_setup<SHADER>(p, A, ox, oy, oz, dx, dy, dz, 0.f, 0.f, 0.f, A.bbox_max[0],
                                        A.bbox_max[1], A.bbox_max[2]);
    const unsigned int samples = volume_group<kGroup, PC, DT, PADDED, GATHER>(p, on && hit, A, S);
    if (on && (lane & (kGroup - 1)) == 0) {
        const float4 v = make_float4(p.vx, p.vy, p.vz, p.vw);
        const size_t idx = size_t(y) * A.view.W + x;
        A.rgba[idx] = quantise(A, v);
        if (A.vout) A.vout[idx] = v;
    }
    count_samples(A, samples);
}

// The Isosurface march of small launches: 8 lanes a ray (iso_group).  A block
// takes 8x4 rays; their hits are shaded by one warp, a ray a lane: shading costs
// a few hundred FP64 instructions a warp whether one lane or all take part
// (linear_to_srgb), which at four rays a warp, where rays hit at once, was most
// of the time (190^2 over 256^3 noise: 158 us, 40 this way, 32 with one ray a lane
// throughout).
constexpr int kIsoGroupThreads = 256, kIsoW = 8, kIsoH = 4;
template <int PC, int DT, bool PADDED>
__global__ void __launch_bounds__(kIsoGroupThreads)
    render_iso_group_kernel(const __grid_constant__ ShadeArgs A) {
    extern __shared__ float4 smem[];
    __shared__ IsoHit hits[kIsoW * kIsoH];
    __shared__ unsigned char found[kIsoW * kIsoH];
    float4 *tf = smem;
    float *lut = reinterpret_cast<float *>(smem + A.ntf + kTfPad);
    load_shared(A, tf, lut);
    const Shared S = make_shared(tf, A.ntf, lut);
    const int ray = threadIdx.x / kGroup;
    const int x = blockIdx.x * kIsoW + ray % kIsoW, y = blockIdx.y * kIsoH + ray / kIsoW;
    {
        const bool on = x < A.view.W && y < A.view.H;
        float ox, oy, oz, dx, dy, dz;
        gen_ray(A.view, x, y, ox, oy, oz, dx, dy, dz);
        Px p;
        const bool hit = emit_setup<HY_SHADER_ISOSURFACE>(p, A, ox, oy, oz, dx, dy, dz, 0.f, 0.f, 0.f,
                                                          A.bbox_max[0], A.bbox_max[1],
                                                          A.bbox_max[2]);
        IsoHit h;
        unsigned int samples;
        const bool f = iso_group<kGroup, PC, DT, PADDED>(p, on && hit, A, S, h, samples);
        if ((threadIdx.x & (kGroup - 1)) == 0) {
            found[ray] = f;
            if (f) hits[ray] = h;
        }
        count_samples(A, samples);
    }
    __syncthreads();
    const int t = threadIdx.x;
    const int px = blockIdx.x * kIsoW + t % kIsoW, py = blockIdx.y * kIsoH + t / kIsoW;
    if (t >= kIsoW * kIsoH || px >= A.view.W || py >= A.view.H) return;
    Px p;
    p.vx = p.vy = p.vz = p.vw = 0.f;
    p.e0 = A.view.ray_o[0];
    p.e1 = A.view.ray_o[1];
    p.e2 = A.view.ray_o[2];
    p.e3 = __int_as_float(0x7f800000);  // INFINITY
    if (found[t]) {
        const IsoHit h = hits[t];
        p.ox = h.o.x;
        p.oy = h.o.y;
        p.oz = h.o.z;
        iso_shade(p, h.at, h.n.x, h.n.y, h.n.z, A, A.view);
    }
    const float4 v = make_float4(p.vx, p.vy, p.vz, p.vw);
    const size_t idx = size_t(py) * A.view.W + px;
    A.rgba[idx] = quantise(A, v);
    if (A.vout) A.vout[idx] = v;
    if (A.aux) A.aux[idx] = make_float4(p.e3, 0.f, 0.f, 0.f);
}

// The per-brick compositing variants of the Volume and Isosurface shaders,
// held to 64 registers (8 resident blocks): on the 512^3 tubes at 1024^2,
// Volume 147 -> 163 and Isosurface 231 -> 237 Gsamples/s against 80
// registers and 6 blocks unbounded (Blocks is 3 % faster unbounded and keeps
// render_kernel); 128 registers with four samples in flight.
template <int SHADER, int PC, int DT, bool PADDED, int LOOP>
__global__ void __launch_bounds__(kThreads, LOOP == kLoopBatch4 ? 4 : 8)
    render_composite_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, PADDED, 1, false, false, LOOP>(A);
}
// The Volume shader's per-brick compositing sampling by gathers (u8 bricks
// with an apron), 64 registers (8 blocks): 64-view step of per-view launches
// 309.2 ms, against 320.7 at 10 blocks, 319.8 at 12 and 334.6 for the loads.
#ifndef HY_RENDER_COMPOSITE_GATHER
#define HY_RENDER_COMPOSITE_GATHER 1
#endif
template <int SHADER, int PC, int DT, bool PADDED, int LOOP>
__global__ void __launch_bounds__(kThreads, LOOP == kLoopBatch4 ? 4 : 8)
    render_composite_gather_kernel(const __grid_constant__ ShadeArgs A) {
    render_body<SHADER, PC, DT, PADDED, 1, false, true, LOOP>(A);
}

template <int SHADER, int PC, int DT, bool PADDED, int LOOP>
void launch_composite(const ShadeArgs &a, cudaStream_t s) {
    const dim3 g = grid_of(a);
    const size_t sm = smem_bytes(a);
    if constexpr (HY_RENDER_COMPOSITE_GATHER && SHADER == HY_SHADER_VOLUME && PADDED &&
                  DT == HY_DTYPE_U8) {
        if (a.vol.tex) {
            render_composite_gather_kernel<SHADER, PC, DT, PADDED, LOOP><<<g, kThreads, sm, s>>>(a);
            return;
        }
    }
    render_composite_kernel<SHADER, PC, DT, PADDED, LOOP><<<g, kThreads, sm, s>>>(a);
}
// Samples in flight by the warps of rays a scheduler gets.  512^3 blobs by
// gathers, half the cells free, 128^2, 256^2, 512^2, 1024^2 (0.8, 3.4, 13.5, 54
// warps): one sample at a time 549, 487, 523, 1321 us, two 393, 367, 466, 1249,
// four 293, 276, 497, 1457; no free cells at 1024^2 1916, 1920, 2477.
template <int SHADER, int PC, int DT, bool PADDED>
void pick_composite(const ShadeArgs &a, cudaStream_t s) {
    if constexpr (PADDED) {
        constexpr bool volume = SHADER == HY_SHADER_VOLUME;
        const long long rays = (long long)a.view.W * a.view.H, per_warp = 32ll * a.schedulers;
        if (a.vol.P <= kMaxBatchesP && (!volume || a.mode == HY_VOLUME_DEFAULT)) {
            if (rays < 8 * per_warp) {
                launch_composite<SHADER, PC, DT, PADDED, kLoopBatch4>(a, s);
                return;
            }
            if constexpr (volume) {
                if (a.skip.d) {
                    launch_composite<SHADER, PC, DT, PADDED, kLoopBatch2>(a, s);
                    return;
                }
            }
        }
    }
    launch_composite<SHADER, PC, DT, PADDED, kLoopOne>(a, s);
}

template <int SHADER, int PC, int DT, bool PADDED, int GATHER>
void launch_group(const ShadeArgs &a, cudaStream_t s) {
    const dim3 g((a.view.W + 2 * kGroupW - 1) / (2 * kGroupW),
                 (a.view.H + 2 * kGroupH - 1) / (2 * kGroupH));
    render_group_kernel<SHADER, PC, DT, PADDED, GATHER><<<g, kThreads, smem_bytes(a), s>>>(a);
}

// The lean march of one view in the form its size wants, by the warps (of 32
// rays) a scheduler would get.  u8 by gathers, 1-voxel steps, us at 0.8, 3.4,
// 13.5 and 54 warps (256^3, 512^3, 512^3, 512^3 blobs at 128^2, 256^2, 512^2,
// 1024^2), half the cells free of effect: 8 lanes a ray 65, 244, 783, 2871; 4
// samples in flight 97, 196, 363, 1100; 2 in flight 112, 247, 323, 904; one at
// a time 163, 361, 364, 941 (without the skip grid 163, 479, 491, 1336).  No
// free cells: 63, 297, 1017, 3867; 83, 208, 483, 1571; 106, 281, 436, 1328; 163,
// 425, 443, 1293.  f32 (200^3, quarter-voxel steps, free cells): 97, 155, 449,
// 1643; 163, 169, 230, 587; 191, 198, 248, 526; 288, 286, 311, 581.  Without an
// apron only the group and the plain march are built: 83, 228, 738 against
// 230, 231, 392.
// Without free cells samples in flight end earlier.  256^3 blobs at 256^2, 320^2,
// 380^2 and 400^2 (3.4, 5.3, 7.4, 8.2 warps): u8 by gathers 90, 125, 156 us with
// four, 118, 144 and 160 with two at the last three, 147, 153, 162, 168 with
// one; u8 by loads 118, 154, 188; 145, 172, 206; 150, 158, 169, 183; f32 135, 178,
// 216; 161, 184, 220; 176, 197, 208, 212.  Rays that are soon opaque (density 0.3)
// lose more where the line is too high: u8 by loads at 380^2 81 with four, 70
// with two, 66 with one.  In bricks of fewer than 32 voxels a batch ends at a face
// after a few steps: f32 by loads at 360x400, bricks of 16^3, 132 with two, 124
// with one; a paged pool of 32^3 bricks at 300^2 (4.6 warps) 221 with four, 200
// with one.
template <int SHADER, int PC, int DT, bool PADDED, int GATHER>
void launch_lean(const ShadeArgs &a, cudaStream_t s) {
    const dim3 g = grid_of(a);
    const size_t sm = smem_bytes(a);
    if (a.ert > 0.f) {
        if constexpr (GATHER != 0)
            render_lean_gather_kernel<SHADER, PC, DT, PADDED, GATHER, kLoopErt><<<g, kThreads, sm, s>>>(a);
        else
            render_lean_kernel<SHADER, PC, DT, PADDED, kLoopErt><<<g, kThreads, sm, s>>>(a);
        return;
    }
    const long long rays = (long long)a.view.W * a.view.H, per_warp = 32ll * a.schedulers;
    if (rays < 2 * per_warp) {
        launch_group<SHADER, PC, DT, PADDED, GATHER>(a, s);
        return;
    }
    if constexpr (PC == 0 && GATHER == 0) {
        if (!PADDED || a.vol.P > kMaxBatchesP) {
            render_lean_kernel<SHADER, PC, DT, PADDED, kLoopOne><<<g, kThreads, sm, s>>>(a);
            return;
        }
    }
    const int four = a.skip.d ? 8 : GATHER ? 5 : 4,
              two = a.vol.P < 34 ? 0 : GATHER ? 24 : DT == HY_DTYPE_F32 ? 8 : 0;
    if (rays < four * per_warp)
        render_batches_kernel<SHADER, PC, DT, GATHER, kLoopBatch4><<<g, kThreads, sm, s>>>(a);
    else if (a.skip.d || rays < two * per_warp)
        render_batches_kernel<SHADER, PC, DT, GATHER, kLoopBatch2><<<g, kThreads, sm, s>>>(a);
    else if constexpr (GATHER != 0)
        render_lean_gather_kernel<SHADER, PC, DT, PADDED, GATHER, kLoopOne><<<g, kThreads, sm, s>>>(a);
    else
        render_lean_kernel<SHADER, PC, DT, PADDED, kLoopOne><<<g, kThreads, sm, s>>>(a);
}

template <int SHADER, int PC, int DT, bool PADDED>
void launch_fused(const ShadeArgs &a, cudaStream_t s) {
    const dim3 g = grid_of(a);
    const size_t sm = smem_bytes(a);
    if (a.composite) {
        if constexpr (SHADER == HY_SHADER_BLOCKS) {
            if (a.mode == HY_BLOCKS_VOLUME)
                render_kernel<SHADER, PC, DT, PADDED, 1, kBlocksVolume><<<g, kThreads, sm, s>>>(a);
            else
                render_kernel<SHADER, PC, DT, PADDED, 1, kBlocksSolid><<<g, kThreads, sm, s>>>(a);
        } else
            pick_composite<SHADER, PC, DT, PADDED>(a, s);
        return;
    }
    if constexpr (SHADER == HY_SHADER_VOLUME) {
        if (a.mode == HY_VOLUME_DEFAULT && !a.aux) {
            if constexpr (DT == HY_DTYPE_U8 && PADDED) {
                if (a.vol.paged_gather) {
                    // A pager's cache in gather textures: its lean march with
                    // 4 samples in flight below 8 warps of rays a scheduler,
                    // 2 above.  Four frames of the 1024x1024x512 noise volume
                    // at 1024^2, half the visible bricks cached: 8.28 ms one
                    // sample at a time, 5.29 with the skip grid, 4.91 two in
                    // flight (5.45 four); 256^2 3.82, 3.57, 2.89 (2.40); opaque
                    // knots 7.99, 8.05, 7.47 (8.19).
                    const long long rays = (long long)a.view.W * a.view.H;
                    if (a.ert > 0.f)
                        render_lean_gather_kernel<SHADER, PC, DT, PADDED, kGatherPaged, kLoopErt>
                            <<<g, kThreads, sm, s>>>(a);
                    else if (rays < 8 * 32ll * a.schedulers)
                        render_batches_kernel<SHADER, PC, DT, kGatherPaged, kLoopBatch4>
                            <<<g, kThreads, sm, s>>>(a);
                    else
                        render_batches_kernel<SHADER, PC, DT, kGatherPaged, kLoopBatch2>
                            <<<g, kThreads, sm, s>>>(a);
                    return;
                }
            }
            if constexpr (HY_RENDER_GATHER && DT == HY_DTYPE_U8 && PADDED) {
                if (a.vol.tex) {  // bricks in gather textures
                    launch_lean<SHADER, PC, DT, PADDED, kGatherResident>(a, s);
                    return;
                }
            }
            launch_lean<SHADER, PC, DT, PADDED, 0>(a, s);
            return;
        }
    }
    if constexpr (SHADER == HY_SHADER_ISOSURFACE) {
        // Eight lanes a ray below 2 warps of rays a scheduler: 256^3 tubes at
        // 128^2 (0.8 warps) 109 us against 191 with four samples in flight.
        // Above, where rays march far (200^2 and 256^2, 2.1 and 3.4 warps) 131
        // and 166 against 198 and 194, where they hit at once (noise) 49 and 68
        // against 43 and 53.
        if ((long long)a.view.W * a.view.H < 2 * 32ll * a.schedulers) {
            const dim3 gg((a.view.W + kIsoW - 1) / kIsoW, (a.view.H + kIsoH - 1) / kIsoH);
            render_iso_group_kernel<PC, DT, PADDED><<<gg, kIsoGroupThreads, sm, s>>>(a);
            return;
        }
    }
    if constexpr (SHADER == HY_SHADER_ISOSURFACE && PADDED) {
        // Samples in flight by the warps of rays a scheduler gets: 512^3 tubes at
        // 256^2 and 512^2 (3.4, 13.5 warps) 414 and 468 us with one, 350 and 415
        // with two, 337 with four at the first; 256^3 of 32^3 bricks at 256^2,
        // 512^2, 670^2 339, 366, 444 with one, 230, 297, 385 with two, 194 with
        // four at the first.  Two from 6 warps on: over 56 volumes and isovalues
        // at 380^2 (7.4 warps) both take as long, but where rays hit soon (noise,
        // 360x400) 138 with four, 123 with two or one.
        const long long rays = (long long)a.view.W * a.view.H, per_warp = 32ll * a.schedulers;
        if (rays < 24 * per_warp && a.vol.P <= kMaxBatchesP) {
            if (rays < 6 * per_warp)
                render_iso_kernel<PC, DT, kLoopBatch4><<<g, kThreads, sm, s>>>(a);
            else
                render_iso_kernel<PC, DT, kLoopBatch2><<<g, kThreads, sm, s>>>(a);
            return;
        }
    }
    if constexpr (SHADER == HY_SHADER_VOLUME && PADDED) {
        if (a.skip.d) {
            render_kernel<SHADER, PC, DT, PADDED, 0, kLoopSkip><<<g, kThreads, sm, s>>>(a);
            return;
        }
    }
    if constexpr (SHADER == HY_SHADER_BLOCKS) {
        if (a.mode == HY_BLOCKS_VOLUME)
            render_kernel<SHADER, PC, DT, PADDED, 0, kBlocksVolume><<<g, kThreads, sm, s>>>(a);
        else
            render_kernel<SHADER, PC, DT, PADDED, 0, kBlocksSolid><<<g, kThreads, sm, s>>>(a);
    } else {
        render_kernel<SHADER, PC, DT, PADDED, 0><<<g, kThreads, sm, s>>>(a);
    }
}

// Instantiations: Blocks reads no bricks; u8 volumes with a 1-voxel apron and
// 64^3 or 128^3 bricks get a compile-time brick edge (immediate offsets).
template <int SHADER>
int dispatch_fused(const ShadeArgs &a, cudaStream_t s) {
    if constexpr (SHADER == HY_SHADER_BLOCKS || SHADER == HY_SHADER_PAGING) {
        launch_fused<SHADER, 0, HY_DTYPE_U8, false>(a, s);
    } else {
        const bool padded = a.vol.pad > 0;
        if (a.vol.dtype == HY_DTYPE_F32) {
            if (padded)
                launch_fused<SHADER, 0, HY_DTYPE_F32, true>(a, s);
            else
                launch_fused<SHADER, 0, HY_DTYPE_F32, false>(a, s);
        } else if (padded && a.vol.P == 66) {
            launch_fused<SHADER, 66, HY_DTYPE_U8, true>(a, s);
        } else if (padded && a.vol.P == 130) {
            launch_fused<SHADER, 130, HY_DTYPE_U8, true>(a, s);
        } else if (padded) {
            launch_fused<SHADER, 0, HY_DTYPE_U8, true>(a, s);
        } else {
            launch_fused<SHADER, 0, HY_DTYPE_U8, false>(a, s);
        }
    }
    return HY_OK;
}

unsigned char sat_host(float f) {
    float x = f * 255.f;
    x = (x < 0.f) ? 0.f : x;
    x = (255.f < x) ? 255.f : x;
    return (unsigned char)x;
}

}  // namespace

int hy_fill_args(hy_ctx *ctx, const hy_volume *vol, const hy_shader_params *p, const hy_view *view,
                 int W, int H, ShadeArgs *a) {
    if (!vol || !p) return hy_fail(ctx, HY_ERR_INVALID, "render: null volume or params");
    if (vol->ctx != ctx) return hy_fail(ctx, HY_ERR_INVALID, "render: volume of another context");
    if (!vol->uploaded) return hy_fail(ctx, HY_ERR_STATE, "render: volume not uploaded");
    // the launch grid is W/16 x H/8 tiles (at most 65535 tile rows)
    if (W <= 0 || H <= 0 || (long long)W * H > (1ll << 31) || (H + kTileH - 1) / kTileH > 65535)
        return hy_fail(ctx, HY_ERR_INVALID, "render: bad resolution");
    if (p->shader < HY_SHADER_VOLUME || p->shader > HY_SHADER_PAGING)
        return hy_fail(ctx, HY_ERR_INVALID, "render: unknown shader");
    if (p->shader == HY_SHADER_PAGING && p->composite)
        return hy_fail(ctx, HY_ERR_UNSUPPORTED, "render: the Paging shader has no compositing");
    if (!(p->sample_rate > 0.f)) return hy_fail(ctx, HY_ERR_INVALID, "render: sample_rate <= 0");
    if (p->shader == HY_SHADER_VOLUME && ctx->ntf <= 0)
        return hy_fail(ctx, HY_ERR_STATE, "render: Volume shader needs a transfer function");
    std::memset(a, 0, sizeof(*a));
    a->skip.stride = 1 << 30;  // no skip grid unless hy_skip_view gives one
    a->vol = DevVolume{vol->pool, vol->info_dev, vol->reg_dev, vol->mean_dev, vol->grid[0],
                       vol->grid[1], vol->grid[2], vol->P, vol->desc.dtype, vol->desc.padding,
                       nullptr, {0ull, 0ull}, vol->k, vol->b, nullptr};
    a->vol.gmx = float(vol->grid[0] - 1);
    a->vol.gmy = float(vol->grid[1] - 1);
    a->vol.gmz = float(vol->grid[2] - 1);
    a->vol.fgx = float(vol->grid[0]);
    a->vol.fgy = float(vol->grid[1]);
    hy_volume_gather_view(vol, &a->vol);
    for (int i = 0; i < 3; ++i) a->bbox_max[i] = vol->bbox_max[i];
    a->du = vol->du;
    a->step = vol->du / 4.f / p->sample_rate;  // basic_renderer.hpp:129
    a->max_steps = p->max_steps;
    a->shader = p->shader;
    a->mode = p->mode;
    a->density = p->density;
    a->isovalue = p->isovalue;
    for (int i = 0; i < 3; ++i) {
        a->surface[i] = p->surface_color[i];
        a->view.eye[i] = p->eye_pos[i];
        a->view.light[i] = p->light_pos[i];
        a->clear_u8[i] = sat_host(p->clear_color[i]);  // raycaster.hpp:211
    }
    a->rank = p->rank;
    a->lowest_blkcnt = p->lowest_blkcnt;
    std::memcpy(a->to_world, p->to_world, sizeof(a->to_world));
    a->composite = p->composite;
    a->srgb = p->srgb;
    a->count = p->count_samples;
    // early ray termination: the lean march only (Volume, Default mode, one
    // march through the volume box; films and compositing need full rays)
    if (!(p->early_termination >= 0.f) || p->early_termination > 1.f)
        return hy_fail(ctx, HY_ERR_INVALID, "render: early_termination must be 0 (off) or in (0, 1]");
    a->ert = (p->shader == HY_SHADER_VOLUME && p->mode == HY_VOLUME_DEFAULT && !p->composite)
                 ? p->early_termination
                 : 0.f;
    if (view) {
        std::memcpy(a->view.trans, view->trans, sizeof(a->view.trans));
        a->view.ctg = view->ctg_fovy_2;
        for (int i = 0; i < 3; ++i) a->view.ray_o[i] = view->ray_o[i];
    }
    a->view.W = W;
    a->view.H = H;
    a->tf = ctx->tf_dev;
    a->ntf = ctx->ntf;
    a->schedulers = 4 * ctx->sms;
    a->counter = ctx->counter_dev;
    return HY_OK;
}

int hy_check_paged_gather(hy_ctx *ctx, const ShadeArgs &a, bool fused) {
    if (!a.vol.paged_gather || a.shader == HY_SHADER_BLOCKS || a.shader == HY_SHADER_PAGING)
        return HY_OK;
    const bool lean = a.shader == HY_SHADER_VOLUME && a.mode == HY_VOLUME_DEFAULT &&
                      !a.composite && !a.aux && a.vol.dtype == HY_DTYPE_U8 && a.vol.pad > 0;
    if (fused && lean) return HY_OK;
    return hy_fail(ctx, HY_ERR_UNSUPPORTED,
                   "a pager's cache in gather textures serves the Volume shader's lean per-view "
                   "march (Default mode, no compositing, no aux output) and the Blocks and "
                   "Paging shaders; create the pager with HY_PAGER_LOADS for this use");
}

int hy_time_begin(hy_ctx *ctx, bool reset_counter) {
    if (reset_counter)
        HY_CUDA(ctx, cudaMemsetAsync(ctx->counter_dev, 0, sizeof(unsigned long long), ctx->stream));
    HY_CUDA(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    return HY_OK;
}

int hy_launch_render(hy_ctx *ctx, const ShadeArgs &a) {
    switch (a.shader) {
        case HY_SHADER_VOLUME:
            dispatch_fused<HY_SHADER_VOLUME>(a, ctx->stream);
            break;
        case HY_SHADER_BLOCKS:
            dispatch_fused<HY_SHADER_BLOCKS>(a, ctx->stream);
            break;
        case HY_SHADER_PAGING:
            dispatch_fused<HY_SHADER_PAGING>(a, ctx->stream);
            break;
        default:
            dispatch_fused<HY_SHADER_ISOSURFACE>(a, ctx->stream);
            break;
    }
    HY_CUDA(ctx, cudaGetLastError());
    HY_CUDA(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    ctx->stats_pending = true;
    ctx->pend_count = a.count;
    ctx->pend_pixels = (int64_t)a.view.W * a.view.H;
    return HY_OK;
}

int hy_finish_stats(hy_ctx *ctx) {
    HY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (!ctx->stats_pending) return HY_OK;
    ctx->stats_pending = false;
    float ms = 0.f;
    HY_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    ctx->stats.ms = ms;
    ctx->stats.pixels = ctx->pend_pixels;
    ctx->stats.samples = -1;
    if (ctx->pend_count) {
        unsigned long long n = 0;
        HY_CUDA(ctx, cudaMemcpy(&n, ctx->counter_dev, sizeof(n), cudaMemcpyDeviceToHost));
        ctx->stats.samples = (int64_t)n;
    }
    return HY_OK;
}

extern "C" int hy_render_device(hy_ctx *ctx, const hy_volume *vol, const hy_shader_params *p,
                                const hy_view *view, int32_t W, int32_t H, uint8_t *rgba_dev,
                                float *v_dev, float *aux_dev) {
    if (!ctx) return HY_ERR_INVALID;
    if (!hy_aligned(rgba_dev, 4) || !hy_aligned(v_dev, 16) || !hy_aligned(aux_dev, 16))
        return hy_fail(ctx, HY_ERR_INVALID,
                       "render: misaligned output (rgba 4-byte, float images 16-byte)");
    if (!view || !rgba_dev) return hy_fail(ctx, HY_ERR_INVALID, "render: null view or output");
    ShadeArgs a;
    int rc = hy_fill_args(ctx, vol, p, view, W, H, &a);
    if (rc) return rc;
    a.rgba = reinterpret_cast<uchar4 *>(rgba_dev);
    a.vout = reinterpret_cast<float4 *>(v_dev);
    a.aux = reinterpret_cast<float4 *>(aux_dev);
    rc = hy_check_paged_gather(ctx, a, true);
    if (!rc) rc = hy_time_begin(ctx, a.count);
    if (!rc) rc = hy_skip_view(ctx, vol, p, &a.skip);
    return rc ? rc : hy_launch_render(ctx, a);
}

uint8_t *hy_mapped_device_ptr(void *host, uintptr_t align) {
    if (!host || !hy_aligned(host, align)) return nullptr;
    cudaPointerAttributes pa{};
    if (cudaPointerGetAttributes(&pa, host) != cudaSuccess) {
        cudaGetLastError();  // not a pointer the runtime knows
        return nullptr;
    }
    if (pa.type != cudaMemoryTypeHost || !hy_aligned(pa.devicePointer, align)) return nullptr;
    return static_cast<uint8_t *>(pa.devicePointer);
}

extern "C" int hy_render(hy_ctx *ctx, const hy_volume *vol, const hy_shader_params *p,
                         const hy_view *view, int32_t W, int32_t H, uint8_t *rgba_out,
                         float *v_out, float *aux_out) {
    if (!ctx) return HY_ERR_INVALID;
    if (!view || !rgba_out) return hy_fail(ctx, HY_ERR_INVALID, "render: null view or output");
    ShadeArgs a;
    int rc = hy_fill_args(ctx, vol, p, view, W, H, &a);
    if (rc) return rc;
    HY_CUDA(ctx, cudaSetDevice(ctx->device));
    // outputs in pinned, mapped host memory are written by the kernel itself
    // (as in hy_batch_render); the others are staged in device memory and
    // copied once
    uint8_t *rgba_d = hy_mapped_device_ptr(rgba_out, 4);
    uint8_t *v_d = v_out ? hy_mapped_device_ptr(v_out, 16) : nullptr;
    uint8_t *aux_d = aux_out ? hy_mapped_device_ptr(aux_out, 16) : nullptr;
    const size_t npx = size_t(W) * H;
    const size_t rgba_b = (npx * 4 + 255) / 256 * 256, f4_b = npx * 16;
    const size_t total =
        (rgba_d ? 0 : rgba_b) + (v_out && !v_d ? f4_b : 0) + (aux_out && !aux_d ? f4_b : 0);
    char *base = nullptr;
    if (total) {
        void *stage = nullptr;
        rc = hy_stage(ctx, total, &stage);
        if (rc) return rc;
        base = static_cast<char *>(stage);
    }
    size_t off = 0;
    auto place = [&](uint8_t *direct, size_t bytes) -> char * {
        if (direct) return reinterpret_cast<char *>(direct);
        char *q = base + off;
        off += bytes;
        return q;
    };
    a.rgba = reinterpret_cast<uchar4 *>(place(rgba_d, rgba_b));
    if (v_out) a.vout = reinterpret_cast<float4 *>(place(v_d, f4_b));
    if (aux_out) a.aux = reinterpret_cast<float4 *>(place(aux_d, f4_b));
    rc = hy_check_paged_gather(ctx, a, true);
    if (!rc) rc = hy_time_begin(ctx, a.count);
    if (!rc) rc = hy_skip_view(ctx, vol, p, &a.skip);
    if (!rc) rc = hy_launch_render(ctx, a);
    if (rc) return rc;
    if (!rgba_d)
        HY_CUDA(ctx, cudaMemcpyAsync(rgba_out, a.rgba, npx * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (v_out && !v_d)
        HY_CUDA(ctx, cudaMemcpyAsync(v_out, a.vout, f4_b, cudaMemcpyDeviceToHost, ctx->stream));
    if (aux_out && !aux_d)
        HY_CUDA(ctx, cudaMemcpyAsync(aux_out, a.aux, f4_b, cudaMemcpyDeviceToHost, ctx->stream));
    return hy_finish_stats(ctx);
}

extern "C" int hy_shade_pass(hy_ctx *ctx, const hy_volume *vol, const hy_shader_params *p,
                             int32_t pass, const hy_view *view, void *film_dev, int32_t W,
                             int32_t H, void *dst_dev, const uint8_t clear_rgb[3]) {
    if (!ctx) return HY_ERR_INVALID;
    // films hold float4 records; the Volume fetch pixel is two float4, the
    // Isosurface one stores a float at byte 4 (16 covers both)
    if (!hy_aligned(film_dev, 16) || (pass == HY_PASS_FETCH && !hy_aligned(dst_dev, 16)))
        return hy_fail(ctx, HY_ERR_INVALID,
                       "pass: misaligned film or fetch destination (16-byte)");
    if (pass < HY_PASS_RAY_EMIT || pass > HY_PASS_FETCH)
        return hy_fail(ctx, HY_ERR_INVALID, "pass: unknown pass");
    if (!film_dev) return hy_fail(ctx, HY_ERR_INVALID, "pass: null film");
    if (pass == HY_PASS_RAY_EMIT && !view) return hy_fail(ctx, HY_ERR_INVALID, "pass: emit needs a view");
    if (pass >= HY_PASS_PIXEL && !dst_dev) return hy_fail(ctx, HY_ERR_INVALID, "pass: null destination");
    if (p && p->composite) return hy_fail(ctx, HY_ERR_UNSUPPORTED, "pass: composite is fused-only");
    ShadeArgs a;
    int rc = hy_fill_args(ctx, vol, p, view, W, H, &a);
    if (rc) return rc;
    a.film = film_dev;
    a.dst = dst_dev;
    if (clear_rgb)
        for (int i = 0; i < 3; ++i) a.clear_u8[i] = clear_rgb[i];
    rc = hy_check_paged_gather(ctx, a, false);
    if (rc) return rc;
    const bool marches = pass <= HY_PASS_RAY_MARCH;
    HY_CUDA(ctx, cudaSetDevice(ctx->device));
    rc = hy_time_begin(ctx, a.count && marches);
    if (!rc && marches) rc = hy_skip_view(ctx, vol, p, &a.skip);
    return rc ? rc : hy_launch_pass(ctx, a, pass);
}
