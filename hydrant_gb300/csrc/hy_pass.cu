// hy_pass.cu -- the reference's four passes over a film (cuda_shading.cu:14-96)
// in its pixel layouts: what hy_shade_pass and the lossless pager launch.
//
// The emit and march passes take the march of the fused kernels: compile-time
// brick edges, the interior sampler (bricks with an apron), the gather textures
// of a resident volume, several samples of a ray in flight and the skip grid;
// the film's bytes are those of the plain march.

#include "hy_tile.cuh"


namespace {

template <int SHADER>
__device__ __forceinline__ size_t film_bytes() {
    return (SHADER == HY_SHADER_BLOCKS || SHADER == HY_SHADER_PAGING) ? 48 : 64;
}

template <int SHADER>
__device__ __forceinline__ void store_film(void *film, size_t idx, const Px &p) {
    float4 *q = reinterpret_cast<float4 *>(static_cast<char *>(film) + idx * film_bytes<SHADER>());
    q[0] = make_float4(p.ox, p.oy, p.oz, p.dx);
    q[1] = make_float4(p.dy, p.dz, __int_as_float(p.nsteps), __int_as_float(p.step_size));
    q[2] = make_float4(p.vx, p.vy, p.vz, p.vw);
    if (SHADER != HY_SHADER_BLOCKS && SHADER != HY_SHADER_PAGING)
        q[3] = make_float4(p.e0, p.e1, p.e2, p.e3);
}

template <int SHADER>
__device__ __forceinline__ Px load_film(const void *film, size_t idx) {
    const float4 *q =
        reinterpret_cast<const float4 *>(static_cast<const char *>(film) + idx * film_bytes<SHADER>());
    Px p;
    float4 a = q[0], b = q[1], c = q[2];
    p.ox = a.x;
    p.oy = a.y;
    p.oz = a.z;
    p.dx = a.w;
    p.dy = b.x;
    p.dz = b.y;
    p.nsteps = __float_as_int(b.z);
    p.step_size = __float_as_int(b.w);
    p.vx = c.x;
    p.vy = c.y;
    p.vz = c.z;
    p.vw = c.w;
    if (SHADER != HY_SHADER_BLOCKS && SHADER != HY_SHADER_PAGING) {
        float4 d = q[3];
        p.e0 = d.x;
        p.e1 = d.y;
        p.e2 = d.z;
        p.e3 = d.w;
    } else {
        p.e0 = p.e1 = p.e2 = p.e3 = 0.f;
    }
    return p;
}

// Resident 128-thread blocks a pass is built for: registers for the samples
// in flight (volume_batches).
constexpr int pass_blocks(int loop, int gather) {
    return loop == kLoopBatch4 ? 4 : loop == kLoopBatch2 ? (gather ? 8 : 6) : 0;
}

// ray_emit_kernel_impl (cuda_shading.cu:14-35)
template <int SHADER, int PC, int DT, bool PADDED, int GATHER, int LOOP>
__global__ void __launch_bounds__(kThreads, pass_blocks(LOOP, GATHER))
    emit_pass_kernel(const __grid_constant__ ShadeArgs A) {
    extern __shared__ float4 smem[];
    float4 *tf = smem;
    float *lut = reinterpret_cast<float *>(smem + A.ntf + kTfPad);
    load_shared(A, tf, lut);
    const Shared S = make_shared(tf, A.ntf, lut);
    int x, y;
    tile_xy(x, y);
    long long samples = 0;
    if (x < A.view.W && y < A.view.H) {
        float ox, oy, oz, dx, dy, dz;
        gen_ray(A.view, x, y, ox, oy, oz, dx, dy, dz);
        Px p;
        samples = emit<SHADER, PC, DT, PADDED, false, GATHER, LOOP>(
            p, A, A.view, S, ox, oy, oz, dx, dy, dz, 0.f, 0.f, 0.f, A.bbox_max[0], A.bbox_max[1],
            A.bbox_max[2]);
        store_film<SHADER>(A.film, size_t(y) * A.view.W + x, p);
    }
    count_samples(A, samples);
}

// Whether a film's pixel is one that a march leaves: the step size its opacity
// asks for, nothing that 0 * t would turn into NaN.  Others (a film that the caller
// wrote) take every sample, as the step size may change at one without effect.
template <int SHADER>
__device__ __forceinline__ bool march_state(const Px &p) {
    if (SHADER != HY_SHADER_VOLUME) return true;
    const float big = 3e38f;
    return fabsf(p.vw) < big && fabsf(p.e3) < big &&
           (!(p.vw >= HY_T85) || p.step_size == (p.vw >= HY_T93 ? 16 : 4));
}

// ray_march_kernel_impl (cuda_shading.cu:41-54): resumes every pixel that has
// steps left (the others keep their bytes).
template <int SHADER, int PC, int DT, bool PADDED, int GATHER, int LOOP>
__global__ void __launch_bounds__(kThreads, pass_blocks(LOOP, GATHER))
    march_pass_kernel(const __grid_constant__ ShadeArgs A) {
    extern __shared__ float4 smem[];
    float4 *tf = smem;
    float *lut = reinterpret_cast<float *>(smem + A.ntf + kTfPad);
    load_shared(A, tf, lut);
    const Shared S = make_shared(tf, A.ntf, lut);
    int x, y;
    tile_xy(x, y);
    long long samples = 0;
    if (x < A.view.W && y < A.view.H) {
        const size_t idx = size_t(y) * A.view.W + x;
        Px p = load_film<SHADER>(A.film, idx);
        if (p.nsteps > 0) {
            if (SHADER != HY_SHADER_VOLUME || LOOP == kLoopOne || march_state<SHADER>(p))
                samples = run_main<SHADER, PC, DT, PADDED, false, GATHER, LOOP>(p, A, A.view, S);
            else
                samples = run_main<SHADER, PC, DT, PADDED, false, GATHER, kLoopOne>(p, A, A.view, S);
            store_film<SHADER>(A.film, idx, p);
        }
    }
    count_samples(A, samples);
}

// pixel_kernel_impl (cuda_shading.cu:60-74): film -> uchar3 via write_to.
template <int SHADER>
__global__ void __launch_bounds__(kThreads) pixel_pass_kernel(const __grid_constant__ ShadeArgs A) {
    int x, y;
    tile_xy(x, y);
    if (x >= A.view.W || y >= A.view.H) return;
    const size_t idx = size_t(y) * A.view.W + x;
    Px p = load_film<SHADER>(A.film, idx);
    unsigned char *d = static_cast<unsigned char *>(A.dst) + idx * 3;
    if (p.vw != 0.f) {
        d[0] = saturate_u8(p.vx);
        d[1] = saturate_u8(p.vy);
        d[2] = saturate_u8(p.vz);
    } else {
        d[0] = A.clear_u8[0];
        d[1] = A.clear_u8[1];
        d[2] = A.clear_u8[2];
    }
}

// fetch_kernel_impl (cuda_shading.cu:80-94): VolumeShaderKernel::fetch
// (volume_shader.cu:23-30), IsosurfaceShaderKernel::fetch
// (isosurface_shader.cu:41-48) and PagingShaderKernel::fetch
// (paging_shader.cu:16-22, uchar3 pixels).  The Blocks shader has no fetch.
template <int SHADER>
__global__ void __launch_bounds__(kThreads) fetch_pass_kernel(const __grid_constant__ ShadeArgs A) {
    int x, y;
    tile_xy(x, y);
    if (x >= A.view.W || y >= A.view.H) return;
    const size_t idx = size_t(y) * A.view.W + x;
    Px p = load_film<SHADER>(A.film, idx);
    if (SHADER == HY_SHADER_VOLUME) {
        float4 *d = reinterpret_cast<float4 *>(static_cast<char *>(A.dst) + idx * 32);
        d[0] = make_float4(p.e0, p.e1, p.e2, p.e3);
        d[1] = make_float4(p.vx, p.vy, p.vz, p.vw);
    } else if (SHADER == HY_SHADER_ISOSURFACE) {
        unsigned char *d = static_cast<unsigned char *>(A.dst) + idx * 8;
        d[0] = saturate_u8(p.vx);
        d[1] = saturate_u8(p.vy);
        d[2] = saturate_u8(p.vz);
        d[3] = 0;
        *reinterpret_cast<float *>(d + 4) = p.e3;
    } else if (SHADER == HY_SHADER_PAGING) {
        unsigned char *d = static_cast<unsigned char *>(A.dst) + idx * 3;
        d[0] = saturate_u8(p.vx);
        d[1] = saturate_u8(p.vy);
        d[2] = saturate_u8(p.vz);
    }
}

template <int SHADER, int PC, int DT, bool PADDED, int GATHER, int LOOP>
void launch_march(const ShadeArgs &a, int pass, cudaStream_t s) {
    const dim3 g = grid_of(a);
    const size_t sm = smem_bytes(a);
    if (pass == HY_PASS_RAY_EMIT)
        emit_pass_kernel<SHADER, PC, DT, PADDED, GATHER, LOOP><<<g, kThreads, sm, s>>>(a);
    else
        march_pass_kernel<SHADER, PC, DT, PADDED, GATHER, LOOP><<<g, kThreads, sm, s>>>(a);
}

// Samples in flight by the warps of rays a scheduler gets, as for the fused
// kernels (launch_lean, hy_render.cu).
template <int SHADER, int PC, int DT, bool PADDED, int GATHER>
void pick_loop(const ShadeArgs &a, int pass, cudaStream_t s) {
    if constexpr (PADDED) {
        const long long rays = (long long)a.view.W * a.view.H, per_warp = 32ll * a.schedulers;
        const bool batches = a.vol.P <= kMaxBatchesP &&
                             (SHADER == HY_SHADER_ISOSURFACE || a.mode == HY_VOLUME_DEFAULT);
        if (batches && rays < 8 * per_warp) {
            launch_march<SHADER, PC, DT, PADDED, GATHER, kLoopBatch4>(a, pass, s);
            return;
        }
        if (batches && (rays < 24 * per_warp || (SHADER == HY_SHADER_VOLUME && a.skip.d))) {
            launch_march<SHADER, PC, DT, PADDED, GATHER, kLoopBatch2>(a, pass, s);
            return;
        }
    }
    launch_march<SHADER, PC, DT, PADDED, GATHER, kLoopOne>(a, pass, s);
}

template <int SHADER, int PC, int DT, bool PADDED>
void pick_sampler(const ShadeArgs &a, int pass, cudaStream_t s) {
    if constexpr (SHADER == HY_SHADER_VOLUME && DT == HY_DTYPE_U8 && PADDED) {
        if (a.vol.tex) {  // bricks in gather textures
            pick_loop<SHADER, PC, DT, PADDED, kGatherResident>(a, pass, s);
            return;
        }
    }
    pick_loop<SHADER, PC, DT, PADDED, 0>(a, pass, s);
}

template <int SHADER>
void dispatch_pass(const ShadeArgs &a, int pass, cudaStream_t s) {
    const dim3 g = grid_of(a);
    if (pass == HY_PASS_PIXEL) {
        pixel_pass_kernel<SHADER><<<g, kThreads, 0, s>>>(a);
    } else if (pass == HY_PASS_FETCH) {
        fetch_pass_kernel<SHADER><<<g, kThreads, 0, s>>>(a);
    } else if constexpr (SHADER == HY_SHADER_BLOCKS) {
        if (a.mode == HY_BLOCKS_VOLUME)
            launch_march<SHADER, 0, HY_DTYPE_U8, false, 0, kBlocksVolume>(a, pass, s);
        else
            launch_march<SHADER, 0, HY_DTYPE_U8, false, 0, kBlocksSolid>(a, pass, s);
    } else if constexpr (SHADER == HY_SHADER_PAGING) {
        launch_march<SHADER, 0, HY_DTYPE_U8, false, 0, kLoopOne>(a, pass, s);
    } else {
        const bool padded = a.vol.pad > 0;
        if (a.vol.dtype == HY_DTYPE_F32) {
            if (padded)
                pick_sampler<SHADER, 0, HY_DTYPE_F32, true>(a, pass, s);
            else
                pick_sampler<SHADER, 0, HY_DTYPE_F32, false>(a, pass, s);
        } else if (padded && a.vol.P == 66) {
            pick_sampler<SHADER, 66, HY_DTYPE_U8, true>(a, pass, s);
        } else if (padded && a.vol.P == 130) {
            pick_sampler<SHADER, 130, HY_DTYPE_U8, true>(a, pass, s);
        } else if (padded) {
            pick_sampler<SHADER, 0, HY_DTYPE_U8, true>(a, pass, s);
        } else {
            pick_sampler<SHADER, 0, HY_DTYPE_U8, false>(a, pass, s);
        }
    }
}

}  // namespace

int hy_launch_pass(hy_ctx *ctx, const ShadeArgs &a, int pass) {
    switch (a.shader) {
        case HY_SHADER_VOLUME:
            dispatch_pass<HY_SHADER_VOLUME>(a, pass, ctx->stream);
            break;
        case HY_SHADER_BLOCKS:
            dispatch_pass<HY_SHADER_BLOCKS>(a, pass, ctx->stream);
            break;
        case HY_SHADER_PAGING:
            dispatch_pass<HY_SHADER_PAGING>(a, pass, ctx->stream);
            break;
        default:
            dispatch_pass<HY_SHADER_ISOSURFACE>(a, pass, ctx->stream);
            break;
    }
    HY_CUDA(ctx, cudaGetLastError());
    HY_CUDA(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    ctx->stats_pending = true;
    ctx->pend_count = a.count && pass <= HY_PASS_RAY_MARCH;
    ctx->pend_pixels = (int64_t)a.view.W * a.view.H;
    return HY_OK;
}

