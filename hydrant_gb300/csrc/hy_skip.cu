// hy_skip.cu -- the skip grid: where a march may pass over samples that
// change nothing.
//
// Most samples of a volume rendering contribute exactly nothing: their
// neighbourhood's values fall where the transfer function's opacity is an
// exact zero (v + 0 * t is v), or cannot cross the isovalue.  The upload
// divides every brick into cells of about 8 voxels and keeps the smallest and
// largest voxel a sample of the cell can touch.  Per transfer function (or
// isovalue) four small kernels turn that into one byte per cell and direction
// octant: 0, samples must be taken, or d > 0, the d^3 cells from this one on
// in the ray's direction are free of effect, so a ray marches to the end of
// that box with three additions per step (the positions round step by step
// as before; nothing else of the sample is computed).  Kept per octant because
// a ray leaving a surface cares only for what lies ahead: boxes around
// the cell on all sides made the 16-view batch 25.7 instead of 24.7 ms and
// small images up to 25 % slower (more and shorter hops).  The grid covers
// the whole volume, so boxes span bricks; cells of empty bricks are 0,
// because rays cross those with the reference's own brick skip.
//
// Cells of 8 voxels against 4: 16-view batch 25.7 and 25.9 ms, the 128^3 view
// 103 and 95 us, the f32 view 192 and 219 us; 4 also takes eight times the
// memory.
//
// Bound: the min/max kernel reads each voxel of the pool from DRAM once and
// from L1 about twice per axis; the distance passes move a byte per cell and
// live in L2 (1024^3 volume: 2 M cells, 14 planes).

#include <algorithm>
#include <cmath>
#include <cstring>

#include "hy_internal.h"

namespace {

constexpr int kStride = 16;     // steps between two looks (hy_shade.cuh, skip_hint)
constexpr int kMaxDist = 16;    // largest stored distance (box of 15 cells each way)
constexpr long long kMaxGridCells = 1ll << 27;

// Voxel range [lo, hi] (padded indices) that samples of cell c along one axis
// can touch: positions l in [c, c + 1] / nc of the brick map to
// u = bs * l + pad - 1/2 and read floor(u) and floor(u) + 1; 1e-3 voxels cover
// the mapping's rounding (P <= 2^12 bricks: below 1e-3).
__host__ __device__ inline void cell_taps(int c, int nc, int bs, int pad, int P, int *lo, int *hi) {
    const float w = float(bs) / float(nc);
    const int a = int(floorf(float(c) * w + float(pad) - .5f - 1e-3f));
    const int b = int(floorf(float(c + 1) * w + float(pad) - .5f + 1e-3f)) + 1;
    *lo = a < 0 ? 0 : a;
    *hi = b > P - 1 ? P - 1 : b;
}

// What a cell keeps: the smallest and largest voxel, or lo > hi for a cell
// that must be sampled whatever the knots (an empty or absent brick, or a
// voxel that is not finite).
template <typename T>
struct MinMax {
    T lo, hi;
};

struct CellArgs {
    const unsigned char *pool;
    const hy::RegEntry *reg;
    const int2 *info;
    int gx, gy, gz;   // bricks
    int nc;           // cells per brick edge
    int bs, pad, P;
};

// gridDim.y blocks per brick, eight lanes per cell, each every eighth row of its taps
// (a thread per cell, a serial chain of 1000 loads, took 91 us for 512 f32
// bricks of 32^3 and 0.99 ms for 1024^3 u8).
constexpr int kCellLanes = 8;
template <typename T>
__global__ void cell_minmax_kernel(const __grid_constant__ CellArgs a, MinMax<T> *__restrict__ out) {
    const int b = blockIdx.x;
    const int bx = b % a.gx, by = (b / a.gx) % a.gy, bz = b / (a.gx * a.gy);
    const int2 in = a.info[b];
    const bool sampled = in.x == 0 && in.y >= 0;
    const T *v = reinterpret_cast<const T *>(a.pool + (sampled ? a.reg[in.y].offset : 0));
    const int nc = a.nc, cells = nc * nc * nc;
    const int cx = a.gx * nc, cy = a.gy * nc;
    const int k = threadIdx.x & (kCellLanes - 1);
    // whole warps go round together (the shuffles below)
    const int step = blockDim.x / kCellLanes;
    for (int c0 = blockIdx.y * step; c0 < cells; c0 += gridDim.y * step) {
        const int c = c0 + threadIdx.x / kCellLanes;
        const int cc = min(c, cells - 1);
        const int x = cc % nc, y = (cc / nc) % nc, z = cc / (nc * nc);
        MinMax<T> m{T(1), T(0)};
        if (sampled) {
            int x0, x1, y0, y1, z0, z1;
            cell_taps(x, nc, a.bs, a.pad, a.P, &x0, &x1);
            cell_taps(y, nc, a.bs, a.pad, a.P, &y0, &y1);
            cell_taps(z, nc, a.bs, a.pad, a.P, &z0, &z1);
            T lo = v[((long long)z0 * a.P + y0) * a.P + x0], hi = lo;
            int finite = 1;
            const int ny = y1 - y0 + 1, rows = ny * (z1 - z0 + 1);
            for (int r = k; r < rows; r += kCellLanes) {
                const int dz = r / ny;
                const T *row = v + ((long long)(z0 + dz) * a.P + y0 + (r - dz * ny)) * a.P;
                for (int i = x0; i <= x1; ++i) {
                    const T t = row[i];
                    lo = t < lo ? t : lo;
                    hi = t > hi ? t : hi;
                    if constexpr (sizeof(T) == 4) finite &= fabsf(t) < 3e38f;
                }
            }
            for (int o = kCellLanes / 2; o > 0; o >>= 1) {
                const T l2 = T(__shfl_xor_sync(0xffffffffu, lo, o)),
                        h2 = T(__shfl_xor_sync(0xffffffffu, hi, o));
                lo = l2 < lo ? l2 : lo;
                hi = h2 > hi ? h2 : hi;
                finite &= __shfl_xor_sync(0xffffffffu, finite, o);
            }
            if (finite) m = MinMax<T>{lo, hi};
        }
        if (k == 0 && c < cells)
            out[((long long)(bz * nc + z) * cy + by * nc + y) * cx + bx * nc + x] = m;
    }
}

// Value bins of the cells' min/max histogram: 64 over [0, 1], the outer ones
// open (a u8 voxel u is u / 255).
constexpr int kBins = 64;
__device__ __forceinline__ int value_bin(float v) {
    return min(max(int(v * float(kBins)), 0), kBins - 1);
}

// hist[i][j]: cells with smallest voxel in bin i and largest in bin j.
template <typename T>
__global__ void cell_hist_kernel(const MinMax<T> *__restrict__ mm, long long n, float scale,
                                 int *__restrict__ hist) {
    __shared__ int h[kBins * kBins];
    for (int i = threadIdx.x; i < kBins * kBins; i += blockDim.x) h[i] = 0;
    __syncthreads();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const MinMax<T> m = mm[i];
        if (!(m.lo > m.hi))
            atomicAdd(&h[value_bin(float(m.lo) * scale) * kBins + value_bin(float(m.hi) * scale)], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kBins * kBins; i += blockDim.x)
        if (h[i]) atomicAdd(&hist[i], h[i]);
}

struct ClassArgs {
    hy_skip_ranges r;
    float scale;  // voxel -> sample value: 1/255 (u8) or 1
    long long n;
};

// 1: every sample of the cell lies in one of the ranges without effect; 0: it
// must be sampled.  A sample is seven lerps x*(1-a) + y*a of the cell's taps:
// each rounds its weight, two products and a sum, so it leaves [lo, hi] by at
// most 3 * 3 * 2^-24 of the largest magnitude, u / 255 and n * s add one
// rounding each: 2e-6 covers them three times over.
template <typename T>
__global__ void classify_kernel(const __grid_constant__ ClassArgs a,
                                const MinMax<T> *__restrict__ mm, unsigned char *__restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const MinMax<T> m = mm[i];
    unsigned char free_ = 0;
    if (!(m.lo > m.hi)) {
        const float lo = float(m.lo) * a.scale, hi = float(m.hi) * a.scale;
        const float e = 2e-6f * fmaxf(fabsf(lo), fabsf(hi)) + 1e-36f;  // and underflows
        for (int k = 0; k < a.r.n; ++k)
            if (lo - e >= a.r.lo[k] && hi + e <= a.r.hi[k]) free_ = 1;
    }
    out[i] = free_;
}

// One axis of the distance, both ways along it: the cells at stride `st`, n
// of them; plane blockIdx.y of `in` holds free flags (first axis) or the
// distances of the axes before, and gives the planes blockIdx.y (rays moving
// up this axis) and blockIdx.y + gridDim.y (down) of `out`.  d(i) = the least
// over k >= 0 of max(k, in(i +- k)), cells outside the grid 0.
template <bool FIRST>
__global__ void distance_kernel(const unsigned char *__restrict__ in,
                                unsigned char *__restrict__ out, long long total, int n, int st) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const unsigned char *p = in + blockIdx.y * total;
    const int c = int((i / st) % n);
    auto at = [&](int k) -> int {
        const int v = p[i + (long long)k * st];
        return FIRST ? (v ? kMaxDist : 0) : v;
    };
    int up = at(0), dn = up;
    for (int k = 1; k < up; ++k) up = min(up, max(k, c + k >= n ? 0 : at(k)));
    for (int k = 1; k < dn; ++k) dn = min(dn, max(k, c - k < 0 ? 0 : at(-k)));
    out[blockIdx.y * total + i] = (unsigned char)up;
    out[(blockIdx.y + gridDim.y) * total + i] = (unsigned char)dn;
}

template <typename T>
int classify(hy_volume *v, const hy_skip_ranges &r, unsigned char *grid) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    const long long n = s.cells;
    const unsigned blocks = unsigned((n + 255) / 256);
    ClassArgs a{r, sizeof(T) == 1 ? 1.f / 255.f : 1.f, n};
    const long long cx = (long long)s.c[0], cxy = cx * s.c[1];
    // free flags in the first plane of the result, then x (2 planes), y (4), z (8)
    classify_kernel<T><<<blocks, 256, 0, ctx->stream>>>(
        a, static_cast<const MinMax<T> *>(s.minmax), grid);
    distance_kernel<true><<<dim3(blocks, 1), 256, 0, ctx->stream>>>(grid, s.tmp, n, s.c[0], 1);
    distance_kernel<false><<<dim3(blocks, 2), 256, 0, ctx->stream>>>(s.tmp, s.tmp2, n, s.c[1],
                                                                     int(cx));
    distance_kernel<false><<<dim3(blocks, 4), 256, 0, ctx->stream>>>(s.tmp2, grid, n, s.c[2],
                                                                     int(cxy));
    HY_CUDA(ctx, cudaGetLastError());
    return HY_OK;
}

// The cells' histogram on the host, summed so that hist[i * kBins + j] counts
// the cells with lo in bin >= i and hi in bin <= j.
template <typename T>
int cell_hist(hy_volume *v) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    int *dev = reinterpret_cast<int *>(s.grid[0]);  // 16 KB of the grids, unused until a render
    int *own = nullptr;
    if (s.cells * 8 < (long long)(sizeof(int) * kBins * kBins)) {
        HY_CUDA(ctx, cudaMalloc(&own, sizeof(int) * kBins * kBins));
        dev = own;
    }
    s.hist.assign(kBins * kBins, 0);
    cudaError_t e = cudaMemsetAsync(dev, 0, sizeof(int) * kBins * kBins, ctx->stream);
    if (e == cudaSuccess) {
        const unsigned blocks = unsigned(std::min<long long>((s.cells + 255) / 256, 4 * ctx->sms));
        cell_hist_kernel<T><<<blocks, 256, 0, ctx->stream>>>(
            static_cast<const MinMax<T> *>(s.minmax), s.cells, sizeof(T) == 1 ? 1.f / 255.f : 1.f, dev);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(s.hist.data(), dev, sizeof(int) * kBins * kBins, cudaMemcpyDeviceToHost,
                            ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (own) cudaFree(own);
    if (e != cudaSuccess) return hy_cuda_fail(ctx, e, "volume: skip grid");
    for (int i = kBins - 1; i >= 0; --i)
        for (int j = 0; j < kBins; ++j) {
            int &h = s.hist[i * kBins + j];
            h += (i + 1 < kBins ? s.hist[(i + 1) * kBins + j] : 0) +
                 (j > 0 ? s.hist[i * kBins + j - 1] : 0) -
                 (i + 1 < kBins && j > 0 ? s.hist[(i + 1) * kBins + j - 1] : 0);
        }
    s.sampled = s.hist[kBins - 1];
    return HY_OK;
}

// Cells free of effect for these ranges, to a value bin's width and no more
// than there are.
long long free_cells(const hy_skip &s, const hy_skip_ranges &r) {
    long long n = 0;
    for (int k = 0; k < r.n; ++k) {
        // the bins that lie in the range (the outer ones are open)
        const float lo = std::ceil(std::max(r.lo[k], 0.f) * kBins);
        const float hi = std::floor(std::min(r.hi[k], 1.f) * kBins) - 1.f;
        const int i = int(std::min(std::max(lo, 0.f), float(kBins)));
        const int j = int(std::min(std::max(hi, -1.f), float(kBins - 1)));
        if (i < kBins && j >= i) n += s.hist[i * kBins + j];
    }
    return n;
}

bool same_ranges(const hy_skip_ranges &a, const hy_skip_ranges &b) {
    return a.n == b.n && std::memcmp(a.lo, b.lo, sizeof(float) * a.n) == 0 &&
           std::memcmp(a.hi, b.hi, sizeof(float) * a.n) == 0;
}

}  // namespace

void hy_skip_free(hy_volume *v) {
    hy_skip &s = v->skip;
    if (s.minmax) cudaFree(s.minmax);
    if (s.tmp) cudaFree(s.tmp);
    s = hy_skip();
}

int hy_skip_build(hy_volume *v) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    hy_skip_free(v);
    const int bs = v->desc.block_size;
    // the interior sampler's bricks only (an apron: no wrapped coordinates)
    if (v->desc.padding < 1 || v->resident <= 0 || v->P > 4096) return HY_OK;
    int nc = 1;  // a power of two (positions scale exactly), cells of >= 8 voxels
    while (nc * 2 * 8 <= bs) nc *= 2;
    long long n = 1;
    int gmax = 1;
    for (int i = 0; i < 3; ++i) {
        s.c[i] = v->grid[i] * nc;
        n *= s.c[i];
        gmax = std::max(gmax, v->grid[i]);
    }
    if (n > kMaxGridCells) return HY_OK;
    // A run of up to 127 steps adds up to 127 roundings of half an ulp of
    // the largest coordinate; 4e-6 brick covers the run length's own
    // arithmetic.  Boxes shrink by this much, so that a run that stays in one
    // by this arithmetic stays in it step by step.
    const float ulp = std::nextafterf(float(gmax), 1e30f) - float(gmax);
    s.shrink = 128.f * ulp + 4e-6f;
    if (s.shrink * float(nc) > .125f) return HY_OK;  // a volume of thousands of bricks an edge
    s.nc = nc;
    s.cells = n;
    const bool u8 = v->desc.dtype == HY_DTYPE_U8;
    cudaError_t e = cudaMalloc(&s.minmax, size_t(n) * (u8 ? sizeof(MinMax<unsigned char>)
                                                          : sizeof(MinMax<float>)));
    // the distances per transfer function and per isovalue, and two work grids
    if (e == cudaSuccess) e = cudaMalloc(&s.tmp, size_t(n) * (2 + 4 + 8 + 8));
    if (e != cudaSuccess) {  // no room: the march samples every cell
        hy_skip_free(v);
        cudaGetLastError();
        return HY_OK;
    }
    s.tmp2 = s.tmp + 2 * n;
    s.grid[0] = s.tmp2 + 4 * n;
    s.grid[1] = s.grid[0] + 8 * n;
    CellArgs a{v->pool, v->reg_dev, v->info_dev, v->grid[0], v->grid[1], v->grid[2], nc, bs,
               v->desc.padding, v->P};
    const int threads = std::min(512, std::max(32, nc * nc * nc * kCellLanes));
    // enough blocks for the GPU when there are few bricks
    const int rounds = (nc * nc * nc * kCellLanes + threads - 1) / threads;
    const dim3 grid(unsigned(v->nbricks),
                    unsigned(std::max(1, std::min(rounds, 8 * ctx->sms / v->nbricks))));
    if (u8)
        cell_minmax_kernel<unsigned char><<<grid, threads, 0, ctx->stream>>>(
            a, static_cast<MinMax<unsigned char> *>(s.minmax));
    else
        cell_minmax_kernel<float><<<grid, threads, 0, ctx->stream>>>(
            a, static_cast<MinMax<float> *>(s.minmax));
    HY_CUDA(ctx, cudaGetLastError());
    return u8 ? cell_hist<unsigned char>(v) : cell_hist<float>(v);
}

// The value ranges in which a sample leaves a Volume march as it is: between
// the first and last of a run of knots whose opacity is zero (the lerp of two
// zeros is zero; colours times zero are zero while they are finite), open
// below 0 and above 1 where the run reaches an end (the lookup clamps below
// and is zero above).  None unless the opacities keep v.w in [0, 1]
// (0 <= alpha, alpha * density <= 1): an overflowing v.w would turn 0 * t
// into NaN.
void hy_skip_tf_ranges(const float *rgba, int n, hy_skip_ranges *r, float *alpha_max) {
    r->n = 0;
    *alpha_max = 0.f;
    for (int i = 0; i < n; ++i) {
        const float a = rgba[4 * i + 3];
        if (!(a >= 0.f) || !std::isfinite(a)) {
            *alpha_max = INFINITY;
            return;
        }
        *alpha_max = std::max(*alpha_max, a);
    }
    for (int i = 0; i < n && r->n < HY_SKIP_RANGES;) {
        auto zero = [&](int k) {
            const float *q = rgba + 4 * k;
            return q[3] == 0.f && std::isfinite(q[0]) && std::isfinite(q[1]) && std::isfinite(q[2]);
        };
        if (!zero(i)) {
            ++i;
            continue;
        }
        int j = i;
        while (j + 1 < n && zero(j + 1)) ++j;
        // knot k sits at s = (k + 1/2) / n; one ulp inwards for the quotient
        const float lo = i == 0 ? -INFINITY : std::nextafterf((float(i) + .5f) / float(n), INFINITY);
        const float hi =
            j == n - 1 ? INFINITY : std::nextafterf((float(j) + .5f) / float(n), -INFINITY);
        if (lo < hi) {
            r->lo[r->n] = lo;
            r->hi[r->n] = hi;
            ++r->n;
        }
        i = j + 1;
    }
}

int hy_skip_view(hy_ctx *ctx, const hy_volume *cv, const hy_shader_params *p, hy::SkipGrid *out) {
    std::memset(out, 0, sizeof(*out));
    out->stride = 1 << 30;
    hy_volume *v = const_cast<hy_volume *>(cv);  // the grids are a cache of its bricks
    hy_skip &s = v->skip;
    if (!s.nc) return HY_OK;
    hy_skip_ranges r;
    int which;
    if (p->shader == HY_SHADER_VOLUME) {
        // (early termination votes among a warp's rays step by step)
        if (p->mode != HY_VOLUME_DEFAULT || p->early_termination > 0.f || !(p->density >= 0.f) ||
            !(ctx->tf_alpha_max * p->density <= 1.f))
            return HY_OK;
        which = 0;
        r = ctx->tf_ranges;
        // With less than a tenth of the cells free the looks cost more than
        // the samples passed over: a march without a free cell takes 3 to 5 %
        // longer with the grid than without.
        if (free_cells(s, r) * 10 < s.sampled) return HY_OK;
    } else if (p->shader == HY_SHADER_ISOSURFACE) {
        // crossed: value and 0 on different sides of the isovalue
        which = 1;
        const float iso = p->isovalue;
        r.n = 1;
        r.lo[0] = -INFINITY;
        r.hi[0] = INFINITY;
        if (iso > 0.f)
            r.hi[0] = std::nextafterf(iso, -INFINITY);  // value < iso
        else if (iso < 0.f)
            r.lo[0] = std::nextafterf(iso, INFINITY);   // value > iso
        else
            r.n = 0;
    } else {
        return HY_OK;
    }
    if (r.n == 0) return HY_OK;
    // A capture would replay against whatever knots the grid holds by then:
    // captured launches sample every cell.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    HY_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) return HY_OK;
    if (!s.valid[which] || !same_ranges(r, s.key[which])) {
        s.valid[which] = false;
        const int rc = v->desc.dtype == HY_DTYPE_U8 ? classify<unsigned char>(v, r, s.grid[which])
                                                    : classify<float>(v, r, s.grid[which]);
        if (rc) return rc;
        s.key[which] = r;
        s.valid[which] = true;
    }
    out->d = s.grid[which];
    out->plane = int(s.cells);
    out->cx = s.c[0];
    out->cy = s.c[1];
    out->fcx = float(s.c[0]);
    out->fcy = float(s.c[1]);
    out->fcz = float(s.c[2]);
    out->nc = float(s.nc);
    out->cell = 1.f / float(s.nc);
    out->shrink = s.shrink;
    out->stride = kStride;
    out->fstride = float(kStride);
    return HY_OK;
}
