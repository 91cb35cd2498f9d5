// hy_skip.cu -- the skip grid: where a march may pass over samples that
// change nothing.
//
// Most samples of a volume rendering contribute exactly nothing: their
// neighbourhood's values fall where the transfer function's opacity is an
// exact zero (v + 0 * t is v), or cannot cross the isovalue.  The upload
// divides every brick into cells of about 8 voxels and keeps the smallest and
// largest voxel a sample of the cell can touch.  Per transfer function (or
// isovalue) six small kernels turn that into one byte per cell and direction
// octant: 0, samples must be taken, or d > 0, the d^3 cells from this one on
// in the ray's direction are free of effect, so a ray marches to the end of
// that box with three additions per step (the positions round step by step
// as before; nothing else of the sample is computed).  Kept per octant because
// a ray leaving a surface cares only for what lies ahead: boxes around
// the cell on all sides made the 16-view batch 4 % and small images up to 25 %
// slower (more and shorter hops).  The grid covers
// the whole volume, so boxes span bricks; cells of empty bricks are 0,
// because rays cross those with the reference's own brick skip.
//
// Cells of 4 voxels instead of 8: 16-view batch 1 % slower, the 128^3 view 8 %
// faster, the f32 view 14 % slower, and eight times the memory.
//
// Bound: the min/max kernel by L1 (each voxel about twice per axis); the
// distances by writing a byte per cell and octant.

#include <algorithm>
#include <cmath>
#include <cstring>

#include "hy_internal.h"

namespace {

constexpr int kStride = 16;     // steps between two looks (hy_shade.cuh, skip_hint)
constexpr long long kMaxGridCells = 1ll << 27;
// A ray crosses few cells of a smaller volume (below 64^3 voxels), and the grid's
// part of its upload shows: 16^3 u8 209 and 258 us, 32^3 f32 90 and 148 (215 and
// 176 by the upload before the grid).
constexpr long long kMinGridCells = 512;

// Voxel range [lo, hi] (padded indices) that samples of cell c along one axis
// can touch: positions l in [c, c + 1] / nc of the brick map to
// u = P * (k * l + b) - 1/2 and read floor(u) and floor(u) + 1; 1e-3 voxels cover
// the mapping's rounding (P <= 2^12: below 1e-3).  A fine brick's mapping, or
// a coarse stand-in's sub-box of its coarse brick.
__device__ inline void cell_taps(int c, int nc, float k, float b, int P, int *lo, int *hi) {
    const float s = 1.f / float(nc);
    const int i = int(floorf(float(P) * (k * (float(c) * s) + b) - .5f - 1e-3f));
    const int j = int(floorf(float(P) * (k * (float(c + 1) * s) + b) - .5f + 1e-3f)) + 1;
    *lo = min(max(i, 0), P - 1);
    *hi = min(max(j, 0), P - 1);
}

// What a cell keeps: the smallest and largest voxel, or lo > hi for a cell
// that must be sampled whatever the knots (an empty or absent brick, or a
// voxel that is not finite).
template <typename T>
struct MinMax {
    T lo, hi;
};

// The min/max of a brick's nc^3 cells, eight lanes per cell, each every eighth
// row of its taps (a thread per cell, a serial chain of 1000 loads, took 91 us
// for 512 f32 bricks of 32^3).  Blocks blockIdx.y of gridDim.y share a brick.
// map: k and the offsets of the three axes; ld(x, y, z): a voxel; put(x, y, z,
// m): the result of a cell.
constexpr int kCellLanes = 8;
template <typename T, typename Load, typename Put>
__device__ __forceinline__ void brick_cells(int nc, int P, float4 map, bool sampled, Load ld,
                                            Put put) {
    const int cells = nc * nc * nc;
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
            cell_taps(x, nc, map.x, map.y, P, &x0, &x1);
            cell_taps(y, nc, map.x, map.z, P, &y0, &y1);
            cell_taps(z, nc, map.x, map.w, P, &z0, &z1);
            T lo = ld(x0, y0, z0), hi = lo;
            int finite = 1;
            const int ny = y1 - y0 + 1, rows = ny * (z1 - z0 + 1);
            for (int r = k; r < rows; r += kCellLanes) {
                const int dz = r / ny;
                for (int i = x0; i <= x1; ++i) {
                    const T t = ld(i, y0 + (r - dz * ny), z0 + dz);
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
        if (k == 0 && c < cells) put(x, y, z, m);
    }
}

// Value bins of the cells' min/max histogram: 64 over [0, 1], the outer ones
// open (a u8 voxel u is u / 255).
constexpr int kBins = 64;

struct CellArgs {
    const unsigned char *pool;
    const hy::RegEntry *reg;
    const int2 *info;
    int gx, gy;  // bricks
    int nc, P;
    int *hist;   // cleared for the histogram's kernel
};

// A resident volume: brick blockIdx.x into the volume's grid of cells.
template <typename T>
__global__ void cell_minmax_kernel(const __grid_constant__ CellArgs a, MinMax<T> *__restrict__ out) {
    const int b = blockIdx.x, nc = a.nc, P = a.P;
    if (b == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < kBins * kBins; i += blockDim.x) a.hist[i] = 0;
    const int bx = b % a.gx, by = (b / a.gx) % a.gy, bz = b / (a.gx * a.gy);
    const int2 in = a.info[b];
    const bool sampled = in.x == 0 && in.y >= 0;
    const hy::RegEntry e = a.reg[sampled ? in.y : 0];
    const T *v = reinterpret_cast<const T *>(a.pool + e.offset);
    const int cx = a.gx * nc, cy = a.gy * nc;
    brick_cells<T>(
        nc, P, make_float4(e.k, e.bx, e.by, e.bz), sampled,
        [&](int x, int y, int z) { return v[((long long)z * P + y) * P + x]; },
        [&](int x, int y, int z, MinMax<T> m) {
            out[((long long)(bz * nc + z) * cy + by * nc + y) * cx + bx * nc + x] = m;
        });
}

// A paged cache: the slots just filled (move list entry blockIdx.x), read back
// from the pool or through the cache textures' surfaces; cells in
// [slot][z][y][x] order.
template <typename T, bool SURF>
__global__ void slot_minmax_kernel(const hy::GatherItem *__restrict__ items,
                                   const __grid_constant__ hy::CacheLayout l, int nc, int P,
                                   float4 map, MinMax<T> *__restrict__ out) {
    const int slot = items[blockIdx.x].dst;
    const int g = l.ncoarse + slot;
    MinMax<T> *o = out + (long long)slot * nc * nc * nc;
    auto put = [&](int x, int y, int z, MinMax<T> m) { o[(z * nc + y) * nc + x] = m; };
    if constexpr (SURF) {
        const int t = g / l.gper, i = g % l.gper;
        const int x0 = (i % l.gcols) * P, y0 = (i / l.gcols) * P * P;
        const cudaSurfaceObject_t so =
            cudaSurfaceObject_t(l.surf[t & (hy::kMaxGatherTextures - 1)]);
        brick_cells<T>(
            nc, P, map, true,
            [&](int x, int y, int z) {
                return T(surf2Dread<unsigned char>(so, x0 + x, y0 + z * P + y, cudaBoundaryModeZero));
            },
            put);
    } else {
        const T *v = reinterpret_cast<const T *>(l.pool + (long long)g * l.stride);
        brick_cells<T>(
            nc, P, map, true,
            [&](int x, int y, int z) { return v[((long long)z * P + y) * P + x]; }, put);
    }
}

// The coarse stand-in of brick blockIdx.x (of one that is not empty): its sub-box
// of coarse brick cid.
template <typename T>
__global__ void coarse_minmax_kernel(const unsigned char *__restrict__ coarse, long long stride,
                                     const hy::RegEntry *__restrict__ reg,
                                     const int2 *__restrict__ info, int gx, int gy, int sc, int cgx,
                                     int cgy, int nc, int P, MinMax<T> *__restrict__ out) {
    const int b = blockIdx.x;
    const int x = b % gx, y = (b / gx) % gy, z = b / (gx * gy);
    const int cid = ((z / sc) * cgy + y / sc) * cgx + x / sc;
    const T *v = reinterpret_cast<const T *>(coarse + (long long)cid * stride);
    const hy::RegEntry e = reg[b];
    MinMax<T> *o = out + (long long)b * nc * nc * nc;
    brick_cells<T>(
        nc, P, make_float4(e.k, e.bx, e.by, e.bz), info[b].x == 0,
        [&](int i, int j, int k) { return v[((long long)k * P + j) * P + i]; },
        [&](int i, int j, int k, MinMax<T> m) { o[(k * nc + j) * nc + i] = m; });
}

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
};

// 1: every sample of the cell lies in one of the ranges without effect; 0: it
// must be sampled.  A sample is seven lerps x*(1-a) + y*a of the cell's taps:
// each rounds its weight, two products and a sum, so it leaves [lo, hi] by at
// most 3 * 3 * 2^-24 of the largest magnitude, u / 255 and n * s add one
// rounding each: 2e-6 covers them three times over.
template <typename T>
__device__ __forceinline__ unsigned char cell_free(const ClassArgs &a, MinMax<T> m) {
    if (m.lo > m.hi) return 0;
    const float lo = float(m.lo) * a.scale, hi = float(m.hi) * a.scale;
    const float e = 2e-6f * fmaxf(fabsf(lo), fabsf(hi)) + 1e-36f;  // and underflows
    for (int k = 0; k < a.r.n; ++k)
        if (lo - e >= a.r.lo[k] && hi + e <= a.r.hi[k]) return 1;
    return 0;
}
// The grid is worked out in bits, 32 cells of a row to a word (rows padded with
// zeros): free flags first, then per direction octant the cells from which a
// cube of 2, 4, 8 and 16 free cells extends -- a cube of 2m is free when the
// eight cubes of m at its corners are -- and last the distances as bytes, with
// cubes of 3, 6 and 12 from overlapping ones of 2, 4 and 8.  A byte per cell
// and scans along the axes took 130 us for a million cells; this takes 44.
struct BitGrid {
    int cx, cy, cz, w;   // cells per axis, words per row
    unsigned int words;  // of one plane: below 2^27 (kMaxGridCells), so that
                         // 32 threads a word number below 2^32
};

template <typename T>
__global__ void classify_kernel(const __grid_constant__ ClassArgs a,
                                const __grid_constant__ BitGrid g,
                                const MinMax<T> *__restrict__ mm, unsigned int *__restrict__ out) {
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x, word = i >> 5;
    if (word >= g.words) return;  // whole warps
    const unsigned int row = word / unsigned(g.w);
    const int x = int(word - row * g.w) * 32 + int(i & 31);
    const bool f = x < g.cx && cell_free(a, mm[(long long)row * g.cx + x]);
    const unsigned int bits = __ballot_sync(0xffffffffu, f);
    if ((i & 31) == 0) out[word] = bits;
}
// The same through a page table: a brick's cells are those of its slot, of its
// coarse stand-in, or (empty or absent) to be looked at by the march.
template <typename T>
__global__ void classify_paged_kernel(const __grid_constant__ ClassArgs a,
                                      const __grid_constant__ BitGrid g,
                                      const int2 *__restrict__ info, int gx, int gy, int lg,
                                      int reg_base, const MinMax<T> *__restrict__ slots,
                                      const MinMax<T> *__restrict__ coarse,
                                      unsigned int *__restrict__ out) {
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x, word = i >> 5;
    if (word >= g.words) return;
    const unsigned int row = word / unsigned(g.w);
    const int x = int(word - row * g.w) * 32 + int(i & 31);
    const int z = int(row / unsigned(g.cy)), y = int(row) - z * g.cy;
    bool f = false;
    if (x < g.cx) {  // nc = 1 << lg cells per brick edge
        const int2 in = info[((z >> lg) * gy + (y >> lg)) * gx + (x >> lg)];
        if (in.x == 0 && in.y >= 0) {
            const int m = (1 << lg) - 1;
            const int cell = ((((z & m) << lg) + (y & m)) << lg) + (x & m);
            f = cell_free(a, in.y < reg_base ? coarse[((long long)in.y << (3 * lg)) + cell]
                                             : slots[((long long)(in.y - reg_base) << (3 * lg)) + cell]);
        }
    }
    const unsigned int bits = __ballot_sync(0xffffffffu, f);
    if ((i & 31) == 0) out[word] = bits;
}

// Word w of row (y, z) of `p` and the same cells moved by m along octant o's
// x, anded; 0 outside the grid.
__device__ __forceinline__ unsigned int row_pair(const unsigned int *__restrict__ p,
                                                 const BitGrid &g, int w, int y, int z, int m,
                                                 int o) {
    if (y < 0 || y >= g.cy || z < 0 || z >= g.cz) return 0u;
    const unsigned int *r = p + ((long long)z * g.cy + y) * g.w;
    const unsigned int v = r[w];
    if (!v) return 0u;
    if (o & 1) return v & ((v << m) | (w > 0 ? r[w - 1] >> (32 - m) : 0u));
    return v & ((v >> m) | (w + 1 < g.w ? r[w + 1] << (32 - m) : 0u));
}
// The cells whose eight corner cubes at distance m are all in `p`.
__device__ __forceinline__ unsigned int cube_and(const unsigned int *__restrict__ p,
                                                 const BitGrid &g, int w, int y, int z, int m,
                                                 int o) {
    const int dy = o & 2 ? -m : m, dz = o & 4 ? -m : m;
    unsigned int v = row_pair(p, g, w, y, z, m, o);
    if (v) v &= row_pair(p, g, w, y + dy, z, m, o);
    if (v) v &= row_pair(p, g, w, y, z + dz, m, o);
    if (v) v &= row_pair(p, g, w, y + dy, z + dz, m, o);
    return v;
}
// Cubes of m (one plane for all octants, or eight) -> cubes of 2 m.
__global__ void double_kernel(const unsigned int *__restrict__ in, int in_planes,
                              const __grid_constant__ BitGrid g, int m,
                              unsigned int *__restrict__ out) {
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.words) return;
    const int o = blockIdx.y;
    const unsigned int row = i / unsigned(g.w);
    const int w = int(i - row * g.w), z = int(row / unsigned(g.cy)), y = int(row) - z * g.cy;
    const long long plane = (long long)o * g.words;
    out[plane + i] = cube_and(in + (in_planes > 1 ? plane : 0), g, w, y, z, m, o);
}
// Four cells' distances from their bits of the planes: 1 for each of the cubes
// of 1, 2, 3 and 4, 2 for 6 and 8, 4 for 12 and 16.
__global__ void distance_kernel(const unsigned int *__restrict__ f1,
                                const unsigned int *__restrict__ cubes,
                                const __grid_constant__ BitGrid g,
                                unsigned char *__restrict__ out) {
    const unsigned int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.words) return;
    const int o = blockIdx.y;
    const unsigned int row = i / unsigned(g.w);
    const int w = int(i - row * g.w), z = int(row / unsigned(g.cy)), y = int(row) - z * g.cy;
    const unsigned int *p = cubes + (long long)o * g.words;
    const long long level = 8ll * g.words;  // planes of one cube size
    const unsigned int b1 = f1[i], b2 = b1 ? p[i] : 0u, b4 = b2 ? p[level + i] : 0u,
                       b8 = b4 ? p[2 * level + i] : 0u, b16 = b8 ? p[3 * level + i] : 0u;
    const unsigned int b3 = b2 ? cube_and(p, g, w, y, z, 1, o) : 0u,
                       b6 = b4 ? cube_and(p + level, g, w, y, z, 2, o) : 0u,
                       b12 = b8 ? cube_and(p + 2 * level, g, w, y, z, 4, o) : 0u;
    unsigned char *q = out + o * ((long long)g.cx * g.cy * g.cz) + (long long)row * g.cx + w * 32;
    const int n = min(32, g.cx - w * 32);
    // bits 0..3 to the low bits of four bytes
    auto spread = [](unsigned int b, int k) {
        return ((((b >> k) & 15u) * 0x00204081u) & 0x01010101u);
    };
    unsigned int d[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
        d[k] = spread(b1, 4 * k) + spread(b2, 4 * k) + spread(b3, 4 * k) + spread(b4, 4 * k) +
               2u * (spread(b6, 4 * k) + spread(b8, 4 * k)) +
               4u * (spread(b12, 4 * k) + spread(b16, 4 * k));
    if ((g.cx & 31) == 0) {  // whole, aligned words of cells
        reinterpret_cast<uint4 *>(q)[0] = make_uint4(d[0], d[1], d[2], d[3]);
        reinterpret_cast<uint4 *>(q)[1] = make_uint4(d[4], d[5], d[6], d[7]);
    } else {
#pragma unroll
        for (int k = 0; k < 32; ++k)
            if (k < n) q[k] = (unsigned char)(d[k >> 2] >> (8 * (k & 3)));
    }
}

BitGrid bit_grid(const hy_skip &s) {
    const int w = (s.c[0] + 31) / 32;
    return BitGrid{s.c[0], s.c[1], s.c[2], w, unsigned(w) * unsigned(s.c[1]) * unsigned(s.c[2])};
}

template <typename T>
int classify(hy_volume *v, const hy_skip_ranges &r, unsigned char *grid) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    const ClassArgs a{r, sizeof(T) == 1 ? 1.f / 255.f : 1.f};
    const BitGrid g = bit_grid(s);
    const unsigned by_cell = (g.words + 7) / 8, by_word = (g.words + 127) / 128;
    unsigned int *f1 = s.bits, *cubes = s.bits + g.words;
    int lg = 0;
    while ((1 << lg) < s.nc) ++lg;
    if (s.slots)
        classify_paged_kernel<T><<<by_cell, 256, 0, ctx->stream>>>(
            a, g, v->info_dev, v->grid[0], v->grid[1], lg, s.reg_base,
            static_cast<const MinMax<T> *>(s.slots), static_cast<const MinMax<T> *>(s.minmax), f1);
    else
        classify_kernel<T><<<by_cell, 256, 0, ctx->stream>>>(
            a, g, static_cast<const MinMax<T> *>(s.minmax), f1);
    for (int k = 0; k < 4; ++k)
        double_kernel<<<dim3(by_word, 8), 128, 0, ctx->stream>>>(
            k ? cubes + (k - 1) * 8ll * g.words : f1, k ? 8 : 1, g, 1 << k,
            cubes + k * 8ll * g.words);
    distance_kernel<<<dim3(by_word, 8), 128, 0, ctx->stream>>>(f1, cubes, g, grid);
    HY_CUDA(ctx, cudaGetLastError());
    return HY_OK;
}

// The cells' histogram on the host, summed so that hist[i * kBins + j] counts
// the cells with lo in bin >= i and hi in bin <= j.
template <typename T>
int cell_hist(hy_volume *v, int *dev) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    s.hist.resize(kBins * kBins);
    const unsigned blocks = unsigned(std::min<long long>((s.cells + 255) / 256, 4 * ctx->sms));
    cell_hist_kernel<T><<<blocks, 256, 0, ctx->stream>>>(
        static_cast<const MinMax<T> *>(s.minmax), s.cells, sizeof(T) == 1 ? 1.f / 255.f : 1.f, dev);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(s.hist.data(), dev, sizeof(int) * kBins * kBins, cudaMemcpyDeviceToHost,
                            ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    if (e != cudaSuccess) return hy_cuda_fail(ctx, e, "volume: skip grid");
    for (int i = kBins - 1; i >= 0; --i) {
        int row = 0;
        for (int j = 0; j < kBins; ++j) {
            row += s.hist[i * kBins + j];
            s.hist[i * kBins + j] = row + (i + 1 < kBins ? s.hist[(i + 1) * kBins + j] : 0);
        }
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
    if (s.slots) {  // paged; else minmax lies in grid[0]'s allocation
        cudaFree(s.slots);
        if (s.minmax) cudaFree(s.minmax);
    }
    if (s.grid[0]) cudaFree(s.grid[0]);
    s = hy_skip();
}

namespace {

// Cells of a volume's bricks and the box margin; s.nc stays 0 where the
// volume has no grid.  The interior sampler's bricks only (an apron: no
// wrapped coordinates).
void skip_geometry(hy_volume *v) {
    hy_skip &s = v->skip;
    const int bs = v->desc.block_size;
    if (v->desc.padding < 1 || v->P > 4096) return;
    int nc = 1;  // a power of two (positions scale exactly), cells of >= 8 voxels
    while (nc * 2 * 8 <= bs) nc *= 2;
    long long n = 1;
    int gmax = 1;
    for (int i = 0; i < 3; ++i) {
        s.c[i] = v->grid[i] * nc;
        n *= s.c[i];
        gmax = std::max(gmax, v->grid[i]);
    }
    if (n < kMinGridCells || n > kMaxGridCells) return;
    // A run of up to 127 steps adds up to 127 roundings of half an ulp of
    // the largest coordinate; 4e-6 brick covers the run length's own
    // arithmetic.  Boxes shrink by this much, so that a run that stays in one
    // by this arithmetic stays in it step by step.
    const float ulp = std::nextafterf(float(gmax), 1e30f) - float(gmax);
    s.shrink = 128.f * ulp + 4e-6f;
    if (s.shrink * float(nc) > .125f) return;  // a volume of thousands of bricks an edge
    s.nc = nc;
    s.cells = n;
}

// Threads and blocks per brick for brick_cells: enough for the GPU when there
// are few bricks.
dim3 cells_grid(const hy_volume *v, int bricks, int *threads) {
    const int lanes = v->skip.nc * v->skip.nc * v->skip.nc * kCellLanes;
    *threads = std::min(512, std::max(32, lanes));
    const int rounds = (lanes + *threads - 1) / *threads;
    return dim3(unsigned(bricks),
                unsigned(std::max(1, std::min(rounds, 8 * v->ctx->sms / std::max(bricks, 1)))));
}

// The distances per transfer function and (iso) per isovalue (at least the
// histogram's size: it is counted there), the bit planes they are worked out in
// and `minmax` bytes of the cells' own (0: none), in one allocation.
cudaError_t alloc_planes(hy_skip &s, bool iso, size_t minmax) {
    const size_t n = size_t(s.cells), hist = sizeof(int) * kBins * kBins,
                 grids = (std::max(n * (iso ? 16 : 8), hist) + 255) / 256 * 256,
                 planes = (size_t(bit_grid(s).words) * 33 * sizeof(unsigned int) + 255) / 256 * 256;
    if (!hy_room_for(grids + planes + minmax)) return cudaErrorMemoryAllocation;
    const cudaError_t e = cudaMalloc(&s.grid[0], grids + planes + minmax);
    if (e != cudaSuccess) return e;
    s.grid[1] = iso ? s.grid[0] + 8 * n : nullptr;
    s.bits = reinterpret_cast<unsigned int *>(s.grid[0] + grids);
    if (minmax) s.minmax = s.grid[0] + grids + planes;
    return e;
}

size_t mm_bytes(const hy_volume *v) {
    return v->desc.dtype == HY_DTYPE_U8 ? sizeof(MinMax<unsigned char>) : sizeof(MinMax<float>);
}

}  // namespace

int hy_skip_build(hy_volume *v) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    hy_skip_free(v);
    if (v->resident <= 0) return HY_OK;
    skip_geometry(v);
    if (!s.nc) return HY_OK;
    const bool u8 = v->desc.dtype == HY_DTYPE_U8;
    const cudaError_t e = alloc_planes(s, true, size_t(s.cells) * mm_bytes(v));
    if (e != cudaSuccess) {  // no room: the march samples every cell
        hy_skip_free(v);
        cudaGetLastError();
        return HY_OK;
    }
    int *hist = reinterpret_cast<int *>(s.grid[0]);  // the grids are unused until a render
    const CellArgs a{v->pool,    v->reg_dev, v->info_dev, v->grid[0],
                     v->grid[1], s.nc,       v->P,        hist};
    int threads;
    const dim3 grid = cells_grid(v, v->nbricks, &threads);
    if (u8)
        cell_minmax_kernel<unsigned char><<<grid, threads, 0, ctx->stream>>>(
            a, static_cast<MinMax<unsigned char> *>(s.minmax));
    else
        cell_minmax_kernel<float><<<grid, threads, 0, ctx->stream>>>(
            a, static_cast<MinMax<float> *>(s.minmax));
    HY_CUDA(ctx, cudaGetLastError());
    return u8 ? cell_hist<unsigned char>(v, hist) : cell_hist<float>(v, hist);
}

int hy_skip_build_paged(hy_volume *v, const hy_store *store, int nslots, int reg_base) {
    hy_ctx *ctx = v->ctx;
    hy_skip &s = v->skip;
    hy_skip_free(v);
    skip_geometry(v);
    if (!s.nc) return HY_OK;
    const bool u8 = v->desc.dtype == HY_DTYPE_U8;
    const size_t per = size_t(s.nc) * s.nc * s.nc * mm_bytes(v);
    unsigned char *coarse = nullptr;  // the coarse level, for its cells alone
    s.reg_base = reg_base;
    const size_t cells = size_t(nslots) * per + (reg_base > 0 ? size_t(v->nbricks) * per : 0);
    cudaError_t e = hy_room_for(cells) ? cudaMalloc(&s.slots, size_t(nslots) * per)
                                       : cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = alloc_planes(s, !v->paged_gather, 0);
    if (e == cudaSuccess && reg_base > 0) {
        e = cudaMalloc(&s.minmax, size_t(v->nbricks) * per);
        if (e == cudaSuccess) e = cudaMalloc(&coarse, store->coarse.size());
    }
    if (e != cudaSuccess) {
        hy_skip_free(v);
        cudaGetLastError();
        return HY_OK;
    }
    if (reg_base > 0) {
        e = cudaMemcpyAsync(coarse, store->coarse.data(), store->coarse.size(),
                            cudaMemcpyHostToDevice, ctx->stream);
        int threads;
        const dim3 grid = cells_grid(v, v->nbricks, &threads);
        const int sc = 1 << store->coarse_level;
        const int *cg = store->coarse_grid;
        if (e == cudaSuccess && u8)
            coarse_minmax_kernel<unsigned char><<<grid, threads, 0, ctx->stream>>>(
                coarse, (long long)v->slot_stride, v->reg_dev, v->info_dev, v->grid[0], v->grid[1], sc,
                cg[0], cg[1], s.nc, v->P, static_cast<MinMax<unsigned char> *>(s.minmax));
        else if (e == cudaSuccess)
            coarse_minmax_kernel<float><<<grid, threads, 0, ctx->stream>>>(
                coarse, (long long)v->slot_stride, v->reg_dev, v->info_dev, v->grid[0], v->grid[1], sc,
                cg[0], cg[1], s.nc, v->P, static_cast<MinMax<float> *>(s.minmax));
        if (e == cudaSuccess) e = cudaGetLastError();
        int *hist = reinterpret_cast<int *>(s.grid[0]);
        if (e == cudaSuccess)
            e = cudaMemsetAsync(hist, 0, sizeof(int) * kBins * kBins, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        cudaFree(coarse);
        if (e != cudaSuccess) return hy_cuda_fail(ctx, e, "pager: skip grid");
        return u8 ? cell_hist<unsigned char>(v, hist) : cell_hist<float>(v, hist);
    }
    return HY_OK;
}

int hy_skip_slots(hy_volume *v, const hy::GatherItem *items, int n, const hy::CacheLayout &l,
                  cudaStream_t stream) {
    hy_skip &s = v->skip;
    if (!s.slots || n <= 0) return HY_OK;
    int threads;
    const dim3 grid = cells_grid(v, n, &threads);
    const float4 map = make_float4(v->k, v->b, v->b, v->b);
    if (v->paged_gather)
        slot_minmax_kernel<unsigned char, true><<<grid, threads, 0, stream>>>(
            items, l, s.nc, v->P, map, static_cast<MinMax<unsigned char> *>(s.slots));
    else if (v->desc.dtype == HY_DTYPE_U8)
        slot_minmax_kernel<unsigned char, false><<<grid, threads, 0, stream>>>(
            items, l, s.nc, v->P, map, static_cast<MinMax<unsigned char> *>(s.slots));
    else
        slot_minmax_kernel<float, false><<<grid, threads, 0, stream>>>(
            items, l, s.nc, v->P, map, static_cast<MinMax<float> *>(s.slots));
    HY_CUDA(v->ctx, cudaGetLastError());
    return HY_OK;
}

void hy_skip_page_table_changed(hy_volume *v) { v->skip.valid[0] = v->skip.valid[1] = false; }

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

int hy_skip_view(hy_ctx *ctx, const hy_volume *cv, const hy_shader_params *p, hy::SkipGrid *out,
                 bool refresh) {
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
        // longer with the grid than without.  A paged cache's cells are
        // counted on the coarse stand-ins (without a coarse level: not).
        if (!s.hist.empty() && free_cells(s, r) * 10 < s.sampled) return HY_OK;
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
    if (r.n == 0 || !s.grid[which]) return HY_OK;
    // A capture would replay against whatever knots the grid holds by then:
    // captured launches sample every cell.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    HY_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) return HY_OK;
    if (refresh && (!s.valid[which] || !same_ranges(r, s.key[which]))) {
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
