// hy_volume.cu -- brick pool, page table and thumbnails on the device.
//
// Replaces, for volumes that stay resident, what the reference does per
// frame on the host: decode bricks and upload one 3-D texture per brick,
// write vaddr[brick] = slot and re-upload the registry
// (src/slave/paging/lossless_block_paging.cc:137-174).  Layout in HBM:
//   pool  : resident bricks, (bs+2*pad)^3 voxels each, x fastest, slots
//           256-byte aligned, u8 (1 B/voxel) or f32 (4 B/voxel);
//   info  : int2 per brick {chebyshev distance, registry id or -1}, the
//           chebyshev thumbnail and the vaddr texture read together
//           (volume_shader.cu:45-50);
//   reg   : RegEntry per registry id {k, b, slot offset} (block_paging.hpp:24-36);
//   mean  : float per brick (the "mean" thumbnail read by blocks_shader.cu:33).
// The dataset definition this builds: the apron of a brick holds the
// neighbouring voxels, clamped at the volume border; a brick is non-empty if
// any voxel of core or apron is non-zero; chebyshev = L-infinity distance in
// bricks to the nearest non-empty brick (0 = non-empty, max(grid) if there is
// none); mean = mean of the normalised core voxels.

#include <algorithm>
#include <cstring>
#include <mutex>

#include "hy_internal.h"

namespace {

// Rows of a padded brick (z, y and x clamped to the volume, as the apron replicates
// the border).  Long rows go to a warp each, its lanes consecutive voxels; of short
// ones (short_rows) a block takes as many at a time as its threads hold, kRows of
// these loaded before the first is used.  What bounds both kernels is issue, and
// FP64 for f32 sums; a thread per voxel with 64-bit divisions took 5.1 + 4.8 ms for
// 1024^3 u8 in bricks of 64^3 (one block per brick for the statistics: 0.8 ms for a
// single 64^3 brick, 6.5 ms for 128^3), a warp a row 2.8 + 1.6, short rows 2.2 + 2.2.
// 200x150x171 f32 in bricks of 16^3, us: 49 + 57 a thread per voxel, 91 + 67 a warp a
// row, 37 + 24 short rows; of 32^3 121 + 58, 57 + 31, 40 + 29.
struct BrickArgs {
    int dim[3];
    int bs, pad, P;
    int gx, gy;
};
constexpr int kThreads = 256, kRows = 4;
template <typename T>
__host__ __device__ constexpr bool short_rows(int P) {
    return P <= (sizeof(T) == 1 ? 40 : 72);
}

// Where a brick's padded rows lie in the volume.
struct BrickOrigin {
    int x, y, z;
    __device__ __forceinline__ BrickOrigin(const BrickArgs &a, int bid) {
        const int q = bid / a.gx, bz = q / a.gy;
        x = (bid - q * a.gx) * a.bs - a.pad;
        y = (q - bz * a.gy) * a.bs - a.pad;
        z = bz * a.bs - a.pad;
    }
    __device__ __forceinline__ long long row(const BrickArgs &a, int pz, int py) const {
        const int Y = min(max(y + py, 0), a.dim[1] - 1), Z = min(max(z + pz, 0), a.dim[2] - 1);
        return ((long long)Z * a.dim[1] + Y) * a.dim[0];
    }
    __device__ __forceinline__ int column(const BrickArgs &a, int px) const {
        return min(max(x + px, 0), a.dim[0] - 1);
    }
};

// This thread's rows of the box [x0, x1) x [y0, y1) x [z0, z1) of a padded brick,
// of which `group` of `groups` blocks takes its share: get(ok, x, y, z) for kRows of
// them, then put(k, ok, x, y, z) for the same ones.
template <typename Get, typename Put>
__device__ __forceinline__ void brick_rows(int x0, int x1, int y0, int y1, int z0, int z1, int group,
                                           int groups, Get get, Put put) {
    const int nx = x1 - x0, ny = y1 - y0, cols = min(nx, kThreads), rows = kThreads / cols;
    const int row = threadIdx.x / cols, col = threadIdx.x - row * cols;
    if (row >= rows) return;
    const int first = group * rows + row, stride = groups * rows;
    const int sz = stride / ny, sy = stride - sz * ny;
    for (int x = x0 + col; x < x1; x += cols) {
        int z = first / ny, y = y0 + first - z * ny;
        z += z0;
        while (z < z1) {
            int ky[kRows], kz[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                ky[k] = y;
                kz[k] = z;
                y += sy;
                z += sz;
                if (y >= y1) {
                    y -= ny;
                    ++z;
                }
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) get(k, kz[k] < z1, x, ky[k], kz[k]);
#pragma unroll
            for (int k = 0; k < kRows; ++k) put(k, kz[k] < z1, x, ky[k], kz[k]);
        }
    }
}

// Emptiness and the sum of the core voxels of brick blockIdx.x, rows of the
// slices of part blockIdx.y of gridDim.y: part sums are added up on the host.
template <typename T, bool SHORT>
__global__ void __launch_bounds__(kThreads) brick_stats_kernel(const T *__restrict__ raw,
                                                               const __grid_constant__ BrickArgs a,
                                                               unsigned int *__restrict__ nonempty,
                                                               double *__restrict__ core_sum) {
    const int bid = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = a.P, hi = a.pad + a.bs;
    const int z0 = int((long long)P * blockIdx.y / gridDim.y),
              z1 = int((long long)P * (blockIdx.y + 1) / gridDim.y);
    const BrickOrigin o(a, bid);
    bool any = false;
    double sum = 0.0;
    unsigned long long whole = 0;  // u8: exact, and no FP64 (slow on this GPU)
    if constexpr (SHORT) {
        T v[kRows];
        auto load = [&](int k, bool ok, int x, int y, int z) {
            v[k] = ok ? raw[o.row(a, z, y) + o.column(a, x)] : T(0);
        };
        brick_rows(0, P, 0, P, z0, z1, 0, 1, load, [&](int k, bool, int x, int y, int z) {
            any |= v[k] != T(0);
            if constexpr (sizeof(T) == 1)
                if (x >= a.pad && x < hi && y >= a.pad && y < hi && z >= a.pad && z < hi)
                    whole += v[k];
        });
        // f32: the core again (L1), full warps of FP64 additions
        if constexpr (sizeof(T) != 1)
            brick_rows(a.pad, hi, a.pad, hi, max(z0, a.pad), min(z1, hi), 0, 1, load,
                       [&](int k, bool, int, int, int) { sum += double(v[k]); });
    } else {
        for (int r = z0 * P + warp; r < z1 * P; r += 8) {
            const int z = r / P, y = r - z * P;
            const T *row = raw + o.row(a, z, y);
            const bool core = z >= a.pad && z < hi && y >= a.pad && y < hi;
            unsigned int rs = 0;  // a row's sum fits: P * 255
            for (int x = lane; x < P; x += 32) {
                const T t = row[o.column(a, x)];
                any |= t != T(0);
                if constexpr (sizeof(T) == 1)
                    if (x >= a.pad && x < hi) rs += t;
            }
            if constexpr (sizeof(T) == 1) {
                if (core) whole += rs;
            } else if (core) {
                for (int x = a.pad + lane; x < hi; x += 32) sum += double(row[o.column(a, x)]);
            }
        }
    }
    if constexpr (sizeof(T) == 1) sum = double(whole);
    __shared__ double ssum[8];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) ssum[warp] = sum;
    const int some = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) sum += ssum[w];
        const size_t i = size_t(bid) * gridDim.y + blockIdx.y;
        nonempty[i] = some != 0;
        core_sum[i] = sum;
    }
}

template <typename T, bool SHORT>
__global__ void __launch_bounds__(kThreads) brick_fill_kernel(const T *__restrict__ raw,
                                                              const __grid_constant__ BrickArgs a,
                                                              const int *__restrict__ slot_brick,
                                                              unsigned char *__restrict__ pool,
                                                              long long slot_stride, int slot0) {
    const int slot = slot0 + blockIdx.y, P = a.P;
    const BrickOrigin o(a, slot_brick[slot]);
    T *dst = reinterpret_cast<T *>(pool + (long long)slot * slot_stride);
    if constexpr (!SHORT) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int r = blockIdx.x * 8 + warp; r < P * P; r += gridDim.x * 8) {
            const int z = r / P, y = r - z * P;
            const T *row = raw + o.row(a, z, y);
            T *out = dst + (long long)r * P;
            for (int x = lane; x < P; x += 32) out[x] = row[o.column(a, x)];
        }
    } else {
        T v[kRows];
        brick_rows(
            0, P, 0, P, 0, P, blockIdx.x, gridDim.x,
            [&](int k, bool ok, int x, int y, int z) {
                if (ok) v[k] = raw[o.row(a, z, y) + o.column(a, x)];
            },
            [&](int k, bool ok, int x, int y, int z) {
                if (ok) dst[((long long)z * P + y) * P + x] = v[k];
            });
    }
}

// ---- gather textures ---------------------------------------------------------
//
// Every resident brick of a u8 volume with an apron is also placed in a 2-D
// u8 texture made for gather: its P slices stacked as P x P tiles in one
// column of texels (slice z at rows y0 + z * P).  The interior sampler then
// fetches the eight taps of a trilinear footprint with two gathers (slices
// z and z + 1), each returning the 2x2 texels at rows y, y + 1 and columns
// x, x + 1 as floats, normalised by the texture unit.  The coordinates are
// whole texel edges (x + 1, y + 1 with x, y integral), so the footprint the
// hardware picks is exactly (x, y) .. (x + 1, y + 1).  Bricks with P^2 rows
// taller than a gather texture allows keep the plain loads.

__global__ void gather_check_kernel(cudaTextureObject_t t, unsigned int *bad) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= 255) return;
    // row 0 holds u = column, row 1 holds 255 - column
    const float4 g = hy::gather_r((unsigned long long)t, float(x) + 1.f, 1.f);
    const float ew = __fdiv_rn(float(x), 255.f), ez = __fdiv_rn(float(x + 1), 255.f);
    const float ex = __fdiv_rn(float(255 - x), 255.f), ey = __fdiv_rn(float(254 - x), 255.f);
    if (__float_as_uint(g.w) != __float_as_uint(ew) || __float_as_uint(g.z) != __float_as_uint(ez) ||
        __float_as_uint(g.x) != __float_as_uint(ex) || __float_as_uint(g.y) != __float_as_uint(ey))
        atomicAdd(bad, 1u);
}

cudaTextureObject_t make_gather_texture(cudaArray_t arr, cudaError_t *err) {
    cudaResourceDesc rd;
    std::memset(&rd, 0, sizeof(rd));
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = arr;
    cudaTextureDesc td;
    std::memset(&td, 0, sizeof(td));
    td.addressMode[0] = td.addressMode[1] = cudaAddressModeClamp;
    td.filterMode = cudaFilterModePoint;
    td.readMode = cudaReadModeNormalizedFloat;
    td.normalizedCoords = 0;
    cudaTextureObject_t t = 0;
    *err = cudaCreateTextureObject(&t, &rd, &td, nullptr);
    return t;
}

// Once per device: the gather order and the u8 -> u / 255 normalisation
// of the texture unit equal what the sampler assumes (for all 256 values,
// against IEEE division).  A device that fails renders with the plain loads.
constexpr int kMaxCheckDevices = 64;
std::mutex g_gather_mu;
int g_gather_ok[kMaxCheckDevices] = {};  // 0 unknown, 1 passed, -1 failed

int gather_check(hy_ctx *ctx, bool *ok) {
    *ok = false;
    if (ctx->device < 0 || ctx->device >= kMaxCheckDevices) return HY_OK;
    std::lock_guard<std::mutex> lock(g_gather_mu);
    if (g_gather_ok[ctx->device] == 0) {
        cudaChannelFormatDesc cd = cudaCreateChannelDesc(8, 0, 0, 0, cudaChannelFormatKindUnsigned);
        cudaArray_t arr = nullptr;
        unsigned int *bad = nullptr;
        cudaTextureObject_t t = 0;
        unsigned char host[2 * 256];
        for (int c = 0; c < 256; ++c) {
            host[c] = (unsigned char)c;
            host[256 + c] = (unsigned char)(255 - c);
        }
        unsigned int nbad = 1;
        cudaError_t e = cudaMallocArray(&arr, &cd, 256, 2, cudaArrayTextureGather);
        if (e == cudaSuccess)
            e = cudaMemcpy2DToArrayAsync(arr, 0, 0, host, 256, 256, 2, cudaMemcpyHostToDevice,
                                         ctx->stream);
        if (e == cudaSuccess) t = make_gather_texture(arr, &e);
        if (e == cudaSuccess) e = cudaMalloc(&bad, sizeof(unsigned int));
        if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(unsigned int), ctx->stream);
        if (e == cudaSuccess) {
            gather_check_kernel<<<1, 256, 0, ctx->stream>>>(t, bad);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&nbad, bad, sizeof(unsigned int), cudaMemcpyDeviceToHost,
                                ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        if (t) cudaDestroyTextureObject(t);
        if (arr) cudaFreeArray(arr);
        if (bad) cudaFree(bad);
        if (e != cudaSuccess) return hy_cuda_fail(ctx, e, "volume: gather texture check");
        g_gather_ok[ctx->device] = nbad == 0 ? 1 : -1;
    }
    *ok = g_gather_ok[ctx->device] == 1;
    return HY_OK;
}

// Slots first .. first + gridDim.y - 1 of the pool into a gather texture: a
// brick's P^2 rows of P voxels are P^2 texel rows (slot i of the texture in
// column i % cols, row block i / cols).  Texel pairs where P is even.  One
// kernel for all bricks: a 2-D copy call per brick took half of a 1024^3
// volume's upload.
template <typename U>
__global__ void __launch_bounds__(256) gather_fill_kernel(const unsigned char *__restrict__ pool,
                                                          long long slot_stride, int P, int first,
                                                          int slot0, int cols,
                                                          cudaSurfaceObject_t surf) {
    const int i = slot0 + blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = (i % cols) * P, y0 = (i / cols) * P * P;
    const U *src = reinterpret_cast<const U *>(pool + (long long)(first + i) * slot_stride);
    const int W = P / int(sizeof(U));
    for (int r = blockIdx.x * 8 + warp; r < P * P; r += gridDim.x * 8)
        for (int x = lane; x < W; x += 32)
            surf2Dwrite(src[(long long)r * W + x], surf, x0 + x * int(sizeof(U)), y0 + r,
                        cudaBoundaryModeZero);
}

void free_gather(hy_volume *v) {
    for (auto t : v->atlas_tex) cudaDestroyTextureObject(cudaTextureObject_t(t));
    for (auto a : v->atlas) cudaFreeArray(a);
    if (v->tex_dev) cudaFree(v->tex_dev);
    if (v->info4_dev) cudaFree(v->info4_dev);
    v->atlas_tex.clear();
    v->atlas.clear();
    v->tex_dev = nullptr;
    v->info4_dev = nullptr;
}

int build_gather(hy_volume *vol) {
    hy_ctx *ctx = vol->ctx;
    const int P = vol->P;
    if (vol->desc.dtype != HY_DTYPE_U8 || vol->desc.padding < 1 || vol->resident <= 0) return HY_OK;
    int gw = 0, gh = 0;
    HY_CUDA(ctx, cudaDeviceGetAttribute(&gw, cudaDevAttrMaxTexture2DGatherWidth, ctx->device));
    HY_CUDA(ctx, cudaDeviceGetAttribute(&gh, cudaDevAttrMaxTexture2DGatherHeight, ctx->device));
    const long long brick_rows = (long long)P * P;
    if (P > gw || brick_rows > gh) return HY_OK;  // too tall for a gather texture
    bool ok = false;
    int rc = gather_check(ctx, &ok);
    if (rc || !ok) return rc;
    const int cols = gw / P, rowblocks = int(gh / brick_rows), per = cols * rowblocks;
    const int n = vol->resident;
    if ((long long)per * hy::kResidentGatherTextures < n) return HY_OK;  // more than two textures hold
    std::vector<hy::TexEntry> table(n);
    std::vector<cudaSurfaceObject_t> surfs;  // for the fill alone
    auto drop_surfs = [&] {
        cudaStreamSynchronize(ctx->stream);
        for (auto sf : surfs) cudaDestroySurfaceObject(sf);
        surfs.clear();
    };
    for (int first = 0; first < n; first += per) {
        const int cnt = std::min(per, n - first);
        const int ucols = std::min(cols, cnt), urows = (cnt + cols - 1) / cols;
        cudaArray_t arr = nullptr;
        unsigned long long t = 0, sf = 0;
        rc = hy_gather_texture_create(ctx, size_t(ucols) * P, size_t(urows) * brick_rows, &arr, &t,
                                      &sf);
        if (rc) {
            drop_surfs();
            free_gather(vol);
            return rc;
        }
        vol->atlas.push_back(arr);
        vol->atlas_tex.push_back(t);
        surfs.push_back(cudaSurfaceObject_t(sf));
        const unsigned gx = unsigned(std::min<long long>((brick_rows + 7) / 8, 64));
        for (int s0 = 0; s0 < cnt; s0 += 65535) {
            const dim3 grid(gx, unsigned(std::min(65535, cnt - s0)));
            if (P % 2 == 0)
                gather_fill_kernel<unsigned short><<<grid, 256, 0, ctx->stream>>>(
                    vol->pool, (long long)vol->slot_stride, P, first, s0, cols, surfs.back());
            else
                gather_fill_kernel<unsigned char><<<grid, 256, 0, ctx->stream>>>(
                    vol->pool, (long long)vol->slot_stride, P, first, s0, cols, surfs.back());
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            drop_surfs();
            free_gather(vol);
            return hy_cuda_fail(ctx, e, "volume: gather texture fill");
        }
        for (int i = 0; i < cnt; ++i) {
            const int slot = first + i, cx = i % cols, ry = i / cols;
            table[slot] = hy::TexEntry{float(cx * P), float(ry * brick_rows),
                                       int(vol->atlas_tex.size()) - 1, 0};
        }
    }
    // the page table with each resident brick's texel origin beside it
    std::vector<int4> info4(vol->nbricks);
    for (int b = 0; b < vol->nbricks; ++b) {
        const int reg = vol->reg_of_brick[b];
        int4 q = make_int4(vol->cheb[b], reg, 0, 0);
        if (reg >= 0) {
            // texel origin + 1 as floats (the sampler's footprint column and
            // row offsets), the texture in the sign of the row (>= 1)
            const float x1 = table[reg].x0 + 1.f, y1 = table[reg].y0 + 1.f;
            const float ys = table[reg].which ? -y1 : y1;
            std::memcpy(&q.z, &x1, 4);
            std::memcpy(&q.w, &ys, 4);
        }
        info4[b] = q;
    }
    cudaError_t e = cudaMalloc(&vol->tex_dev, size_t(n) * sizeof(hy::TexEntry));
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(vol->tex_dev, table.data(), size_t(n) * sizeof(hy::TexEntry),
                            cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaMalloc(&vol->info4_dev, size_t(vol->nbricks) * sizeof(int4));
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(vol->info4_dev, info4.data(), size_t(vol->nbricks) * sizeof(int4),
                            cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    drop_surfs();
    if (e != cudaSuccess) {
        free_gather(vol);
        return hy_cuda_fail(ctx, e, "volume: gather table");
    }
    return HY_OK;
}

void free_volume_device(hy_volume *v) {
    free_gather(v);
    hy_skip_free(v);
    if (v->pool) cudaFree(v->pool);
    if (v->info_dev) cudaFree(v->info_dev);
    if (v->reg_dev) cudaFree(v->reg_dev);
    if (v->mean_dev) cudaFree(v->mean_dev);
    v->pool = nullptr;
    v->info_dev = nullptr;
    v->reg_dev = nullptr;
    v->mean_dev = nullptr;
    v->pool_bytes = 0;
    v->uploaded = false;
}

template <typename T>
int upload_impl(hy_volume *vol, const void *host) {
    hy_ctx *ctx = vol->ctx;
    const hy_volume_desc &d = vol->desc;
    const size_t nvox = size_t(d.dim[0]) * d.dim[1] * d.dim[2];
    T *raw = nullptr;
    unsigned int *ne_dev = nullptr;
    double *sum_dev = nullptr;
    int *slot_brick_dev = nullptr;
    auto cleanup = [&] {
        if (raw) cudaFree(raw);
        if (ne_dev) cudaFree(ne_dev);
        if (sum_dev) cudaFree(sum_dev);
        if (slot_brick_dev) cudaFree(slot_brick_dev);
    };
#define HY_UP(call)                                            \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess) {                               \
            cleanup();                                         \
            return hy_cuda_fail(ctx, e_, #call);               \
        }                                                      \
    } while (0)
    free_volume_device(vol);
    HY_UP(cudaMalloc(&raw, nvox * sizeof(T)));
    HY_UP(cudaMemcpyAsync(raw, host, nvox * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
    const int nb = vol->nbricks;
    // enough blocks for the GPU when there are few bricks
    const int parts = std::max(1, std::min(vol->P, 8 * ctx->sms / nb));
    const size_t np = size_t(nb) * parts;
    const BrickArgs ba{{d.dim[0], d.dim[1], d.dim[2]}, d.block_size, d.padding, vol->P,
                       vol->grid[0], vol->grid[1]};
    HY_UP(cudaMalloc(&ne_dev, np * sizeof(unsigned int)));
    HY_UP(cudaMalloc(&sum_dev, np * sizeof(double)));
    const bool rows_short = short_rows<T>(vol->P);
    const auto stats = rows_short ? &brick_stats_kernel<T, true> : &brick_stats_kernel<T, false>;
    stats<<<dim3(unsigned(nb), unsigned(parts)), kThreads, 0, ctx->stream>>>(raw, ba, ne_dev,
                                                                             sum_dev);
    HY_UP(cudaGetLastError());
    std::vector<unsigned int> ne_part(np);
    std::vector<double> sum_part(np);
    HY_UP(cudaMemcpyAsync(ne_part.data(), ne_dev, np * sizeof(unsigned int),
                          cudaMemcpyDeviceToHost, ctx->stream));
    HY_UP(cudaMemcpyAsync(sum_part.data(), sum_dev, np * sizeof(double), cudaMemcpyDeviceToHost,
                          ctx->stream));
    HY_UP(cudaStreamSynchronize(ctx->stream));
    std::vector<unsigned char> ne(nb, 0);
    std::vector<double> sums(nb, 0.0);
    for (int i = 0; i < nb; ++i)
        for (int k = 0; k < parts; ++k) {
            ne[i] |= ne_part[size_t(i) * parts + k] ? 1 : 0;
            sums[i] += sum_part[size_t(i) * parts + k];
        }

    hy_chebyshev_transform(ne, vol->grid, vol->cheb);
    const double ncore = double(d.block_size) * d.block_size * d.block_size;
    vol->mean.resize(nb);
    for (int i = 0; i < nb; ++i)
        vol->mean[i] = (sizeof(T) == 1) ? float(sums[i] / 255.0 / ncore) : float(sums[i] / ncore);
    std::vector<int> slot_brick;
    vol->reg_of_brick.assign(nb, -1);
    for (int i = 0; i < nb; ++i)
        if (ne[i]) {
            vol->reg_of_brick[i] = int(slot_brick.size());
            slot_brick.push_back(i);
        }
    vol->nonempty = int(slot_brick.size());
    vol->resident = vol->nonempty;
    const int nslots = std::max(vol->resident, 1);
    vol->pool_bytes = size_t(nslots) * vol->slot_stride;
    HY_UP(cudaMalloc(&vol->pool, vol->pool_bytes));
    HY_UP(cudaMemsetAsync(vol->pool, 0, vol->pool_bytes, ctx->stream));
    if (vol->resident > 0) {
        HY_UP(cudaMalloc(&slot_brick_dev, slot_brick.size() * sizeof(int)));
        HY_UP(cudaMemcpyAsync(slot_brick_dev, slot_brick.data(), slot_brick.size() * sizeof(int),
                              cudaMemcpyHostToDevice, ctx->stream));
        // rows a block takes at a time
        const int rows = rows_short ? kRows * (kThreads / vol->P) : kThreads / 32;
        const unsigned gx =
            unsigned(std::min<long long>(((long long)vol->P * vol->P + rows - 1) / rows, 64));
        const auto fill = rows_short ? &brick_fill_kernel<T, true> : &brick_fill_kernel<T, false>;
        for (int s0 = 0; s0 < vol->resident; s0 += 65535) {
            const int n = std::min(65535, vol->resident - s0);
            fill<<<dim3(gx, unsigned(n)), kThreads, 0, ctx->stream>>>(
                raw, ba, slot_brick_dev, vol->pool, (long long)vol->slot_stride, s0);
            HY_UP(cudaGetLastError());
        }
    }
    std::vector<int2> info(nb);
    for (int i = 0; i < nb; ++i) info[i] = make_int2(vol->cheb[i], vol->reg_of_brick[i]);
    std::vector<hy::RegEntry> reg(nslots);
    for (int s = 0; s < nslots; ++s) {
        reg[s] = hy::RegEntry{vol->k, vol->b, vol->b, vol->b, (long long)s * (long long)vol->slot_stride,
                              {0, 0}};
    }
    HY_UP(cudaMalloc(&vol->info_dev, nb * sizeof(int2)));
    HY_UP(cudaMalloc(&vol->reg_dev, nslots * sizeof(hy::RegEntry)));
    HY_UP(cudaMalloc(&vol->mean_dev, nb * sizeof(float)));
    HY_UP(cudaMemcpyAsync(vol->info_dev, info.data(), nb * sizeof(int2), cudaMemcpyHostToDevice,
                          ctx->stream));
    HY_UP(cudaMemcpyAsync(vol->reg_dev, reg.data(), nslots * sizeof(hy::RegEntry),
                          cudaMemcpyHostToDevice, ctx->stream));
    HY_UP(cudaMemcpyAsync(vol->mean_dev, vol->mean.data(), nb * sizeof(float),
                          cudaMemcpyHostToDevice, ctx->stream));
    HY_UP(cudaStreamSynchronize(ctx->stream));
#undef HY_UP
    cleanup();
    vol->uploaded = true;
    // what the upload needs first: the skip grid gives way where memory is short
    const int rc = build_gather(vol);
    if (rc) return rc;
    return hy_skip_build(vol);
}

}  // namespace

int hy_volume_init(hy_ctx *ctx, const hy_volume_desc *desc, hy_volume *v) {
    if (desc->dtype != HY_DTYPE_U8 && desc->dtype != HY_DTYPE_F32)
        return hy_fail(ctx, HY_ERR_INVALID, "volume: dtype must be u8 or f32");
    if (desc->block_size <= 0 || desc->padding < 0 || desc->padding > desc->block_size)
        return hy_fail(ctx, HY_ERR_INVALID, "volume: bad block_size/padding");
    for (int i = 0; i < 3; ++i)
        if (desc->dim[i] <= 0) return hy_fail(ctx, HY_ERR_INVALID, "volume: bad dims");
    v->ctx = ctx;
    v->desc = *desc;
    for (int i = 0; i < 3; ++i) v->grid[i] = (desc->dim[i] + desc->block_size - 1) / desc->block_size;
    long long nb = (long long)v->grid[0] * v->grid[1] * v->grid[2];
    if (nb > (1 << 24)) return hy_fail(ctx, HY_ERR_INVALID, "volume: more than 2^24 bricks");
    v->nbricks = int(nb);
    v->P = desc->block_size + 2 * desc->padding;
    v->elem = desc->dtype == HY_DTYPE_U8 ? 1 : 4;
    size_t bytes = size_t(v->P) * v->P * v->P * v->elem;
    v->slot_stride = (bytes + 255) / 256 * 256;
    // lossless_block_paging.cc:20-22 / rt_block_paging.cc:219-221
    v->k = float(desc->block_size) / float(v->P);
    v->b = float(desc->padding) / float(desc->block_size) * v->k;
    // basic_renderer.hpp:104-118: bbox = [0, raw / block_size], du = 1 / block_size
    float blksz = float(desc->block_size);
    for (int i = 0; i < 3; ++i) v->bbox_max[i] = float(desc->dim[i]) / blksz;
    v->du = 1.f / blksz;
    return HY_OK;
}

extern "C" int hy_volume_create(hy_ctx *ctx, const hy_volume_desc *desc, hy_volume **out) {
    if (!ctx || !desc || !out) return HY_ERR_INVALID;
    *out = nullptr;
    hy_volume *v = new hy_volume();
    int rc = hy_volume_init(ctx, desc, v);
    if (rc) {
        delete v;
        return rc;
    }
    *out = v;
    return HY_OK;
}

extern "C" int hy_volume_destroy(hy_volume *vol) {
    if (!vol) return HY_OK;
    cudaSetDevice(vol->ctx->device);
    cudaStreamSynchronize(vol->ctx->stream);
    free_volume_device(vol);
    delete vol;
    return HY_OK;
}

extern "C" int hy_volume_upload(hy_volume *vol, const void *host_voxels) {
    if (!vol || !host_voxels) return HY_ERR_INVALID;
    if (vol->uploaded || vol->paged)
        return hy_fail(vol->ctx, HY_ERR_STATE,
                       "volume: already has its bricks (create a new volume for new data)");
    HY_CUDA(vol->ctx, cudaSetDevice(vol->ctx->device));
    if (vol->desc.dtype == HY_DTYPE_U8) return upload_impl<unsigned char>(vol, host_voxels);
    return upload_impl<float>(vol, host_voxels);
}

const hy::TexEntry *hy_volume_gather_table(const hy_volume *v) {
    return (v->tex_sampling && v->tex_dev) ? v->tex_dev : nullptr;
}

void hy_volume_gather_view(const hy_volume *v, hy::DevVolume *dv) {
    dv->tex = v->paged_gather ? nullptr : hy_volume_gather_table(v);
    dv->info4 = dv->tex ? v->info4_dev : nullptr;
    dv->paged_gather = v->paged_gather ? 1 : 0;
    // every entry a valid handle (the last texture repeated)
    const int n = int(v->atlas_tex.size());
    const bool any = (dv->tex || v->paged_gather) && n > 0;
    for (int i = 0; i < hy::kMaxGatherTextures; ++i)
        dv->gtex[i] = any ? v->atlas_tex[std::min(i, n - 1)] : 0ull;
}

int hy_gather_layout(hy_ctx *ctx, int P, bool *ok, int *cols, int *rowblocks) {
    *ok = false;
    *cols = *rowblocks = 0;
    int gw = 0, gh = 0;
    HY_CUDA(ctx, cudaDeviceGetAttribute(&gw, cudaDevAttrMaxTexture2DGatherWidth, ctx->device));
    HY_CUDA(ctx, cudaDeviceGetAttribute(&gh, cudaDevAttrMaxTexture2DGatherHeight, ctx->device));
    const long long brick_rows = (long long)P * P;
    if (P <= 0 || P > gw || brick_rows > gh) return HY_OK;
    int rc = gather_check(ctx, ok);
    if (rc) return rc;
    *cols = gw / P;
    *rowblocks = int(gh / brick_rows);
    return HY_OK;
}

int hy_gather_texture_create(hy_ctx *ctx, size_t width, size_t height, cudaArray_t *arr,
                             unsigned long long *tex, unsigned long long *surf) {
    *arr = nullptr;
    *tex = 0;
    if (surf) *surf = 0;
    cudaChannelFormatDesc cd = cudaCreateChannelDesc(8, 0, 0, 0, cudaChannelFormatKindUnsigned);
    const unsigned int flags = cudaArrayTextureGather | (surf ? cudaArraySurfaceLoadStore : 0u);
    cudaError_t e = cudaMallocArray(arr, &cd, width, height, flags);
    if (e != cudaSuccess) {
        *arr = nullptr;
        return hy_cuda_fail(ctx, e, "gather texture allocation");
    }
    cudaTextureObject_t t = make_gather_texture(*arr, &e);
    if (e != cudaSuccess) {
        cudaFreeArray(*arr);
        *arr = nullptr;
        return hy_cuda_fail(ctx, e, "gather texture object");
    }
    if (surf) {
        cudaResourceDesc rd;
        std::memset(&rd, 0, sizeof(rd));
        rd.resType = cudaResourceTypeArray;
        rd.res.array.array = *arr;
        cudaSurfaceObject_t so = 0;
        e = cudaCreateSurfaceObject(&so, &rd);
        if (e != cudaSuccess) {
            cudaDestroyTextureObject(t);
            cudaFreeArray(*arr);
            *arr = nullptr;
            return hy_cuda_fail(ctx, e, "gather texture surface");
        }
        *surf = (unsigned long long)so;
    }
    *tex = (unsigned long long)t;
    return HY_OK;
}

void hy_volume_free_gather(hy_volume *v) { free_gather(v); }

extern "C" int hy_volume_set_gather_sampling(hy_volume *vol, int32_t enable) {
    if (!vol) return HY_ERR_INVALID;
    vol->tex_sampling = enable != 0;
    return HY_OK;
}

extern "C" int hy_volume_gather_sampling(const hy_volume *vol, int32_t *active) {
    if (!vol || !active) return HY_ERR_INVALID;
    *active = hy_volume_gather_table(vol) ? 1 : 0;
    return HY_OK;
}

extern "C" int hy_volume_get_info(const hy_volume *vol, hy_volume_info *out) {
    if (!vol || !out) return HY_ERR_INVALID;
    for (int i = 0; i < 3; ++i) {
        out->grid[i] = vol->grid[i];
        out->bbox_max[i] = vol->bbox_max[i];
    }
    out->nbricks = vol->nbricks;
    out->nonempty = vol->nonempty;
    out->resident = vol->resident;
    out->padded = vol->P;
    out->slot_bytes = (int64_t)vol->slot_stride;
    out->pool_bytes = (int64_t)vol->pool_bytes;
    return HY_OK;
}

extern "C" int hy_volume_thumbnails(const hy_volume *vol, int32_t *chebyshev, float *mean) {
    if (!vol) return HY_ERR_INVALID;
    if (!vol->uploaded) return hy_fail(vol->ctx, HY_ERR_STATE, "volume: not uploaded");
    for (int i = 0; i < vol->nbricks; ++i) {
        if (chebyshev) chebyshev[i] = vol->cheb[i];
        if (mean) mean[i] = vol->mean[i];
    }
    return HY_OK;
}
