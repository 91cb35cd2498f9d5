// hy_diff.cu -- differentiable Volume rendering: forward with per-ray
// checkpoints and the adjoint ray march.
//
// The forward is the Volume shader's march (volume_shader.cu:32-81) over one
// dense f32 brick with a 1-voxel replicate apron, in the reference's float
// operations, with the discontinuous parts fixed: step_size stays 1 (no
// adaptive stepping) and there is no empty-space skipping.  Sampling the
// padded brick at index i is sampling the raw volume at clamp(i-1, 0, n-1),
// so the kernels read the caller's raw n^3 volume directly and the gradient
// of an apron voxel lands on the voxel it replicates.
//
// Every K steps the forward stores the ray state (position, v.w) in a
// checkpoint buffer.  The adjoint walks a ray's segments back to front: it
// restores a checkpoint, recomputes the K samples of that segment (positions,
// sample values, transmittance) into per-thread arrays, and back-propagates
// through front-to-back compositing, the transfer-function lookup and the
// trilinear weights without fetching the voxels a second time.  With c_n = (r a, g a, b a, a), T_n = 1 - v.w before sample n and
// R_n = c_n + (1 - a_n) R_{n+1} the colour composited behind sample n:
//   dL/dc_n = T_n g,   dL/da_n += -T_n (g . R_{n+1}),
// with g = dL/dv of the pixel.  A ray sums its knot and voxel gradients in
// registers while consecutive samples stay in one knot interval / voxel cell;
// knot sums then go through shared memory (one global atomic per knot channel
// and block), voxel sums straight to global atomics (eight per cell).

#include <algorithm>
#include <cstring>

#include "hy_shade.cuh"

using namespace hy;
using namespace hy::dev;

namespace {

constexpr int kMaxDiffViews = 64;
constexpr int kMaxK = 64;
constexpr int kMaxKnots = 256;

struct DiffView {
    float trans[16];
    float ctg;
    float ray_o[3];
};

struct DiffArgs {
    const float *vol;  // raw n^3, x fastest
    int n;             // edge (brick = whole volume)
    float k, b;        // BlockSamplerMapping of the padded brick
    float step;
    int max_steps;
    float density;
    const float4 *tf;
    int ntf;
    int K;             // checkpoint interval
    int max_ckpt;      // checkpoints per ray
    int W, H, nviews;
    DiffView views[kMaxDiffViews];
    float4 *image;     // nviews * H * W
    float4 *ckpt;      // nviews * H * W * max_ckpt (position.xyz, v.w)
    int *nsteps_out;   // steps taken per ray (for the adjoint)
    const float4 *dimage;
    float *dvol;
    float *dtf;        // ntf * 4
    // the padded volume as a gather texture (0: none): slice s of P = n + 2
    // in tile (s / gper, s % gper) of P x P texels, column tiles P apart,
    // with slice (c + 1) * gper repeated as row gper of column c, so slice
    // s + 1 of a footprint is always P rows below slice s
    unsigned long long gtex;
    int gper;
    unsigned int gmagic;  // floor(2^32 / gper) + 1: s / gper = umulhi(s, gmagic) for s < 2^16
};

// Trilinear footprint of the padded brick at brick-local x in [0,1] (the
// interior case of sample_brick: apron >= 1, no wrap, no clamps): the raw
// volume rows and columns of the 2x2x2 taps and the lerp fractions.  Voxel
// indices fit in int (n^3 < 2^31 is checked on the host).
struct Cell {
    int r00, r10, r01, r11;  // row bases (z, y) -> (z * n + y) * n
    int x0, x1;
    float ax, ay, az;
};

// The footprint's lower padded indices (whole numbers) and the lerp fractions.
__device__ __forceinline__ void diff_place(const DiffArgs &a, float lx, float ly, float lz,
                                           float &flx, float &fly, float &flz, float &ax,
                                           float &ay, float &az) {
    const float fd = float(a.n + 2);
    // x and y in packed pairs (products summed by scalar adds), z alone
    const float2 kl = mul2(f2(a.k, a.k), f2(lx, ly));
    const float2 fxy = mul2(f2(fd, fd), f2(__fadd_rn(kl.x, a.b), __fadd_rn(kl.y, a.b)));
    const float fz = fd * (a.k * lz + a.b);
    const float ux = fxy.x - .5f, uy = fxy.y - .5f, uz = fz - .5f;
    flx = floorf(ux);
    fly = floorf(uy);
    flz = floorf(uz);
    const float2 axy = sub2(f2(ux, uy), f2(flx, fly));
    ax = axy.x;
    ay = axy.y;
    az = uz - flz;
}

__device__ __forceinline__ void diff_cell(const DiffArgs &a, float lx, float ly, float lz,
                                          Cell &c) {
    float flx, fly, flz;
    diff_place(a, lx, ly, lz, flx, fly, flz, c.ax, c.ay, c.az);
    const int ix = int(flx), iy = int(fly), iz = int(flz);
    // padded index i -> raw clamp(i - 1, 0, n - 1)
    const int n = a.n;
    c.x0 = iclamp(ix - 1, 0, n - 1);
    c.x1 = iclamp(ix, 0, n - 1);
    const int y0 = iclamp(iy - 1, 0, n - 1), y1 = iclamp(iy, 0, n - 1);
    const int z0 = iclamp(iz - 1, 0, n - 1), z1 = iclamp(iz, 0, n - 1);
    c.r00 = (z0 * n + y0) * n;
    c.r10 = (z0 * n + y1) * n;
    c.r01 = (z1 * n + y0) * n;
    c.r11 = (z1 * n + y1) * n;
}

__device__ __forceinline__ float diff_fetch(const DiffArgs &a, const Cell &c) {
    // taps in z pairs: c<y><x> = (v_xy0, v_xy1); the lerps of sample_brick
    const float2 c00 = f2(__ldg(a.vol + c.r00 + c.x0), __ldg(a.vol + c.r01 + c.x0));
    const float2 c01 = f2(__ldg(a.vol + c.r00 + c.x1), __ldg(a.vol + c.r01 + c.x1));
    const float2 c10 = f2(__ldg(a.vol + c.r10 + c.x0), __ldg(a.vol + c.r11 + c.x0));
    const float2 c11 = f2(__ldg(a.vol + c.r10 + c.x1), __ldg(a.vol + c.r11 + c.x1));
    const float2 bxy = sub2(f2(1.f, 1.f), f2(c.ax, c.ay));
    const float bz = 1.f - c.az;
    const float2 bx2 = f2(bxy.x, bxy.x), ax2 = f2(c.ax, c.ax);
    const float2 X0 = lerp2(c00, bx2, c01, ax2);  // (x0_0, x0_1)
    const float2 X1 = lerp2(c10, bx2, c11, ax2);  // (x1_0, x1_1)
    const float2 Y = lerp2(X0, f2(bxy.y, bxy.y), X1, f2(c.ay, c.ay));
    const float2 Z = mul2(Y, f2(bz, c.az));
    return __fadd_rn(Z.x, Z.y);
}

__device__ __forceinline__ float diff_sample(const DiffArgs &a, float lx, float ly, float lz) {
    Cell c;
    diff_cell(a, lx, ly, lz, c);
    return diff_fetch(a, c);
}

// U samples' values at positions q: through the gather texture (the fractions
// and lerps of diff_sample, the eight taps by two gathers from slices iz and
// iz + 1 of the padded volume, whose texels repeat the clamped border exactly as
// diff_cell's indices do; in the interior a footprint's lower index lies in
// [0, P - 2], so the whole-number texel coordinates stay inside the slice's
// tile), or by loads.  All footprints first, then all taps, then the lerps, so
// that the fetches are in flight together.
template <int U, bool GATHER>
__device__ __forceinline__ void diff_values(const DiffArgs &a, const float (&qx)[U],
                                            const float (&qy)[U], const float (&qz)[U],
                                            float (&v)[U]) {
    if constexpr (!GATHER) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            v[u] = diff_sample(a, qx[u] - floorf(qx[u]), qy[u] - floorf(qy[u]),
                               qz[u] - floorf(qz[u]));
    } else {
        const float fd = float(a.n + 2);
        float X[U], Y[U], az[U];
        float2 axy[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float lx = qx[u] - floorf(qx[u]), ly = qy[u] - floorf(qy[u]),
                        lz = qz[u] - floorf(qz[u]);
            const float2 kl = mul2(f2(a.k, a.k), f2(lx, ly));
            const float2 fxy = mul2(f2(fd, fd), f2(__fadd_rn(kl.x, a.b), __fadd_rn(kl.y, a.b)));
            const float fz = fd * (a.k * lz + a.b);
            const float ux = fxy.x - .5f, uy = fxy.y - .5f, uz = fz - .5f;
            const float flx = floorf(ux), fly = floorf(uy), flz = floorf(uz);
            axy[u] = sub2(f2(ux, uy), f2(flx, fly));
            az[u] = uz - flz;
            const int iz = int(flz);
            const int col = int(__umulhi(unsigned(iz), a.gmagic)), row = iz - col * a.gper;
            // whole numbers below 2^24: exact in any order
            X[u] = __fmaf_rn(float(col), fd, flx + 1.f);
            Y[u] = __fmaf_rn(float(row), fd, fly + 1.f);
        }
        float4 g0[U], g1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            g0[u] = gather_r(a.gtex, X[u], Y[u]);
            g1[u] = gather_r(a.gtex, X[u], Y[u] + fd);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = gather_lerp(g0[u], g1[u], axy[u], az[u]);
    }
}

// The padded volume into the gather texture.  A block takes kFillRows rows of a
// slice, its threads texel pairs along them (8-byte surface writes; single
// texels when P is odd).  256^3: 20-30 us (67 MB read, 69 MB written) against
// 103 us with a thread per texel in 200 k blocks.
constexpr int kFillRows = 32;
template <bool PAIRS>
__global__ void __launch_bounds__(256) diff_fill_kernel(const float *__restrict__ vol, int n,
                                                        int gper, unsigned long long surf) {
    const int P = n + 2, s = blockIdx.y;
    const int vz = min(max(s - 1, 0), n - 1);
    const cudaSurfaceObject_t so = cudaSurfaceObject_t(surf);
    const int col = s / gper, row = s - col * gper;
    const bool twice = row == 0 && col > 0;
    constexpr int W = PAIRS ? 2 : 1;
    const int lane = threadIdx.x & 63;
    const int y1 = min((int(blockIdx.x) + 1) * kFillRows, P);
    for (int y = blockIdx.x * kFillRows + (threadIdx.x >> 6); y < y1; y += 4) {
        const float *src = vol + (size_t(vz) * n + min(max(y - 1, 0), n - 1)) * n;
        for (int x = lane * W; x < P; x += 64 * W) {
            const float v0 = src[min(max(x - 1, 0), n - 1)];
            if constexpr (PAIRS) {
                const float2 v = make_float2(v0, src[min(x, n - 1)]);
                surf2Dwrite(v, so, (col * P + x) * int(sizeof(float)), row * P + y,
                            cudaBoundaryModeZero);
                if (twice)
                    surf2Dwrite(v, so, ((col - 1) * P + x) * int(sizeof(float)), gper * P + y,
                                cudaBoundaryModeZero);
            } else {
                surf2Dwrite(v0, so, (col * P + x) * int(sizeof(float)), row * P + y,
                            cudaBoundaryModeZero);
                if (twice)
                    surf2Dwrite(v0, so, ((col - 1) * P + x) * int(sizeof(float)), gper * P + y,
                                cudaBoundaryModeZero);
            }
        }
    }
}

// emit against the unit box; returns nsteps, sets o and d
__device__ __forceinline__ int diff_emit(const DiffArgs &a, int view, int x, int y, float &ox,
                                         float &oy, float &oz, float &dx, float &dy, float &dz) {
    const DiffView &vw = a.views[view];
    ViewArgs va;
    // gen_ray reads trans / ctg / ray_o / W / H only
    for (int i = 0; i < 16; ++i) va.trans[i] = vw.trans[i];
    va.ctg = vw.ctg;
    va.ray_o[0] = vw.ray_o[0];
    va.ray_o[1] = vw.ray_o[1];
    va.ray_o[2] = vw.ray_o[2];
    va.W = a.W;
    va.H = a.H;
    gen_ray(va, x, y, ox, oy, oz, dx, dy, dz);
    float tnear, tfar;
    if (!intersect(ox, oy, oz, 1.f / dx, 1.f / dy, 1.f / dz, 0.f, 0.f, 0.f, 1.f, 1.f, 1.f, tnear,
                   tfar))
        return 0;
    if (tnear < 0) tnear = 0;
    if (tfar < 0) tfar = 0;
    ox = ox + dx * tnear;
    oy = oy + dy * tnear;
    oz = oz + dz * tnear;
    return min(a.max_steps, int((tfar - tnear) / a.step));
}

// Where a value falls among the knots staged by stage_tf (end knots repeated,
// two zero knots after them): between entries k and k + 1 at fraction al; out
// of [0, 1] (or NaN) between the zeros.
struct TfAt {
    int k;
    float al;
    bool in;
};
__device__ __forceinline__ TfAt tf_at(int n, float fn, float s) {
    float fx = fn * s;
    const bool in = 0.f <= fx && fx <= fn;
    fx = in ? fx : 0.f;
    const float u = fx - .5f;
    const float flr = floorf(u);
    return TfAt{in ? int(flr) + 1 : n + 2, u - flr, in};
}
__device__ __forceinline__ float4 tf_value(const float4 *tf, const TfAt &t) {
    const float4 p = tf[t.k], q = tf[t.k + 1];
    const float bb = 1.f - t.al;
    const float2 b2 = f2(bb, bb), a2 = f2(t.al, t.al);
    const float2 rg = lerp2(f2(p.x, p.y), b2, f2(q.x, q.y), a2);
    const float2 ba = lerp2(f2(p.z, p.w), b2, f2(q.z, q.w), a2);
    return make_float4(rg.x, rg.y, ba.x, ba.y);
}

__device__ __forceinline__ void pixel_of(const DiffArgs &a, int &x, int &y, int &view) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    x = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7);
    y = blockIdx.y * 8 + (warp >> 1) * 4 + (lane >> 3);
    view = blockIdx.z;
}

// U steps of a ray at a time: their taps are fetched together (a step's
// position does not depend on the sample before it).  256^3, four views of
// 512^2, K = 32: 5.30 ms by loads one at a time, 2.9 ms by gathers with 4 in
// flight (L1 86 % busy: the texture's f32 wavefronts); 3 views of 75x51 over
// 48^3 104 and 50 us.
template <int U, bool GATHER>
__global__ void __launch_bounds__(128, U >= 4 ? 4 : 8)
    diff_forward_kernel(const __grid_constant__ DiffArgs a) {
    __shared__ float4 tf[kMaxKnots + kTfPad];
    stage_tf(a.tf, a.ntf, tf);
    __syncthreads();
    int x, y, view;
    pixel_of(a, x, y, view);
    if (x >= a.W || y >= a.H) return;
    const size_t ray = (size_t(view) * a.H + y) * a.W + x;
    float ox, oy, oz, dx, dy, dz;
    const int nsteps = diff_emit(a, view, x, y, ox, oy, oz, dx, dy, dz);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const float sx = dx * a.step, sy = dy * a.step, sz = dz * a.step;  // step_size 1
    float4 *cp = a.ckpt ? a.ckpt + ray * a.max_ckpt : nullptr;
    const float fn = float(a.ntf);
    int left = nsteps;
    while (left > 0) {
        // a checkpoint before steps 0, K, 2K, ...
        if (cp) *cp++ = make_float4(ox, oy, oz, v.w);
        int cnt = a.ckpt ? min(a.K, left) : left;
        left -= cnt;
        while (cnt > 0) {
            float qx[U], qy[U], qz[U], val[U];
            qx[0] = ox;
            qy[0] = oy;
            qz[0] = oz;
#pragma unroll
            for (int u = 1; u < U; ++u) {
                const bool on = u < cnt;  // beyond the segment: the last position again
                qx[u] = on ? qx[u - 1] + sx : qx[u - 1];
                qy[u] = on ? qy[u - 1] + sy : qy[u - 1];
                qz[u] = on ? qz[u - 1] + sz : qz[u - 1];
            }
            diff_values<U, GATHER>(a, qx, qy, qz, val);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                float4 ub = tf_value(tf, tf_at(a.ntf, fn, val[u]));
                ub.w = ub.w * a.density;
                const float w = ub.w;
                const float2 uxy = mul2(f2(ub.x, ub.y), f2(w, w));
                ub.z = ub.z * w;
                if (u < cnt) {
                    const float t = 1.f - v.w;
                    // packed products, scalar sums (see mul2)
                    const float2 txy = mul2(uxy, f2(t, t)), tzw = mul2(f2(ub.z, ub.w), f2(t, t));
                    v.x = __fadd_rn(v.x, txy.x);
                    v.y = __fadd_rn(v.y, txy.y);
                    v.z = __fadd_rn(v.z, tzw.x);
                    v.w = __fadd_rn(v.w, tzw.y);
                }
            }
            ox = qx[U - 1] + sx;
            oy = qy[U - 1] + sy;
            oz = qz[U - 1] + sz;
            cnt -= U;
        }
    }
    a.image[ray] = v;
    if (a.nsteps_out) a.nsteps_out[ray] = nsteps;
}

// Gradient accumulators of one ray.  Consecutive samples mostly share a knot
// interval and a voxel cell, so gradients are summed in registers and flushed
// (one atomic per knot channel / cell corner) only when those change.
struct GradAcc {
    int k = -1;  // knot entries k and k + 1 of stage_tf
    float4 acc_i = make_float4(0.f, 0.f, 0.f, 0.f), acc_j = make_float4(0.f, 0.f, 0.f, 0.f);
    float fx, fy, fz;  // the cell's padded lower indices (whole numbers)
    bool has_cell = false;
    float cacc[8];

    static __device__ __forceinline__ void add4(float4 *e, const float4 &v) {
        atomicAdd(&e->x, v.x);
        atomicAdd(&e->y, v.y);
        atomicAdd(&e->z, v.z);
        atomicAdd(&e->w, v.w);
    }
    // On to interval nk.  A value mostly moves to the next interval up or
    // down, which shares an entry with this one: its sum stays in registers
    // and only the other entry's is added to the block's (shared float adds
    // are compare-and-swap loops, the lanes of a warp after the same few
    // entries).  256^3, four views of 512^2: 9.18 -> 8.89 ms forward and
    // adjoint; 64^3, two of 200^2: 609 -> 442 us.
    __device__ __forceinline__ void to_knots(float4 *gtf, int nk) {
        const bool up = nk == k + 1, down = nk == k - 1;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k >= 0) {
            add4(gtf + (down ? k + 1 : k), down ? acc_j : acc_i);
            if (!up && !down) add4(gtf + k + 1, acc_j);
            const float4 i = acc_i;
            acc_i = up ? acc_j : zero;
            acc_j = down ? i : zero;
        }
        k = nk;
    }
    __device__ __forceinline__ void flush_knots(float4 *gtf) {
        if (k < 0) return;
        add4(gtf + k, acc_i);
        add4(gtf + k + 1, acc_j);
    }
    // The indices are worked out here and not per sample, and away from the
    // border from one base: nearly every step some lane of the warp flushes
    // (256^3, four views of 512^2: 9.50 -> 9.19 ms forward and adjoint).
    __device__ __forceinline__ void flush_cell(const DiffArgs &a) {
        if (!has_cell) return;
        // padded index i -> raw clamp(i - 1, 0, n - 1)
        const int n = a.n, ix = int(fx), iy = int(fy), iz = int(fz);
        const unsigned int m = unsigned(n - 1);
        if (unsigned(ix - 1) < m && unsigned(iy - 1) < m && unsigned(iz - 1) < m) {
            float *p = a.dvol + (((iz - 1) * n + iy - 1) * n + ix - 1);
            float *q = p + n * n;
            add2(p, cacc[0], cacc[1]);
            add2(p + n, cacc[2], cacc[3]);
            add2(q, cacc[4], cacc[5]);
            add2(q + n, cacc[6], cacc[7]);
            return;
        }
        const int x[2] = {iclamp(ix - 1, 0, n - 1), iclamp(ix, 0, n - 1)};
        const int y[2] = {iclamp(iy - 1, 0, n - 1), iclamp(iy, 0, n - 1)};
        const int z[2] = {iclamp(iz - 1, 0, n - 1), iclamp(iz, 0, n - 1)};
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (cacc[t] != 0.f)
                atomicAdd(a.dvol + ((z[t >> 2] * n + y[(t >> 1) & 1]) * n + x[t & 1]), cacc[t]);
    }
    static __device__ __forceinline__ void add2(float *p, float u, float v) {
        if (u != 0.f) atomicAdd(p, u);
        if (v != 0.f) atomicAdd(p + 1, v);
    }
};

// A block's sums of the gradients of stage_tf's entries 0 .. ntf + 1, in as
// many copies as fit (a power of two, at most one a lane): neighbouring lanes,
// whose values mostly lie in the same interval, add to different ones.  64^3,
// two views of 200x150, 32 knots (4 copies) 440 -> 344 us forward and adjoint,
// 256^3, four of 512^2 8.91 -> 8.81 ms; room for twice or four times the copies
// (8 or 16 KB a block, out of the L1) 360 and 347 us, 8.77 and 8.92 ms.
constexpr int kSums = kMaxKnots + 2;
__device__ __forceinline__ int knot_copies(int ntf) {
    int c = 1;
    while (c < 32 && 2 * c * (ntf + 2) <= kSums) c *= 2;
    return c;
}

// The block's sums into dtf: entry i is knot clamp(i - 1, 0, ntf - 1).
__device__ __forceinline__ void add_knots(const DiffArgs &a, const float4 *sums, int copies) {
    for (int i = threadIdx.x; i < a.ntf + 2; i += blockDim.x) {
        float4 v = sums[i];
        for (int c = 1; c < copies; ++c) {
            const float4 w = sums[c * (a.ntf + 2) + i];
            v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
        }
        float *d = a.dtf + 4 * min(max(i - 1, 0), a.ntf - 1);
        if (v.x != 0.f) atomicAdd(d + 0, v.x);
        if (v.y != 0.f) atomicAdd(d + 1, v.y);
        if (v.z != 0.f) atomicAdd(d + 2, v.z);
        if (v.w != 0.f) atomicAdd(d + 3, v.w);
    }
}

// Gradients of one sample: its value's place among the knots (`at`, q its knot
// lerp, aa = q.w * density), the transmittance T before it, R the colour
// composited behind it, its position.
__device__ __forceinline__ void diff_adjoint_sample(const DiffArgs &a, const float4 *tf,
                                                    float4 *gtf, GradAcc &G, const float4 &g,
                                                    const float4 &R, float px, float py, float pz,
                                                    const TfAt &at, const float4 &q, float aa,
                                                    float T) {
    const float al = at.al;
    // The gradient arithmetic has no float-exact counterpart to follow, so it
    // uses fused multiply-adds (the file is compiled with contraction off).
    // dL/dc = T g ; transmittance term through later samples
    const float2 gcxy = mul2(f2(T, T), f2(g.x, g.y)), gczw = mul2(f2(T, T), f2(g.z, g.w));
    const float gcx = gcxy.x, gcy = gcxy.y, gcz = gczw.x, gcw = gczw.y;
    const float gdot = __fmaf_rn(g.w, R.w, __fmaf_rn(g.z, R.z, __fmaf_rn(g.y, R.y, g.x * R.x)));
    const float da =
        __fmaf_rn(-T, gdot, __fmaf_rn(gcz, q.z, __fmaf_rn(gcy, q.y, __fmaf_rn(gcx, q.x, gcw))));
    if (!at.in) return;
    // gradient of the TF output (r, g, b, A)
    const float2 gqxy = mul2(gcxy, f2(aa, aa)), gqzw = mul2(f2(gcz, da), f2(aa, a.density));
    const float4 gq = make_float4(gqxy.x, gqxy.y, gqzw.x, gqzw.y);
    const float bb = 1.f - al;
    if (at.k != G.k) G.to_knots(gtf, at.k);
    {
        const float2 b2 = f2(bb, bb), a2 = f2(al, al);
        const float2 ixy = fma2(gqxy, b2, f2(G.acc_i.x, G.acc_i.y));
        const float2 izw = fma2(gqzw, b2, f2(G.acc_i.z, G.acc_i.w));
        const float2 jxy = fma2(gqxy, a2, f2(G.acc_j.x, G.acc_j.y));
        const float2 jzw = fma2(gqzw, a2, f2(G.acc_j.z, G.acc_j.w));
        G.acc_i = make_float4(ixy.x, ixy.y, izw.x, izw.y);
        G.acc_j = make_float4(jxy.x, jxy.y, jzw.x, jzw.y);
    }
    // d TF / d s = (knot_j - knot_i) * n
    const float4 kj = tf[at.k + 1], ki = tf[at.k];
    const float fn = float(a.ntf);
    const float ds = fn * __fmaf_rn(gq.w, kj.w - ki.w,
                                    __fmaf_rn(gq.z, kj.z - ki.z,
                                              __fmaf_rn(gq.y, kj.y - ki.y, gq.x * (kj.x - ki.x))));
    if (ds == 0.f) return;
    float cx, cy, cz, ax, ay, az;
    diff_place(a, px - floorf(px), py - floorf(py), pz - floorf(pz), cx, cy, cz, ax, ay, az);
    if (!G.has_cell || cx != G.fx || cy != G.fy || cz != G.fz) {
        G.flush_cell(a);
        G.fx = cx;
        G.fy = cy;
        G.fz = cz;
        G.has_cell = true;
#pragma unroll
        for (int t = 0; t < 8; ++t) G.cacc[t] = 0.f;
    }
    // trilinear weights w = (x-weight) * (y-weight) * (z-weight), times ds
    const float bx = 1.f - ax, by = 1.f - ay, bz = 1.f - az;
    const float2 ds2 = f2(ds, ds), yw = f2(by, ay);
    const float2 dz0 = mul2(ds2, mul2(yw, f2(bz, bz)));  // (d00, d10)
    const float2 dz1 = mul2(ds2, mul2(yw, f2(az, az)));  // (d01, d11)
    const float2 xw = f2(bx, ax);
    const float2 c01 = fma2(xw, f2(dz0.x, dz0.x), f2(G.cacc[0], G.cacc[1]));
    const float2 c23 = fma2(xw, f2(dz0.y, dz0.y), f2(G.cacc[2], G.cacc[3]));
    const float2 c45 = fma2(xw, f2(dz1.x, dz1.x), f2(G.cacc[4], G.cacc[5]));
    const float2 c67 = fma2(xw, f2(dz1.y, dz1.y), f2(G.cacc[6], G.cacc[7]));
    G.cacc[0] = c01.x;
    G.cacc[1] = c01.y;
    G.cacc[2] = c23.x;
    G.cacc[3] = c23.y;
    G.cacc[4] = c45.x;
    G.cacc[5] = c45.y;
    G.cacc[6] = c67.x;
    G.cacc[7] = c67.y;
}

// R_n = c_n + (1 - a_n) R_{n+1}
__device__ __forceinline__ float4 diff_behind(const float4 &q, float aa, const float4 &R) {
    const float om = 1.f - aa;
    const float2 om2 = f2(om, om);
    const float2 Rxy = fma2(om2, f2(R.x, R.y), mul2(f2(q.x, q.y), f2(aa, aa)));
    const float2 Rzw = fma2(om2, f2(R.z, R.w), f2(q.z * aa, aa));
    return make_float4(Rxy.x, Rxy.y, Rzw.x, Rzw.y);
}

// The adjoint walks a ray's segments back to front; a segment's recomputed
// sample values and transmittances sit in a per-thread array (8 bytes per
// step), and the reverse walk recomputes each sample position from the
// checkpoint as c + s * step (one rounding per axis instead of the forward's
// s additions: the positions agree to a few ulps, and the trilinear weights'
// derivative is continuous across cell faces, so a sample that lands in the
// neighbouring cell gets the same gradient to first order).
// BLOCKS: resident 128-thread blocks per SM the registers are fitted to.  256^3,
// four views of 512^2, K = 32, forward and adjoint: 8 blocks (64 registers)
// 8.78 ms, 6 (80) 9.03, 5 9.40; launches of fewer than 8 warps of rays a
// scheduler are bound by latency and take 4 (128 registers) with four samples
// of the recompute in flight: 2 of 200^2 over 128^3 (4 warps) 635 against 732 us.
template <int U, int BLOCKS, bool GATHER>
__global__ void __launch_bounds__(128, BLOCKS)
    diff_backward_kernel(const __grid_constant__ DiffArgs a) {
    __shared__ float4 tf[kMaxKnots + kTfPad];
    __shared__ float4 sums[kSums];
    stage_tf(a.tf, a.ntf, tf);
    const int copies = knot_copies(a.ntf);
    for (int i = threadIdx.x; i < copies * (a.ntf + 2); i += blockDim.x)
        sums[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    float4 *gtf = sums + (threadIdx.x & (copies - 1)) * (a.ntf + 2);
    int x, y, view;
    pixel_of(a, x, y, view);
    if (x < a.W && y < a.H) {
        const size_t ray = (size_t(view) * a.H + y) * a.W + x;
        const int nsteps = a.nsteps_out[ray];
        const float4 g = a.dimage[ray];
        float ox0, oy0, oz0, dx, dy, dz;
        diff_emit(a, view, x, y, ox0, oy0, oz0, dx, dy, dz);
        const float sx = dx * a.step, sy = dy * a.step, sz = dz * a.step;
        float4 R = make_float4(0.f, 0.f, 0.f, 0.f);
        const int K = a.K;
        float2 seg_vw[kMaxK];  // (sample value, v.w before the sample)
        const int nseg = (nsteps + K - 1) / K;
        const float fn = float(a.ntf);
        GradAcc G;
        const float4 *cps = a.ckpt + ray * a.max_ckpt;
        for (int seg = nseg - 1; seg >= 0; --seg) {
            const float4 c = cps[seg];
            float ox = c.x, oy = c.y, oz = c.z, vw = c.w;
            const int cnt = min(K, nsteps - seg * K);
            // recompute the segment: values and v.w before each sample, U
            // samples' taps in flight
            for (int s = 0; s < cnt; s += U) {
                float qx[U], qy[U], qz[U], val[U];
                qx[0] = ox;
                qy[0] = oy;
                qz[0] = oz;
#pragma unroll
                for (int u = 1; u < U; ++u) {
                    const bool on = s + u < cnt;
                    qx[u] = on ? qx[u - 1] + sx : qx[u - 1];
                    qy[u] = on ? qy[u - 1] + sy : qy[u - 1];
                    qz[u] = on ? qz[u - 1] + sz : qz[u - 1];
                }
                diff_values<U, GATHER>(a, qx, qy, qz, val);
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const float aa = tf_value(tf, tf_at(a.ntf, fn, val[u])).w * a.density;
                    if (s + u < cnt) {
                        seg_vw[s + u] = make_float2(val[u], vw);
                        vw = vw + aa * (1.f - vw);
                    }
                }
                ox = qx[U - 1] + sx;
                oy = qy[U - 1] + sy;
                oz = qz[U - 1] + sz;
            }
            for (int s = cnt - 1; s >= 0; --s) {
                const float fs = float(s);
                const float2 e = seg_vw[s];
                const TfAt at = tf_at(a.ntf, fn, e.x);
                const float4 q = tf_value(tf, at);
                const float aa = q.w * a.density;
                diff_adjoint_sample(a, tf, gtf, G, g, R, __fmaf_rn(fs, sx, c.x),
                                    __fmaf_rn(fs, sy, c.y), __fmaf_rn(fs, sz, c.z), at, q, aa,
                                    1.f - e.y);
                R = diff_behind(q, aa, R);
            }
        }
        G.flush_knots(gtf);
        G.flush_cell(a);
    }
    __syncthreads();
    add_knots(a, sums, copies);
}

// Small launches: a ray's samples on kLanes neighbouring lanes.  A march of few
// rays is a chain of samples waiting for their taps; here kLanes of them wait
// together, and what has to go in order (compositing, the transmittance, the
// colour behind) every lane of the group works out for itself from the others'
// values, in the order and arithmetic of the kernels above.  A warp holds
// 2x2 rays, a block 4 warps; the lanes of a group stay together (the shuffles
// name the group), groups may part.  Below 2 warps of rays a scheduler: forward
// and adjoint 8 lanes a ray against one, 2 views of 64^2 over 128^3 311 and 541
// us, 3 of 75x51 over 48^3 306 and 372, 2 of 128x96 over 64^3 (1.3 warps) 320 and
// 337, 2 of 200x150 over 64^3 (3 warps) 380 and 353, 2 of 200^2 over 128^3 (4
// warps) 941 and 635.
constexpr int kLanes = 8;
__device__ __forceinline__ bool group_pixel(const DiffArgs &a, int &x, int &y, int &view, int &j,
                                            unsigned int &mask) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane / kLanes;
    j = lane & (kLanes - 1);
    mask = ((1u << kLanes) - 1u) << (lane - j);
    x = blockIdx.x * 4 + (warp & 1) * 2 + (r & 1);
    y = blockIdx.y * 4 + (warp >> 1) * 2 + (r >> 1);
    view = blockIdx.z;
    return x < a.W && y < a.H;
}
dim3 group_grid(const DiffArgs &a) { return dim3((a.W + 3) / 4, (a.H + 3) / 4, a.nviews); }

// Lane j's position: j steps on (no further than step n - 1 of the group).
__device__ __forceinline__ void group_position(int j, int n, float sx, float sy, float sz,
                                               float &x, float &y, float &z) {
#pragma unroll
    for (int i = 1; i < kLanes; ++i)
        if (i <= j && i < n) {
            x = x + sx;
            y = y + sy;
            z = z + sz;
        }
}

template <bool GATHER>
__global__ void __launch_bounds__(128) diff_forward_group_kernel(const __grid_constant__ DiffArgs a) {
    __shared__ float4 tf[kMaxKnots + kTfPad];
    stage_tf(a.tf, a.ntf, tf);
    __syncthreads();
    int x, y, view, j;
    unsigned int mask;
    if (!group_pixel(a, x, y, view, j, mask)) return;  // whole groups
    const size_t ray = (size_t(view) * a.H + y) * a.W + x;
    float ox, oy, oz, dx, dy, dz;
    const int nsteps = diff_emit(a, view, x, y, ox, oy, oz, dx, dy, dz);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    const float sx = dx * a.step, sy = dy * a.step, sz = dz * a.step;
    float4 *cp = a.ckpt ? a.ckpt + ray * a.max_ckpt : nullptr;
    const float fn = float(a.ntf);
    int left = nsteps;
    while (left > 0) {
        if (cp) {
            if (j == 0) *cp = make_float4(ox, oy, oz, v.w);
            ++cp;
        }
        int cnt = a.ckpt ? min(a.K, left) : left;
        left -= cnt;
        for (; cnt > 0; cnt -= kLanes) {
            const int n = min(cnt, kLanes);
            float qx[1] = {ox}, qy[1] = {oy}, qz[1] = {oz}, val[1];
            group_position(j, n, sx, sy, sz, qx[0], qy[0], qz[0]);
            diff_values<1, GATHER>(a, qx, qy, qz, val);
            float4 c = tf_value(tf, tf_at(a.ntf, fn, val[0]));
            c.w = c.w * a.density;
            c.x = c.x * c.w;
            c.y = c.y * c.w;
            c.z = c.z * c.w;
#pragma unroll
            for (int i = 0; i < kLanes; ++i) {
                const float4 q = make_float4(
                    __shfl_sync(mask, c.x, i, kLanes), __shfl_sync(mask, c.y, i, kLanes),
                    __shfl_sync(mask, c.z, i, kLanes), __shfl_sync(mask, c.w, i, kLanes));
                if (i < n) {
                    const float t = 1.f - v.w;
                    const float2 txy = mul2(f2(q.x, q.y), f2(t, t)), tzw = mul2(f2(q.z, q.w), f2(t, t));
                    v.x = __fadd_rn(v.x, txy.x);
                    v.y = __fadd_rn(v.y, txy.y);
                    v.z = __fadd_rn(v.z, tzw.x);
                    v.w = __fadd_rn(v.w, tzw.y);
                }
            }
            ox = __shfl_sync(mask, qx[0], kLanes - 1, kLanes) + sx;
            oy = __shfl_sync(mask, qy[0], kLanes - 1, kLanes) + sy;
            oz = __shfl_sync(mask, qz[0], kLanes - 1, kLanes) + sz;
        }
    }
    if (j) return;
    a.image[ray] = v;
    if (a.nsteps_out) a.nsteps_out[ray] = nsteps;
}

template <bool GATHER>
__global__ void __launch_bounds__(128) diff_backward_group_kernel(const __grid_constant__ DiffArgs a) {
    __shared__ float4 tf[kMaxKnots + kTfPad];
    __shared__ float4 sums[kSums];
    stage_tf(a.tf, a.ntf, tf);
    const int copies = knot_copies(a.ntf);
    for (int i = threadIdx.x; i < copies * (a.ntf + 2); i += blockDim.x)
        sums[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    float4 *gtf = sums + (threadIdx.x & (copies - 1)) * (a.ntf + 2);
    int x, y, view, j;
    unsigned int mask;
    if (group_pixel(a, x, y, view, j, mask)) {
        const size_t ray = (size_t(view) * a.H + y) * a.W + x;
        const int nsteps = a.nsteps_out[ray];
        const float4 g = a.dimage[ray];
        float ox0, oy0, oz0, dx, dy, dz;
        diff_emit(a, view, x, y, ox0, oy0, oz0, dx, dy, dz);
        const float sx = dx * a.step, sy = dy * a.step, sz = dz * a.step;
        float4 R = make_float4(0.f, 0.f, 0.f, 0.f);
        const int K = a.K, nseg = (nsteps + K - 1) / K;
        const float fn = float(a.ntf);
        GradAcc G;
        const float4 *cps = a.ckpt + ray * a.max_ckpt;
        for (int seg = nseg - 1; seg >= 0; --seg) {
            const float4 c = cps[seg];
            float ox = c.x, oy = c.y, oz = c.z, vw = c.w;
            const int cnt = min(K, nsteps - seg * K);
            float2 mine[kMaxK / kLanes];  // this lane's (sample value, v.w before it)
            for (int s = 0; s < cnt; s += kLanes) {
                const int n = min(cnt - s, kLanes);
                float qx[1] = {ox}, qy[1] = {oy}, qz[1] = {oz}, val[1];
                group_position(j, n, sx, sy, sz, qx[0], qy[0], qz[0]);
                diff_values<1, GATHER>(a, qx, qy, qz, val);
                const float aa = tf_value(tf, tf_at(a.ntf, fn, val[0])).w * a.density;
                float before = vw;
#pragma unroll
                for (int i = 0; i < kLanes; ++i) {
                    const float ai = __shfl_sync(mask, aa, i, kLanes);
                    if (i == j) before = vw;
                    if (i < n) vw = vw + ai * (1.f - vw);
                }
                mine[s / kLanes] = make_float2(val[0], before);
                ox = __shfl_sync(mask, qx[0], kLanes - 1, kLanes) + sx;
                oy = __shfl_sync(mask, qy[0], kLanes - 1, kLanes) + sy;
                oz = __shfl_sync(mask, qz[0], kLanes - 1, kLanes) + sz;
            }
            for (int s = (cnt - 1) / kLanes * kLanes; s >= 0; s -= kLanes) {
                const int n = min(cnt - s, kLanes);
                const float2 e = mine[s / kLanes];
                const TfAt at = tf_at(a.ntf, fn, e.x);
                const float4 q = tf_value(tf, at);
                const float aa = q.w * a.density;
                float4 behind = R;
#pragma unroll
                for (int i = kLanes - 1; i >= 0; --i) {
                    const float4 qi = make_float4(
                        __shfl_sync(mask, q.x, i, kLanes), __shfl_sync(mask, q.y, i, kLanes),
                        __shfl_sync(mask, q.z, i, kLanes), 0.f);
                    const float ai = __shfl_sync(mask, aa, i, kLanes);
                    if (i == j) behind = R;
                    if (i < n) R = diff_behind(qi, ai, R);
                }
                if (j < n) {
                    const float fs = float(s + j);
                    diff_adjoint_sample(a, tf, gtf, G, g, behind, __fmaf_rn(fs, sx, c.x),
                                        __fmaf_rn(fs, sy, c.y), __fmaf_rn(fs, sz, c.z), at, q, aa,
                                        1.f - e.y);
                }
                __syncwarp(mask);
            }
        }
        G.flush_knots(gtf);
        G.flush_cell(a);
    }
    __syncthreads();
    add_knots(a, sums, copies);
}

int fill_diff(hy_ctx *ctx, const hy_diff_params *p, const float *vol, const float *tf,
              const hy_view *views, int nviews, int W, int H, DiffArgs &a) {
    if (!p || !vol || !tf || !views) return hy_fail(ctx, HY_ERR_INVALID, "diff: null argument");
    if (p->n <= 1) return hy_fail(ctx, HY_ERR_INVALID, "diff: volume edge must be > 1");
    if ((long long)p->n * p->n * p->n >= (1LL << 31))
        return hy_fail(ctx, HY_ERR_INVALID, "diff: volume edge must be <= 1290 (n^3 < 2^31)");
    if (nviews <= 0 || nviews > kMaxDiffViews)
        return hy_fail(ctx, HY_ERR_INVALID, "diff: 1..64 views");
    // the launch grid is W/16 x H/8 tiles (at most 65535 tile rows) per view
    if (W <= 0 || H <= 0 || (long long)W * H > (1ll << 31) || (H + 7) / 8 > 65535)
        return hy_fail(ctx, HY_ERR_INVALID, "diff: bad resolution");
    if (p->ntf <= 0 || p->ntf > kMaxKnots) return hy_fail(ctx, HY_ERR_INVALID, "diff: 1..256 knots");
    if (p->ckpt_k <= 0 || p->ckpt_k > kMaxK)
        return hy_fail(ctx, HY_ERR_INVALID, "diff: checkpoint interval 1..64");
    if (!(p->sample_rate > 0.f)) return hy_fail(ctx, HY_ERR_INVALID, "diff: sample_rate <= 0");
    std::memset(&a, 0, sizeof(a));
    a.vol = vol;
    a.n = p->n;
    // one brick of edge n with a 1-voxel apron (lossless_block_paging.cc:20-22)
    a.k = float(p->n) / float(p->n + 2);
    a.b = float(1) / float(p->n) * a.k;
    const float du = 1.f / float(p->n);
    a.step = du / 4.f / p->sample_rate;
    a.max_steps = p->max_steps;
    a.density = p->density;
    a.tf = reinterpret_cast<const float4 *>(tf);
    a.ntf = p->ntf;
    a.K = p->ckpt_k;
    // the unit box's diagonal bounds every ray's step count
    const long long maxn = std::min<long long>(p->max_steps, (long long)(1.7320509f / a.step) + 2);
    a.max_ckpt = int((maxn + a.K - 1) / a.K) + 1;
    a.W = W;
    a.H = H;
    a.nviews = nviews;
    for (int v = 0; v < nviews; ++v) {
        std::memcpy(a.views[v].trans, views[v].trans, sizeof(a.views[v].trans));
        a.views[v].ctg = views[v].ctg_fovy_2;
        for (int i = 0; i < 3; ++i) a.views[v].ray_o[i] = views[v].ray_o[i];
    }
    return HY_OK;
}

dim3 diff_grid(const DiffArgs &a) { return dim3((a.W + 15) / 16, (a.H + 7) / 8, a.nviews); }

// Both passes sample the volume through a gather texture refreshed from the
// caller's volume at each call (inside the timed launch); by loads where the
// device cannot make it, and while the stream is captured: a graph would keep the
// texture after the context has replaced it.
struct DiffGather {
    cudaArray_t arr = nullptr;
    unsigned long long tex = 0, surf = 0;
    int w = 0, h = 0;  // texels
};

void free_diff_gather(DiffGather *g) {
    if (!g) return;
    if (g->surf) cudaDestroySurfaceObject(cudaSurfaceObject_t(g->surf));
    if (g->tex) cudaDestroyTextureObject(cudaTextureObject_t(g->tex));
    if (g->arr) cudaFreeArray(g->arr);
    delete g;
}

// Slices per column in h rows (plus the repeated one; less than 2: too few rows)
// and the columns of the footprints' lower slices.
int slices_per_column(int P, int h) { return std::max(0, std::min(h / P, P) - 1); }
int slice_columns(int P, int gper) { return (P - 2) / gper + 1; }

DiffGather *make_diff_gather(int w, int h) {
    DiffGather *g = new DiffGather();
    g->w = w;
    g->h = h;
    cudaChannelFormatDesc cd = cudaCreateChannelDesc(32, 0, 0, 0, cudaChannelFormatKindFloat);
    cudaError_t e = cudaMallocArray(&g->arr, &cd, size_t(w), size_t(h),
                                    cudaArrayTextureGather | cudaArraySurfaceLoadStore);
    cudaResourceDesc rd;
    std::memset(&rd, 0, sizeof(rd));
    rd.resType = cudaResourceTypeArray;
    rd.res.array.array = g->arr;
    cudaTextureDesc td;
    std::memset(&td, 0, sizeof(td));
    td.addressMode[0] = td.addressMode[1] = cudaAddressModeClamp;
    td.filterMode = cudaFilterModePoint;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 0;
    cudaTextureObject_t t = 0;
    cudaSurfaceObject_t so = 0;
    if (e == cudaSuccess) e = cudaCreateTextureObject(&t, &rd, &td, nullptr);
    if (e == cudaSuccess) g->tex = (unsigned long long)t;
    if (e == cudaSuccess) e = cudaCreateSurfaceObject(&so, &rd);
    if (e == cudaSuccess) g->surf = (unsigned long long)so;
    if (e == cudaSuccess) return g;
    free_diff_gather(g);  // e.g. no room: the loads serve this call
    cudaGetLastError();
    return nullptr;
}

// The context's texture, filled from the n^3 volume on the stream.  A texture
// that holds a smaller volume's slices too is kept for it (edges that alternate
// neither allocate nor wait), one too small is replaced once the launches that
// read it are through.  *ok = false (no error): by loads.
int diff_gather_refresh(hy_ctx *ctx, const float *vol, int n, DiffArgs &a, bool *ok) {
    *ok = false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    HY_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) return HY_OK;
    DiffGather *g = static_cast<DiffGather *>(ctx->diff_gather);
    const int P = n + 2;
    int gper = g ? slices_per_column(P, g->h) : 0;
    if (gper < 2 || (long long)slice_columns(P, gper) * P > g->w) {
        int gw = 0, gh = 0;
        HY_CUDA(ctx, cudaDeviceGetAttribute(&gw, cudaDevAttrMaxTexture2DGatherWidth, ctx->device));
        HY_CUDA(ctx, cudaDeviceGetAttribute(&gh, cudaDevAttrMaxTexture2DGatherHeight, ctx->device));
        gper = slices_per_column(P, gh);
        if (gper < 2 || (long long)slice_columns(P, gper) * P > gw) return HY_OK;
        if (g) {
            HY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
            free_diff_gather(g);
            ctx->diff_gather = nullptr;
        }
        const int w = slice_columns(P, gper) * P, h = (gper + 1) * P;
        g = hy_room_for(size_t(w) * h * sizeof(float)) ? make_diff_gather(w, h) : nullptr;
        if (!g) return HY_OK;
        ctx->diff_gather = g;
    }
    const dim3 grid((P + kFillRows - 1) / kFillRows, P);
    if (P % 2 == 0)
        diff_fill_kernel<true><<<grid, 256, 0, ctx->stream>>>(vol, n, gper, g->surf);
    else
        diff_fill_kernel<false><<<grid, 256, 0, ctx->stream>>>(vol, n, gper, g->surf);
    HY_CUDA(ctx, cudaGetLastError());
    a.gtex = g->tex;
    a.gper = gper;
    a.gmagic = unsigned((1ull << 32) / unsigned(gper) + 1);
    *ok = true;
    return HY_OK;
}

// Whether the forward is worth the texture's refresh, which takes a launch and some
// 1.5 ps a voxel while the volume stays in L2 and 3.3 ps beyond.  By loads, up to 64 k
// rays wait about as long as one: 0.3 us a step while the volume stays in L1, 0.5 us
// for a few rays or a volume in L2, else 1 us.  One view of 768^3 at 8^2, 32^2 and 256^2: 1430, 3200, 2920 us by loads and
// 1860, 1880, 2740 through the texture; a quarter of the steps, 394, 925 and (128^2)
// 934 against 1520, 1520 and 1570; 512^3 at 8^2 968 and 664, a quarter of the
// steps 265 and 442; 33^3, 33 steps, 27 and 33; 64^3, 64 steps, 50 and 33.  The
// adjoint, whose samples cost several times as much, is always worth it.
bool forward_through_texture(const DiffArgs &a, long long rays) {
    const double voxels = double(a.n) * a.n * a.n;
    const bool in_l2 = voxels * 4 < 100e6;
    const double refresh = 15. + voxels * (in_l2 ? 1.5e-6 : 3.3e-6);
    const double steps = std::min<double>(a.max_steps, 1.0 / a.step);
    const double step = voxels * 4 < 128e3 ? .3 : in_l2 || rays < 512 ? .5 : 1.;
    const double loads = steps * step * std::max(1., double(rays) / 65536);
    return refresh < .75 * loads;
}

}  // namespace

extern "C" int hy_diff_ckpt_bytes(const hy_diff_params *p, int32_t W, int32_t H, int32_t nviews,
                                  int64_t *bytes) {
    if (!p || !bytes || p->ckpt_k <= 0 || p->n <= 1 || !(p->sample_rate > 0.f))
        return HY_ERR_INVALID;
    const float step = 1.f / float(p->n) / 4.f / p->sample_rate;
    const long long maxn = std::min<long long>(p->max_steps, (long long)(1.7320509f / step) + 2);
    const long long per_ray = (maxn + p->ckpt_k - 1) / p->ckpt_k + 1;
    *bytes = (int64_t)per_ray * 16 * W * H * nviews;
    return HY_OK;
}

extern "C" int hy_diff_forward(hy_ctx *ctx, const hy_diff_params *p, const float *vol_dev,
                               const float *tf_dev, const hy_view *views, int32_t nviews,
                               int32_t W, int32_t H, float *image_dev, float *ckpt_dev,
                               int32_t *nsteps_dev) {
    if (!ctx) return HY_ERR_INVALID;
    // float4 records: knots, image, checkpoints; scalars: volume, step counts
    if (!hy_aligned(tf_dev, 16) || !hy_aligned(image_dev, 16) || !hy_aligned(ckpt_dev, 16) ||
        !hy_aligned(vol_dev, 4) || !hy_aligned(nsteps_dev, 4))
        return hy_fail(ctx, HY_ERR_INVALID,
                       "diff: misaligned buffer (knots, image, checkpoints 16-byte; others 4)");
    if (!image_dev) return hy_fail(ctx, HY_ERR_INVALID, "diff: null image");
    DiffArgs a;
    int rc = fill_diff(ctx, p, vol_dev, tf_dev, views, nviews, W, H, a);
    if (rc) return rc;
    if ((ckpt_dev == nullptr) != (nsteps_dev == nullptr))
        return hy_fail(ctx, HY_ERR_INVALID, "diff: checkpoints and step counts go together");
    a.image = reinterpret_cast<float4 *>(image_dev);
    a.ckpt = reinterpret_cast<float4 *>(ckpt_dev);
    a.nsteps_out = nsteps_dev;
    HY_CUDA(ctx, cudaSetDevice(ctx->device));
    // the texture's refresh is part of the timed launch
    HY_CUDA(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    bool gathers = false;
    const long long rays = (long long)W * H * nviews, per_warp = 32ll * 4 * ctx->sms;
    if (forward_through_texture(a, rays)) {
        rc = diff_gather_refresh(ctx, vol_dev, p->n, a, &gathers);
        if (rc) return rc;
    }
    if (gathers && rays < 2 * per_warp)
        diff_forward_group_kernel<true><<<group_grid(a), 128, 0, ctx->stream>>>(a);
    else if (gathers)
        diff_forward_kernel<4, true><<<diff_grid(a), 128, 0, ctx->stream>>>(a);
    else
        diff_forward_kernel<1, false><<<diff_grid(a), 128, 0, ctx->stream>>>(a);
    HY_CUDA(ctx, cudaGetLastError());
    HY_CUDA(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    ctx->stats_pending = true;
    ctx->pend_count = 0;
    ctx->pend_pixels = (int64_t)W * H * nviews;
    return HY_OK;
}

extern "C" int hy_diff_backward(hy_ctx *ctx, const hy_diff_params *p, const float *vol_dev,
                                const float *tf_dev, const hy_view *views, int32_t nviews,
                                int32_t W, int32_t H, const float *dimage_dev,
                                const float *ckpt_dev, const int32_t *nsteps_dev,
                                float *dvol_dev, float *dtf_dev) {
    if (!ctx) return HY_ERR_INVALID;
    if (!hy_aligned(tf_dev, 16) || !hy_aligned(dimage_dev, 16) || !hy_aligned(ckpt_dev, 16) ||
        !hy_aligned(vol_dev, 4) || !hy_aligned(nsteps_dev, 4) || !hy_aligned(dvol_dev, 4) ||
        !hy_aligned(dtf_dev, 4))
        return hy_fail(ctx, HY_ERR_INVALID,
                       "diff: misaligned buffer (knots, image, checkpoints 16-byte; others 4)");
    if (!dimage_dev || !ckpt_dev || !nsteps_dev || !dvol_dev || !dtf_dev)
        return hy_fail(ctx, HY_ERR_INVALID, "diff: null argument");
    DiffArgs a;
    int rc = fill_diff(ctx, p, vol_dev, tf_dev, views, nviews, W, H, a);
    if (rc) return rc;
    a.dimage = reinterpret_cast<const float4 *>(dimage_dev);
    a.ckpt = const_cast<float4 *>(reinterpret_cast<const float4 *>(ckpt_dev));
    a.nsteps_out = const_cast<int *>(nsteps_dev);
    a.dvol = dvol_dev;
    a.dtf = dtf_dev;
    HY_CUDA(ctx, cudaSetDevice(ctx->device));
    // the texture's refresh is part of the timed launch
    HY_CUDA(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
    bool gathers = false;
    rc = diff_gather_refresh(ctx, vol_dev, p->n, a, &gathers);
    if (rc) return rc;
    const long long rays = (long long)W * H * nviews, per_warp = 32ll * 4 * ctx->sms;
    if (gathers && rays < 2 * per_warp)
        diff_backward_group_kernel<true><<<group_grid(a), 128, 0, ctx->stream>>>(a);
    else if (gathers && rays < 8 * per_warp)
        diff_backward_kernel<4, 4, true><<<diff_grid(a), 128, 0, ctx->stream>>>(a);
    else if (gathers)
        diff_backward_kernel<2, 8, true><<<diff_grid(a), 128, 0, ctx->stream>>>(a);
    else
        diff_backward_kernel<1, 6, false><<<diff_grid(a), 128, 0, ctx->stream>>>(a);
    HY_CUDA(ctx, cudaGetLastError());
    HY_CUDA(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
    ctx->stats_pending = true;
    ctx->pend_count = 0;
    ctx->pend_pixels = (int64_t)W * H * nviews;
    return HY_OK;
}

void hy_diff_release(hy_ctx *ctx) {
    if (!ctx) return;
    free_diff_gather(static_cast<DiffGather *>(ctx->diff_gather));
    ctx->diff_gather = nullptr;
}
