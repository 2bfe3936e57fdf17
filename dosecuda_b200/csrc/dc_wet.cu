// dc_wet.cu — radiological depth: per-voxel ray march to the source and the
// proton beam's-eye-view smoothing.
//
// wet_march_kernel restates rayTraceKernel (CudaClasses.cu:180-228): from
// each voxel centre, 1 mm steps towards the source, hardware-trilinear
// density samples, WET(cm) = -0.05 + sum 0.1*max(rho,0) until the sample's
// texture coordinate leaves [0,n).  wet_smooth_kernel restates
// smoothRayKernel (IMPTClasses.cu:139-202): the mean of the voxel's WET and
// the nearest-voxel WET at radii 1,2,.. mm (r < min(10*WET, 10)) along six
// BEV directions.
//
// B200 mapping: the march is bound by the texture unit's trilinear fetches,
// one per 1 mm sample: by their latency in small volumes (wet_march_kernel,
// eight lanes per ray), by their rate in larger ones, where samples in uniform
// density are added without a fetch (wet_march_leap_kernel).  The smoothing
// adds 54 voxels at constant index offsets; see there.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "../../include/dosecuda.h"
#include "dc_common.cuh"
#include "dc_runtime.cuh"
#include "dc_kernels.cuh"

namespace dc {

DC_BOUNDS_WORD

// March of the smaller volumes (march_leaps): eight lanes per ray, two samples
// of each in flight; a block takes 16 voxels of a row.  Measured on B200 (us,
// a thread per ray of 32 x 4 voxels per block -> eight lanes): 24^3 at 3 mm
// 18.6 -> 11.3, 44 x 40 x 36 at 3 mm 24 -> 18.5, 56^3 at 2 mm 41 -> 32.5, 80^3 at
// 2 mm 103 -> 92; in larger volumes the texture rate binds either way (127 x
// 113 x 91 288 -> 318).  Four lanes of four samples are 2 us slower at 24^3 and
// 1.5 us faster at 80^3.
constexpr int kRayLanes = 8, kRayEach = 2;
__global__ void __launch_bounds__(128) wet_march_kernel(Grid g, Frame f, cudaTextureObject_t density,
                                                        float *__restrict__ wet) {
    const int i = blockIdx.x * (128 / kRayLanes) + threadIdx.x / kRayLanes, j = blockIdx.y, k = blockIdx.z;
    const float3 p = voxel_xyz(g, f, i, j, k);
    const float3 u = unit_to_source(f, p);
    const float sum = march_lanes<kRayLanes, kRayEach>(g, f, density, p, u, i < g.nx);
    const long long v = (long long)i + (long long)g.nx * (j + (long long)g.ny * k);
    if (i < g.nx && threadIdx.x % kRayLanes == 0 && DC_IN_BOUNDS(v, g.n(), 1)) wet[v] = sum;
}

// Uniform density leapt over, in the larger volumes.  A plain march is bound by
// the texture unit (1.9 trilinear samples per clock and SM, one per mm of ray).
// Where all eight voxels of a sample hold one number c the filter returns c
// (its weights are multiples of 1/256 that add up to 1), so such a sample
// needs no fetch: phantoms, the air around a patient, structures overridden to
// one density.  A map of bricks of kBrick^3 voxels holds each brick's value
// and the radius r (in bricks, Chebyshev) within which every brick of the
// volume is uniform with that value; from a point in such a brick a ray may
// take kBrick r - 1 voxels of steps, along the axis it crosses fastest, as
// additions of c.  They are the plain march's additions in its order, so the
// sum is the same bit for bit.  The map is built from the texture in every
// call, its radii only where enough bricks are uniform; otherwise the march
// does not look at it.
//
// Measured on B200 (us, map + march, before -> after): 96^3 at 2 mm of water
// with inserts 190 -> 18 + 67; 127 x 113 x 91 oblique 288 -> 21 + 228; 256 x
// 256 x 160, noisy body in air 3735 -> 50 + 2360; the same filled with one
// value 51 + 414.  With noise in every voxel the map is a loss: 38 + 3711 there
// (3710), 96^3 14 + 184 (186), 80^3 11 + 101 (104).  The looks at the map cost
// 1 %; every 4 samples instead of every 6 2 %, every 8 loses 3 % on the body.
// Bricks of 8 voxels gave 2750 on the body (fewer leaps near its surface), of 2
// voxels 2367 with a map of 210.  Testing 256 bricks in a kernel of its own first
// cost more than it saved (28 us instead of 17 where the map is made), so did
// the eight-lane march as a second launch where nothing is uniform (its empty
// blocks take 8 to 15 us).  The photon depth's marched voxels gain less than the
// map costs (their rays run through the noisy body) and do not leap.
constexpr int kBrick = 4;
constexpr int kBrickRadius = 4;
constexpr int kFetches = 6;  // samples fetched between two looks at the map

struct Bricks {
    float *value = nullptr;           // NaN: not uniform
    unsigned char *radius = nullptr;  // 0: the brick or a neighbour differs
    unsigned *uniform = nullptr;      // uniform bricks; with fewer than `least` of them nothing is leapt over
    unsigned least = 0;
    int nx = 0, ny = 0, nz = 0;
};

// Leaps of one ray, p + t u: steps t may not leave the voxel centres' box
// (beyond it the filter blends in the border value).
struct Leaps {
    float per_brick;  // steps per kBrick voxels of the fastest axis
    float one;        // and per voxel
    int last;         // last step inside the box

    __device__ __forceinline__ Leaps(const Grid &g, const Frame &f, float3 p, float3 u) {
        const float3 c = tex_coord(g, f, p);
        const float cc[3] = {c.x, c.y, c.z}, rate[3] = {u.x * g.inv_sx, u.y * g.inv_sy, u.z * g.inv_sz};
        const float n[3] = {(float)g.nx, (float)g.ny, (float)g.nz};
        float fast = 0.0f, box = 1.0e6f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            fast = fmaxf(fast, fabsf(rate[a]));
            const float edge = fmaf(1.0e-6f, n[a], 0.5f);  // more than a coordinate's rounding inside
            if (rate[a] != 0.0f) box = fminf(box, (rate[a] > 0.0f ? n[a] - edge - cc[a] : edge - cc[a]) / rate[a]);
        }
        one = 1.0f / fast;
        per_brick = (float)kBrick * one;
        last = (int)floorf(box);
    }
    // Samples from step t on (at tc) that all read *value; 0 where the map cannot tell.
    __device__ __forceinline__ int at(const Bricks &B, float3 tc, int t, float *value) const {
        if (t > last) return 0;
        const long long b = (int)tc.x / kBrick + (long long)B.nx * ((int)tc.y / kBrick + (long long)B.ny * ((int)tc.z / kBrick));
        if (!DC_IN_BOUNDS(b, (long long)B.nx * B.ny * B.nz, 5)) return 0;
        const int r = __ldg(B.radius + b);
        if (r == 0) return 0;
        *value = __ldg(B.value + b);
        return min((int)(fmaf((float)r, per_brick, -one)), last - t) + 1;
    }
};

// Value of a brick, NaN where its voxels differ (bit for bit) or hold a number
// whose filtered value might not be exact.  By a warp; reading at a texel's
// centre returns the stored value.
__device__ __forceinline__ float brick_value(const Grid &g, const Bricks &B, cudaTextureObject_t density, int b) {
    const int lane = threadIdx.x & 31;
    const int bz = b / (B.nx * B.ny), by = (b - bz * B.nx * B.ny) / B.nx, bx = b - (bz * B.ny + by) * B.nx;
    const int x0 = bx * kBrick, y0 = by * kBrick, z0 = bz * kBrick;
    const float c = tex3D<float>(density, x0 + 0.5f, y0 + 0.5f, z0 + 0.5f);
    bool same = true;
#pragma unroll
    for (int q = 0; q < kBrick * kBrick * kBrick; q += 32) {
        const int e = q + lane;
        // beyond the volume's end the brick's own last voxels again
        const int i = min(x0 + e % kBrick, g.nx - 1), j = min(y0 + e / kBrick % kBrick, g.ny - 1);
        const int k = min(z0 + e / (kBrick * kBrick), g.nz - 1);
        same = same && __float_as_uint(tex3D<float>(density, i + 0.5f, j + 0.5f, k + 0.5f)) == __float_as_uint(c);
    }
    const bool plain = c == 0.0f || (fabsf(c) >= 1.0e-30f && fabsf(c) <= 1.0e30f);
    return __all_sync(0xffffffffu, same) && plain ? c : NAN;
}

// Values of all bricks, and the number of uniform ones (0 before).
__global__ void __launch_bounds__(128) brick_value_kernel(Grid g, Bricks B, cudaTextureObject_t density) {
    const int n = B.nx * B.ny * B.nz;
    int uniform = 0;
    for (int b = blockIdx.x * 4 + (threadIdx.x >> 5); b < n; b += gridDim.x * 4) {
        const float c = brick_value(g, B, density, b);
        uniform += c == c;
        if ((threadIdx.x & 31) == 0 && DC_IN_BOUNDS(b, n, 6)) B.value[b] = c;
    }
    __shared__ int s_uniform;
    if (threadIdx.x == 0) s_uniform = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && uniform > 0) atomicAdd(&s_uniform, uniform);
    __syncthreads();
    if (threadIdx.x == 0 && s_uniform > 0) atomicAdd(B.uniform, (unsigned)s_uniform);
}

// Radius of each brick: the Chebyshev distance to the nearest brick of another
// value, less one, capped.  Separable: the distance along x, then the smallest
// max(|dy|, that of the row dy away), then likewise along z; a block takes
// kTile^3 bricks with their surroundings in shared memory.
constexpr int kTile = 8, kSpan = kTile + 2 * kBrickRadius;
__global__ void __launch_bounds__(512) brick_radius_kernel(Bricks B) {
    __shared__ float val[kSpan][kSpan][kSpan];
    __shared__ unsigned char dx[kSpan][kSpan][kTile], dxy[kSpan][kTile][kTile];
    if (*B.uniform < B.least) return;
    const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile, z0 = blockIdx.z * kTile;
    for (int e = threadIdx.x; e < kSpan * kSpan * kSpan; e += 512) {
        const int lx = e % kSpan, ly = e / kSpan % kSpan, lz = e / (kSpan * kSpan);
        // outside the volume the nearest brick inside again, which adds no nearer difference
        const int x = min(max(x0 + lx - kBrickRadius, 0), B.nx - 1), y = min(max(y0 + ly - kBrickRadius, 0), B.ny - 1);
        const int z = min(max(z0 + lz - kBrickRadius, 0), B.nz - 1);
        val[lz][ly][lx] = __ldg(B.value + x + B.nx * (y + B.ny * z));
    }
    __syncthreads();
    constexpr int kFar = kBrickRadius + 1;
    for (int e = threadIdx.x; e < kSpan * kSpan * kTile; e += 512) {
        const int lx = e % kTile, ly = e / kTile % kSpan, lz = e / (kTile * kSpan);
        const float c = val[lz][ly][lx + kBrickRadius];
        int d = kFar;
#pragma unroll
        for (int o = -kBrickRadius; o <= kBrickRadius; ++o)
            if (val[lz][ly][lx + kBrickRadius + o] != c) d = min(d, abs(o));  // NaN differs from itself: 0
        dx[lz][ly][lx] = (unsigned char)d;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kSpan * kTile * kTile; e += 512) {
        const int lx = e % kTile, ly = e / kTile % kTile, lz = e / (kTile * kTile);
        const float c = val[lz][ly + kBrickRadius][lx + kBrickRadius];
        int d = kFar;
#pragma unroll
        for (int o = -kBrickRadius; o <= kBrickRadius; ++o) {
            const int y = ly + kBrickRadius + o;
            d = min(d, val[lz][y][lx + kBrickRadius] != c ? abs(o) : max(abs(o), (int)dx[lz][y][lx]));
        }
        dxy[lz][ly][lx] = (unsigned char)d;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kTile * kTile * kTile; e += 512) {
        const int lx = e % kTile, ly = e / kTile % kTile, lz = e / (kTile * kTile);
        const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
        if (x >= B.nx || y >= B.ny || z >= B.nz) continue;
        const float c = val[lz + kBrickRadius][ly + kBrickRadius][lx + kBrickRadius];
        int d = kFar;
#pragma unroll
        for (int o = -kBrickRadius; o <= kBrickRadius; ++o) {
            const int w = lz + kBrickRadius + o;
            d = min(d, val[w][ly + kBrickRadius][lx + kBrickRadius] != c ? abs(o) : max(abs(o), (int)dxy[w][ly][lx]));
        }
        const int b = x + B.nx * (y + B.ny * z);
        if (DC_IN_BOUNDS(b, B.nx * B.ny * B.nz, 7)) B.radius[b] = (unsigned char)max(d - 1, 0);
    }
}

// Lanes of a warp: 8 x 4 voxels, warps of a block along z.
constexpr int kMarchX = 8, kMarchY = 4, kMarchZ = 4;

__global__ void __launch_bounds__(32 * kMarchZ) wet_march_leap_kernel(Grid g, Frame f, Bricks B,
                                                                      cudaTextureObject_t density,
                                                                      float *__restrict__ wet) {
    const int i = blockIdx.x * kMarchX + threadIdx.x, j = blockIdx.y * kMarchY + threadIdx.y;
    const int k = blockIdx.z * kMarchZ + threadIdx.z;
    if (i >= g.nx || j >= g.ny || k >= g.nz) return;

    const float3 p = voxel_xyz(g, f, i, j, k);
    const float3 u = unit_to_source(f, p);
    const Leaps leaps(g, f, p, u);
    const bool worth = *B.uniform >= B.least;

    float wet_sum = -0.05f;
    int t = 0;
    auto coord = [&](int step) {
        float3 q;
        q.x = fmaf(u.x, (float)step, p.x);
        q.y = fmaf(u.y, (float)step, p.y);
        q.z = fmaf(u.z, (float)step, p.z);
        return tex_coord(g, f, q);
    };
    // The samples inside the volume form a prefix of t = 0,1,2,... (each
    // coordinate is monotonic in t), so the loop stops at the first exit.
    for (bool inside = true; inside;) {
        float3 tc = coord(t);
        inside = tex_inside(g, tc);
        if (!inside) break;
        float c;
        const int n = worth ? leaps.at(B, tc, t, &c) : 0;
        if (n > 0) {
            c = fmaxf(c, 0.0f);
#pragma unroll 4
            for (int q = 0; q < n; ++q) wet_sum = fmaf(c, 0.1f, wet_sum);
            t += n;
            continue;
        }
#pragma unroll
        for (int q = 0; q < kFetches; ++q) {
            if (q > 0) {
                tc = coord(t);
                if (!tex_inside(g, tc)) {
                    inside = false;
                    break;
                }
            }
            const float rho = tex3D<float>(density, tc.x, tc.y, tc.z);
            wet_sum = fmaf(fmaxf(rho, 0.0f), 0.1f, wet_sum);
            ++t;
        }
    }
    const long long v = (long long)i + (long long)g.nx * (j + (long long)g.ny * k);
    if (DC_IN_BOUNDS(v, g.n(), 1)) wet[v] = wet_sum;
}

// Nearest voxel index (int)roundf(v / s) of the reference's smoothing
// (CudaClasses.cuh:112-116: IEEE division, then round half away from zero),
// without the division and the float-to-int conversion on the common path.
// With r = RN(1/s), qa = RN(v * r) differs from Q = RN(v / s) by less than
// |qa| * 2^-22 (two relative roundings of 2^-24 each on r and qa, one on Q).
// When no half-integer lies within |qa| * 2^-21 of qa, Q and qa round to the
// same integer, which the magic-number addition (1.5 * 2^23, exact for
// |qa| < 2^21) delivers as bits of a float.  Otherwise — and for inf/NaN —
// the reference's expression itself is evaluated, so the index is always
// exactly the reference's.
__device__ __forceinline__ int nearest_index(float v, float s, float r) {
    const float magic = 12582912.0f;  // 1.5 * 2^23
    const float qa = __fmul_rn(v, r);
    const float t = __fadd_rn(qa, magic);
    const float d = fabsf(__fsub_rn(qa, __fsub_rn(t, magic)));  // distance to the nearest integer
    const float aq = fabsf(qa);
    if (aq < 2097152.0f && __fsub_rn(0.5f, d) > __fmul_rn(aq, 4.76837158203125e-07f)) {  // 2^-21
        return __float_as_int(t) - 0x4B400000;
    }
    return (int)roundf(v / s);
}

// (int)roundf(v / s) (CudaClasses.cuh:112-116): half away from zero, for any spacing; a power-of-two
// spacing's reciprocal is exact, so the quotient is one product.
__device__ __forceinline__ int reference_index(float v, float s, float r, bool pow2) {
    if (!pow2) return nearest_index(v, s, r);
    const float q = __fmul_rn(v, r);
    return __float2int_rz(__fadd_rz(q, copysignf(0.5f, q)));
}

// Smoothing.  The reference samples, per voxel, the nearest voxel at 54 points
// h + dr (cos, sin, 0) of the head frame (six directions, dr = 1 .. 9 mm).
// The displacement from the voxel to such a point is the same for every
// voxel, so the nearest voxel is the voxel's own index plus a constant offset
// per axis, except where the displacement lies next to a half-integer number
// of voxels: there the float rounding of the reference's expression decides,
// and the axis is marked to be evaluated exactly (WetSmoothTable).  The sum
// keeps the reference's order, so the result is the reference's bit for bit.
//
// Bounds: a sample used to be some 40 instructions of rotation and rounding;
// as a constant offset it is one load and one add.  The loads hit L1 (blocks
// of 32 x 4 x 4 voxels share most of their neighbours in whichever plane the
// disk lies) at about 4 clocks per warp, an unaligned row touching two lines.
// Measured (ms): 96^3 at 2 mm, gantry 0, where a third of the samples fall on
// half-integers, 0.138 -> 0.096; 127 x 113 x 91 oblique 0.132 -> 0.045;
// 256 x 256 x 160 0.854 -> 0.228.  Staging the block and its reach in shared
// memory (one wavefront per sample) gave 0.21 on the last, where the staging
// itself takes as many instructions as the sums, and twice the time on small
// grids with fewer blocks than SMs.

// Coordinates (relative to the grid's origin) of a voxel's sample point, as
// the reference's head_to_image and its float sums give them.  Written with
// explicit fused multiply-adds: which product of a rotation is rounded decides
// the picks at half-integers, and left to the compiler it changes with the
// code around it.
struct SmoothPoint {
    const Frame &f;
    float3 h;
    float dr, si, co;
    __device__ __forceinline__ float gx() const {
        return __fmaf_rn(-__fmaf_rn(dr, co, h.x), f.cga, -__fmul_rn(h.z, f.sga));
    }
    __device__ __forceinline__ float gz() const { return __fmaf_rn(dr, si, h.y); }
    __device__ __forceinline__ float x() const {
        return __fadd_rn(__fmaf_rn(gx(), f.cta, __fmul_rn(gz(), f.sta)), f.isox);
    }
    __device__ __forceinline__ float y() const {
        return __fadd_rn(__fmaf_rn(-__fmaf_rn(dr, co, h.x), f.sga, __fmul_rn(h.z, f.cga)), f.isoy);
    }
    __device__ __forceinline__ float z() const {
        return __fadd_rn(__fmaf_rn(-gx(), f.sta, __fmul_rn(gz(), f.cta)), f.isoz);
    }
};

template <bool kInside, bool kExact>
__device__ __forceinline__ void smooth_general(const Grid &g, const Frame &f, const WetSmoothTable &T,
                                               const float (&s_dir)[2][6], const float *__restrict__ wet, int i, int j,
                                               int k, long long v, float rmax, float &sum, int &n) {
    float3 h = make_float3(0.f, 0.f, 0.f);
    if (kExact) h = image_to_head<false>(f, voxel_xyz(g, f, i, j, k));
    // samples per direction of the warp's widest radius; narrower lanes mask theirs, so that the
    // loads of several samples are in flight at once
    const int mine = rmax > 9.0f ? 9 : (rmax > 1.0f ? (int)ceilf(rmax) - 1 : 0);
    const int cnt = __reduce_max_sync(__activemask(), mine);
    for (int d = 0; d < 6; ++d) {
#pragma unroll 3
        for (int m = 0; m < cnt; ++m) {
            const float dr = (float)(m + 1);
            const int e = d * 9 + m;
            int qi = i + T.dx[e], qj = j + T.dy[e], qk = k + T.dz[e];
            long long u = v + T.lin[e];
            const int exact = kExact ? T.exact[e] : 0;
            if (exact != 0) {
                const SmoothPoint P{f, h, dr, s_dir[0][d], s_dir[1][d]};
                if (exact & 1) qi = reference_index(P.x(), g.sx, g.inv_sx, T.pow2 & 1);
                if (exact & 2) qj = reference_index(P.y(), g.sy, g.inv_sy, T.pow2 & 2);
                if (exact & 4) qk = reference_index(P.z(), g.sz, g.inv_sz, T.pow2 & 4);
                u = (long long)qi + (long long)g.nx * (qj + (long long)g.ny * qk);
            }
            const bool ok = dr < rmax && ((kInside && exact == 0) ||
                                          ((unsigned)qi < (unsigned)g.nx && (unsigned)qj < (unsigned)g.ny &&
                                           (unsigned)qk < (unsigned)g.nz));
            const float value = ok && DC_IN_BOUNDS(u, g.n(), 3) ? __ldg(wet + u) : 0.0f;
            sum += value;
            n += ok ? 1 : 0;
        }
    }
}

__global__ void __launch_bounds__(512) wet_smooth_kernel(Grid g, Frame f, const __grid_constant__ WetSmoothTable T,
                                                         const float *__restrict__ wet, float *__restrict__ wet_s) {
    // The six direction cosines/sines, evaluated once per block by the device's own sincosf.
    __shared__ float s_dir[2][6];
    if (T.n_exact > 0) {
        const int tid = (threadIdx.z * blockDim.y + threadIdx.y) * blockDim.x + threadIdx.x;
        if (tid < 6) sincosf((float)tid * CUDART_PI_F / 3.0f, &s_dir[0][tid], &s_dir[1][tid]);
        __syncthreads();
    }
    const int i0 = blockIdx.x * 32, i = i0 + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= g.nx || j >= g.ny || k >= g.nz) return;
    // every sample of the warp's row inside the grid
    const bool inside = i0 >= T.reach[0] && i0 + 32 + T.reach[0] <= g.nx && j >= T.reach[1] && j + T.reach[1] < g.ny &&
                        k >= T.reach[2] && k + T.reach[2] < g.nz;
    const long long v = (long long)i + (long long)g.nx * (j + (long long)g.ny * k);
    const float c = DC_IN_BOUNDS(v, g.n(), 2) ? __ldg(wet + v) : 0.0f;
    const float rmax = c * 10.0f;
    float sum = c;
    int n = 1;
    if (T.n_exact == 0) {
        if (inside && __all_sync(__activemask(), rmax > 9.0f)) {
#pragma unroll 18
            for (int e = 0; e < kSmoothSamples; ++e) {
                const long long u = v + T.lin[e];
                sum += DC_IN_BOUNDS(u, g.n(), 3) ? __ldg(wet + u) : 0.0f;
            }
            n += kSmoothSamples;
        } else if (inside) {
            smooth_general<true, false>(g, f, T, s_dir, wet, i, j, k, v, rmax, sum, n);
        } else {
            smooth_general<false, false>(g, f, T, s_dir, wet, i, j, k, v, rmax, sum, n);
        }
    } else {
        if (inside)
            smooth_general<true, true>(g, f, T, s_dir, wet, i, j, k, v, rmax, sum, n);
        else
            smooth_general<false, true>(g, f, T, s_dir, wet, i, j, k, v, rmax, sum, n);
    }
    if (DC_IN_BOUNDS(v, g.n(), 2)) wet_s[v] = sum / (float)n;
}

WetSmoothTable make_wet_smooth_table(const Grid &g, const Frame &f) {
    WetSmoothTable T{};
    const double sp[3] = {g.sx, g.sy, g.sz};
    const double iso[3] = {f.isox, f.isoy, f.isoz};
    const int nn[3] = {g.nx, g.ny, g.nz};
    // Largest coordinate the reference's float chain meets (relative to the
    // isocentre, and to the grid's origin), mm.  The chain rounds about a
    // dozen times at up to half an ulp of it and its float sines and cosines
    // rotate by up to 1e-7 too far or too short: 1.2e-6 of it in all; eps
    // allows 3e-6.
    double m = 0.0;
    for (int a = 0; a < 3; ++a) {
        const double hi = std::max(std::fabs(iso[a]), std::fabs(nn[a] * sp[a] - iso[a]));
        m += hi * hi;
    }
    m = std::sqrt(m) + std::max({nn[0] * sp[0], nn[1] * sp[1], nn[2] * sp[2]}) + 20.0;
    const double eps = 3e-6 * m;
    const float inv[3] = {g.inv_sx, g.inv_sy, g.inv_sz};
    for (int a = 0; a < 3; ++a) {
        int e2 = 0;
        if (std::frexp(sp[a], &e2) == 0.5 && (double)inv[a] * sp[a] == 1.0) T.pow2 |= 1 << a;
    }
    for (int d = 0; d < 6; ++d) {
        const double ang = (double)((float)d * CUDART_PI_F / 3.0f);
        for (int q = 0; q < 9; ++q) {
            // head_to_image<false> of (dr cos, dr sin, 0)
            const double x = -(q + 1) * std::cos(ang), z = (q + 1) * std::sin(ang);
            const double xg = x * f.cga, yg = x * f.sga;
            const double delta[3] = {xg * f.cta + z * f.sta, yg, -xg * f.sta + z * f.cta};
            int off[3], exact = 0;
            for (int a = 0; a < 3; ++a) {
                const double v = delta[a] / sp[a], lo = std::floor(v);
                // written so that a NaN anywhere asks for the exact form
                if (!(std::fabs(v - (lo + 0.5)) * sp[a] > eps) || !(std::fabs(v) < 30000.0)) exact |= 1 << a;
                off[a] = std::fabs(v) < 30000.0 ? (int)std::floor(v + 0.5) : 0;
                const int reach = std::fabs(v) < 30000.0 ? std::abs(off[a]) + (exact >> a & 1) : 1 << 28;
                T.reach[a] = std::max(T.reach[a], reach);
            }
            const int e = d * 9 + q;
            T.dx[e] = (short)off[0];
            T.dy[e] = (short)off[1];
            T.dz[e] = (short)off[2];
            T.exact[e] = (short)exact;
            T.n_exact += exact != 0;
        }
    }
    for (int e = 0; e < kSmoothSamples; ++e)
        T.lin[e] = T.dx[e] + (long long)g.nx * (T.dy[e] + (long long)g.ny * T.dz[e]);
    return T;
}

void enqueue_wet_smooth(const Grid &g, const Frame &f, const float *wet, float *wet_s, cudaStream_t s) {
    const dim3 block(32, 4, 4);
    const dim3 grid((unsigned)((g.nx + 31) / 32), (unsigned)((g.ny + 3) / 4), (unsigned)((g.nz + 3) / 4));
    wet_smooth_kernel<<<grid, block, 0, s>>>(g, f, make_wet_smooth_table(g, f), wet, wet_s);
    check_launch("wet_smooth_kernel");
}

DC_BOUNDS_TAKE(take_bounds_wet)

static Bricks brick_shape(const Grid &g) {
    Bricks B;
    B.nx = (g.nx + kBrick - 1) / kBrick;
    B.ny = (g.ny + kBrick - 1) / kBrick;
    B.nz = (g.nz + kBrick - 1) / kBrick;
    return B;
}

size_t march_bytes(const Grid &g) {
    const Bricks B = brick_shape(g);
    return (size_t)g.n() * sizeof(float) + (size_t)B.nx * B.ny * B.nz * (sizeof(float) + 1) + sizeof(unsigned);
}

// Samples of a plain march: a voxel's mean path is half the volume's mean extent.
static double march_samples(const Grid &g) {
    return (double)g.n() * (g.nx * (double)g.sx + g.ny * (double)g.sy + g.nz * (double)g.sz) / 6.0;
}

static Bricks launch_bricks(DeviceContext &ctx, const Grid &g, cudaTextureObject_t density, float *wet, cudaStream_t s) {
    Bricks B = brick_shape(g);
    const long long n = (long long)B.nx * B.ny * B.nz;
    B.value = wet + g.n();
    B.uniform = reinterpret_cast<unsigned *>(B.value + n);
    B.radius = reinterpret_cast<unsigned char *>(B.uniform + 1);
    // the rest of the map and the looks at it pay off from some 6 % of uniform bricks on, in short marches 20 %
    B.least = (unsigned)((double)n * (0.06 + 0.15 * 4.0e7 / march_samples(g)));
    KernelTimer kt(ctx, "march_bricks", s);
    int sms = 0;
    DC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
    DC_CUDA(cudaMemsetAsync(B.uniform, 0, sizeof(unsigned), s));
    brick_value_kernel<<<(unsigned)std::min((n + 3) / 4, 32LL * sms), 128, 0, s>>>(g, B, density);
    check_launch("brick_value_kernel");
    const dim3 tiles((unsigned)((B.nx + kTile - 1) / kTile), (unsigned)((B.ny + kTile - 1) / kTile),
                     (unsigned)((B.nz + kTile - 1) / kTile));
    brick_radius_kernel<<<tiles, 512, 0, s>>>(B);
    check_launch("brick_radius_kernel");
    return B;
}

// Whether the march may leap.  The map takes 11 to 20 us, so a march shorter than
// some 90 us (4e7 samples) would win little: 80^3 at 2 mm takes 91 us with eight
// lanes per ray; leaping 16 + 21 where all is uniform, 15 + 65 for a body in
// uniform air and 11 + 102 where nothing is.
void launch_wet_march(DeviceContext &ctx, const Grid &g, const Frame &f, cudaTextureObject_t density,
                      float *wet, cudaStream_t s) {
    if (march_samples(g) > 4.0e7) {
        const Bricks B = launch_bricks(ctx, g, density, wet, s);
        KernelTimer kt(ctx, "wet_march", s);
        const dim3 grid((unsigned)((g.nx + kMarchX - 1) / kMarchX), (unsigned)((g.ny + kMarchY - 1) / kMarchY),
                        (unsigned)((g.nz + kMarchZ - 1) / kMarchZ));
        wet_march_leap_kernel<<<grid, dim3(kMarchX, kMarchY, kMarchZ), 0, s>>>(g, f, B, density, wet);
        check_launch("wet_march_leap_kernel");
        return;
    }
    KernelTimer kt(ctx, "wet_march", s);
    const dim3 grid((unsigned)((g.nx + 128 / kRayLanes - 1) / (128 / kRayLanes)), (unsigned)g.ny, (unsigned)g.nz);
    wet_march_kernel<<<grid, 128, 0, s>>>(g, f, density, wet);
    check_launch("wet_march_kernel");
}

void launch_wet_smooth(DeviceContext &ctx, const Grid &g, const Frame &f, const float *wet, float *wet_s,
                       cudaStream_t s) {
    KernelTimer kt(ctx, "wet_smooth", s);
    enqueue_wet_smooth(g, f, wet, wet_s, s);
}

}  // namespace dc

extern "C" int dc_wet_smooth_offsets(int nz, int ny, int nx, const float spacing[3], const float origin[3],
                                     const float iso[3], double gantry_deg, float couch_deg, float src_dist,
                                     int *offsets) {
    using namespace dc;
    return guarded([&] {
        if (!spacing || !origin || !iso || !offsets) throw Error(DC_ERR_VALUE, "NULL argument.");
        const WetSmoothTable T = make_wet_smooth_table(make_grid(nz, ny, nx, spacing),
                                                       make_frame(iso, origin, gantry_deg, couch_deg, 0.0, src_dist));
        for (int e = 0; e < kSmoothSamples; ++e) {
            offsets[4 * e] = T.dx[e];
            offsets[4 * e + 1] = T.dy[e];
            offsets[4 * e + 2] = T.dz[e];
            offsets[4 * e + 3] = T.exact[e];
        }
    });
}
