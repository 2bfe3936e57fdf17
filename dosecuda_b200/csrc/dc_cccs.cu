// dc_cccs.cu — photon collapsed-cone superposition, per voxel.
//
// cccs_kernel restates cccKernel (IMRTClasses.cu:252-350) with kernelTilt
// (:173-203): per voxel with TERMA > 0.01, for 6 zenith cones x 12 azimuths,
// a backward recursive march from ray_length (cm) down to 0 in steps of one
// voxel spacing, sampling TERMA and density (trilinear, weights in 1/256 as
// the texture unit rounds them), with the cone direction tilted so that its
// axis points at the source.
//
// What bounds it: trilinear samples.  The texture unit delivers 1.77 of them
// per clock and SM (measured, float2 texels; 1.00 for float4 layered ones,
// 1.99 for float2 layered ones, two of which make a sample); interpolating in
// software from shared memory reaches the same rate through another pipe, and
// the two run side by side (from global memory they would share the texture
// unit's L1 path).
//  * A block owns a tile of voxels.  The samples nearest to the voxel, the
//    last K of every cone, reach at most K voxels far: their texels, the tile
//    with K voxels around it, are staged in shared memory and interpolated
//    there; the farther samples go to the texture unit.  K is the count that
//    brings about a quarter of all samples to shared memory (kShare).
//  * A sample's coordinates are one fused multiply-add per axis: in voxels
//    for the texture unit; in 1/256 voxel, rounded by adding 1.5 * 2^23, for
//    shared memory, where the low byte is the fraction and the next the cell.
//    The weights are the texture unit's own (box_sample): with plain products
//    of the fractions the dose would differ by 5e-5.
//  * The tile's voxels above the TERMA mask (a bit per voxel, from the TERMA
//    kernel) are compacted over the block's threads.
//  * The recursions run without the cone's constant factors, applied once at
//    the end: 7 operations per sample.
//  * Small grids take smaller tiles whose directions are shared by 4 groups
//    of threads, added in a fixed order.
//
// Measured (ms; before = all samples from the texture unit, one thread per
// listed voxel): 128^3 at 2.5 mm, 10 x 10 cm field 0.893 -> 0.704; 143 x 131
// x 97 at 3 mm, shaped field 1.66 -> 1.14; 36 x 32 x 30 at 4 mm 0.060 ->
// 0.038.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "../../include/dosecuda.h"
#include "dc_common.cuh"
#include "dc_kernels.cuh"
#include "dc_photon.cuh"
#include "dc_runtime.cuh"

namespace dc {

DC_BOUNDS_WORD

namespace {

constexpr int kThreads = 256;
// Large tiles per SM from which on they are taken; below (a grid of 32^3 has
// one per two SMs) the small ones keep more SMs busy: 36 x 32 x 30 at 4 mm
// takes 0.038 ms with small tiles, 0.060 with large ones.
constexpr long long kLargeTiles = 8;
// Share of the samples interpolated from shared memory: measured at 0, 0.25,
// 0.38 and 0.5 of the samples of 128^3 at 2.5 mm: 0.85, 0.70, 0.79, 0.90 ms.
// The texture unit alone would allow 0.5; the instructions of the software
// interpolation (about 60 per sample against 13) set the line.
constexpr double kShare = 0.26;
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the low bits

// Which samples of each cone come from where: the first n_far from the
// texture unit, the next n_near from shared memory, and the one at distance 0
// (n_zero), which is the voxel's own texel.  The staged box: the tile with h
// voxels below and h + 1 above; a record holds a texel's and its upper z
// neighbour's values (T, T up, density, density up): four 16-byte loads per
// sample, and the lanes of a row read consecutive records.
struct CccsPlan {
    int n_far[kMaxCones], n_near[kMaxCones], n_zero[kMaxCones];
    int hx, hy, hz, wx, wy, wz;
};

template <int TX, int TY, int TZ, int G>
struct CccsTile {
    static constexpr int x = TX, y = TY, z = TZ, groups = G, voxels = TX * TY * TZ;
    static_assert(voxels * G == kThreads && TX == 8, "a thread per voxel and group; rows of 8 match the mask's bytes");
};
using TileLarge = CccsTile<8, 8, 4, 1>;
using TileSmall = CccsTile<8, 4, 2, 4>;

// 256 x the trilinear (TERMA, density) at box coordinates tx, ty, tz (magic
// floats in 1/256 voxel), with the texture unit's weights: the eight weights
// are multiples of 1/256 that sum to 1, split off 1 by z, then x, then y, each
// split rounded to 1/256, ties to the upper side except in the y split of the
// lower x side (found by sampling volumes with a single non-zero texel at
// 20000 fractions; every one of the 160000 weights agrees).  A register holds
// the two z sides of a weight in 16-bit fields, so that one multiply-add
// splits both and one byte permute shifts both; as floats they ride in the
// paired lanes, like the texels in the box's records.  The index is kept
// inside the box whatever the coordinates.
__device__ __forceinline__ float2 box_sample(const float4 *__restrict__ box, int row, int plane, int cap, float tx,
                                             float ty, float tz) {
    const unsigned bx = __float_as_uint(tx), by = __float_as_uint(ty), bz = __float_as_uint(tz);
    const int cx = __byte_perm(bx, 0, 0x4441), cy = __byte_perm(by, 0, 0x4441), cz = __byte_perm(bz, 0, 0x4441);
    const unsigned fx = __byte_perm(bx, 0, 0x4440), fy = __byte_perm(by, 0, 0x4440), fz = __byte_perm(bz, 0, 0x4440);
    const float4 *p = box + min(cx + cy * row + cz * plane, cap);
    const float4 a = p[0], b = p[1], c = p[row], d = p[row + 1];
    const unsigned z = fz * 65535u + 256u;  // (256 - fz, fz)
    const unsigned x1 = __byte_perm(z * fx + 0x00800080u, 0, 0x4341), x0 = z - x1;
    const unsigned w11 = __byte_perm(x1 * fy + 0x00800080u, 0, 0x4341), w10 = x1 - w11;
    const unsigned w01 = __byte_perm(x0 * fy + 0x007F007Fu, 0, 0x4341), w00 = x0 - w01;
    auto pair = [](unsigned w) {  // both fields as floats: the mantissa of 2^23 + w
        return __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7410)),
                                      __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7432))),
                          make_float2(-8388608.0f, -8388608.0f));
    };
    const float2 u00 = pair(w00), u10 = pair(w10), u01 = pair(w01), u11 = pair(w11);
    const float2 t = __ffma2_rn(u11, make_float2(d.x, d.y), __ffma2_rn(u01, make_float2(c.x, c.y),
                     __ffma2_rn(u10, make_float2(b.x, b.y), __fmul2_rn(u00, make_float2(a.x, a.y)))));
    const float2 r = __ffma2_rn(u11, make_float2(d.z, d.w), __ffma2_rn(u01, make_float2(c.z, c.w),
                     __ffma2_rn(u10, make_float2(b.z, b.w), __fmul2_rn(u00, make_float2(a.z, a.w)))));
    return make_float2(t.x + t.y, r.x + r.y);
}

// One step of the recursions R = R e + T (1 - e), S = S (1 - b rho) + T rho
// (the reference's Rp and Rs over their constant factors), e = exp(-a rho).
__device__ __forceinline__ void cccs_step(float2 td, float nal, float nb, float &R, float &S) {
    const float rho = fmaxf(td.y, kAirDensity);
    const float e = fast_exp2(nal * rho);
    R = fmaf(e, R - td.x, td.x);
    S = fmaf(rho, fmaf(nb, S, td.x), S);
}

}  // namespace

template <class Tile>
__global__ void __launch_bounds__(kThreads, 4)
    cccs_kernel(Grid g, Frame f, const __grid_constant__ CccsCones C, const __grid_constant__ CccsPlan B, float sp_cm,
                float dose_scale, const float4 *__restrict__ dirs, cudaTextureObject_t td_tex,
                const float *__restrict__ electron, const unsigned *__restrict__ mask, float *__restrict__ dose) {
    extern __shared__ float4 s_box[];  // [wz - 1][wy][wx]
    __shared__ float4 s_dir[kMaxCones * 12];
    __shared__ float s_rl10[kMaxConeSteps];
    __shared__ float s_part[Tile::groups > 1 ? kThreads : 1];
    __shared__ unsigned short s_voxel[Tile::voxels];
    __shared__ int s_count[Tile::voxels / 32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int i0 = blockIdx.x * Tile::x, j0 = blockIdx.y * Tile::y, k0 = blockIdx.z * Tile::z;

    // the tile's active voxels, in order, over the first threads
    bool act = false;
    unsigned bal = 0;
    if (tid < Tile::voxels) {
        const int i = i0 + tid % Tile::x, j = j0 + tid / Tile::x % Tile::y, k = k0 + tid / (Tile::x * Tile::y);
        if (i < g.nx && j < g.ny && k < g.nz) {
            const long long word = ((long long)k * g.ny + j) * mask_words(g.nx) + (i >> 5);
            act = DC_IN_BOUNDS(word, (long long)g.nz * g.ny * mask_words(g.nx), 14) && (__ldg(mask + word) >> (i & 31) & 1u);
        }
        bal = __ballot_sync(0xffffffffu, act);
        if (lane == 0) s_count[w] = __popc(bal);
    }
    __syncthreads();
    int n = 0, base = 0;
#pragma unroll
    for (int q = 0; q < Tile::voxels / 32; ++q) {
        base += q < w ? s_count[q] : 0;
        n += s_count[q];
    }
    if (n == 0) return;
    if (act) s_voxel[base + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)tid;
    for (int q = tid; q < C.n_cones * 12; q += kThreads) s_dir[q] = dirs[q];
    for (int q = tid; q < C.total_steps; q += kThreads) s_rl10[q] = C.rl10[q];
    // the staged texels: fetched at their centres, where linear filtering
    // returns the stored value (outside the volume, the border's)
    const int plane = B.wx * B.wy;
    for (int q = tid; q < plane * B.wz; q += kThreads) {
        const int row = q / B.wx, x = q - row * B.wx, z = row / B.wy, y = row - z * B.wy;
        const float2 t = tex3D<float2>(td_tex, (float)(i0 - B.hx + x) + 0.5f, (float)(j0 - B.hy + y) + 0.5f,
                                       (float)(k0 - B.hz + z) + 0.5f);
        float *r = reinterpret_cast<float *>(s_box + q);
        if (z < B.wz - 1) r[0] = t.x, r[2] = t.y;
        if (z > 0) r[1 - 4 * plane] = t.x, r[3 - 4 * plane] = t.y;
    }
    __syncthreads();

    const int slot = tid % Tile::voxels, group = tid / Tile::voxels;
    float sum = 0.0f;
    long long v = 0;
    if (slot < n) {
        const int u = s_voxel[slot];
        const int li = u % Tile::x, lj = u / Tile::x % Tile::y, lk = u / (Tile::x * Tile::y);
        const int i = i0 + li, j = j0 + lj, k = k0 + lk;
        v = (long long)i + (long long)g.nx * (j + (long long)g.ny * k);
        const float3 p = voxel_xyz(g, f, i, j, k);
        // kernelTilt (IMRTClasses.cu:173-203): rotate each direction by the
        // rotation taking the central axis (iso -> source) onto voxel -> source.
        const float3 uvec = unit_to_source(f, p);
        const float3 axis0 = unit_to_source(f, make_float3(0.f, 0.f, 0.f));
        const float costh = axis0.x * uvec.x + axis0.y * uvec.y + axis0.z * uvec.z;
        const float3 ax = make_float3(axis0.y * uvec.z - axis0.z * uvec.y, axis0.z * uvec.x - axis0.x * uvec.z,
                                      axis0.x * uvec.y - axis0.y * uvec.x);
        const float inv1c = 1.0f / (1.0f + costh);
        const float3 tc = tex_coord(g, f, p);
        const float bx = (float)((li + B.hx) * 256) + kMagic, by = (float)((lj + B.hy) * 256) + kMagic,
                    bz = (float)((lk + B.hz) * 256) + kMagic;
        const int cap = (B.wz - 2) * plane + (B.wy - 2) * B.wx + B.wx - 2;
        const float4 own = s_box[(lk + B.hz) * plane + (lj + B.hy) * B.wx + li + B.hx];
        const float2 td0 = make_float2(own.x, own.z);

        for (int c = 0; c < C.n_cones; ++c) {
            const float nal = -C.am[c] * kLog2e * sp_cm, nb = -C.bm[c] * sp_cm;
            const int n_far = B.n_far[c], n_near = B.n_near[c];
            const float *rl = s_rl10 + C.step_off[c];
            float cone = 0.0f;
            for (int az = group; az < 12; az += Tile::groups) {
                const float4 dv = s_dir[c * 12 + az];
                // Rodrigues: r = ax x v + v cos + ax (ax.v)/(1+cos)
                float3 r;
                r.x = ax.y * dv.z - ax.z * dv.y;
                r.y = ax.z * dv.x - ax.x * dv.z;
                r.z = ax.x * dv.y - ax.y * dv.x;
                r.x += dv.x * costh;
                r.y += dv.y * costh;
                r.z += dv.z * costh;
                const float sc = (ax.x * dv.x + ax.y * dv.y + ax.z * dv.z) * inv1c;
                r.x = (r.x + ax.x * sc) * g.inv_sx;
                r.y = (r.y + ax.y * sc) * g.inv_sy;
                r.z = (r.z + ax.z * sc) * g.inv_sz;

                float R = 0.0f, S = 0.0f;
                // a batch's fetches are all in flight before the first is used; the remainder is
                // a batch of its own (one by one it would wait for every fetch)
                auto far = [&](auto count, int s) {
                    constexpr int N = decltype(count)::value;
                    float2 td[N];
#pragma unroll
                    for (int q = 0; q < N; ++q) {
                        const float L = rl[s + q];
                        td[q] = tex3D<float2>(td_tex, fmaf(r.x, L, tc.x), fmaf(r.y, L, tc.y), fmaf(r.z, L, tc.z));
                    }
#pragma unroll
                    for (int q = 0; q < N; ++q) cccs_step(td[q], nal, nb, R, S);
                };
                int s = 0;
                for (; s + 6 <= n_far; s += 6) far(std::integral_constant<int, 6>{}, s);
                switch (n_far - s) {
                    case 1: far(std::integral_constant<int, 1>{}, s); break;
                    case 2: far(std::integral_constant<int, 2>{}, s); break;
                    case 3: far(std::integral_constant<int, 3>{}, s); break;
                    case 4: far(std::integral_constant<int, 4>{}, s); break;
                    case 5: far(std::integral_constant<int, 5>{}, s); break;
                }
                r.x *= 256.0f;
                r.y *= 256.0f;
                r.z *= 256.0f;
                auto near_step = [&](int s) {
                    const float L = rl[n_far + s];
                    float2 td = box_sample(s_box, B.wx, plane, cap, fmaf(r.x, L, bx), fmaf(r.y, L, by), fmaf(r.z, L, bz));
                    td.x *= 1.0f / 256.0f;
                    td.y *= 1.0f / 256.0f;
                    cccs_step(td, nal, nb, R, S);
                };
                if (n_near == 2) {  // the count at most spacings, see kShare
                    near_step(0);
                    near_step(1);
                } else if (n_near == 3) {
                    near_step(0);
                    near_step(1);
                    near_step(2);
                } else {
                    for (int s = 0; s < n_near; ++s) near_step(s);
                }
                for (int s = 0; s < B.n_zero[c]; ++s) cccs_step(td0, nal, nb, R, S);
                // am Rp + bm Rs with Rp = sin Am / am^2 R, Rs = sin Bm / bm sp S
                cone = fmaf(dv.w, fmaf(C.Am[c] / C.am[c], R, C.Bm[c] * sp_cm * S), cone);
            }
            sum += cone;
        }
    }
    if (Tile::groups > 1) {  // add the groups in order
        s_part[tid] = sum;
        __syncthreads();
        if (group != 0) return;
#pragma unroll
        for (int q = 1; q < Tile::groups; ++q) sum += s_part[q * Tile::voxels + slot];
    }
    if (slot < n && DC_IN_BOUNDS(v, g.n(), 13)) {
        const float d = sum + __ldg(electron + v);
        dose[v] = (!isnan(d) && d >= 0.0f) ? dose_scale * d : 0.0f;
    }
}

// Mask bits of the listed voxels that the TERMA mask keeps (the probe).
__global__ void __launch_bounds__(128) points_mask_kernel(Grid g, const int *__restrict__ voxels, int n,
                                                          const unsigned *__restrict__ mask,
                                                          unsigned *__restrict__ points) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int v = __ldg(voxels + t);
    if (v < 0 || (long long)v >= g.n()) return;
    const int row = v / g.nx, i = v - row * g.nx;
    const long long word = (long long)row * mask_words(g.nx) + (i >> 5);
    if (__ldg(mask + word) >> (i & 31) & 1u) atomicOr(points + word, 1u << (i & 31));
}

// Doses of the listed voxels (0: masked, or not a voxel of the grid).
__global__ void __launch_bounds__(128) points_gather_kernel(Grid g, const int *__restrict__ voxels, int n,
                                                            const unsigned *__restrict__ points,
                                                            const float *__restrict__ dose, float *__restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int v = __ldg(voxels + t);
    float d = 0.0f;
    if (v >= 0 && (long long)v < g.n()) {
        const int row = v / g.nx, i = v - row * g.nx;
        const long long word = (long long)row * mask_words(g.nx) + (i >> 5);
        if (__ldg(points + word) >> (i & 31) & 1u) d = __ldg(dose + v);
    }
    out[t] = d;
}

DC_BOUNDS_TAKE(take_bounds_cccs)

namespace {

// Fills B for a tile and returns the staged box's bytes.  Where no near sample
// fits (spacings far below the cones' ray lengths never do that; very uneven
// ones may) only the tile's own texels are staged and all others are fetched.
template <class Tile>
size_t cccs_plan(const CccsCones &C, const Grid &g, CccsPlan &B) {
    constexpr size_t kMostBytes = 104 * 1024;  // two blocks per SM
    int total = 0, longest = 0;
    for (int c = 0; c < C.n_cones; ++c) {
        B.n_zero[c] = C.n_steps[c] > 0 && C.rl10[C.step_off[c] + C.n_steps[c] - 1] == 0.0f;
        total += C.n_steps[c] - B.n_zero[c];
        longest = std::max(longest, C.n_steps[c] - B.n_zero[c]);
    }
    auto fill = [&](int K) -> size_t {
        float reach = 0.0f;
        for (int c = 0; c < C.n_cones; ++c) {
            const int n = C.n_steps[c] - B.n_zero[c];
            B.n_near[c] = std::min(K, n);
            B.n_far[c] = n - B.n_near[c];
            if (B.n_near[c] > 0) reach = std::max(reach, C.rl10[C.step_off[c] + B.n_far[c]]);
        }
        auto halo = [&](float sp) { return (int)std::min(200.0, std::ceil((double)reach / sp * 1.0001)); };
        B.hx = halo(g.sx), B.hy = halo(g.sy), B.hz = halo(g.sz);
        B.wx = Tile::x + 2 * B.hx + 1, B.wy = Tile::y + 2 * B.hy + 1, B.wz = Tile::z + 2 * B.hz + 1;
        return (size_t)B.wx * B.wy * (B.wz - 1) * sizeof(float4);
    };
    int best = 0;
    double off = kShare;  // K = 0: none
    for (int K = 1; K <= longest; ++K) {
        if (fill(K) > kMostBytes || B.wx > 255 || B.wy > 255 || B.wz > 255) break;
        int near = 0;
        for (int c = 0; c < C.n_cones; ++c) near += B.n_near[c];
        const double d = std::fabs((double)near / std::max(total, 1) - kShare);
        if (d < off) off = d, best = K;
    }
    return fill(best);
}

template <class Tile>
void cccs_launch(const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w, float dose_scale,
                 const unsigned *mask, float *dose, cudaStream_t s) {
    CccsPlan B;
    const size_t smem = cccs_plan<Tile>(C, g, B);
    if (smem > 48 * 1024)
        DC_CUDA(cudaFuncSetAttribute(cccs_kernel<Tile>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const dim3 grid((unsigned)((g.nx + Tile::x - 1) / Tile::x), (unsigned)((g.ny + Tile::y - 1) / Tile::y),
                    (unsigned)((g.nz + Tile::z - 1) / Tile::z));
    cccs_kernel<Tile><<<grid, kThreads, smem, s>>>(g, f, C, B, g.sx / 10.0f, dose_scale, w.dirs, w.td_tex, w.electron,
                                                   mask, dose);
    check_launch("cccs_kernel");
}

void cccs(DeviceContext &ctx, const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w, float dose_scale,
          const unsigned *mask, float *dose, cudaStream_t s) {
    int sms = 0;
    DC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
    const long long tiles = (long long)((g.nx + TileLarge::x - 1) / TileLarge::x) * ((g.ny + TileLarge::y - 1) / TileLarge::y) *
                            ((g.nz + TileLarge::z - 1) / TileLarge::z);
    if (tiles >= kLargeTiles * sms)
        cccs_launch<TileLarge>(g, f, C, w, dose_scale, mask, dose, s);
    else
        cccs_launch<TileSmall>(g, f, C, w, dose_scale, mask, dose, s);
}

}  // namespace

void enqueue_cccs(DeviceContext &ctx, const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w,
                  float dose_scale, float *dose_dev, cudaStream_t s) {
    KernelTimer kt(ctx, "cccs", s);
    cccs(ctx, g, f, C, w, dose_scale, w.mask, dose_dev, s);
}

size_t cccs_points_bytes(const Grid &g) {
    return ((mask_bytes(g) + 255) & ~(size_t)255) + (size_t)g.n() * sizeof(float);
}

// The listed voxels go through the same kernel as the full volume, behind
// their own mask, so their doses are the full calculation's bit for bit.
void enqueue_cccs_points(DeviceContext &ctx, const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w,
                         float dose_scale, const int *voxels, int n, float *out, void *scratch, cudaStream_t s) {
    if (n <= 0) return;
    const size_t mb = mask_bytes(g);
    unsigned *points = static_cast<unsigned *>(scratch);
    float *dose = reinterpret_cast<float *>(static_cast<char *>(scratch) + ((mb + 255) & ~(size_t)255));
    KernelTimer kt(ctx, "cccs_points", s);
    DC_CUDA(cudaMemsetAsync(points, 0, mb, s));
    const unsigned blocks = (unsigned)((n + 127) / 128);
    points_mask_kernel<<<blocks, 128, 0, s>>>(g, voxels, n, w.mask, points);
    check_launch("points_mask_kernel");
    cccs(ctx, g, f, C, w, dose_scale, points, dose, s);
    points_gather_kernel<<<blocks, 128, 0, s>>>(g, voxels, n, points, dose, out);
    check_launch("points_gather_kernel");
}

}  // namespace dc
