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
//    The weights are the texture unit's own (CornerWeights): with plain products
//    of the fractions the dose would differ by 5e-5.
//  * The tile's voxels above the TERMA mask (a bit per voxel, from the TERMA
//    kernel) are compacted over the block's threads.
//  * The recursions run without the cone's constant factors, applied once at
//    the end: 7 operations per sample.
//  * Tiles are small, 8 x 4 x 2 voxels, and the directions are shared by 4
//    groups of threads, added in a fixed order: a masked tile has few voxels,
//    and a narrow field few tiles.  Tiles of 8 x 8 x 4 without groups take 2 %
//    less on 128^3 with a 10 x 10 cm field and 10 % less on a field that fills
//    143 x 131 x 97 at 3 mm (5.9 staged texels per voxel instead of 12.8), but twice the
//    time under narrow fields; 8 x 4 x 4 with two groups lie between (3 and 5 %
//    less, 1.4 times).  Which is better depends on the number of active voxels,
//    which is on the device; launching both, one to return at once, costs 20 us.
//
// Measured (ms; before = all samples from the texture unit, one thread per
// listed voxel): 128^3 at 2.5 mm, 10 x 10 cm field 0.889 -> 0.720, 2 x 2 cm field
// 0.076 -> 0.061; 143 x 131 x 97 at 3 mm, shaped field 1.66 -> 1.27; 36 x 32 x 30
// at 4 mm 0.060 -> 0.039; 91 x 82 x 35 at 2.5 mm, 4 x 2 cm 0.080 -> 0.056; 10 x 10 cm
// on 87^3 at 1.5 mm 1.45 -> 1.13, on 96^3 at 1 mm 2.65 -> 2.30 (there a tile stages 3705
// texels; one voxel more of margin, 5355, made it 2.65, and a 2 cm field 0.28
// instead of 0.24).
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
// Share of the samples interpolated from shared memory: measured at 0, 0.25,
// 0.38 and 0.5 of the samples of 128^3 at 2.5 mm: 0.85, 0.70, 0.79, 0.90 ms
// (tiles of 8 x 8 x 4 voxels).
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

struct Tile {
    static constexpr int x = 8, y = 4, z = 2, groups = 4, voxels = x * y * z;
};
static_assert(Tile::voxels * Tile::groups == kThreads, "a thread per voxel and group");

// The texture unit's weights of a sample at box coordinates tx, ty, tz (magic
// floats in 1/256 voxel): multiples of 1/256 that sum to 1, split off 1 by z,
// then x, then y, each split rounded to 1/256, ties to the upper side except in
// the y split of the lower x side (found by sampling volumes with a single
// non-zero texel at 20000 fractions; every one of the 160000 weights agrees).
// Times 256, both z sides of a weight in one pair.  A register holds the two in
// 16-bit fields, so that one multiply-add splits both and one byte permute
// shifts both; as floats they ride in the paired lanes.
struct CornerWeights {
    float2 u00, u10, u01, u11;  // of (x, y) corner (0, 0), (1, 0), (0, 1), (1, 1): lower z, upper z
    __device__ __forceinline__ CornerWeights(float tx, float ty, float tz) {
        const unsigned fx = __byte_perm(__float_as_uint(tx), 0, 0x4440), fy = __byte_perm(__float_as_uint(ty), 0, 0x4440);
        const unsigned fz = __byte_perm(__float_as_uint(tz), 0, 0x4440);
        const unsigned z = fz * 65535u + 256u;  // (256 - fz, fz)
        const unsigned x1 = __byte_perm(z * fx + 0x00800080u, 0, 0x4341), x0 = z - x1;
        const unsigned w11 = __byte_perm(x1 * fy + 0x00800080u, 0, 0x4341), w10 = x1 - w11;
        const unsigned w01 = __byte_perm(x0 * fy + 0x007F007Fu, 0, 0x4341), w00 = x0 - w01;
        auto pair = [](unsigned w) {  // both fields as floats: the mantissa of 2^23 + w
            return __fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7410)),
                                          __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7432))),
                              make_float2(-8388608.0f, -8388608.0f));
        };
        u00 = pair(w00), u10 = pair(w10), u01 = pair(w01), u11 = pair(w11);
    }
};
__device__ __forceinline__ int box_cell(float t) { return __byte_perm(__float_as_uint(t), 0, 0x4441); }

// 256 x the trilinear (TERMA, density) in a box of records.  The index is kept
// inside the box whatever the coordinates.
struct RecordBox {
    const float4 *box;
    int row, plane, cap;
    __device__ __forceinline__ float2 operator()(float tx, float ty, float tz) const {
        const float4 *p = box + min(box_cell(tx) + box_cell(ty) * row + box_cell(tz) * plane, cap);
        const float4 a = p[0], b = p[1], c = p[row], d = p[row + 1];
        const CornerWeights w(tx, ty, tz);
        const float2 t = __ffma2_rn(w.u11, make_float2(d.x, d.y), __ffma2_rn(w.u01, make_float2(c.x, c.y),
                         __ffma2_rn(w.u10, make_float2(b.x, b.y), __fmul2_rn(w.u00, make_float2(a.x, a.y)))));
        const float2 r = __ffma2_rn(w.u11, make_float2(d.z, d.w), __ffma2_rn(w.u01, make_float2(c.z, c.w),
                         __ffma2_rn(w.u10, make_float2(b.z, b.w), __fmul2_rn(w.u00, make_float2(a.z, a.w)))));
        return make_float2(t.x + t.y, r.x + r.y);
    }
};
// The same products and sums in a box of single texels, half the size.
struct TexelBox {
    const float2 *box;
    int row, plane, cap;
    __device__ __forceinline__ float2 operator()(float tx, float ty, float tz) const {
        const float2 *p = box + min(box_cell(tx) + box_cell(ty) * row + box_cell(tz) * plane, cap);
        const CornerWeights w(tx, ty, tz);
        auto side = [&](const float2 *q, float w00, float w10, float w01, float w11) {
            return __ffma2_rn(make_float2(w11, w11), q[row + 1], __ffma2_rn(make_float2(w01, w01), q[row],
                   __ffma2_rn(make_float2(w10, w10), q[1], __fmul2_rn(make_float2(w00, w00), q[0]))));
        };
        const float2 l = side(p, w.u00.x, w.u10.x, w.u01.x, w.u11.x), h = side(p + plane, w.u00.y, w.u10.y, w.u01.y, w.u11.y);
        return make_float2(l.x + h.x, l.y + h.y);
    }
};

// One step of the recursions R = R e + T (1 - e), S = S (1 - b rho) + T rho
// (the reference's Rp and Rs over their constant factors), e = exp(-a rho).
__device__ __forceinline__ void cccs_step(float2 td, float nal, float nb, float &R, float &S) {
    const float rho = fmaxf(td.y, kAirDensity);
    const float e = fast_exp2(nal * rho);
    R = fmaf(e, R - td.x, td.x);
    S = fmaf(rho, fmaf(nb, S, td.x), S);
}

// kernelTilt (IMRTClasses.cu:173-203) of a voxel: the rotation taking the
// central axis (iso -> source) onto voxel -> source.  Products are fused
// explicitly here and in tilt(), so that both kernels round alike.
struct CccsVoxel {
    float3 ax, tc;  // rotation axis times its sine; texture coordinates
    float costh, inv1c;

    CccsVoxel() = default;
    __device__ __forceinline__ CccsVoxel(const Grid &g, const Frame &f, int i, int j, int k) {
        const float3 p = voxel_xyz(g, f, i, j, k);
        const float3 u = unit_to_source(f, p), a = unit_to_source(f, make_float3(0.f, 0.f, 0.f));
        costh = __fmaf_rn(a.z, u.z, __fmaf_rn(a.y, u.y, __fmul_rn(a.x, u.x)));
        ax = make_float3(__fmaf_rn(a.y, u.z, -__fmul_rn(a.z, u.y)), __fmaf_rn(a.z, u.x, -__fmul_rn(a.x, u.z)),
                         __fmaf_rn(a.x, u.y, -__fmul_rn(a.y, u.x)));
        inv1c = 1.0f / (1.0f + costh);
        tc = tex_coord(g, f, p);
    }
    // Rodrigues: r = ax x v + v cos + ax (ax.v)/(1+cos), in voxels per mm
    __device__ __forceinline__ float3 tilt(const Grid &g, float4 v) const {
        const float sc = __fmul_rn(__fmaf_rn(ax.z, v.z, __fmaf_rn(ax.y, v.y, __fmul_rn(ax.x, v.x))), inv1c);
        const float x = __fmaf_rn(v.x, costh, __fmaf_rn(ax.y, v.z, -__fmul_rn(ax.z, v.y)));
        const float y = __fmaf_rn(v.y, costh, __fmaf_rn(ax.z, v.x, -__fmul_rn(ax.x, v.z)));
        const float z = __fmaf_rn(v.z, costh, __fmaf_rn(ax.x, v.y, -__fmul_rn(ax.y, v.x)));
        return make_float3(__fmul_rn(__fmaf_rn(ax.x, sc, x), g.inv_sx), __fmul_rn(__fmaf_rn(ax.y, sc, y), g.inv_sy),
                           __fmul_rn(__fmaf_rn(ax.z, sc, z), g.inv_sz));
    }
};

// am Rp + bm Rs of one direction r of cone c, from the farthest sample to the
// voxel's own; b: the voxel's box coordinates (magic floats in 1/256 voxel).
template <class Box>
__device__ __forceinline__ float cccs_direction(const CccsCones &C, const CccsPlan &B, int c, const float *rl, float3 r,
                                                float3 tc, float3 b, float sp_cm, cudaTextureObject_t td_tex,
                                                const Box &box, float2 td0) {
    const float nal = -C.am[c] * kLog2e * sp_cm, nb = -C.bm[c] * sp_cm;
    const int n_far = B.n_far[c], n_near = B.n_near[c];
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
    auto near_step = [&](int q) {
        const float L = rl[n_far + q];
        float2 td = box(fmaf(r.x, L, b.x), fmaf(r.y, L, b.y), fmaf(r.z, L, b.z));
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
        for (int q = 0; q < n_near; ++q) near_step(q);
    }
    for (int q = 0; q < B.n_zero[c]; ++q) cccs_step(td0, nal, nb, R, S);
    // Rp = sin Am / am^2 R, Rs = sin Bm / bm sp S, the sine by the caller
    return fmaf(C.Am[c] / C.am[c], R, C.Bm[c] * sp_cm * S);
}

__device__ __forceinline__ float cccs_dose(float sum, float electron, float dose_scale) {
    const float d = sum + electron;
    return (!isnan(d) && d >= 0.0f) ? dose_scale * d : 0.0f;
}

// Stages a texel: its record's lower z halves, and the upper ones of the record below.
__device__ __forceinline__ void stage_texel(float4 *box, int q, int z, int wz, int plane, float2 t) {
    float *r = reinterpret_cast<float *>(box + q);
    if (z < wz - 1) r[0] = t.x, r[2] = t.y;
    if (z > 0) r[1 - 4 * plane] = t.x, r[3 - 4 * plane] = t.y;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 4)
    cccs_kernel(Grid g, Frame f, const __grid_constant__ CccsCones C, const __grid_constant__ CccsPlan B, float sp_cm,
                float dose_scale, const float4 *__restrict__ dirs, cudaTextureObject_t td_tex,
                const float *__restrict__ electron, const unsigned *__restrict__ mask, float *__restrict__ dose) {
    extern __shared__ float4 s_box[];  // [wz - 1][wy][wx]
    __shared__ float4 s_dir[kMaxCones * 12];
    __shared__ float s_rl10[kMaxConeSteps];
    __shared__ float s_part[kThreads];
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
        stage_texel(s_box, q, z, B.wz, plane, t);
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
        const CccsVoxel V(g, f, i, j, k);
        const float3 b = make_float3((float)((li + B.hx) * 256) + kMagic, (float)((lj + B.hy) * 256) + kMagic,
                                     (float)((lk + B.hz) * 256) + kMagic);
        const RecordBox box{s_box, B.wx, plane, (B.wz - 2) * plane + (B.wy - 2) * B.wx + B.wx - 2};
        const float4 own = s_box[(lk + B.hz) * plane + (lj + B.hy) * B.wx + li + B.hx];
        for (int c = 0; c < C.n_cones; ++c) {
            float cone = 0.0f;
            for (int az = group; az < 12; az += Tile::groups) {
                const float4 dv = s_dir[c * 12 + az];
                const float x = cccs_direction(C, B, c, s_rl10 + C.step_off[c], V.tilt(g, dv), V.tc, b, sp_cm, td_tex,
                                               box, make_float2(own.x, own.z));
                cone = fmaf(dv.w, x, cone);
            }
            sum += cone;
        }
    }
    // add the groups in order
    s_part[tid] = sum;
    __syncthreads();
    if (group != 0) return;
#pragma unroll
    for (int q = 1; q < Tile::groups; ++q) sum += s_part[q * Tile::voxels + slot];
    if (slot < n && DC_IN_BOUNDS(v, g.n(), 13)) dose[v] = cccs_dose(sum, __ldg(electron + v), dose_scale);
}

// The dose of listed voxels (a probe on a few lines and a lattice through the
// field), bit for bit cccs_kernel's: the same samples from the same sources,
// added in the order of its groups.  Tiles around so few voxels would stage far
// more texels than they use, so each voxel has a box of its own, of which only
// the texels within reach of its near samples are staged (some 150 at 128^3,
// 2.5 mm), and the directions of a block's voxels are dealt to its threads.  A
// block takes 4 voxels: 8 leave 27 warps per SM, 2 or half-masked blocks idle
// threads.  Measured (us; before = one thread per listed voxel, every sample
// from the texture unit), 34 k voxels of 128^3 at 2.5 mm: 2 cm field 69 -> 24, 10 cm
// 75 -> 60, 20 cm 108 -> 110; 5 k of 64^3 at 3 mm 74 -> 21.
constexpr int kListThreads = 288, kListVoxels = 4;
__global__ void __launch_bounds__(kListThreads, 5)
    cccs_list_kernel(Grid g, Frame f, const __grid_constant__ CccsCones C, const __grid_constant__ CccsPlan B,
                     int per_block, float reach, float sp_cm, float dose_scale, const float4 *__restrict__ dirs,
                     cudaTextureObject_t td_tex, const float *__restrict__ electron, const int *__restrict__ voxels,
                     int n, float *__restrict__ out) {
    extern __shared__ float4 s_boxes[];  // [per_block][wz - 1][wy][wx]
    __shared__ float4 s_dir[kMaxCones * 12];
    __shared__ float s_rl10[kMaxConeSteps];
    __shared__ float s_x[kListVoxels][kMaxCones * 12], s_part[kListVoxels][Tile::groups];
    __shared__ int s_voxel[kListVoxels];  // -1: masked, or not a voxel of the grid
    __shared__ CccsVoxel s_geo[kListVoxels];
    __shared__ float3 s_centre[kListVoxels];
    const int tid = threadIdx.x, e0 = blockIdx.x * per_block, n_dirs = C.n_cones * 12;
    int v = -1;
    if (tid < per_block) {
        if (e0 + tid < n) v = __ldg(voxels + e0 + tid);
        if (v < 0 || (long long)v >= g.n()) v = -1;
        if (v >= 0) {
            // masked by the texel itself (read at its centre), which a fluence map may have scaled since the mask
            const int row = v / g.nx, i = v - row * g.nx, k = row / g.ny, j = row - k * g.ny;
            if (tex3D<float2>(td_tex, i + 0.5f, j + 0.5f, k + 0.5f).x <= 0.01f) v = -1;
        }
        s_voxel[tid] = v;
        if (v >= 0) {
            const int vr = v / g.nx, i = v - vr * g.nx, k = vr / g.ny, j = vr - k * g.ny;
            s_geo[tid] = CccsVoxel(g, f, i, j, k);
            s_centre[tid] = make_float3(i + 0.5f, j + 0.5f, k + 0.5f);
        }
    }
    if (!__syncthreads_or(v >= 0)) {
        if (tid < per_block && e0 + tid < n) out[e0 + tid] = 0.0f;
        return;
    }
    for (int q = tid; q < n_dirs; q += kListThreads) s_dir[q] = dirs[q];
    for (int q = tid; q < C.total_steps; q += kListThreads) s_rl10[q] = C.rl10[q];
    const int plane = B.wx * B.wy, texels = plane * B.wz, records = plane * (B.wz - 1);
    for (int t = tid; t < texels; t += kListThreads) {
        const int row = t / B.wx, x = t - row * B.wx, z = row / B.wy, y = row - z * B.wy;
        const int ox = x - B.hx, oy = y - B.hy, oz = z - B.hz;
        // a sample reads texels less than a voxel away on each axis
        const float mx = fmaxf((float)abs(ox) - 1.01f, 0.0f) * g.sx, my = fmaxf((float)abs(oy) - 1.01f, 0.0f) * g.sy;
        const float mz = fmaxf((float)abs(oz) - 1.01f, 0.0f) * g.sz;
        if (mx * mx + my * my + mz * mz > reach * reach) continue;
        for (int e = 0; e < per_block; ++e) {
            if (s_voxel[e] < 0) continue;
            const float3 at = s_centre[e];
            stage_texel(s_boxes + e * records, t, z, B.wz, plane,
                        tex3D<float2>(td_tex, at.x + (float)ox, at.y + (float)oy, at.z + (float)oz));
        }
    }
    __syncthreads();
    const int cap = (B.wz - 2) * plane + (B.wy - 2) * B.wx + B.wx - 2;
    const float3 b = make_float3((float)(B.hx * 256) + kMagic, (float)(B.hy * 256) + kMagic, (float)(B.hz * 256) + kMagic);
    for (int q = tid; q < n_dirs * per_block; q += kListThreads) {
        const int e = q / n_dirs, d = q - e * n_dirs, c = d / 12;
        if (s_voxel[e] < 0) continue;
        const CccsVoxel V = s_geo[e];
        const RecordBox box{s_boxes + e * records, B.wx, plane, cap};
        const float4 own = box.box[B.hz * plane + B.hy * B.wx + B.hx];
        s_x[e][d] = cccs_direction(C, B, c, s_rl10 + C.step_off[c], V.tilt(g, s_dir[d]), V.tc, b, sp_cm, td_tex, box,
                                   make_float2(own.x, own.z));
    }
    __syncthreads();
    const int e = tid / Tile::groups, group = tid % Tile::groups;
    if (e < per_block && s_voxel[min(e, kListVoxels - 1)] >= 0) {
        float sum = 0.0f;
        for (int c = 0; c < C.n_cones; ++c) {
            float cone = 0.0f;
            for (int az = group; az < 12; az += Tile::groups) cone = fmaf(s_dir[c * 12 + az].w, s_x[e][c * 12 + az], cone);
            sum += cone;
        }
        s_part[e][group] = sum;
    }
    __syncthreads();
    if (tid < per_block && e0 + tid < n) {
        float sum = s_part[tid][0];
#pragma unroll
        for (int q = 1; q < Tile::groups; ++q) sum += s_part[tid][q];
        out[e0 + tid] = v < 0 ? 0.0f : cccs_dose(sum, __ldg(electron + v), dose_scale);
    }
}

// The same for long lists, where a box per voxel costs more than its samples.  A
// block compacts its entries above the mask and works through them in runs: a
// run is as many of the next entries as share a staged box that fits and holds
// no more texels than a box for each would (neighbours along a row of a sorted
// list do).  A run's pairs of direction and voxel are dealt to the threads,
// voxels innermost, so that a warp's lanes march alike.  Boxes hold single
// texels: half the shared memory, twice the blocks per SM.
//
// Measured (us; before = one thread per listed voxel, every sample from the
// texture unit; in brackets a box per voxel), 10 x 10 cm fields: every voxel of 128^3
// at 2.5 mm 1118 -> 907 (2540), of 95^3 at 2 mm 1307 -> 1340 (3263), of 96^3 at 1 mm 2621 ->
// 2870 (14970); every other per axis 189 -> 198 (341), 215 -> 256 (430), 430 -> 520 (1980);
// every fourth of 248^3 at 2.5 mm, 241 k, 92 -> 102 (137).  Where a box per voxel no
// longer fits four to a block: 15 k of 96^3 at 1 mm 173 -> 182 (285).
constexpr int kRunThreads = 256, kRunVoxels = 32, kRunEntries = 128;
__global__ void __launch_bounds__(kRunThreads, 4)
    cccs_runs_kernel(Grid g, Frame f, const __grid_constant__ CccsCones C, const __grid_constant__ CccsPlan B,
                     int per_block, int most_texels, float sp_cm, float dose_scale, const float4 *__restrict__ dirs,
                     cudaTextureObject_t td_tex, const float *__restrict__ electron, const int *__restrict__ voxels,
                     int n, float *__restrict__ out) {
    extern __shared__ float2 s_texels[];  // most_texels
    __shared__ float4 s_dir[kMaxCones * 12];
    __shared__ float s_rl10[kMaxConeSteps];
    __shared__ float s_x[kMaxCones * 12 * kRunVoxels];
    __shared__ CccsVoxel s_geo[kRunVoxels];
    __shared__ int s_voxel[kRunEntries], s_entry[kRunEntries], s_count[kRunEntries / 32];
    __shared__ int s_run[7];  // voxels, low corner, widths of the box
    const int tid = threadIdx.x, lane = tid & 31, e0 = blockIdx.x * per_block, n_dirs = C.n_cones * 12;
    auto index3 = [&](int v) {
        const int row = v / g.nx, k = row / g.ny;
        return make_int3(v - row * g.nx, row - k * g.ny, k);
    };
    int v = -1;
    if (tid < kRunEntries) {
        if (tid < per_block && e0 + tid < n) {
            v = __ldg(voxels + e0 + tid);
            if (v < 0 || (long long)v >= g.n()) v = -1;
            if (v >= 0) {
                // masked by the texel itself (read at its centre), which a fluence map may have scaled since the mask
                const int3 q = index3(v);
                if (tex3D<float2>(td_tex, q.x + 0.5f, q.y + 0.5f, q.z + 0.5f).x <= 0.01f) v = -1;
            }
            if (v < 0) out[e0 + tid] = 0.0f;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, v >= 0);
        if (lane == 0) s_count[tid >> 5] = __popc(bal);
    }
    __syncthreads();
    int left = 0, base = 0;
#pragma unroll
    for (int q = 0; q < kRunEntries / 32; ++q) {
        base += q < (tid >> 5) ? s_count[q] : 0;
        left += s_count[q];
    }
    if (left == 0) return;
    if (tid < kRunEntries) {
        const unsigned bal = __ballot_sync(0xffffffffu, v >= 0);
        if (v >= 0) {
            const int at = base + __popc(bal & ((1u << lane) - 1u));
            s_voxel[at] = v;
            s_entry[at] = e0 + tid;
        }
    }
    for (int q = tid; q < n_dirs; q += kRunThreads) s_dir[q] = dirs[q];
    for (int q = tid; q < C.total_steps; q += kRunThreads) s_rl10[q] = C.rl10[q];
    __syncthreads();
    const int single = (2 * B.hx + 2) * (2 * B.hy + 2) * (2 * B.hz + 2);  // texels of one voxel's box
    for (int first = 0; left > 0;) {
        if (tid < 32) {
            const int3 q = index3(s_voxel[first + min(lane, left - 1)]);
            int3 lo = q, hi = q;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int3 l = make_int3(__shfl_up_sync(0xffffffffu, lo.x, o), __shfl_up_sync(0xffffffffu, lo.y, o),
                                         __shfl_up_sync(0xffffffffu, lo.z, o));
                const int3 h = make_int3(__shfl_up_sync(0xffffffffu, hi.x, o), __shfl_up_sync(0xffffffffu, hi.y, o),
                                         __shfl_up_sync(0xffffffffu, hi.z, o));
                if (lane >= o) {
                    lo = make_int3(min(lo.x, l.x), min(lo.y, l.y), min(lo.z, l.z));
                    hi = make_int3(max(hi.x, h.x), max(hi.y, h.y), max(hi.z, h.z));
                }
            }
            const int wx = hi.x - lo.x + 2 * B.hx + 2, wy = hi.y - lo.y + 2 * B.hy + 2, wz = hi.z - lo.z + 2 * B.hz + 2;
            const bool fits = lane < left && max(wx, max(wy, wz)) <= 255 &&
                              (long long)wx * wy * wz <= min(most_texels, single * (lane + 1));
            const int last = 31 - __clz(__ballot_sync(0xffffffffu, fits));  // lane 0's box of its own always fits
            if (lane == last) {
                s_run[0] = last + 1;
                s_run[1] = lo.x, s_run[2] = lo.y, s_run[3] = lo.z;
                s_run[4] = wx, s_run[5] = wy, s_run[6] = wz;
            }
        }
        __syncthreads();
        const int m = s_run[0], wx = s_run[4], wy = s_run[5], wz = s_run[6], plane = wx * wy;
        const int3 lo = make_int3(s_run[1], s_run[2], s_run[3]);
        if (tid < m) {
            const int3 q = index3(s_voxel[first + tid]);
            s_geo[tid] = CccsVoxel(g, f, q.x, q.y, q.z);
        }
        {
            int row = tid / wx, x = tid - row * wx, z = row / wy, y = row - z * wy;
            const int drow = kRunThreads / wx, dx = kRunThreads - drow * wx, dz = drow / wy, dy = drow - dz * wy;
            for (int t = tid; t < plane * wz; t += kRunThreads) {
                s_texels[t] = tex3D<float2>(td_tex, (float)(lo.x - B.hx + x) + 0.5f, (float)(lo.y - B.hy + y) + 0.5f,
                                            (float)(lo.z - B.hz + z) + 0.5f);
                x += dx, y += dy, z += dz;
                if (x >= wx) x -= wx, ++y;
                if (y >= wy) y -= wy, ++z;
            }
        }
        __syncthreads();
        const TexelBox box{s_texels, wx, plane, (wz - 2) * plane + (wy - 2) * wx + wx - 2};
        // voxels innermost, padded to a power of two: a thread keeps its voxel
        const int bits = m > 1 ? 32 - __clz(m - 1) : 0, e = tid & ((1 << bits) - 1);
        if (e < m) {
            const int3 l = index3(s_voxel[first + e]);
            const int3 at = make_int3(l.x - lo.x + B.hx, l.y - lo.y + B.hy, l.z - lo.z + B.hz);
            const float3 b = make_float3((float)(at.x * 256) + kMagic, (float)(at.y * 256) + kMagic, (float)(at.z * 256) + kMagic);
            const float2 own = s_texels[at.z * plane + at.y * wx + at.x];
            const CccsVoxel V = s_geo[e];
            int c = 0;
            for (int d = tid >> bits; d < n_dirs; d += kRunThreads >> bits) {
                while (d >= 12 * (c + 1)) ++c;
                s_x[d * m + e] = cccs_direction(C, B, c, s_rl10 + C.step_off[c], V.tilt(g, s_dir[d]), V.tc, b, sp_cm, td_tex,
                                                box, own);
            }
        }
        __syncthreads();
        if (tid < kRunVoxels * Tile::groups) {  // four neighbouring lanes add a voxel's groups, in their order
            const int e = tid / Tile::groups, group = tid % Tile::groups;
            float sum = 0.0f;
            if (e < m)
                for (int c = 0; c < C.n_cones; ++c) {
                    float cone = 0.0f;
                    for (int az = group; az < 12; az += Tile::groups)
                        cone = fmaf(s_dir[c * 12 + az].w, s_x[(c * 12 + az) * m + e], cone);
                    sum += cone;
                }
            float all = sum;
#pragma unroll
            for (int q = 1; q < Tile::groups; ++q) all += __shfl_sync(0xffffffffu, sum, (lane & ~(Tile::groups - 1)) + q);
            if (group == 0 && e < m) out[s_entry[first + e]] = cccs_dose(all, __ldg(electron + s_voxel[first + e]), dose_scale);
        }
        first += m;
        left -= m;
        // s_run and s_geo are written again: the reads above lie before the barrier that follows the run's pairs
    }
}

DC_BOUNDS_TAKE(take_bounds_cccs)

namespace {

// Most bytes of a staged box: two blocks per SM.
constexpr size_t kMostBytes = 104 * 1024;

// Opts a kernel with `fixed` bytes of static shared memory in to kMostBytes of
// dynamic, where the launch needs it.  Always the same limit: it belongs to the
// function, and calls of several threads share it.
template <class K>
void allow_shared(K *kernel, size_t fixed, size_t smem) {
    if (smem + fixed > 48 * 1024)
        DC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostBytes));
}

// Fills B for a tile and returns the staged box's bytes.  Where no near sample
// fits (spacings far below the cones' ray lengths never do that; very uneven
// ones may) only the tile's own texels are staged and all others are fetched.
size_t cccs_plan(const CccsCones &C, const Grid &g, CccsPlan &B) {
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
        // a sample's offset is rounded to 1/256 voxel, so up to 1/512 voxel past a whole number it still lies in
        // that voxel, with no weight on the next; 1/600 leaves 3e-4 for the rounding of directions and products
        auto halo = [&](float sp) { return (int)std::min(200.0, std::ceil((double)reach / sp - 1.0 / 600.0)); };
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

}  // namespace

void enqueue_cccs(DeviceContext &ctx, const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w,
                  float dose_scale, float *dose_dev, cudaStream_t s) {
    KernelTimer kt(ctx, "cccs", s);
    CccsPlan B;
    const size_t smem = cccs_plan(C, g, B);
    allow_shared(cccs_kernel, 8 * 1024, smem);
    const dim3 grid((unsigned)((g.nx + Tile::x - 1) / Tile::x), (unsigned)((g.ny + Tile::y - 1) / Tile::y),
                    (unsigned)((g.nz + Tile::z - 1) / Tile::z));
    cccs_kernel<<<grid, kThreads, smem, s>>>(g, f, C, B, g.sx / 10.0f, dose_scale, w.dirs, w.td_tex, w.electron, w.mask,
                                             dose_dev);
    check_launch("cccs_kernel");
}

void enqueue_cccs_points(DeviceContext &ctx, const Grid &g, const Frame &f, const CccsCones &C, const PhotonWork &w,
                         float dose_scale, const int *voxels, int n, float *out, cudaStream_t s) {
    if (n <= 0) return;
    KernelTimer kt(ctx, "cccs_points", s);
    CccsPlan B;
    cccs_plan(C, g, B);  // the tiles' split of the samples
    const size_t texels = (size_t)(2 * B.hx + 2) * (2 * B.hy + 2) * (2 * B.hz + 2);  // of one voxel's box
    const size_t box = texels / (2 * B.hz + 2) * (2 * B.hz + 1) * sizeof(float4);
    // A box per voxel for short lists (100 k entries, 24 k where more than one voxel in 32 is listed: there
    // neighbours share most of theirs), as long as at least three fit
    const bool runs = 56 * 1024 / box < 3 || n >= 100000 || (n >= 24000 && 32LL * n >= g.n());
    if (runs) {
        const size_t one = texels * sizeof(float2);
        const size_t smem = std::max(one, std::min<size_t>(30 * 1024, std::max<size_t>(20 * 1024, 8 * one)));
        allow_shared(cccs_runs_kernel, 20 * 1024, smem);
        // few entries per block keep a sparse list's many short runs apart; a dense one has long runs
        const bool dense = 4LL * n >= g.n();
        const int per_block = dense && n >= 500000 ? 128 : dense && n >= 200000 ? 64 : 16;
        cccs_runs_kernel<<<(unsigned)((n + per_block - 1) / per_block), kRunThreads, smem, s>>>(
            g, f, C, B, per_block, (int)(smem / sizeof(float2)), g.sx / 10.0f, dose_scale, w.dirs, w.td_tex, w.electron,
            voxels, n, out);
        check_launch("cccs_runs_kernel");
        return;
    }
    float reach = 0.0f;
    for (int c = 0; c < C.n_cones; ++c)
        if (B.n_near[c] > 0) reach = std::max(reach, C.rl10[C.step_off[c] + B.n_far[c]]);
    B.wx = 2 * B.hx + 2, B.wy = 2 * B.hy + 2, B.wz = 2 * B.hz + 2;
    const int per_block = (int)std::min<size_t>(kListVoxels, 56 * 1024 / box);
    const size_t smem = box * per_block;
    allow_shared(cccs_list_kernel, 8 * 1024, smem);
    cccs_list_kernel<<<(unsigned)((n + per_block - 1) / per_block), kListThreads, smem, s>>>(
        g, f, C, B, per_block, reach * 1.0001f, g.sx / 10.0f, dose_scale, w.dirs, w.td_tex, w.electron, voxels, n,
        out);
    check_launch("cccs_list_kernel");
}

}  // namespace dc
