// dc_pencil.cu — proton pencil-beam dose and its adjoint, one warp per voxel tile.
//
// The per-pair influence is dc_proton.cu's: for a voxel with smoothed WET w
// and a spot at squared distance r^2 of its divergent axis,
//   K = pf exp2(ps2 r^2) + hf exp2(hs2 r^2),
// dose(v) = sum_s mu_s K_s(v) and grad_mu(s) = sum_v g(v) K_s(v).
//
// What bounds it: the two exponentials per (voxel, spot) pair on the
// special-function unit (4 lanes per clock and SM quarter: 8 clocks per warp
// exponential), so everything else is arranged to stay below that.
//  * A warp owns an 8 x 4 x 4 voxel tile (4 voxels of a thread along z) and
//    walks the energy layers by itself: no block-wide barrier, and a tile half
//    the size of a block's in every lateral direction, which culls more spots.
//  * The lanes test 32 spots at a time against the tile's box and compact the
//    records of those within reach into the warp's shared memory: first the
//    spots whose primary Gaussian matters to the tile, then those of which
//    only the halo does.  Where  pf exp2(ps2 r^2) < 2^-26 hf exp2(hs2 r^2)
//    for every voxel of the tile the primary term is below a quarter ulp of
//    the halo term of the same pair and is not evaluated (the primary falls
//    off within ~7 sigma_t, the halo's reach is 6 sigma_ht, about twice that).
//    It counts where sigma_t is narrow: 65 % of the evaluated pairs of 256 x 256 x
//    160, 32 % of 96^3, but 5 % of the listed voxels' and 0.3 % of the oblique
//    beam's with its range shifter below.
//  * r^2 = U^2 + W^2 with U, W the components of the voxel along two unit
//    vectors normal to the spot's axis, taken relative to the tile's centre.
//    Along the thread's four voxels r^2 is a parabola: 15 operations give the
//    four values (the previous form took 10 per voxel).
//  * Small volumes split the layers of a tile over 2 or 4 warps of the block
//    and add the parts in a fixed order, so the result stays deterministic.
//
// Measured on B200 (ms; before = the 16 x 8 x 4 tile per block of 256 threads
// with its per-layer barriers): 96^3 beam of 2034 spots 0.95 -> 0.41; oblique
// 127 x 113 x 91 with range shifter, 2831 spots 1.08 -> 0.63; 256 x 256 x 160,
// 2655 spots 2.32 -> 1.27; six beams of 160 x 160 x 96 in one batch 5.90 ->
// 2.86; dose / adjoint at 50 k listed voxels, 6025 spots 0.48 -> 0.30 / 1.63
// -> 0.31.  Of the batch's cycles the exponentials take 62 %.  Fewer or more
// registers (24 to 40 warps per SM) changed nothing above 1 %; evaluating a
// quarter of the exponentials as polynomials on the FP32 pipe cost 5 %, tiles
// of 8 x 4 x 8 voxels 4 to 15 %.
#include <algorithm>
#include <cmath>

#include "../../include/dosecuda.h"
#include "dc_common.cuh"
#include "dc_kernels.cuh"
#include "dc_runtime.cuh"

namespace dc {

DC_BOUNDS_WORD

namespace {

constexpr int kVox = 4;                       // voxels per thread, along z
constexpr int kLanesX = 8, kLanesY = 4;       // lanes of a warp along x and y
constexpr int kTileX = kLanesX, kTileY = kLanesY, kTileZ = kVox;
constexpr int kWarpVox = 32 * kVox;
constexpr float kLn2 = 0.6931471805599453f;
constexpr float kPrimaryBits = 26.0f;         // primary terms below 2^-26 of their pair's halo term are left out

// The spots a warp's pair loops read (broadcast), relative to the tile's
// centre: U = p.x lx + p.y ly + p.z lz + p.w, W = q.x ly + q.y lz + q.z for
// head-frame offsets l; per voxel step along z U changes by q.w and W by d.x,
// d.y = (q.w^2 + d.x^2) / 4, and d.z = d.w = the spot's weight.  For listed
// voxels, which share no centre, l is the position itself and p.w, q.z are the
// spot's: U = p.x (lx - p.w) + p.y (ly - q.z) + p.z lz, W = q.x (ly - q.z) + q.y lz.
// The differences are small and nearly exact where the Gaussian is not; sums
// about a common origin would round at the size of lx.  Spots with
// both terms fill the arrays from the front, those with the halo term alone
// from the back.  One array per field keeps the lanes' stores free of bank
// conflicts.
template <bool kAdj>
struct __align__(16) WarpMem {
    static constexpr int kCap = kAdj ? 32 : 64;
    float4 p[kCap], q[kCap], d[kCap];
    int orig[kAdj ? kCap : 1];              // the spot's row in the caller's list
    float part[kAdj ? kCap : 1][33];        // adjoint: [spot][lane] partial sums, padded
};

struct VoxelLayer {
    float pf, hf, ps2, hs2;
};

// The special-function unit's forms without the denormal handling of
// __fdividef and __log2f (several instructions each; none of the operands
// here is denormal).
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float log2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Layer constants of voxel_layer, from LayerRec in five 16-byte loads.
struct LayerView {
    int spot_start, n_spots, energy_id;
    float r80, A, B, C, rcut, lut_d0, lut_inv, lut_step, hs_log, hs_pole, hw_arg, hw_num, hw_edge, hw_lin;
};
__device__ __forceinline__ LayerView load_layer(const LayerRec *L) {
    const float4 *v = reinterpret_cast<const float4 *>(L);
    const float4 a = __ldg(v), b = __ldg(v + 1), d = __ldg(v + 3), e = __ldg(v + 4), f = __ldg(v + 5);
    return LayerView{__float_as_int(a.x), __float_as_int(a.y), __float_as_int(a.z), a.w, b.x, b.y, b.z, b.w,
                     d.w, e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
}

// Per (voxel, layer) Gaussian parameters (interpolateProtonLUT, sigmaAir,
// nuclearHalo, IMPTClasses.cu:69-121).  `dw` = |voxel - source| - wet.  The
// LUT row is computed where the depths are evenly spaced (lut_step > 0: every
// difference of neighbouring depths is the step, so the factor is the searched
// form's; the interpolant is continuous, so a product rounded across a row
// boundary does not matter) and searched for otherwise.
//
// Errors against 64 bits over all energies and depths (rms, largest), in
// brackets the same with logf, hypotf and IEEE divisions throughout: pf 6.3e-8,
// 2.5e-7 (6.5e-8, 3.1e-7); hf relative to pf 4.3e-9, 6.5e-8 (5.7e-9, 7.3e-8);
// ps2 4.6e-8, 1.5e-7 (the same); hs2 8.8e-8, 4.6e-7 (1.1e-7, 5.8e-7).  The
// approximate logarithms and reciprocals serve only the small terms of sigma_h
// and of the halo weight; pf and hf are quotients with their remainder added,
// ps2 and hs2 take a Newton step.  IEEE forms throughout cost the batch kernel
// 19 % (2.83 -> 3.37 ms).
__device__ __forceinline__ VoxelLayer voxel_layer(const LayerView &L, const ProtonTables &t, int l, float wet, float dw) {
    const int n = t.lut_len;
    int i;
    float fac;
    if (L.lut_step > 0.0f) {
        i = min(max((int)ceilf((wet - L.lut_d0) * L.lut_inv), 0), n);
        const float past = wet - fmaf((float)(i - 1), L.lut_step, L.lut_d0);
        fac = past * L.lut_inv;
        fac = fmaf(fmaf(-L.lut_step, fac, past), L.lut_inv, fac);  // past / step, rounded once
    } else {
        const float *D = t.lut_depths + (size_t)L.energy_id * n;
        int a = 0, b = n;
        while (a < b) {  // first row with wet <= depth
            const int mid = (a + b) >> 1;
            if (wet <= __ldg(D + mid)) b = mid; else a = mid + 1;
        }
        i = a;
        fac = i > 0 && i < n ? (wet - __ldg(D + i - 1)) / (__ldg(D + i) - __ldg(D + i - 1)) : 0.0f;
    }
    const float4 row = __ldg(t.rows + (size_t)l * (n + 1) + i);
    const float sig = fmaf(row.z, fac, row.x), idd = fmaf(row.w, fac, row.y);
    const float r80 = L.r80;
    const float d = dw + 0.7f * r80;
    const float sigma_t = fmaf(fmaf(L.A, d, L.B), d, L.C) + sig;
    const float w = clampf(wet, 0.1f, r80 - 0.1f);
    const float hs = fmaf(w, fmaf(-7.4e-5f, w, 0.06f), fmaf(L.hs_log, log2_approx(w + 3.0f), 2.85f)) -
                     L.hs_pole * rcp_approx(sqr(w - r80 - 5.0f));
    const float hw = fmaf(0.052f * kLn2, log2_approx(fmaf(w, L.hw_arg, 1.13f)),
                          fmaf(L.hw_num, rcp_approx((L.hw_edge - w) * (L.hw_edge + w)), -L.hw_lin * w));
    const float sigma_h = fmaxf(hs, 0.0f);
    const float wh = clampf(hw, 0.0f, 0.9f);
    const float t2 = sqr(sigma_t), h2 = fmaf(sigma_t, sigma_t, sqr(sigma_h));
    const float rt = rcp_approx(t2), rh = rcp_approx(h2);
    auto over_2pi = [](float a, float s2, float r) {  // a / (2 pi s2), r ~ 1 / s2
        const float inv = r * (0.5f / CUDART_PI_F), q = a * inv;
        return fmaf(fmaf(-2.0f * CUDART_PI_F * s2, q, a), inv, q);
    };
    VoxelLayer o;
    o.pf = over_2pi((1.0f - wh) * idd, t2, rt);
    o.hf = over_2pi(wh * idd, h2, rh);
    o.ps2 = (-0.5f * kLog2e) * fmaf(rt, fmaf(-t2, rt, 1.0f), rt);
    o.hs2 = (-0.5f * kLog2e) * fmaf(rh, fmaf(-h2, rh, 1.0f), rh);
    return o;
}

__device__ __forceinline__ float warp_max_pos(float x) {  // max over the warp of values >= 0 (NaN ignored)
    return __uint_as_float(__reduce_max_sync(0xffffffffu, x > 0.0f ? __float_as_uint(x) : 0u));
}
__device__ __forceinline__ float warp_min(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

__device__ __forceinline__ float2 ex2_pair(float2 x) { return make_float2(fast_exp2(x.x), fast_exp2(x.y)); }

// Head-frame position of an image position, in double (image_to_head<false>).
__device__ __forceinline__ void head_centre(const Frame &f, double x, double y, double z, float3 &c, float2 &cl) {
    const double xt = x * f.cta - z * f.sta, zt = x * f.sta + z * f.cta;
    const double hx = -(xt * f.cga + y * f.sga), hz = y * f.cga - xt * f.sga;
    c = make_float3((float)hx, (float)zt, (float)hz);
    cl = make_float2((float)(hx - c.x), (float)(zt - c.y));
}

// Voxels of one warp: head-frame offsets from the centre `c` (per thread: the
// middle of its voxels in tile mode, each voxel in list mode), the offset per
// voxel step along z, and the head-frame box of all its voxels.
template <bool kList>
struct WarpGeom {
    float3 c;                       // centre, head frame,
    float2 cl;                      // and what the rounding of c.x, c.y left (the tile's voxels share it)
    float3 l[kList ? kVox : 1];     // offsets from it
    float3 dz;                      // offset of one voxel step (tile mode)
    float bx0, bx1, by0, by1, bz0, bz1;
    float wet[kVox], dw[kVox];      // WET (mm), |voxel - source| - WET; +inf WET where there is no voxel
};

// Layers l0 + bit (one per lane) whose range reaches depth wmin and whose
// spots, as a whole, come within the layer's cut-off of the tile's box: their
// axes at the box's heights span [x0 fx, x1 fx] with fx = 1 - hz / VSAD.
template <bool kList>
__device__ __forceinline__ unsigned layers_reaching(const ProtonTables &t, const WarpGeom<kList> &G, int l0, float wmin) {
    const int l = l0 + (int)(threadIdx.x & 31);
    bool hit = false;
    if (l < t.n_layers) {
        const LayerRec &L = t.layers[l];
        const float fx0 = fmaf(-G.bz0, L.inv_vx, 1.0f), fx1 = fmaf(-G.bz1, L.inv_vx, 1.0f);
        const float fy0 = fmaf(-G.bz0, L.inv_vy, 1.0f), fy1 = fmaf(-G.bz1, L.inv_vy, 1.0f);
        const float xl = fminf(fminf(L.x0 * fx0, L.x0 * fx1), fminf(L.x1 * fx0, L.x1 * fx1));
        const float xh = fmaxf(fmaxf(L.x0 * fx0, L.x0 * fx1), fmaxf(L.x1 * fx0, L.x1 * fx1));
        const float yl = fminf(fminf(L.y0 * fy0, L.y0 * fy1), fminf(L.y1 * fy0, L.y1 * fy1));
        const float yh = fmaxf(fmaxf(L.y0 * fy0, L.y0 * fy1), fmaxf(L.y1 * fy0, L.y1 * fy1));
        const float dx = fmaxf(0.0f, fmaxf(xl - G.bx1, G.bx0 - xh)), dy = fmaxf(0.0f, fmaxf(yl - G.by1, G.by0 - yh));
        hit = !(wmin > 1.1f * L.r80) && !((dx * dx + dy * dy) * L.it2_min * 0.9999f > L.rcut * L.rcut);
    }
    return __ballot_sync(0xffffffffu, hit);
}

// Sum over the beam's layers that reach the tile, every step-th one from the
// first-th on (for warps that share the tile).  kAdj: gv holds
// the voxels' dose gradients and each spot's sum goes to x.grad_mu; else the
// dose of each voxel is added to acc.
template <bool kAdj, bool kList>
__device__ __forceinline__ void warp_beam(const ProtonTables &t, const PbExtra &x, const WarpGeom<kList> &G,
                                          WarpMem<kAdj> &mem, int first, int step,
                                          const float (&gv)[kVox], float (&acc)[kVox]) {
    const int lane = threadIdx.x & 31;
    float wmin = INFINITY;  // shallowest voxel that takes part (NaN counts as reached by every layer)
#pragma unroll
    for (int v = 0; v < kVox; ++v)
        // a voxel with zero gradient adds exactly zero to every spot's sum
        if (!kAdj || gv[v] != 0.0f) wmin = fminf(wmin, G.wet[v] == G.wet[v] ? G.wet[v] : -INFINITY);
    wmin = warp_min(wmin);
    int turn = 0;  // layers taken so far by the warps that share this tile
    for (int l0 = 0; l0 < t.n_layers; l0 += 32) {
        unsigned todo = layers_reaching(t, G, l0, wmin);
        for (; todo != 0u; todo &= todo - 1u) {
            const int l = l0 + __ffs(todo) - 1;
            // in turn over the tile's layers; a listed voxel's parts must not depend on which layers its warp reaches
            if ((kList ? l : turn++) % step != first) continue;
            const LayerView L = load_layer(t.layers + l);
            const float r80 = L.r80;
            bool act[kVox];
#pragma unroll
            for (int v = 0; v < kVox; ++v) act[v] = !(G.wet[v] > 1.1f * r80) && (!kAdj || gv[v] != 0.0f);
            VoxelLayer pv[kVox];
            float hmax = -INFINITY, ratio = 0.0f, dmin = INFINITY;
#pragma unroll
            for (int v = 0; v < kVox; ++v) {
                pv[v] = VoxelLayer{0.f, 0.f, 0.f, 0.f};
                if (!act[v]) continue;
                pv[v] = voxel_layer(L, t, l, G.wet[v], G.dw[v]);
                if (pv[v].hs2 < 0.0f) hmax = fmaxf(hmax, pv[v].hs2);
                const float q = pv[v].pf * rcp_approx(pv[v].hf);
                ratio = fmaxf(ratio, q == q ? q : INFINITY);  // no halo: the primary is never left out
                dmin = fminf(dmin, pv[v].hs2 - pv[v].ps2);
            }
            // smallest r^2 from which on every primary term is below 2^-26 of its halo term; a lane without a
            // voxel has no say
            const bool any = act[0] || act[1] || act[2] || act[3];
            const float rp = any ? (kPrimaryBits + log2_approx(ratio)) * rcp_approx(dmin) * 1.0001f : 0.0f;
            // Lateral cut-off of this tile for this layer: 6 x the widest halo
            // sigma of its active voxels, never wider than the layer's bound.  A
            // spot whose axis stays farther than that from the tile's box lies
            // beyond 6 sigma_ht of every voxel here, where both Gaussians are
            // below exp(-18) of their peaks.
            const float s2 = hmax < 0.0f ? (-0.5f * kLog2e) * rcp_approx(hmax) : 0.0f;
            const float rc = 6.0f * (sqrtf(warp_max_pos(s2)) * 1.01f + 0.1f);
            const float rcut2 = fminf(L.rcut * L.rcut, rc * rc);
            const float rprim2 = warp_max_pos(rp == rp ? rp : INFINITY);

            float2 ps01, ps23, hs01, hs23;
            ps01 = make_float2(pv[0].ps2, pv[1].ps2);
            ps23 = make_float2(pv[2].ps2, pv[3].ps2);
            hs01 = make_float2(pv[0].hs2, pv[1].hs2);
            hs23 = make_float2(pv[2].hs2, pv[3].hs2);
            // dose: sums of mu exp2; adjoint: the factors g pf, g hf
            float2 p01 = make_float2(0.f, 0.f), p23 = p01, h01 = p01, h23 = p01;
            if (kAdj) {
                p01 = make_float2(gv[0] * pv[0].pf, gv[1] * pv[1].pf);
                p23 = make_float2(gv[2] * pv[2].pf, gv[3] * pv[3].pf);
                h01 = make_float2(gv[0] * pv[0].hf, gv[1] * pv[1].hf);
                h23 = make_float2(gv[2] * pv[2].hf, gv[3] * pv[3].hf);
            }

            constexpr int kCap = WarpMem<kAdj>::kCap;
            int nf = 0, nh = 0;
            for (int c0 = 0;; c0 += 32) {
                const bool last = c0 >= L.n_spots;
                if (last || nf + nh > kCap - 32) {  // the lists are full: evaluate their pairs
                    __syncwarp();
                    auto distances = [&](int q, const float4 &D, float2 &r01, float2 &r23) {
                        const float4 P = mem.p[q], Q = mem.q[q];
                        if constexpr (kList) {
                            float r2[kVox];
#pragma unroll
                            for (int v = 0; v < kVox; ++v) {
                                const float rx = G.l[v].x - P.w, ry = G.l[v].y - Q.z;
                                const float U = fmaf(P.x, rx, fmaf(P.y, ry, P.z * G.l[v].z));
                                const float W = fmaf(Q.x, ry, Q.y * G.l[v].z);
                                r2[v] = fmaf(U, U, W * W);
                            }
                            r01 = make_float2(r2[0], r2[1]);
                            r23 = make_float2(r2[2], r2[3]);
                        } else {
                            const float U = fmaf(P.x, G.l[0].x, fmaf(P.y, G.l[0].y, fmaf(P.z, G.l[0].z, P.w)));
                            const float W = fmaf(Q.x, G.l[0].y, fmaf(Q.y, G.l[0].z, Q.z));
                            const float m = fmaf(U, U, W * W), b2 = fmaf(U, Q.w, W * D.x);
                            const float A = fmaf(9.0f, D.y, m), B = m + D.y;
                            r01 = make_float2(fmaf(-3.0f, b2, A), B - b2);
                            r23 = make_float2(B + b2, fmaf(3.0f, b2, A));
                        }
                    };
                    if constexpr (kAdj) {
                        float2 r01, r23;
                        for (int q = 0; q < nf; ++q) {
                            distances(q, mem.d[q], r01, r23);
                            float2 c = __fmul2_rn(p01, ex2_pair(__fmul2_rn(ps01, r01)));
                            c = __ffma2_rn(h01, ex2_pair(__fmul2_rn(hs01, r01)), c);
                            c = __ffma2_rn(p23, ex2_pair(__fmul2_rn(ps23, r23)), c);
                            c = __ffma2_rn(h23, ex2_pair(__fmul2_rn(hs23, r23)), c);
                            mem.part[q][lane] = c.x + c.y;
                        }
                        for (int q = kCap - nh; q < kCap; ++q) {
                            distances(q, mem.d[q], r01, r23);
                            const float2 c = __ffma2_rn(h01, ex2_pair(__fmul2_rn(hs01, r01)),
                                                        __fmul2_rn(h23, ex2_pair(__fmul2_rn(hs23, r23))));
                            mem.part[q][lane] = c.x + c.y;
                        }
                        __syncwarp();
                        if (lane < nf || lane >= kCap - nh) {  // lane q sums spot q over the warp: one atomic per spot
                            float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                            for (int k = 0; k < 32; ++k) c[k & 3] += mem.part[lane][k];
                            const double sum = ((double)c[0] + c[1]) + ((double)c[2] + c[3]);
                            if (sum != 0.0) atomicAdd(x.grad_mu + mem.orig[lane], sum);
                        }
                    } else {
                        float2 r01, r23;
#pragma unroll 2
                        for (int q = 0; q < nf; ++q) {
                            const float4 D = mem.d[q];
                            const float2 mu = make_float2(D.z, D.w);
                            distances(q, D, r01, r23);
                            p01 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(ps01, r01)), p01);
                            h01 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(hs01, r01)), h01);
                            p23 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(ps23, r23)), p23);
                            h23 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(hs23, r23)), h23);
                        }
#pragma unroll 2
                        for (int q = kCap - nh; q < kCap; ++q) {
                            const float4 D = mem.d[q];
                            const float2 mu = make_float2(D.z, D.w);
                            distances(q, D, r01, r23);
                            h01 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(hs01, r01)), h01);
                            h23 = __ffma2_rn(mu, ex2_pair(__fmul2_rn(hs23, r23)), h23);
                        }
                    }
                    __syncwarp();
                    nf = nh = 0;
                    if (last) break;
                }
                const int s = c0 + lane;
                bool keep = false, full = false;
                float4 a, b;
                if (s < L.n_spots) {
                    const float4 *sp = reinterpret_cast<const float4 *>(t.spots + L.spot_start + s);
                    a = __ldg(sp);
                    b = __ldg(sp + 1);
                    const float ax0 = a.x - b.x * G.bz0, ax1 = a.x - b.x * G.bz1;
                    const float ay0 = a.y - b.y * G.bz0, ay1 = a.y - b.y * G.bz1;
                    const float dx = fmaxf(0.0f, fmaxf(fminf(ax0, ax1) - G.bx1, G.bx0 - fmaxf(ax0, ax1)));
                    const float dy = fmaxf(0.0f, fmaxf(fminf(ay0, ay1) - G.by1, G.by0 - fmaxf(ay0, ay1)));
                    // perpendicular distance >= lateral distance * cos(tilt), cos^2 = inv_t2
                    const float r2min = (dx * dx + dy * dy) * b.z;
                    keep = !(r2min > rcut2);
                    full = keep && !(r2min > rprim2);
                }
                const unsigned mf = __ballot_sync(0xffffffffu, full), mh = __ballot_sync(0xffffffffu, keep && !full);
                if (keep) {
                    const unsigned below = (1u << lane) - 1u;
                    const int pos = full ? nf + __popc(mf & below) : kCap - 1 - (nh + __popc(mh & below));
                    const float tx = b.x, ty = b.y;
                    // unit vectors normal to the axis: (e.x, e.y, e.z) and (0, e.w, e.w ty)
                    const float4 e = __ldg(t.axes + L.spot_start + s);
                    const float k2 = e.w * ty;
                    const float cu = fmaf(G.c.z, tx, G.c.x - a.x) + G.cl.x, cw = fmaf(G.c.z, ty, G.c.y - a.y) + G.cl.y;
                    const float uw = kList ? a.x : fmaf(e.x, cu, e.y * cw), wz = kList ? a.y : e.w * cw;
                    const float du = fmaf(e.x, G.dz.x, fmaf(e.y, G.dz.y, e.z * G.dz.z)), dw = fmaf(e.w, G.dz.y, k2 * G.dz.z);
                    float mu = a.z;
                    if (!kAdj && x.mu != nullptr) mu = __ldg(x.mu + __float_as_int(a.w));
                    mem.p[pos] = make_float4(e.x, e.y, e.z, uw);
                    mem.q[pos] = make_float4(e.w, k2, wz, du);
                    mem.d[pos] = make_float4(dw, 0.25f * fmaf(du, du, dw * dw), mu, mu);
                    if (kAdj) mem.orig[pos] = __float_as_int(a.w);
                }
                nf += __popc(mf);
                nh += __popc(mh);
            }
            if constexpr (!kAdj) {
                if (act[0]) acc[0] += fmaf(pv[0].pf, p01.x, pv[0].hf * h01.x);
                if (act[1]) acc[1] += fmaf(pv[1].pf, p01.y, pv[1].hf * h01.y);
                if (act[2]) acc[2] += fmaf(pv[2].pf, p23.x, pv[2].hf * h23.x);
                if (act[3]) acc[3] += fmaf(pv[3].pf, p23.y, pv[3].hf * h23.y);
            }
        }
    }
}

// The warp's index in its block through a shuffle, which lets the compiler see
// that it is the same in all lanes: the addresses of the warp's shared memory
// then live in uniform registers and cost the pair loops no instructions (batch
// of six beams 3.24 -> 2.83 ms, 256 x 256 x 160 1.35 -> 1.27).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

// WET of voxel u in mm.  At -infinity the air sigma is infinite and the dose 0:
// no voxel.
__device__ __forceinline__ float voxel_wet(const float *__restrict__ wet_s, long long u) {
    const float w = __ldg(wet_s + u) * 10.0f;
    return w == -INFINITY ? INFINITY : w;
}

// Geometry of the tile with low corner (i0, j0, k0) and, when a layer of the
// beam comes near its box, the voxels' depths; false when none does.  gv: the
// voxels' gradients where grad is given (0 outside the grid).
__device__ __forceinline__ bool tile_geom(const Grid &g, const Frame &f, const ProtonTables &t,
                                          const float *__restrict__ wet_s, int i0, int j0, int k0,
                                          const float *__restrict__ grad, WarpGeom<false> &G, float (&gv)[kVox]) {
    const int lane = threadIdx.x & 31;
    const int i = i0 + (lane & (kLanesX - 1)), j = j0 + lane / kLanesX;
    const float3 ex = image_to_head<false>(f, make_float3(1.f, 0.f, 0.f));
    const float3 ey = image_to_head<false>(f, make_float3(0.f, 1.f, 0.f));
    const float3 ez = image_to_head<false>(f, make_float3(0.f, 0.f, 1.f));
    const float hx = 0.5f * (kTileX - 1) * g.sx, hy = 0.5f * (kTileY - 1) * g.sy, hz = 0.5f * (kTileZ - 1) * g.sz;
    head_centre(f, (i0 + 0.5 * (kTileX - 1)) * g.sx - f.isox, (j0 + 0.5 * (kTileY - 1)) * g.sy - f.isoy,
                (k0 + 0.5 * (kTileZ - 1)) * g.sz - f.isoz, G.c, G.cl);
    const float ox = (float)(i - i0) * g.sx - hx, oy = (float)(j - j0) * g.sy - hy;
    G.l[0] = make_float3(fmaf(ex.x, ox, ey.x * oy), fmaf(ex.y, ox, ey.y * oy), fmaf(ex.z, ox, ey.z * oy));
    G.dz = make_float3(ez.x * g.sz, ez.y * g.sz, ez.z * g.sz);
    const float rx = fabsf(ex.x) * hx + fabsf(ey.x) * hy + fabsf(ez.x) * hz;
    const float ry = fabsf(ex.y) * hx + fabsf(ey.y) * hy + fabsf(ez.y) * hz;
    const float rz = fabsf(ex.z) * hx + fabsf(ey.z) * hy + fabsf(ez.z) * hz;
    G.bx0 = G.c.x - rx, G.bx1 = G.c.x + rx;
    G.by0 = G.c.y - ry, G.by1 = G.c.y + ry;
    G.bz0 = G.c.z - rz, G.bz1 = G.c.z + rz;
    unsigned near = 0u;
    for (int l0 = 0; l0 < t.n_layers && near == 0u; l0 += 32) near = layers_reaching(t, G, l0, -INFINITY);
    if (near == 0u) return false;
#pragma unroll
    for (int v = 0; v < kVox; ++v) {
        const int k = k0 + v;
        const bool inside = i < g.nx && j < g.ny && k < g.nz;
        G.wet[v] = INFINITY;
        G.dw[v] = 0.0f;
        gv[v] = 0.0f;
        if (!inside) continue;
        const long long u = (long long)i + (long long)g.nx * (j + (long long)g.ny * k);
        if (!DC_IN_BOUNDS(u, g.n(), 25)) continue;
        G.wet[v] = voxel_wet(wet_s, u);
        G.dw[v] = distance_to_source(f, voxel_xyz(g, f, i, j, k)) - G.wet[v];
        if (grad != nullptr) gv[v] = __ldg(grad + u);
    }
    return true;
}

constexpr int kWarps = 4;  // warps of a block of the one-beam kernels

// One-beam kernels over the image: a block's warps take 4 / split tiles
// (2 x 2, 2 x 1 or one) and `split` warps share a tile's layers.
template <bool kAdj>
__global__ void __launch_bounds__(32 * kWarps, 7)
    pencil_tile_kernel(Grid g, Frame f, ProtonTables t, const float *__restrict__ wet_s, float *__restrict__ dose,
                       PbExtra x, int split) {
    extern __shared__ float4 smem4[];
    WarpMem<kAdj> *mems = reinterpret_cast<WarpMem<kAdj> *>(smem4);
    const int w = warp_index(), lane = threadIdx.x & 31;
    const int tile = w / split, part = w - tile * split;
    const int bx = split == 4 ? 1 : 2, by = split == 1 ? 2 : 1;  // tiles of the block along x and y
    const int i0 = (blockIdx.x * bx + tile % bx) * kTileX, j0 = (blockIdx.y * by + tile / bx) * kTileY;
    const int k0 = ((int)blockIdx.z + x.tile_z0) * kTileZ;
    WarpGeom<false> G;
    float gv[kVox], acc[kVox];
#pragma unroll
    for (int v = 0; v < kVox; ++v) acc[v] = 0.0f;
    if (tile_geom(g, f, t, wet_s, i0, j0, k0, kAdj ? x.grad_dose : nullptr, G, gv))
        warp_beam<kAdj, false>(t, x, G, mems[w], part, split, gv, acc);
    if (kAdj) return;
    if (split > 1) {  // add the parts of a tile in warp order
        float *s_acc = reinterpret_cast<float *>(smem4);
        __syncthreads();
#pragma unroll
        for (int v = 0; v < kVox; ++v) s_acc[(w * kVox + v) * 32 + lane] = acc[v];
        __syncthreads();
        if (part != 0) return;
        for (int q = 1; q < split; ++q)
#pragma unroll
            for (int v = 0; v < kVox; ++v) acc[v] += s_acc[((w + q) * kVox + v) * 32 + lane];
    }
    const int i = i0 + (lane & (kLanesX - 1)), j = j0 + lane / kLanesX;
    if (i >= g.nx || j >= g.ny) return;
#pragma unroll
    for (int v = 0; v < kVox; ++v) {
        const long long u = (long long)i + (long long)g.nx * (j + (long long)g.ny * (k0 + v));
        if (k0 + v < g.nz && DC_IN_BOUNDS(u, g.n(), 20)) dose[u] = acc[v];
    }
}

// Voxel-list kernel: a warp takes 128 consecutive list entries, 32 per step
// (a sorted list keeps them close together).  A voxel's distances and the split
// of its layers are its own; the cut-offs are the warp's.  In another list the
// same voxel may lose or gain terms beyond 6 sigma_ht (1.5e-8 of the halo's peak
// each) and primaries below 2^-26 of their halo term, and add its spots in
// another order.
template <bool kAdj>
__global__ void __launch_bounds__(32 * kWarps, 6)
    pencil_list_kernel(Grid g, Frame f, ProtonTables t, const float *__restrict__ wet_s, PbExtra x, int split) {
    extern __shared__ float4 smem4[];
    WarpMem<kAdj> *mems = reinterpret_cast<WarpMem<kAdj> *>(smem4);
    const int w = warp_index(), lane = threadIdx.x & 31;
    const int tile = w / split, part = w - tile * split;
    const long long e0 = ((long long)blockIdx.x * (kWarps / split) + tile) * kWarpVox;
    WarpGeom<true> G;
    float gv[kVox], acc[kVox];
    const long long plane = (long long)g.nx * g.ny;
    // Positions relative to the isocentre, not to a voxel of the warp: a
    // voxel's distances then do not depend on the list's other entries.
    G.c = make_float3(0.f, 0.f, 0.f);
    G.cl = make_float2(0.f, 0.f);
    G.dz = make_float3(0.f, 0.f, 0.f);
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool have = false;
#pragma unroll
    for (int v = 0; v < kVox; ++v) {
        const long long e = e0 + v * 32 + lane;
        const long long vi = e < x.n_list ? (long long)__ldg(x.list + e) : -1;
        const bool valid = vi >= 0 && vi < plane * g.nz;  // out-of-grid entries give 0
        const long long u = valid ? vi : 0;
        const int k = (int)(u / plane);
        const long long rem = u - (long long)k * plane;
        const int j = (int)(rem / g.nx), i = (int)(rem - (long long)j * g.nx);
        const float3 p = voxel_xyz(g, f, i, j, k);
        G.l[v] = image_to_head<false>(f, p);
        G.wet[v] = INFINITY;
        G.dw[v] = 0.0f;
        gv[v] = 0.0f;
        acc[v] = 0.0f;
        if (valid && DC_IN_BOUNDS(u, g.n(), 21)) {
            have = true;
            G.wet[v] = voxel_wet(wet_s, u);
            G.dw[v] = distance_to_source(f, p) - G.wet[v];
            if (kAdj) gv[v] = __ldg(x.grad_dose + e);
            lo[0] = fminf(lo[0], G.l[v].x), hi[0] = fmaxf(hi[0], G.l[v].x);
            lo[1] = fminf(lo[1], G.l[v].y), hi[1] = fmaxf(hi[1], G.l[v].y);
            lo[2] = fminf(lo[2], G.l[v].z), hi[2] = fmaxf(hi[2], G.l[v].z);
        }
    }
    have = __any_sync(0xffffffffu, have);
    G.bx0 = warp_min(lo[0]), G.bx1 = warp_max(hi[0]);
    G.by0 = warp_min(lo[1]), G.by1 = warp_max(hi[1]);
    G.bz0 = warp_min(lo[2]), G.bz1 = warp_max(hi[2]);
    if (have) warp_beam<kAdj, true>(t, x, G, mems[w], part, split, gv, acc);
    if (kAdj) return;
    if (split > 1) {
        float *s_acc = reinterpret_cast<float *>(smem4);
        __syncthreads();
#pragma unroll
        for (int v = 0; v < kVox; ++v) s_acc[(w * kVox + v) * 32 + lane] = acc[v];
        __syncthreads();
        if (part != 0) return;
        for (int q = 1; q < split; ++q)
#pragma unroll
            for (int v = 0; v < kVox; ++v) acc[v] += s_acc[((w + q) * kVox + v) * 32 + lane];
    }
#pragma unroll
    for (int v = 0; v < kVox; ++v) {
        const long long e = e0 + v * 32 + lane;
        if (e < x.n_list && DC_IN_BOUNDS(e, x.n_list, 22)) x.list_out[e] = acc[v];
    }
}

// Persistent batch kernel: each warp takes (plan, tile) items from a device
// queue (most expensive plans first) and sums the dose of all the plan's
// beams for the tile in registers before one write per voxel.  The plan and
// beam records are staged in the warp's shared memory and read from there.
template <class T>
__device__ __forceinline__ void stage_record(T *dst, const T *__restrict__ src) {
    static_assert(sizeof(T) % sizeof(int) == 0, "records are copied as words");
    const int *s = reinterpret_cast<const int *>(src);
    int *d = reinterpret_cast<int *>(dst);
    for (int q = threadIdx.x & 31; q < (int)(sizeof(T) / sizeof(int)); q += 32) d[q] = __ldg(s + q);
}

struct __align__(16) BatchMem {
    WarpMem<false> w;
    PbBatchPlan plan;
    PbBatchBeam beam;
};

template <int kW>
__global__ void __launch_bounds__(32 * kW, 28 / kW)
    pencil_batch_kernel(const PbBatchPlan *__restrict__ plans, const PbBatchBeam *__restrict__ beams,
                        const long long *__restrict__ first_tile, int n_plans, unsigned *__restrict__ next) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31;
    BatchMem &M = reinterpret_cast<BatchMem *>(smem4)[warp_index()];
    const long long n_items = __ldg(first_tile + n_plans);
    while (true) {
        unsigned it = 0;
        if (lane == 0) it = atomicAdd(next, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if ((long long)it >= n_items) break;
        int lo = 0, hi = n_plans - 1;  // last plan (in queue order) whose first tile is <= it
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(first_tile + mid) <= (long long)it) lo = mid; else hi = mid - 1;
        }
        __syncwarp();
        stage_record(&M.plan, plans + lo);
        __syncwarp();
        const PbBatchPlan &P = M.plan;
        const int nx = (P.g.nx + kTileX - 1) / kTileX, ny = (P.g.ny + kTileY - 1) / kTileY;
        const int tile = (int)((long long)it - __ldg(first_tile + lo));
        const int bz = tile / (nx * ny), rem = tile - bz * nx * ny;
        const int i0 = (rem % nx) * kTileX, j0 = (rem / nx) * kTileY, k0 = bz * kTileZ;
        float acc[kVox], gv[kVox];
#pragma unroll
        for (int v = 0; v < kVox; ++v) acc[v] = 0.0f;
        for (int b = P.beam0; b < P.beam0 + P.n_beams; ++b) {
            __syncwarp();
            stage_record(&M.beam, beams + b);
            __syncwarp();
            PbExtra x;
            x.mu = M.beam.mu;
            WarpGeom<false> G;
            if (tile_geom(P.g, M.beam.f, M.beam.t, M.beam.wet, i0, j0, k0, nullptr, G, gv))
                warp_beam<false, false>(M.beam.t, x, G, M.w, 0, 1, gv, acc);
        }
        const int i = i0 + (lane & (kLanesX - 1)), j = j0 + lane / kLanesX;
#pragma unroll
        for (int v = 0; v < kVox; ++v) {
            const long long u = (long long)i + (long long)P.g.nx * (j + (long long)P.g.ny * (k0 + v));
            if (i < P.g.nx && j < P.g.ny && k0 + v < P.g.nz && DC_IN_BOUNDS(u, P.g.n(), 23)) P.dose[u] = acc[v];
        }
    }
}

// Warps per tile: layers are split while the tiles alone make fewer than
// kWaves rounds of the chip's 28 warps per SM.  Tiles differ in cost by the
// spots and layers that reach them (many have none), so few rounds end in a
// long tail.
constexpr int kWaves = 8;
int layer_split(const DeviceContext &ctx, long long tiles, int n_layers) {
    int sms = 0;
    DC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
    int split = 1;
    while (split < 4 && 2 * split <= n_layers && tiles * split < (long long)sms * 28 * kWaves) split *= 2;
    return split;
}

template <bool kAdj>
void tile_launch(DeviceContext &ctx, const char *name, const Grid &g, const Frame &f, const ProtonTables &t,
                 const float *wet_s, float *dose, const PbExtra &x, cudaStream_t s) {
    const int tx = (g.nx + kTileX - 1) / kTileX, ty = (g.ny + kTileY - 1) / kTileY, tz = (g.nz + kTileZ - 1) / kTileZ;
    const int z1 = x.tile_z1 < 0 ? tz : std::min(x.tile_z1, tz);
    if (x.tile_z0 < 0 || x.tile_z0 >= z1) return;
    // by the whole volume's tiles, so that a call in slabs sums as one without
    const int split = layer_split(ctx, (long long)tx * ty * tz, t.n_layers);
    const int bx = split == 4 ? 1 : 2, by = split == 1 ? 2 : 1;
    const dim3 grid((unsigned)((tx + bx - 1) / bx), (unsigned)((ty + by - 1) / by), (unsigned)(z1 - x.tile_z0));
    constexpr size_t smem = kWarps * sizeof(WarpMem<kAdj>);
    static_assert(smem <= 48 * 1024, "fits without opt-in");
    KernelTimer kt(ctx, name, s);
    pencil_tile_kernel<kAdj><<<grid, 32 * kWarps, smem, s>>>(g, f, t, wet_s, dose, x, split);
    check_launch(name);
}

template <bool kAdj>
void list_launch(DeviceContext &ctx, const char *name, const Grid &g, const Frame &f, const ProtonTables &t,
                 const float *wet_s, const PbExtra &x, cudaStream_t s) {
    if (x.n_list <= 0) return;
    const long long tiles = ((long long)x.n_list + kWarpVox - 1) / kWarpVox;
    const int split = layer_split(ctx, 0, t.n_layers);  // the same for every list, so that the layers' parts are
    const long long per = kWarps / split;
    constexpr size_t smem = kWarps * sizeof(WarpMem<kAdj>);
    KernelTimer kt(ctx, name, s);
    pencil_list_kernel<kAdj><<<(unsigned)((tiles + per - 1) / per), 32 * kWarps, smem, s>>>(g, f, t, wet_s, x, split);
    check_launch(name);
}

template <int kW>
void batch_launch(DeviceContext &ctx, const PbBatchPlan *plans, const PbBatchBeam *beams, const long long *first_tile,
                  int n_plans, long long n_items, unsigned *next, cudaStream_t s) {
    constexpr size_t smem = kW * sizeof(BatchMem);
    static_assert(smem <= 48 * 1024, "fits without opt-in");
    int sms = 0, per_sm = 0;
    DC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx.device));
    DC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pencil_batch_kernel<kW>, 32 * kW, smem));
    const long long blocks = std::max(1LL, std::min((n_items + kW - 1) / kW, (long long)sms * std::max(per_sm, 1)));
    DC_CUDA(cudaMemsetAsync(next, 0, sizeof(unsigned), s));
    KernelTimer kt(ctx, "pencil_beam_batch", s);
    pencil_batch_kernel<kW><<<(unsigned)blocks, 32 * kW, smem, s>>>(plans, beams, first_tile, n_plans, next);
    check_launch("pencil_batch_kernel");
}

}  // namespace

DC_BOUNDS_TAKE(take_bounds_pencil)

void launch_pencil_beam(DeviceContext &ctx, const Grid &g, const Frame &f, const ProtonTables &t,
                        const float *wet_s, float *dose, cudaStream_t s, const float *mu_dev, int tile_z0,
                        int tile_z1) {
    PbExtra x;
    x.mu = mu_dev;
    x.tile_z0 = tile_z0;
    x.tile_z1 = tile_z1;
    tile_launch<false>(ctx, "pencil_beam", g, f, t, wet_s, dose, x, s);
}

int pencil_beam_tile_depth() { return kTileZ; }

void launch_pencil_beam_adjoint(DeviceContext &ctx, const Grid &g, const Frame &f, const ProtonTables &t,
                                const float *wet_s, const PbExtra &x, cudaStream_t s) {
    tile_launch<true>(ctx, "pencil_beam_adjoint", g, f, t, wet_s, nullptr, x, s);
}

void launch_pencil_beam_list(DeviceContext &ctx, int mode, const Grid &g, const Frame &f, const ProtonTables &t,
                             const float *wet_s, const PbExtra &x, cudaStream_t s) {
    switch (mode) {
        case kPbDose: list_launch<false>(ctx, "pencil_beam_list", g, f, t, wet_s, x, s); break;
        case kPbAdjoint: list_launch<true>(ctx, "pencil_beam_list_adjoint", g, f, t, wet_s, x, s); break;
        default: throw Error(DC_ERR_VALUE, "voxel-list mode is for the dose and the adjoint");
    }
}

// Variants of the batch kernel: warps per block.  The warps work alone, so
// the variants differ only in how blocks share an SM.
static const int kBatchWarps[] = {4, 2, 1, 7};
int pencil_beam_batch_variants() { return (int)(sizeof(kBatchWarps) / sizeof(kBatchWarps[0])); }
long long pencil_beam_batch_tiles(const Grid &g) {
    return (long long)((g.nx + kTileX - 1) / kTileX) * ((g.ny + kTileY - 1) / kTileY) * ((g.nz + kTileZ - 1) / kTileZ);
}

void launch_pencil_beam_batch(DeviceContext &ctx, int variant, const PbBatchPlan *plans, const PbBatchBeam *beams,
                              const long long *first_tile, int n_plans, long long n_items, unsigned *next,
                              cudaStream_t s) {
    switch (variant) {
        case 0: batch_launch<4>(ctx, plans, beams, first_tile, n_plans, n_items, next, s); break;
        case 1: batch_launch<2>(ctx, plans, beams, first_tile, n_plans, n_items, next, s); break;
        case 2: batch_launch<1>(ctx, plans, beams, first_tile, n_plans, n_items, next, s); break;
        case 3: batch_launch<7>(ctx, plans, beams, first_tile, n_plans, n_items, next, s); break;
        default: throw Error(DC_ERR_VALUE, "unknown pencil-beam tile variant");
    }
}

}  // namespace dc
