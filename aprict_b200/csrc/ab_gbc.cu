// ab_gbc.cu -- the GBC reconstruction's device work: backprojection with the
// cylindrical-locus GBC weights into a volume and a weight-sum volume, the
// expected weight sum over a perfect cylindrical trajectory, the volume-domain
// cone-beam ramp filter's spectral multiplier, and the trilinear low-resolution
// correction.
//
// Reference: backproject_CB_voltex_GBC_cyl / _backproject_CB_getval_GBC_cyl /
// _GBC_weightfun / cossq_soft (src/aprict/data/cusrc/CB_backproject.cu:273-311,
// 736-905, 1030-1105), get_GBC_weight_integ (:1108-1168, driven by
// src/aprict/gbc/weightinteg.py:22-91), ramp_filter_conebeam and
// _conebeam_kfactor_unchunked (src/aprict/gbc/filters.py:59-147, 256-504).
//
// The backprojection launches once for all views (the reference: once per 10
// views, the volume read-modified-written each time). One thread per voxel,
// consecutive threads on consecutive voxels in memory order, per-view
// coefficients staged in shared memory. The weight is evaluated in FP32 from
// reciprocal square roots and one division (the angles' sines and cosines by
// trigonometric identities, the soft windows on squared sines), the detector coordinate
// by the same linear forms as the other backprojection modes, and the
// nearest-pixel choice re-decided in FP64 near ties, so the result follows
// the FP64 restatement. The spectral filter is one pass over the cuFFT
// spectrum with all per-frequency factors (ramp, 1 / k-factor, sinc
// corrections, DC) folded into one FP64 factor; the reference makes about
// ten array passes.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "ab_bpcol.cuh"

namespace {

constexpr int kGThreads = 256;
constexpr int kGChunk = 64;  // views per shared-memory chunk

// Soft window s(a, b; c) of cossq_soft (CB_backproject.cu:273-311): 0 beyond
// |c| = a, 1 inside |c| = a - b, 3x^2 - 2x^3 between, x = gamma sin|c| - chi,
// gamma = 1 / (sin(a - b) - sin a), chi = gamma sin a. Both angles the weight
// feeds it lie in [0, pi/2], where sin is increasing, so the window is taken
// as a function of s = sin|c| with the comparisons made on sines: no
// transcendental per voxel-view. The constants come from the host in FP64.
struct SoftWin {
    float sa2, sab2, gamma, chi;  // sin^2 a (4 if a >= pi/2), sin^2(a - b) (-1 if a - b <= 0, 4 if >= pi/2), gamma, chi
};

struct GbcSoft {
    SoftWin v, h;  // vertical (elevation) and horizontal windows
};

SoftWin soft_win(double a, double b) {
    const double half_pi = 1.5707963267948966;
    SoftWin w;
    w.sa2 = a >= half_pi ? 4.f : (float)(sin(a) * sin(a));
    w.sab2 = a - b <= 0.0 ? -1.f : (a - b >= half_pi ? 4.f : (float)(sin(a - b) * sin(a - b)));
    const double g = 1.0 / (sin(a - b) - sin(a));
    w.gamma = (float)g;
    w.chi = (float)(g * sin(a));
    return w;
}

// The soft band's cubic at s = sin|angle|.
__device__ __forceinline__ float soft_cubic(float s, const SoftWin &w) {
    const float x = w.gamma * s - w.chi;
    return fmaxf(0.f, fminf(1.f, 3.f * x * x - 2.f * x * x * x));
}

// The window at s = sqrt(s2), s = sin|angle| in [0, 1]: compared on squares,
// a square root only inside the soft band.
__device__ __forceinline__ float soft_of_sin2(float s2, const SoftWin &w) {
    if (s2 > w.sa2) return 0.f;
    if (s2 < w.sab2) return 1.f;
    return soft_cubic(sqrtf(s2), w);
}

// The same window when s itself is at hand (s2 = s * s): no square root.
__device__ __forceinline__ float soft_of_sin(float s, float s2, const SoftWin &w) {
    if (s2 > w.sa2) return 0.f;
    if (s2 < w.sab2) return 1.f;
    return soft_cubic(s, w);
}

// GBC weight (eq. 23 of the GBC method with the soft windows,
// CB_backproject.cu:736-787) of the voxel at world position p for the source
// at s (inv_ls = 1 / |(s_x, s_y)|), on a cylinder of radius R (inv_R = 1/R)
// about the world z axis. With r = p - s, q = r_x^2 + r_y^2:
//   ell = sqrt(q) / R, c = clamp(|Z / R / ell|) = clamp(|r . L| / (|L| sqrt(q))),
//   theta = atan2(r_z / R, ell): cos theta = ell / h, sin|theta| = |r_z / R| / h,
//   h = hypot(ell, r_z / R); phi = acos(c): sin^2 phi = 1 - c^2.
// Reciprocal square roots and one fast division, as the reference's
// fast-math build evaluates its transcendental form; the limits at q = 0 and
// h = 0 are the reference's (c = 1, cos theta = 1).
__device__ float gbc_weight(float inv_R, float px, float py, float pz, float sx, float sy, float sz, float inv_ls,
                            const GbcSoft &S) {
    const float rx = px - sx, ry = py - sy, rz = pz - sz;
    const float q = rx * rx + ry * ry;
    const float rq = rsqrtf(q);
    const float ell = q > 0.f ? q * rq * inv_R : 0.f;
    const float c = fmaxf(0.f, fminf(1.f, fabsf((rx * sx + ry * sy) * inv_ls * rq)));  // NaN at q = 0 -> 1
    const float d = c - ell;
    const float zr = rz * inv_R;
    const float h2 = ell * ell + zr * zr;
    const float ih = rsqrtf(h2);
    const float cos_el = h2 > 0.f ? ell * ih : 1.f;
    const float sin_el = h2 > 0.f ? fabsf(zr) * ih : 0.f;
    const float weight = __fdividef(cos_el * cos_el * cos_el * c, fmaxf(1e-9f, c * c + d * d));
    return weight * soft_of_sin(sin_el, sin_el * sin_el, S.v) * soft_of_sin2(fmaxf(0.f, 1.f - c * c), S.h);
}

struct GbcParams {
    float *vol2;  // weight-sum volume (same layout as the volume)
    float inv_R;  // 1 / R
    GbcSoft soft;
    float pos000[3];  // world centre of voxel (0, 0, 0): corner + voxwid / 2
};

// Resident CTAs per SM: the kernel is bound by the latency of its detector
// gathers, and at the unconstrained ~105 registers only 2 CTAs fit; a few
// registers spilled (view derivation, FP64 tie refinement) cost less than the
// lost occupancy (198^3 x 360 views: bilinear 22.7 -> 17.2 ms at 3 CTAs,
// nearest 19.7 -> 12.9 ms at 4).
template <bool BILIN>
__global__ void __launch_bounds__(kGThreads, BILIN ? 3 : 4) k_backproject_gbc(const ab_bp::BPParams P, const GbcParams G,
                                                               int order_f) {
    using namespace ab_bp;
    __shared__ ab_bpview sv[kGChunk];
    __shared__ ab_bpview_d svd[BILIN ? 1 : kGChunk];
    __shared__ float ssrc[kGChunk][4];  // source x, y, z, 1 / |(x, y)|
    if (P.views == (int)APRICT_VIEWS_UNKNOWN && P.col.gb[0] != 0 && all_upright(P)) return;  // k_backproject_gbc_columns'

    const int64_t nvox = (int64_t)P.n[0] * P.n[1] * P.n[2];
    const int64_t e = (int64_t)blockIdx.x * kGThreads + threadIdx.x;
    const bool live = e < nvox;
    int id[3];
    if (order_f) {  // x fastest
        id[0] = (int)(e % P.n[0]);
        id[1] = (int)((e / P.n[0]) % P.n[1]);
        id[2] = (int)(e / ((int64_t)P.n[0] * P.n[1]));
    } else {  // z fastest
        id[2] = (int)(e % P.n[2]);
        id[1] = (int)((e / P.n[2]) % P.n[1]);
        id[0] = (int)(e / ((int64_t)P.n[1] * P.n[2]));
    }
    const float vw = P.voxwid;
    const float offs[3] = {1.f / (float)P.ssx, 1.f / (float)P.ssy, 1.f / (float)P.ssz};
    const int n_sub = P.ssx * P.ssy * P.ssz;
    float acc = 0.f, acc2 = 0.f;

    for (uint32_t v0 = 0; v0 < P.n_views; v0 += kGChunk) {
        const int cn = (int)min((uint32_t)kGChunk, P.n_views - v0);
        __syncthreads();
        for (int t = threadIdx.x; t < cn; t += kGThreads) {
            const ab_d3 c0d{P.cornerd[0] + 0.5 * P.vwd * P.n[0], P.cornerd[1] + 0.5 * P.vwd * P.n[1],
                            P.cornerd[2] + 0.5 * P.vwd * P.n[2]};
            const aprict_proj_spec sp = P.specs[v0 + t];
            const double hext[3] = {(0.5 * P.n[0] + 1.0) * P.vwd, (0.5 * P.n[1] + 1.0) * P.vwd,
                                    (0.5 * P.n[2] + 1.0) * P.vwd};
            if (!ab_derive_bpview(sp, c0d, vw, 0.f, hext, sv[t], BILIN ? nullptr : &svd[t]) && P.status)
                atomicOr(P.status, APRICT_STATUS_BAD_GEOMETRY);
            ssrc[t][0] = sp.source_pos.x;
            ssrc[t][1] = sp.source_pos.y;
            ssrc[t][2] = sp.source_pos.z;
            ssrc[t][3] = rsqrtf(sp.source_pos.x * sp.source_pos.x + sp.source_pos.y * sp.source_pos.y);
        }
        __syncthreads();
        if (!live) continue;
        for (int isub = 0; isub < n_sub; ++isub) {
            const int sidx[3] = {isub / (P.ssy * P.ssz), (isub / P.ssz) % P.ssy, isub % P.ssz};
            float fsub[3], rel[3], wp[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                fsub[a] = -0.5f + offs[a] * (0.5f + (float)sidx[a]);  // sub_offset, contracted
                // relative to the volume centre, for the detector coordinate
                rel[a] = ((float)id[a] + 0.5f - 0.5f * (float)P.n[a]) * vw + fsub[a] * vw;
                // world position as the reference forms it (pos_000_c + idx voxwid + offset voxwid)
                wp[a] = (G.pos000[a] + (float)id[a] * vw) + fsub[a] * vw;
            }
            float s = 0.f, s2 = 0.f;
            for (int t = 0; t < cn; ++t) {
                const float w =
                    gbc_weight(G.inv_R, wp[0], wp[1], wp[2], ssrc[t][0], ssrc[t][1], ssrc[t][2], ssrc[t][3], G.soft);
                s2 += w;
                if (w == 0.f) continue;
                const ab_bpview &b = sv[t];
                const float rD = rcp_fast(dot4(b.den, rel[0], rel[1], rel[2]));
                const float fu = dot4(b.nu, rel[0], rel[1], rel[2]) * rD;
                const float fv = dot4(b.nv, rel[0], rel[1], rel[2]) * rD;
                const float *pvw = P.projs + (int64_t)(v0 + t) * P.stride_view;
                float pv;
                if (BILIN) {
                    pv = fetch_bilinear(P, pvw, fu, fv);
                } else {
                    float du, dv;
                    int iu = round_index(fu, -2.f, P.fnu1, du);
                    int iv = round_index(fv, -2.f, P.fnv1, dv);
                    const bool tu = fabsf(du) > b.tie_u, tv = fabsf(dv) > b.tie_v;
                    if (tu || tv) {
                        const VoxRef vr{((double)id[0] + 0.5 + (double)fsub[0] - 0.5 * P.n[0]) * P.vwd,
                                        ((double)id[1] + 0.5 + (double)fsub[1] - 0.5 * P.n[1]) * P.vwd,
                                        ((double)id[2] + 0.5 + (double)fsub[2] - 0.5 * P.n[2]) * P.vwd};
                        const ab_bpview_d &cd = svd[BILIN ? 0 : t];
                        if (tu) iu = refine_index(cd.nu, cd.den, vr, iu, du);
                        if (tv) iv = refine_index(cd.nv, cd.den, vr, iv, dv);
                    }
                    const bool inb = (unsigned)iu < P.nu && (unsigned)iv < P.nv;
                    pv = inb ? __ldg(pvw + (iu * P.su + iv * P.sv)) : 0.f;
                }
                s = fmaf(pv, w, s);
            }
            acc += s;
            acc2 += s2;
        }
    }
    if (!live) return;
    const float value = n_sub == 1 ? acc : acc / (float)n_sub;
    const float value2 = n_sub == 1 ? acc2 : acc2 / (float)n_sub;
    if (value == 0.f && value2 == 0.f) return;  // the reference writes neither (:1068-1075)
    const int64_t o = (int64_t)id[0] * P.vs[0] + (int64_t)id[1] * P.vs[1] + (int64_t)id[2] * P.vs[2];
    const float m = P.mult ? P.mult[o] : 1.f;
    if (value != 0.f) P.vol[o] = value * m + P.vol[o];
    if (value2 != 0.f) G.vol2[o] = value2 * m + G.vol2[o];
}

// Z-column layout for C-order volumes: the 32 lanes of a warp and each
// thread's kGZ voxels lie along z (voxel k of a lane 32 k further), warps
// along y, one x layer per CTA. For a view whose detector u axis and normal
// have no z component (the GBC's cylindrical scans) the thread's voxels share
// x and y, and with them everything horizontal: the depth and its
// reciprocal, u (the pixel column or the bilinear columns and their weight),
// the horizontal distance ell, the horizontal angle's cosine c, its window,
// and the weight's factor c / max(1e-9, c^2 + (c - ell)^2). Per voxel only
// the elevation (its cosine cubed and window) and v remain. Other views take
// the per-voxel formulas of k_backproject_gbc.
constexpr int kGZ = 4;

template <bool BILIN>
__global__ void __launch_bounds__(kGThreads, BILIN ? 3 : 4) k_backproject_gbc_z(const ab_bp::BPParams P, const GbcParams G,
                                                                 int gb0, int gb1) {
    using namespace ab_bp;
    __shared__ ab_bpview sv[kGChunk];
    __shared__ ab_bpview_d svd[BILIN ? 1 : kGChunk];
    __shared__ float ssrc[kGChunk][4];  // source x, y, z, 1 / |(x, y)|
    __shared__ uint8_t szinv[kGChunk];
    if (P.views == (int)APRICT_VIEWS_UNKNOWN && P.col.gb[0] != 0 && all_upright(P)) return;  // k_backproject_gbc_columns'

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b0 = (int)(blockIdx.x % (unsigned)gb0), b1 = (int)((blockIdx.x / (unsigned)gb0) % (unsigned)gb1);
    const int ix = (int)(blockIdx.x / ((unsigned)gb0 * (unsigned)gb1));
    const int iy = b1 * 8 + warp, iz0 = b0 * 32 * kGZ + lane;
    const bool col_live = iy < P.n[1];
    bool live[kGZ];
#pragma unroll
    for (int k = 0; k < kGZ; ++k) live[k] = col_live && iz0 + 32 * k < P.n[2];
    const float vw = P.voxwid;
    const float offs[3] = {1.f / (float)P.ssx, 1.f / (float)P.ssy, 1.f / (float)P.ssz};
    const int n_sub = P.ssx * P.ssy * P.ssz;
    float acc[kGZ], acc2[kGZ];
#pragma unroll
    for (int k = 0; k < kGZ; ++k) acc[k] = acc2[k] = 0.f;

    for (uint32_t v0 = 0; v0 < P.n_views; v0 += kGChunk) {
        const int cn = (int)min((uint32_t)kGChunk, P.n_views - v0);
        __syncthreads();
        for (int t = threadIdx.x; t < cn; t += kGThreads) {
            const ab_d3 c0d{P.cornerd[0] + 0.5 * P.vwd * P.n[0], P.cornerd[1] + 0.5 * P.vwd * P.n[1],
                            P.cornerd[2] + 0.5 * P.vwd * P.n[2]};
            const aprict_proj_spec sp = P.specs[v0 + t];
            const double hext[3] = {(0.5 * P.n[0] + 1.0) * P.vwd, (0.5 * P.n[1] + 1.0) * P.vwd,
                                    (0.5 * P.n[2] + 1.0) * P.vwd};
            if (!ab_derive_bpview(sp, c0d, vw, 0.f, hext, sv[t], BILIN ? nullptr : &svd[t]) && P.status)
                atomicOr(P.status, APRICT_STATUS_BAD_GEOMETRY);
            ssrc[t][0] = sp.source_pos.x;
            ssrc[t][1] = sp.source_pos.y;
            ssrc[t][2] = sp.source_pos.z;
            ssrc[t][3] = rsqrtf(sp.source_pos.x * sp.source_pos.x + sp.source_pos.y * sp.source_pos.y);
            const ab_bpview &bt = sv[t];
            szinv[t] = (uint8_t)(bt.den.z == 0.f && bt.nu.z == 0.f && (BILIN || (svd[t].nu[2] == 0.0 && svd[t].den[2] == 0.0)));
        }
        __syncthreads();
        if (!__any_sync(0xffffffffu, col_live && live[0])) continue;  // warp-uniform
        for (int isub = 0; isub < n_sub; ++isub) {
            const int sidx[3] = {isub / (P.ssy * P.ssz), (isub / P.ssz) % P.ssy, isub % P.ssz};
            float fsub[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) fsub[a] = -0.5f + offs[a] * (0.5f + (float)sidx[a]);  // sub_offset, contracted
            const int idv[2] = {ix, iy};
            float rel[2], wp[2];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                rel[a] = ((float)idv[a] + 0.5f - 0.5f * (float)P.n[a]) * vw + fsub[a] * vw;
                wp[a] = (G.pos000[a] + (float)idv[a] * vw) + fsub[a] * vw;
            }
            float relz[kGZ], wpz[kGZ];
#pragma unroll
            for (int k = 0; k < kGZ; ++k) {
                const int iz = iz0 + 32 * k;
                relz[k] = ((float)iz + 0.5f - 0.5f * (float)P.n[2]) * vw + fsub[2] * vw;
                wpz[k] = (G.pos000[2] + (float)iz * vw) + fsub[2] * vw;
            }
            float s[kGZ], s2[kGZ];
#pragma unroll
            for (int k = 0; k < kGZ; ++k) s[k] = s2[k] = 0.f;
            for (int t = 0; t < cn; ++t) {
                const ab_bpview &b = sv[t];
                const float sx = ssrc[t][0], sy = ssrc[t][1], sz = ssrc[t][2], inv_ls = ssrc[t][3];
                const float *pvw = P.projs + (int64_t)(v0 + t) * P.stride_view;
                if (szinv[t]) {
                    // horizontal: shared by the thread's voxels
                    const float rx = wp[0] - sx, ry = wp[1] - sy;
                    const float q = rx * rx + ry * ry;
                    const float rq = rsqrtf(q);
                    const float ell = q > 0.f ? q * rq * G.inv_R : 0.f;
                    const float c = fmaxf(0.f, fminf(1.f, fabsf((rx * sx + ry * sy) * inv_ls * rq)));
                    const float d = c - ell;
                    const float ac = __fdividef(c, fmaxf(1e-9f, c * c + d * d)) *
                                     soft_of_sin2(fmaxf(0.f, 1.f - c * c), G.soft.h);
                    const float rD = rcp_fast(dot4(b.den, rel[0], rel[1], relz[0]));
                    const float fu = dot4(b.nu, rel[0], rel[1], relz[0]) * rD;
                    // u: the pixel column (nearest) or the two columns and their weight (bilinear)
                    int iu = -1, i0 = 0;
                    float fx = 0.f;
                    bool ucol = false;
                    if (BILIN) {
                        ucol = !(fu <= -1.f || fu >= (float)P.nu);
                        i0 = (int)floorf(fu);
                        fx = fu - (float)i0;
                    } else {
                        float du;
                        iu = round_index(fu, -2.f, P.fnu1, du);
                        if (fabsf(du) > b.tie_u) {
                            const VoxRef vr{((double)ix + 0.5 + (double)fsub[0] - 0.5 * P.n[0]) * P.vwd,
                                            ((double)iy + 0.5 + (double)fsub[1] - 0.5 * P.n[1]) * P.vwd, 0.0};
                            iu = refine_index(svd[BILIN ? 0 : t].nu, svd[BILIN ? 0 : t].den, vr, iu, du);
                        }
                        ucol = (unsigned)iu < P.nu;
                    }
#pragma unroll
                    for (int k = 0; k < kGZ; ++k) {
                        const float zr = (wpz[k] - sz) * G.inv_R;
                        const float h2 = ell * ell + zr * zr;
                        const float ih = rsqrtf(h2);
                        const float cos_el = h2 > 0.f ? ell * ih : 1.f;
                        const float sin_el = h2 > 0.f ? fabsf(zr) * ih : 0.f;
                        const float w = cos_el * cos_el * cos_el * ac * soft_of_sin(sin_el, sin_el * sin_el, G.soft.v);
                        s2[k] += w;
                        if (w == 0.f || !ucol) continue;
                        const float fv = dot4(b.nv, rel[0], rel[1], relz[k]) * rD;
                        float pv;
                        if (BILIN) {
                            if (fv <= -1.f || fv >= (float)P.nv) continue;
                            const int j0 = (int)floorf(fv);
                            const float fy = fv - (float)j0;
                            auto get = [&](int i, int j) -> float {
                                if (i < 0 || i >= (int)P.nu || j < 0 || j >= (int)P.nv) return 0.f;
                                return __ldg(pvw + (i * P.su + j * P.sv));
                            };
                            const float v00 = get(i0, j0), v01 = get(i0, j0 + 1), v10 = get(i0 + 1, j0),
                                        v11 = get(i0 + 1, j0 + 1);
                            const float t1 = v00 * (1.f - fx) + v10 * fx;
                            const float t2 = v01 * (1.f - fx) + v11 * fx;
                            pv = t1 * (1.f - fy) + t2 * fy;
                        } else {
                            float dv;
                            int iv = round_index(fv, -2.f, P.fnv1, dv);
                            if (fabsf(dv) > b.tie_v) {
                                const VoxRef vr{((double)ix + 0.5 + (double)fsub[0] - 0.5 * P.n[0]) * P.vwd,
                                                ((double)iy + 0.5 + (double)fsub[1] - 0.5 * P.n[1]) * P.vwd,
                                                ((double)(iz0 + 32 * k) + 0.5 + (double)fsub[2] - 0.5 * P.n[2]) *
                                                    P.vwd};
                                iv = refine_index(svd[BILIN ? 0 : t].nv, svd[BILIN ? 0 : t].den, vr, iv, dv);
                            }
                            pv = (unsigned)iv < P.nv ? __ldg(pvw + (iu * P.su + iv * P.sv)) : 0.f;
                        }
                        s[k] = fmaf(pv, w, s[k]);
                    }
                } else {
#pragma unroll
                    for (int k = 0; k < kGZ; ++k) {
                        const float w = gbc_weight(G.inv_R, wp[0], wp[1], wpz[k], sx, sy, sz, inv_ls, G.soft);
                        s2[k] += w;
                        if (w == 0.f) continue;
                        const float rD = rcp_fast(dot4(b.den, rel[0], rel[1], relz[k]));
                        const float fu = dot4(b.nu, rel[0], rel[1], relz[k]) * rD;
                        const float fv = dot4(b.nv, rel[0], rel[1], relz[k]) * rD;
                        float pv;
                        if (BILIN) {
                            pv = fetch_bilinear(P, pvw, fu, fv);
                        } else {
                            float du, dv;
                            int iu = round_index(fu, -2.f, P.fnu1, du);
                            int iv = round_index(fv, -2.f, P.fnv1, dv);
                            const bool tu = fabsf(du) > b.tie_u, tv = fabsf(dv) > b.tie_v;
                            if (tu || tv) {
                                const VoxRef vr{((double)ix + 0.5 + (double)fsub[0] - 0.5 * P.n[0]) * P.vwd,
                                                ((double)iy + 0.5 + (double)fsub[1] - 0.5 * P.n[1]) * P.vwd,
                                                ((double)(iz0 + 32 * k) + 0.5 + (double)fsub[2] - 0.5 * P.n[2]) *
                                                    P.vwd};
                                const ab_bpview_d &cd = svd[BILIN ? 0 : t];
                                if (tu) iu = refine_index(cd.nu, cd.den, vr, iu, du);
                                if (tv) iv = refine_index(cd.nv, cd.den, vr, iv, dv);
                            }
                            const bool inb = (unsigned)iu < P.nu && (unsigned)iv < P.nv;
                            pv = inb ? __ldg(pvw + (iu * P.su + iv * P.sv)) : 0.f;
                        }
                        s[k] = fmaf(pv, w, s[k]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kGZ; ++k) {
                acc[k] += s[k];
                acc2[k] += s2[k];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kGZ; ++k) {
        if (!live[k]) continue;
        const float value = n_sub == 1 ? acc[k] : acc[k] / (float)n_sub;
        const float value2 = n_sub == 1 ? acc2[k] : acc2[k] / (float)n_sub;
        if (value == 0.f && value2 == 0.f) continue;  // the reference writes neither (:1068-1075)
        const int64_t o = (int64_t)ix * P.vs[0] + (int64_t)iy * P.vs[1] + (int64_t)(iz0 + 32 * k) * P.vs[2];
        const float m = P.mult ? P.mult[o] : 1.f;
        if (value != 0.f) P.vol[o] = value * m + P.vol[o];
        if (value2 != 0.f) G.vol2[o] = value2 * m + G.vol2[o];
    }
}

// Upright views into z columns (ab_bpcol.cuh's layout and per-warp table): one
// lane per view evaluates in FP64 the column's u, the row coordinate f = A + n S
// and, once per column and view, everything horizontal of the weight
// (k_backproject_gbc_z's factor times ell^3), and sorts the column's blocks of
// 32 voxels: inside the vertical window's flat part and on the detector
// (fast), past the window (weight 0: skipped) or neither. A fast voxel-view
// is then ell^3 A / h^3 from one reciprocal square root, the row, the gathers
// and two fmas, on pairs of voxels. Measured, 198^3 x 360 views x 256^2
// bilinear: 13.0 ms (k_backproject_gbc_z) -> 5.6 ms, 4.7e9 warp instructions against
// 1.2e10, at 4 CTAs per SM (64 registers; 6.4 ms at 3, 7.9 ms at 2; 7.8 ms at 3 with
// the window's band left to the per-voxel branch).
struct GbcView {
    ab_bpview_d d;
    float sx, sy, sz, inv_ls;  // source, 1 / |(sx, sy)|
    int ok;
    int pad;
};
static_assert(sizeof(GbcView) % 16 == 8, "an odd number of 8-byte words (see ColView)");

struct GbcRec {
    float4 a;  // A, S, fx (bilinear) or trust threshold (nearest), factor times ell^3
    uint4 b;   // column address (lo, hi), block masks (fast | weight not 0 << 8 | on detector << 16 | inside
               // it << 24), columns on the detector
    float4 c;  // ell^2, (z_0 - s_z) / R, factor, unused
};

constexpr int kGCol = 8;  // voxels per thread

struct GbcColSmem {
    GbcView view[kGChunk];
    GbcRec rec[kGThreads / 32][32];
    float vol[kGThreads / 32][32 * kGCol], wsum[kGThreads / 32][32 * kGCol];
    double pos[kGThreads / 32][4];  // the warp's column, as ColSmem's
};

template <bool BILIN>
__global__ void __launch_bounds__(kGThreads, 4) k_backproject_gbc_columns(const ab_bp::BPParams P, const GbcParams G,
                                                                          float tan_flat, float tan_zero, int clamped) {
    using namespace ab_bp;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    GbcColSmem &sm = *reinterpret_cast<GbcColSmem *>(smem_raw);
    if (!all_upright(P)) return;  // the other kernels'
    int b0, b1, b2;
    if (!brick_coords(P.col, blockIdx.x, b0, b1, b2)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ix = b2, iy = b1 * 8 + warp, z0 = b0 * 32 * kGCol;
    const bool col_live = iy < P.n[1];
    const int nb = min(kGCol, (P.n[2] - z0 + 31) / 32);
    const unsigned blocks = (1u << nb) - 1u, pairs = (1u << ((nb + 1) & ~1)) - 1u;
    float *tv = sm.vol[warp], *tw = sm.wsum[warp];
#pragma unroll
    for (int k = 0; k < kGCol; ++k) tv[lane + 32 * k] = tw[lane + 32 * k] = 0.f;
    const int crow = (int)(P.nv >> 1);
    const float coff = 0.5f * ((float)P.nv - 1.f) - (float)crow;
    const float halfv = 0.5f * (float)P.nv;
    const float insidev = BILIN ? halfv - 0.5f : halfv, offv = BILIN ? halfv + 0.5f : halfv;
    const uint32_t sv4 = 4u * (uint32_t)P.sv, su4 = 4u * (uint32_t)P.su;
    const f32x2 magic = pk(kMagic, kMagic), nmagic = pk(-kMagic, -kMagic), minus1 = pk(-1.f, -1.f), one = pk(1.f, 1.f),
                mhalf = pk(-0.5f, -0.5f);
    const float dzR = P.voxwid * G.inv_R, s32z = 32.f * dzR;
    const int n_sub = P.ssx * P.ssy * P.ssz;

    for (int isub = 0; isub < n_sub; ++isub) {
        const float ox = sub_offset(1.f / (float)P.ssx, isub / (P.ssy * P.ssz));
        const float oy = sub_offset(1.f / (float)P.ssy, (isub / P.ssz) % P.ssy);
        const float oz = sub_offset(1.f / (float)P.ssz, isub % P.ssz);
        if (lane == 0) {
            sm.pos[warp][0] = (ix + 0.5 + ox - 0.5 * P.n[0]) * P.vwd;
            sm.pos[warp][1] = (iy + 0.5 + oy - 0.5 * P.n[1]) * P.vwd;
            sm.pos[warp][2] = z0 + 0.5 + oz - 0.5 * P.n[2];
        }
        // world position of the column's first voxel
        const float wx = (G.pos000[0] + (float)ix * P.voxwid) + ox * P.voxwid;
        const float wy = (G.pos000[1] + (float)iy * P.voxwid) + oy * P.voxwid;
        const float wz = (G.pos000[2] + (float)z0 * P.voxwid) + oz * P.voxwid;
        for (uint32_t v0 = 0; v0 < P.n_views; v0 += kGChunk) {
            const int cn = (int)min((uint32_t)kGChunk, P.n_views - v0);
            __syncthreads();
            if ((int)threadIdx.x < cn) {
                const ab_d3 c0d{P.cornerd[0] + 0.5 * P.vwd * P.n[0], P.cornerd[1] + 0.5 * P.vwd * P.n[1],
                                P.cornerd[2] + 0.5 * P.vwd * P.n[2]};
                const aprict_proj_spec sp = P.specs[v0 + threadIdx.x];
                GbcView &gv = sm.view[threadIdx.x];
                double Dn, uu, vv;
                ab_d3 Ps, c0s;
                gv.ok = derive_upright(sp, c0d, gv.d, Dn, uu, vv, Ps, c0s);
                if (!gv.ok && P.status) atomicOr(P.status, APRICT_STATUS_BAD_GEOMETRY);
                gv.sx = sp.source_pos.x;
                gv.sy = sp.source_pos.y;
                gv.sz = sp.source_pos.z;
                gv.inv_ls = rsqrtf(gv.sx * gv.sx + gv.sy * gv.sy);
            }
            __syncthreads();
            if (!col_live) continue;  // warp-uniform
            f32x2 acc2[kGCol / 2], accw2[kGCol / 2];
#pragma unroll
            for (int k = 0; k < kGCol / 2; ++k) acc2[k] = accw2[k] = pk(0.f, 0.f);
            for (int g0 = 0; g0 < cn; g0 += 32) {
                __syncwarp();
                {
                    const int t = g0 + lane;
                    GbcRec rec;
                    rec.a = make_float4(0.f, 0.f, 0.f, 0.f);
                    rec.b = make_uint4(0u, 0u, 0u, 0u);
                    rec.c = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (t < cn) {
                        const GbcView &gv = sm.view[t];
                        // horizontal part of the weight, as k_backproject_gbc_z
                        const float rx = wx - gv.sx, ry = wy - gv.sy;
                        const float q = rx * rx + ry * ry;
                        const float rq = rsqrtf(q);
                        const float ell = q > 0.f ? q * rq * G.inv_R : 0.f;
                        const float c = fmaxf(0.f, fminf(1.f, fabsf((rx * gv.sx + ry * gv.sy) * gv.inv_ls * rq)));
                        const float d = c - ell;
                        const float ac = __fdividef(c, fmaxf(1e-9f, c * c + d * d)) *
                                         soft_of_sin2(fmaxf(0.f, 1.f - c * c), G.soft.h);
                        const float zr0 = (wz - gv.sz) * G.inv_R;
                        if (ac != 0.f) {
                            // the blocks' part of the vertical window: |z - s_z| / R against ell tan(angle)
                            unsigned flat = 0, past = 0;
#pragma unroll
                            for (int k = 0; k < kGCol; ++k) {
                                const float e0 = fmaf((float)(32 * k), dzR, zr0), e1 = fmaf((float)(32 * k + 31), dzR, zr0);
                                if (fmaxf(fabsf(e0), fabsf(e1)) < ell * tan_flat) flat |= 1u << k;
                                if (fminf(fabsf(e0), fabsf(e1)) > ell * tan_zero && (e0 > 0.f) == (e1 > 0.f)) past |= 1u << k;
                            }
                            unsigned in = 0, across = 0, cols = 0;
                            float Af = 0.f, Sf = 0.f, du = 0.f, eps = 0.f;
                            uint64_t col = 0;
                            const double X = sm.pos[warp][0], Y = sm.pos[warp][1], Z0 = sm.pos[warp][2] * P.vwd;
                            const double D = fma(gv.d.den[0], X, fma(gv.d.den[1], Y, gv.d.den[3]));
                            const double rD = 1.0 / D;
                            const double fu = fma(gv.d.nu[0], X, fma(gv.d.nu[1], Y, gv.d.nu[3])) * rD;
                            if (gv.ok && fabs(fu) < 4194304.0) {
                                int iu = BILIN ? __double2int_rd(fu) : __double2int_rn(fu);
                                du = (float)(fu - (double)iu);
                                if (!BILIN && fabsf(du) > 0.499f)
                                    iu = refine_index(gv.d.nu, gv.d.den, VoxRef{X, Y, 0.0}, iu, du);
                                if (BILIN ? fu > -1.0 && iu < (int)P.nu : (unsigned)iu < P.nu) {
                                    Af = (float)(fma(gv.d.nv[0], X, fma(gv.d.nv[1], Y, fma(gv.d.nv[2], Z0, gv.d.nv[3]))) * rD -
                                                 (double)crow);
                                    Sf = (float)(gv.d.nv[2] * P.vwd * rD);
                                    eps = fmaf(1.5f * 5.9604645e-8f,
                                               3.f * fabsf(Af) + (3.f * 32 * kGCol) * fabsf(Sf) + (float)P.nv, 1e-6f);
#pragma unroll
                                    for (int k = 0; k < kGCol; ++k) {
                                        const float e0 = fmaf((float)(32 * k), Sf, Af) - coff;
                                        const float e1 = fmaf((float)(32 * k + 31), Sf, Af) - coff;
                                        const float lo = fminf(e0, e1), hi = fmaxf(e0, e1);
                                        if (lo - eps >= -insidev && hi + eps <= insidev)
                                            in |= 1u << k;
                                        else if (!(lo - eps > offv || hi + eps < -offv))
                                            across |= 1u << k;
                                    }
                                    cols = 3u;
                                    if (BILIN && (iu < 0 || iu + 1 >= (int)P.nu)) {
                                        cols = (iu >= 0 ? 1u : 0u) | (iu + 1 < (int)P.nu ? 2u : 0u);
                                        across |= in;
                                        in = 0u;
                                    }
                                    col = (uint64_t)(uintptr_t)(P.projs + (int64_t)(v0 + t) * P.stride_view +
                                                                (int64_t)iu * P.su + (int64_t)crow * P.sv) -
                                          4ull * 0x4B400000ull * (uint64_t)(uint32_t)P.sv;
                                }
                            }
                            const unsigned fast = in & flat & pairs, partly = blocks & ~past;
                            rec.a = make_float4(Af, Sf, BILIN ? du : 0.5f - eps, ac * (ell * ell * ell));
                            rec.b = make_uint4((uint32_t)col, (uint32_t)(col >> 32),
                                               fast | partly << 8 | (in | across) << 16 | (in & pairs) << 24, cols);
                            rec.c = make_float4(ell * ell, zr0, ac, 0.f);
                        }
                    }
                    sm.rec[warp][lane] = rec;
                }
                __syncwarp();
                const int gn = min(32, cn - g0);
                for (int j = 0; j < gn; ++j) {
                    const GbcRec &rc = sm.rec[warp][j];
                    const uint4 rb = rc.b;
                    if ((rb.z & 0xffffu) == 0u) continue;  // weight 0 (warp-uniform)
                    const float4 ra = rc.a, rcc = rc.c;
                    const uint64_t col = ((uint64_t)rb.y << 32) | rb.x, col1 = col + su4;
                    const float a = fmaf((float)lane, ra.y, ra.x), s32 = 32.f * ra.y;
                    const float zl = fmaf((float)lane, dzR, rcc.y);
                    const f32x2 f0 = pk(a, a + s32), s2 = pk(s32, s32), zr0 = pk(zl, zl + s32z), sz2 = pk(s32z, s32z);
                    const f32x2 e2 = pk(rcc.x, rcc.x), ae2 = pk(ra.w, ra.w), fx2 = pk(ra.z, ra.z), gx2 = pk(1.f - ra.z, 1.f - ra.z);
                    auto fast_pair = [&](int k, bool windowed) {
                        const f32x2 f = k == 0 ? f0 : fma2(pk(2.f * k, 2.f * k), s2, f0);
                        const f32x2 zr = k == 0 ? zr0 : fma2(pk(2.f * k, 2.f * k), sz2, zr0);
                        f32x2 pv;
                        float ta, tb;
                        if constexpr (BILIN) {
                            const f32x2 t = add2(add2(f, mhalf), magic);
                            const f32x2 fy = fma2(add2(t, nmagic), minus1, f);
                            upk(t, ta, tb);
                            const char *pa = reinterpret_cast<const char *>(col + (uint64_t)(uint32_t)__float_as_int(ta) * sv4);
                            const char *pb = reinterpret_cast<const char *>(col + (uint64_t)(uint32_t)__float_as_int(tb) * sv4);
                            const char *qa = reinterpret_cast<const char *>(col1 + (uint64_t)(uint32_t)__float_as_int(ta) * sv4);
                            const char *qb = reinterpret_cast<const char *>(col1 + (uint64_t)(uint32_t)__float_as_int(tb) * sv4);
                            auto at = [](const char *p, int o) { return __ldg(reinterpret_cast<const float *>(p) + o); };
                            const f32x2 v00 = pk(at(pa, 0), at(pb, 0)), v01 = pk(at(pa, 1), at(pb, 1));
                            const f32x2 v10 = pk(at(qa, 0), at(qb, 0)), v11 = pk(at(qa, 1), at(qb, 1));
                            const f32x2 t1 = fma2(v10, fx2, mul2(v00, gx2)), t2 = fma2(v11, fx2, mul2(v01, gx2));
                            pv = fma2(t2, fy, mul2(t1, fma2(fy, minus1, one)));
                        } else {
                            const f32x2 t = add2(f, magic);
                            const f32x2 d = fma2(add2(t, nmagic), minus1, f);
                            float da, db, fa, fb;
                            upk(t, ta, tb);
                            upk(d, da, db);
                            float pa = __ldg(reinterpret_cast<const float *>(col + (uint64_t)(uint32_t)__float_as_int(ta) * sv4));
                            float pb = __ldg(reinterpret_cast<const float *>(col + (uint64_t)(uint32_t)__float_as_int(tb) * sv4));
                            if (fmaxf(fabsf(da), fabsf(db)) > ra.z) {
                                upk(f, fa, fb);
                                const ab_bpview_d &vd = sm.view[g0 + j].d;
                                const double X = sm.pos[warp][0], Y = sm.pos[warp][1], zi0 = sm.pos[warp][2];
                                if (fabsf(da) > ra.z)
                                    pa = col_exact_row(vd, X, Y, (zi0 + (double)(lane + 64 * k)) * P.vwd, fa, crow, (int)P.nv, col, sv4);
                                if (fabsf(db) > ra.z)
                                    pb = col_exact_row(vd, X, Y, (zi0 + (double)(lane + 64 * k + 32)) * P.vwd, fb, crow, (int)P.nv,
                                                       col, sv4);
                            }
                            pv = pk(pa, pb);
                        }
                        float ha, hb;
                        upk(fma2(zr, zr, e2), ha, hb);
                        const f32x2 ih = pk(rsqrtf(ha), rsqrtf(hb));
                        f32x2 w = mul2(mul2(ih, ih), mul2(ih, ae2));
                        if (windowed) {  // soft_cubic with its argument clamped to [0, 1]: the whole window
                            float za, zb, ia, ib;
                            upk(zr, za, zb);
                            upk(ih, ia, ib);
                            const f32x2 x = pk(__saturatef(fmaf(G.soft.v.gamma, fabsf(za) * ia, -G.soft.v.chi)),
                                               __saturatef(fmaf(G.soft.v.gamma, fabsf(zb) * ib, -G.soft.v.chi)));
                            w = mul2(w, mul2(mul2(x, x), fma2(x, pk(-2.f, -2.f), pk(3.f, 3.f))));
                            // past the window nothing is sampled: 0 times an infinite pixel is no 0
                            float wa, wb, sa, sb;
                            upk(w, wa, wb);
                            upk(pv, sa, sb);
                            pv = pk(wa == 0.f ? 0.f : sa, wb == 0.f ? 0.f : sb);
                        }
                        accw2[k] = add2(accw2[k], w);
                        acc2[k] = fma2(pv, w, acc2[k]);
                    };
                    // one block in the window's band or across the detector's edge: weight and sample
                    auto slow_block = [&](int k, float &w, float &pv) {
                        w = pv = 0.f;
                        if (!(rb.z >> (8 + k) & 1u) || z0 + lane + 32 * k >= P.n[2]) return;
                        const float zr = fmaf((float)(32 * k), dzR, zl);
                        const float h2 = fmaf(zr, zr, rcc.x);
                        const float ih = rsqrtf(h2);
                        const float sin_el = h2 > 0.f ? fabsf(zr) * ih : 0.f;
                        w = (h2 > 0.f ? ra.w * (ih * ih * ih) : rcc.z) * soft_of_sin(sin_el, sin_el * sin_el, G.soft.v);
                        if (w == 0.f || !(rb.z >> (16 + k) & 1u)) return;
                        const float fo = (k & 1) ? a + s32 : a;
                        const float f = fminf(fmaxf(k < 2 ? fo : fmaf((float)(k & ~1), s32, fo), -2097152.f), 2097152.f);
                        if constexpr (BILIN) {
                            const float fl = floorf(f), fy = f - fl;
                            const int j0 = (int)fl + crow;
                            const float *p = reinterpret_cast<const float *>(col + 4ull * 0x4B400000ull) + (j0 - crow);
                            const bool r0 = (unsigned)j0 < P.nv, r1 = (unsigned)(j0 + 1) < P.nv, c0 = rb.w & 1u, c1 = rb.w & 2u;
                            const float v00 = r0 && c0 ? __ldg(p) : 0.f, v01 = r1 && c0 ? __ldg(p + 1) : 0.f;
                            const float v10 = r0 && c1 ? __ldg(p + P.su) : 0.f, v11 = r1 && c1 ? __ldg(p + P.su + 1) : 0.f;
                            const float t1 = v00 * (1.f - ra.z) + v10 * ra.z, t2 = v01 * (1.f - ra.z) + v11 * ra.z;
                            pv = t1 * (1.f - fy) + t2 * fy;
                        } else {
                            const float t = __fadd_rn(f, kMagic);
                            if (fabsf(__fsub_rn(f, __fsub_rn(t, kMagic))) > ra.z)
                                pv = col_exact_row(sm.view[g0 + j].d, sm.pos[warp][0], sm.pos[warp][1],
                                                   (sm.pos[warp][2] + (double)(lane + 32 * k)) * P.vwd, f, crow, (int)P.nv, col, sv4);
                            else if ((unsigned)(__float_as_int(t) - 0x4B400000 + crow) < P.nv)
                                pv = __ldg(reinterpret_cast<const float *>(col + (uint64_t)(uint32_t)__float_as_int(t) * sv4));
                        }
                    };
#pragma unroll
                    for (int k = 0; k < kGCol / 2; ++k) {  // warp-uniform branches
                        if ((rb.z >> (2 * k) & 3u) == 3u) {
                            fast_pair(k, false);
                        } else if (clamped && (rb.z >> (24 + 2 * k) & 3u) == 3u) {
                            if (rb.z >> (8 + 2 * k) & 3u) fast_pair(k, true);
                        } else if (rb.z >> (8 + 2 * k) & 3u) {
                            float wa, wb, pa, pb;
                            slow_block(2 * k, wa, pa);
                            slow_block(2 * k + 1, wb, pb);
                            const f32x2 w = pk(wa, wb);
                            accw2[k] = add2(accw2[k], w);
                            acc2[k] = fma2(pk(pa, pb), w, acc2[k]);
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kGCol / 2; ++k) {
                float a, b, wa, wb;
                upk(acc2[k], a, b);
                upk(accw2[k], wa, wb);
                tv[lane + 64 * k] += a;
                tv[lane + 64 * k + 32] += b;
                tw[lane + 64 * k] += wa;
                tw[lane + 64 * k + 32] += wb;
            }
        }
    }
    if (!col_live) return;
#pragma unroll
    for (int k = 0; k < kGCol; ++k) {
        const int i = lane + 32 * k;
        if (z0 + i >= P.n[2]) continue;
        const float value = n_sub == 1 ? tv[i] : tv[i] / (float)n_sub;
        const float value2 = n_sub == 1 ? tw[i] : tw[i] / (float)n_sub;
        if (value == 0.f && value2 == 0.f) continue;  // the reference writes neither (:1068-1075)
        const int64_t o = (int64_t)ix * P.vs[0] + (int64_t)iy * P.vs[1] + (int64_t)(z0 + i) * P.vs[2];
        const float m = P.mult ? P.mult[o] : 1.f;
        if (value != 0.f) P.vol[o] = value * m + P.vol[o];
        if (value2 != 0.f) G.vol2[o] = value2 * m + G.vol2[o];
    }
}

// Expected GBC weight sum at radius r (units of R) over a perfect cylindrical
// source locus: sum over num_z heights z in [0, tan(vartheta_v) (1 + r_max)]
// (the first with weight 1/2) and num_ang source angles t in [0, pi) of the
// weight of the voxel (r, 0, 0) for the source (cos t, sin t, z), times
// 4 z_max pi / (num_z num_ang) (get_GBC_weight_integ, CB_backproject.cu:1108-1168).
//
// The weight factorises: with the voxel at (r, 0, 0) and the source at
// (cos t, sin t, z), ell and the horizontal angle depend on (r, t) only, so
//   w(r, t, z) = A(r, t) cos^3(theta) s_v(sin^2 theta),
//   A = c / max(1e-9, c^2 + (c - ell)^2) s_h(1 - c^2),
//   cos theta = ell / h, sin^2 theta = z^2 / h^2, h^2 = ell^2 + z^2.
// The inner sum over heights is a function F of ell alone, smooth on the scale
// of ell, so it is evaluated at kNodes values of ell over the call's range
// (k_gbc_height_table, one warp each, the samples and weights of the rule) and
// taken by four-point Lagrange interpolation for each (radius, angle): 4096
// height sums instead of n_r num_ang of them (396 x 6000: 2.4 million).
// Interpolation error, relative to F, node spacing h: (h / ell)^4 from the
// smooth part, below 4e-9 where ell >= 128 h; and from the window, whose second
// derivative jumps at its two edges. A sample whose edge lies within a node of ell
// is off by a share of gamma^2 (h / ell)^2, and of the N = ell (num_z - 1) /
// (1 + r_max) samples in the window there are about N h / ell of them, at least
// one now and then:
//   error <= 0.06 gamma^2 (h / ell)^2 max(h / ell, 1 / N)
// (the rule in FP64 over window angles 0.1 .. 1, r_max 0.3 .. 1.1, gamma 5 .. 193, 100 ..
// 6000 heights: 0.045 at most). Where that exceeds kTol, a third of the samples'
// FP32 rounding, and below 128 h, the heights are summed directly, as in calls
// without scratch for the table.
// 396 radii x 6000 x 6000 samples, the whole call: 7.0 -> 0.53-0.68 ms (most of it host
// work; sums equal to 1e-8).
// sin^2 theta grows with z, so a height sum stops at the first height past the
// vertical window, where the window is 0 (it reaches 0 continuously at its
// edge). Heights are summed in FP32 in runs of 64, the runs in FP64; per
// radius an FP64 block sum over angles and one atomic add.
constexpr int kNodes = 4096;        // interpolation nodes of the height sum
constexpr int kDirectBelow = 128;   // node spacings below which ell is summed directly
constexpr float kTol = 2e-8f;       // largest relative error of an interpolated height sum
constexpr int kZRun = 64;  // heights per FP32 partial sum

// sum over heights iz = 0 .. num_z - 1 (iz = 0 with weight 1/2) of
// cos^3(theta) s_v(sin^2 theta), for horizontal distance ell. sin^2 theta
// grows with z, so the heights fall into three ranges: the window's flat part
// (s_v = 1, sin^2 < sin^2(a - b)), its soft band, and beyond (s_v = 0). The
// flat part runs first without the window's test; from the first height
// that leaves it, every sample takes the full rule until the window closes.
__device__ double height_sum(float ell, int num_z, float dz, const SoftWin &v) {
    const float e2 = ell * ell, e3 = e2 * ell;
    double tot = 0.5 * (double)soft_of_sin2(0.f, v);  // z = 0: cos theta = 1, sin theta = 0
    if (e3 == 0.f) return tot;  // ell = 0: cos theta = 0 at every z > 0
    int iz = 1;
    bool flat = true;
    while (flat && iz < num_z) {  // flat part, runs of kZRun summed in FP32
        const int stop = min(num_z, iz + kZRun);
        float part = 0.f;
        for (; iz < stop; ++iz) {
            const float z = (float)iz * dz;
            const float ih = rsqrtf(fmaf(z, z, e2));
            const float s = fabsf(z) * ih;  // sin|theta| (z < 0 when the vertical window passes pi/2)
            if (!(s * s < v.sab2)) {
                flat = false;  // this height starts the band: not consumed here
                break;
            }
            part = fmaf(e3 * ih, ih * ih, part);
        }
        tot += (double)part;
    }
    bool done = false;
    while (!done && iz < num_z) {  // soft band, until the window closes
        const int stop = min(num_z, iz + kZRun);
        float part = 0.f;
        for (; iz < stop; ++iz) {
            const float z = (float)iz * dz;
            const float ih = rsqrtf(fmaf(z, z, e2));
            const float s = fabsf(z) * ih;
            const float s2 = s * s;
            if (s2 > v.sa2) {
                done = true;
                break;
            }
            const float win = s2 < v.sab2 ? 1.f : soft_cubic(s, v);
            part = fmaf(e3 * ih * (ih * ih), win, part);
        }
        tot += (double)part;
    }
    return tot;
}

// One lane's share of height_sum (heights 1 + lane, 33 + lane, ...): the same
// samples and weights, a warp per ell.
__device__ double height_sum_lane(float ell, int num_z, float dz, const SoftWin &v, int lane) {
    const float e2 = ell * ell, e3 = e2 * ell;
    double tot = lane == 0 ? 0.5 * (double)soft_of_sin2(0.f, v) : 0.0;
    if (e3 == 0.f) return tot;
    for (int iz = 1 + lane; iz < num_z;) {
        float part = 0.f;
        bool done = false;
        for (int k = 0; k < kZRun && iz < num_z; ++k, iz += 32) {
            const float z = (float)iz * dz;
            const float ih = rsqrtf(fmaf(z, z, e2));
            const float s = fabsf(z) * ih;
            const float s2 = s * s;
            if (s2 > v.sa2) {
                done = true;
                break;
            }
            const float win = s2 < v.sab2 ? 1.f : soft_cubic(s, v);
            part = fmaf(e3 * ih * (ih * ih), win, part);
        }
        tot += (double)part;
        if (done) break;
    }
    return tot;
}

// The nodes' range of ell: [|1 - r|, 1 + r] over the call's radii (increasing).
__device__ __forceinline__ void ell_nodes(float r_max, float &lo, float &h) {
    lo = fmaxf(0.f, 1.f - r_max);
    h = (1.f + r_max - lo) / (float)(kNodes - 3);  // one node to spare at each end
    lo -= h;
}

// The least ell that is interpolated (see above; infinite for a steep window).
__device__ __forceinline__ float ell_direct(float r_max, float lo, float h, int num_z, const SoftWin &v) {
    if (!(h > 0.f)) return INFINITY;
    const float gh = v.gamma * h;
    const float edge = cbrtf(0.06f / kTol * gh * gh * fmaxf(h, (1.f + r_max) / (float)(num_z - 1)));
    return edge >= 0.f ? fmaxf(edge, fmaxf((float)kDirectBelow * h, lo + h)) : INFINITY;
}

__global__ void __launch_bounds__(kGThreads) k_gbc_height_table(const float *r_on_R, int nr, double *table, int num_z, SoftWin v,
                                                                float tan_v) {
    const int lane = threadIdx.x & 31, node = (blockIdx.x * kGThreads + threadIdx.x) >> 5;
    if (node >= kNodes) return;
    float lo, h;
    ell_nodes(r_on_R[nr - 1], lo, h);
    if (fmaf((float)(node + 3), h, lo) < ell_direct(r_on_R[nr - 1], lo, h, num_z, v)) return;  // never read
    const float dz = tan_v * (1.f + r_on_R[nr - 1]) / (float)(num_z - 1);
    double s = height_sum_lane(fmaxf(0.f, fmaf((float)node, h, lo)), num_z, dz, v, lane);
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
    if (lane == 0) table[node] = s;
}

// Four-point Lagrange interpolation of the height sum at ell.
__device__ __forceinline__ double height_at(float ell, float lo, float h, const double *__restrict__ table) {
    const double x = ((double)ell - (double)lo) / (double)h;
    int i = (int)x;
    i = i < 1 ? 1 : (i > kNodes - 3 ? kNodes - 3 : i);
    const double t = x - (double)i;
    const double a = __ldg(table + i - 1), b = __ldg(table + i), c = __ldg(table + i + 1), d = __ldg(table + i + 2);
    const double t1 = t + 1.0, tm = t - 1.0, t2 = t - 2.0;
    return (t1 * t * tm * d - t * tm * t2 * a) * (1.0 / 6.0) + (t1 * tm * t2 * b - t1 * t * t2 * c) * 0.5;
}

// table: the nodes' height sums, or null (every height sum taken directly).
__global__ void __launch_bounds__(kGThreads) k_gbc_weight_integ(const float *r_on_R, int nr, double *out, int num_z,
                                                                int num_ang, GbcSoft S, float tan_v,
                                                                const double *__restrict__ table) {
    __shared__ double warp_sums[kGThreads / 32];
    const float maxz = tan_v * (1.f + r_on_R[nr - 1]);  // tan(soft_vartheta_v) (1 + r_max)
    const float dz = maxz / (float)(num_z - 1);
    float lo, h;
    ell_nodes(r_on_R[nr - 1], lo, h);
    const float direct = table ? ell_direct(r_on_R[nr - 1], lo, h, num_z, S.v) : INFINITY;
    const double mult = (double)((4.f * maxz * 3.1415926535898f) / ((float)num_z * (float)num_ang));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int r = blockIdx.y; r < nr; r += gridDim.y) {
        double w = 0.0;
        for (int ia = blockIdx.x * kGThreads + threadIdx.x; ia < num_ang; ia += gridDim.x * kGThreads) {
            const float t = (float)ia / (float)num_ang * 3.1415926535898f;
            const float ct = cosf(t), st = sinf(t);
            const float rx = r_on_R[r] - ct, ry = -st;  // voxel minus source, in units of R
            const float q = rx * rx + ry * ry;
            const float rq = rsqrtf(q);
            const float ell = q > 0.f ? q * rq : 0.f;
            const float c = fmaxf(0.f, fminf(1.f, fabsf((rx * ct + ry * st) * rq)));  // NaN at q = 0 -> 1
            const float d = c - ell;
            const float a = __fdividef(c, fmaxf(1e-9f, c * c + d * d)) * soft_of_sin2(fmaxf(0.f, 1.f - c * c), S.h);
            // (radii out of order may lie outside the nodes)
            if (a != 0.f)
                w += (double)a * (ell >= direct && ell <= fmaf((float)(kNodes - 2), h, lo) ? height_at(ell, lo, h, table)
                                                                                          : height_sum(ell, num_z, dz, S.v));
        }
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) w += __shfl_xor_sync(0xffffffffu, w, k);
        if (lane == 0) warp_sums[warp] = w;
        __syncthreads();
        if (threadIdx.x == 0) {
            double b = 0.0;
            for (int k = 0; k < kGThreads / 32; ++k) b += warp_sums[k];
            if (b != 0.0) atomicAdd(out + r, b * mult);
        }
        __syncthreads();
    }
}

// k-factor of the softened Colsher window at polar angle th (radians from
// the k_z axis, |th| taken), cone angle `cone` and softening `soft`
// (_conebeam_kfactor_unchunked, gbc/filters.py:59-147): 2 pi outside
// (cone/2 - soft, pi - (cone/2 - soft)), else the cubic in sin(th).
__device__ double conebeam_kfactor(double th, double cone, double soft) {
    th = fabs(th);
    const double h = cone / 2 - soft;
    if (!(h < th && th < M_PI - h)) return 2 * M_PI;
    const double gamma = 1.0 / (sin(cone / 2 - soft) - sin(cone / 2));
    const double chi = gamma * sin(cone / 2);
    const double s = sin(th);
    const double alpha = h <= 0 ? 0.0 : fmax(0.0, fmin(1.0, sin(h) / s));
    const double beta = fmax(0.0, fmin(1.0, sin(cone / 2) >= s ? 1.0 : sin(cone / 2) / s));
    const double t1 = asin(beta) - asin(alpha);
    const double t2 = sqrt(1 - beta * beta);
    const double t3 = sqrt(1 - alpha * alpha);
    double out = t1 * 4 * (chi * chi) * (3 + 2 * chi) + 4 * asin(alpha);
    out += s * (24 * gamma * chi * (1 + chi) * (t2 - t3));
    out += s * s * (6 * gamma * gamma * (1 + 2 * chi) * (t1 - beta * t2 + alpha * t3));
    out += s * s * s * (-2.0 / 3.0 * gamma * gamma * gamma * (-9 * (t2 - t3) + (cos(3 * asin(beta)) - cos(3 * asin(alpha)))));
    return out;
}

__device__ double fftfreq(int k, int n) { return (double)(k < (n + 1) / 2 ? k : k - n) / (double)n; }

__device__ double sinc(double x) {
    if (x == 0.0) return 1.0;
    const double px = M_PI * x;
    return sin(px) / px;
}

struct SpecParams {
    float2 *spec;  // (n0, n1, n2 / 2 + 1) complex, C order
    int n0, n1, n2;
    double multiplier, cone, soft;
};

// One pass over the rfftn spectrum of an (n0, n1, n2) volume (axis 2 = z,
// the cylinder axis): times |k| * multiplier, divided by the k-factor of the
// polar angle (cone > 0; cone = pi gives 2 pi; cone = 0 uses the lateral |k|
// without a k-factor), times sinc(f0) sinc(f1) sinc(f2); the DC term is set
// to 0 (filters.py:340-398).
__global__ void __launch_bounds__(kGThreads) k_conebeam_spectral(const SpecParams P) {
    const int m2 = P.n2 / 2 + 1;
    const int64_t n = (int64_t)P.n0 * P.n1 * m2;
    const int64_t step = (int64_t)gridDim.x * kGThreads;
    for (int64_t e = (int64_t)blockIdx.x * kGThreads + threadIdx.x; e < n; e += step) {
        const int k2 = (int)(e % m2);
        const int64_t r = e / m2;
        const int k1 = (int)(r % P.n1), k0 = (int)(r / P.n1);
        const double f0 = fftfreq(k0, P.n0), f1 = fftfreq(k1, P.n1), f2 = (double)k2 / (double)P.n2;
        const double lat2 = f0 * f0 + f1 * f1;
        double factor;
        if (P.cone == 0.0) {
            factor = sqrt(lat2) * P.multiplier;
        } else {
            factor = sqrt(lat2 + f2 * f2) * P.multiplier;
            const double th = fabs(M_PI / 2 - atan2(f2, sqrt(lat2)));
            factor /= P.cone == M_PI ? 2 * M_PI : conebeam_kfactor(th, P.cone, P.soft);
        }
        factor *= sinc(f0) * sinc(f1) * sinc(f2);
        if (e == 0) factor = 0.0;
        const float2 z = P.spec[e];
        P.spec[e] = make_float2((float)((double)z.x * factor), (float)((double)z.y * factor));
    }
}

// out[x][y][z] += trilinear value of low at (x, y, z) / d - 1/2 + 1/(2d) per
// axis, neighbour indices clamped to the array (scipy.ndimage.map_coordinates
// order 1, mode "nearest", the reference's low-resolution correction,
// filters.py:403-455). Both arrays C order (z fastest).
__global__ void __launch_bounds__(kGThreads) k_add_upsampled(float *out, int n0, int n1, int n2, const float *low,
                                                             int m0, int m1, int m2, int d) {
    const int64_t n = (int64_t)n0 * n1 * n2;
    const int64_t step = (int64_t)gridDim.x * kGThreads;
    for (int64_t e = (int64_t)blockIdx.x * kGThreads + threadIdx.x; e < n; e += step) {
        const int z = (int)(e % n2);
        const int64_t r = e / n2;
        const int y = (int)(r % n1), x = (int)(r / n1);
        const int idx[3] = {x, y, z}, lim[3] = {m0, m1, m2};
        int i0[3], i1[3];
        double t[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const double c = (double)idx[a] / d - 0.5 + 1.0 / d / 2;
            const double f = floor(c);
            t[a] = c - f;
            const int fi = (int)f;
            i0[a] = min(max(fi, 0), lim[a] - 1);
            i1[a] = min(max(fi + 1, 0), lim[a] - 1);
        }
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int a = c >> 2 & 1, b = c >> 1 & 1, g = c & 1;
            const double w = (a ? t[0] : 1 - t[0]) * (b ? t[1] : 1 - t[1]) * (g ? t[2] : 1 - t[2]);
            const int ix = a ? i1[0] : i0[0], iy = b ? i1[1] : i0[1], iz = g ? i1[2] : i0[2];
            v += w * (double)low[((int64_t)ix * m1 + iy) * m2 + iz];
        }
        out[e] += (float)v;
    }
}

unsigned grid_for(int64_t n) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    const int64_t want = (n + kGThreads - 1) / kGThreads, cap = (int64_t)sms * 16;
    return (unsigned)(want < cap ? want : cap);
}

bool finite_soft(const aprict_backproject_config *c) {
    return std::isfinite(c->soft_vartheta_v) && std::isfinite(c->soft_vartheta_v_softspan) &&
           std::isfinite(c->soft_vartheta_h) && std::isfinite(c->soft_vartheta_h_softspan);
}

}  // namespace

extern "C" int aprict_b200_backproject_gbc_views(const aprict_proj_spec *specs_dev, const aprict_proj_desc *pd,
                                                 const float *projs_dev, const aprict_vol_desc *vd, float *vol_dev,
                                                 float *weightsum_dev, const float *multiplier_dev,
                                                 const aprict_backproject_config *cfg, uint32_t views, uint32_t *status_dev,
                                                 aprict_stream_t stream) {
    if (views > APRICT_VIEWS_MIXED) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "GBC: unknown view promise %u", views);
    if (views == APRICT_VIEWS_MIXED) views = APRICT_VIEWS_GENERAL;  // one kernel for both
    if (cfg == nullptr) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "null backproject config");
    if (cfg->weighting_preset != 7)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "the GBC backprojection takes weighting preset 7");
    if (cfg->exact) return ab_fail(APRICT_ERR_UNSUPPORTED, "the GBC backprojection is a fast (approximate) mode");
    if (!(cfg->Z_on_val_factor_val > 0.f) || !finite_soft(cfg))
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "GBC needs R > 0 in Z_on_val_factor_val and finite soft windows");
    if (weightsum_dev == nullptr) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "GBC needs a weight-sum volume");
    if ((reinterpret_cast<uintptr_t>(weightsum_dev) & 3u) != 0)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "weight-sum volume pointer not 4-byte aligned");
    if (weightsum_dev == vol_dev) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "the weight sums need their own volume");
    aprict_backproject_config c = *cfg;
    c.weighting_preset = 0;  // validated here; the shared checks below know presets 0-6
    ab_bp::BPParams P;
    uint64_t units = 0;
    int xb = 2;
    int cxb = kGCol;
    uint64_t col_units = 0;
    int rc = ab_bp::make_bp_params(specs_dev, pd, projs_dev, vd, vol_dev, multiplier_dev, &c, status_dev, P, units,
                                   xb, 2, nullptr, &cxb, &col_units);
    if (rc != APRICT_OK || units == 0) return rc;
    // (super-bricks of one wave: 198^3 x 360 views 5.59 ms, of four 5.61)
    if (cxb != 0 && !ab_bp::order_bricks(P.col, 1, ab_bp::kColBlocks, col_units))
        return ab_fail(APRICT_ERR_TOO_LARGE, "volume too large for the grid");
    P.views = (int)views;
    GbcParams G;
    G.vol2 = weightsum_dev;
    G.inv_R = (float)(1.0 / (double)cfg->Z_on_val_factor_val);
    G.soft = GbcSoft{soft_win(cfg->soft_vartheta_v, cfg->soft_vartheta_v_softspan),
                     soft_win(cfg->soft_vartheta_h, cfg->soft_vartheta_h_softspan)};
    G.pos000[0] = vd->corner.x + 0.5f * vd->voxwid;
    G.pos000[1] = vd->corner.y + 0.5f * vd->voxwid;
    G.pos000[2] = vd->corner.z + 0.5f * vd->voxwid;
    const int64_t nvox = (int64_t)vd->nx * vd->ny * vd->nz;
    const int64_t blocks = (nvox + kGThreads - 1) / kGThreads;
    if (blocks > 0x7fffffffLL) return ab_fail(APRICT_ERR_TOO_LARGE, "volume too large for the grid");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int order_f = vd->order != 0;
    // C order: the columns at every size. F order: its lanes along x have a flat volume's
    // voxels side by side and need no column, a small one's are too few for 8 voxels a
    // lane, and a column reads and writes both volumes 4 bytes a line. 198^2 x nz from 120
    // views bilinear, columns and k_backproject_gbc: 8: 1096, 292 us; 48: 1557, 1470; 64:
    // 791, 1971; 24^2 x 100: 164, 79; 48^2 x 64: 91, 157; nearest 99^2 x 65: 455, 383.
    if (cxb != 0 && order_f &&
        !(pd->n_views > ab_bp::views_f(cfg) && vd->nz > 48u && !(vd->nz > 64u && vd->nz < ab_bp::kSecondPair) &&
          ab_bp::col_units_of(vd, kGCol) >= 3 * (uint64_t)ab_bp::bp_sms() / 2))
        P.views = (int)(views = APRICT_VIEWS_GENERAL);
    if (cxb != 0 && views != APRICT_VIEWS_GENERAL) {
        // The window's flat part and its end as bounds on |z - s_z| / (R ell),
        // with 1e-5 to spare (the band's rule decides there); none where the
        // angle reaches pi/2 or the flat part is empty.
        const double a = cfg->soft_vartheta_v, b = a - cfg->soft_vartheta_v_softspan, half_pi = 1.5707963267948966;
        const float tan_a = a >= half_pi ? 3e38f : (float)tan(a);
        const float tan_flat = a <= 0.0 || b <= 0.0 ? 0.f : std::min(tan_a, b >= half_pi ? 3e38f : (float)tan(b)) * (1.f - 1e-5f);
        const float tan_zero = a >= half_pi || a <= 0.0 ? INFINITY : tan_a * (1.f + 1e-5f);
        // 0 < b < a < pi/2: the window is the cubic of its argument clamped to [0, 1]
        const int clamped = b > 0.0 && b < a && a < half_pi;
        for (auto *k : {k_backproject_gbc_columns<true>, k_backproject_gbc_columns<false>}) {
            rc = ab_cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GbcColSmem)),
                               "backproject_gbc smem");
            if (rc != APRICT_OK) return rc;
        }
        auto *kern = cfg->approx_mode_linear_interpolate ? k_backproject_gbc_columns<true> : k_backproject_gbc_columns<false>;
        kern<<<(unsigned)col_units, kGThreads, sizeof(GbcColSmem), st>>>(P, G, tan_flat, tan_zero, clamped);
        if (views == APRICT_VIEWS_UPRIGHT) return ab_cuda_check(cudaGetLastError(), "backproject_gbc launch");
    }
    if (!order_f) {  // C order: z columns (see k_backproject_gbc_z)
        const int64_t gb0 = ((int64_t)vd->nz + 32 * kGZ - 1) / (32 * kGZ), gb1 = ((int64_t)vd->ny + 7) / 8;
        const int64_t zblocks = gb0 * gb1 * (int64_t)vd->nx;
        if (zblocks > 0x7fffffffLL) return ab_fail(APRICT_ERR_TOO_LARGE, "volume too large for the grid");
        if (cfg->approx_mode_linear_interpolate)
            k_backproject_gbc_z<true><<<(unsigned)zblocks, kGThreads, 0, st>>>(P, G, (int)gb0, (int)gb1);
        else
            k_backproject_gbc_z<false><<<(unsigned)zblocks, kGThreads, 0, st>>>(P, G, (int)gb0, (int)gb1);
    } else if (cfg->approx_mode_linear_interpolate) {
        k_backproject_gbc<true><<<(unsigned)blocks, kGThreads, 0, st>>>(P, G, order_f);
    } else {
        k_backproject_gbc<false><<<(unsigned)blocks, kGThreads, 0, st>>>(P, G, order_f);
    }
    return ab_cuda_check(cudaGetLastError(), "backproject_gbc launch");
}

extern "C" int aprict_b200_backproject_gbc(const aprict_proj_spec *specs_dev, const aprict_proj_desc *pd,
                                           const float *projs_dev, const aprict_vol_desc *vd, float *vol_dev,
                                           float *weightsum_dev, const float *multiplier_dev,
                                           const aprict_backproject_config *cfg, uint32_t *status_dev,
                                           aprict_stream_t stream) {
    return aprict_b200_backproject_gbc_views(specs_dev, pd, projs_dev, vd, vol_dev, weightsum_dev, multiplier_dev, cfg,
                                             APRICT_VIEWS_UNKNOWN, status_dev, stream);
}

extern "C" int64_t aprict_b200_gbc_weight_integral_scratch_bytes(int32_t n_r, int32_t num_ang) {
    // The table pays from a few tables' worth of height sums on: 16384 of them in
    // warps of 32 cost about what the table's 4096 warps do.
    return (int64_t)n_r * num_ang >= 4 * (int64_t)kNodes ? (int64_t)(kNodes * sizeof(double)) : 0;
}

extern "C" int aprict_b200_gbc_weight_integral_scratch(const float *r_on_R_dev, int32_t n_r, double *out_dev, int32_t num_z,
                                                       int32_t num_ang, const aprict_backproject_config *cfg,
                                                       void *scratch_dev, aprict_stream_t stream) {
    if (cfg == nullptr) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "null backproject config");
    if (n_r <= 0) return APRICT_OK;
    if (r_on_R_dev == nullptr || out_dev == nullptr)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "null radius or output array");
    if (num_z < 2 || num_ang < 1 || (int64_t)num_z * num_ang > (int64_t)1 << 31)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "num_z must be >= 2, num_ang >= 1, num_z * num_ang <= 2^31");
    if (!finite_soft(cfg)) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "non-finite soft windows");
    const GbcSoft S{soft_win(cfg->soft_vartheta_v, cfg->soft_vartheta_v_softspan),
                    soft_win(cfg->soft_vartheta_h, cfg->soft_vartheta_h_softspan)};
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const float tan_v = (float)tan((double)cfg->soft_vartheta_v);
    if ((reinterpret_cast<uintptr_t>(scratch_dev) & 7u) != 0)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "gbc_weight_integral: scratch not 8-byte aligned");
    double *table = static_cast<double *>(scratch_dev);
    if (table != nullptr && aprict_b200_gbc_weight_integral_scratch_bytes(n_r, num_ang) > 0) {
        k_gbc_height_table<<<kNodes * 32 / kGThreads, kGThreads, 0, st>>>(r_on_R_dev, n_r, table, num_z, S.v, tan_v);
        // a CTA per radius where the radii alone fill the GPU
        const int per_r = n_r >= 296 ? 1 : (num_ang + kGThreads - 1) / kGThreads;
        k_gbc_weight_integ<<<dim3((unsigned)per_r, (unsigned)min(n_r, 65535)), kGThreads, 0, st>>>(
            r_on_R_dev, n_r, out_dev, num_z, num_ang, S, tan_v, table);
        return ab_cuda_check(cudaGetLastError(), "gbc_weight_integral launch");
    }
    const dim3 grid((unsigned)((num_ang + kGThreads - 1) / kGThreads), (unsigned)min(n_r, 65535));
    k_gbc_weight_integ<<<grid, kGThreads, 0, st>>>(r_on_R_dev, n_r, out_dev, num_z, num_ang, S, tan_v, nullptr);
    return ab_cuda_check(cudaGetLastError(), "gbc_weight_integral launch");
}

extern "C" int aprict_b200_gbc_weight_integral(const float *r_on_R_dev, int32_t n_r, double *out_dev, int32_t num_z,
                                               int32_t num_ang, const aprict_backproject_config *cfg,
                                               aprict_stream_t stream) {
    return aprict_b200_gbc_weight_integral_scratch(r_on_R_dev, n_r, out_dev, num_z, num_ang, cfg, nullptr, stream);
}

extern "C" int aprict_b200_conebeam_spectral(void *spec_dev, int32_t n0, int32_t n1, int32_t n2, double multiplier,
                                             double cone_angle, double theta_soft, aprict_stream_t stream) {
    if (n0 <= 0 || n1 <= 0 || n2 <= 0) return APRICT_OK;
    if (spec_dev == nullptr) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "null spectrum");
    if ((reinterpret_cast<uintptr_t>(spec_dev) & 7u) != 0)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "spectrum pointer not 8-byte aligned");
    if (!(cone_angle >= 0.0 && cone_angle <= M_PI))
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "cone angle must lie in [0, pi]");
    if (!std::isfinite(multiplier) || !std::isfinite(theta_soft))
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "non-finite multiplier or softening");
    SpecParams P{static_cast<float2 *>(spec_dev), n0, n1, n2, multiplier, cone_angle, theta_soft};
    const int64_t n = (int64_t)n0 * n1 * (n2 / 2 + 1);
    k_conebeam_spectral<<<grid_for(n), kGThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(P);
    return ab_cuda_check(cudaGetLastError(), "conebeam_spectral launch");
}

extern "C" int aprict_b200_add_upsampled(float *out_dev, int32_t n0, int32_t n1, int32_t n2, const float *low_dev,
                                         int32_t m0, int32_t m1, int32_t m2, int32_t factor, aprict_stream_t stream) {
    if (n0 <= 0 || n1 <= 0 || n2 <= 0) return APRICT_OK;
    if (out_dev == nullptr || low_dev == nullptr) return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "null array");
    if (m0 <= 0 || m1 <= 0 || m2 <= 0 || factor <= 0)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "empty low-resolution array or non-positive factor");
    const int64_t n = (int64_t)n0 * n1 * n2;
    k_add_upsampled<<<grid_for(n), kGThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(out_dev, n0, n1, n2,
                                                                                          low_dev, m0, m1, m2, factor);
    return ab_cuda_check(cudaGetLastError(), "add_upsampled launch");
}
