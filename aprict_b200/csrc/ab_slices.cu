// ab_slices.cu -- fan-beam backprojection of a stack of slices that share one
// scan: every slice's sinogram and image in one launch.
//
// The slices of a fan-beam stack (src/aprict/scripts/recon_cbfp_cyl_fbp.py with
// fan_beam=True reconstructs them one by one) have the same views, so a pixel's
// detector column and weight (CB_backproject.cu:512-528) are those of every
// slice. The filtered data is taken with the slices interleaved, (view, u,
// slice): what one voxel gathers from one view for all slices is contiguous,
// and its coordinate is computed once for the whole stack.
//
// Work split: LS lanes of a warp hold 4 slices each (one 16-byte gather), the
// 32 / LS voxel groups of a warp kVox voxels each. A CTA computes the detector
// columns and weights of its tile of voxels for a few views into shared memory
// (each entry once: the same steps and FP64 near-tie decisions as bp_brick's
// one-row path), then every thread reads an entry, gathers 4 slices and adds
// them to 4 accumulators. Per voxel and view of 4 slices that is one shared
// load, one 16-byte gather and 4 fmas.
// Bound: the L1's 128 bytes per clock (4 B per voxel, view and slice).
// Measured, 64 slices 512^2 x 720 views x 1024: 24 ms (every slice by itself, one
// persistent launch) -> 3.4 ms with 8 voxels per thread and 16 warps per SM; with 4
// and 32, as here, the whole reconstruction of the stack takes 4.6 ms instead of
// 5.1 (the gathers' latency wants the warps more than the shared loads the reuse).
// Accumulation as in bp_brick: FP32 over a chunk of views, the chunks under
// Kahan's compensation (totals and compensations in shared memory).
#include <cuda_runtime.h>

#include "ab_bpbrick.cuh"

namespace {

using namespace ab_bp;

constexpr int kVox = 4;       // voxels per thread
constexpr int kMaxSlices = 64;
constexpr int kEntries = 1024;  // (view, voxel) entries per table fill
constexpr int kViews = 64;      // views per coefficient chunk (and per FP32 partial sum)
constexpr int kTileY = 16;

struct SliceArgs {
    BPParams P;                 // scan, volume grid and config of every slice (projs: the interleaved data)
    float *vol[kMaxSlices];
    int n_slices;
    int pitch;                  // floats from pixel to pixel (a multiple of 4)
    uint32_t zero_pixel;        // index of a pixel of zeros after the last view's
};

struct SliceSmem {
    ab_bpview sv[kViews];
    ab_bpview_d svd[kViews];
    uint2 table[kEntries];      // pixel index, weight bits
    float sum[kVox * 4][kThreads], comp[kVox * 4][kThreads];
};

// LS: lanes per voxel (4 LS >= slices).
template <int LS>
__global__ void __launch_bounds__(kThreads, 4) k_backproject_slices(const __grid_constant__ SliceArgs A) {
    constexpr int kGroups = 32 / LS;             // voxel groups per warp
    constexpr int kTile = kWarps * kGroups * kVox;  // voxels per CTA
    constexpr int kStep = kEntries / kTile;      // views per table fill
    constexpr int kTileX = kTile / kTileY;
    const BPParams &P = A.P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SliceSmem &sm = *reinterpret_cast<SliceSmem *>(smem_raw);

    const int x0 = blockIdx.y * kTileX, y0 = blockIdx.x * kTileY;
    const float vw = P.voxwid;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = warp * kGroups + lane / LS, ls = lane % LS;
    // position of tile voxel e relative to the volume centre, and whether it is reconstructed
    auto voxel = [&](int e, float &X, float &Y) -> bool {
        const int ix = x0 + e / kTileY, iy = y0 + e % kTileY;
        X = ((float)ix + 0.5f - 0.5f * (float)P.n[0]) * vw;
        Y = ((float)iy + 0.5f - 0.5f * (float)P.n[1]) * vw;
        if (ix >= P.n[0] || iy >= P.n[1]) return false;
        const float xw = X + P.c0[0], yw = Y + P.c0[1];
        return !(P.mask && xw * xw + yw * yw > P.mask_r2);
    };
    bool any = false;
    for (int e = threadIdx.x; e < kTile; e += kThreads) {
        float X, Y;
        any = any || voxel(e, X, Y);
    }
    if (!__syncthreads_or(any)) return;  // the tile lies outside the cylinder

#pragma unroll
    for (int i = 0; i < kVox * 4; ++i) sm.sum[i][threadIdx.x] = sm.comp[i][threadIdx.x] = 0.f;
    const bool needZ = P.pL != 0 || P.pV != 0;
    const float4 *data = reinterpret_cast<const float4 *>(P.projs) + ls;
    const uint32_t pitch16 = 4u * (uint32_t)A.pitch;  // bytes from pixel to pixel
    const bool lane_on = 4 * ls < A.pitch;

    for (uint32_t v0 = 0; v0 < P.n_views; v0 += kViews) {
        const int cn = (int)min((uint32_t)kViews, P.n_views - v0);
        __syncthreads();
        if ((int)threadIdx.x < cn) {
            const ab_d3 c0d{P.cornerd[0] + 0.5 * P.vwd * P.n[0], P.cornerd[1] + 0.5 * P.vwd * P.n[1],
                            P.cornerd[2] + 0.5 * P.vwd * P.n[2]};
            const aprict_proj_spec sp = P.specs[v0 + threadIdx.x];
            const double hext[3] = {(0.5 * P.n[0] + 1.0) * P.vwd, (0.5 * P.n[1] + 1.0) * P.vwd, (0.5 * P.n[2] + 1.0) * P.vwd};
            if (!ab_derive_bpview(sp, c0d, vw, P.sep, hext, sm.sv[threadIdx.x], &sm.svd[threadIdx.x]) && P.status)
                atomicOr(P.status, APRICT_STATUS_BAD_GEOMETRY);
        }
        float acc[kVox][4];
#pragma unroll
        for (int k = 0; k < kVox; ++k)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[k][c] = 0.f;
        for (int s0 = 0; s0 < cn; s0 += kStep) {
            __syncthreads();  // coefficients written; the previous table no longer read
            for (int q = threadIdx.x; q < kEntries; q += kThreads) {
                const int t = s0 + q / kTile, e = q % kTile;
                uint32_t pix = A.zero_pixel;
                float w = 0.f;
                float X, Y;
                if (t < cn && voxel(e, X, Y)) {
                    const ab_bpview &b = sm.sv[t];
                    const float D = dot4(b.den, X, Y, 0.f);
                    const float rD = rcp_fast(D);
                    const float fu = dot4(b.nu, X, Y, 0.f) * rD;
                    float du;
                    int iu = round_index(fu, -2.f, P.fnu1, du);
                    if (fabsf(du) > b.tie_u) {
                        const VoxRef vr{((double)(x0 + e / kTileY) + 0.5 - 0.5 * P.n[0]) * P.vwd,
                                        ((double)(y0 + e % kTileY) + 0.5 - 0.5 * P.n[1]) * P.vwd, 0.0};
                        iu = refine_index(sm.svd[t].nu, sm.svd[t].den, vr, iu, du);
                    }
                    if ((unsigned)iu < P.nu) {  // else the pixel of zeros, weight 0
                        pix = (v0 + (uint32_t)t) * P.nu + (uint32_t)iu;
                        w = needZ ? zpow(P, b, dot4(b.zl, X, Y, 0.f)) : 1.f;
                    }
                }
                sm.table[q] = make_uint2(pix, __float_as_uint(w));
            }
            __syncthreads();
            const int sn = min(kStep, cn - s0);
            const uint2 *tab = sm.table + group * kVox;
            if (lane_on) {
#pragma unroll 1
                for (int t = 0; t < sn; ++t, tab += kTile) {
                    float4 p[kVox];
                    float w[kVox];
#pragma unroll
                    for (int k = 0; k < kVox; k += 2) {
                        const uint4 two = *reinterpret_cast<const uint4 *>(tab + k);
                        w[k] = __uint_as_float(two.y);
                        w[k + 1] = __uint_as_float(two.w);
                        p[k] = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(data) +
                                                                      (uint64_t)two.x * pitch16));
                        p[k + 1] = __ldg(reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(data) +
                                                                          (uint64_t)two.z * pitch16));
                    }
#pragma unroll
                    for (int k = 0; k < kVox; ++k) {
                        acc[k][0] = fmaf(p[k].x, w[k], acc[k][0]);
                        acc[k][1] = fmaf(p[k].y, w[k], acc[k][1]);
                        acc[k][2] = fmaf(p[k].z, w[k], acc[k][2]);
                        acc[k][3] = fmaf(p[k].w, w[k], acc[k][3]);
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kVox * 4; ++i) {  // the chunk's partial sums into the compensated totals
            const float sk = sm.sum[i][threadIdx.x];
            const float y = acc[i >> 2][i & 3] - sm.comp[i][threadIdx.x];
            const float tk = sk + y;
            sm.comp[i][threadIdx.x] = (tk - sk) - y;
            sm.sum[i][threadIdx.x] = tk;
        }
    }
    __syncthreads();
    // rows of 16 voxels of one slice per half warp
    for (int o = threadIdx.x; o < kTile * A.n_slices; o += kThreads) {
        const int e = o % kTile, s = o / kTile;
        const int ix = x0 + e / kTileY, iy = y0 + e % kTileY;
        if (ix >= P.n[0] || iy >= P.n[1]) continue;
        const int g = e / kVox, i = (e % kVox) * 4 + (s & 3);
        const int owner = (g / kGroups) * 32 + (g % kGroups) * LS + (s >> 2);
        const float value = sm.sum[i][owner] - sm.comp[i][owner];
        if (value == 0.f) continue;  // the reference skips the write (:1010)
        float *p = A.vol[s] + (int64_t)ix * P.vs[0] + (int64_t)iy * P.vs[1];
        *p += value;
    }
}

template <int LS>
int launch_slices(const SliceArgs &A, cudaStream_t st) {
    constexpr int kTile = kWarps * (32 / LS) * kVox;
    const int rc = ab_cuda_check(cudaFuncSetAttribute(k_backproject_slices<LS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      (int)sizeof(SliceSmem)),
                                 "backproject_slices smem");
    if (rc != APRICT_OK) return rc;
    const unsigned gy = (unsigned)((A.P.n[0] + kTile / kTileY - 1) / (kTile / kTileY));
    if (gy > 65535u) return ab_fail(APRICT_ERR_TOO_LARGE, "slice too large for the grid");
    const dim3 grid((unsigned)((A.P.n[1] + kTileY - 1) / kTileY), gy);
    k_backproject_slices<LS><<<grid, kThreads, sizeof(SliceSmem), st>>>(A);
    return ab_cuda_check(cudaGetLastError(), "backproject_slices launch");
}

}  // namespace

extern "C" int aprict_b200_backproject_slices(const aprict_proj_spec *specs_dev, uint32_t n_views, uint32_t nu,
                                              const float *data_dev, int64_t pitch, int32_t n_slices,
                                              const aprict_vol_desc *vd, float *const *vols_dev,
                                              const aprict_backproject_config *cfg, uint32_t *status_dev,
                                              aprict_stream_t stream) {
    if (vd == nullptr || cfg == nullptr || vols_dev == nullptr)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "backproject_slices: null argument");
    if (n_slices < 0 || n_slices > kMaxSlices)
        return ab_fail(APRICT_ERR_UNSUPPORTED, "backproject_slices: 0 to %d slices a call", kMaxSlices);
    if (pitch < n_slices || pitch % 4 != 0 || pitch > kMaxSlices)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "backproject_slices: the pitch is a multiple of 4 from n_slices to %d", kMaxSlices);
    if ((reinterpret_cast<uintptr_t>(data_dev) & 15u) != 0)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "backproject_slices: data not 16-byte aligned");
    if (vd->nz != 1 || vd->order != 0)
        return ab_fail(APRICT_ERR_UNSUPPORTED, "backproject_slices: C-order slices of one layer");
    if (cfg->exact || !cfg->approx_mode_direct_raycast || cfg->approx_mode_linear_interpolate || cfg->weighting_preset != 0 ||
        cfg->apply_summand_multiplier || cfg->soften_edge_proportion != 0.f || cfg->ssx != 1 || cfg->ssy != 1 || cfg->ssz != 1)
        return ab_fail(APRICT_ERR_UNSUPPORTED, "backproject_slices: plain nearest-pixel direct-raycast mode only");
    if ((uint64_t)n_views * nu >= 0xffffffffull) return ab_fail(APRICT_ERR_TOO_LARGE, "backproject_slices: too many pixels");
    if (n_slices == 0 || n_views == 0 || nu == 0) return APRICT_OK;
    aprict_proj_desc pd{};
    pd.n_views = n_views;
    pd.nu = nu;
    pd.nv = 1;
    pd.stride_view = (int64_t)nu * pitch;
    pd.stride_u = pitch;
    pd.stride_v = 1;
    SliceArgs A{};
    for (int s = 0; s < n_slices; ++s) {
        const int rc = ab_check_vol(vd, vols_dev[s], "slice volume");
        if (rc != APRICT_OK) return rc;
        A.vol[s] = vols_dev[s];
    }
    uint64_t units = 0;
    int xb = 2;
    const int rc = make_bp_params(specs_dev, &pd, data_dev, vd, vols_dev[0], nullptr, cfg, status_dev, A.P, units, xb, 2);
    if (rc != APRICT_OK || units == 0) return rc;
    A.n_slices = n_slices;
    A.pitch = (int)pitch;
    A.zero_pixel = n_views * nu;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const int quads = (int)pitch / 4;
    if (quads > 8) return launch_slices<16>(A, st);
    if (quads > 4) return launch_slices<8>(A, st);
    if (quads > 2) return launch_slices<4>(A, st);
    if (quads > 1) return launch_slices<2>(A, st);
    return launch_slices<1>(A, st);
}
