// ab_backproject.cu -- voxel-driven cone-beam backprojection, all views in
// one launch (one scan). The work unit lives in ab_bpbrick.cuh.
#include <cuda_runtime.h>

#include "ab_bpcol.cuh"

namespace {

using namespace ab_bp;

template <int ORD, bool EXACT, bool RAYCAST, bool BILIN, int XB, bool ZT = false>
__global__ void __launch_bounds__(kThreads, bp_min_blocks(XB, EXACT)) k_backproject(const BPParams P) {
    __shared__ BPSmem<EXACT, BILIN, XB, ZT> sm;
    if constexpr (!EXACT && ORD != 2) {
        if (P.views == (int)APRICT_VIEWS_UNKNOWN && P.col.gb[0] != 0 && all_upright(P)) return;  // k_backproject_columns'
    }
    bp_brick<ORD, EXACT, RAYCAST, BILIN, XB, RAYCAST, ZT>(P, blockIdx.x, sm);
}

template <bool RAYCAST, bool BILIN, int XB>
__global__ void __launch_bounds__(kThreads, kColBlocks) k_backproject_columns(const BPParams P) {
    __shared__ ColSmem<XB> sm;
    if (!all_upright(P)) return;  // k_backproject's
    bp_columns<RAYCAST, BILIN, XB>(P, blockIdx.x, sm);
}

template <int XB>
void launch_columns(const BPParams &P, bool raycast, bool lin, unsigned grid, cudaStream_t st) {
    if (raycast && lin)
        k_backproject_columns<true, true, XB><<<grid, kThreads, 0, st>>>(P);
    else if (raycast)
        k_backproject_columns<true, false, XB><<<grid, kThreads, 0, st>>>(P);
    else if (lin)
        k_backproject_columns<false, true, XB><<<grid, kThreads, 0, st>>>(P);
    else
        k_backproject_columns<false, false, XB><<<grid, kThreads, 0, st>>>(P);
}

template <int ORD, int XB>
void launch_bp(const BPParams &P, const aprict_backproject_config *cfg, bool lin, unsigned grid, cudaStream_t st) {
    if (cfg->exact) {
        k_backproject<ORD, true, false, false, XB><<<grid, kThreads, 0, st>>>(P);
    } else if (cfg->approx_mode_direct_raycast) {
        if constexpr (ORD != 3) {
            if (lin)
                k_backproject<ORD, false, true, true, XB><<<grid, kThreads, 0, st>>>(P);
            else
                k_backproject<ORD, false, true, false, XB><<<grid, kThreads, 0, st>>>(P);
        }
    } else if (lin) {
        if constexpr (ORD != 3) k_backproject<ORD, false, false, true, XB><<<grid, kThreads, 0, st>>>(P);
    } else if (ORD == 3 && P.views != (int)APRICT_VIEWS_GENERAL) {  // some views may be upright
        k_backproject<ORD, false, false, false, XB, ORD == 3><<<grid, kThreads, 0, st>>>(P);
    } else {
        k_backproject<ORD, false, false, false, XB><<<grid, kThreads, 0, st>>>(P);
    }
}

}  // namespace

extern "C" int aprict_b200_backproject_views(const aprict_proj_spec *specs_dev, const aprict_proj_desc *pd,
                                             const float *projs_dev, const aprict_vol_desc *vd, float *vol_dev,
                                             const float *multiplier_dev, const aprict_backproject_config *cfg,
                                             uint32_t views, uint32_t *status_dev, aprict_stream_t stream) {
    if (views > APRICT_VIEWS_MIXED)
        return ab_fail(APRICT_ERR_INVALID_ARGUMENT, "backproject: unknown view promise %u", views);
    BPParams P;
    uint64_t grid = 0, col_grid = 0;
    int xb = 2;
    int ord = 0;
    int cxb = 0;
    // Slice stacks (one z layer) always take two voxels per thread.
    const int rc = make_bp_params(specs_dev, pd, projs_dev, vd, vol_dev, multiplier_dev, cfg, status_dev, P, grid, xb,
                                  vd != nullptr && bp_ord(vd) == 2 ? 2 : 0, &ord, &cxb, &col_grid);
    if (rc != APRICT_OK || grid == 0) return rc;
    P.views = (int)views;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const bool lin = cfg->approx_mode_linear_interpolate != 0;
    if (cxb != 0 && views != APRICT_VIEWS_MIXED && !columns_pay(vd, pd->n_views, cfg, col_units_of(vd, cxb), false)) P.views = (int)(views = APRICT_VIEWS_GENERAL);
    if (cxb != 0 && (views == APRICT_VIEWS_UNKNOWN || views == APRICT_VIEWS_UPRIGHT)) {
        const bool ray = cfg->approx_mode_direct_raycast != 0;
        if (cxb == 8)
            launch_columns<8>(P, ray, lin, (unsigned)col_grid, st);
        else if (cxb == 4)
            launch_columns<4>(P, ray, lin, (unsigned)col_grid, st);
        else
            launch_columns<2>(P, ray, lin, (unsigned)col_grid, st);
        if (views == APRICT_VIEWS_UPRIGHT) return ab_cuda_check(cudaGetLastError(), "backproject launch");
    }
    if (ord == 2) {
        launch_bp<2, 2>(P, cfg, lin, (unsigned)grid, st);  // slices (xb forced to 2 above)
    } else if (ord == 3) {  // C order, lanes and a thread's voxels along z
        if (xb == 8)
            launch_bp<3, 8>(P, cfg, lin, (unsigned)grid, st);
        else if (xb == 4)
            launch_bp<3, 4>(P, cfg, lin, (unsigned)grid, st);
        else
            launch_bp<3, 2>(P, cfg, lin, (unsigned)grid, st);
    } else if (xb == 8) {
        if (ord == 0)
            launch_bp<0, 8>(P, cfg, lin, (unsigned)grid, st);
        else
            launch_bp<1, 8>(P, cfg, lin, (unsigned)grid, st);
    } else if (xb == 4) {
        if (ord == 0)
            launch_bp<0, 4>(P, cfg, lin, (unsigned)grid, st);
        else
            launch_bp<1, 4>(P, cfg, lin, (unsigned)grid, st);
    } else {
        if (ord == 0)
            launch_bp<0, 2>(P, cfg, lin, (unsigned)grid, st);
        else
            launch_bp<1, 2>(P, cfg, lin, (unsigned)grid, st);
    }
    return ab_cuda_check(cudaGetLastError(), "backproject launch");
}

extern "C" int aprict_b200_backproject(const aprict_proj_spec *specs_dev, const aprict_proj_desc *pd,
                                       const float *projs_dev, const aprict_vol_desc *vd, float *vol_dev,
                                       const float *multiplier_dev, const aprict_backproject_config *cfg,
                                       uint32_t *status_dev, aprict_stream_t stream) {
    return aprict_b200_backproject_views(specs_dev, pd, projs_dev, vd, vol_dev, multiplier_dev, cfg, APRICT_VIEWS_UNKNOWN,
                                         status_dev, stream);
}
