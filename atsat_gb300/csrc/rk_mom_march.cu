// Launches of the radial-march momentum / temperature kernel on its own (rk_march_body.cuh): every stage that does not
// share a launch with the tracers. That is any stage of a grid beyond the waves of stage_fusable (rk_stage_fused.cu; the
// 41x181x361 shell among them), and on smaller grids the intermediate stages of knob sets with more than 12 point arrays
// or with the regular rings.
#include "rk_march_body.cuh"

namespace atsat {

namespace {

using namespace march;

template <int MODE, bool HAS_DL, bool CMP>
__global__ void __launch_bounds__(march::THREADS, (CMP ? 3 : 2))
rk_mom_march_kernel(const __grid_constant__ CUtensorMap map_plane, const __grid_constant__ CUtensorMap map_seam,
                    const __grid_constant__ CUtensorMap map_pt, const MixedConstF K, const MixedIO io,
                    const StageParams sp, const MarchPlan plan) {
    extern __shared__ __align__(128) float smem[];
    march::block<MODE, HAS_DL, CMP>(map_plane, map_seam, map_pt, K, io, sp, plan, smem, blockIdx.x, blockIdx.y, blockIdx.z);
}

template <int MODE, bool HAS_DL, bool CMP>
cudaError_t launch_one(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                       const MarchPlan& plan, dim3 grid, cudaStream_t s) {
    constexpr size_t smem = Shape<MODE, CMP>::SMEM;
    static SharedMemory shared;
    const cudaError_t e = shared.allow((const void*)rk_mom_march_kernel<MODE, HAS_DL, CMP>, smem);
    if (e != cudaSuccess) return e;
    rk_mom_march_kernel<MODE, HAS_DL, CMP><<<grid, THREADS, smem, s>>>(
        *reinterpret_cast<const CUtensorMap*>(maps.plane1), *reinterpret_cast<const CUtensorMap*>(maps.seam1),
        *reinterpret_cast<const CUtensorMap*>(maps.pt1), kf, io, sp, plan);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_rk_mom_march(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                                const MarchPlan& plan, int mode, cudaStream_t s) {
    const int nk = (kf.km - 1 + TILE_K - 1) / TILE_K;
    const int nj = (kf.jm - 4 + TILE_J - 1) / TILE_J;
    if (nk <= 0 || nj <= 0 || kf.im < 3) return cudaSuccess;
    const bool has_dl = io.dl_in[0] != nullptr;
    const int nha = has_dl ? 9 : 5;
    const int npt_max = mode == MODE_FINAL ? Shape<MODE_FINAL, false>::NPT : Shape<MODE_STAGE, false>::NPT;
    if (mode == MODE_RHS || kf.divu_on || plan.levels < 1 || plan.n_halo != nha || plan.n_pt < N_PT_FIXED ||
        plan.n_pt > npt_max || (mode == MODE_FINAL) != (plan.p_dl >= 0) || plan.withhold < 0)
        return cudaErrorInvalidValue;
    const dim3 grid(nk, nj, (kf.im - 2 + plan.levels - 1) / plan.levels);
    if (mode == MODE_STAGE && plan.compact && plan.n_pt <= Shape<MODE_STAGE, true>::NPT)
        return has_dl ? launch_one<MODE_STAGE, true, true>(maps, kf, io, sp, plan, grid, s)
                      : launch_one<MODE_STAGE, false, true>(maps, kf, io, sp, plan, grid, s);
    if (mode == MODE_STAGE)
        return has_dl ? launch_one<MODE_STAGE, true, false>(maps, kf, io, sp, plan, grid, s)
                      : launch_one<MODE_STAGE, false, false>(maps, kf, io, sp, plan, grid, s);
    return has_dl ? launch_one<MODE_FINAL, true, false>(maps, kf, io, sp, plan, grid, s)
                  : launch_one<MODE_FINAL, false, false>(maps, kf, io, sp, plan, grid, s);
}

}  // namespace atsat
