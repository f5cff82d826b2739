// Launches of the TMA-tiled tracer kernel on its own (rk_tracer_body.cuh): the split_tiled and tiled2 variants and the
// march variant's final stage. The march variant's intermediate stages run it fused (rk_stage_fused.cu).
#include "rk_tracer_body.cuh"

namespace atsat {

namespace {

using namespace tracer;

template <int MODE, bool HAS_DL, int NG>
__global__ void __launch_bounds__(tracer::THREADS, 3)
rk_tracer_tile_kernel(const __grid_constant__ CUtensorMap map_main, const __grid_constant__ CUtensorMap map_seam,
                      const __grid_constant__ CUtensorMap map_pt, const MixedConstF K, const MixedIO io,
                      const StageParams sp, const TracerPlan plan) {
    extern __shared__ __align__(128) float smem[];
    const int bz = blockIdx.z / NG;
    tracer::group_block<MODE, HAS_DL, NG>(map_main, map_seam, map_pt, K, io, sp, plan, smem, blockIdx.x, blockIdx.y, bz,
                                          blockIdx.z - bz * NG);
}

template <int MODE, bool HAS_DL, int NG>
cudaError_t launch_groups(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                          const TracerPlan& plan, dim3 grid, cudaStream_t s) {
    static bool attr = false;
    if (!attr) {
        const cudaError_t e = cudaFuncSetAttribute(rk_tracer_tile_kernel<MODE, HAS_DL, NG>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    grid.z *= NG;
    rk_tracer_tile_kernel<MODE, HAS_DL, NG><<<grid, THREADS, SMEM_BYTES, s>>>(
        *reinterpret_cast<const CUtensorMap*>(maps.main4), *reinterpret_cast<const CUtensorMap*>(maps.seam4),
        *reinterpret_cast<const CUtensorMap*>(maps.pt4), kf, io, sp, plan);
    return cudaGetLastError();
}

template <int MODE, bool HAS_DL>
cudaError_t launch_one(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                       const TracerPlan& plan, dim3 grid, cudaStream_t s) {
    switch (tracer_groups((int64_t)grid.x * grid.y * grid.z)) {
        case 13: return launch_groups<MODE, HAS_DL, 13>(maps, kf, io, sp, plan, grid, s);
        case 4: return launch_groups<MODE, HAS_DL, 4>(maps, kf, io, sp, plan, grid, s);
        default: return launch_groups<MODE, HAS_DL, 1>(maps, kf, io, sp, plan, grid, s);
    }
}

}  // namespace

// What bounds a small grid is the serial stream of 13 fields through each of too few blocks (8 tiles at 10x20x36:
// 22.8 us per intermediate launch, 38.6 us at the final stage, mostly latency). So where the resident blocks (three
// per SM) outnumber the tiles, the fields of a tile go to several blocks, each streaming the winds again: 13 blocks
// per tile while all of them are resident at once, 4 while they make at most two waves. Two iterations of the march
// variant (us): 10x20x36 309 -> 240 with 13 groups (261 with 4), 9x31x61 294 -> 246 (250), 14x40x97 301 -> 279 with 4
// (342 with 13), 21x60x121 451 -> 420 with 4 (615 with 13), 21x91x181 587 with one group (675 with 4).
int tracer_groups(int64_t tiles) {
    const int64_t slots = 3 * sm_count();
    return tiles * 13 <= slots ? 13 : (tiles * 4 <= 2 * slots ? 4 : 1);
}

cudaError_t launch_rk_tracer_tile(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io,
                                  const StageParams& sp, const TracerPlan& plan, int mode, cudaStream_t s) {
    const int nk = (kf.km - 1 + TILE_K - 1) / TILE_K;
    const int nj = (kf.jm - 4 + TILE_J - 1) / TILE_J;
    const int ni = (kf.im - 2 + TI - 1) / TI;
    if (nk <= 0 || nj <= 0 || ni <= 0) return cudaSuccess;
    if (mode == MODE_RHS || kf.divu_on || kf.fsz_over_int || plan.n_items > TRACER_MAX_ITEMS) return cudaErrorInvalidValue;
    const dim3 grid(nk, nj, ni);
    const bool has_dl = io.dl_in[0] != nullptr;
    if (mode == MODE_STAGE)
        return has_dl ? launch_one<MODE_STAGE, true>(maps, kf, io, sp, plan, grid, s)
                      : launch_one<MODE_STAGE, false>(maps, kf, io, sp, plan, grid, s);
    cudaError_t e = has_dl ? launch_one<MODE_FINAL, true>(maps, kf, io, sp, plan, grid, s)
                           : launch_one<MODE_FINAL, false>(maps, kf, io, sp, plan, grid, s);
    if (e != cudaSuccess) return e;
    return launch_final_combine(kf, io, ATSAT_F_H2O, kf.turb ? ATSAT_F_DIS : ATSAT_F_NH4SH, s);
}

// the number of items the kernel consumes (the host's plan must match)
int tracer_plan_items(int mode, bool has_dl, bool turb) {
    int n = has_dl ? 8 : 5;
    for (int q = ATSAT_F_H2O; q < NPROG; q++) {
        if (turb_field(q) && !turb) continue;
        n += (has_dl ? 2 : 1) + ((mode == MODE_FINAL) ? n_pt<MODE_FINAL>(q) : n_pt<MODE_STAGE>(q));
    }
    return n;
}

}  // namespace atsat
