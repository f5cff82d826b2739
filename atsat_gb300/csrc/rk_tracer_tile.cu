// Launches of the TMA-tiled tracer kernel on its own (rk_tracer_body.cuh): the split_tiled and tiled2 variants, and the
// march variant where its two kernels do not share a launch (stage_fusable in rk_stage_fused.cu).
#include "rk_tracer_body.cuh"

namespace atsat {

namespace {

using namespace tracer;

template <int MODE, bool HAS_DL, int TK>
__global__ void __launch_bounds__(tracer::THREADS, 3)
rk_tracer_tile_kernel(const __grid_constant__ CUtensorMap map_main, const __grid_constant__ CUtensorMap map_seam,
                      const __grid_constant__ CUtensorMap map_pt, const MixedConstF K, const MixedIO io,
                      const StageParams sp, const TracerPlan plan, const int ng) {
    extern __shared__ __align__(128) float smem[];
    const int bz = blockIdx.z / ng, g = blockIdx.z - bz * ng;
    tracer::block<MODE, HAS_DL, TK>(map_main, map_seam, map_pt, K, io, sp, plan, smem, blockIdx.x, blockIdx.y, bz,
                                group_q0(ng, g), group_q0(ng, g + 1));
}

template <int MODE, bool HAS_DL, int TK>
cudaError_t launch_one(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                       const TracerPlan& plan, cudaStream_t s) {
    static SharedMemory shared;
    const cudaError_t e = shared.allow((const void*)rk_tracer_tile_kernel<MODE, HAS_DL, TK>, Tile<TK>::SMEM);
    if (e != cudaSuccess) return e;
    dim3 grid((kf.km - 1 + TK - 1) / TK, (kf.jm - 4 + Tile<TK>::TJ - 1) / Tile<TK>::TJ, (kf.im - 2 + TI - 1) / TI);
    const int ng = tracer_groups((int64_t)grid.x * grid.y * grid.z), m = TK == 64 ? 0 : 1;
    grid.z *= ng;
    rk_tracer_tile_kernel<MODE, HAS_DL, TK><<<grid, THREADS, Tile<TK>::SMEM, s>>>(
        *reinterpret_cast<const CUtensorMap*>(maps.main4[m]), *reinterpret_cast<const CUtensorMap*>(maps.seam4[m]),
        *reinterpret_cast<const CUtensorMap*>(maps.pt4[m]), kf, io, sp, plan, ng);
    return cudaGetLastError();
}

template <int MODE, bool HAS_DL>
cudaError_t launch_tiles(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                         const TracerPlan& plan, cudaStream_t s) {
    return tracer_tile_k(kf.jm, kf.km) == 64 ? launch_one<MODE, HAS_DL, 64>(maps, kf, io, sp, plan, s)
                                             : launch_one<MODE, HAS_DL, 32>(maps, kf, io, sp, plan, s);
}

}  // namespace

// What bounds a small grid is the serial stream of 13 fields through each of too few blocks (10 tiles at 10x20x36,
// mostly latency). So where the resident blocks (three per SM) outnumber the tiles, the fields of a tile go to several
// blocks, each streaming the winds again: 13, 4 or 2 blocks per tile while all of them are resident at once. Two
// iterations of the march variant (us), a lone state's replays and, after the bar, three states' in turn, whose blocks
// fill idle SMs anyway and pay for the winds:
//   tiles                    1           2           4          13 groups
//      8  10x20x36   185 |  70   148 |  58   132 |  54   114 |  50
//     45  14x40x97   189 | 110   157 | 102   156 | 106   167 | 122
//    108  26x49x97   293 | 193   257 | 184   237 | 186   287 | 242
//    135  61x40x60   331 | 232   299 | 230   309 | 247   351 | 312
//    180  50x21x154  352 | 243   314 | 241   323 | 263   382 | 349
//    240  31x121x61  378 | 284   366 | 287   375 | 307   457 | 411
//    330  21x91x181  453 | 366   454 | 390   474 | 396   605 | 541
int tracer_groups(int64_t tiles) {
    const int64_t slots = 3 * sm_count();
    for (int ng : {13, 4, 2})
        if (tiles * ng <= slots) return ng;
    return 1;
}

// 64 x 4 tiles read a halo a tenth smaller per cell and in longer rows than 32 x 8, so they are taken unless they pad
// the grid by more (a ring of 66 meridians fills 128 columns of 64-wide tiles, 96 of 32-wide ones): two iterations (us)
// at 41x181x361 (the same padding) 2194 with 64 against 2221 with 32, at 81x361x721 (276480 columns against 264960)
// 16640 against 16500.
int tracer_tile_k(int jm, int km) {
    auto cells = [&](int tk, int tj) { return (int64_t)((km - 1 + tk - 1) / tk * tk) * ((jm - 4 + tj - 1) / tj * tj); };
    return cells(64, 4) <= cells(32, 8) ? 64 : 32;
}

cudaError_t launch_rk_tracer_tile(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io,
                                  const StageParams& sp, const TracerPlan& plan, int mode, cudaStream_t s) {
    if (kf.km < 2 || kf.jm < 5 || kf.im < 3) return cudaSuccess;
    if (mode == MODE_RHS || kf.divu_on || kf.fsz_over_int || plan.n_items > TRACER_MAX_ITEMS) return cudaErrorInvalidValue;
    const bool has_dl = io.dl_in[0] != nullptr;
    if (mode == MODE_STAGE)
        return has_dl ? launch_tiles<MODE_STAGE, true>(maps, kf, io, sp, plan, s)
                      : launch_tiles<MODE_STAGE, false>(maps, kf, io, sp, plan, s);
    return has_dl ? launch_tiles<MODE_FINAL, true>(maps, kf, io, sp, plan, s) : cudaErrorInvalidValue;
}

// the number of items the kernel consumes (the host's plan must match)
int tracer_plan_items(int mode, bool has_dl, bool turb) {
    int n = n_state(has_dl);
    for (int q = ATSAT_F_H2O; q < NPROG; q++) {
        if (turb_field(q) && !turb) continue;
        n += (has_dl ? 2 : 1) + n_pt(mode, q);
    }
    return n;
}

}  // namespace atsat
