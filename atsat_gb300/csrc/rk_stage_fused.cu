// One launch per RK stage of the march variant: the blocks of the radial-march momentum kernel (rk_march_body.cuh) and
// those of the TMA-tiled tracer kernel (rk_tracer_body.cuh) in one grid. The two read the same stage input and write
// different fields, so they need no order between them.
#include "rk_march_body.cuh"
#include "rk_tracer_body.cuh"

namespace atsat {

namespace {

static_assert(march::THREADS == tracer::THREADS, "one block size");

struct FusedGrid {
    int nm, nt;                    // momentum blocks, tracer tiles
    int nk, nj, tk, tj;            // their tiles along k and j
    int ng;                        // field groups per tracer tile
};

template <int MODE, int TK>
struct Fused {
    static constexpr bool CMP = MODE == MODE_STAGE;
    static constexpr size_t SMEM = march::Shape<MODE, CMP>::SMEM > tracer::Tile<TK>::SMEM ? march::Shape<MODE, CMP>::SMEM
                                                                                          : tracer::Tile<TK>::SMEM;
};

template <int MODE, bool HAS_DL, int TK>
__global__ void __launch_bounds__(march::THREADS, Fused<MODE, TK>::CMP ? 3 : 2)
rk_stage_fused_kernel(const __grid_constant__ CUtensorMap plane, const __grid_constant__ CUtensorMap plane_seam,
                      const __grid_constant__ CUtensorMap plane_pt, const __grid_constant__ CUtensorMap box,
                      const __grid_constant__ CUtensorMap box_seam, const __grid_constant__ CUtensorMap box_pt,
                      const MixedConstF K, const MixedIO io, const StageParams sp, const MarchPlan mp,
                      const TracerPlan tp, const FusedGrid G) {
    extern __shared__ __align__(128) float smem[];
    // momentum blocks first (they are the longer ones), then the tracer tiles, their field groups side by side
    const bool mom = (int)blockIdx.x < G.nm;
    const int m = mom ? (int)blockIdx.x : (int)blockIdx.x - G.nm, n = mom ? m : m / G.ng, g = m - n * G.ng;
    const int nk = mom ? G.nk : G.tk, nj = mom ? G.nj : G.tj;
    const int bx = n % nk, r = n / nk, by = r % nj, bz = r / nj;
    if (mom)
        march::block<MODE, HAS_DL, Fused<MODE, TK>::CMP>(plane, plane_seam, plane_pt, K, io, sp, mp, smem, bx, by, bz);
    else
        tracer::block<MODE, HAS_DL, TK>(box, box_seam, box_pt, K, io, sp, tp, smem, bx, by, bz, tracer::group_q0(G.ng, g),
                                    tracer::group_q0(G.ng, g + 1));
}

template <int MODE, bool HAS_DL, int TK>
cudaError_t launch_tile(const TileMaps& m, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                       const MarchPlan& mp, const TracerPlan& tp, const FusedGrid& G, cudaStream_t s) {
    constexpr size_t smem = Fused<MODE, TK>::SMEM;
    static SharedMemory shared;
    const cudaError_t e = shared.allow((const void*)rk_stage_fused_kernel<MODE, HAS_DL, TK>, smem);
    if (e != cudaSuccess) return e;
    constexpr int t = TK == 64 ? 0 : 1;
    auto map = [](const unsigned char* p) -> const CUtensorMap& { return *reinterpret_cast<const CUtensorMap*>(p); };
    rk_stage_fused_kernel<MODE, HAS_DL, TK><<<G.nm + G.nt * G.ng, march::THREADS, smem, s>>>(
        map(m.plane1), map(m.seam1), map(m.pt1), map(m.main4[t]), map(m.seam4[t]), map(m.pt4[t]), kf, io, sp, mp, tp, G);
    return cudaGetLastError();
}

template <int MODE, bool HAS_DL>
cudaError_t launch_one(const TileMaps& m, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                       const MarchPlan& mp, const TracerPlan& tp, const FusedGrid& G, cudaStream_t s) {
    return tracer_tile_k(kf.jm, kf.km) == 64 ? launch_tile<MODE, HAS_DL, 64>(m, kf, io, sp, mp, tp, G, s)
                                             : launch_tile<MODE, HAS_DL, 32>(m, kf, io, sp, mp, tp, G, s);
}

// blocks of the momentum kernel and tiles of the tracer kernel
FusedGrid fused_grid(int im, int jm, int km, int levels) {
    FusedGrid G{};
    G.nk = (km - 1 + TILE_K - 1) / TILE_K;
    G.nj = (jm - 4 + TILE_J - 1) / TILE_J;
    if (G.nk <= 0 || G.nj <= 0 || im < 3) return G;
    const int tk = tracer_tile_k(jm, km), tj = 256 / tk;
    G.tk = (km - 1 + tk - 1) / tk;
    G.tj = (jm - 4 + tj - 1) / tj;
    G.nm = G.nk * G.nj * ((im - 2 + levels - 1) / levels);
    G.nt = G.tk * G.tj * ((im - 2 + TTILE_I - 1) / TTILE_I);
    G.ng = tracer_groups(G.nt);
    return G;
}

}  // namespace

// Up to four waves of resident blocks (three per SM) the stage's two kernels are short enough that their launch and
// their thin last waves show: one launch takes two iterations at 10x20x36 from 247 to 214 us, 21x60x121 395 -> 361,
// 21x91x181 575 -> 549, 31x121x241 1063 -> 1018. Beyond, a lone run still gains (41x181x361 replayed 2408 -> 2351 us,
// 61x271x541 7457 -> 7238), but handles that run concurrently fill those waves with each other's blocks already and
// lose (three replaying in turn at 41x181x361 2193 -> 2203 us): the launches stay apart.
// The final stage's momentum blocks need 109 KB (two blocks per SM), so there the line is two waves of those: two
// iterations at 10x20x36 206 -> 188 us, 9x31x61 204 -> 188, 14x40x97 243 -> 238; at four waves 21x91x181 goes 548 -> 581.
// Interleaving the momentum blocks with the tracer blocks, so that both kinds share an SM, is slower the finer it is
// (with the unrolled tracer code, 2489 us apart: every 3rd block 2755, every 4th 2820).
bool stage_fusable(const MixedConstF& kf, const MarchPlan& mp, int mode) {
    if (mode == MODE_RHS || mp.levels < 1) return false;
    const FusedGrid G = fused_grid(kf.im, kf.jm, kf.km, mp.levels);
    if (mode == MODE_FINAL)
        return mp.p_dl >= 0 && mp.n_pt <= march::Shape<MODE_FINAL, false>::NPT && G.nm + G.nt * G.ng <= 2 * 2 * sm_count();
    if (!mp.compact || mp.n_pt > march::Shape<MODE_STAGE, true>::NPT) return false;
    return G.nm + G.nt <= 4 * 3 * sm_count();
}

cudaError_t launch_rk_stage_fused(const TileMaps& maps, const MixedConstF& kf, const MixedIO& io, const StageParams& sp,
                                  const MarchPlan& mp, const TracerPlan& tp, int mode, cudaStream_t s) {
    const bool has_dl = io.dl_in[0] != nullptr;
    if (!stage_fusable(kf, mp, mode) || kf.divu_on || kf.fsz_over_int || mp.n_halo != (has_dl ? 9 : 5) ||
        mp.n_pt < march::N_PT_FIXED || tp.n_items > TRACER_MAX_ITEMS || mp.withhold < 0)
        return cudaErrorInvalidValue;
    const FusedGrid G = fused_grid(kf.im, kf.jm, kf.km, mp.levels);
    if (G.nm + G.nt == 0) return cudaSuccess;
    if (mode == MODE_FINAL)
        return has_dl ? launch_one<MODE_FINAL, true>(maps, kf, io, sp, mp, tp, G, s) : cudaErrorInvalidValue;
    return has_dl ? launch_one<MODE_STAGE, true>(maps, kf, io, sp, mp, tp, G, s)
                  : launch_one<MODE_STAGE, false>(maps, kf, io, sp, mp, tp, G, s);
}

}  // namespace atsat
