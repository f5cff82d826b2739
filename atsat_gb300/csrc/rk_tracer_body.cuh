// TMA-tiled RK stage of the 13 tracer fields (h2o .. nh4sh, tke, dis: RHS_Sat_Turb.cpp:580-1000 with the
// stage handling of RungeKutta_Sat_Turb.cpp:250-375), run after the momentum / temperature kernel of the
// split variant (rk_mixed.cu) when species_divu is off.
//
// A block owns TK x 256 / TK x 4 cells (k, j, i), TK 64 or 32 (tracer_tile_k). A producer warp streams every array
// the tracers read with tensor copies, in groups: the advecting winds and the eddy viscosity (three groups of point
// boxes, without a halo), then one group per field: the halo boxes (72 x 6 x 6 or 40 x 10 x 6 floats) of its y_n copy
// and stage increment and the point boxes of its sources, the tke/dis running sum and, at the final stage, dl_1 and
// dl_2. A group has one "full" barrier for all of its copies and one "empty" barrier; with increments two groups are
// in flight, without four. Eight consumer warps (32 columns of a row j, four radial levels per lane) read the boxes
// from shared memory; at the final stage each lane loads its y_n (FP64) before it waits for the field's boxes and forms
// y_{n+1} there. A block needs 73 KB of shared memory and 72 registers a thread: three blocks fit on an SM.
//
// What bounds it: memory (84-88 % of a plain copy's rate at 41x181x361) and, close behind, issue (60 %). Launches at
// 41x181x361, before -> now: intermediate with increments 144 -> 134 us, final stage with its FP64 half 184 + 118 ->
// 255 us. Prefetching the next groups into L2 did not help (2209-2240 us a step pair against 2193).
//
// The fields run through three copies of the code (one source, two sources, tke / dis) in a loop that is not
// unrolled. With one copy per field the program was 90 KB: at the final stage a warp in eight waited for instructions,
// and with the FP64 half in it most did (419 us at 41x181x361), which is why that half was a kernel of its own.
//
// The arithmetic is mixed_physics.cuh's scalar() with its constant factors folded: with the raw
// differences a0..a5 of the field (each part differenced on its own),
//   transport = (u / 2dr) a0 + (v / (2 dtheta rm)) a2 + (w / (2 dphi rm sin)) a4
//   diffusion = a1 / dr^2 + (two_inv_rm / 2dr) a0 + (inv_rm2 / dtheta^2) a3
//             + (costhe_inv_rm2sinthe / 2dtheta) a2 + (inv_rm2sinthe2 / dphi^2) a5
// (per-cell wind factors, per-column diffusion factors), r = kappa diffusion - transport + sources.
//
// The block's body is a device function, so that a launch of its own (rk_tracer_tile.cu) and the fused stage launch
// (rk_stage_fused.cu) run the same code.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "mixed_physics.cuh"
#include "tma_pipe.cuh"

namespace atsat {
namespace tracer {

using namespace mixed;
using namespace tma;

constexpr int TI = TTILE_I;                               // 4 radial levels per thread
constexpr int NHS = 4, NPS = 7;                           // halo and point slots
constexpr int NCW = 8;                                    // consumer warps
constexpr int THREADS = (NCW + 1) * 32;
constexpr int GEO_F = TI * NCW * 16;                      // ColGeoF of each warp's four columns
constexpr int COEF_F = TI * NCW * 4;                      // their four diffusion factors

// a tile TK cells wide (k), 256 / TK rows, TI levels
template <int TK>
struct Tile {
    static constexpr int TJ = 256 / TK, BX = TK + 8, BY = TJ + 2;
    static constexpr int PL = BX * BY;                    // floats per plane of a halo box
    static constexpr int BOX_F = PL * TTILE_BZ, SEAM_F = TILE_SEAM_X * TJ * TI;
    static constexpr int HSLOT_F = (BOX_F + SEAM_F + 31) / 32 * 32;
    static constexpr int PP = TK * TJ, PSLOT_F = PP * TI; // floats per plane of a point box, per box
    static constexpr uint32_t BOX_BYTES = BOX_F * 4, SEAM_BYTES = SEAM_F * 4, PT_BYTES = PSLOT_F * 4;
    static constexpr int WPR = TK / 32;                   // warps per row
    static constexpr size_t SMEM = (size_t)NHS * HSLOT_F * 4 + (size_t)NPS * PSLOT_F * 4 + (size_t)(GEO_F + COEF_F) * 4
                                 + 2 * NHS * 8;
    static_assert((HSLOT_F * 4) % 128 == 0 && (PSLOT_F * 4) % 128 == 0 && (BOX_F * 4) % 128 == 0, "slot alignment");
    static_assert(WPR * TJ == NCW && 3 * (SMEM + 1024) <= 228 * 1024, "three blocks per SM");
};

// ---- the stream layout (the host builds the same, make_plan_tracer) ----
constexpr int NTRACER = NPROG - ATSAT_F_H2O;
__host__ __device__ constexpr bool turb_field(int q) { return q == ATSAT_F_TKE || q == ATSAT_F_DIS; }
__host__ __device__ constexpr int n_src(int q) { return (q == ATSAT_F_NH3 || q == ATSAT_F_NH4SH) ? 2 : 1; }
__host__ __device__ constexpr int n_pt(int mode, int q) {
    return n_src(q) + (turb_field(q) ? 1 : 0) + ((mode == MODE_FINAL && !turb_field(q)) ? 2 : 0);
}
// the wind groups' point boxes: u, [du] | v, [dv], nue | w, wlo, [dw]
constexpr int NWIND = TRACER_WIND_GROUPS;
__host__ __device__ constexpr int n_wind(bool dl, int g) { return (g == 0 ? 1 : 2) + (dl ? 1 : 0); }
__host__ __device__ constexpr int n_state(bool dl) { return n_wind(dl, 0) + n_wind(dl, 1) + n_wind(dl, 2); }
__host__ __device__ constexpr int groups_ahead(bool dl) { return dl ? 2 : 4; }   // NHS halo boxes
// Field group g of ng: the tracers [group_q0(g), group_q0(g + 1)).
__host__ __device__ constexpr int group_q0(int ng, int g) { return ATSAT_F_H2O + NTRACER * g / ng; }

// Point slots are handed out in stream order, and a group waits for the release of the group groups_ahead before it:
// so any groups_ahead consecutive groups of a block's stream must fit the point slots.
constexpr bool slots_fit(int mode, bool dl, int ng) {
    for (int g = 0; g < ng; g++) {
        int n[NWIND + NTRACER] = {}, m = 0;
        for (int w = 0; w < NWIND; w++) n[m++] = n_wind(dl, w);
        for (int q = group_q0(ng, g); q < group_q0(ng, g + 1); q++) n[m++] = n_pt(mode, q);
        for (int a = 0; a < m; a++) {
            int s = 0;
            for (int b = a; b < m && b < a + groups_ahead(dl); b++) s += n[b];
            if (s > NPS) return false;
        }
    }
    return true;
}
constexpr bool slots_fit(int ng) {
    return slots_fit(MODE_STAGE, false, ng) && slots_fit(MODE_STAGE, true, ng) && slots_fit(MODE_FINAL, true, ng);
}
static_assert(slots_fit(1) && slots_fit(2) && slots_fit(4) && slots_fit(13), "point slots");

// One array's stencil of a lane's column of TI cells: the centre values at i-1 and i stay in registers from cell to
// cell, so a cell costs five shared loads instead of seven.
template <int TK>
struct Column {
    static constexpr int PL = Tile<TK>::PL, BX = Tile<TK>::BX;
    float rn, x;                   // the values at i-1 and i

    __device__ __forceinline__ void start(const float* s, int o) {
        rn = s[o - PL];
        x = s[o];
    }
    // the raw differences of cell i; returns its centre value and moves on to i+1
    __device__ __forceinline__ float d7(const float* s, int o, int ow, int oe, float* e) {
        const float rp = s[o + PL];
        const float tp = s[o + BX], tn = s[o - BX];
        const float pe = s[oe], pw = s[ow];
        const float c = x;
        e[0] = rp - rn;
        e[1] = rp - 2.0f * c + rn;
        e[2] = tp - tn;
        e[3] = tp - 2.0f * c + tn;
        e[4] = pe - pw;
        e[5] = pe - 2.0f * c + pw;
        rn = c;
        x = rp;
        return c;
    }
};

// A global store that the compiler may move shared loads across (a plain one could alias them as far as it knows, and
// each cell's loads would wait for the stores of the cell before); it stays ahead of the slot's release, which is
// volatile too.
__device__ __forceinline__ void store(float* p, float x) {
    asm volatile("st.global.f32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "f"(x));
}
__device__ __forceinline__ void store(double* p, double x) {
    asm volatile("st.global.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "d"(x));
}

// the tracers [q0, q1) of tile (bx, by, bz): the winds' groups, then those fields' groups of the plan
template <int MODE, bool HAS_DL, int TK>
__device__ __forceinline__ void block(const CUtensorMap& map_main, const CUtensorMap& map_seam, const CUtensorMap& map_pt,
                                      const MixedConstF& K, const MixedIO& io, const StageParams& sp,
                                      const TracerPlan& plan, float* smem, int bx, int by, int bz, int q0, int q1) {
    static_assert(MODE == MODE_STAGE || (MODE == MODE_FINAL && HAS_DL), "stages of the stream layout");
    constexpr int NH = HAS_DL ? 2 : 1, AHEAD = groups_ahead(HAS_DL);
    using T = Tile<TK>;
    constexpr int TJ = T::TJ, PL = T::PL, BOX_F = T::BOX_F, HSLOT_F = T::HSLOT_F, PSLOT_F = T::PSLOT_F, PP = T::PP;
    float* hs = smem;
    float* ps = hs + NHS * HSLOT_F;
    float* sgeo = ps + NPS * PSLOT_F;
    float* scoef = sgeo + GEO_F;
    uint64_t* bars = reinterpret_cast<uint64_t*>(scoef + COEF_F);
    const Ring rg{smem_u32(bars), smem_u32(bars + AHEAD)};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int k0 = bx * TK;
    const int j0 = 2 + by * TJ;
    const int i0 = 1 + bz * TI;
    int seam = 0, xs = 0;
    if (k0 == 0 && K.km - 2 > k0 + TK + 3) { seam = 1; xs = (K.km - 2) & ~3; }
    else if (k0 > 0 && K.km - 2 >= k0 && K.km - 2 < k0 + TK) { seam = 2; xs = 0; }

    if (smem_u32(smem) & 127u) {
        if (threadIdx.x == 0) atomicOr(plan.err, ERR_ALIGN);
        return;
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < AHEAD; s++) { mbar_init(rg.full(s), 1); mbar_init(rg.empty(s), NCW); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    const int q_end = K.turb ? q1 : (q1 < ATSAT_F_TKE ? q1 : ATSAT_F_TKE);   // tke and dis come last

    if (warp == NCW) {
        // ---- producer: the plan's groups in order ----
        if (lane == 0) {
            const int ng = NWIND + (q_end > q0 ? q_end - q0 : 0);
            const int last = plan.first[NWIND + (q_end > q0 ? q_end : q0) - ATSAT_F_H2O] - plan.withhold;
            int n = 0, pslot = 0;
            bool ok = true;
            for (; n < ng; n++) {
                const int g = n < NWIND ? n : n + (q0 - ATSAT_F_H2O);
                const int m0 = plan.first[g], m1 = plan.first[g + 1], nh = n < NWIND ? 0 : NH, s = n % AHEAD;
                if (m1 > last) break;                       // withheld
                if (n >= AHEAD && !mbar_wait(rg.empty(s), (uint32_t)(((n / AHEAD) - 1) & 1), plan.wait_limit)) {
                    ok = false;
                    break;
                }
                const uint32_t bar = rg.full(s);
                mbar_expect_tx(bar, nh * (T::BOX_BYTES + (seam ? T::SEAM_BYTES : 0u)) + (m1 - m0 - nh) * T::PT_BYTES);
                for (int m = m0; m < m0 + nh; m++) {
                    const uint32_t dst = smem_u32(hs + (s * NH + m - m0) * HSLOT_F);
                    tma_load_4d(dst, &map_main, k0 - 4, j0 - 1, i0 - 1, plan.arr[m], bar);
                    if (seam) tma_load_4d(dst + T::BOX_BYTES, &map_seam, xs, j0, i0, plan.arr[m], bar);
                }
                for (int m = m0 + nh; m < m1; m++) {
                    tma_load_4d(smem_u32(ps + pslot * PSLOT_F), &map_pt, k0, j0, i0, plan.arr[m], bar);
                    pslot = pslot + 1 == NPS ? 0 : pslot + 1;
                }
            }
            if (!ok) atomicOr(plan.err, ERR_PRODUCER);
            // a copy in flight lands by itself: none may land after the block is gone
            for (int m = (n > AHEAD ? n - AHEAD : 0); m < n; m++)
                if (!mbar_wait(rg.full(m % AHEAD), (uint32_t)((m / AHEAD) & 1))) break;
        }
        return;
    }

    // ---- consumers ----
    const int row_j = warp / T::WPR, kl = warp % T::WPR * 32 + lane;   // the lane's place in the tile
    const int j = j0 + row_j, k = k0 + kl;
    {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int e = lane + 32 * h;
            const int ii = e >> 4, f = e & 15;
            const int i = i0 + ii;
            float v = 0.0f;
            if (i < K.im && j < K.jm) v = __ldg(reinterpret_cast<const float*>(io.geof + ((int64_t)i * K.jm + j)) + f);
            sgeo[(ii * NCW + warp) * 16 + f] = v;
        }
        __syncwarp();
        if (lane < TI) {
            const ColGeoF& g = *reinterpret_cast<const ColGeoF*>(sgeo + (lane * NCW + warp) * 16);
            float* cf = scoef + (lane * NCW + warp) * 4;
            cf[0] = K.inv_2dr * g.two_inv_rm;
            cf[1] = K.inv_dthe2 * g.inv_rm2;
            cf[2] = K.inv_2dthe * g.costhe_inv_rm2sinthe;
            cf[3] = K.inv_dphi2 * g.inv_rm2sinthe2;
        }
        __syncwarp();
    }
    // the lane's cells: c0 + ii plane for ii < nv; their places in a halo box: o + ii PL, the neighbours in k at
    // ow + ii ows and oe + ii oes (in the seam box for the periodic partner)
    const int nv = (k <= K.km - 2 && j <= K.jm - 3) ? K.im - 1 - i0 : 0;
    const int c0 = (i0 * K.jm + j) * K.kp + k, plane = (int)K.plane;
    const int row = PL + (row_j + 1) * T::BX;
    const int o = row + kl + 4;
    int ow = o - 1, oe = o + 1, ows = PL, oes = PL;
    if (k == 0) {
        if (seam == 1) { ow = BOX_F + row_j * TILE_SEAM_X + ((K.km - 2) - xs); ows = TJ * TILE_SEAM_X; }
        else ow = row + (K.km - 2) - (k0 - 4);
    }
    if (k == K.km - 2) {
        if (seam == 2) { oe = BOX_F + row_j * TILE_SEAM_X + (0 - xs); oes = TJ * TILE_SEAM_X; }
        else oe = row + 0 - (k0 - 4);
    }
    const int px = row_j * TK + kl;                      // the lane's place in a point box's plane
    auto wait = [&](int n) -> bool {
        const bool ok = mbar_wait(rg.full(n % AHEAD), (uint32_t)((n / AHEAD) & 1), plan.wait_limit);
        if (!__any_sync(0xffffffffu, !ok)) return true;
        if (lane == 0) atomicOr(plan.err, ERR_CONSUMER);
        return false;
    };
    auto release = [&](int n) {
        __syncwarp();
        if (lane == 0) mbar_arrive(rg.empty(n % AHEAD));
    };

    // ---- the winds and the eddy viscosity: point boxes u, [du] | v, [dv], nue | w, wlo, [dw] ----
    float tu[TI], tv[TI], tw[TI], nts[TI], nuec[TI];
    {
        constexpr int sV = n_wind(HAS_DL, 0), sW = sV + n_wind(HAS_DL, 1);
        const float* p = ps + px;
        auto P = [&](int slot, int ii) { return p[(slot % NPS) * PSLOT_F + ii * PP]; };
        if (!wait(0)) return;
#pragma unroll
        for (int ii = 0; ii < TI; ii++) {
            const float u = HAS_DL ? P(0, ii) + P(1, ii) : P(0, ii);
            tu[ii] = u * K.inv_2dr;
        }
        slot_reads_done();
        release(0);
        if (!wait(1)) return;
#pragma unroll
        for (int ii = 0; ii < TI; ii++) {
            const float v = HAS_DL ? P(sV, ii) + P(sV + 1, ii) : P(sV, ii);
            const ColGeoF& g = *reinterpret_cast<const ColGeoF*>(sgeo + (ii * NCW + warp) * 16);
            tv[ii] = v * (K.inv_2dthe * g.inv_rm);
            const float nue_c = P(sW - 1, ii);
            const float nue_t = (K.turb_coupling != 0.0f && isfinite(nue_c)) ? K.turb_coupling * smaxf(0.0f, nue_c) : 0.0f;
            nts[ii] = nue_t * K.inv_pr_t;
            nuec[ii] = nue_c;
        }
        slot_reads_done();
        release(1);
        // w = (y_n + low word) + increment
        if (!wait(2)) return;
#pragma unroll
        for (int ii = 0; ii < TI; ii++) {
            float w = P(sW, ii) + P(sW + 1, ii);
            if (HAS_DL) w = w + P(sW + 2, ii);
            const ColGeoF& g = *reinterpret_cast<const ColGeoF*>(sgeo + (ii * NCW + warp) * 16);
            tw[ii] = w * (K.inv_2dphi * g.inv_rmsinthe);
        }
        slot_reads_done();
        release(2);
    }

    int pslot = n_state(HAS_DL) % NPS;                        // the next point slot
    // field q, group n of the stream
    auto field = [&](auto nsrc, auto is_turb_field, int q, int n) -> bool {
        constexpr int NSRC = decltype(nsrc)::value;
        constexpr bool TURB = decltype(is_turb_field)::value;
        constexpr int NPT = NSRC + (TURB ? 1 : 0) + ((MODE == MODE_FINAL && !TURB) ? 2 : 0);
        double yn64[TI];                                      // the final stage's y_n: in flight during the wait
        if (MODE == MODE_FINAL) {
            const double* y = io.yn64[q] + c0;
#pragma unroll
            for (int ii = 0; ii < TI; ii++) yn64[ii] = ii < nv ? ldd(y + (int64_t)ii * plane) : 0.0;
        }
        const TracerField F = plan.fld[q - ATSAT_F_H2O];
        if (!wait(n)) return false;
        const float* Y = hs + (n % AHEAD) * NH * HSLOT_F;
        const float* D = Y + HSLOT_F;
        const float* P[NPT];
#pragma unroll
        for (int m = 0; m < NPT; m++) {
            P[m] = ps + pslot * PSLOT_F + px;
            pslot = pslot + 1 == NPS ? 0 : pslot + 1;
        }
        Column<TK> cy, cd;
        cy.start(Y, o);
        if (HAS_DL) cd.start(D, o);
#pragma unroll
        for (int ii = 0; ii < TI; ii++) {
            // cells outside the interior compute on the box's zeros and store nothing
            float a[6];
            const float yn_c = cy.d7(Y, o + ii * PL, ow + ii * ows, oe + ii * oes, a);
            float dl_c = 0.0f;
            if (HAS_DL) {
                float b[6];
                dl_c = cd.d7(D, o + ii * PL, ow + ii * ows, oe + ii * oes, b);
#pragma unroll
                for (int r = 0; r < 6; r++) a[r] += b[r];
            }
            const float* cf = scoef + (ii * NCW + warp) * 4;
            const float df = K.inv_dr2 * a[1] + cf[0] * a[0] + cf[1] * a[3] + cf[2] * a[2] + cf[3] * a[5];
            const float tr = tu[ii] * a[0] + tv[ii] * a[2] + tw[ii] * a[4];
            float S = F.w0 * P[0][ii * PP];
            if (NSRC == 2) S = fmaf(F.w0, P[0][ii * PP], F.w1 * P[1][ii * PP]);
            const float kap = TURB ? F.kap0 + nuec[ii] * F.inv_sig : F.kap0 + nts[ii];
            const float r = kap * df - tr + S;
            const int cc = c0 + ii * plane;
            if (MODE == MODE_STAGE) {
                const float cr = sp.c_in_f * r;
                float d = cr;
                if (TURB) {
                    const float accv = P[NSRC][ii * PP];
                    const float acc = (sp.stage == 0) ? sp.wgt_f * r : accv + sp.wgt_f * r;
                    if (ii < nv) store(io.acc_turb[q - ATSAT_F_TKE] + cc, acc);
                    const float y = yn_c + cr;
                    const float yc = (q == ATSAT_F_TKE) ? sminf(smaxf(y, 0.0f), K.tke_max) : smaxf(y, K.dis_min);
                    d = yc - yn_c;
                }
                if (ii < nv) store(io.dl_out[q] + cc, d);
            } else {
                // y_{n+1} = y_n + increment: the increment in FP32, the sum in FP64
                float inc;
                if (TURB) inc = sp.sixth_dt_f * (P[1][ii * PP] + r);
                else inc = THIRD * (P[NSRC][ii * PP] + 2.0f * P[NSRC + 1][ii * PP] + dl_c) + sp.sixth_dt_f * r;
                double y = yn64[ii] + f2d(inc);
                if (TURB) y = (q == ATSAT_F_TKE) ? smin(smax(y, 0.0), K.tke_max_d) : smax(y, K.dis_min_d);
                if (ii < nv) {
                    store(io.out64[q] + cc, y);
                    if (io.out32[q]) store(io.out32[q] + cc, d2f(y));
                    if (sp.write_all_rhs) store(io.rhs[q] + cc, f2d(r));
                }
            }
        }
        release(n);
        return true;
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
#pragma unroll 1
    for (int q = q0, n = NWIND; q < q_end; q++, n++) {
        const bool ok = turb_field(q) ? field(One{}, std::true_type{}, q, n)
                      : n_src(q) == 2 ? field(Two{}, std::false_type{}, q, n)
                                      : field(One{}, std::false_type{}, q, n);
        if (!ok) return;
    }
    if (MODE == MODE_FINAL && q1 == NPROG && !K.turb && sp.write_all_rhs) {
#pragma unroll
        for (int ii = 0; ii < TI; ii++)
            if (ii < nv) {
                io.rhs[ATSAT_F_TKE][c0 + ii * plane] = 0.0;
                io.rhs[ATSAT_F_DIS][c0 + ii * plane] = 0.0;
            }
    }
}

}  // namespace tracer
}  // namespace atsat
