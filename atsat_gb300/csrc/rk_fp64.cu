// FP64 drop-in kernels of RungeKuttaSat (planet/RungeKutta_Sat_Turb.cpp:110-387) and RHSSat
// (planet/RHS_Sat_Turb.cpp:25-1016).
//
// One fused kernel per RK stage: every thread owns one cell of the RK interior
// (i = 1..im-2, j = 2..jm-3, k = 0..km-2 with the periodic seam), evaluates the full right-hand side
// of the 17 prognostic fields from the stage input Y_s, folds it into the FP64 accumulator and
// writes the next stage input Y_{s+1} = y_n + c_in * rhs (the reference's pass A and pass B,
// :220-320, in one pass over memory). The last stage writes y_{n+1} = y_n + dt/6 * acc directly
// (:324-375). Y_s and Y_{s+1} live in different buffers, so no cell reads a half-updated
// neighbour -- the property the reference's separated passes exist for (:178-202).
//
// The arithmetic follows the reference's expressions. Divisions by configuration constants are
// multiplications by reciprocals formed on the host, and exp_rm (identically 1: ATSAT has no radial
// stretching) is not multiplied; both change results by at most an ulp per operation.
#include "dyn_common.cuh"

namespace atsat {

namespace {

__device__ __forceinline__ double ldg(const double* p) { return __ldg(p); }

__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }

// Comparisons on the integer pipe: GB300's FP64 pipe issues two operations per SM per cycle and a DSETP takes a
// slot like an addition. Each test settles the common case on the double's high word and leaves the rest to the
// comparison itself.
__device__ __forceinline__ uint32_t hi_word(double x) {
    uint32_t lo, hi;
    split_f64(x, lo, hi);
    return hi;
}
__device__ __forceinline__ bool finite(double x) { return (hi_word(x) & 0x7FF00000u) != 0x7FF00000u; }
// true: lim < x < inf for sure (lim > 0); false: unknown
__device__ __forceinline__ bool surely_above(double x, double lim) { return hi_word(x) - hi_word(lim) - 1u < 0x7FEFFFFFu - hi_word(lim); }
// max(0, x) of a finite x, +0 for x = -0
__device__ __forceinline__ double positive(double x) { return (hi_word(x) >> 31) ? 0.0 : x; }
// x clipped to [-0.5, 0.5], 0 where x is not finite
__device__ __forceinline__ double clip_half(double x) {
    const uint32_t a = hi_word(x) & 0x7FFFFFFFu;
    if (a < 0x3FE00000u) return x;
    if (a >= 0x7FF00000u) return 0.0;
    return (hi_word(x) >> 31) ? -0.5 : 0.5;
}

// The tendency r of field q into the state; `out` the tendency as it is written where it is asked for. What is written
// must not change the state, so the sums are pinned: every instance rounds them alike.
template <int MODE>
__device__ __forceinline__ void emit(const StageIO<double>& io, const StageParams& sp, const KConst& K, int q,
                                     int64_t c, double r, double out) {
    if (MODE == MODE_RHS) {
        io.rhs[q][c] = out;
        return;
    }
    double y;
    if (MODE == MODE_STAGE) {
        const double a = fma(sp.wgt, r, (sp.stage == 0) ? 0.0 : io.acc[q][c]);
        io.acc[q][c] = a;
        y = fma(sp.c_in, r, ldg(io.yn[q] + c));
    } else {
        const double a = fma(sp.wgt, r, io.acc[q][c]);
        y = fma(sp.sixth_dt, a, ldg(io.yn[q] + c));
        if (sp.write_all_rhs || q < 3) io.rhs[q][c] = out;
    }
    if (q == ATSAT_F_TKE) {
        if (hi_word(y) >= hi_word(K.tke_max)) y = smin(smax(y, 0.0), K.tke_max);
    } else if (q == ATSAT_F_DIS) {
        if (!surely_above(y, K.dis_min)) y = smax(y, K.dis_min);
    }
    io.out[q][c] = y;
}

// The stencil of one field: the centre and its six neighbours.
struct S7 { double c, rp, rm, tp, tm, pe, pw; };

__device__ __forceinline__ S7 stencil(const double* __restrict__ f, int64_t c, int64_t plane, int kp, int dkw, int dke) {
    return S7{ldg(f + c), ldg(f + c + plane), ldg(f + c - plane), ldg(f + c + kp), ldg(f + c - kp), ldg(f + c + dke),
              ldg(f + c + dkw)};
}
// neighbours minus the centre
__device__ __forceinline__ S7 centred(const S7& f) {
    return S7{f.c, f.rp - f.c, f.rm - f.c, f.tp - f.c, f.tm - f.c, f.pe - f.c, f.pw - f.c};
}

// kappa diffusion - transport of a field as one weight per stencil value (the transport's weights sum to zero
// over the neighbours, the diffusion's centre weight is kappa l_0).
struct Wt { double rp, rm, tp, tm, pe, pw, c; };

__device__ __forceinline__ Wt weights(double kappa, double U, double V, double W, const StageGeo& g) {
    return Wt{fma(kappa, g.l_rp, -U), fma(kappa, g.l_rm, U), fma(kappa, g.l_tp, -V), fma(kappa, g.l_tm, V),
              fma(kappa, g.l_p, -W), fma(kappa, g.l_p, W), kappa * g.l_0};
}

// sum over the neighbours of weight times difference to the centre
__device__ __forceinline__ double apply_centred(const Wt& w, const S7& d) {
    return fma(w.rp, d.rp, fma(w.rm, d.rm, fma(w.tp, d.tp, fma(w.tm, d.tm, fma(w.pe, d.pe, w.pw * d.pw)))));
}
// the same and `extra`, first in the chain: no operation of its own, but six roundings at its size
__device__ __forceinline__ double apply_centred(const Wt& w, const S7& d, double extra) {
    return fma(w.rp, d.rp, fma(w.rm, d.rm, fma(w.tp, d.tp, fma(w.tm, d.tm, fma(w.pe, d.pe, fma(w.pw, d.pw, extra))))));
}
// the same on the values themselves
__device__ __forceinline__ double apply_values(const Wt& w, const S7& f, double extra) {
    return fma(w.rp, f.rp, fma(w.rm, f.rm, fma(w.tp, f.tp, fma(w.tm, f.tm,
           fma(w.pe, f.pe, fma(w.pw, f.pw, fma(w.c, f.c, extra)))))));
}

// The default switches: metric split on, no hydro-buoyancy, no legacy buoyancy, no radiation or thermal-mass-flux
// source, no flux-form species term, and couplings of exactly 1 (whose products are the factors themselves).
bool plain_knobs(const KConst& K) {
    return K.metric_split && !K.hydro_buoy && !K.buoy_legacy && !K.rad_on && !K.tmf_on && !K.divu_on &&
           K.precip_coupling == 1.0 && K.chem == 1.0 && K.turb_coupling == 1.0;
}

// Rows of 32 cells per block and blocks per SM: 4 x 128 threads at 128 registers, no spills. The two-iteration
// step at 41x181x361 took 13.36 ms with 2 x 256, 13.21 with 4 x 128, 13.24 / 13.27 / 13.29 with 5 / 6 / 8 x 128
// (spilling), 15.05 with 1 x 256: a few warps fill the FP64 pipe, the finer blocks even out the last wave.
constexpr int RKS_ROWS = 4, RKS_BLOCKS = 4;

// What bounds it: the FP64 pipe (two operations per SM per cycle). With the differences of each field scaled and
// combined one by one it was 590 FP64 instructions per interior cell and 2.38 ms per launch at 41x181x361, while
// the launch's 1.97 GB take 0.29 ms. So the kernel is written for the fewest FP64 operations: 308 per cell, 1.47 ms
// (the two-iteration step 20.03 -> 12.72 ms). Transport and diffusion of
// RHS_Sat_Turb.cpp:300-1000 together are one weight per stencil value: seven fused multiply-adds per field with
// weights that cost seven more per diffusivity -- shared by the three phases of a species, by u, v and w, and by the
// water and ammonia groups where their Schmidt numbers are equal. Comparisons run on the integer pipe.
//   u, v, w always combine differences to the centre (five operations more per field): their tendencies are
//   results (the projection's source), w's zonal differences are small against w, and differences of near-equal
//   values are exact. So do k* and omega*: the closure floors k* to a uniform value and divides by gradients that
//   a uniform field must leave at zero. t and the species enter y + dt r by weights on the values: the rounding,
//   eps sum |weight| |f|, is there below eps |f| times dt sum |weight| -- the Courant number that a stable step keeps
//   under 3. Where their tendencies are results too (CENTRED), those are formed from the differences beside.
// PLAIN: the default switches (`plain_knobs`), whose branches are then left out at compile time: an instruction
// the compiler predicates off still takes its slot of the FP64 pipe.
template <int MODE, bool CENTRED, bool PLAIN>
__global__ void __launch_bounds__(32 * RKS_ROWS, RKS_BLOCKS) rk_stage_fp64_kernel(const KConst K,
                                                                                  const StageIO<double> io,
                                                                                  const StageParams sp) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * RKS_ROWS + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= K.km || j >= K.jm) return;
    const int64_t plane = K.plane;
    const int kp = K.kp;
    const int64_t c = ((int64_t)i * K.jm + j) * kp + k;
    const bool interior = (i >= 1 && i <= K.im - 2 && j >= 2 && j <= K.jm - 3 && k <= K.km - 2);
    if (!interior) {
        // Cells the step does not integrate keep their values: the stage buffer takes them once.
        if (MODE == MODE_STAGE && sp.stage == 0) {
#pragma unroll 1
            for (int q = 0; q < NPROG; q++) io.out[q][c] = ldg(io.in[q] + c);
        }
        return;
    }
    const int kw = (k == 0) ? K.km - 2 : k - 1;
    const int ke = (k == K.km - 2) ? 0 : k + 1;
    const int dkw = kw - k, dke = ke - k;
    const StageGeo& g = io.geo[(int64_t)i * K.jm + j];
    auto load = [&](int q) { return stencil(io.in[q], c, plane, kp, dkw, dke); };

    const S7 su = load(ATSAT_F_U), sv = load(ATSAT_F_V), sw = load(ATSAT_F_W);
    const double u = su.c, v = sv.c, w = sw.c;
    const double U = u * K.inv_2dr, V = v * g.s_the, W = w * g.s_phi;
    const double dpr = (ldg(io.p_dyn + c + plane) - ldg(io.p_dyn + c - plane)) * K.inv_2dr;
    const double dpth = (ldg(io.p_dyn + c + kp) - ldg(io.p_dyn + c - kp)) * g.s_the;
    const double dpph = (ldg(io.p_dyn + c + dke) - ldg(io.p_dyn + c + dkw)) * g.s_phi;

    // eddy viscosity as the momentum / scalar equations read it (RHS_Sat_Turb.cpp:577-582)
    const double nue_c = ldg(io.nue + c);
    const double nue_t = finite(nue_c) ? (PLAIN ? 1.0 : K.turb_coupling) * positive(nue_c) : 0.0;
    const double nue_t_s = nue_t * K.inv_pr_t;
    double sd = 0.0;              // flux-form factor of the species (RHS_Sat_Turb.cpp:979-1009)

    // ---- momentum (RHS_Sat_Turb.cpp:310-350, 388-399, 435-456, 700-714, 780-835) ----
    {
        const S7 du = centred(su), dv = centred(sv), dw = centred(sw);
        const double visc = K.inv_re + nue_t;
        const Wt wt = weights(visc, U, V, W, g);
        Wt wu = wt;
        wu.rp = fma(visc, g.lu_rp, -U);
        wu.rm = fma(visc, g.lu_rm, U);
        const double u_t = du.tp - du.tm, u_p = du.pe - du.pw, v_p = dv.pe - dv.pw, w_p = dw.pe - dw.pw;

        double buoyancy_u = 0.0;
        const double t_c = ldg(io.in[ATSAT_F_T] + c);
        if (PLAIN || !K.hydro_buoy) {
            const double ps = ldg(io.p_stat + c);
            if ((PLAIN || !K.buoy_legacy) && in_rcp_range(t_c)) {
                buoyancy_u = K.kbuoy * ((K.buoy_c * ps) * recip_nr(t_c) - ldg(io.buoy + i));
            } else if (t_c > 0.0) {
                if (!PLAIN && K.buoy_legacy) buoyancy_u = K.legacy_buoy * (ps + ldg(io.p_dyn + c)) / (K.rR * t_c * K.t_ref);
                else buoyancy_u = K.kbuoy * (K.g * ps / (K.rR * t_c * K.t_ref) - ldg(io.buoy + i));
            }
        }
        double fu = fma(visc, g.u_metric * u, fma(-g.c_rad, w, g.cent_rad + buoyancy_u));
        if (!PLAIN && !K.metric_split) fu = fma(K.metric_on * g.inv_rm, fma(v, v, w * w), fu);

        // p_metric's gradient with the metric terms (theta) and with the Coriolis force (phi)
        const double wcot = w * g.cot;
        double mv = fma(u, v, -(w * wcot));
        const double mw = fma(w, u, v * wcot);
        double fw = fma(-g.c_v, v - g.vbar0, -(g.c_u * (u - g.ubar0)));
        if (PLAIN || K.metric_split) {
            mv = fma(ldg(io.p_metric + c + kp) - ldg(io.p_metric + c - kp), K.inv_2dthe, mv);
            fw = fma(-(ldg(io.p_metric + c + dke) - ldg(io.p_metric + c + dkw)), g.s_phi, fw);
        }
        const double xv = fma(g.x_v1, u_t, -fma(g.x_v2, w_p, g.v_metric * v));
        const double xw = fma(g.x_w1, u_p, fma(g.x_v2, v_p, -(g.v_metric * w)));
        // The tendencies without p_dyn's gradient (aux), which would round away part of them: it comes last. The large
        // forces of v and w come after their stencil sums too, whose steps would each round at the forces' size.
        const double aux_u = apply_centred(wu, du, fu);
        const double aux_v = fma(-mv, g.inv_rm, fma(visc, xv, apply_centred(wt, dv))) + fma(-g.c_the, w, g.cent_the);
        const double aux_w = fma(-mw, g.inv_rm, fma(visc, xw, apply_centred(wt, dw))) + fw;
        const double rhs_u = aux_u - dpr, rhs_v = aux_v - dpth, rhs_w = aux_w - dpph;
        emit<MODE>(io, sp, K, ATSAT_F_U, c, rhs_u, rhs_u);
        emit<MODE>(io, sp, K, ATSAT_F_V, c, rhs_v, rhs_v);
        emit<MODE>(io, sp, K, ATSAT_F_W, c, rhs_w, rhs_w);
        if (MODE != MODE_STAGE) {
            io.aux[0][c] = aux_u;
            io.aux[1][c] = aux_v;
            io.aux[2][c] = aux_w;
        }
        if (!PLAIN && K.divu_on)
            sd = K.species_divu * ((du.rp - du.rm) * K.inv_2dr + 2.0 * u * g.inv_rm + (dv.tp - dv.tm) * g.s_the
                                   + v * g.cot * g.inv_rm + w_p * g.s_phi);
    }

    // kappa diffusion - transport + extra of t or a species
    auto tendency = [&](int q, const Wt& wt, double extra) {
        const S7 f = load(q);
        const double out = CENTRED ? apply_centred(wt, centred(f), extra) : 0.0;
        const double r = MODE == MODE_RHS ? out : apply_values(wt, f, extra);
        emit<MODE>(io, sp, K, q, c, r, out);
    };

    // ---- temperature (RHS_Sat_Turb.cpp:368-386, 409, 435-437, 611-665, 752-759) ----
    {
        double dps = 0.0;
        if (K.adiabatic) {
            dps = (ldg(io.p_stat + c + plane) - ldg(io.p_stat + c - plane)) * K.dps_scale;
            const double rho_l = ldg(io.rho_mix + c);
            if (K.adiabatic_rho) {
                if (in_rcp_range(rho_l)) dps *= K.r_mix * recip_nr(rho_l);
                else if (rho_l > 0.0 && isfinite(rho_l)) dps *= K.r_mix / rho_l;
            }
        }
        double r = K.coeff_energy_p * fma(u, dpr + dps, fma(v, dpth, w * dpph));
        if (!PLAIN && K.rad_on) {
            const double rho_f = ldg(io.rho_mix + c);
            const double rho = (rho_f > 0.0 && isfinite(rho_f)) ? rho_f : K.r_mix;
            if (rho > 0.0) r += clip_half(K.rad_coupling * ldg(io.q_rad + c) * K.rad_num / (rho * K.rad_den_c));
        }
        if (K.precip_on) r += clip_half(K.precip_factor * ldg(io.q_precip + c));
        if (!PLAIN && K.tmf_on) r -= K.tmf_chem * ldg(io.thermalmassflux + c);
        tendency(ATSAT_F_T, weights(K.inv_re_pr + nue_t_s, U, V, W, g), r);
    }

    // ---- species (RHS_Sat_Turb.cpp:409-431, 457-491, 839-937) ----
    auto species = [&](int q, const Wt& wt, double extra) {
        double r = extra;
        if (!PLAIN && K.divu_on) r -= sd * ldg(io.in[q] + c);
        tendency(q, wt, r);
    };
    const double pc = PLAIN ? 1.0 : K.precip_coupling, chem = PLAIN ? 1.0 : K.chem;
    // fma(1, a, b) is a + b bit for bit
    Wt wt = weights(K.inv_sc_re_h2o + nue_t_s, U, V, W, g);
    species(ATSAT_F_H2O, wt, pc * ldg(io.s_precip[0] + c));
    species(ATSAT_F_H2O_CLOUD, wt, pc * ldg(io.s_precip[1] + c));
    species(ATSAT_F_H2O_ICE, wt, pc * ldg(io.s_precip[2] + c));
    if (!K.nh3_as_h2o) wt = weights(K.inv_sc_re_nh3 + nue_t_s, U, V, W, g);
    species(ATSAT_F_NH3, wt, fma(chem, ldg(io.massflux_nh3 + c), pc * ldg(io.s_precip[3] + c)));
    species(ATSAT_F_NH3_CLOUD, wt, pc * ldg(io.s_precip[4] + c));
    species(ATSAT_F_NH3_ICE, wt, pc * ldg(io.s_precip[5] + c));
    wt = weights(K.inv_sc_re_ch4 + nue_t_s, U, V, W, g);
    species(ATSAT_F_CH4, wt, pc * ldg(io.s_precip[6] + c));
    species(ATSAT_F_CH4_CLOUD, wt, pc * ldg(io.s_precip[7] + c));
    species(ATSAT_F_CH4_ICE, wt, pc * ldg(io.s_precip[8] + c));
    wt = weights(K.inv_sc_re_h2s + nue_t_s, U, V, W, g);
    species(ATSAT_F_H2S, wt, chem * ldg(io.massflux_h2s + c));
    // nh4sh carries the flux-limiter correction (RHS_Sat_Turb.cpp:932-937)
    wt = weights(K.inv_sc_re_nh4sh + nue_t_s, U, V, W, g);
    species(ATSAT_F_NH4SH, wt, fma(chem, ldg(io.massflux_nh4sh + c), ldg(io.fluxlim_nh4sh + c)));

    // ---- k-omega transport (RHS_Sat_Turb.cpp:511-538) ----
    // The eddy viscosity enters as it is: an infinite one makes the diffusion infinite, which the limits of k* and
    // omega* in emit take; as weights on differences of either sign it would make it NaN.
    auto closure = [&](int q, double inv_sig, double source) {
        const double kappa = fma(nue_c, inv_sig, K.inv_re);
        const S7 d = centred(load(q));
        double r;
        if (finite(nue_c)) r = apply_centred(weights(kappa, U, V, W, g), d) + source;
        else r = fma(kappa, apply_centred(weights(1.0, 0.0, 0.0, 0.0, g), d), apply_centred(weights(0.0, U, V, W, g), d) + source);
        emit<MODE>(io, sp, K, q, c, r, r);
    };
    if (K.turb) {
        closure(ATSAT_F_TKE, K.inv_sig_k, ldg(io.tke_source + c));
        closure(ATSAT_F_DIS, K.inv_sig_w, ldg(io.dis_source + c));
    } else if (MODE == MODE_RHS || (MODE == MODE_FINAL && sp.write_all_rhs)) {
        io.rhs[ATSAT_F_TKE][c] = 0.0;
        io.rhs[ATSAT_F_DIS][c] = 0.0;
    }
}

// ---- computeBuoyancyRefLevel (RungeKutta_Sat_Turb.cpp:31-50): two-level deterministic reduction ----
// One block per (level, chunk of rows); a warp takes whole rows, its lanes the meridians, four at a time
// so that eight loads are in flight per lane.
constexpr int LM_CHUNKS = LEVEL_MEAN_CHUNKS;
constexpr int LM_THREADS = 128;

// the buoyancy g p / (r_mix R_mix T t_ref) = bc p / t of one cell (bc formed on the host); false where
// the reference skips the cell (!(t > 0), non-finite b). The level mean's rows take the fast path below
// and come here only for cells outside it.
__device__ __forceinline__ bool cell_buoyancy(const KConst& K, double tc, double pc, double& b) {
    if (in_rcp_range(tc)) {
        b = (K.buoy_c * pc) * recip_nr(tc);
    } else {
        if (!(tc > 0.0)) return false;
        b = K.g * pc / (K.rR * tc * K.t_ref);
    }
    return isfinite(b);
}

// rest + the cell's buoyancy, and whether the cell counts. A call that does the sum too: inlined, or with the sum in
// the caller, it was if-converted, and its FP64 operations took their slots of the FP64 pipe in every cell.
struct RareSum { double rest; int counts; };
__device__ __noinline__ RareSum add_buoyancy_rare(const KConst& K, double tc, double pc, double rest) {
    double b;
    if (!cell_buoyancy(K, tc, pc, b)) return {rest, 0};
    return {rest + b, 1};
}

// |x| < 2^e (zero and subnormals included), finite: an exponent test on the integer pipe
__device__ __forceinline__ bool below_pow2(double x, uint32_t e) {
    uint32_t lo, hi;
    split_f64(x, lo, hi);
    return ((hi >> 20) & 0x7FFu) < 1023u + e;
}

// GB300 issues two FP64 operations per SM per cycle, so the per-cell work is three of them: each lane
// sums p / t over its cells of a row (the Newton-Raphson reciprocal and one fma) and the row's weight
// and the constant bc are applied once per row: sum += sin(theta_j) (bc * sum_k p/t + rest), with the
// weight sum sin(theta_j) * (cells counted). Cells with t outside the reciprocal's range or a huge p
// ("rest") take the reference's own expression and skip rule. With |p| < 2^512, 1/t < 2^127 and
// |bc| < 2^256 every fast-path term and sum is finite, as the reference's isfinite test needs.
// Measured at 41x181x361: 33.8 -> 28 us with the rare path called (5.1 -> 3.9 FP64 slots a cell); two or three warps
// of a block sharing a running sum's rows changed nothing (28, 27 us), four filled two waves (42 us).
//
// The last of a level's blocks to finish adds the chunks' sums in order (`done` counts the level's finished blocks
// and is zero again afterwards).
__device__ __forceinline__ void level_mean_block(const KConst& K, const double* __restrict__ t,
                                                 const double* __restrict__ ps, const double* __restrict__ sin_j,
                                                 double* partial, unsigned int* done, double* buoy, int i, int chunk) {
    const int j0 = (int)((int64_t)K.jm * chunk / LM_CHUNKS), j1 = (int)((int64_t)K.jm * (chunk + 1) / LM_CHUNKS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool bc_ok = below_pow2(K.buoy_c, 256);
    double sum = 0.0, wsum = 0.0;
    for (int j = j0 + warp; j < j1; j += LM_THREADS / 32) {
        const int64_t row = ((int64_t)i * K.jm + j) * K.kp;
        double rs = 0.0, rest = 0.0;
        int cnt = 0;
        for (int k0 = 0; k0 < K.km; k0 += 128) {
            double tv[4], pv[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = k0 + q * 32 + lane;
                tv[q] = (k < K.km) ? __ldg(t + row + k) : 0.0;
                pv[q] = (k < K.km) ? __ldg(ps + row + k) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (k0 + q * 32 + lane >= K.km) continue;
                if (bc_ok && in_rcp_range(tv[q]) && below_pow2(pv[q], 512)) {
                    rs = fma(pv[q], recip_nr(tv[q]), rs);
                    cnt++;
                } else {
                    const RareSum r = add_buoyancy_rare(K, tv[q], pv[q], rest);
                    rest = r.rest;
                    cnt += r.counts;
                }
            }
        }
        const double wgt = __ldg(sin_j + j);
        sum = fma(wgt, fma(K.buoy_c, rs, rest), sum);
        wsum = fma(wgt, (double)cnt, wsum);
    }
    __shared__ double s_sum[LM_THREADS / 32], s_w[LM_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_down_sync(0xffffffffu, sum, o);
        wsum += __shfl_down_sync(0xffffffffu, wsum, o);
    }
    if (lane == 0) { s_sum[warp] = sum; s_w[warp] = wsum; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int q = 0; q < LM_THREADS / 32; q++) { a += s_sum[q]; b += s_w[q]; }
        double* part = partial + (int64_t)i * LM_CHUNKS * 2;
        __stcg(part + chunk * 2 + 0, a);
        __stcg(part + chunk * 2 + 1, b);
        __threadfence();
        if (atomicAdd(done + i, 1u) == LM_CHUNKS - 1) {
            __threadfence();
            double s = 0.0, w = 0.0;
            for (int q = 0; q < LM_CHUNKS; q++) {
                s += __ldcg(part + q * 2 + 0);
                w += __ldcg(part + q * 2 + 1);
            }
            buoy[i] = (w > 0.0) ? s / w : 0.0;
            done[i] = 0u;
        }
    }
}

// ---- computeMetricPressure (RungeKutta_Sat_Turb.cpp:60-108): one radial trapezoid scan per column ----
// The scan is serial in i. inv_rm holds
// 1 / rm(i) (a product instead of the reference's quotient: at most one rounding apart). Six FP64 operations
// per cell (seven with p_baro): f = (v^2 + w^2) / rm + cor w as two products and two fmas, and the
// trapezoid acc += dr/2 (f_{i-1} + f_i) as one add and one fma.
// The next four levels' loads are in flight while these are summed (two, four or eight alike), and p_baro is a switch
// of the code: 45.5 -> 39.7 us by itself at 41x181x361 (26 us of FP64 issue).
constexpr int MS_BATCH = 4;

template <bool BARO>
__device__ __forceinline__ void metric_scan_column(const KConst& K, const double* __restrict__ v,
                                                   const double* __restrict__ w, const double* __restrict__ inv_rm,
                                                   const double* __restrict__ cor_j,
                                                   const double* __restrict__ p_baro, double* __restrict__ pm,
                                                   double half_dr, int j, int k) {
    const double cor = __ldg(cor_j + j);
    const int64_t c0 = (int64_t)j * K.kp + k;
    double vv[MS_BATCH], ww[MS_BATCH], pb[MS_BATCH];
    auto load = [&](int i0) {
#pragma unroll
        for (int q = 0; q < MS_BATCH; q++) {
            const int64_t c = c0 + (int64_t)(i0 + q) * K.plane;
            const bool in = i0 + q < K.im;
            vv[q] = in ? __ldg(v + c) : 0.0;
            ww[q] = in ? __ldg(w + c) : 0.0;
            if (BARO) pb[q] = in ? __ldg(p_baro + c) : 0.0;
        }
    };
    const double v0 = __ldg(v + c0), w0 = __ldg(w + c0);
    load(1);
    double f_prev = fma(fma(w0, w0, v0 * v0), __ldg(inv_rm), cor * w0), acc = 0.0;
    pm[c0] = BARO ? acc + __ldg(p_baro + c0) : acc;
    for (int i0 = 1; i0 < K.im; i0 += MS_BATCH) {
        double cv[MS_BATCH], cw[MS_BATCH], cb[MS_BATCH];
#pragma unroll
        for (int q = 0; q < MS_BATCH; q++) {
            cv[q] = vv[q];
            cw[q] = ww[q];
            if (BARO) cb[q] = pb[q];
        }
        load(i0 + MS_BATCH);
#pragma unroll
        for (int q = 0; q < MS_BATCH; q++) {
            const int i = i0 + q;
            if (i >= K.im) break;
            const double f = fma(fma(cw[q], cw[q], cv[q] * cv[q]), __ldg(inv_rm + i), cor * cw[q]);
            acc = fma(half_dr, f_prev + f, acc);
            f_prev = f;
            pm[c0 + (int64_t)i * K.plane] = BARO ? acc + cb[q] : acc;
        }
    }
}

// The step's two FP64-bound scans in one launch: the level mean's blocks (one per level and chunk), then the metric
// scan's (32 x 4 columns; the other order is 0.6 % of a step slower). They read different fields of y_n and fill each other's thin waves: 66 us at 41x181x361
// (44 us of FP64 issue). Apart, on two streams forked and joined by events, with the level mean's last sum a launch of
// its own, they took three launches: two iterations at 10x20x36 214 -> 206 us, 41x181x361 replayed 2408 -> 2385.
struct LevelMetricArgs {
    const double *t, *ps, *sin_j;                  // level mean
    double *partial, *buoy;
    unsigned int* done;
    const double *v, *w, *inv_rm, *cor_j, *p_baro; // metric scan
    double* pm;
    double half_dr;
    int mean_blocks, bk;                           // level mean blocks; metric scan blocks along k
};

template <bool BARO>
__global__ void __launch_bounds__(LM_THREADS) level_metric_kernel(const KConst K, const LevelMetricArgs A) {
    if ((int)blockIdx.x < A.mean_blocks) {
        level_mean_block(K, A.t, A.ps, A.sin_j, A.partial, A.done, A.buoy, blockIdx.x / LM_CHUNKS, blockIdx.x % LM_CHUNKS);
        return;
    }
    const int b = blockIdx.x - A.mean_blocks;
    const int k = b % A.bk * 32 + (threadIdx.x & 31), j = b / A.bk * 4 + (threadIdx.x >> 5);
    if (k < K.km && j < K.jm)
        metric_scan_column<BARO>(K, A.v, A.w, A.inv_rm, A.cor_j, A.p_baro, A.pm, A.half_dr, j, k);
}

// ---- computeMixtureDensity (Pressure_Sat.cpp:49-62) ----
// rho = p_stat 1e5 / (R_mix t t_ref). Where t is in [2^-60, 2^60), |p_stat| < 2^60 and the constant
// c2 = 1e5 / (R_mix t_ref) is moderate (`fast`, set by the host), rho = p_stat (c2 / t) with c2 / t the
// FP32 quotient corrected once in FP64 (q = q0 + (c2 - t q0) rcp(t), relative error ~2^-44): three FP64
// operations per cell. Elsewhere the reference's expression and skip rules.
__global__ void __launch_bounds__(256) density_kernel(const KConst K, const double* __restrict__ t,
                                                      const double* __restrict__ ps, double R_mix, double c2,
                                                      float c2f, int fast, double* __restrict__ rho) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= K.km || j >= K.jm) return;
    const int64_t c = ((int64_t)i * K.jm + j) * K.kp + k;
    const double tc = __ldg(t + c), pc = __ldg(ps + c);
    uint32_t lo, th, ph;
    split_f64(tc, lo, th);
    split_f64(pc, lo, ph);
    if (fast && ((th >> 20) & 0xFFFu) - 963u < 120u && ((ph >> 20) & 0x7FFu) < 1083u) {
        const float rf = __frcp_rn(d2f(tc));
        const double q0 = f2d(c2f * rf);
        rho[c] = pc * fma(fma(-tc, q0, c2), f2d(rf), q0);
        return;
    }
    const double T = tc * K.t_ref;
    if (!(T > 0.0) || !(R_mix > 0.0)) { rho[c] = 0.0; return; }
    const double den = R_mix * T;
    const double r = in_rcp_range(den) ? (pc * 1.0e5) * recip_nr(den) : (pc * 1.0e5) / den;
    rho[c] = isfinite(r) ? r : 0.0;
}

}  // namespace

cudaError_t launch_rk_stage_fp64(const KConst& kc, const StageIO<double>& io, const StageParams& sp, int mode,
                                 cudaStream_t s) {
    const dim3 block(32, RKS_ROWS), grid((kc.km + 31) / 32, (kc.jm + RKS_ROWS - 1) / RKS_ROWS, kc.im);
    const bool plain = plain_knobs(kc);
    auto go = [&](auto kernel) { kernel<<<grid, block, 0, s>>>(kc, io, sp); };
    if (mode == MODE_RHS) plain ? go(rk_stage_fp64_kernel<MODE_RHS, true, true>) : go(rk_stage_fp64_kernel<MODE_RHS, true, false>);
    else if (mode == MODE_STAGE)
        plain ? go(rk_stage_fp64_kernel<MODE_STAGE, false, true>) : go(rk_stage_fp64_kernel<MODE_STAGE, false, false>);
    else if (sp.write_all_rhs)
        plain ? go(rk_stage_fp64_kernel<MODE_FINAL, true, true>) : go(rk_stage_fp64_kernel<MODE_FINAL, true, false>);
    else plain ? go(rk_stage_fp64_kernel<MODE_FINAL, false, true>) : go(rk_stage_fp64_kernel<MODE_FINAL, false, false>);
    return cudaGetLastError();
}

cudaError_t launch_level_metric(const KConst& kc, const LevelMean* m, const MetricScan* c, cudaStream_t s) {
    LevelMetricArgs A{};
    if (m) {
        A.t = m->t; A.ps = m->p_stat; A.sin_j = m->sin_j;
        A.partial = m->partial; A.done = m->done; A.buoy = m->buoy;
    }
    if (c) {
        A.v = c->v; A.w = c->w; A.inv_rm = c->inv_rm; A.cor_j = c->cor_j; A.p_baro = c->p_baro; A.pm = c->p_metric;
        A.half_dr = 0.5 * kc.dr;
        A.bk = (kc.km + 31) / 32;
    }
    A.mean_blocks = m ? kc.im * LM_CHUNKS : 0;
    const int blocks = A.mean_blocks + A.bk * ((kc.jm + 3) / 4);
    auto kernel = A.p_baro ? level_metric_kernel<true> : level_metric_kernel<false>;
    kernel<<<blocks, LM_THREADS, 0, s>>>(kc, A);
    return cudaGetLastError();
}

cudaError_t launch_density(const KConst& kc, const double* t, const double* p_stat, double R_mix, double* rho,
                           cudaStream_t s) {
    dim3 block(32, 8), grid((kc.km + 31) / 32, (kc.jm + 7) / 8, kc.im);
    const double c2 = (R_mix > 0.0 && kc.t_ref > 0.0) ? 1.0e5 / (R_mix * kc.t_ref) : 0.0;
    const int fast = c2 > 0x1p-60 && c2 < 0x1p60;
    density_kernel<<<grid, block, 0, s>>>(kc, t, p_stat, R_mix, c2, (float)c2, fast, rho);
    return cudaGetLastError();
}

}  // namespace atsat
