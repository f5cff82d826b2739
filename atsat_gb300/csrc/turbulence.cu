// Turbulence<cSaturnModel>::run (planet/Turbulence.h:306-329) on the device, FP64: the friction velocity, the
// floors of k* and omega*, the sources of the chosen closure (k-omega SST by default, k-omega, k-epsilon) with
// the production P_k of the curvature-corrected velocity-gradient tensor and the moist buoyancy sink of k, the
// floors and caps after the source loop, the zero-gradient copy at i = 0, the eddy-viscosity cap, the seam
// copy and the two lid corners -- in the reference's order of passes. ATSAT has no
// solid body (cSaturnModel.h:254-255), so the land branches are constant.
//
// Per-level and per-row factors come from the host (TurbTables) with the reference's expressions: the model's
// float layer-height table (cSaturnModel.h:1062-1074), the closure's own sine (exact-zero guard, no floor),
// inv_2dthe / rm and inv_2dphi / (rm sin). The sources loop reads only the other cells' k* and omega*, which
// no thread of it writes (the floors run as separate passes), so its result does not depend on the order. The default
// closure (SST) has a source kernel of its own that applies the floors and caps where it reads and writes (sst_kernel).
#include "dyn_common.cuh"

#include <cmath>

namespace atsat {
namespace {

constexpr double C_NUE = 0.028, DIS_MIN = 1.0e-10;

__device__ __forceinline__ double dmax(double a, double b) { return (a < b) ? b : a; }   // std::max
__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }   // std::min
__device__ __forceinline__ double clamp3(double x, double lo, double hi) { return (x < lo) ? lo : ((x > hi) ? hi : x); }

struct TurbArgs {
    int im, jm, km, kp, periodic, model, turb_free, curv, buoy, abl_taper, local_rho, turb_active;
    int64_t plane;
    double u_0, t_ref, g, cp_mix, r_mix, R_mix, L_m, nue_air, re_turb, nue_max, k_bg_nd, vel_star_max;
    double dr, dthe, dphi, inv_2dr, abl_height, taper_dz;
    // quotients of constants, formed once on the host
    double inv_L_m, nue_air_nd, gam_ad, tL2_pr, inv_R_mix, inv_cpR, inv_2dr2;
    double la[3], lb[3], sa[3], sb[3];   // L / R_mix and ep L^2 / (cp R_mix) over liquid and over ice
    float inv_ys_free_f, nue_air_nd_f;
    int kbg_pos, t0_pos, rmix_pos;   // constants whose signs allow integer comparisons
    int sst_bound_ok;                // the constants of the FP32 bounds are in range
    double ep[3], lv[3], ls[3], t_0[3];
    TurbTables tab;
    double *u, *v, *w, *t, *rho, *tke, *dis, *tken, *disn, *nue, *tks, *dss, *prod, *vel_star;
    double *gv[3], *gc[3], *gi[3];
};

__device__ __forceinline__ int64_t cidx(const TurbArgs& A, int i, int j, int k) {
    return ((int64_t)i * A.jm + j) * A.kp + k;
}

// compute_vel_star (Turbulence.h:335-378): u_tau per (j, k), at the first fluid cell i = 1
__global__ void turb_vel_star_kernel(const TurbArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (k >= A.km || j >= A.jm) return;
    double vs = 0.05;
    if (!A.turb_free) {
        const int i_surf = (1 < A.im - 1) ? 1 : A.im - 1;
        const int64_t c = cidx(A, i_surf, j, k);
        const double v_s = A.v[c], w_s = A.w[c];
        const double vw2 = v_s * v_s + w_s * w_s;
        vs = !isfinite(vw2) ? 0.05 : clamp3(sqrt(0.002) * (A.u_0 * sqrt(vw2)), 0.05, A.vel_star_max);
    }
    A.vel_star[(int64_t)j * A.kp + k] = vs;
}

__device__ __forceinline__ bool interior(const TurbArgs& A, int i, int j, int k) {
    return i >= 1 && i <= A.im - 2 && j >= 1 && j <= A.jm - 2 && k >= (A.periodic ? 0 : 1) && k <= A.km - 2;
}

// the floors before the source loop (Turbulence.h:628-630, 645-650)
__global__ void __launch_bounds__(256) turb_clamp_in_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (!interior(A, i, j, k)) return;
    const int64_t c = cidx(A, i, j, k);
    A.tke[c] = dmax(0.0, A.tke[c]);
    A.dis[c] = dmax(DIS_MIN, A.dis[c]);
}

// k-omega and k-epsilon (SST: sst_kernel)
__device__ void sources_cell(const TurbArgs& A, int i, int j, int k) {
    const TurbTables& T = A.tab;
    const int64_t c = cidx(A, i, j, k);
    const int64_t P = A.plane, kp = A.kp;
    const int N = A.km - 1;
    const int kw = A.periodic ? (k == 0 ? N - 1 : k - 1) : k - 1;
    const int ke = A.periodic ? (k == N - 1 ? 0 : k + 1) : k + 1;
    const int64_t cw = c - k + kw, ce = c - k + ke;
    const double rm = T.rm[i], inv_rm = T.inv_rm[i];
    const double cotanthe = T.cotanthe[j];
    const double inv_rm2dthe = T.inv_rm2dthe[i];
    const double inv_rmsinthe2dphi = T.inv_rmsinthe2dphi[(int64_t)i * A.jm + j];
    const double inv_2dr = A.inv_2dr;
    const double* u = A.u; const double* v = A.v; const double* w = A.w;
    const double* tk = A.tke; const double* ds = A.dis;
    const double dudr = (u[c + P] - u[c - P]) * inv_2dr * 1.0;
    const double dvdr = (v[c + P] - v[c - P]) * inv_2dr * 1.0;
    const double dwdr = (w[c + P] - w[c - P]) * inv_2dr * 1.0;
    const double dudthe = (u[c + kp] - u[c - kp]) * inv_rm2dthe;
    const double dvdthe = (v[c + kp] - v[c - kp]) * inv_rm2dthe;
    const double dwdthe = (w[c + kp] - w[c - kp]) * inv_rm2dthe;
    const double dudphi = (u[ce] - u[cw]) * inv_rmsinthe2dphi;
    const double dvdphi = (v[ce] - v[cw]) * inv_rmsinthe2dphi;
    const double dwdphi = (w[ce] - w[cw]) * inv_rmsinthe2dphi;
    const double tkc = tk[c], dsc = ds[c];
    const double dtkedr = (tk[c + P] - tk[c - P]) * inv_2dr * 1.0;
    const double ddisdr = (ds[c + P] - ds[c - P]) * inv_2dr * 1.0;
    double cnue;
    {
        const double dis_here = dmax(dsc, DIS_MIN);
        const double tke_here = dmax(tkc, 0.0);
        cnue = (A.model == 0) ? qdiv(C_NUE * tke_here * tke_here, dis_here) : qdiv(tke_here, dis_here);
        cnue = dmin(cnue, A.nue_max);
    }
    const double u_r = A.curv ? u[c] * inv_rm : 0.0;
    const double v_r = A.curv ? v[c] * inv_rm : 0.0;
    const double w_r = A.curv ? w[c] * inv_rm : 0.0;
    const double v_cot_r = v_r * cotanthe, w_cot_r = w_r * cotanthe;
    const double g_rr = dudr, g_rt = dudthe - v_r, g_rp = dudphi - w_r;
    const double g_tr = dvdr, g_tt = dvdthe + u_r, g_tp = dvdphi - w_cot_r;
    const double g_pr = dwdr, g_pt = dwdthe, g_pp = dwdphi + u_r + v_cot_r;
    const double der = 0.66667 * (g_rr + g_tt + g_pp);
    const double prod = dmax(0.0, (cnue * (2.0 * g_rr - der) - 0.66667 * tkc) * g_rr
                                + (cnue * (g_rt + g_tr)) * g_rt
                                + (cnue * (g_rp + g_pr)) * g_rp
                                + (cnue * (2.0 * g_tt - der) - 0.66667 * tkc) * g_tt
                                + (cnue * (g_tr + g_rt)) * g_tr
                                + (cnue * (g_tp + g_pt)) * g_tp
                                + (cnue * (2.0 * g_pp - der) - 0.66667 * tkc) * g_pp
                                + (cnue * (g_pr + g_rp)) * g_pr
                                + (cnue * (g_pt + g_tp)) * g_pt);
    A.prod[c] = prod;
    const double W12 = g_rt - g_tr, W13 = g_rp - g_pr, W23 = g_tp - g_pt;
    const double Omega = sqrt(W12 * W12 + W13 * W13 + W23 * W23);
    const double L_m = A.L_m;
    double nue, tks, dss;
    if (A.model == 1) {            // compute_k_omega (Turbulence.h:929-1017)
        const double bet_star = 0.09, gam = 0.52, C_lim = 0.875, bet_0 = 0.0708;
        // the reference's quotients by rm 2 dthe, rm sin 2 dphi and 2 dr (rm + 1) as products with the
        // column's reciprocals (one division per cell)
        const double inv_r1 = qdiv(A.inv_2dr, rm + 1.0);
        const double dtkedthe = (tk[c + kp] - tk[c - kp]) * inv_rm2dthe;
        const double ddisdthe = (ds[c + kp] - ds[c - kp]) * inv_rm2dthe;
        const double dtkedphi = (tk[ce] - tk[cw]) * inv_rmsinthe2dphi;
        const double ddisdphi = (ds[ce] - ds[cw]) * inv_rmsinthe2dphi;
        const double dudr_k = (u[c + P] - u[c - P]) * inv_r1;
        const double dvdthe_k = dvdthe;
        const double dwdphi_k = dwdphi;
        const double dudthe_u = dudthe;
        const double dudphi_u = dudphi;
        const double dvdr_u = (v[c + P] - v[c - P]) * inv_r1;
        const double dwdr_u = (w[c + P] - w[c - P]) * inv_r1;
        const double dvdphi_u = dvdphi;
        const double dwdthe_u = dwdthe;
        const double S11 = dudr_k, S22 = dvdthe_k, S33 = dwdphi_k;
        const double S12 = 0.5 * (dudthe_u + dvdr_u), S13 = 0.5 * (dudphi_u + dwdr_u), S23 = 0.5 * (dvdphi_u + dwdthe_u);
        const double S_mag = sqrt(2.0 * (S11 * S11 + S22 * S22 + S33 * S33 + 2.0 * (S12 * S12 + S13 * S13 + S23 * S23)));
        const double w_hat = dmax(dsc, C_lim * S_mag / sqrt(bet_star));
        const double gd = dtkedr * ddisdr + dtkedthe * ddisdthe + dtkedphi * ddisdphi;
        const double sig_d = (gd <= 0.0) ? 0.0 : 0.125;
        const double b3 = bet_star * dmax(dsc, 1.0e-20);
        const double chi_w = fabs(qdiv(Omega * Omega * S_mag, b3 * b3 * b3));
        const double f_bet = qdiv(1.0 + 85.0 * chi_w, 1.0 + 100.0 * chi_w);
        nue = qdiv(tkc, dmax(w_hat, 1.0e-20));
        const double P_k = dmin(prod, 20.0 * bet_star * tkc * dsc);
        const double Y_k = bet_star * tkc * dsc;
        const double P_w = qdiv(gam * dsc, dmax(tkc, 1.0e-20)) * P_k;
        const double Y_w = bet_0 * f_bet * dsc * dsc;
        const double D_w = qdiv(sig_d, dmax(dsc, 1.0e-20)) * gd;
        tks = P_k - Y_k;
        dss = P_w - Y_w + D_w;
    } else {                       // compute_k_epsilon (Turbulence.h:885-926)
        const double C_eps_1 = 1.35, C_eps_2 = 1.80;
        const double y_phys = A.turb_free ? 1.0e20 : dmax(T.height_m[i] - T.height_m[0], L_m);
        const double y_star = y_phys / L_m;
        nue = C_NUE * tkc * tkc / dmax(dsc, DIS_MIN);
        const double d_plus = y_phys * A.vel_star[(int64_t)j * kp + k] / A.nue_air;
        const double f_nue = 1.0 - exp(-0.0115 * d_plus);
        const double Re_T = tkc * tkc * A.u_0 * L_m / dmax(dsc * A.nue_air, DIS_MIN * A.nue_air);
        const double f_2 = 1.0 - 0.4 / 1.8 * exp(-Re_T * Re_T / 36.0);
        nue *= f_nue;
        const double y_star2 = y_star * y_star;
        const double L_k = -2.0 * tkc / y_star2;
        const double L_w = -2.0 * dsc / y_star2 * exp(-d_plus / 2.0);
        const double tke_safe = dmax(tkc, DIS_MIN);
        const double P_w = C_eps_1 * dsc / tke_safe * prod;
        const double Y_w = C_eps_2 * f_2 * dsc * dsc / tke_safe;
        tks = prod - dsc + L_k / A.re_turb;
        dss = P_w - Y_w + L_w / A.re_turb;
    }
    // the buoyancy sink of k (Turbulence.h:800-835): B = -nu_t N^2 / Pr_t, moist N^2 in saturated cells
    if (A.buoy != 0) {
        // quotients as products with 1 / dz, 1 / T, 1 / rho and the host's constant quotients
        const double Tc = A.t[c] * A.t_ref;
        const double dz = T.height_m[i + 1] - T.height_m[i - 1];
        const double dTdz = qdiv((A.t[c + P] - A.t[c - P]) * A.t_ref, dz);
        const double inv_T = qdiv(1.0, Tc);
        double Gam = A.gam_ad, fac = 1.0;
        if (A.buoy == 3 && Tc > 0.0) {
            double rho = A.r_mix;
            if (A.local_rho) {
                const double r_ = A.rho[c];
                rho = (r_ > 0.0 && isfinite(r_)) ? r_ : A.r_mix;
            }
            double a = 0.0, b = 0.0;
            const double inv_rho = qdiv(1.0, rho);
            for (int n = 0; rho > 0.0 && n < 3; n++) {
                const double qc = (dmax(0.0, A.gc[n][c]) + dmax(0.0, A.gi[n][c])) * inv_rho;
                if (!(qc > 1.0e-9)) continue;
                const double qv = dmax(0.0, A.gv[n][c]) * inv_rho;
                const double L = Tc >= A.t_0[n] ? A.lv[n] : A.ls[n];
                a += L * qv * A.inv_R_mix * inv_T;
                b += A.ep[n] * L * L * qv * A.inv_cpR * inv_T * inv_T;
            }
            if (isfinite(a + b)) { Gam *= qdiv(1.0 + a, 1.0 + b); fac = 1.0 + a; }
        }
        const double N2 = (Tc > 0.0 && dz > 0.0) ? A.g * inv_T * (dTdz + Gam) * fac : 0.0;
        if (isfinite(N2) && (N2 > 0.0 || A.buoy == 2)) tks -= dmax(0.0, nue) * N2 * A.tL2_pr;
    }
    A.nue[c] = nue;
    A.tks[c] = tks;
    A.dss[c] = dss;
}

// ---- the SST closure (Turbulence.h:1020-1106 with 628-650, 800-881) ----
// Comparisons on the integer pipe (a DSETP takes a slot of the FP64 pipe like an addition): non-negative doubles order
// as their bit patterns.
__device__ __forceinline__ unsigned long long bits_of(double x) { return (unsigned long long)__double_as_longlong(x); }
constexpr unsigned long long INF_BITS = 0x7FF0000000000000ull, SIGN_BIT = 0x8000000000000000ull;
// (lo < x) ? x : lo for lo >= 0 (NaN: lo)
__device__ __forceinline__ double floor_at(double x, double lo) {
    const unsigned long long b = bits_of(x);
    return b > bits_of(lo) && b <= INF_BITS ? x : lo;
}
// (hi < x) ? hi : x for x >= +0 or NaN, hi any but -0 and a NaN with its sign bit set (as signed integers a negative hi
// is below every x)
__device__ __forceinline__ double cap_at(double x, double hi) {
    const unsigned long long b = bits_of(x);
    return (long long)b > __double_as_longlong(hi) && b <= INF_BITS ? hi : x;
}
// clamp3(x, -s, s), s >= 0
__device__ __forceinline__ double clip_to(double x, double s) {
    const unsigned long long b = bits_of(x), m = b & ~SIGN_BIT;
    return m > bits_of(s) && m <= INF_BITS ? __longlong_as_double((long long)(bits_of(s) | (b & SIGN_BIT))) : x;
}
// clamp3(x, 0, hi), hi as in cap_at
__device__ __forceinline__ double clip_positive(double x, double hi) {
    const unsigned long long b = bits_of(x);
    if (b > SIGN_BIT) return b <= (SIGN_BIT | INF_BITS) ? 0.0 : x;
    if (b == SIGN_BIT) return __double_as_longlong(hi) < 0 ? hi : x;
    return cap_at(x, hi);
}
__device__ __forceinline__ bool finite_double(double x) { return (bits_of(x) & INF_BITS) != INF_BITS; }

// Menter's blending where it is not negligible: F1, F2 and the eddy viscosity's denominator
struct SstBlend { double F1, nue; };
__device__ __noinline__ SstBlend sst_blend(double tkc, double dsc, double inv_dis, double inv_ys, double nue_air_nd,
                                           double grad_dot, double W2) {
    const double a1 = 0.31, inv_bet_star = 1.0 / 0.09, sig_w2 = 1.168;
    const double inv_ys2 = inv_ys * inv_ys;
    const double CD_kw = dmax(2.0 * sig_w2 * inv_dis * grad_dot, 1.0e-20);
    const double t_a = sqrt(tkc) * inv_bet_star * inv_dis * inv_ys;        // sqrt(k) / (beta* omega y*)
    const double t_b = 500.0 * nue_air_nd * inv_ys2 * inv_dis;             // 500 nu / (y*^2 omega)
    const double arg1 = dmin(dmax(t_a, t_b), qdiv(4.0 * sig_w2 * tkc * inv_ys2, CD_kw));
    const double arg2 = dmax(2.0 * t_a, t_b);
    const double a1sq = arg1 * arg1;
    const double F2 = tanh(arg2 * arg2);
    return {tanh(a1sq * a1sq), qdiv(a1 * tkc, dmax(a1 * dsc, sqrt(W2) * F2))};
}

// k* at its background after the source loop (Turbulence.h:634-643)
__device__ __forceinline__ double sst_floor(const TurbArgs& A, double tk, int j, int k) {
    double k_bg = A.k_bg_nd;
    if (!A.turb_free) {
        const double vs = A.vel_star[(int64_t)j * A.kp + k];
        k_bg = 0.01 * vs * vs / (sqrt(C_NUE) * A.u_0 * A.u_0);
    }
    return A.kbg_pos ? floor_at(tk, k_bg) : dmax(k_bg, tk);
}

// The sources, the production and the eddy viscosity of one cell, floors and caps included: k* and omega* enter floored
// (neighbours in the interior too, as the reference's pass before the loop leaves them) and are not written here
// (turb_floor_kernel does, after every cell has read its neighbours).
//
// Bound by the FP64 pipe (two operations per SM per cycle): about 110 operations per cell where the reference's expressions
// term by term, with a pass per floor, took 337 and 1347 us at 41x181x361 (1.50 ms with the passes around them). What
// went: the tensor products sum to cnue (2 (rr^2 + tt^2 + pp^2) - 2/3 S^2 + (rt + tr)^2 + (rp + pr)^2 + (tp + pt)^2)
// - 2/3 k S; scales are fused into the differences; quotients share 1 / omega, 1 / k, 1 / rho, 1 / T; comparisons are
// integer; and the blending functions are evaluated only where FP32 bounds with a margin do not already settle them
// (F1 < 1e-18 leaves 1 - F1 = 1 and the blended constants at their second values to the last bit, Omega F2 < a1 omega
// the viscosity's maximum): away from walls, with the closure's y* of 1e20 m, nowhere. Now 580 us, 0.63 ms a run
// (four to eight blocks per SM measured alike).
__global__ void __launch_bounds__(128, 4) sst_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y, i = blockIdx.z;
    if (!interior(A, i, j, k)) return;
    const TurbTables& T = A.tab;
    const int64_t c = cidx(A, i, j, k), P = A.plane, kp = A.kp;
    const int N = A.km - 1;
    const int64_t cw = c - k + (A.periodic ? (k == 0 ? N - 1 : k - 1) : k - 1);
    const int64_t ce = c - k + (A.periodic ? (k == N - 1 ? 0 : k + 1) : k + 1);
    const double inv_rm = A.curv ? T.inv_rm[i] : 0.0;
    const double s_r = A.inv_2dr, s_t = T.inv_rm2dthe[i], s_p = T.inv_rmsinthe2dphi[(int64_t)i * A.jm + j];

    // k*, omega* and their gradients' product
    const double tkc = floor_at(A.tke[c], 0.0), dsc = floor_at(A.dis[c], DIS_MIN);
    double grad_dot;
    {
        const bool up = i < A.im - 2, dn = i > 1, so = j < A.jm - 2, no = j > 1;
        auto tk = [&](int64_t n, bool in) { const double x = A.tke[n]; return in ? floor_at(x, 0.0) : x; };
        auto ds = [&](int64_t n, bool in) { const double x = A.dis[n]; return in ? floor_at(x, DIS_MIN) : x; };
        const double gr = (tk(c + P, up) - tk(c - P, dn)) * (ds(c + P, up) - ds(c - P, dn));
        const double gt = (tk(c + kp, so) - tk(c - kp, no)) * (ds(c + kp, so) - ds(c - kp, no));
        const bool edge_e = !A.periodic && k == N - 1, edge_w = !A.periodic && k == 1;
        const double gp = (tk(ce, !edge_e) - tk(cw, !edge_w)) * (ds(ce, !edge_e) - ds(cw, !edge_w));
        grad_dot = fma(gr, A.inv_2dr2, fma(gt, T.s_t2[i], gp * T.s_p2[(int64_t)i * A.jm + j]));
    }
    const double inv_dis = in_rcp_range(dsc) ? recip_nr(dsc) : 1.0 / dsc;
    const double k_over_d = tkc * inv_dis;

    // the velocity-gradient tensor and the production
    double prod;
    float W2f;
    {
        const double *u = A.u, *v = A.v, *w = A.w;
        const double u_r = u[c] * inv_rm, v_r = v[c] * inv_rm, w_r = w[c] * inv_rm, cot = T.cotanthe[j];
        const double rr = (u[c + P] - u[c - P]) * s_r, tr = (v[c + P] - v[c - P]) * s_r, pr = (w[c + P] - w[c - P]) * s_r;
        const double rt = fma(u[c + kp] - u[c - kp], s_t, -v_r), rp = fma(u[ce] - u[cw], s_p, -w_r);
        const double tt = fma(v[c + kp] - v[c - kp], s_t, u_r), tp = fma(v[ce] - v[cw], s_p, -(w_r * cot));
        const double pt = (w[c + kp] - w[c - kp]) * s_t, pp = fma(w[ce] - w[cw], s_p, fma(v_r, cot, u_r));
        const double S = rr + tt + pp, h = 0.66667 * S;
        const double a = rt + tr, b = rp + pr, d = tp + pt;
        const double diag = fma(rr, rr, fma(tt, tt, pp * pp)), off = fma(a, a, fma(b, b, d * d));
        const double cnue = cap_at(k_over_d, A.nue_max);
        prod = floor_at(fma(cnue, fma(2.0, diag, fma(-h, S, off)), -(h * tkc)), 0.0);
        // an upper bound of the rotation rate's square, free of cancellation
        const float w12 = fabsf(d2f(rt)) + fabsf(d2f(tr)), w13 = fabsf(d2f(rp)) + fabsf(d2f(pr));
        const float w23 = fabsf(d2f(tp)) + fabsf(d2f(pt));
        W2f = w12 * w12 + w13 * w13 + w23 * w23;
    }
    A.prod[c] = prod;

    const double bet_star = 0.09, bet1 = 0.0333, bet2 = 0.0368, gam1 = 0.413, gam2 = 0.2, sig_w2 = 1.168;
    double gam = gam2, bet = bet2, d_w = 2.0 * sig_w2, nue = k_over_d;
    {
        double y_phys = 1.0e20;
        if (!A.turb_free)
            y_phys = dmax(T.height_m[i] - T.height_m[0], dmax(1.0, T.thick_m[i - 1 > 0 ? i - 1 : 0]));
        // upper bounds of max(t_a, t_b) and of Omega F2 (tanh x <= x), one percent above FP32's rounding
        const float kf = d2f(tkc), df = d2f(dsc), iyf = A.turb_free ? A.inv_ys_free_f : 1.0f / d2f(y_phys * A.inv_L_m);
        const float ta = 1.01f * sqrtf(kf) * (1.0f / 0.09f) * iyf / df, tb = 1.01f * 500.0f * A.nue_air_nd_f * iyf * iyf / df;
        const float m2 = fmaxf(2.0f * ta, tb);
        const bool settled = fmaxf(ta, tb) < 1.0e-5f && 1.02f * sqrtf(W2f) * m2 * m2 < 0.3f * df && W2f < 1.0e30f &&
                             df < 1.0e30f && kf < 1.0e30f && A.sst_bound_ok;
        if (!settled) {
            // the exact rotation rate, formed again
            const double *u = A.u, *v = A.v, *w = A.w;
            const double v_r = v[c] * inv_rm, w_r = w[c] * inv_rm, cot = T.cotanthe[j];
            const double W12 = fma(u[c + kp] - u[c - kp], s_t, -v_r) - (v[c + P] - v[c - P]) * s_r;
            const double W13 = fma(u[ce] - u[cw], s_p, -w_r) - (w[c + P] - w[c - P]) * s_r;
            const double W23 = fma(v[ce] - v[cw], s_p, -(w_r * cot)) - (w[c + kp] - w[c - kp]) * s_t;
            const SstBlend B = sst_blend(tkc, dsc, inv_dis, qdiv(1.0, y_phys * A.inv_L_m), A.nue_air_nd, grad_dot,
                                         fma(W12, W12, fma(W13, W13, W23 * W23)));
            gam = B.F1 * gam1 + (1.0 - B.F1) * gam2;
            bet = B.F1 * bet1 + (1.0 - B.F1) * bet2;
            d_w = 2.0 * (1.0 - B.F1) * sig_w2;
            nue = B.nue;
        }
    }
    const double tke_safe = floor_at(tkc, 1.0e-20);
    const double kd = tke_safe * dsc, Y_k = bet_star * kd;
    const double P_k = cap_at(prod, 20.0 * Y_k);
    const double inv_k = in_rcp_range(tke_safe) ? recip_nr(tke_safe) : 1.0 / tke_safe;
    double tks = P_k - Y_k;
    const double P_w = gam * P_k * (dsc * inv_k);
    const double dss = fma(d_w * inv_dis, grad_dot, fma(-(bet * dsc), dsc, P_w));

    // the buoyancy sink of k (Turbulence.h:800-835): B = -nu_t N^2 / Pr_t, moist N^2 in saturated cells
    if (A.buoy != 0) {
        const double Tc = A.t[c] * A.t_ref, tref_dz = T.tref_dz[i];
        const bool fast_T = in_rcp_range(Tc);
        if (fast_T || Tc > 0.0) {
            const double inv_T = fast_T ? recip_nr(Tc) : 1.0 / Tc;
            double Gam = A.gam_ad, fac = 1.0;
            if (A.buoy == 3) {
                double rho = A.r_mix;
                if (A.local_rho) {
                    const double r_ = A.rho[c];
                    if (in_rcp_range(r_) || (r_ > 0.0 && isfinite(r_))) rho = r_;
                }
                const double inv_rho = in_rcp_range(rho) ? recip_nr(rho) : 1.0 / rho;
                const double inv_rT = inv_rho * inv_T;
                double a = 0.0, b = 0.0;
                bool moist = false;
                if (A.rmix_pos || rho > 0.0) {
#pragma unroll
                    for (int n = 0; n < 3; n++) {
                        const double qc = (floor_at(A.gc[n][c], 0.0) + floor_at(A.gi[n][c], 0.0)) * inv_rho;
                        if (!(bits_of(qc) > bits_of(1.0e-9) && bits_of(qc) <= INF_BITS)) continue;
                        const bool liquid = A.t0_pos ? bits_of(Tc) >= bits_of(A.t_0[n]) : Tc >= A.t_0[n];   // Tc > 0
                        const double q = floor_at(A.gv[n][c], 0.0) * inv_rT;
                        a = fma(liquid ? A.la[n] : A.sa[n], q, a);
                        b = fma(liquid ? A.lb[n] : A.sb[n], q * inv_T, b);
                        moist = true;
                    }
                }
                if (moist && finite_double(a + b)) {
                    fac = 1.0 + a;
                    Gam = Gam * fac * qdiv(1.0, 1.0 + b);
                }
            }
            if (bits_of(tref_dz) != 0ull) {
                const double N2 = A.g * inv_T * fma(A.t[c + P] - A.t[c - P], tref_dz, Gam) * fac;
                const unsigned long long nb = bits_of(N2);
                const bool positive = nb > 0ull && nb < INF_BITS;
                if (positive || (A.buoy == 2 && finite_double(N2))) tks = fma(-(floor_at(nue, 0.0) * N2), A.tL2_pr, tks);
            }
        }
    }
    // the caps after the source loop, from the floored k* (its background) and omega*
    const double tk_out = sst_floor(A, tkc, j, k);
    A.nue[c] = clip_positive(nue, A.nue_max);
    const double d20 = 20.0 * dsc;
    A.dss[c] = clip_to(dss, d20 * dsc);
    A.tks[c] = clip_to(tks, d20 * tk_out);
}

// k* and omega* at their floors (the passes before and after the source loop together)
__global__ void __launch_bounds__(256) turb_floor_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (!interior(A, i, j, k)) return;
    const int64_t c = cidx(A, i, j, k);
    A.tke[c] = sst_floor(A, floor_at(A.tke[c], 0.0), j, k);
    A.dis[c] = floor_at(A.dis[c], DIS_MIN);
}

// The wall copy at i = 0 and the cap of nue on the cells the source kernel leaves alone (no taper, a cap >= 0: it is then
// idempotent there). blockIdx.z: the planes i = 0 and im-1; the rows j = 0 and jm-1; the meridian km-1, and k = 0 where
// the seam is not periodic.
__global__ void __launch_bounds__(128) turb_edges_kernel(const TurbArgs A) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, im = A.im, jm = A.jm, km = A.km;
    int i, j, k;
    switch (blockIdx.z) {
        case 0: case 1: i = blockIdx.z ? im - 1 : 0; j = y; k = x; break;
        case 2: case 3: i = 1 + y; j = blockIdx.z == 3 ? jm - 1 : 0; k = x; break;
        default: i = 1 + y; j = 1 + x; k = blockIdx.z == 5 ? 0 : km - 1; break;
    }
    if (k >= km || j >= jm || (blockIdx.z >= 2 && i > im - 2) || (blockIdx.z >= 4 && j > jm - 2)) return;
    const int64_t c = cidx(A, i, j, k);
    double nue = A.nue[c];
    if (i == 0) {
        A.tke[c] = A.tke[c + A.plane];
        A.dis[c] = A.dis[c + A.plane];
        nue = A.nue[c + A.plane];
    }
    A.nue[c] = clip_positive(nue, A.nue_max);
}

__global__ void __launch_bounds__(128) turb_sources_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 4 + threadIdx.y, i = blockIdx.z;
    if (!interior(A, i, j, k)) return;
    sources_cell(A, i, j, k);
}

// the floors and caps after the source loop (Turbulence.h:634-643, 873-881)
__global__ void __launch_bounds__(256) turb_clamp_out_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (!interior(A, i, j, k)) return;
    const int64_t c = cidx(A, i, j, k);
    const double vs = A.vel_star[(int64_t)j * A.kp + k];
    const double k_bg = A.turb_free ? A.k_bg_nd : 0.01 * vs * vs / (sqrt(C_NUE) * A.u_0 * A.u_0);
    const double tk = dmax(k_bg, A.tke[c]);
    const double ds = dmax(DIS_MIN, A.dis[c]);
    A.tke[c] = tk;
    A.dis[c] = ds;
    A.nue[c] = clamp3(A.nue[c], 0.0, A.nue_max);
    const double dsm = 20.0 * ds * ds;
    A.dss[c] = clamp3(A.dss[c], -dsm, dsm);
    const double tsm = 20.0 * tk * ds;
    A.tks[c] = clamp3(A.tks[c], -tsm, tsm);
}

// apply_wall_bc (Turbulence.h:382-423) without an obstacle: the zero-gradient copy at i = 0
__global__ void turb_wall_kernel(const TurbArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (k >= A.km || j >= A.jm) return;
    const int64_t c0 = cidx(A, 0, j, k), c1 = c0 + A.plane;
    A.tke[c0] = A.tke[c1];
    A.dis[c0] = A.dis[c1];
    A.nue[c0] = A.nue[c1];
}

// clamp_nue (Turbulence.h:564-589)
__global__ void __launch_bounds__(256) turb_nue_cap_kernel(const TurbArgs A) {
    const int k = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, i = blockIdx.z;
    if (k >= A.km || j >= A.jm) return;
    double f = 1.0;
    if (A.abl_taper) {
        const double z_agl = A.tab.height_m[i] - A.tab.height_m[0];
        f = clamp3((A.abl_height + A.taper_dz - z_agl) / A.taper_dz, 0.0, 1.0);
    }
    const int64_t c = cidx(A, i, j, k);
    A.nue[c] = clamp3(A.nue[c], 0.0, A.nue_max) * f;
}

// seam_copy (Turbulence.h:542-561) and fill_lid_corners (:510-540), the closure's eight arrays
__device__ __forceinline__ double* turb_array(const TurbArgs& A, int q) {
    switch (q) {
        case 0: return A.tke; case 1: return A.dis; case 2: return A.tken; case 3: return A.disn;
        case 4: return A.nue; case 5: return A.prod; case 6: return A.tks; default: return A.dss;
    }
}

__global__ void turb_seam_kernel(const TurbArgs A) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= A.im * A.jm * 8) return;
    const int q = e % 8, r = e / 8;
    double* a = turb_array(A, q);
    const int64_t row = (int64_t)r * A.kp;
    a[row + A.km - 1] = a[row];
}

__global__ void turb_corners_kernel(const TurbArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
    if (k >= A.km) return;
    double* a = turb_array(A, q);
    const int il = A.im - 1, jm = A.jm;
    a[cidx(A, il, 0, k)] = 0.5 * (a[cidx(A, il, 1, k)] + a[cidx(A, il - 1, 0, k)]);
    a[cidx(A, il, jm - 1, k)] = 0.5 * (a[cidx(A, il, jm - 2, k)] + a[cidx(A, il - 1, jm - 1, k)]);
}

// bc_turb_active false: the lid from i = im-2 (j = 1..jm-2), then the pole rows from j = 1, jm-2 at every level
__global__ void turb_lid_kernel(const TurbArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = 1 + blockIdx.y, q = blockIdx.z;
    if (k >= A.km || j > A.jm - 2) return;
    double* a = turb_array(A, q);
    a[cidx(A, A.im - 1, j, k)] = a[cidx(A, A.im - 2, j, k)];
}
__global__ void turb_poles_kernel(const TurbArgs A) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y, q = blockIdx.z;
    if (k >= A.km || i >= A.im) return;
    double* a = turb_array(A, q);
    a[cidx(A, i, 0, k)] = a[cidx(A, i, 1, k)];
    a[cidx(A, i, A.jm - 1, k)] = a[cidx(A, i, A.jm - 2, k)];
}

}  // namespace

cudaError_t launch_turbulence(const KConst& K, const atsat_dyn_params& p, const atsat_dyn_turb_params& tp,
                              const TurbTables& tab, double* const* f, double* prod, double* vel_star, cudaStream_t s,
                              int* launches) {
    TurbArgs A{};
    A.im = K.im; A.jm = K.jm; A.km = K.km; A.kp = K.kp; A.plane = K.plane;
    A.periodic = p.phi_periodic; A.model = tp.model; A.turb_free = tp.turb_free; A.curv = tp.curv; A.buoy = tp.buoy;
    A.abl_taper = tp.abl_taper; A.local_rho = p.local_rho; A.turb_active = p.turb_active;
    A.u_0 = p.u_0; A.t_ref = p.t_ref; A.g = p.g; A.cp_mix = p.cp_mix; A.r_mix = p.r_mix; A.R_mix = p.R_mix;
    A.L_m = p.L_atm * 1.0e3;
    A.nue_air = tp.nue_gas;
    A.re_turb = tp.vel_star_ref * tp.z_0 / tp.nue_gas;
    A.nue_max = tp.nue_max_phys / (p.u_0 * A.L_m) + 0.0;     // -0 becomes +0, which compares the same
    if (std::isnan(A.nue_max)) A.nue_max = std::fabs(A.nue_max);
    A.k_bg_nd = tp.k_bg / (p.u_0 * p.u_0);
    A.vel_star_max = tp.vel_star_max;
    A.dr = tab.dr; A.dthe = tab.dthe; A.dphi = tab.dphi;
    A.inv_2dr = 1.0 / (2.0 * tab.dr);
    A.inv_L_m = 1.0 / A.L_m;
    A.nue_air_nd = A.nue_air / (A.u_0 * A.L_m);
    A.gam_ad = p.g / p.cp_mix;
    A.tL2_pr = (A.L_m / A.u_0) * (A.L_m / A.u_0) / 0.9;
    A.inv_R_mix = 1.0 / p.R_mix;
    A.inv_cpR = 1.0 / (p.cp_mix * p.R_mix);
    A.inv_2dr2 = A.inv_2dr * A.inv_2dr;
    A.inv_ys_free_f = (float)(1.0 / (1.0e20 * A.inv_L_m));
    A.nue_air_nd_f = (float)A.nue_air_nd;
    A.kbg_pos = A.k_bg_nd >= 0.0;
    A.rmix_pos = p.r_mix > 0.0;
    A.t0_pos = tp.t_0[0] > 0.0 && tp.t_0[1] > 0.0 && tp.t_0[2] > 0.0;
    A.sst_bound_ok = A.inv_ys_free_f > 1.0e-30f && A.inv_ys_free_f < 1.0e30f && A.nue_air_nd_f >= 0.0f && A.nue_air_nd_f < 1.0e30f;
    A.abl_height = tp.abl_height;
    A.taper_dz = tab.taper_dz;
    for (int n = 0; n < 3; n++) { A.ep[n] = tp.ep[n]; A.lv[n] = tp.lv[n]; A.ls[n] = tp.ls[n]; A.t_0[n] = tp.t_0[n]; }
    for (int n = 0; n < 3; n++) {
        A.la[n] = tp.lv[n] * A.inv_R_mix;
        A.sa[n] = tp.ls[n] * A.inv_R_mix;
        A.lb[n] = tp.ep[n] * tp.lv[n] * tp.lv[n] * A.inv_cpR;
        A.sb[n] = tp.ep[n] * tp.ls[n] * tp.ls[n] * A.inv_cpR;
    }
    A.tab = tab;
    A.u = f[ATSAT_F_U]; A.v = f[ATSAT_F_V]; A.w = f[ATSAT_F_W]; A.t = f[ATSAT_F_T]; A.rho = f[ATSAT_F_RHO_MIX];
    A.tke = f[ATSAT_F_TKE]; A.dis = f[ATSAT_F_DIS]; A.tken = f[ATSAT_F_TKEN]; A.disn = f[ATSAT_F_DISN];
    A.nue = f[ATSAT_F_NUE]; A.tks = f[ATSAT_F_TKE_SOURCE]; A.dss = f[ATSAT_F_DIS_SOURCE];
    A.prod = prod; A.vel_star = vel_star;
    const int gv[3] = {ATSAT_F_H2O, ATSAT_F_NH3, ATSAT_F_CH4};
    const int gc[3] = {ATSAT_F_H2O_CLOUD, ATSAT_F_NH3_CLOUD, ATSAT_F_CH4_CLOUD};
    const int gi[3] = {ATSAT_F_H2O_ICE, ATSAT_F_NH3_ICE, ATSAT_F_CH4_ICE};
    for (int n = 0; n < 3; n++) { A.gv[n] = f[gv[n]]; A.gc[n] = f[gc[n]]; A.gi[n] = f[gi[n]]; }

    const dim3 b8(32, 8), g8((K.km + 31) / 32, (K.jm + 7) / 8, K.im);
    const dim3 b4(32, 4), g4((K.km + 31) / 32, (K.jm + 3) / 4, K.im);
    turb_vel_star_kernel<<<dim3((K.km + 127) / 128, K.jm), 128, 0, s>>>(A);
    const dim3 gw((K.km + 127) / 128, K.jm);
    if (tp.model == ATSAT_TURB_K_OMEGA_SST) {
        sst_kernel<<<g4, b4, 0, s>>>(A);
        turb_floor_kernel<<<g8, b8, 0, s>>>(A);
        *launches += 3;
        if (tp.abl_taper || !(A.nue_max >= 0.0)) {           // capping twice is not capping once
            turb_wall_kernel<<<gw, 128, 0, s>>>(A);
            turb_nue_cap_kernel<<<g8, b8, 0, s>>>(A);
            *launches += 2;
        } else {
            const int width = K.km > K.jm ? K.km : K.jm, rows = K.jm > K.im ? K.jm : K.im;
            turb_edges_kernel<<<dim3((width + 127) / 128, rows, p.phi_periodic ? 5 : 6), 128, 0, s>>>(A);
            *launches += 1;
        }
    } else {
        turb_clamp_in_kernel<<<g8, b8, 0, s>>>(A);
        turb_sources_kernel<<<g4, b4, 0, s>>>(A);
        turb_clamp_out_kernel<<<g8, b8, 0, s>>>(A);
        turb_wall_kernel<<<gw, 128, 0, s>>>(A);
        turb_nue_cap_kernel<<<g8, b8, 0, s>>>(A);
        *launches += 6;
    }
    if (p.phi_periodic) {
        turb_seam_kernel<<<(K.im * K.jm * 8 + 255) / 256, 256, 0, s>>>(A);
        *launches += 1;
    }
    if (tp.turb_free) {
        if (p.turb_active) {
            turb_corners_kernel<<<dim3((K.km + 127) / 128, 8), 128, 0, s>>>(A);
            *launches += 1;
        } else {
            turb_lid_kernel<<<dim3((K.km + 127) / 128, K.jm - 2, 8), 128, 0, s>>>(A);
            turb_poles_kernel<<<dim3((K.km + 127) / 128, K.im, 8), 128, 0, s>>>(A);
            *launches += 2;
        }
    }
    return cudaGetLastError();
}

}  // namespace atsat
