// The two optional passes of PressureSolver<cSaturnModel>::run, FP64, run after each sweep's red-black
// colours (PressureSolver.h:300-316, 502-708, 750-755):
//
// PRESS_LINE: per colour ((j + k) & 1) every (j, k) column is relaxed exactly in r -- a Thomas solve over
// i = 1..im-2 with the theta / phi neighbours lagged and both radial ends folded (p0 = c43 p1 - c13 p2) --
// and after the boundary pass the interior mean of p_dyn is held at its value on entry. One thread per
// column; the matrix does not depend on k, so its elimination is tabulated once per (i, j) (LineGeo). The columns of one
// colour read only the other colour, except across an odd periodic seam where k = 0 and k = km-2 share a
// colour: as in a single thread's visit of the reference's loop, k = km-2 is solved after k = 0 (a second
// launch) and reads its new values.
//
// PRESS_BAROTROPIC: the column residual R(j, k) = sum_i (src - Lc(p)) / sum_i 1/rm^2, its real DFT over
// the N = km-1 meridians (press_baro_fft.cu; modes below 1e-12 of the row's sum |R| dropped), per mode a
// tridiagonal in theta (mode 0 made consistent, pinned at j = 1, shifted to zero sin-weighted mean; its elimination
// tabulated too), and the correction q(j, k) added to every level of the column.
//
// Rounding. The residual is a sum of nearly cancelling terms and the theta solve amplifies its rounding, so this file is
// compiled without multiply-add contraction and the line pass and the residual take the values that the reference's
// expressions round to: quotients by a tabulated divisor are formed from its reciprocal and corrected to the division's
// own rounding (div_tab). The theta solve itself does not: products with rounded reciprocals, fused multiply-adds and
// mode 0's sums across a warp. Its error is not what counts: over 66 seeded states on four grids the pass's error
// against long double is that of the reference's form (medians of the rms, in 1e-16: 10x20x36 9.6 and now 8.3,
// 21x91x182 107 and 104, 27x118x222 185 and 189).
//
// Weights: lc_num1..3 of ColGeo are the line pass's num1, num2, num3 expression for expression.
#include "dyn_common.cuh"

namespace atsat {
namespace {

__device__ __forceinline__ double ldg(const double* p) { return __ldg(p); }

// isfinite on the integer pipe
__device__ __forceinline__ bool finite_bits(double x) {
    uint32_t lo, hi;
    split_f64(x, lo, hi);
    return (hi & 0x7FF00000u) != 0x7FF00000u;
}

// x / d from y = 1 / d (rounded): two corrections by the exact residual give the correctly rounded quotient where
// nothing over- or underflows (P. Markstein, IA-64 and Elementary Functions, 2000, ch. 8); the division elsewhere. Five
// FP64 operations in a chain instead of about a dozen and a call.
__device__ __forceinline__ double div_tab(double x, double d, double y) {
    double q = x * y;
    uint32_t lo, hi;
    split_f64(q, lo, hi);
    if (((hi >> 20) & 0x7FFu) - 200u < 1600u) {
        q = fma(fma(-q, d, x), y, q);
        return fma(fma(-q, d, x), y, q);
    }
    return x / d;
}

// The elimination of a column's matrix per (i, j): the coupling to the row above as eliminated (a), the pivot and its
// reciprocal, and cp (PressureSolver.h:506-567 with the fold of both ends).
__global__ void line_table_kernel(const KConst K, const ColGeo* __restrict__ geo, LineGeo* __restrict__ tab) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < 1 || j > K.jm - 2) return;
    const int lo = 1, hi = K.im - 2;
    const bool fold = hi > lo;
    double cprev = 0.0;
    for (int i = lo; i <= hi; i++) {
        const ColGeo* g = geo + ((int64_t)i * K.jm + j);
        const double num1 = g->lc_num1, num2 = g->lc_num2, num3 = g->lc_num3;
        double a = -num1, b = 2.0 * (num1 + num2 + num3), cc = -num1;
        if (i == lo && fold) { b += a * K.c43; cc -= a * K.c13; }
        if (i == hi && fold) { b += cc * K.c43; a -= cc * K.c13; }
        const double dn = i == lo ? b : b - a * cprev;
        LineGeo& t = tab[(int64_t)i * K.jm + j];
        t.num1 = num1; t.num2 = num2; t.num3 = num3;
        t.a = a; t.dn = dn; t.rdn = 1.0 / dn;
        t.cp = cprev = cc / dn;
        t.pad = 0.0;
    }
}

// One column. Bound by the FP64 pipe: 15 operations per cell, where forming the elimination in every column took about
// 45 and two divisions (151 us per colour at 41x181x361; 39 dependent steps per thread, the loads of LINE_AHEAD levels
// issued ahead; 4 to 13 measured alike): 64 us.
constexpr int LINE_AHEAD = 4;

__device__ void line_column(const KConst& K, const LineGeo* __restrict__ tab, const double* __restrict__ src,
                            double* __restrict__ p, double* __restrict__ dpb, int j, int k) {
    const int64_t P = K.plane, kp = K.kp;
    const int kw = (k == 0) ? K.km - 2 : k - 1;
    const int ke = (k == K.km - 2) ? 0 : k + 1;
    const int lo = 1, hi = K.im - 2;
    double dprev = 0.0;
    const int64_t c1 = ((int64_t)lo * K.jm + j) * kp + k;
    for (int i0 = lo; i0 <= hi; i0 += LINE_AHEAD) {
        double n[LINE_AHEAD], s[LINE_AHEAD], e[LINE_AHEAD], w[LINE_AHEAD], f[LINE_AHEAD];
#pragma unroll
        for (int u = 0; u < LINE_AHEAD; u++) {
            const int64_t c = c1 + (int64_t)(i0 - lo + u) * P;
            if (i0 + u <= hi) {
                n[u] = p[c - kp]; s[u] = p[c + kp]; e[u] = p[c - k + ke]; w[u] = p[c - k + kw]; f[u] = ldg(src + c);
            }
        }
#pragma unroll
        for (int u = 0; u < LINE_AHEAD; u++) {
            const int i = i0 + u;
            if (i > hi) break;
            const LineGeo& t = tab[(int64_t)i * K.jm + j];
            const double d = t.num2 * (s[u] + n[u]) + t.num3 * (e[u] + w[u]) - f[u];
            dprev = div_tab(i == lo ? d : d - t.a * dprev, t.dn, t.rdn);
            dpb[c1 + (int64_t)(i - lo) * P] = dprev;
        }
    }
    double x = dprev;
    int64_t c = c1 + (int64_t)(hi - lo) * P;
    if (finite_bits(x)) p[c] = x;
#pragma unroll 4
    for (int i = hi - 1; i >= lo; i--) {
        c -= P;
        x = dpb[c] - tab[(int64_t)i * K.jm + j].cp * x;
        if (finite_bits(x)) p[c] = x;
    }
}

constexpr int LINE_THREADS = 64;   // 181 columns of a colour and row are 3 x 64: the blocks even out over the SMs

__global__ void __launch_bounds__(LINE_THREADS) line_kernel(const KConst K, const LineGeo* __restrict__ tab,
                                                   const double* __restrict__ src, double* __restrict__ p,
                                                   double* __restrict__ dpb, int colour) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    if (j > K.jm - 2) return;
    const int k = 2 * m + ((colour - j) & 1);
    if (k > K.km - 2) return;
    if (k == K.km - 2 && k > 0 && ((K.km - 1) & 1)) return;     // after its seam partner k = 0
    line_column(K, tab, src, p, dpb, j, k);
}

__global__ void line_seam_kernel(const KConst K, const LineGeo* __restrict__ tab, const double* __restrict__ src,
                                 double* __restrict__ p, double* __restrict__ dpb, int colour) {
    const int j = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (j > K.jm - 2) return;
    const int k = K.km - 2;
    if (((j + k) & 1) != colour) return;
    line_column(K, tab, src, p, dpb, j, k);
}

// ---- interior mean (PressureSolver.h:310-316): per level partial sums over row chunks, then in order ----
constexpr int IM_CHUNKS = 16;

__global__ void __launch_bounds__(128) imean_partial_kernel(const KConst K, const double* __restrict__ p,
                                                            double* __restrict__ partial) {
    const int i = 1 + blockIdx.x, chunk = blockIdx.y;
    const int nj = K.jm - 2;
    const int j0 = 1 + (int)((int64_t)nj * chunk / IM_CHUNKS), j1 = 1 + (int)((int64_t)nj * (chunk + 1) / IM_CHUNKS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
    for (int j = j0 + warp; j < j1; j += 4) {
        const double* row = p + ((int64_t)i * K.jm + j) * K.kp;
#pragma unroll 4
        for (int k = lane; k <= K.km - 2; k += 32) s += ldg(row + k);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ double ws[4];
    if (lane == 0) ws[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) partial[(int64_t)(i - 1) * IM_CHUNKS + chunk] = ((ws[0] + ws[1]) + ws[2]) + ws[3];
}

__global__ void imean_final_kernel(const double* __restrict__ partial, int n, double count, double* __restrict__ out) {
    double s = 0.0;
    for (int q = threadIdx.x; q < n; q += 32) s += partial[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *out = s / count;
}

// p -= mean_now - mean_entry on every cell (PressureSolver.h:750-755)
__global__ void __launch_bounds__(256) mean_shift_kernel(const KConst K, double* __restrict__ p,
                                                         const double* __restrict__ mean) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int i = blockIdx.z;
    if (k >= K.km || j >= K.jm) return;
    const double shift = mean[1] - mean[0];
    p[((int64_t)i * K.jm + j) * K.kp + k] -= shift;
}

// ---- PRESS_BAROTROPIC (PressureSolver.h:573-708) ----
// the column residual of PressureSolver.h:581-604, end rows read as the boundary pass sets them. 13 FP64 operations per
// cell, each rounded as the reference's ((x + y) - 2 p0 as one fma: the product is exact); the column marches in i with
// its radial neighbours in registers, and the polar rows' folds and the lid are branches of
// their own, not predicated instructions that would take the pipe's slots: 183 -> 86 us at 41x181x361 (the operations
// alone are 52).
template <bool NORTH, bool SOUTH>
__device__ __forceinline__ double column_residual(const KConst& K, const ColGeo* __restrict__ geo,
                                                  const double* __restrict__ src, const double* __restrict__ p, int j, int k) {
    const int N = K.km - 1;
    const int kw = (k == 0) ? N - 1 : k - 1;
    const int ke = (k == N - 1) ? 0 : k + 1;
    const int64_t P = K.plane, kp = K.kp;
    int64_t c = ((int64_t)K.jm + j) * kp + k;
    double s = 0.0, p0 = p[c], pn = p[c + P];
    double pm = K.c43 * p0 - K.c13 * pn;                     // i = 0
    const ColGeo* g = geo + ((int64_t)K.jm + j);
    auto term = [&](double pip) {
        const double pjp = SOUTH ? K.c43 * p0 - K.c13 * p[c - kp] : p[c + kp];
        const double pjm = NORTH ? K.c43 * p0 - K.c13 * p[c + kp] : p[c - kp];
        const double lc = ldg(&g->lc_num1) * fma(-2.0, p0, pip + pm)
                        + ldg(&g->lc_num2) * fma(-2.0, p0, pjp + pjm)
                        + ldg(&g->lc_num3) * fma(-2.0, p0, p[c - k + ke] + p[c - k + kw]);
        s += ldg(src + c) - lc;
    };
#pragma unroll 4
    for (int i = 1; i < K.im - 2; i++) {
        const double ahead = p[c + 2 * P];                   // level i + 2: an interior level or the lid (not used)
        term(pn);
        pm = p0;
        p0 = pn;
        pn = ahead;
        c += P;
        g += K.jm;
    }
    term(K.c43 * p0 - K.c13 * pm);                           // the level below the lid
    return s;
}

__global__ void __launch_bounds__(128) baro_resid_kernel(const KConst K, const ColGeo* __restrict__ geo,
                                                         const double* __restrict__ src, const double* __restrict__ p,
                                                         double A2, double* __restrict__ R) {
    const int N = K.km - 1;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    if (k >= N || j > K.jm - 2) return;
    const double s = j == 1 ? column_residual<true, false>(K, geo, src, p, j, k)
                   : j == K.jm - 2 ? column_residual<false, true>(K, geo, src, p, j, k)
                                   : column_residual<false, false>(K, geo, src, p, j, k);
    R[(int64_t)(j - 1) * N + k] = s / A2;
}

// The elimination of each mode's tridiagonal in theta (PressureSolver.h:638-680): cp, the pivot's reciprocal and the
// coupling times it at [jj * NU + mode]; mode 0's weight sums.
__global__ void baro_table_kernel(const BaroTables B, double e, double c43, double c13) {
    const int mm = blockIdx.x * blockDim.x + threadIdx.x;
    if (mm > B.NM) return;
    const int J = B.J;
    const double lam = B.lam[mm];
    double cprev = 0.0;
    for (int jj = 0; jj < J; jj++) {
        const double s_ = B.sinthe[jj + 1];
        double a = e, b = -2.0 * e - lam / (s_ * s_), c = e;
        if (jj == 0) { a = 0.0; b += c43 * e; c -= c13 * e; }
        if (jj == J - 1) { c = 0.0; b += c43 * e; a -= c13 * e; }
        if (mm == 0 && jj == 0) { b = 1.0; c = 0.0; }
        const double dn = jj == 0 ? b : b - a * cprev;
        const int64_t o = (int64_t)jj * B.NU + mm;
        B.rdn[o] = 1.0 / dn;
        B.ar[o] = a / dn;
        B.cp[o] = cprev = c / dn;
    }
    if (mm == 0) {
        double ys = 0.0, sw = 0.0;
        for (int jj = 0; jj < J; jj++) {
            ys += ((jj == 0 || jj == J - 1) ? 1.5 : 1.0) * B.abs_sin[jj];
            sw += B.abs_sin[jj];
        }
        B.sums[0] = ys;
        B.sums[1] = sw;
    }
}

// One lane per (mode, part), block 0 mode 0 alone: its sums over theta are chains of their own. What counts is the chain,
// one fma a row each way; what it reads is loaded a batch of MODES_AHEAD rows ahead, side by side over the modes. With
// the elimination formed in the chain (two divisions a row) and a mode's rows read one by one it took 809 us at
// 41x181x361, with tabulated divisors and quotients rounded as the division's 163 us; now 70 us, most
// of it mode 0's.
constexpr int MODES_AHEAD = 8;

__global__ void __launch_bounds__(32) baro_modes_kernel(const BaroTables B) {
    const int J = B.J, NM = B.NM;
    const int lane = threadIdx.x;
    const int u = ((int)blockIdx.x - 1) * 32 + lane;         // modes 1 .. NM of part 0, then of part 1
    const bool zero = blockIdx.x == 0;
    const int mm = zero ? 0 : (u < NM ? u + 1 : u - NM + 1), part = zero || u < NM ? 0 : 1;
    if (!zero && (u >= 2 * NM || (part == 1 && 2 * mm == B.N))) return;
    double* __restrict__ d = (part == 0 ? B.Ac : B.As) + mm;
    const double* __restrict__ ar = B.ar + mm;
    const double* __restrict__ rdn = B.rdn + mm;
    const double* __restrict__ cp = B.cp + mm;
    const int NU = B.NU;
    auto warp_sum = [](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    if (zero) {                                              // the whole warp; then lane 0 solves
        double yr = 0.0;
        for (int jj = lane; jj < J; jj += 32) yr += ((jj == 0 || jj == J - 1) ? 1.5 : 1.0) * d[(int64_t)jj * NU];
        const double f = warp_sum(yr) / B.sums[0];
        for (int jj = lane; jj < J; jj += 32) {
            const int64_t o = (int64_t)jj * NU;
            d[o] = jj == 0 ? 0.0 : d[o] - f * B.abs_sin[jj];
        }
        __syncwarp();
    }
    double dprev = 0.0;
    double x[MODES_AHEAD], c[MODES_AHEAD];
    auto forward = [&](int j0) {
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++)
            if (j0 + q < J) {
                const int64_t o = (int64_t)(j0 + q) * NU;
                x[q] = d[o] * rdn[o];
                c[q] = ar[o];
            }
    };
    const int Jn = zero && lane ? 0 : J;                     // rows this lane solves
    if (Jn) forward(0);
    for (int j0 = 0; j0 < Jn; j0 += MODES_AHEAD) {
        double y[MODES_AHEAD], b[MODES_AHEAD];
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++) { y[q] = x[q]; b[q] = c[q]; }
        forward(j0 + MODES_AHEAD);
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++) {
            if (j0 + q >= J) break;
            dprev = fma(-b[q], dprev, y[q]);
            d[(int64_t)(j0 + q) * NU] = dprev;
        }
    }
    auto backward = [&](int j0) {
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++)
            if (j0 - q >= 0) {
                const int64_t o = (int64_t)(j0 - q) * NU;
                x[q] = d[o];
                c[q] = cp[o];
            }
    };
    if (Jn) backward(J - 2);
    for (int j0 = Jn - 2; j0 >= 0; j0 -= MODES_AHEAD) {
        double y[MODES_AHEAD], b[MODES_AHEAD];
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++) { y[q] = x[q]; b[q] = c[q]; }
        backward(j0 - MODES_AHEAD);
#pragma unroll
        for (int q = 0; q < MODES_AHEAD; q++) {
            if (j0 - q < 0) break;
            dprev = fma(-b[q], dprev, y[q]);
            d[(int64_t)(j0 - q) * NU] = dprev;
        }
    }
    if (zero) {
        __syncwarp();
        double sq = 0.0;
        for (int jj = lane; jj < J; jj += 32) sq += B.abs_sin[jj] * d[(int64_t)jj * NU];
        const double f = warp_sum(sq) / B.sums[1];
        for (int jj = lane; jj < J; jj += 32) d[(int64_t)jj * NU] -= f;
    }
}

// q(j, k) added to every level of the column (PressureSolver.h:684-697)
__global__ void __launch_bounds__(256) baro_add_kernel(const KConst K, int N, const double* __restrict__ q,
                                                       double* __restrict__ p) {
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = 1 + blockIdx.y * 8 + threadIdx.y;
    if (k >= N || j > K.jm - 2) return;
    const double v = ldg(q + (int64_t)(j - 1) * N + k);
    const int i0 = blockIdx.z * 4;
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (i0 + u < K.im) p[((int64_t)(i0 + u) * K.jm + j) * K.kp + k] += v;
}

}  // namespace

cudaError_t launch_line_table(const KConst& kc, const ColGeo* geo, LineGeo* tab, cudaStream_t s) {
    line_table_kernel<<<(kc.jm + 63) / 64, 64, 0, s>>>(kc, geo, tab);
    return cudaGetLastError();
}

cudaError_t launch_line_pass(const KConst& kc, const LineGeo* tab, const double* src, double* p, double* dpb, int colour,
                             cudaStream_t s, int* launches) {
    const int nm = (kc.km - 1 + 1) / 2 + 1;
    line_kernel<<<dim3((nm + LINE_THREADS - 1) / LINE_THREADS, kc.jm - 2), LINE_THREADS, 0, s>>>(kc, tab, src, p, dpb, colour);
    *launches += 1;
    if (((kc.km - 1) & 1) && kc.km - 2 > 0) {
        line_seam_kernel<<<(kc.jm - 2 + 127) / 128, 128, 0, s>>>(kc, tab, src, p, dpb, colour);
        *launches += 1;
    }
    return cudaGetLastError();
}

// the interior mean of p into *out; partial holds (im-2) * IM_CHUNKS doubles
cudaError_t launch_interior_mean(const KConst& kc, const double* p, double* partial, double* out, cudaStream_t s,
                                 int* launches) {
    const int n = (kc.im - 2) * IM_CHUNKS;
    const double count = (double)((int64_t)(kc.im - 2) * (kc.jm - 2) * (kc.km - 1));
    imean_partial_kernel<<<dim3(kc.im - 2, IM_CHUNKS), 128, 0, s>>>(kc, p, partial);
    imean_final_kernel<<<1, 32, 0, s>>>(partial, n, count, out);
    *launches += 2;
    return cudaGetLastError();
}

int interior_mean_partials(const KConst& kc) { return (kc.im - 2) * IM_CHUNKS; }

cudaError_t launch_mean_shift(const KConst& kc, double* p, const double* mean, cudaStream_t s) {
    mean_shift_kernel<<<dim3((kc.km + 31) / 32, (kc.jm + 7) / 8, kc.im), dim3(32, 8), 0, s>>>(kc, p, mean);
    return cudaGetLastError();
}

cudaError_t launch_baro_table(const KConst& kc, const BaroTables& T, cudaStream_t s) {
    baro_table_kernel<<<(T.NM + 1 + 31) / 32, 32, 0, s>>>(T, kc.inv_dthe2, kc.c43, kc.c13);
    return cudaGetLastError();
}

cudaError_t launch_barotropic(const KConst& kc, const ColGeo* geo, const double* src, double* p, const BaroTables& T,
                              cudaStream_t s, int* launches) {
    const int N = T.N, J = T.J;
    baro_resid_kernel<<<dim3((N + 127) / 128, J), 128, 0, s>>>(kc, geo, src, p, T.A2, T.R);
    cudaError_t e = launch_baro_forward(T, s);
    if (e != cudaSuccess) return e;
    baro_modes_kernel<<<1 + (2 * T.NM + 31) / 32, 32, 0, s>>>(T);
    if ((e = launch_baro_inverse(T, s)) != cudaSuccess) return e;
    baro_add_kernel<<<dim3((N + 31) / 32, (J + 7) / 8, (kc.im + 3) / 4), dim3(32, 8), 0, s>>>(kc, N, T.R, p);
    *launches += 5;
    return cudaGetLastError();
}

}  // namespace atsat
