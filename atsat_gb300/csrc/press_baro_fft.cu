// The transforms over phi of PRESS_BAROTROPIC (PressureSolver.h:606-636, 684-697): the column residual's cosine and sine
// sums per row and mode, and the correction back on the meridians.
//
// Two rows per complex transform, one block each (poisson_spectral.cuh). The reference's sums run over the meridians in
// order, n terms each; the transform's rounding error is smaller than theirs, but relative to the larger of its two rows.
// So each row enters scaled by a power of two that brings its sum of magnitudes to [1, 2) and leaves unscaled, both
// exact: the error is then relative to the row itself, as the reference's is and as its dropping of modes below 1e-12 of
// the row's own sum needs (the noise of a row 1e4 times stronger would pass for modes of the weak one). As direct sums, a
// thread per (row, mode), the two passes took 163 and 159 us at 41x181x361 (179 rows of 360), the row sums 32 us; as
// transforms 14 and 15 us (13.5 and 11.5 unscaled).
#include "poisson_spectral.cuh"

namespace atsat {
namespace {

using namespace spectral;

// The pairs alone do not fill the GPU (90 at 41x181x361) and the FP64 chains are long: four warps share a transform
// (30.5 us with one warp per pair).
constexpr int BT = 128;

__device__ __forceinline__ Cx<double>* tables(unsigned char* dsm, const BaroTables& B, Cx<double>*& buf) {
    Cx<double>* tw = reinterpret_cast<Cx<double>*>(dsm);
    buf = tw + B.N;
    for (int k = threadIdx.x; k < B.N; k += blockDim.x) tw[k] = {B.ct[k], B.st[k]};
    return tw;
}

__device__ __forceinline__ double keep(double x, double tol) { return fabs(x) < tol ? 0.0 : x; }

// the sums over the block of a and b
__device__ __forceinline__ void block_sums(double& a, double& b) {
    __shared__ double ws[2][BT / 32];
    const int t = threadIdx.x;
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if ((t & 31) == 0) { ws[0][t >> 5] = a; ws[1][t >> 5] = b; }
    __syncthreads();
    a = (ws[0][0] + ws[0][1]) + (ws[0][2] + ws[0][3]);
    b = (ws[1][0] + ws[1][1]) + (ws[1][2] + ws[1][3]);
}

// A row's scale from its sum of magnitudes m: x = 2^-e brings m to [1, 2), y = 2^e undoes it; y = 0 for a row of zeros,
// x = y = 1 where m is subnormal or not finite.
struct RowScale { double x, y; };
__device__ __forceinline__ RowScale row_scale(double m) {
    if (m == 0.0) return {1.0, 0.0};
    const int e = (__double2hiint(m) >> 20) & 0x7FF;
    if (e == 0 || e >= 0x7FE) return {1.0, 1.0};
    return {__hiloint2double((0x7FE - e) << 20, 0), __hiloint2double(e << 20, 0)};
}

__global__ void baro_forward_kernel(const BaroTables B, const FftPlan F) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Cx<double>* buf;
    const Cx<double>* tw = tables(dsm, B, buf);
    const int t = threadIdx.x, N = B.N, jj = 2 * blockIdx.x;
    Cx<double>* a = buf;
    const bool two = jj + 1 < B.J;
    const double* r0 = B.R + (int64_t)jj * N;
    double ra0 = 0.0, ra1 = 0.0;
    for (int k = t; k < N; k += BT) {
        const double x = r0[k], y = two ? r0[N + k] : 0.0;
        a[k] = {x, y};
        ra0 += fabs(x);
        ra1 += fabs(y);
    }
    block_sums(ra0, ra1);
    const RowScale f0 = row_scale(ra0), f1 = row_scale(ra1);
    for (int k = t; k < N; k += BT) a[k] = {a[k].re * f0.x, a[k].im * f1.x};
    __syncthreads();
    const Cx<double>* z = fft(a, a + F.stride, tw, N, F, t, BT, [] { __syncthreads(); });
    // modes below 1e-12 of the row's sum |R| are dropped (mode 0 is kept)
    for (int m = t; m <= B.NM; m += BT) {
        const Cx<double> u = z[m], v = z[m ? N - m : 0];
        const double t0 = m ? 1.0e-12 * ra0 : 0.0, t1 = m ? 1.0e-12 * ra1 : 0.0;
        const int64_t o = (int64_t)jj * B.NU + m;
        const double h0 = 0.5 * f0.y, h1 = 0.5 * f1.y;
        B.Ac[o] = keep(h0 * (u.re + v.re), t0);
        B.As[o] = keep(h0 * (v.im - u.im), t0);
        if (two) {
            B.Ac[o + B.NU] = keep(h1 * (u.im + v.im), t1);
            B.As[o + B.NU] = keep(h1 * (u.re - v.re), t1);
        }
    }
}

__global__ void baro_inverse_kernel(const BaroTables B, const FftPlan F) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Cx<double>* buf;
    const Cx<double>* tw = tables(dsm, B, buf);
    const int t = threadIdx.x, N = B.N, jj = 2 * blockIdx.x;
    Cx<double>* z = buf;
    const bool two = jj + 1 < B.J;
    double s0 = 0.0, s1 = 0.0;
    for (int m = t; m <= B.NM; m += BT) {
        const int64_t o = (int64_t)jj * B.NU + m;
        const bool real = m == 0 || 2 * m == N;                // its sine sums are not used
        s0 += fabs(B.Ac[o]) + (real ? 0.0 : fabs(B.As[o]));
        if (two) s1 += fabs(B.Ac[o + B.NU]) + (real ? 0.0 : fabs(B.As[o + B.NU]));
    }
    block_sums(s0, s1);
    const RowScale f0 = row_scale(s0), f1 = row_scale(s1);
    for (int m = t; m <= B.NM; m += BT) {
        const int64_t o = (int64_t)jj * B.NU + m;
        const double a1 = f0.x * B.Ac[o], a2 = two ? f1.x * B.Ac[o + B.NU] : 0.0;
        if (m == 0 || 2 * m == N) {
            z[m] = {a1, -a2};
            continue;
        }
        const double b1 = f0.x * B.As[o], b2 = two ? f1.x * B.As[o + B.NU] : 0.0;
        z[m] = {a1 + b2, b1 - a2};
        z[N - m] = {a1 - b2, -a2 - b1};
    }
    __syncthreads();
    const Cx<double>* r = fft(z, z + F.stride, tw, N, F, t, BT, [] { __syncthreads(); });
    double* q = B.R + (int64_t)jj * N;
    const double inv_n = 1.0 / (double)N;
    for (int k = t; k < N; k += BT) {
        q[k] = r[k].re * inv_n * f0.y;
        if (two) q[N + k] = -r[k].im * inv_n * f1.y;
    }
}

// rings beyond one row pair in shared memory: a thread per (row, mode) and per (row, meridian), sums in order
__global__ void baro_forward_sums_kernel(const BaroTables B) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x, jj = blockIdx.y;
    if (m > B.NM) return;
    const double* r = B.R + (int64_t)jj * B.N;
    double sc = 0.0, ss = 0.0, ra = 0.0;
    for (int k = 0, idx = 0; k < B.N; k++) {
        sc += r[k] * B.ct[idx];
        ss += r[k] * B.st[idx];
        ra += fabs(r[k]);
        if ((idx += m) >= B.N) idx -= B.N;
    }
    const double tol = m ? 1.0e-12 * ra : 0.0;
    B.Ac[(int64_t)jj * B.NU + m] = keep(sc, tol);
    B.As[(int64_t)jj * B.NU + m] = keep(ss, tol);
}
__global__ void baro_inverse_sums_kernel(const BaroTables B) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, jj = blockIdx.y;
    if (k >= B.N) return;
    const double *a = B.Ac + (int64_t)jj * B.NU, *b = B.As + (int64_t)jj * B.NU;
    double q = 0.0;
    for (int m = 0, idx = 0; m <= B.NM; m++) {
        const bool real = m == 0 || 2 * m == B.N;
        q += (real ? 1.0 : 2.0) * (a[m] * B.ct[idx] + (real ? 0.0 : b[m] * B.st[idx]));
        if ((idx += k) >= B.N) idx -= B.N;
    }
    B.R[(int64_t)jj * B.N + k] = q / B.N;
}

// the stages for N and the shared memory, 0 where a pair does not fit
size_t plan(int N, FftPlan& F) {
    fft_plan(N, F);
    F.pairs = 1;
    F.lanes = BT;
    const size_t b = fft_smem<double>(F, N);
    return b > 220 * 1024 ? 0 : b;
}

template <class Kernel>
cudaError_t launch_rows(Kernel kernel, const BaroTables& T, const FftPlan& F, size_t smem, cudaStream_t s) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return e;
    kernel<<<(T.J + 1) / 2, BT, smem, s>>>(T, F);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_baro_forward(const BaroTables& T, cudaStream_t s) {
    FftPlan F;
    if (const size_t smem = plan(T.N, F)) return launch_rows(baro_forward_kernel, T, F, smem, s);
    baro_forward_sums_kernel<<<dim3((T.NM + 128) / 128, T.J), 128, 0, s>>>(T);
    return cudaGetLastError();
}

cudaError_t launch_baro_inverse(const BaroTables& T, cudaStream_t s) {
    FftPlan F;
    if (const size_t smem = plan(T.N, F)) return launch_rows(baro_inverse_kernel, T, F, smem, s);
    baro_inverse_sums_kernel<<<dim3((T.N + 127) / 128, T.J), 128, 0, s>>>(T);
    return cudaGetLastError();
}

}  // namespace atsat
