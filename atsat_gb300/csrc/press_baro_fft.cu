// The transforms over phi of PRESS_BAROTROPIC (PressureSolver.h:606-636, 684-697): the column residual's cosine and sine
// sums per row and mode, and the correction back on the meridians.
//
// Two rows per complex transform, one block each (poisson_spectral.cuh). The reference's sums run over the meridians in
// order, n terms each; the transform's rounding error is smaller than theirs and relative to the row itself, far below
// the residual's own (press_variants.cu). As direct sums, a thread per (row, mode), the two passes took 163 and 159 us
// at 41x181x361 (179 rows of 360), the row sums 32 us; as transforms 13.5 and 11.5 us.
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
    __shared__ double ws[2][BT / 32];
    for (int o = 16; o > 0; o >>= 1) {
        ra0 += __shfl_xor_sync(0xffffffffu, ra0, o);
        ra1 += __shfl_xor_sync(0xffffffffu, ra1, o);
    }
    if ((t & 31) == 0) { ws[0][t >> 5] = ra0; ws[1][t >> 5] = ra1; }
    __syncthreads();
    ra0 = (ws[0][0] + ws[0][1]) + (ws[0][2] + ws[0][3]);
    ra1 = (ws[1][0] + ws[1][1]) + (ws[1][2] + ws[1][3]);
    const Cx<double>* z = fft(a, a + F.stride, tw, N, F, t, BT, [] { __syncthreads(); });
    // modes below 1e-12 of the row's sum |R| are dropped (mode 0 is kept)
    for (int m = t; m <= B.NM; m += BT) {
        const Cx<double> u = z[m], v = z[m ? N - m : 0];
        const double t0 = m ? 1.0e-12 * ra0 : 0.0, t1 = m ? 1.0e-12 * ra1 : 0.0;
        const int64_t o = (int64_t)jj * B.NU + m;
        B.Ac[o] = keep(0.5 * (u.re + v.re), t0);
        B.As[o] = keep(0.5 * (v.im - u.im), t0);
        if (two) {
            B.Ac[o + B.NU] = keep(0.5 * (u.im + v.im), t1);
            B.As[o + B.NU] = keep(0.5 * (u.re - v.re), t1);
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
    for (int m = t; m <= B.NM; m += BT) {
        const int64_t o = (int64_t)jj * B.NU + m;
        const double a1 = B.Ac[o], a2 = two ? B.Ac[o + B.NU] : 0.0;
        if (m == 0 || 2 * m == N) {
            z[m] = {a1, -a2};
            continue;
        }
        const double b1 = B.As[o], b2 = two ? B.As[o + B.NU] : 0.0;
        z[m] = {a1 + b2, b1 - a2};
        z[N - m] = {a1 - b2, -a2 - b1};
    }
    __syncthreads();
    const Cx<double>* r = fft(z, z + F.stride, tw, N, F, t, BT, [] { __syncthreads(); });
    double* q = B.R + (int64_t)jj * N;
    const double inv_n = 1.0 / (double)N;
    for (int k = t; k < N; k += BT) {
        q[k] = r[k].re * inv_n;
        if (two) q[N + k] = -r[k].im * inv_n;
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
    F.warps = 1;                       // one pair per block
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
