// The spectral solve of poisson.cu: real transforms over phi and the block-tridiagonal solve of each mode.
//
// Spectrum: mode m, polar row jj, radial row ii as the pair (a, b), a the cosine and b the sine sum, at
// ((m NJ + jj) RS + 2 ii): RS = 2 NI rounded up to four, so that a row pair is one vector access.
#pragma once

#include <cstdint>

#include "dyn_common.cuh"

namespace atsat {
namespace spectral {

struct Spec {
    int n, M, NI, NJ;     // ring length km-1, modes n/2+1, radial and polar unknowns
    int RS;               // spectrum values per (mode, polar row)
};

template <typename T> struct Vec2;
template <> struct Vec2<float> { using V = float2; };
template <> struct Vec2<double> { using V = double2; };
template <typename T> struct alignas(4 * sizeof(T)) Quad { T x, y, z, w; };

// ---- transforms over phi ----
// The stages of a mixed-radix transform of length n (Stockham, decimation in frequency: no reordering pass), s the
// product of the radices before the stage and mag = ceil(2^32 / s) for the division by it.
constexpr int FFT_MAX_STAGES = 16;
struct FftPlan {
    int stages, pairs, lanes, stride;    // row pairs per block; threads per pair; complex values per pair and buffer
    int radix[FFT_MAX_STAGES], s[FFT_MAX_STAGES];
    uint32_t mag[FFT_MAX_STAGES];
};

template <typename T>
struct Cx { T re, im; };
template <typename T>
__device__ __forceinline__ Cx<T> operator+(Cx<T> a, Cx<T> b) { return {a.re + b.re, a.im + b.im}; }
template <typename T>
__device__ __forceinline__ Cx<T> operator-(Cx<T> a, Cx<T> b) { return {a.re - b.re, a.im - b.im}; }
// a (c - i s)
template <typename T>
__device__ __forceinline__ Cx<T> turn(Cx<T> a, T c, T s) { return {a.re * c + a.im * s, a.im * c - a.re * s}; }

// b_u = sum_t a_t exp(-2 pi i t u / R), in place
template <typename T, int R>
__device__ __forceinline__ void butterfly(Cx<T>* a) {
    if constexpr (R == 2) {
        const Cx<T> x = a[0], y = a[1];
        a[0] = x + y; a[1] = x - y;
    } else if constexpr (R == 3) {
        const T h = (T)0.86602540378443864676372317075294;      // sin(pi / 3)
        const Cx<T> p = a[1] + a[2], m = a[1] - a[2];
        const Cx<T> c = {a[0].re - (T)0.5 * p.re, a[0].im - (T)0.5 * p.im};
        a[0] = a[0] + p;
        a[1] = {c.re + h * m.im, c.im - h * m.re};
        a[2] = {c.re - h * m.im, c.im + h * m.re};
    } else if constexpr (R == 4) {
        const Cx<T> p = a[0] + a[2], m = a[0] - a[2], q = a[1] + a[3], d = a[1] - a[3];
        a[0] = p + q; a[2] = p - q;
        a[1] = {m.re + d.im, m.im - d.re};
        a[3] = {m.re - d.im, m.im + d.re};
    } else {
        const T c1 = (T)0.30901699437494742410229341718282, s1 = (T)0.95105651629515357211643933337938;   // 2 pi / 5
        const T c2 = (T)-0.80901699437494742410229341718282, s2 = (T)0.58778525229247312916870595463907;  // 4 pi / 5
        const Cx<T> p1 = a[1] + a[4], m1 = a[1] - a[4], p2 = a[2] + a[3], m2 = a[2] - a[3], x = a[0];
        const Cx<T> e = {x.re + c1 * p1.re + c2 * p2.re, x.im + c1 * p1.im + c2 * p2.im};
        const Cx<T> f = {x.re + c2 * p1.re + c1 * p2.re, x.im + c2 * p1.im + c1 * p2.im};
        const Cx<T> g = {s1 * m1.re + s2 * m2.re, s1 * m1.im + s2 * m2.im};
        const Cx<T> h = {s2 * m1.re - s1 * m2.re, s2 * m1.im - s1 * m2.im};
        a[0] = x + p1 + p2;
        a[1] = {e.re + g.im, e.im - g.re};
        a[4] = {e.re - g.im, e.im + g.re};
        a[2] = {f.re + h.im, f.im - h.re};
        a[3] = {f.re - h.im, f.im + h.re};
    }
}

template <typename T, int R>
__device__ __forceinline__ void stage(const Cx<T>* x, Cx<T>* y, const Cx<T>* tw, int n, int s, uint32_t mag, int lane,
                                      int step) {
    const int items = n / R;
    for (int e = lane; e < items; e += step) {
        const int p = s == 1 ? e : (int)__umulhi((uint32_t)e, mag), q = e - p * s;
        Cx<T> a[R];
#pragma unroll
        for (int t = 0; t < R; t++) a[t] = x[e + t * items];         // q + s (p + m t), s m = items
        butterfly<T, R>(a);
        const int o = q + s * R * p, w = p * s;
        y[o] = a[0];
#pragma unroll
        for (int u = 1; u < R; u++) {
            const Cx<T> c = tw[w * u];                               // angle 2 pi p u s / n, below n
            y[o + u * s] = turn(a[u], c.re, c.im);
        }
    }
}

// Any other radix, an odd one: the inputs t and R - t become their sum and difference in place, and a lane forms the
// outputs u and R - u together from the sums' cosine part and the differences' sine part, 2 R operations a pair of
// outputs where R complex products each took 8 R. A ring of one prime R takes R^2 / 2 operations per real row; the direct
// real sums took R^2.
template <typename T, class Sync>
__device__ __forceinline__ void stage_any(Cx<T>* x, Cx<T>* y, const Cx<T>* tw, int n, int R, int s, uint32_t mag,
                                          int lane, int step, Sync sync) {
    const int items = n / R, h = R / 2;
    const int du = step / items, de = step - du * items;
    int u = lane / items, e = lane - u * items;
    for (int w = lane; w < h * items; w += step) {
        Cx<T>*p = x + e + (u + 1) * items, *q = x + e + (R - 1 - u) * items;
        const Cx<T> a = *p, b = *q;
        *p = a + b;
        *q = a - b;
        u += du;
        if ((e += de) >= items) { e -= items; u++; }
    }
    sync();
    u = lane / items;
    e = lane - u * items;
    for (int w = lane; w < (h + 1) * items; w += step) {
        const int p = s == 1 ? e : (int)__umulhi((uint32_t)e, mag), q = e - p * s, turn_by = u * items;
        Cx<T> c = x[e], d = {(T)0, (T)0};
        int idx = 0;
#pragma unroll 4
        for (int t = 1; t <= h; t++) {
            idx += turn_by;                                          // t u (n / R) mod n
            if (idx >= n) idx -= n;
            const Cx<T> f = tw[idx], a = x[e + t * items], b = x[e + (R - t) * items];
            c.re = fma(f.re, a.re, c.re);
            c.im = fma(f.re, a.im, c.im);
            d.re = fma(f.im, b.re, d.re);
            d.im = fma(f.im, b.im, d.im);
        }
        const Cx<T> f = tw[p * s * u];
        Cx<T>* o = y + q + s * R * p;
        o[s * u] = turn(Cx<T>{c.re + d.im, c.im - d.re}, f.re, f.im);
        if (u) {
            const Cx<T> g = tw[p * s * (R - u)];
            o[s * (R - u)] = turn(Cx<T>{c.re - d.im, c.im + d.re}, g.re, g.im);
        }
        u += du;
        if ((e += de) >= items) { e -= items; u++; }
    }
}

// Transforms the complex sequence in `x` with `step` threads (`lane` this one's index; `sync` orders their shared-memory
// accesses); returns the buffer that holds the result in natural order.
template <typename T, class Sync>
__device__ __forceinline__ Cx<T>* fft(Cx<T>* x, Cx<T>* y, const Cx<T>* tw, int n, const FftPlan& F, int lane, int step,
                                      Sync sync) {
    for (int st = 0; st < F.stages; st++) {
        const int R = F.radix[st], s = F.s[st];
        const uint32_t mag = F.mag[st];
        switch (R) {
            case 2: stage<T, 2>(x, y, tw, n, s, mag, lane, step); break;
            case 3: stage<T, 3>(x, y, tw, n, s, mag, lane, step); break;
            case 4: stage<T, 4>(x, y, tw, n, s, mag, lane, step); break;
            case 5: stage<T, 5>(x, y, tw, n, s, mag, lane, step); break;
            default: stage_any<T>(x, y, tw, n, R, s, mag, lane, step, sync); break;
        }
        sync();
        Cx<T>* z = x; x = y; y = z;
    }
    return x;
}
// by a warp, or by a block of LANES threads
template <typename T, int LANES>
__device__ __forceinline__ Cx<T>* fft_lanes(Cx<T>* x, Cx<T>* y, const Cx<T>* tw, int n, const FftPlan& F, int lane) {
    if constexpr (LANES == 32) return fft(x, y, tw, n, F, lane, 32, [] { __syncwarp(); });
    else return fft(x, y, tw, n, F, lane, LANES, [] { __syncthreads(); });
}

template <typename T>
size_t fft_smem(const FftPlan& F, int n) { return ((size_t)F.pairs * 2 * F.stride + n) * sizeof(Cx<T>); }

// Two real rows per complex transform (radial rows 2q and 2q + 1 as real and imaginary part), LANES threads per pair: a
// warp, whose stages in shared memory need no block barrier, or a block (plan_spectral). The direct sums this replaces
// took n (n + 2) multiply-adds per row: 343 us forward and 387 us inverse (FP32) for the 39 x 179 rows of 360 at
// 41x181x361, 104 and 178 us (FP64) at 21x91x181; now 15.8 and 29.2 us (with the FP64 p += e), 24.8 and 25.5 us. The
// FP32 passes' 20 MB take 3 us at the copy rate: the rest is the stages' steps through shared memory; FP64 is bound by
// its pipe. The rounding error is relative to the larger row of a pair. The equation couples the two more strongly than
// any other neighbours, so a row's own rounding reaches the other through the solve at the same size.
template <typename T, int LANES>
__global__ void fft_fwd_kernel(const KConst K, const Spec S, const FftPlan F, const T* __restrict__ x,
                               const T* __restrict__ twt, T* __restrict__ spec) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Cx<T>* tw = reinterpret_cast<Cx<T>*>(dsm);
    Cx<T>* buf = tw + S.n;
    const int lane = threadIdx.x % LANES, pair = threadIdx.x / LANES;
    const int jj = blockIdx.y, pair0 = blockIdx.x * F.pairs, ii = 2 * (pair0 + pair);
    for (int k = threadIdx.x; k < S.n; k += blockDim.x) tw[k] = {twt[k], twt[S.n + k]};
    Cx<T>* a = buf + (size_t)pair * 2 * F.stride;
    const int64_t row = ((int64_t)(ii + 1) * K.jm + jj + 1) * K.kp;
    const bool two = ii + 1 < S.NI;
    if (ii < S.NI)
        for (int k = lane; k < S.n; k += LANES) a[k] = {x[row + k], two ? x[row + K.plane + k] : (T)0};
    __syncthreads();
    if (ii < S.NI) {
        Cx<T>* r = fft_lanes<T, LANES>(a, a + F.stride, tw, S.n, F, lane);
        if (r != a)
            for (int k = lane; k < S.n; k += LANES) a[k] = r[k];
    }
    __syncthreads();
    // split Z into the rows' cosine and sine sums; the pairs of a mode side by side
    const int np = min(F.pairs, (S.NI + 1) / 2 - pair0);
    for (int e = threadIdx.x; e < np * S.M; e += blockDim.x) {
        const int m = e / np, q = e - m * np;
        const Cx<T>* z = buf + (size_t)q * 2 * F.stride;
        const Cx<T> u = z[m], v = z[m ? S.n - m : 0];
        const T h = (T)0.5;
        *reinterpret_cast<Quad<T>*>(spec + ((int64_t)m * S.NJ + jj) * S.RS + 4 * (pair0 + q)) =
            Quad<T>{h * (u.re + v.re), h * (v.im - u.im), h * (u.im + v.im), h * (u.re - v.re)};
    }
}

// The inverse; ADD: add the result to `x` in FP64 (the defect correction's p += e) instead of storing it.
template <typename T, int LANES, typename To, bool ADD>
__global__ void fft_inv_kernel(const KConst K, const Spec S, const FftPlan F, const T* __restrict__ spec,
                               const T* __restrict__ twt, To* __restrict__ x) {
    extern __shared__ __align__(16) unsigned char dsm[];
    Cx<T>* tw = reinterpret_cast<Cx<T>*>(dsm);
    Cx<T>* buf = tw + S.n;
    const int lane = threadIdx.x % LANES, pair = threadIdx.x / LANES;
    const int jj = blockIdx.y, pair0 = blockIdx.x * F.pairs, ii = 2 * (pair0 + pair);
    for (int k = threadIdx.x; k < S.n; k += blockDim.x) tw[k] = {twt[k], twt[S.n + k]};
    const int np = min(F.pairs, (S.NI + 1) / 2 - pair0);
    for (int e = threadIdx.x; e < np * S.M; e += blockDim.x) {
        const int m = e / np, q = e - m * np;
        const Quad<T> v = *reinterpret_cast<const Quad<T>*>(spec + ((int64_t)m * S.NJ + jj) * S.RS + 4 * (pair0 + q));
        Cx<T>* z = buf + (size_t)q * 2 * F.stride;
        // conj(Z), so that the forward transform gives the inverse's conjugate
        if (m == 0 || 2 * m == S.n) {
            z[m] = {v.x, -v.z};                                      // sine sums are zero there
        } else {
            z[m] = {v.x + v.w, v.y - v.z};
            z[S.n - m] = {v.x - v.w, -v.z - v.y};
        }
    }
    __syncthreads();
    if (ii >= S.NI) return;
    Cx<T>* a = buf + (size_t)pair * 2 * F.stride;
    const Cx<T>* r = fft_lanes<T, LANES>(a, a + F.stride, tw, S.n, F, lane);
    const T inv_n = (T)1 / (T)S.n;
    const int64_t row = ((int64_t)(ii + 1) * K.jm + jj + 1) * K.kp;
    const bool two = ii + 1 < S.NI;
    for (int k = lane; k < S.n; k += LANES) {
        const T u = r[k].re * inv_n, v = -r[k].im * inv_n;
        if constexpr (ADD) {
            x[row + k] += f2d(u);
            if (two) x[row + K.plane + k] += f2d(v);
        } else {
            x[row + k] = u;
            if (two) x[row + K.plane + k] = v;
        }
    }
}

// ---- block Thomas per mode ----
// g_j = f_j - b_j (W_{j-1} g_{j-1}); x_NJ = W_NJ g_NJ; x_j = W_j (g_j - c_j x_{j+1}); b, c are the theta couplings. The
// zero mode pins the cell (1, 1) (its row of D_1 is the identity, its c is 0, f = 0) and leaves with the average of its
// solution removed, which is the zero mean of the result over the interior.
//
// One block per mode solves its cosine and sine part together. The recurrence is a chain of 2 NJ - 1 dependent
// matrix-vector products, so what counts is the latency of one step, and with a few warps per SM that is its number of
// instructions. W, f and g are in registers before the vector is ready, loaded DEPTH steps ahead; W is laid out so that
// a thread's share of a product is NC / 2 vector loads without bounds (BtLayout); the vector is read from shared memory
// in 16-byte words; one barrier a step. In FP32 LANES lanes share a dot product, each a contiguous range of columns: the
// defect that a correction leaves oscillates from row to row, so sums over neighbours stay small where sums over every
// LANES-th row grow and cancel only at the end. (With strided lanes the corrections contracted by 0.8 instead of 0.63 at
// 42x9x9, and a solve at 61x61x121 took 16 of them instead of 12.) In FP64 a lane keeps the sequential sum: on this
// ill-conditioned operator another order moves the result by as much as its error.
// At 41x181x361 (181 modes, 357 steps), FP32: 2487 us with W and f read from global memory inside the chain, a mode part
// per block; 248 us with W streamed through a shared-memory ring by bulk copies (waiting for a phase, reading the ring
// and releasing the slot took 550 of a step's 1140 cycles); 235 us with plain column-major W in registers (260 cycles of
// addresses and bounds); 193 us in this layout. DEPTH 8 against 4 (FP32): 2.15 -> 2.02 ms per five-correction solve.
// FP64 at 21x91x181: 480 -> 232 us, 19 dependent operations of ~90 cycles in each of 177 steps.
template <typename T> struct BtShape { static constexpr int LANES = sizeof(T) == 4 ? 4 : 1; };

// W of a (mode, polar row): value u of thread t at (u / 2 * width + t) * 2 + u % 2, zero beyond the matrix.
//   FP32: t = 4 r + q (width: the block's threads), u -> column q nc + u;  FP64: t = r (width: NI), u -> column u
// nc = 0: plain column-major, element (r, c) at c NI + r (the wide kernel).
struct BtLayout {
    int nc, width, threads;
    int64_t stride;                // values per (mode, polar row)
};
template <typename T>
inline BtLayout bt_layout(int NI) {
    constexpr int LANES = BtShape<T>::LANES;
    const int share = (NI + LANES - 1) / LANES;
    BtLayout L{0, NI, ((LANES == 1 ? 2 : LANES) * NI + 31) / 32 * 32, (int64_t)NI * NI};
    if (LANES == 4) L.nc = share <= 6 ? 6 : (share <= 10 ? 10 : (share <= 20 ? 20 : 0));
    else L.nc = share <= 10 ? 10 : (share <= 20 ? 20 : (share <= 40 ? 40 : 0));
    if (L.nc) {
        if (LANES == 4) L.width = L.threads;
        L.stride = (int64_t)L.nc * L.width;
    }
    return L;
}
// place of element (r, c)
template <typename T>
inline int64_t bt_place(const BtLayout& L, int NI, int r, int c) {
    constexpr int LANES = BtShape<T>::LANES;
    if (!L.nc) return (int64_t)c * NI + r;
    const int t = LANES == 4 ? 4 * r + c / L.nc : r, u = LANES == 4 ? c % L.nc : c;
    return ((int64_t)(u / 2) * L.width + t) * 2 + (u & 1);
}

template <typename T, int NC, int DEPTH>
__global__ void bt_solve_kernel(const Spec S, const BtLayout L, const T* __restrict__ W, const double* __restrict__ bvec,
                                const double* __restrict__ cvec, T* __restrict__ spec) {
    using V2 = typename Vec2<T>::V;
    constexpr int LANES = BtShape<T>::LANES;
    // the vector, double buffered: FP32 the pairs (a, b) of the columns in order; FP64 a part after the other. Zero
    // beyond NI.
    constexpr int HALF = LANES == 4 ? 2 * NC : NC;          // values of one lane (FP32) or part (FP64)
    constexpr int NV = LANES == 4 ? 4 * HALF : 2 * HALF;
    __shared__ __align__(16) T gb[2][NV];
    __shared__ double red[32];
    const int NI = S.NI, NJ = S.NJ, m = blockIdx.x, t = threadIdx.x;
    for (int e = t; e < 2 * NV; e += blockDim.x) gb[0][e] = (T)0;
    T* f = spec + (int64_t)m * NJ * S.RS;
    // FP64: thread (part, r); FP32: thread (r, lane q), both parts, lanes 0 and 1 own a part's result
    int r, part, q;
    bool own;
    if (LANES == 1) {
        part = t >= NI ? 1 : 0; r = t - part * NI; q = 0;
        own = r < NI;
    } else {
        r = t / LANES; q = t - r * LANES; part = q & 1;
        own = r < NI && q < 2;
    }
    const int wt = LANES == 4 ? t : (own ? r : 0);          // this thread's W values
    if (r >= NI) r = 0;
    const bool pin = m == 0 && r == 0;
    const int o = 2 * r + part;
    const int place = LANES == 4 ? o : part * HALF + r;
    // the couplings do not depend on j but for the folded end rows
    const T b_mid = (T)bvec[NI + r], b_end = (T)bvec[(NJ - 1) * NI + r];
    const T c_mid = (T)cvec[NI + r], c_0 = pin ? (T)0 : (T)cvec[r];
    V2 wr[DEPTH][NC / 2];
    T pre[DEPTH];
    const int width = L.width, wstep = NC / 2 * width;
    const V2* wp = reinterpret_cast<const V2*>(W) + (int64_t)m * NJ * wstep + wt;   // block row to be loaded next
    auto load_w = [&](V2* w) {
#pragma unroll
        for (int u = 0; u < NC / 2; u++) w[u] = wp[u * width];
    };
    auto product = [&](const V2* w, const T* g) -> T {      // (W g) of this thread's row and part
        if constexpr (LANES == 1) {
            const V2* gp = reinterpret_cast<const V2*>(g + part * HALF);
            V2 gv[NC / 2];
#pragma unroll
            for (int u = 0; u < NC / 2; u++) gv[u] = gp[u];
            T acc = 0;
#pragma unroll
            for (int u = 0; u < NC / 2; u++) {
                acc += w[u].x * gv[u].x;
                acc += w[u].y * gv[u].y;
            }
            return acc;
        } else {
            const Quad<T>* gp = reinterpret_cast<const Quad<T>*>(g + q * HALF);
            T a0 = 0, a1 = 0;
#pragma unroll
            for (int u = 0; u < NC / 2; u++) {
                const Quad<T> v = gp[u];
                a0 += w[u].x * v.x;
                a1 += w[u].x * v.y;
                a0 += w[u].y * v.z;
                a1 += w[u].y * v.w;
            }
#pragma unroll
            for (int d = 1; d < LANES; d <<= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, d);
                a1 += __shfl_xor_sync(0xffffffffu, a1, d);
            }
            return part ? a1 : a0;
        }
    };
    __syncthreads();
    // forward: step jj uses W_{jj-1}
    T* row = f + o;                                         // this thread's value of row jj
    const int rs = S.RS;
#pragma unroll
    for (int u = 0; u < DEPTH; u++) {
        if (u < NJ - 1) { load_w(wr[u]); wp += wstep; }
        pre[u] = (own && 1 + u < NJ) ? row[(1 + u) * rs] : (T)0;
    }
    if (own) {
        const T g = pin ? (T)0 : *row;
        gb[0][place] = g;
        *row = g;
    }
    row += rs;
    __syncthreads();
    for (int j0 = 1; j0 < NJ; j0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; u++) {
            const int jj = j0 + u;
            if (jj >= NJ) break;
            const T acc = product(wr[u], gb[(jj - 1) & 1]);
            const T g = pre[u] - (jj == NJ - 1 ? b_end : b_mid) * acc;
            if (own) {
                gb[jj & 1][place] = g;
                *row = g;                                   // kept for the backward pass
                if (jj + DEPTH < NJ) pre[u] = row[DEPTH * rs];
            }
            if (jj + DEPTH < NJ) { load_w(wr[u]); wp += wstep; }
            row += rs;
            __syncthreads();
        }
    }
    // backward: row jj from W_jj; pre holds g of row jj - 1
    double sum = 0.0;
    row -= rs;
    wp = reinterpret_cast<const V2*>(W) + ((int64_t)m * NJ + NJ - 1) * wstep + wt;
#pragma unroll
    for (int u = 0; u < DEPTH; u++) {
        if (NJ - 1 - u >= 0) { load_w(wr[u]); wp -= wstep; }
        pre[u] = (own && NJ - 2 - u >= 0) ? row[-(1 + u) * rs] : (T)0;
    }
    for (int k0 = 0; k0 < NJ; k0 += DEPTH) {
#pragma unroll
        for (int u = 0; u < DEPTH; u++) {
            const int jj = NJ - 1 - k0 - u;
            if (jj < 0) break;
            const T x = product(wr[u], gb[jj & 1]);
            if (own) {
                *row = x;
                if (m == 0) sum += (double)x;
                if (jj > 0) gb[(jj - 1) & 1][place] = pre[u] - (jj - 1 == 0 ? c_0 : c_mid) * x;
                if (jj - 1 - DEPTH >= 0) pre[u] = row[-(1 + DEPTH) * rs];
            }
            if (jj - DEPTH >= 0) { load_w(wr[u]); wp -= wstep; }
            row -= rs;
            __syncthreads();
        }
    }
    if (m != 0) return;
    if (!own || part != 0) sum = 0.0;
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
    if ((t & 31) == 0) red[t >> 5] = sum;
    __syncthreads();
    double s = 0.0;
    for (unsigned w = 0; w < blockDim.x / 32; w++) s += red[w];
    const T avg = (T)(s / ((double)NI * NJ));
    if (own && part == 0)
        for (int jj = 0; jj < NJ; jj++) f[(int64_t)jj * rs + o] -= avg;
}

// The same solve for radial systems whose rows do not fit the registers: one block per mode and part, the FP64 kernel's
// sums, W from global memory (column-major) in batches of AHEAD columns. A batch is loaded while the one before is summed,
// and a product's first batch and its row of f before the barrier that releases the vector: with single loads the
// chain waited for a load every four columns (the FP64 direct solve at
// 61x61x121, 59 rows: 1266 -> 555 us; FP32 at 90x61x121: 1729 -> 547).
template <typename T, int AHEAD, int THREADS>
__global__ void __launch_bounds__(THREADS) bt_solve_wide_kernel(const Spec S, const T* __restrict__ W,
                                                                const double* __restrict__ bvec,
                                                                const double* __restrict__ cvec, T* __restrict__ spec) {
    const int m = blockIdx.x >> 1, part = blockIdx.x & 1;
    const int NI = S.NI, NJ = S.NJ, r = threadIdx.x;
    extern __shared__ __align__(16) unsigned char dsm[];
    T* g = reinterpret_cast<T*>(dsm);
    T* f = spec + (int64_t)m * NJ * S.RS + part;
    const int64_t ws = (int64_t)NI * NI;
    const bool own = r < NI, pin = m == 0 && r == 0;
    const T* Wr = W + (int64_t)m * NJ * ws + (own ? r : 0);
    T w[AHEAD];                                             // the next product's first batch
    auto load = [&](T* b, const T* wp, int c0) {
#pragma unroll
        for (int u = 0; u < AHEAD; u++) b[u] = c0 + u < NI ? wp[(int64_t)(c0 + u) * NI] : (T)0;
    };
    auto product = [&](int jj) {
        const T* wp = Wr + jj * ws;
        T acc = 0;
        for (int c0 = 0; c0 < NI; c0 += AHEAD) {
            T next[AHEAD];
            if (c0 + AHEAD < NI) load(next, wp, c0 + AHEAD);
#pragma unroll
            for (int u = 0; u < AHEAD; u++)
                if (c0 + u < NI) acc += w[u] * g[c0 + u];
#pragma unroll
            for (int u = 0; u < AHEAD; u++) w[u] = next[u];
        }
        return acc;
    };
    load(w, Wr, 0);
    if (own) f[2 * r] = g[r] = pin ? (T)0 : f[2 * r];
    __syncthreads();
    for (int jj = 1; jj < NJ; jj++) {
        T* row = f + (int64_t)jj * S.RS + 2 * r;
        const T fj = own ? *row : (T)0, b = own ? (T)bvec[jj * NI + r] : (T)0;
        const T acc = product(jj - 1);
        load(w, Wr + jj * ws, 0);
        __syncthreads();
        if (own) *row = g[r] = fj - b * acc;
        __syncthreads();
    }
    double sum = 0.0;
    for (int jj = NJ - 1; jj >= 0; jj--) {
        T* row = f + (int64_t)jj * S.RS + 2 * r;
        const T fj = own && jj > 0 ? row[-S.RS] : (T)0;
        const T cj = own && jj > 0 && !(pin && jj == 1) ? (T)cvec[(jj - 1) * NI + r] : (T)0;
        const T x = product(jj);
        if (jj > 0) load(w, Wr + (jj - 1) * ws, 0);
        __syncthreads();
        if (own) {
            *row = x;
            sum += (double)x;
            if (jj > 0) g[r] = fj - cj * x;
        }
        __syncthreads();
    }
    if (m == 0 && part == 0) {
        __shared__ double red[32];
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
        if ((r & 31) == 0) red[r >> 5] = sum;
        __syncthreads();
        double s = 0.0;
        for (unsigned w_ = 0; w_ < blockDim.x / 32; w_++) s += red[w_];
        const T avg = (T)(s / ((double)NI * NJ));
        if (own)
            for (int jj = 0; jj < NJ; jj++) f[(int64_t)jj * S.RS + 2 * r] -= avg;
    }
}

// ---- host side ----
template <typename T>
cudaError_t launch_bt(const Spec& S, const BtLayout& L, const T* W, const double* bvec, const double* cvec, T* spec,
                      cudaStream_t s) {
    auto go = [&](auto kernel) { kernel<<<S.M, L.threads, 0, s>>>(S, L, W, bvec, cvec, spec); };
    if constexpr (sizeof(T) == 4) {
        if (L.nc == 6) go(bt_solve_kernel<T, 6, 8>);
        else if (L.nc == 10) go(bt_solve_kernel<T, 10, 8>);
        else if (L.nc == 20) go(bt_solve_kernel<T, 20, 4>);
    } else {
        if (L.nc == 10) go(bt_solve_kernel<T, 10, 1>);
        else if (L.nc == 20) go(bt_solve_kernel<T, 20, 1>);
        else if (L.nc == 40) go(bt_solve_kernel<T, 40, 1>);
    }
    if (!L.nc) {                       // the wider batch where the registers of a larger block allow it
        auto wide = [&](auto kernel) {
            kernel<<<2 * S.M, (S.NI + 31) / 32 * 32, (size_t)S.NI * sizeof(T), s>>>(S, W, bvec, cvec, spec);
        };
        if (S.NI <= 256) wide(bt_solve_wide_kernel<T, 16, 256>);
        else wide(bt_solve_wide_kernel<T, 4, 1024>);
    }
    return cudaGetLastError();
}

inline void fft_plan(int n, FftPlan& F) {
    F = FftPlan{};
    int left = n, s = 1;
    auto add = [&](int r) {
        F.radix[F.stages] = r;
        F.s[F.stages] = s;
        F.mag[F.stages] = s > 1 ? (uint32_t)(((1ull << 32) + s - 1) / s) : 0u;
        F.stages++;
        s *= r;
        left /= r;
    };
    // odd radices first: their stores at small strides fall on different banks
    int odd = n;
    while (odd % 2 == 0) odd /= 2;
    for (int r : {5, 3})
        for (; odd % r == 0; odd /= r) add(r);
    for (int r = 7; r * r <= odd; r += 2)
        for (; odd % r == 0; odd /= r) add(r);
    if (odd > 1) add(odd);
    while (left % 4 == 0) add(4);
    if (left % 2 == 0) add(2);
    F.stride = n | 1;
}

}  // namespace spectral
}  // namespace atsat
