// kernels_fft.cuh -- the complex transform of the dipole grid with its
// convolution, for grids whose sizes are products of two small radices.
//
// A line of n = r1 r2 points (Cooley & Tukey 1965; Gentleman & Sande's
// decimation) is transformed in two steps: r2 transforms of r1 points in the
// registers of a thread each, the twiddles, one exchange through shared
// memory, r1 transforms of r2 points.  Five kernels take the grid through
//   z forward (reading the spreading grid, which is cleared on the way),
//   y forward, x forward times the influence function and x backward,
//   y backward, z backward
// where a library transform pair with the scaling between takes seven: the
// passes are short (54^3: 3 us each) and bound by latency, so fewer of them is
// what counts, and the x pass saves two trips of the grid through L2.
// Measured (cold, all passes of one convolution, library then these): FP32
// 24^3 28 -> 18 us (k_fft_planes 13), 54^3 33 -> 24, 108^3 53 -> 44; FP64 72^3
// 46 -> 35.
// Unnormalised both ways, forward exp(-2 pi i jk/n), backward as the forward
// transform of the numbers with their parts exchanged.
#pragma once
#include "kernels.cuh"
#include "kernels_pme.cuh"

namespace amg {

// cos and sin of 2 pi m / n at compile time: the angle reduced to at most an
// eighth of the circle, then the power series
__host__ __device__ constexpr double trig_series(double x, bool sine) {
    double term = sine ? x : 1.0, sum = term;
    for (int k = 1; k < 14; k++) {
        const double a = 2 * k + (sine ? 0 : -1), b = a + 1;
        term *= -x * x / (a * b);
        sum += term;
    }
    return sum;
}
__host__ __device__ constexpr double root_cos(int m, int n) {
    m %= n;
    if (2 * m > n) m = n - m;                              // cos is even
    if (4 * m > n) return -root_cos(n - 2 * m, 2 * n);     // cos(pi - x) = -cos x
    if (8 * m > n) return trig_series(2 * kPi * (n - 4 * m) / (4.0 * n), true);  // sin(pi/2 - x)
    return trig_series(2 * kPi * m / n, false);
}
__host__ __device__ constexpr double root_sin(int m, int n) { return root_cos(4 * m + 3 * n, 4 * n); }  // cos(x - pi/2)

// the n-th roots of unity exp(-2 pi i m / n) as compile-time constants
template <int N>
struct Roots {
    double re[N], im[N];
    constexpr Roots() : re{}, im{} {
        for (int m = 0; m < N; m++) {
            re[m] = root_cos(m, N);
            im[m] = -root_sin(m, N);
        }
    }
};
template <int N>
__device__ constexpr Roots<N> kRoots{};

template <class R>
struct Cx {
    R x, y;
};
template <class R>
__device__ __forceinline__ Cx<R> operator+(Cx<R> a, Cx<R> b) { return {a.x + b.x, a.y + b.y}; }
template <class R>
__device__ __forceinline__ Cx<R> operator-(Cx<R> a, Cx<R> b) { return {a.x - b.x, a.y - b.y}; }
template <class R>
__device__ __forceinline__ Cx<R> operator*(R s, Cx<R> a) { return {s * a.x, s * a.y}; }
template <class R>
__device__ __forceinline__ Cx<R> cmul(Cx<R> a, Cx<R> b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
template <class R>
__device__ __forceinline__ Cx<R> neg_i(Cx<R> a) { return {a.y, -a.x}; }  // -i a

// forward transform of N values in registers, in place, natural order
template <int N>
struct Dft {
    static constexpr int A = N % 4 == 0 && N > 8 ? 4 : N % 3 == 0 ? 3 : N % 2 == 0 ? 2 : 5, B = N / A;
    static_assert(A * B == N && B > 1, "a product of 2, 3, 4 and 5");
    template <class R>
    static __device__ __forceinline__ void run(Cx<R> (&x)[N]) {
        Cx<R> y[B][A];
#pragma unroll
        for (int j = 0; j < B; j++) {
#pragma unroll
            for (int t = 0; t < A; t++) y[j][t] = x[j + B * t];
            Dft<A>::run(y[j]);
#pragma unroll
            for (int k = 1; k < A; k++)
                if (j) y[j][k] = cmul(y[j][k], Cx<R>{(R)kRoots<N>.re[j * k], (R)kRoots<N>.im[j * k]});
        }
#pragma unroll
        for (int k = 0; k < A; k++) {
            Cx<R> z[B];
#pragma unroll
            for (int j = 0; j < B; j++) z[j] = y[j][k];
            Dft<B>::run(z);
#pragma unroll
            for (int m = 0; m < B; m++) x[k + A * m] = z[m];
        }
    }
};
template <>
struct Dft<2> {
    template <class R>
    static __device__ __forceinline__ void run(Cx<R> (&x)[2]) {
        const Cx<R> a = x[0];
        x[0] = a + x[1];
        x[1] = a - x[1];
    }
};
template <>
struct Dft<3> {
    template <class R>
    static __device__ __forceinline__ void run(Cx<R> (&x)[3]) {
        const Cx<R> s = x[1] + x[2], d = neg_i((R)-kRoots<3>.im[1] * (x[1] - x[2]));
        const Cx<R> m = x[0] - R(0.5) * s;
        x[0] = x[0] + s;
        x[1] = m + d;
        x[2] = m - d;
    }
};
template <>
struct Dft<4> {
    template <class R>
    static __device__ __forceinline__ void run(Cx<R> (&x)[4]) {
        const Cx<R> a = x[0] + x[2], b = x[0] - x[2], c = x[1] + x[3], d = neg_i(x[1] - x[3]);
        x[0] = a + c;
        x[1] = b + d;
        x[2] = a - c;
        x[3] = b - d;
    }
};
template <>
struct Dft<5> {
    template <class R>
    static __device__ __forceinline__ void run(Cx<R> (&x)[5]) {
        const R c1 = (R)kRoots<5>.re[1], c2 = (R)kRoots<5>.re[2], s1 = (R)-kRoots<5>.im[1], s2 = (R)-kRoots<5>.im[2];
        const Cx<R> p = x[1] + x[4], q = x[2] + x[3], u = x[1] - x[4], v = x[2] - x[3];
        const Cx<R> a = x[0] + c1 * p + c2 * q, b = x[0] + c2 * p + c1 * q;
        const Cx<R> c = neg_i(s1 * u + s2 * v), d = neg_i(s2 * u - s1 * v);
        x[0] = x[0] + p + q;
        x[1] = a + c;
        x[2] = b + d;
        x[3] = b - d;
        x[4] = a - c;
    }
};

// the radices; BIG: with those above 12, whose registers cost the kernels of
// the others occupancy
#define FFT_RADIX(r, BIG, ...)                                       \
    switch (r) {                                                     \
        case 3: { constexpr int Q = 3; __VA_ARGS__ } break;          \
        case 4: { constexpr int Q = 4; __VA_ARGS__ } break;          \
        case 5: { constexpr int Q = 5; __VA_ARGS__ } break;          \
        case 6: { constexpr int Q = 6; __VA_ARGS__ } break;          \
        case 8: { constexpr int Q = 8; __VA_ARGS__ } break;          \
        case 9: { constexpr int Q = 9; __VA_ARGS__ } break;          \
        case 10: { constexpr int Q = 10; __VA_ARGS__ } break;        \
        case 12: { constexpr int Q = 12; __VA_ARGS__ } break;        \
        case 15:                                                     \
            if constexpr (BIG) { constexpr int Q = 15; __VA_ARGS__ } \
            break;                                                   \
        case 16:                                                     \
            if constexpr (BIG) { constexpr int Q = 16; __VA_ARGS__ } \
            break;                                                   \
        default: break;                                              \
    }

// one axis: n = r1 r2 and the twiddles w^(j k), j < r2, k < r1, w =
// exp(-2 pi i / n), at [k r2 + j]
template <class R>
struct FftAxis {
    int n, r1, r2;
    const Cx<R>* tw;
};

template <class R>
__device__ __forceinline__ Cx<R> exchanged(Cx<R> a, bool yes) { return yes ? Cx<R>{a.y, a.x} : a; }

// Lines along the contiguous axis: blockDim = (max(r1, r2), lines per block).
// `in` and `out` may be the same grid; `clear` (null or `in`) is set to zero.
template <class R, bool BIG>
__global__ void __launch_bounds__(256) k_fft_rows(FftAxis<R> ax, int lines, bool backward, const Cx<R>* in, Cx<R>* out,
                                                  Cx<R>* clear) {
    extern __shared__ __align__(16) unsigned char fft_sm[];
    Cx<R>* sm = reinterpret_cast<Cx<R>*>(fft_sm);
    const int j = threadIdx.x, l = threadIdx.y, line = blockIdx.x * blockDim.y + l;
    const int r1 = ax.r1, r2 = ax.r2, ld = r2 | 1;  // odd row length: no bank conflicts in the second step
    const size_t base = (size_t)line * ax.n;
    if (j < r2 && line < lines) FFT_RADIX(r1, BIG, {
        Cx<R> x[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) x[q] = exchanged(in[base + j + r2 * q], backward);
        if (clear) {
#pragma unroll
            for (int q = 0; q < Q; q++) clear[base + j + r2 * q] = Cx<R>{0, 0};
        }
        Dft<Q>::run(x);
#pragma unroll
        for (int k = 0; k < Q; k++) sm[(l * Q + k) * ld + j] = k ? cmul(x[k], ax.tw[k * r2 + j]) : x[k];
    })
    __syncthreads();
    if (j < r1 && line < lines) FFT_RADIX(r2, BIG, {
        Cx<R> x[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) x[q] = sm[(l * r1 + j) * ld + q];
        Dft<Q>::run(x);
#pragma unroll
        for (int k = 0; k < Q; k++) out[base + j + r1 * k] = exchanged(x[k], backward);
    })
}

// Lines along a strided axis, in place: blockDim = (lines per block,
// max(r1, r2)); blockIdx.y the batch, `inner` lines side by side in each.
// With G (forward only): times the influence function and backward again,
// the backward transform taking the radices in the other order, so that its
// first step starts on the values that the forward's last one left in the
// same registers.
template <class R, bool BIG, bool CONV>
__global__ void __launch_bounds__(256) k_fft_strided(FftAxis<R> ax, size_t stride, int inner, size_t batch,
                                                     bool backward, Cx<R>* g, const R* __restrict__ G) {
    extern __shared__ __align__(16) unsigned char fft_sm[];
    Cx<R>* sm = reinterpret_cast<Cx<R>*>(fft_sm);
    const int t = threadIdx.x, T = blockDim.x, j = threadIdx.y, m = blockIdx.x * T + t;
    const int r1 = ax.r1, r2 = ax.r2;
    const bool ok = m < inner;
    const size_t base = blockIdx.y * batch + m;
    Cx<R>* line = g + base;
    if (j < r2 && ok) FFT_RADIX(r1, BIG, {
        Cx<R> x[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) x[q] = exchanged(line[(j + r2 * q) * stride], backward);
        Dft<Q>::run(x);
#pragma unroll
        for (int k = 0; k < Q; k++) sm[(k * r2 + j) * T + t] = k ? cmul(x[k], ax.tw[k * r2 + j]) : x[k];
    })
    __syncthreads();
    if constexpr (!CONV) {
        if (j < r1 && ok) FFT_RADIX(r2, BIG, {
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = sm[(j * Q + q) * T + t];
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) line[(j + r1 * k) * stride] = exchanged(x[k], backward);
        })
    } else {
        // (every thread of the block takes the same case, so the barrier
        // between the reads and the writes of the exchange is met by all)
        const bool mine = j < r1 && ok;
        FFT_RADIX(r2, BIG, {
            Cx<R> x[Q];
            if (mine) {
                R w[Q];
#pragma unroll
                for (int q = 0; q < Q; q++) w[q] = G[base + (j + r1 * q) * stride];
#pragma unroll
                for (int q = 0; q < Q; q++) x[q] = sm[(j * Q + q) * T + t];
                Dft<Q>::run(x);
#pragma unroll
                for (int k = 0; k < Q; k++) x[k] = exchanged(w[k] * x[k], true);
                Dft<Q>::run(x);
            }
            __syncthreads();
            if (mine) {
#pragma unroll
                for (int k = 0; k < Q; k++) sm[(k * r1 + j) * T + t] = k ? cmul(x[k], ax.tw[j * Q + k]) : x[k];
            }
        })
        __syncthreads();
        if (j < r2 && ok) FFT_RADIX(r1, BIG, {
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = sm[(j * Q + q) * T + t];
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) line[(j + r2 * k) * stride] = exchanged(x[k], true);
        })
    }
}

// Small planes: both contiguous axes in one kernel, a block per plane of K2 x
// K3 points held in shared memory (two buffers: A for the exchanges of either
// axis, B between the axes), so that the grid takes three kernels instead of
// five.  z then y for both directions (the axes commute); the parts are
// exchanged at the first load and the last store.
template <class R>
__host__ __device__ inline size_t fft_plane_words(const FftAxis<R>& z, const FftAxis<R>& y) {
    const size_t a = (size_t)y.n * z.r1 * (z.r2 | 1), p = (size_t)y.n * z.n;
    return (a > p ? a : p) + (size_t)y.n * (z.n | 1);
}

template <class R, bool BIG>
__global__ void __launch_bounds__(512) k_fft_planes(FftAxis<R> az, FftAxis<R> ay, bool backward, const Cx<R>* in,
                                                    Cx<R>* out, Cx<R>* clear) {
    extern __shared__ __align__(16) unsigned char fft_sm[];
    const int K2 = ay.n, K3 = az.n, ldz = az.r2 | 1, ldb = K3 | 1;
    Cx<R>* A = reinterpret_cast<Cx<R>*>(fft_sm);
    Cx<R>* B = A + max(K2 * az.r1 * ldz, K2 * K3);
    const size_t base = (size_t)blockIdx.x * K2 * K3;
    FFT_RADIX(az.r1, BIG, {
        for (int b = threadIdx.x; b < K2 * az.r2; b += blockDim.x) {
            const int l = b / az.r2, j = b - l * az.r2;
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = exchanged(in[base + l * K3 + j + az.r2 * q], backward);
            if (clear) {
#pragma unroll
                for (int q = 0; q < Q; q++) clear[base + l * K3 + j + az.r2 * q] = Cx<R>{0, 0};
            }
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) A[(l * Q + k) * ldz + j] = k ? cmul(x[k], az.tw[k * az.r2 + j]) : x[k];
        }
    })
    __syncthreads();
    FFT_RADIX(az.r2, BIG, {
        for (int b = threadIdx.x; b < K2 * az.r1; b += blockDim.x) {
            const int l = b / az.r1, j = b - l * az.r1;
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = A[b * ldz + q];
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) B[l * ldb + j + az.r1 * k] = x[k];
        }
    })
    __syncthreads();
    FFT_RADIX(ay.r1, BIG, {
        for (int b = threadIdx.x; b < K3 * ay.r2; b += blockDim.x) {
            const int j = b / K3, t = b - j * K3;
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = B[(j + ay.r2 * q) * ldb + t];
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) A[(k * ay.r2 + j) * K3 + t] = k ? cmul(x[k], ay.tw[k * ay.r2 + j]) : x[k];
        }
    })
    __syncthreads();
    FFT_RADIX(ay.r2, BIG, {
        for (int b = threadIdx.x; b < K3 * ay.r1; b += blockDim.x) {
            const int j = b / K3, t = b - j * K3;
            Cx<R> x[Q];
#pragma unroll
            for (int q = 0; q < Q; q++) x[q] = A[(j * Q + q) * K3 + t];
            Dft<Q>::run(x);
#pragma unroll
            for (int k = 0; k < Q; k++) out[base + (j + ay.r1 * k) * K3 + t] = exchanged(x[k], backward);
        }
    })
}

}  // namespace amg
