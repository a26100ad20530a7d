// FP64 fast Fourier transforms of the PME mesh (hand-written; no library):
// the forward real-to-complex and the inverse complex-to-real 3D transforms of
// an n0 x n1 x n2 mesh (n2 fastest; half spectrum n0 x n1 x (n2 / 2 + 1)),
// each built from 1D passes over lines held in shared memory.
//
// A line of length n = 2^a 3^b (n <= kFftMax) is transformed by the
// self-sorting Stockham algorithm, decimation in frequency: with the stride s
// (the product of the radices so far, initially 1) and the remaining length
// l = n / s, a radix-r stage maps x to y by
//     y[q + s (r p + k)] = w_l^(p k) sum_j x[q + s (p + j l / r)] w_r^(j k),
// p < l / r, q < s, k < r, w_m = exp(-+ 2 pi i / m); the output is in natural
// order.  Sign -1: forward (exp(-2 pi i k x / n)), +1: inverse, unnormalised.
// Radices 8, 4, 2 and 3, so that 64 points take two stages and 128 three (a
// stage costs one pass through shared memory and one barrier); the twiddles
// w_l^(p k) = w_n^(p k s) come from a table of the n roots (fft_twiddles),
// which sincospi per butterfly made the transforms' largest cost.
//
// The lines of a batch are interleaved (element i of line b at x[i * ld + b],
// consecutive threads take consecutive lines), so that the 16-byte shared
// memory accesses of every stage are conflict-free whatever its stride.
//
// The stages are __host__ __device__ functions over a "thread" index range, so
// the host test build runs the same arithmetic.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace gcmc {

constexpr int kFftMax = 256;  // longest line

__host__ __device__ inline bool fft_size_ok(int n) {
    if (n < 1 || n > kFftMax) return false;
    while (n % 2 == 0) n /= 2;
    while (n % 3 == 0) n /= 3;
    return n == 1;
}

// The radix of the stage that leaves the remaining length l: 8 while the power
// of two left is 8 or 32 and more (16 goes as 4 x 4), then 4, 2, 3.
__host__ __device__ inline int fft_radix(int l) {
    if ((l & 7) == 0 && (l & 31) != 16) return 8;
    if ((l & 3) == 0) return 4;
    return (l & 1) == 0 ? 2 : 3;
}

__host__ __device__ inline double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ inline double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ inline double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a times sign i
__host__ __device__ inline double2 cmuli(double2 a, double sign) { return make_double2(-sign * a.y, sign * a.x); }

// The n roots exp(-2 pi i k / n) (host; long double, rounded once).
inline void fft_twiddles(int n, double2* tw) {
    const long double two_pi = 6.283185307179586476925286766559005768L;
    for (int k = 0; k < n; ++k) {
        const long double th = two_pi * k / n;
        tw[k] = make_double2((double)std::cos(th), (double)-std::sin(th));
    }
}

// Division by d of 0 <= t < 2^32 / d with one multiplication (m = ceil(2^32 / d),
// d > 1): the index arithmetic of a butterfly costs as much as its sums with the
// compiler's general division.
struct FastDiv {
    unsigned m, d;
    __host__ __device__ explicit FastDiv(int d_) : m(0xffffffffu / (unsigned)d_ + 1u), d((unsigned)d_) {}
    __host__ __device__ int quot(int t) const {
        if (d == 1u) return t;
#ifdef __CUDA_ARCH__
        return (int)__umulhi((unsigned)t, m);
#else
        return (int)(((unsigned long long)(unsigned)t * m) >> 32);
#endif
    }
};

// v[k] <- sum_j v[j] w_R^(j k)
__host__ __device__ inline void fft_dft2(double2* v) {
    const double2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}
__host__ __device__ inline void fft_dft3(double2* v, double sign) {
    // w3 = -1/2 + sign i sqrt(3)/2
    const double2 cd = cadd(v[1], v[2]), cm = csub(v[1], v[2]);
    const double2 base = make_double2(v[0].x - 0.5 * cd.x, v[0].y - 0.5 * cd.y);
    const double2 rot = cmuli(make_double2(0.86602540378443864676 * cm.x, 0.86602540378443864676 * cm.y), sign);
    v[0] = cadd(v[0], cd);
    v[1] = cadd(base, rot);
    v[2] = csub(base, rot);
}
__host__ __device__ inline void fft_dft4(double2* v, double sign) {
    const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const double2 c = cadd(v[1], v[3]), d = cmuli(csub(v[1], v[3]), sign);
    v[0] = cadd(a, c);
    v[1] = cadd(b, d);
    v[2] = csub(a, c);
    v[3] = csub(b, d);
}
__host__ __device__ inline void fft_dft8(double2* v, double sign) {
    const double h = 0.70710678118654752440;
    double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    fft_dft4(e, sign);
    fft_dft4(o, sign);
    // w8^k, k = 1..3: h (1 + sign i), sign i, h (-1 + sign i)
    o[1] = make_double2(h * (o[1].x - sign * o[1].y), h * (o[1].y + sign * o[1].x));
    o[2] = cmuli(o[2], sign);
    o[3] = make_double2(-h * (o[3].x + sign * o[3].y), h * (sign * o[3].x - o[3].y));
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = cadd(e[k], o[k]);
        v[k + 4] = csub(e[k], o[k]);
    }
}

// One radix-R Stockham stage on nl interleaved lines, work items t in
// [t0, nl * n / R) step dt (t = butterfly * nl + line).
template <int R>
__host__ __device__ inline void fft_stage(const double2* x, double2* y, int ld, int nl, int n, int s,
                                          const double2* tw, int sign, int t0, int dt) {
    const int per = n / R;  // butterflies per line
    const bool last = s * R == n;  // p = 0: no twiddles
    const double sg = (double)sign;
    const FastDiv by_nl(nl), by_s(s);
    for (int t = t0; t < nl * per; t += dt) {
        const int u = by_nl.quot(t), b = t - u * nl;
        const int p = by_s.quot(u), q = u - p * s;
        double2 v[R];
#pragma unroll
        for (int j = 0; j < R; ++j) v[j] = x[(u + j * per) * ld + b];
        if (R == 2) fft_dft2(v);
        if (R == 3) fft_dft3(v, sg);
        if (R == 4) fft_dft4(v, sg);
        if (R == 8) fft_dft8(v, sg);
        double2* out = y + (q + s * R * p) * ld + b;
        out[0] = v[0];
#pragma unroll
        for (int k = 1; k < R; ++k) {
            if (!last) {
                double2 w = tw[k * p * s];
                w.y *= -sg;
                v[k] = cmul(v[k], w);
            }
            out[k * s * ld] = v[k];
        }
    }
}

__host__ __device__ inline void fft_any_stage(int r, const double2* x, double2* y, int ld, int nl, int n, int s,
                                              const double2* tw, int sign, int t0, int dt) {
    if (r == 8) fft_stage<8>(x, y, ld, nl, n, s, tw, sign, t0, dt);
    else if (r == 4) fft_stage<4>(x, y, ld, nl, n, s, tw, sign, t0, dt);
    else if (r == 3) fft_stage<3>(x, y, ld, nl, n, s, tw, sign, t0, dt);
    else fft_stage<2>(x, y, ld, nl, n, s, tw, sign, t0, dt);
}

#ifdef __CUDACC__
// nl interleaved lines of length n in shared memory (x, y: n * ld each; tw the
// n roots), whole CTA; returns the buffer holding the result.
__device__ __forceinline__ double2* fft_lines_block(double2* x, double2* y, int ld, int nl, int n, const double2* tw,
                                                    int sign) {
    for (int s = 1; s < n;) {
        const int r = fft_radix(n / s);
        __syncthreads();
        fft_any_stage(r, x, y, ld, nl, n, s, tw, sign, threadIdx.x, blockDim.x);
        s *= r;
        double2* t = x; x = y; y = t;
    }
    __syncthreads();
    return x;
}
#endif

// Host reference of one line (test build): the transform of x in x.
inline void fft_line_host(double2* x, int n, int sign) {
    double2 y[kFftMax], tw[kFftMax];
    fft_twiddles(n, tw);
    double2 *a = x, *b = y;
    for (int s = 1; s < n;) {
        const int r = fft_radix(n / s);
        fft_any_stage(r, a, b, 1, 1, n, s, tw, sign, 0, 1);
        s *= r;
        double2* t = a; a = b; b = t;
    }
    if (a != x)
        for (int i = 0; i < n; ++i) x[i] = a[i];
}

}  // namespace gcmc
