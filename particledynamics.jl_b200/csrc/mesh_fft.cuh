// Transforms of the mesh engine: real 3D FFTs fused with the influence multiply.
//
// A transform pair of one mesh (charge grid -> potential grid, or the three ik fields) is three
// kernels instead of a library R2C, a multiply and a library C2R (six transform kernels and one
// multiply, two more per ik field):
//   k_plane_forward  one z plane per CTA: real x lines (two rows per complex line), then the y lines, all
//                    in shared memory; the consumed charges are cleared on the way;
//   k_lines_z        z lines forward, times the influence function (FP64 energy and virial sums when asked),
//                    z lines back, the spectrum's values staying in registers across the multiply;
//   k_plane_inverse  y lines, then x lines back to the real grid.
// Planes too large for shared memory go through k_rows_forward / k_lines_y / k_rows_inverse instead of the
// plane kernels (five kernels).
//
// In principle L2-bound (20 bytes per mode and kernel), in fact latency-bound: a 120^3 mesh is 120 planes, one
// CTA each, between whose passes stand barriers.  120^3, warm: planes 11.3 us each way, z lines 7.3 us (the
// library's six kernels and the multiply: 54 us of a launch list with cold caches; with the planes' lines as
// separate kernels the step of 64 000 ions takes 1 % more, of 18 302 ions on 70 x 70 x 112 16 % more).
//
// A line of length n = a b (a, b: 1 to 10, 12, 14, 15 or 16) takes two register passes: DFTs of length a over stride-b
// elements, the twiddles exp(-2 pi i q k / n) from a table computed in FP64, DFTs of length b (the
// Cooley-Tukey decomposition).  Inverse transforms run the forward code on values with real and
// imaginary part exchanged.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "mesh_fft.hpp"

namespace pdb {

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cswap(float2 a) { return make_float2(a.y, a.x); }

// cos and sin of 2 pi k / n at compile time: the angle reduced to [0, pi/4], then the Taylor series
// (eleven terms, below the round-off of FP64 there).
constexpr double fft_series(double x, bool odd) {
    double term = odd ? x : 1.0, sum = term;
    for (int i = odd ? 2 : 1; i < 24; i += 2) {
        term *= -x * x / (i * (i + 1.0));
        sum += term;
    }
    return sum;
}
constexpr double fft_cos(int k, int n) {
    k = ((k % n) + n) % n;
    int e = 8 * k;                        // eighths of the angle, in units of 1 / n of a turn
    if (2 * k > n) return fft_cos(n - k, n);
    if (4 * k > n) return -fft_cos(n - 2 * k, 2 * n);
    if (e > n) return fft_series(2.0 * 3.14159265358979323846 * (n - 4.0 * k) / (4.0 * n), true);
    return fft_series(2.0 * 3.14159265358979323846 * k / n, false);
}
constexpr double fft_sin(int k, int n) { return fft_cos(4 * k - n, 4 * n); }

template <int K, int N>
struct Root {   // exp(-2 pi i K / N)
    static constexpr float c = (float)fft_cos(K, N);
    static constexpr float s = (float)-fft_sin(K, N);
};

// In-register DFT of length R (natural order in and out).
template <int R>
struct Dft;

template <>
struct Dft<1> {
    static __device__ __forceinline__ void run(float2 *) {}
};
template <>
struct Dft<2> {
    static __device__ __forceinline__ void run(float2 *x) {
        const float2 t = x[0];
        x[0] = cadd(t, x[1]);
        x[1] = csub(t, x[1]);
    }
};
template <>
struct Dft<4> {
    static __device__ __forceinline__ void run(float2 *x) {
        const float2 s0 = cadd(x[0], x[2]), d0 = csub(x[0], x[2]), s1 = cadd(x[1], x[3]), d1 = csub(x[1], x[3]);
        x[0] = cadd(s0, s1);
        x[2] = csub(s0, s1);
        x[1] = make_float2(d0.x + d1.y, d0.y - d1.x);   // d0 - i d1
        x[3] = make_float2(d0.x - d1.y, d0.y + d1.x);
    }
};

// Odd prime length: pairs x_k +- x_{R-k} against the real cosine and sine sums.
template <int R, int M, int K>
struct OddTerm {
    static __device__ __forceinline__ void add(const float2 *t, const float2 *d, float2 &re, float2 &im) {
        constexpr float c = Root<M * K, R>::c, s = -Root<M * K, R>::s;
        re = make_float2(fmaf(c, t[K - 1].x, re.x), fmaf(c, t[K - 1].y, re.y));
        im = make_float2(fmaf(s, d[K - 1].y, im.x), fmaf(-s, d[K - 1].x, im.y));   // -i s d
        if constexpr (K < (R - 1) / 2) OddTerm<R, M, K + 1>::add(t, d, re, im);
    }
};
template <int R, int M>
struct OddRow {
    static __device__ __forceinline__ void row(float2 *x, float2 x0, const float2 *t, const float2 *d) {
        float2 re = x0, im = make_float2(0.f, 0.f);
        OddTerm<R, M, 1>::add(t, d, re, im);
        x[M] = cadd(re, im);
        x[R - M] = csub(re, im);
        if constexpr (M < (R - 1) / 2) OddRow<R, M + 1>::row(x, x0, t, d);
    }
};
template <int R>
struct DftOdd {
    static __device__ __forceinline__ void run(float2 *x) {
        constexpr int H = (R - 1) / 2;
        float2 t[H], d[H];
        const float2 x0 = x[0];
        float2 s = x0;
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            t[k - 1] = cadd(x[k], x[R - k]);
            d[k - 1] = csub(x[k], x[R - k]);
            s = cadd(s, t[k - 1]);
        }
        x[0] = s;
        OddRow<R, 1>::row(x, x0, t, d);
    }
};
template <> struct Dft<3> : DftOdd<3> {};
template <> struct Dft<5> : DftOdd<5> {};
template <> struct Dft<7> : DftOdd<7> {};

// Composite length R = A B: DFTs of length A over stride B, twiddles, DFTs of length B.
template <int A, int B, int N2, int K1>
struct CompTwiddle {
    static __device__ __forceinline__ void apply(float2 *y) {   // y[k1] of one n2
        if constexpr (N2 > 0 && K1 > 0) y[K1] = cmul(y[K1], make_float2(Root<N2 * K1, A * B>::c, Root<N2 * K1, A * B>::s));
        if constexpr (K1 + 1 < A) CompTwiddle<A, B, N2, K1 + 1>::apply(y);
    }
};
template <int A, int B, int N2>
struct CompColumn {
    static __device__ __forceinline__ void run(const float2 *x, float2 (*y)[A]) {
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) y[N2][n1] = x[B * n1 + N2];
        Dft<A>::run(y[N2]);
        CompTwiddle<A, B, N2, 0>::apply(y[N2]);
        if constexpr (N2 + 1 < B) CompColumn<A, B, N2 + 1>::run(x, y);
    }
};
template <int A, int B>
struct DftComp {
    static __device__ __forceinline__ void run(float2 *x) {
        float2 y[B][A];
        CompColumn<A, B, 0>::run(x, y);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            float2 z[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
            Dft<B>::run(z);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = z[k2];
        }
    }
};
template <> struct Dft<6> : DftComp<2, 3> {};
template <> struct Dft<8> : DftComp<2, 4> {};
template <> struct Dft<9> : DftComp<3, 3> {};
template <> struct Dft<10> : DftComp<2, 5> {};
template <> struct Dft<12> : DftComp<3, 4> {};
template <> struct Dft<14> : DftComp<2, 7> {};
template <> struct Dft<15> : DftComp<3, 5> {};
template <> struct Dft<16> : DftComp<4, 4> {};

// Calls f with the radix as a compile-time constant (block-uniform).
template <typename F>
__device__ __forceinline__ void with_radix(int r, F &&f) {
    switch (r) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        case 12: f(std::integral_constant<int, 12>{}); break;
        case 14: f(std::integral_constant<int, 14>{}); break;
        case 15: f(std::integral_constant<int, 15>{}); break;
        case 16: f(std::integral_constant<int, 16>{}); break;
        default: break;
    }
}

}  // namespace pdb
