// Transform kernels of the mesh engine and their launchers (mesh_fft.cuh has the layout and the DFTs).
#include <cmath>
#include <vector>

#include "chain.cuh"
#include "common.cuh"
#include "ell_common.cuh"
#include "internal.hpp"
#include "mesh_fft.cuh"

namespace pdb {

// i / d for 0 <= i < 2^18, 1 <= d < 2^10 with inv = 1 / d in FP32: (i + 1/2) / d lies at least 1 / 2d from an
// integer, above the product's rounding error.
__device__ __forceinline__ int fdiv(int i, float inv) { return (int)(((float)i + 0.5f) * inv); }

// First register pass of a line: DFTs of length a over elements j + q b, then second: DFTs of length b over
// the a-pass outputs with twiddles exp(-2 pi i q j / n).  ld(line, j, q) reads and st(line, j, q, v) writes;
// items are (line, j) pairs of `lines` lines, line fastest when LINE_FAST.  INPLACE: the block has a thread for
// every item, and a barrier parts its reads from its writes, so that source and target may be the same buffer.
template <bool TWIDDLE, bool LINE_FAST, bool INPLACE, typename Ld, typename St>
__device__ __forceinline__ void fft_pass(int radix, int per_line, int lines, const float2 *__restrict__ w, Ld &&ld,
                                         St &&st) {
    const int count = per_line * lines;
    const float inv = 1.f / (float)(LINE_FAST ? lines : per_line);
    with_radix(radix, [&](auto R) {
        constexpr int r = decltype(R)::value;
        for (int i = threadIdx.x; INPLACE || i < count; i += blockDim.x) {
            const bool on = !INPLACE || i < count;
            const int hi = fdiv(i, inv), lo = i - hi * (LINE_FAST ? lines : per_line);
            const int line = LINE_FAST ? lo : hi, j = LINE_FAST ? hi : lo;
            float2 x[r];
            if (on) {
#pragma unroll
                for (int q = 0; q < r; ++q) x[q] = ld(line, j, q);
            }
            if (INPLACE) __syncthreads();
            if (on) {
                if (TWIDDLE) {
#pragma unroll
                    for (int q = 1; q < r; ++q) x[q] = cmul(x[q], __ldg(w + q * j));
                }
                Dft<r>::run(x);
#pragma unroll
                for (int q = 0; q < r; ++q) st(line, j, q, x[q]);
            }
            if (INPLACE) break;
        }
    });
}

// The spectra of two real rows from the complex line that carries them as real and imaginary part:
// z1 = Z[m], z2 = Z[n - m].
__device__ __forceinline__ float2 split_row(float2 z1, float2 z2, bool odd) {
    return odd ? make_float2(0.5f * (z1.y + z2.y), 0.5f * (z2.x - z1.x))
               : make_float2(0.5f * (z1.x + z2.x), 0.5f * (z1.y - z2.y));
}

// The complex line of two real rows at element n, from their half spectra at m = min(n, N - n): the rows'
// imaginary parts at m = 0 and N / 2 are not part of a real row's spectrum.
__device__ __forceinline__ float2 join_rows(float2 a, float2 b, bool mirrored, bool real_mode) {
    if (real_mode) return make_float2(a.x, b.x);
    return mirrored ? make_float2(a.x + b.y, b.x - a.y) : make_float2(a.x - b.y, a.y + b.x);
}

// Shared memory of the plane kernels: one buffer where every pass has a thread per item (INPLACE), otherwise
// two.  S0 holds the x lines between their passes (row pitch b | 1, so that
// the second pass's strided loads spread over the banks) and the y lines between theirs; S1 the lines
// between the x and the y transforms.
__host__ __device__ inline int fft_plane_s0(const FftAxis &x, int K2, int K1h) {
    const int xs = ((K2 + 1) / 2) * x.a * (x.b | 1), ys = K2 * K1h;
    return xs > ys ? xs : ys;
}
__host__ __device__ inline int fft_plane_s1(const FftAxis &x, int K2, int K1h) {
    const int xs = ((K2 + 1) / 2) * x.n, ys = K2 * K1h;
    return xs > ys ? xs : ys;
}

// Zero n consecutive grid nodes (16-byte stores where the start and the count allow).
__device__ __forceinline__ void clear_charges(float *p, int n) {
    if ((((size_t)p & 15) | (n & 3)) == 0) {
        float4 *p4 = reinterpret_cast<float4 *>(p);
        for (int i = threadIdx.x; i < (n >> 2); i += blockDim.x) p4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = 0.f;
    }
}

// One z plane: charges -> y-transformed half spectrum, the charges cleared.
template <bool INPLACE>
__device__ __forceinline__ void plane_forward(const FftMesh &m, int z, float2 *S0) {
    const FftAxis X = m.ax[0], Y = m.ax[1];
    const int K1 = X.n, K2 = Y.n, K1h = m.K1h, P = (K2 + 1) >> 1, bp = X.b | 1;
    float2 *S1 = INPLACE ? S0 : S0 + fft_plane_s0(X, K2, K1h);
    float *plane = m.grid + (size_t)z * K2 * K1;
    const int xb = X.b, xa = X.a, ya = Y.a, yb = Y.b;
    fft_pass<false, false, false>(
        xa, xb, P, nullptr,
        [&](int p, int j, int q) {
            const float *r = plane + (size_t)(2 * p) * K1 + j + q * xb;
            return make_float2(r[0], 2 * p + 1 < K2 ? r[K1] : 0.f);
        },
        [&](int p, int j, int q, float2 v) { S0[(p * xa + q) * bp + j] = v; });
    __syncthreads();
    clear_charges(plane, K1 * K2);   // every thread has read its charges
    fft_pass<true, false, INPLACE>(
        xb, xa, P, X.w, [&](int p, int j, int q) { return S0[(p * xa + j) * bp + q]; },
        [&](int p, int j, int q, float2 v) { S1[p * K1 + j + q * xa] = v; });
    __syncthreads();
    fft_pass<false, true, INPLACE>(
        ya, yb, K1h, nullptr,
        [&](int c, int j, int q) {
            const int n = j + q * yb;
            const float2 *line = S1 + (n >> 1) * K1;
            return split_row(line[c], line[c ? K1 - c : 0], n & 1);
        },
        [&](int c, int j, int q, float2 v) { S0[(j * ya + q) * K1h + c] = v; });
    __syncthreads();
    float2 *out = m.spec + (size_t)z * K2 * K1h;
    fft_pass<true, true, false>(
        yb, ya, K1h, Y.w, [&](int c, int j, int q) { return S0[(j + q * ya) * K1h + c]; },
        [&](int c, int j, int q, float2 v) { out[(size_t)(j + q * ya) * K1h + c] = v; });
}

// One z plane back: half spectrum of output f -> real grid.
template <bool INPLACE>
__device__ __forceinline__ void plane_inverse(const FftMesh &m, int z, int f, float2 *S0) {
    const FftAxis X = m.ax[0], Y = m.ax[1];
    const int K1 = X.n, K2 = Y.n, K1h = m.K1h, P = (K2 + 1) >> 1, bp = X.b | 1;
    float2 *S1 = INPLACE ? S0 : S0 + fft_plane_s0(X, K2, K1h);
    const float2 *in = m.zspec[f] + (size_t)z * K2 * K1h;
    float *plane = m.out[f] + (size_t)z * K2 * K1;
    const int xb = X.b, xa = X.a, ya = Y.a, yb = Y.b;
    fft_pass<false, true, false>(
        ya, yb, K1h, nullptr, [&](int c, int j, int q) { return cswap(in[(size_t)(j + q * yb) * K1h + c]); },
        [&](int c, int j, int q, float2 v) { S0[(j * ya + q) * K1h + c] = v; });
    __syncthreads();
    fft_pass<true, true, INPLACE>(
        yb, ya, K1h, Y.w, [&](int c, int j, int q) { return S0[(j + q * ya) * K1h + c]; },
        [&](int c, int j, int q, float2 v) { S1[(j + q * ya) * K1h + c] = cswap(v); });
    __syncthreads();
    fft_pass<false, false, INPLACE>(
        xa, xb, P, nullptr,
        [&](int p, int j, int q) {
            const int n = j + q * xb;
            const bool mir = 2 * n > K1;
            const int c = mir ? K1 - n : n;
            const float2 va = S1[(2 * p) * K1h + c];
            const float2 vb = 2 * p + 1 < K2 ? S1[(2 * p + 1) * K1h + c] : make_float2(0.f, 0.f);
            return cswap(join_rows(va, vb, mir, n == 0 || 2 * n == K1));
        },
        [&](int p, int j, int q, float2 v) { S0[(p * xa + q) * bp + j] = v; });
    __syncthreads();
    fft_pass<true, false, false>(
        xb, xa, P, X.w, [&](int p, int j, int q) { return S0[(p * xa + j) * bp + q]; },
        [&](int p, int j, int q, float2 v) {   // exchanged: the imaginary part is the even row
            float *r = plane + (size_t)(2 * p) * K1 + j + q * xa;
            r[0] = v.y;
            if (2 * p + 1 < K2) r[K1] = v.x;
        });
}

// Up to FFT_LINES_C adjacent lines with element stride `stride` (in float2) through registers and shared
// memory (pitch FFT_LINES_C), one block of FFT_LINES_C x max(a, b) threads.
template <bool INVERSE>
__device__ __forceinline__ void lines_through(const FftAxis &A, const float2 *in, float2 *out, size_t stride, int ncol,
                                              float2 *S) {
    const int c = threadIdx.x & (FFT_LINES_C - 1), j = threadIdx.x / FFT_LINES_C;
    const bool live = c < ncol;
    const int a = A.a, b = A.b;
    with_radix(a, [&](auto R) {
        constexpr int r = decltype(R)::value;
        if (!live || j >= b) return;
        float2 x[r];
#pragma unroll
        for (int q = 0; q < r; ++q) {
            x[q] = in[(size_t)(j + q * b) * stride + c];
            if (INVERSE) x[q] = cswap(x[q]);
        }
        Dft<r>::run(x);
#pragma unroll
        for (int q = 0; q < r; ++q) S[(j * r + q) * FFT_LINES_C + c] = x[q];
    });
    __syncthreads();
    with_radix(b, [&](auto R) {
        constexpr int r = decltype(R)::value;
        if (!live || j >= a) return;
        float2 x[r];
#pragma unroll
        for (int q = 0; q < r; ++q) {
            x[q] = S[(j + q * a) * FFT_LINES_C + c];
            if (q > 0) x[q] = cmul(x[q], __ldg(A.w + q * j));
        }
        Dft<r>::run(x);
#pragma unroll
        for (int q = 0; q < r; ++q) out[(size_t)(j + q * a) * stride + c] = INVERSE ? cswap(x[q]) : x[q];
    });
}

// z lines: forward, times G, back.  The second forward pass leaves a thread the elements j + q a of its line,
// exactly what the first inverse pass (radix b, stride a) takes, so the spectrum is multiplied and turned
// around in registers.  ENERGY adds the FP64 energy and virial sums of _solve_kernel! (MeshKernels.jl:57-81);
// IK writes the three field spectra -i k_d G S (_ik_field_kernel!, MeshKernels.jl:84-102; the Nyquist
// component of the operator is zero), and with ENERGY the potential's as a fourth.
template <bool ENERGY, bool IK>
__device__ __forceinline__ void lines_z(const FftMesh &m, int col0, float2 *S, const float *__restrict__ Vc,
                                        double *__restrict__ acc) {
    const FftAxis A = m.ax[2];
    const int a = A.a, b = A.b, K1h = m.K1h, ncols = m.ax[1].n * K1h;
    const int c = threadIdx.x & (FFT_LINES_C - 1), j = threadIdx.x / FFT_LINES_C;
    const int col = col0 + c;
    const bool live = col < ncols;
    const size_t stride = (size_t)ncols;
    with_radix(a, [&](auto R) {
        constexpr int r = decltype(R)::value;
        if (!live || j >= b) return;
        float2 x[r];
        const float2 *in = m.spec + col;
#pragma unroll
        for (int q = 0; q < r; ++q) x[q] = in[(size_t)(j + q * b) * stride];
        Dft<r>::run(x);
#pragma unroll
        for (int q = 0; q < r; ++q) S[(j * r + q) * FFT_LINES_C + c] = x[q];
    });
    __syncthreads();
    constexpr int NOUT = IK ? (ENERGY ? 4 : 3) : 1;
    double e = 0, v[6] = {0, 0, 0, 0, 0, 0};
    float2 *T = S + A.n * FFT_LINES_C;   // IK: the multiplied spectrum, kept for the fields
    float kx = 0.f, ky = 0.f;
    if (IK) {
        const int m1 = col % K1h, m2 = col / K1h, K1 = m.ax[0].n, K2 = m.ax[1].n;
        kx = 2 * m1 == K1 ? 0.f : m.kd[0] * (float)m1;
        ky = 2 * m2 == K2 ? 0.f : m.kd[1] * (float)(2 * m2 < K2 ? m2 : m2 - K2);
    }
    // The forward transform's end, the multiply, and (one output) the inverse transform's start.
    with_radix(b, [&](auto R) {
        constexpr int r = decltype(R)::value;
        float2 x[r];
        if (live && j < a) {
            float g[r];
#pragma unroll
            for (int q = 0; q < r; ++q) g[q] = __ldg(m.G + (size_t)(j + q * a) * stride + col);
#pragma unroll
            for (int q = 0; q < r; ++q) {
                x[q] = S[(j + q * a) * FFT_LINES_C + c];
                if (q > 0) x[q] = cmul(x[q], __ldg(A.w + q * j));
            }
            Dft<r>::run(x);
            if (ENERGY) {
                const int m1 = col % K1h;
                const double wgt = (m1 == 0 || 2 * m1 == m.ax[0].n) ? 0.5 : 1.0;
                const size_t nmodes = stride * A.n;
#pragma unroll
                for (int q = 0; q < r; ++q) {
                    const size_t idx = (size_t)(j + q * a) * stride + col;
                    const double s2 = wgt * ((double)x[q].x * x[q].x + (double)x[q].y * x[q].y);
                    e += s2 * (double)g[q];
#pragma unroll
                    for (int k = 0; k < 6; ++k) v[k] += s2 * (double)__ldg(Vc + k * nmodes + idx);
                }
            }
#pragma unroll
            for (int q = 0; q < r; ++q) x[q] = make_float2(x[q].x * g[q], x[q].y * g[q]);
            if (IK) {
#pragma unroll
                for (int q = 0; q < r; ++q) T[(j + q * a) * FFT_LINES_C + c] = x[q];   // read back by this thread
            } else {
#pragma unroll
                for (int q = 0; q < r; ++q) x[q] = cswap(x[q]);
                Dft<r>::run(x);
            }
        }
        __syncthreads();   // every thread holds its values of the exchange
        if (!IK && live && j < a) {
#pragma unroll
            for (int q = 0; q < r; ++q) S[(j * r + q) * FFT_LINES_C + c] = x[q];
        }
    });
#pragma unroll 1
    for (int f = 0; f < NOUT; ++f) {
        if (IK) {
            int jf = j;
            asm volatile("" : "+r"(jf));   // keeps the mode numbers of every radix from being hoisted out of the loop
            with_radix(b, [&](auto R) {
                constexpr int r = decltype(R)::value;
                if (!live || jf >= a) return;
                float2 x[r];
#pragma unroll
                for (int q = 0; q < r; ++q) {
                    const int m3 = jf + q * a;
                    const float2 t = T[m3 * FFT_LINES_C + c];
                    float k = f == 0 ? kx : ky;
                    if (f == 2) k = 2 * m3 == A.n ? 0.f : m.kd[2] * (float)(2 * m3 < A.n ? m3 : m3 - A.n);
                    x[q] = f == 3 ? cswap(t) : make_float2(-t.x * k, t.y * k);   // -i k t, exchanged
                }
                Dft<r>::run(x);
#pragma unroll
                for (int q = 0; q < r; ++q) S[(jf * r + q) * FFT_LINES_C + c] = x[q];
            });
        }
        __syncthreads();
        int ji = j;
        asm volatile("" : "+r"(ji));
        with_radix(a, [&](auto R) {
            constexpr int r = decltype(R)::value;
            if (!live || ji >= b) return;
            float2 x[r];
#pragma unroll
            for (int q = 0; q < r; ++q) {
                x[q] = S[(ji + q * b) * FFT_LINES_C + c];
                if (q > 0) x[q] = cmul(x[q], __ldg(A.w + q * ji));
            }
            Dft<r>::run(x);
            float2 *out = m.zspec[f] + col;
#pragma unroll
            for (int q = 0; q < r; ++q) out[(size_t)(ji + q * b) * stride] = cswap(x[q]);
        });
        if (IK) __syncthreads();   // the lines' values are in registers before the next field's exchange
    }
    if (ENERGY) {
        __shared__ double sh[7][FFT_RADIX_MAX * FFT_LINES_C / 32];
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
        double vals[7] = {e, v[0], v[1], v[2], v[3], v[4], v[5]};
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const double s = warp_sum_d(vals[k]);
            if (lane == 0) sh[k][w] = s;
        }
        __syncthreads();
        if (threadIdx.x < 7) {
            double s = 0.0;
            for (int k = 0; k < nw; ++k) s += sh[threadIdx.x][k];
            if (s != 0.0) red_add_d(&acc[threadIdx.x], s);
        }
    }
}

// ------------------------------------------------------------------ kernels: one mesh

// Planes come in three CTA sizes (up to 256, 512 or FFT_PLANE_THREADS threads): the registers are capped so that
// four, two or one of them share an SM, as a plane alone leaves most of an SM waiting on its own barriers (12 melts of
// 2050 to 16 282 ions, 5 steps: 926 us with one size, 814 with three).
constexpr int fft_plane_blocks(int maxt) { return maxt <= 256 ? 4 : maxt <= 512 ? 2 : 1; }

template <bool INPLACE, int MAXT>
__global__ void __launch_bounds__(MAXT, fft_plane_blocks(MAXT)) k_plane_forward(const __grid_constant__ FftMesh m) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    plane_forward<INPLACE>(m, blockIdx.x, fft_smem);
}
template <bool INPLACE, int MAXT>
__global__ void __launch_bounds__(MAXT, fft_plane_blocks(MAXT)) k_plane_inverse(const __grid_constant__ FftMesh m) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    plane_inverse<INPLACE>(m, blockIdx.x, blockIdx.y, fft_smem);
}
template <bool ENERGY, bool IK>
__global__ void __launch_bounds__(FFT_RADIX_MAX *FFT_LINES_C) k_lines_z(const __grid_constant__ FftMesh m,
                                                                       const float *__restrict__ Vc,
                                                                       double *__restrict__ acc) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    lines_z<ENERGY, IK>(m, blockIdx.x * FFT_LINES_C, fft_smem, Vc, acc);
}

// Rows of planes that exceed shared memory: FFT_ROW_PAIRS pairs of adjacent rows per CTA.
constexpr int FFT_ROW_PAIRS = 8;

__global__ void __launch_bounds__(FFT_RADIX_MAX *FFT_ROW_PAIRS) k_rows_forward(const __grid_constant__ FftMesh m) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    const FftAxis X = m.ax[0];
    const int K1 = X.n, K2 = m.ax[1].n, K1h = m.K1h, P = (K2 + 1) >> 1, bp = X.b | 1, xa = X.a, xb = X.b;
    const int g0 = blockIdx.x * FFT_ROW_PAIRS, lines = min(FFT_ROW_PAIRS, P * m.ax[2].n - g0);
    float2 *S0 = fft_smem, *S1 = fft_smem + FFT_ROW_PAIRS * xa * bp;
    fft_pass<false, false, false>(
        xa, xb, lines, nullptr,
        [&](int l, int j, int q) {
            const int g = g0 + l, z = g / P, p = g - z * P;
            const float *r = m.grid + ((size_t)z * K2 + 2 * p) * K1 + j + q * xb;
            return make_float2(r[0], 2 * p + 1 < K2 ? r[K1] : 0.f);
        },
        [&](int l, int j, int q, float2 v) { S0[(l * xa + q) * bp + j] = v; });
    __syncthreads();
    fft_pass<true, false, false>(
        xb, xa, lines, X.w, [&](int l, int j, int q) { return S0[(l * xa + j) * bp + q]; },
        [&](int l, int j, int q, float2 v) { S1[l * K1 + j + q * xa] = v; });
    __syncthreads();
    for (int l = 0; l < lines; ++l) {
        const int g = g0 + l, z = g / P, p = g - z * P;
        clear_charges(m.grid + ((size_t)z * K2 + 2 * p) * K1, 2 * p + 1 < K2 ? 2 * K1 : K1);
        float2 *o = m.spec + ((size_t)z * K2 + 2 * p) * K1h;
        for (int c = threadIdx.x; c < K1h; c += blockDim.x) {
            const float2 z1 = S1[l * K1 + c], z2 = S1[l * K1 + (c ? K1 - c : 0)];
            o[c] = split_row(z1, z2, false);
            if (2 * p + 1 < K2) o[K1h + c] = split_row(z1, z2, true);
        }
    }
}

__global__ void __launch_bounds__(FFT_RADIX_MAX *FFT_ROW_PAIRS) k_rows_inverse(const __grid_constant__ FftMesh m) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    const FftAxis X = m.ax[0];
    const int K1 = X.n, K2 = m.ax[1].n, K1h = m.K1h, P = (K2 + 1) >> 1, bp = X.b | 1, xa = X.a, xb = X.b;
    const int f = blockIdx.y, g0 = blockIdx.x * FFT_ROW_PAIRS, lines = min(FFT_ROW_PAIRS, P * m.ax[2].n - g0);
    float2 *S0 = fft_smem, *S1 = fft_smem + FFT_ROW_PAIRS * xa * bp;
    for (int l = 0; l < lines; ++l) {
        const int g = g0 + l, z = g / P, p = g - z * P;
        const float2 *in = m.zspec[f] + ((size_t)z * K2 + 2 * p) * K1h;
        for (int c = threadIdx.x; c < K1h; c += blockDim.x) {
            S1[(2 * l) * K1h + c] = in[c];
            S1[(2 * l + 1) * K1h + c] = 2 * p + 1 < K2 ? in[K1h + c] : make_float2(0.f, 0.f);
        }
    }
    __syncthreads();
    fft_pass<false, false, false>(
        xa, xb, lines, nullptr,
        [&](int l, int j, int q) {
            const int n = j + q * xb;
            const bool mir = 2 * n > K1;
            const int c = mir ? K1 - n : n;
            return cswap(join_rows(S1[(2 * l) * K1h + c], S1[(2 * l + 1) * K1h + c], mir, n == 0 || 2 * n == K1));
        },
        [&](int l, int j, int q, float2 v) { S0[(l * xa + q) * bp + j] = v; });
    __syncthreads();
    fft_pass<true, false, false>(
        xb, xa, lines, X.w, [&](int l, int j, int q) { return S0[(l * xa + j) * bp + q]; },
        [&](int l, int j, int q, float2 v) {
            const int g = g0 + l, z = g / P, p = g - z * P;
            float *r = m.out[f] + ((size_t)z * K2 + 2 * p) * K1 + j + q * xa;
            r[0] = v.y;
            if (2 * p + 1 < K2) r[K1] = v.x;
        });
}

// y lines of one z plane, in place.
template <bool INVERSE>
__global__ void __launch_bounds__(FFT_RADIX_MAX *FFT_LINES_C) k_lines_y(const __grid_constant__ FftMesh m) {
    chain_begin();
    extern __shared__ float2 fft_smem[];
    const int K1h = m.K1h, c0 = blockIdx.x * FFT_LINES_C;
    float2 *base = (INVERSE ? m.zspec[blockIdx.z] : m.spec) + (size_t)blockIdx.y * m.ax[1].n * K1h + c0;
    lines_through<INVERSE>(m.ax[1], base, base, (size_t)K1h, min(FFT_LINES_C, K1h - c0), fft_smem);
}

// ------------------------------------------------------------------ kernels: batched meshes

// blocks[i] = (mesh, plane or first column); every kernel returns while the rows are invalid, as the other
// stages of the batched step do.
template <bool INPLACE, int MAXT>
__global__ void __launch_bounds__(MAXT, fft_plane_blocks(MAXT)) k_bplane_forward(const FftMesh *__restrict__ tab,
                                                                     const int2 *__restrict__ blocks,
                                                                     const long long *__restrict__ st) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    extern __shared__ float2 fft_smem[];
    __shared__ FftMesh m;
    const int2 w = blocks[blockIdx.x];
    if (threadIdx.x == 0) m = tab[w.x];
    __syncthreads();
    plane_forward<INPLACE>(m, w.y, fft_smem);
}
template <bool INPLACE, int MAXT>
__global__ void __launch_bounds__(MAXT, fft_plane_blocks(MAXT)) k_bplane_inverse(const FftMesh *__restrict__ tab,
                                                                     const int2 *__restrict__ blocks,
                                                                     const long long *__restrict__ st) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    extern __shared__ float2 fft_smem[];
    __shared__ FftMesh m;
    const int2 w = blocks[blockIdx.x];
    if (threadIdx.x == 0) m = tab[w.x];
    __syncthreads();
    plane_inverse<INPLACE>(m, w.y, 0, fft_smem);
}
__global__ void __launch_bounds__(FFT_RADIX_MAX *FFT_LINES_C) k_blines_z(const FftMesh *__restrict__ tab,
                                                                        const int2 *__restrict__ blocks,
                                                                        const long long *__restrict__ st) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    extern __shared__ float2 fft_smem[];
    __shared__ FftMesh m;
    const int2 w = blocks[blockIdx.x];
    if (threadIdx.x == 0) m = tab[w.x];
    __syncthreads();
    lines_z<false, false>(m, w.y, fft_smem, nullptr, nullptr);
}

// ------------------------------------------------------------------ host side

static bool fft_factor(int n, int *a, int *b) {
    auto ok = [](int r) { return r >= 1 && r <= FFT_RADIX_MAX && r != 11 && r != 13; };
    for (int d = (int)std::sqrt((double)n) + 1; d >= 1; --d)   // the most balanced pair
        if (n % d == 0 && d * d <= n && ok(d) && ok(n / d)) {
            *a = d;
            *b = n / d;
            return true;
        }
    return false;
}

// Items of a plane's largest pass.
static int fft_plane_items(const FftMesh &m) {
    const FftAxis &X = m.ax[0], &Y = m.ax[1];
    return std::max((Y.n + 1) / 2 * std::max(X.a, X.b), m.K1h * std::max(Y.a, Y.b));
}
bool fft_plane_inplace(const FftMesh &m) { return fft_plane_items(m) <= FFT_PLANE_THREADS; }

size_t fft_plane_smem(const FftMesh &m, bool inplace) {
    const size_t s0 = fft_plane_s0(m.ax[0], m.ax[1].n, m.K1h), s1 = fft_plane_s1(m.ax[0], m.ax[1].n, m.K1h);
    return sizeof(float2) * (inplace ? std::max(s0, s1) : s0 + s1);
}

int fft_route(const int K[3], FftMesh *m) {
    for (int d = 0; d < 3; ++d) {
        m->ax[d].n = K[d];
        m->ax[d].w = nullptr;
        if (!fft_factor(K[d], &m->ax[d].a, &m->ax[d].b)) return FFT_CUFFT;
    }
    m->K1h = K[0] / 2 + 1;
    return fft_plane_smem(*m, fft_plane_inplace(*m)) <= FFT_PLANE_SMEM_MAX ? FFT_PLANES : FFT_LINES;
}

int fft_twiddles(int n, float2 **out) {
    std::vector<float2> w((size_t)n);
    for (int k = 0; k < n; ++k) {
        const double t = 2.0 * M_PI * k / n;
        w[(size_t)k] = make_float2((float)std::cos(t), (float)-std::sin(t));
    }
    int rc = dalloc(out, (size_t)n);
    if (rc) return rc;
    PD_CUDA(cudaMemcpy(*out, w.data(), sizeof(float2) * (size_t)n, cudaMemcpyHostToDevice));
    return PD_OK;
}

// Threads of a plane CTA: its largest pass in as few rounds as the limit allows.
int fft_plane_threads(const FftMesh &m) {
    const int items = fft_plane_items(m), rounds = (items + FFT_PLANE_THREADS - 1) / FFT_PLANE_THREADS;
    return std::min(FFT_PLANE_THREADS, ((items + rounds - 1) / rounds + 31) / 32 * 32);
}

int fft_plane_class(const FftMesh &m) {
    const int nt = fft_plane_threads(m);
    return !fft_plane_inplace(m) ? 3 : nt <= 256 ? 0 : nt <= 512 ? 1 : 2;
}

// Whole warps: the energy sums shuffle across all 32 lanes (a factor of 9 alone would give four and a half warps).
int fft_line_threads(const FftAxis &a) { return (FFT_LINES_C * std::max(a.a, a.b) + 31) / 32 * 32; }
size_t fft_line_smem(const FftAxis &a) { return sizeof(float2) * (size_t)a.n * FFT_LINES_C; }

int fft_init() {
    const int most = (int)FFT_PLANE_SMEM_MAX;
#define PD_PLANE_SIZES(K) (const void *)K<true, 256>, (const void *)K<true, 512>, (const void *)K<true, FFT_PLANE_THREADS>, \
                          (const void *)K<false, FFT_PLANE_THREADS>
    const void *fns[] = {PD_PLANE_SIZES(k_plane_forward), PD_PLANE_SIZES(k_plane_inverse),
                         PD_PLANE_SIZES(k_bplane_forward), PD_PLANE_SIZES(k_bplane_inverse)};
#undef PD_PLANE_SIZES
    for (const void *f : fns) PD_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    const int line = 2 * FFT_RADIX_MAX * FFT_RADIX_MAX * FFT_LINES_C * (int)sizeof(float2);   // two exchanges (ik)
    PD_CUDA(cudaFuncSetAttribute((const void *)k_lines_z<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, line));
    PD_CUDA(cudaFuncSetAttribute((const void *)k_lines_z<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, line));
    return PD_OK;
}

static size_t fft_rows_smem(const FftMesh &m) {
    const FftAxis &X = m.ax[0];
    return sizeof(float2) * FFT_ROW_PAIRS * ((size_t)X.a * (X.b | 1) + std::max(X.n, 2 * m.K1h));
}

#define PD_UNPAREN(...) __VA_ARGS__
// A plane kernel in the CTA size of nt threads (two buffers: always the largest).
#define PD_PLANE_LAUNCH(K, inplace, nt, grid, shm, s, args)                                \
    do {                                                                                   \
        if (!(inplace)) launch_chained(K<false, FFT_PLANE_THREADS>, grid, nt, shm, s, PD_UNPAREN args);            \
        else if ((nt) <= 256) launch_chained(K<true, 256>, grid, nt, shm, s, PD_UNPAREN args);                     \
        else if ((nt) <= 512) launch_chained(K<true, 512>, grid, nt, shm, s, PD_UNPAREN args);                     \
        else launch_chained(K<true, FFT_PLANE_THREADS>, grid, nt, shm, s, PD_UNPAREN args);                        \
    } while (0)

int fft_forward(const FftMesh &m, int route, cudaStream_t s) {
    if (route == FFT_PLANES) {
        const bool in = fft_plane_inplace(m);
        const int nt = fft_plane_threads(m);
        const size_t shm = fft_plane_smem(m, in);
        const dim3 g(m.ax[2].n);
        PD_PLANE_LAUNCH(k_plane_forward, in, nt, g, shm, s, (m));
        PD_LAUNCHED();
        return PD_OK;
    }
    const int pairs = (m.ax[1].n + 1) / 2 * m.ax[2].n;
    launch_chained(k_rows_forward, (pairs + FFT_ROW_PAIRS - 1) / FFT_ROW_PAIRS, FFT_RADIX_MAX * FFT_ROW_PAIRS, fft_rows_smem(m), s, m);
    PD_LAUNCHED();
    const dim3 g((m.K1h + FFT_LINES_C - 1) / FFT_LINES_C, m.ax[2].n);
    launch_chained(k_lines_y<false>, g, fft_line_threads(m.ax[1]), fft_line_smem(m.ax[1]), s, m);
    PD_LAUNCHED();
    return PD_OK;
}

int fft_solve(const FftMesh &m, bool ik, bool energy, const float *Vc, double *acc, cudaStream_t s) {
    const int blocks = (m.ax[1].n * m.K1h + FFT_LINES_C - 1) / FFT_LINES_C;
    const int threads = fft_line_threads(m.ax[2]);
    const size_t shm = fft_line_smem(m.ax[2]) * (ik ? 2 : 1);
    if (ik) {
        if (energy) launch_chained(k_lines_z<true, true>, blocks, threads, shm, s, m, Vc, acc);
        else launch_chained(k_lines_z<false, true>, blocks, threads, shm, s, m, Vc, acc);
    } else {
        if (energy) launch_chained(k_lines_z<true, false>, blocks, threads, shm, s, m, Vc, acc);
        else launch_chained(k_lines_z<false, false>, blocks, threads, shm, s, m, Vc, acc);
    }
    PD_LAUNCHED();
    return PD_OK;
}

int fft_inverse(const FftMesh &m, int route, int nout, cudaStream_t s) {
    if (route == FFT_PLANES) {
        const bool in = fft_plane_inplace(m);
        const int nt = fft_plane_threads(m);
        const size_t shm = fft_plane_smem(m, in);
        const dim3 g(m.ax[2].n, nout);
        PD_PLANE_LAUNCH(k_plane_inverse, in, nt, g, shm, s, (m));
        PD_LAUNCHED();
        return PD_OK;
    }
    const dim3 g((m.K1h + FFT_LINES_C - 1) / FFT_LINES_C, m.ax[2].n, nout);
    launch_chained(k_lines_y<true>, g, fft_line_threads(m.ax[1]), fft_line_smem(m.ax[1]), s, m);
    PD_LAUNCHED();
    const int pairs = (m.ax[1].n + 1) / 2 * m.ax[2].n;
    launch_chained(k_rows_inverse, dim3((pairs + FFT_ROW_PAIRS - 1) / FFT_ROW_PAIRS, nout), FFT_RADIX_MAX * FFT_ROW_PAIRS, fft_rows_smem(m), s, m);
    PD_LAUNCHED();
    return PD_OK;
}

int fft_batch(const FftBatch &f, const long long *st, cudaStream_t s) {
    for (int c = 0; c < f.nclass; ++c) {
        const FftBatch::Class &k = f.cls[c];
        PD_PLANE_LAUNCH(k_bplane_forward, k.inplace, k.threads, k.count, k.smem, s, (f.tab, f.planes + k.first, st));
        PD_LAUNCHED();
    }
    launch_chained(k_blines_z, f.ncols, f.line_threads, f.line_smem, s, f.tab, f.cols, st);
    PD_LAUNCHED();
    for (int c = 0; c < f.nclass; ++c) {
        const FftBatch::Class &k = f.cls[c];
        PD_PLANE_LAUNCH(k_bplane_inverse, k.inplace, k.threads, k.count, k.smem, s, (f.tab, f.planes + k.first, st));
        PD_LAUNCHED();
    }
    return PD_OK;
}

}  // namespace pdb
