// Transforms of the mesh engine: what their callers see (mesh_fft.cu has the kernels, mesh_fft.cuh the DFTs).
#pragma once

#include <cuda_runtime.h>

namespace pdb {

constexpr int FFT_RADIX_MAX = 16;
constexpr int FFT_LINES_C = 16;          // adjacent lines per CTA of the line kernels
constexpr int FFT_PLANE_THREADS = 768;
constexpr size_t FFT_PLANE_SMEM_MAX = 220 * 1024;

// How a mesh is transformed: cuFFT (an axis is no product of two lengths of 1 to 10, 12, 14, 15 or 16: those with a
// factor 11 or 13, 125, 147, 162, 175, 189, 200, 216, 243, 245, 250, 252 and most above 256), whole z planes in shared
// memory, or separate x and y lines.
enum { FFT_CUFFT = 0, FFT_PLANES = 1, FFT_LINES = 2 };

// One axis: n = a b, w[k] = exp(-2 pi i k / n).
struct FftAxis {
    int n, a, b;
    const float2 *w;
};

// One mesh: the real charge grid (K3 x K2 x K1), the half spectrum (K3 x K2 x K1h), the outputs.
struct FftMesh {
    FftAxis ax[3];
    int K1h;
    float *grid;        // charges, cleared by the forward transform
    float2 *spec;       // half spectrum
    const float *G;     // influence function
    float2 *zspec[4];   // spectra after the multiply: [0] potential (may be spec), ik: [0..2] fields, [3] potential
    float *out[4];      // real outputs of the same order
    float kd[3];        // ik: 2 pi / L per axis
};

// Batched meshes: a table of meshes and the (mesh, plane) and (mesh, first column) of every CTA; the planes
// by CTA size (one launch each way per class).
struct FftBatch {
    struct Class {
        int first, count, threads;
        size_t smem;
        bool inplace;
    };
    const FftMesh *tab;
    const int2 *planes, *cols;
    int ncols, line_threads;
    size_t line_smem;
    int nclass;
    Class cls[4];   // up to 256, 512 and FFT_PLANE_THREADS threads in place, then two buffers
};
int fft_plane_class(const FftMesh &m);

// Route of a mesh; fills the axes' factors (twiddle tables stay null).
int fft_route(const int K[3], FftMesh *m);
// Device table of exp(-2 pi i k / n), k < n.
int fft_twiddles(int n, float2 **out);
int fft_init();
bool fft_plane_inplace(const FftMesh &m);
size_t fft_plane_smem(const FftMesh &m, bool inplace);
int fft_plane_threads(const FftMesh &m);
int fft_line_threads(const FftAxis &a);
size_t fft_line_smem(const FftAxis &a);
// grid -> spec without the z transform (the grid is cleared); spec -> zspec (z forward, multiply, z back);
// zspec -> out for nout outputs.
int fft_forward(const FftMesh &m, int route, cudaStream_t s);
int fft_solve(const FftMesh &m, bool ik, bool energy, const float *Vc, double *acc, cudaStream_t s);
int fft_inverse(const FftMesh &m, int route, int nout, cudaStream_t s);
// The whole transform pair of every batched mesh: three launches per class and z lines.
int fft_batch(const FftBatch &f, const long long *st, cudaStream_t s);

}  // namespace pdb
