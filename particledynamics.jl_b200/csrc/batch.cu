// Batched replicas of libpdb200: hundreds of independent LJ / WCA systems of uneven size (their
// own box, density and pair model) stepped together, one launch per stage over all replicas,
// the whole velocity-Verlet step captured into one CUDA graph.
//
// The replicas' particles are concatenated (replica r owns [first_r, first_r + N_r)); every
// replica has its own cell grid, and the grids are concatenated too (global cell = cell_base_r +
// local cell), so the counting sort of the ELL route (scan, scatter, id order per cell) serves
// all replicas in one pass.  Per-replica geometry and pair model sit in a small device table
// read through the read-only cache.  Stages per step:
//   1. k_batch_drift: half kick, drift, centred wrap in the replica's box, per-replica
//      displacement maxima since each replica's last build; the last block flags the replicas to
//      rebuild and sets the graph's IF condition when there is one;
//   2. the rebuild (IF node): k_batch_bin (flagged replicas re-binned, the others keep their
//      cells), the shared counting sort (which leaves the others' cell order unchanged),
//      k_batch_rows for the flagged replicas' cells only (one warp per cell, the replica's
//      stencil staged in shared memory, rows identical to the single-system kernels'), the
//      capacity commit by the last block;
//   3. k_batch_pack (coordinates in cell order) and k_batch_pairs<G>: G lanes per row (G chosen by
//      the caller's autotuner), the replica's LJ or WCA model; the closing half kick is fused into
//      it for small batches, and runs in k_batch_finish for those of BATCH_SLOT_MIN particles or
//      more and in the meshes' gather for charged ones; the device step advances.
// Rows live in cell order (entry t of the particle at position k of the cell order at k * cap + t,
// entries are cell-order positions), so a row's entries are contiguous and the neighbours' packed
// records of a row sit in nearby cells.
//
// Charged replicas (the batched ionic melts) add the real-space Coulomb polynomial to the pair kernel
// and a mesh per replica (batch_mesh.cu): the step's force pass packs coordinates and charges once,
// runs the pair kernel while the mesh branch (spread, transforms with the influence multiply) runs on
// a second stream, and the gather joins both and applies the closing half kick.
#include <cmath>
#include <cstring>
#include <vector>

#include "chain.cuh"
#include "common.cuh"
#include "ell_common.cuh"
#include "internal.hpp"
#include "rows.cuh"

#include <algorithm>
#include <numeric>
#include <tuple>

using namespace pdb;

namespace pdb {

constexpr int B_THREADS = 256;

struct BatchRep {
    float L[3];
    int nx, ny, nz, cell_base;
    int kind;
    float eps, sig2, rc2, eshift;
};

__device__ __forceinline__ float wrap_centred(float x, float L) {
    x -= (x >= 0.5f * L) ? L : 0.f;
    x += (x < -0.5f * L) ? L : 0.f;
    return x;
}

// Rebuild decision per replica, taken by the whole last block of the drift kernel: replica r is
// rebuilt when one of its particles moved more than skin / 2 since its last build, and every replica
// when the list is invalid or the rebuild interval is reached.  Sets the device request (and the
// graph's IF condition) when any replica is rebuilt.
template <bool COND>
__device__ void batch_decide(long long *st, unsigned *rep_dmax, int *rep_flag, int nrep, float threshold,
                             bool thread0, cudaGraphConditionalHandle h) {
    __shared__ int any, all, bad;
    if (thread0) {
        st[E_CHECKS] += 1;
        st[E_REQUEST] = 0;
        bad = !isfinite(__uint_as_float((unsigned)st[E_DMAX]));
        all = st[E_VALID] == 0 || st[E_STEP] - st[E_LAST_BUILD] >= st[E_INTERVAL];
        any = 0;
        st[E_DMAX] = 0;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < nrep; r += blockDim.x) {
        const int f = (all || __uint_as_float(rep_dmax[r]) > threshold) ? 1 : 0;
        rep_flag[r] = f;
        rep_dmax[r] = 0u;
        if (f) any = 1;   // benign race: every writer stores 1
    }
    __syncthreads();
    if (thread0) {
        if (bad) {
            st[E_ERROR] = E_ERR_COORD;
            st[E_VALID] = 0;
        } else if (any) {
            st[E_REQUEST] = 1;
            st[E_VALID] = 0;
        }
        if (COND) cudaGraphSetConditional(h, ell_requested(st) ? 1u : 0u);
    }
}

// Half kick, drift, wrap and displacement (DRIFT), or the displacement of the current coordinates
// alone; per-replica displacement maxima, the decision by the last block.
template <bool DRIFT, bool COND>
__global__ void __launch_bounds__(B_THREADS) k_batch_drift(int n, int items, float *__restrict__ x, float *__restrict__ y,
                                                           float *__restrict__ z, float *__restrict__ vx,
                                                           float *__restrict__ vy, float *__restrict__ vz,
                                                           const float *__restrict__ fx, const float *__restrict__ fy,
                                                           const float *__restrict__ fz,
                                                           const float *__restrict__ inv_mass, float dt,
                                                           const int *__restrict__ rep_of,
                                                           const BatchRep *__restrict__ reps,
                                                           const float4 *__restrict__ ref, float threshold,
                                                           const int *__restrict__ pos_of, float4 *__restrict__ xq,
                                                           unsigned *__restrict__ rep_dmax, int *__restrict__ rep_flag,
                                                           int nrep, long long *__restrict__ st,
                                                           cudaGraphConditionalHandle h) {
    chain_begin();
    if (st[E_ERROR] != 0) {
        if (COND && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(h, 0u);
        return;
    }
    unsigned most = 0;
    // `items` rounds per block: the fence and the ticket come once for all of them
    for (int it = 0; it < items; ++it) {
        const int i = (blockIdx.x * items + it) * B_THREADS + threadIdx.x;
        float v = 0.f;
        int r = -1;
        if (i < n) {
            r = __ldg(rep_of + i);
            const BatchRep &R = reps[r];
            const float L[3] = {R.L[0], R.L[1], R.L[2]};
            float p[3] = {x[i], y[i], z[i]};
            if (DRIFT) {
                const float c = 0.5f * dt * inv_mass[i];
                const float u[3] = {fmaf(c, fx[i], vx[i]), fmaf(c, fy[i], vy[i]), fmaf(c, fz[i], vz[i])};
                vx[i] = u[0];
                vy[i] = u[1];
                vz[i] = u[2];
#pragma unroll
                for (int d = 0; d < 3; ++d) p[d] = wrap_centred(fmaf(dt, u[d], p[d]), L[d]);
                x[i] = p[0];
                y[i] = p[1];
                z[i] = p[2];
                if (pos_of) xq[pos_of[i]] = make_float4(p[0], p[1], p[2], 0.f);   // packed for the pair pass
            }
            v = ell_displacement<3>(p, ref[i], L, st[E_VALID] != 0);
        }
        // per-replica maximum: one atomic per warp where the warp's particles share a replica
        const unsigned bits = __float_as_uint(v);
        most = max(most, bits);
        const int r0 = __shfl_sync(0xffffffffu, r, 0);
        if (__all_sync(0xffffffffu, r == r0)) {
            const unsigned m = __reduce_max_sync(0xffffffffu, bits);
            if ((threadIdx.x & 31) == 0 && r0 >= 0) atomicMax(rep_dmax + r0, m);
        } else if (r >= 0) {
            atomicMax(rep_dmax + r, bits);
        }
    }
    __threadfence();   // the per-replica maxima are visible before this block's ticket
    __shared__ bool last_block;
    const bool t0last = ell_block_max_last(most, st, E_DMAX, E_TICKET_D);
    if (threadIdx.x == 0) last_block = t0last;
    __syncthreads();
    if (last_block) {
        __threadfence();
        if (threadIdx.x == 0) st[E_TICKET_D] = 0;
        batch_decide<COND>(st, rep_dmax, rep_flag, nrep, threshold, threadIdx.x == 0, h);
    }
}

// Global cell of every particle (its replica's grid) and the cell histogram.
// Particles of replicas that are not rebuilt keep their cells, so that their cell-order positions,
// and with them their rows, stay valid through the counting sort.
__global__ void k_batch_bin(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                            int n, const int *__restrict__ rep_of, const BatchRep *__restrict__ reps,
                            const int *__restrict__ rep_flag, int *__restrict__ cell_of, int *__restrict__ cell_count,
                            const long long *__restrict__ st) {
    chain_begin();
    if (!ell_requested(st)) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = __ldg(rep_of + i);
    if (!rep_flag[r]) {
        atomicAdd(&cell_count[cell_of[i]], 1);
        return;
    }
    const BatchRep &R = reps[r];
    const float p[3] = {x[i], y[i], z[i]};
    const int ng[3] = {R.nx, R.ny, R.nz};
    int cc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float u = p[d] + 0.5f * R.L[d];
        u -= floorf(u / R.L[d]) * R.L[d];
        cc[d] = min(max((int)floorf(u * ((float)ng[d] / R.L[d])), 0), ng[d] - 1);
    }
    const int c = R.cell_base + (cc[2] * R.ny + cc[1]) * R.nx + cc[0];
    cell_of[i] = c;
    atomicAdd(&cell_count[c], 1);
}

// Rows of the flagged replicas' cells, nsplit warps per global cell (rows.cuh): rows, their lengths and their
// entries are in cell order (positions in `sorted`).  Five blocks per SM, 96 registers: at the 80 of six the replica's
// grid spills (96 replicas, five steps: 1588 us with six, 1359 with five; 12 melts 859, 818).
__global__ void __launch_bounds__(32 * ROWS_WARPS, 5) k_batch_rows(
    const float4 *__restrict__ xq, int ncell, int nsplit, const int *__restrict__ cell_rep,
    const BatchRep *__restrict__ reps, const int *__restrict__ rep_flag, const int *__restrict__ sorted,
    const int *__restrict__ cell_off, float rl2, int cap, int *__restrict__ rows, int *__restrict__ counts,
    float4 *__restrict__ ref, long long *__restrict__ st) {
    chain_begin();
    if (!ell_requested(st)) return;
    extern __shared__ float4 batch_stage[];
    const int w = threadIdx.x >> 5;
    const int item = blockIdx.x * ROWS_WARPS + w, c = item / nsplit;
    unsigned fmax = 0;
    if (c < ncell) {
        const int r = __ldg(cell_rep + c);
        if (rep_flag[r]) {   // warp-uniform; only replicas being rebuilt
            const BatchRep &R = reps[r];
            const RowGrid g{{R.L[0], R.L[1], R.L[2]}, R.nx, R.ny, R.nz, R.cell_base};
            fmax = cell_rows<3>(g, c - g.base, item - c * nsplit, nsplit, xq, sorted, cell_off, rl2, cap, rows, counts,
                                ref, batch_stage + w * ROWS_CAP);
        }
    }
    if (ell_block_max_last(fmax, st, E_RMAX, E_TICKET_R)) rows_commit(st, cap);
}

// The rows in the exported layout (slot t of position k at t n + k) for callers that read them.
__global__ void k_batch_export(const int *__restrict__ rows, const int *__restrict__ counts, int n, int cap,
                               int *__restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = min(counts[k], cap);
    for (int t = 0; t < c; ++t) out[(size_t)t * n + k] = rows[(size_t)k * cap + t];
}

// Packed coordinates (and charges, when q is given) in cell order: xq[k] = (x, y, z, q) of particle
// sorted[k].  REBUILD: the pack that feeds the row build of a rebuild (runs while the rows are being
// rebuilt); otherwise the pack of the pair pass (skipped while the rows are invalid).
template <bool REBUILD>
__global__ void k_batch_pack(const float *__restrict__ x, const float *__restrict__ y, const float *__restrict__ z,
                             const float *__restrict__ q, const int *__restrict__ sorted, int n,
                             int *__restrict__ pos_of, float4 *__restrict__ xq, const long long *__restrict__ st) {
    chain_begin();
    if (REBUILD ? !ell_requested(st) : st[E_VALID] == 0) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = sorted[k];
    if (REBUILD) pos_of[i] = k;
    xq[k] = make_float4(x[i], y[i], z[i], q ? q[i] : 0.f);
}

struct BatchKick {
    float *vx, *vy, *vz;
    const float *inv_mass;
    float half_dt;
    int on;
};

// Real-space Coulomb of charged replicas, shared by every replica (one split and cutoff): the
// cluster route's fitted polynomial (pair_force, PairFunctor.jl:127-156), f/r = C qq (r^-3 - P_f(x)),
// e = C qq (1/r + P_e(x) - eshift), x = r^2 sx - 1, inside rc2.  Monomial coefficients, constant term
// first, zero above the fitted degree.
constexpr int BATCH_NP = 16;
struct BatchCoul {
    float C, rc2, sx, eshift;
    float pf[BATCH_NP], pe[BATCH_NP];
};

// Row pair kernel over all replicas: the model of particle i's replica (LJ or WCA, the ELL route's
// UniformLJ / UniformWCA arithmetic), forces stored, optional energy (half of each pair).  G lanes per row.
// The packed coordinates are refreshed by the pack of the same stage.
// COUL: the packed records carry the charges (xq.w) and the pair adds the Coulomb polynomial term,
// evaluated with NP coefficients (the fitted ones, zeros above them); one reciprocal square root
// serves both terms.
// SLOT: forces (and the energy) are stored by position in fc, one coalesced record, for the kernel that carries
// them to particle order with the closing half kick (k_batch_finish, or the charged replicas' gather).
template <int G, bool ENERGY, bool COUL, bool SLOT, int NP = BATCH_NP>
__global__ void __launch_bounds__(B_THREADS) k_batch_pairs(const float4 *__restrict__ xq, int n, int cap,
                                                           const int *__restrict__ rows,
                                                           const int *__restrict__ counts,
                                                           const int *__restrict__ sorted,
                                                           const int *__restrict__ rep_of,
                                                           const BatchRep *__restrict__ reps, float *__restrict__ fx,
                                                           float *__restrict__ fy, float *__restrict__ fz,
                                                           float *__restrict__ epot, float4 *__restrict__ fc,
                                                           BatchKick kick, long long *__restrict__ st, int advance,
                                                           float face, const __grid_constant__ BatchCoul cp) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x;
    const int k = tid / G, lane = tid % G;   // position in cell order
    const int i = k < n ? sorted[k] : -1;
    float a[3] = {0.f, 0.f, 0.f}, e = 0.f;
    const BatchRep &R = reps[k < n ? __ldg(rep_of + i) : 0];
    const float L[3] = {R.L[0], R.L[1], R.L[2]};
    const float rc2 = R.rc2;
    const LjRow lj = lj_row(R.eps, R.sig2, rc2, R.kind == PD_PAIR_WCA ? R.eps : -R.eshift);
    const float4 pi = k < n ? xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int cnt = k < n ? counts[k] : 0;
    const float cqi = COUL ? cp.C * pi.w : 0.f;
    const float cut2 = COUL ? fmaxf(rc2, cp.rc2) : rc2;
    f2 npf[COUL ? NP : 1];   // minus the force polynomial
    if (COUL) {
#pragma unroll
        for (int t = 0; t < NP; ++t) npf[t] = pk_held(-cp.pf[t]);
    }
    auto walk = [&](auto wrap) {
        constexpr bool WRAP = decltype(wrap)::value;
        walk_row<G, true>(rows + (size_t)k * cap, 1, lane, cnt, k, xq, [&](const float4 &pa, const float4 &pb) {
            float dx[2], dy[2], dz[2], r2[2], f[2], u[2];
            pair_delta<3, WRAP>(pi, pa, L, dx[0], dy[0], dz[0]);
            pair_delta<3, WRAP>(pi, pb, L, dx[1], dy[1], dz[1]);
#pragma unroll
            for (int c = 0; c < 2; ++c) r2[c] = fmaf(dx[c], dx[c], fmaf(dy[c], dy[c], dz[c] * dz[c]));
            const f2 r22 = pk(r2[0], r2[1]);
            f2 fr, un, rinv, ir2;
            if (COUL) {
                rinv = pk(rsqrt_fast(r2[0]), rsqrt_fast(r2[1]));
                ir2 = mul2(rinv, rinv);
            } else {
                ir2 = rcp2(r22);
            }
            lj_two<ENERGY>(lj, ir2, fr, un);
            unpk(fr, f[0], f[1]);
            if (ENERGY) unpk(un, u[0], u[1]);
            bool in[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                in[c] = r2[c] > 0.f && r2[c] < rc2;
                f[c] = in[c] ? f[c] : 0.f;
                if (ENERGY) e += in[c] ? 0.5f * u[c] : 0.f;
            }
            if (COUL) {
                const f2 x = fma2(r22, pk(cp.sx), pk(-1.f));
                f2 g = npf[NP - 1];
#pragma unroll
                for (int t = NP - 2; t >= 0; --t) g = fma2(g, x, npf[t]);
                float q[2], h[2];
                unpk(fma2(rinv, ir2, g), h[0], h[1]);
                unpk(mul2(pk(cqi), pk(pa.w, pb.w)), q[0], q[1]);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    in[c] = r2[c] > 0.f && r2[c] < cp.rc2;
                    f[c] = fmaf(q[c], in[c] ? h[c] : 0.f, f[c]);
                }
                if (ENERGY) {
                    f2 pe = pk(cp.pe[NP - 1]);
#pragma unroll
                    for (int t = NP - 2; t >= 0; --t) pe = fma2(pe, x, pk(cp.pe[t]));
                    unpk(add2(add2(rinv, pe), pk(-cp.eshift)), h[0], h[1]);
#pragma unroll
                    for (int c = 0; c < 2; ++c) e = fmaf(0.5f * q[c], in[c] ? h[c] : 0.f, e);
                }
            }
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (!(r2[c] > 0.f && r2[c] < cut2)) continue;   // a difference that is not finite adds nothing
                a[0] = fmaf(f[c], dx[c], a[0]);
                a[1] = fmaf(f[c], dy[c], a[1]);
                a[2] = fmaf(f[c], dz[c], a[2]);
            }
        });
    };
    // face: 1.001 keeps the faces farther than the cutoff by more than the coordinates' rounding; infinite for
    // coordinates that may lie beyond them
    if (__all_sync(0xffffffffu, cnt == 0 || clear_of_faces<3>(pi, L, face * sqrtf(cut2)))) walk(std::false_type{});
    else walk(std::true_type{});
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int d = 0; d < 3; ++d) a[d] += __shfl_down_sync(0xffffffffu, a[d], off, G);
        if (ENERGY) e += __shfl_down_sync(0xffffffffu, e, off, G);
    }
    if (lane == 0 && k < n) {
        if (SLOT) {
            fc[k] = make_float4(a[0], a[1], a[2], e);
        } else {
            fx[i] = a[0];
            fy[i] = a[1];
            fz[i] = a[2];
            if (ENERGY) epot[i] = e;
            if (kick.on) {
                const float c = kick.half_dt * kick.inv_mass[i];
                kick.vx[i] = fmaf(c, a[0], kick.vx[i]);
                kick.vy[i] = fmaf(c, a[1], kick.vy[i]);
                kick.vz[i] = fmaf(c, a[2], kick.vz[i]);
            }
        }
    }
    if (advance && blockIdx.x == 0 && threadIdx.x == 0) st[E_STEP] += 1;
}

// The uncharged pair pass with one lane per row: a thread adds its row's terms in row order, so the sums are those
// of the row order itself.  A warp's 32 rows are read eight entries at a time by eight lanes each (whole sectors of
// the row-major rows) and turned around in shared memory.  96 replicas, 568 986 atoms: 158 us (eight lanes per row:
// 133 us, slot-major rows read entry by entry: 225 us).
constexpr int SEQ_E = 8;   // entries per turn
template <bool ENERGY, bool SLOT>
__global__ void __launch_bounds__(B_THREADS, 3) k_batch_pairs_seq(const float4 *__restrict__ xq, int n, int cap,
                                                               const int *__restrict__ rows,
                                                               const int *__restrict__ counts,
                                                               const int *__restrict__ sorted,
                                                               const int *__restrict__ rep_of,
                                                               const BatchRep *__restrict__ reps,
                                                               float *__restrict__ fx, float *__restrict__ fy,
                                                               float *__restrict__ fz, float *__restrict__ epot,
                                                               float4 *__restrict__ fc, BatchKick kick,
                                                               long long *__restrict__ st, int advance,
                                                               float face) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    __shared__ int turn[B_THREADS / 32][32 * (SEQ_E + 1)];
    const int k = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    int *mine = turn[threadIdx.x >> 5];
    const bool live = k < n;
    const int i = live ? sorted[k] : -1;
    const BatchRep &R = reps[live ? __ldg(rep_of + i) : 0];
    const float L[3] = {R.L[0], R.L[1], R.L[2]};
    const LjRow lj = lj_row(R.eps, R.sig2, R.rc2, R.kind == PD_PAIR_WCA ? R.eps : -R.eshift);
    const float4 pi = live ? xq[k] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int cnt = live ? counts[k] : 0;
    const int most = __reduce_max_sync(0xffffffffu, cnt);
    float a[3] = {0.f, 0.f, 0.f}, e = 0.f;
    // lane reads entry c0 + (lane & 7) of rows (lane >> 3) + 4 u, u < 8; past a row's end its own position
    int at[SEQ_E], rc[SEQ_E];
    const int k0 = k - lane, er = lane & (SEQ_E - 1);
#pragma unroll
    for (int u = 0; u < SEQ_E; ++u) rc[u] = __shfl_sync(0xffffffffu, cnt, (lane >> 3) + 4 * u);
    auto fetch = [&](int c0) {
#pragma unroll
        for (int u = 0; u < SEQ_E; ++u) {
            const int r = k0 + (lane >> 3) + 4 * u, t = c0 + er;
            at[u] = t < rc[u] ? __ldg(rows + (size_t)r * cap + t) : min(r, n - 1);
        }
    };
    auto walk = [&](auto wrap) {
        constexpr bool WRAP = decltype(wrap)::value;
        fetch(0);
        for (int c0 = 0; c0 < most; c0 += SEQ_E) {
            __syncwarp();
#pragma unroll
            for (int u = 0; u < SEQ_E; ++u) mine[((lane >> 3) + 4 * u) * (SEQ_E + 1) + er] = at[u];
            __syncwarp();
            float4 p[SEQ_E];
#pragma unroll
            for (int u = 0; u < SEQ_E; ++u) p[u] = __ldg(xq + mine[lane * (SEQ_E + 1) + u]);
            if (c0 + SEQ_E < most) fetch(c0 + SEQ_E);
#pragma unroll
            for (int u = 0; u < SEQ_E; u += 2) {
                float dx[2], dy[2], dz[2], r2[2], f[2], v[2];
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    pair_delta<3, WRAP>(pi, p[u + c], L, dx[c], dy[c], dz[c]);
                    r2[c] = fmaf(dx[c], dx[c], fmaf(dy[c], dy[c], dz[c] * dz[c]));
                }
                f2 fr, un;
                lj_two<ENERGY>(lj, rcp2(pk(r2[0], r2[1])), fr, un);
                unpk(fr, f[0], f[1]);
                if (ENERGY) unpk(un, v[0], v[1]);
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    if (!(r2[c] > 0.f && r2[c] < lj.rc2)) continue;   // a difference that is not finite adds nothing
                    a[0] = fmaf(f[c], dx[c], a[0]);
                    a[1] = fmaf(f[c], dy[c], a[1]);
                    a[2] = fmaf(f[c], dz[c], a[2]);
                    if (ENERGY) e += 0.5f * v[c];
                }
            }
        }
    };
    if (__all_sync(0xffffffffu, cnt == 0 || clear_of_faces<3>(pi, L, face * sqrtf(lj.rc2)))) walk(std::false_type{});
    else walk(std::true_type{});
    if (live) {
        if (SLOT) {
            fc[k] = make_float4(a[0], a[1], a[2], e);
        } else {
            fx[i] = a[0];
            fy[i] = a[1];
            fz[i] = a[2];
            if (ENERGY) epot[i] = e;
            if (kick.on) {
                const float c = kick.half_dt * kick.inv_mass[i];
                kick.vx[i] = fmaf(c, a[0], kick.vx[i]);
                kick.vy[i] = fmaf(c, a[1], kick.vy[i]);
                kick.vz[i] = fmaf(c, a[2], kick.vz[i]);
            }
        }
    }
    if (advance && blockIdx.x == 0 && threadIdx.x == 0) st[E_STEP] += 1;
}

// Positions' forces to particle order, with the closing half kick when there is one.
template <bool ENERGY>
__global__ void __launch_bounds__(B_THREADS) k_batch_finish(const float4 *__restrict__ fc,
                                                            const int *__restrict__ pos_of, int n,
                                                            float *__restrict__ fx, float *__restrict__ fy,
                                                            float *__restrict__ fz, float *__restrict__ epot,
                                                            BatchKick kick, long long *__restrict__ st, int advance) {
    chain_begin();
    if (st[E_VALID] == 0) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float4 f = fc[pos_of[i]];
        fx[i] = f.x;
        fy[i] = f.y;
        fz[i] = f.z;
        if (ENERGY) epot[i] = f.w;
        if (kick.on) {
            const float c = kick.half_dt * kick.inv_mass[i];
            kick.vx[i] = fmaf(c, f.x, kick.vx[i]);
            kick.vy[i] = fmaf(c, f.y, kick.vy[i]);
            kick.vz[i] = fmaf(c, f.z, kick.vz[i]);
        }
    }
    if (advance && blockIdx.x == 0 && threadIdx.x == 0) st[E_STEP] += 1;
}

}  // namespace pdb

struct pd_batch {
    int nrep = 0, n = 0, ncell = 0, cap = 0, lanes = 4;
    int num_sms = device_sms();
    double mean_row = 0.0;           // expected entries per row at the replicas' densities
    float rl2 = 0.f, threshold = 0.f;
    std::vector<BatchRep> hreps;
    std::vector<int> first;
    BatchRep *reps = nullptr;
    int *rep_of = nullptr, *cell_rep = nullptr;
    int *rep_flag = nullptr;         // replicas rebuilt by the current decision
    unsigned *rep_dmax = nullptr;    // per-replica displacement maxima (float bits)
    long long *st = nullptr;
    int *cell_of = nullptr, *cell_count = nullptr, *cell_off = nullptr, *sorted = nullptr, *tmp = nullptr;
    int *rows = nullptr, *counts = nullptr;
    int *pos_of = nullptr, *scan_part = nullptr;   // inverse of sorted; tile sums of the cell scan
    int *xrows = nullptr;            // rows in the exported layout, kept current once pd_batch_rows was called
    float4 *ref = nullptr, *xq = nullptr, *fc = nullptr;
    // bound state (pd_batch_bind)
    pd_md_state state;
    bool bound = false;
    cudaStream_t body = nullptr;
    bool cond_nodes = true;
    cudaGraphExec_t exec = nullptr;
    float exec_dt = 0.f;
    int exec_lanes = 0;
    cudaStream_t exec_stream = nullptr;
    int exec_chunk = 0;
    std::vector<double> box;          // 3 per replica, as given
    // charged replicas: real-space Coulomb and the batched meshes
    bool coul = false;
    BatchCoul cp{};
    int coul_ne = 0, coul_nf = 0;
    float half_c_self = 0.f;
    bool mesh = false;
    int morder = 5, mchunk = 64, nchunk = 0, mtpi = 2;
    std::vector<BMeshRep> hmreps;
    BMeshRep *mreps = nullptr;
    int *chunk_rep = nullptr, *slot_src = nullptr, *mid = nullptr;
    float4 *mq = nullptr;
    float *gridA = nullptr, *gridB = nullptr, *G = nullptr;
    float2 *spec = nullptr;
    long long total_nodes = 0, total_modes = 0;
    struct FftGroup {
        int K1, K2, K3, count;
        long long grid, modes;
        cufftHandle fwd, bwd;
    };
    std::vector<FftGroup> groups;
    // every replica's mesh on this library's transforms: three launches for the whole set (fft.tab set);
    // otherwise the cuFFT groups
    FftBatch fft{};
    FftMesh *fft_tab = nullptr;
    int2 *fft_planes = nullptr, *fft_cols = nullptr;
    std::vector<float2 *> twiddles;
    // the mesh sizes' transforms run on NFFT streams at once, group g on stream g % NFFT with that
    // stream's own cuFFT work area
    static constexpr int NFFT = 4;
    void *fft_work[NFFT] = {};
    cudaStream_t fft_stream[NFFT] = {};
    cudaEvent_t ev_fft[NFFT] = {};
    cudaEvent_t ev_fft_fork = nullptr;
    cudaStream_t mesh_stream = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
};

namespace pdb {

static void batch_free_chunks(pd_batch *b) {
    dfree(b->chunk_rep);
    dfree(b->slot_src);
    dfree(b->mid);
    dfree(b->mq);
    b->nchunk = 0;
}

static void batch_free_mesh(pd_batch *b) {
    for (auto &g : b->groups) {
        if (g.fwd) cufftDestroy(g.fwd);
        if (g.bwd) cufftDestroy(g.bwd);
    }
    b->groups.clear();
    for (auto &w : b->twiddles) dfree(w);
    b->twiddles.clear();
    dfree(b->fft_tab);
    dfree(b->fft_planes);
    dfree(b->fft_cols);
    b->fft = FftBatch{};
    batch_free_chunks(b);
    dfree(b->mreps);
    dfree(b->gridA);
    dfree(b->gridB);
    dfree(b->G);
    dfree(b->spec);
    for (int k = 0; k < pd_batch::NFFT; ++k) {
        if (b->fft_work[k]) cudaFree(b->fft_work[k]);
        if (b->fft_stream[k]) cudaStreamDestroy(b->fft_stream[k]);
        if (b->ev_fft[k]) cudaEventDestroy(b->ev_fft[k]);
        b->fft_work[k] = nullptr;
        b->fft_stream[k] = nullptr;
        b->ev_fft[k] = nullptr;
    }
    if (b->ev_fft_fork) cudaEventDestroy(b->ev_fft_fork);
    b->ev_fft_fork = nullptr;
    if (b->mesh_stream) cudaStreamDestroy(b->mesh_stream);
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->ev_join) cudaEventDestroy(b->ev_join);
    b->mesh_stream = nullptr;
    b->ev_fork = b->ev_join = nullptr;
    b->mesh = false;
}

static void batch_free(pd_batch *b) {
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    batch_free_mesh(b);
    if (b->body) cudaStreamDestroy(b->body);
    b->body = nullptr;
    dfree(b->reps);
    dfree(b->rep_of);
    dfree(b->cell_rep);
    dfree(b->rep_flag);
    dfree(b->rep_dmax);
    dfree(b->st);
    dfree(b->cell_of);
    dfree(b->cell_count);
    dfree(b->cell_off);
    dfree(b->sorted);
    dfree(b->tmp);
    dfree(b->rows);
    dfree(b->counts);
    dfree(b->ref);
    dfree(b->xq);
    dfree(b->fc);
    dfree(b->pos_of);
    dfree(b->scan_part);
    dfree(b->xrows);
}

static int batch_blocks(const pd_batch *b) { return (b->n + B_THREADS - 1) / B_THREADS; }

static int batch_rebuild_launch(pd_batch *b, const float *x, const float *y, const float *z, cudaStream_t s) {
    const int blocks = (b->n + B_THREADS - 1) / B_THREADS;
    launch_chained(k_batch_bin, blocks, B_THREADS, 0, s, x, y, z, b->n, b->rep_of, b->reps, b->rep_flag, b->cell_of,
                                             b->cell_count, b->st);
    PD_LAUNCHED();
    int rc;
    if ((rc = ell_sort_launch(b->cell_of, b->n, b->ncell, b->cell_count, b->cell_off, b->scan_part, b->sorted, b->tmp,
                              b->st, s)))
        return rc;
    launch_chained(k_batch_pack<true>, blocks, B_THREADS, 0, s, x, y, z, nullptr, b->sorted, b->n, b->pos_of, b->xq, b->st);
    PD_LAUNCHED();
    const int nsplit = rows_split(b->ncell, b->num_sms);
    const int grid = (int)(((long long)b->ncell * nsplit + ROWS_WARPS - 1) / ROWS_WARPS);
    launch_chained(k_batch_rows, grid, 32 * ROWS_WARPS, sizeof(float4) * ROWS_WARPS * ROWS_CAP, s, 
        b->xq, b->ncell, nsplit, b->cell_rep, b->reps, b->rep_flag, b->sorted, b->cell_off, b->rl2, b->cap, b->rows,
        b->counts, b->ref, b->st);
    PD_LAUNCHED();
    if (b->xrows) {
        k_batch_export<<<blocks, B_THREADS, 0, s>>>(b->rows, b->counts, b->n, b->cap, b->xrows);
        PD_LAUNCHED();
    }
    return PD_OK;
}

// Lanes per row that the pair kernel runs with.  Charged rows are long and every choice below 8 lanes reads their
// sectors several times; uncharged rows take the caller's choice.
static int batch_lanes(const pd_batch *b) {
    return b->coul ? std::max(b->lanes, b->mean_row < 4.0 ? 1 : b->mean_row < 12.0 ? 4 : 8) : b->lanes;
}

template <bool COUL, int NP = BATCH_NP>
static void launch_batch_pairs(pd_batch *b, float *fx, float *fy, float *fz, float *epot, int energy,
                               const BatchKick &kick, int advance, bool slot, bool centred, cudaStream_t s) {
    const float face = centred ? 1.001f : INFINITY;
    const int G = batch_lanes(b);
    const int blocks = (int)(((long long)b->n * G + B_THREADS - 1) / B_THREADS);
    if constexpr (!COUL) {
        if (G == 1) {
#define PD_BS(EE, SS)                                                                                               \
    launch_chained(k_batch_pairs_seq<EE, SS>, blocks, B_THREADS, 0, s, b->xq, b->n, b->cap, b->rows, b->counts,     \
                   b->sorted, b->rep_of, b->reps, fx, fy, fz, epot, b->fc, kick, b->st, advance, face)
            if (slot) {
                if (energy) PD_BS(true, true);
                else PD_BS(false, true);
            } else {
                if (energy) PD_BS(true, false);
                else PD_BS(false, false);
            }
#undef PD_BS
            return;
        }
    }
#define PD_BP2(GG, EE, SS)                                                                                            \
    launch_chained(k_batch_pairs<GG, EE, COUL, SS, NP>, blocks, B_THREADS, 0, s, b->xq, b->n, b->cap, b->rows, b->counts,         \
                                                                     b->sorted, b->rep_of, b->reps, fx, fy, fz, epot, \
                                                                     b->fc, kick, b->st, advance, face, b->cp)
#define PD_BP(GG)                                                                                                     \
    if (slot) {                                                                                                       \
        if (energy) PD_BP2(GG, true, true);                                                                           \
        else PD_BP2(GG, false, true);                                                                                 \
    } else if constexpr (!COUL) {                                                                                     \
        if (energy) PD_BP2(GG, true, false);                                                                          \
        else PD_BP2(GG, false, false);                                                                                \
    }
    switch (G) {
        case 1:
            if constexpr (COUL) { PD_BP(1) }
            break;
        case 2: PD_BP(2) break;
        case 4: PD_BP(4) break;
        default: PD_BP(8) break;
    }
#undef PD_BP
#undef PD_BP2
}

static BMeshView batch_mesh_view(const pd_batch *b) {
    BMeshView v;
    v.order = b->morder;
    v.chunk = b->mchunk;
    v.tpi = b->mtpi;
    v.nchunk = b->nchunk;
    v.nrep = b->nrep;
    v.reps = b->mreps;
    v.chunk_rep = b->chunk_rep;
    v.slot_src = b->slot_src;
    v.mq = b->mq;
    v.mid = b->mid;
    v.fc = b->fc;
    v.gridA = b->gridA;
    v.gridB = b->gridB;
    v.spec = b->spec;
    v.G = b->G;
    v.total_nodes = b->total_nodes;
    v.total_modes = b->total_modes;
    return v;
}

// The mesh branch of charged replicas: spread, the batched forward transforms (one per mesh size),
// the influence multiply, the batched inverse transforms.
// Transforms of every mesh size, forked from s onto the FFT streams and joined back into s.
static int batch_fft_all(pd_batch *b, bool forward, cudaStream_t s) {
    const int ns = std::min<int>(pd_batch::NFFT, (int)b->groups.size());
    PD_CUDA(cudaEventRecord(b->ev_fft_fork, s));
    for (int k = 0; k < ns; ++k) PD_CUDA(cudaStreamWaitEvent(b->fft_stream[k], b->ev_fft_fork, 0));
    for (size_t gi = 0; gi < b->groups.size(); ++gi) {
        auto &g = b->groups[gi];
        cudaStream_t fs = b->fft_stream[gi % pd_batch::NFFT];
        if (forward) {
            PD_CHECK(cufftSetStream(g.fwd, fs) == CUFFT_SUCCESS, PD_ECUFFT, "batched mesh: cufftSetStream failed");
            PD_CHECK(cufftExecR2C(g.fwd, b->gridA + g.grid, reinterpret_cast<cufftComplex *>(b->spec + g.modes)) ==
                         CUFFT_SUCCESS,
                     PD_ECUFFT, "batched mesh: forward transform failed");
        } else {
            PD_CHECK(cufftSetStream(g.bwd, fs) == CUFFT_SUCCESS, PD_ECUFFT, "batched mesh: cufftSetStream failed");
            PD_CHECK(cufftExecC2R(g.bwd, reinterpret_cast<cufftComplex *>(b->spec + g.modes), b->gridB + g.grid) ==
                         CUFFT_SUCCESS,
                     PD_ECUFFT, "batched mesh: inverse transform failed");
        }
    }
    for (int k = 0; k < ns; ++k) {
        PD_CUDA(cudaEventRecord(b->ev_fft[k], b->fft_stream[k]));
        PD_CUDA(cudaStreamWaitEvent(s, b->ev_fft[k], 0));
    }
    return PD_OK;
}

static int batch_mesh_transform(pd_batch *b, cudaStream_t s) {
    const BMeshView v = batch_mesh_view(b);
    int rc;
    if ((rc = bmesh_spread_launch(v, b->st, s))) return rc;
    if (b->fft.tab) return fft_batch(b->fft, b->st, s);
    if ((rc = batch_fft_all(b, true, s))) return rc;
    if ((rc = bmesh_solve_launch(v, b->st, s))) return rc;
    return batch_fft_all(b, false, s);
}

// From this size the pair kernel stores its forces by position and k_batch_finish carries them to particle order. Below
// it the two are within 4 % of each other either way (five steps, by particle / by position: 4757 atoms 242 / 251 us,
// 17 316 atoms 318 / 307), and the launch is saved.
constexpr int BATCH_SLOT_MIN = 32768;

// The force pass: pack (unless the drift has packed the coordinates), then the row pair kernel; with charges and meshes
// the pair kernel runs on s while the mesh branch runs on the batch's mesh stream (forked and joined by events, so the
// same code is captured into the step graph), and the gather joins both and applies the closing kick.
static int batch_pairs_launch(pd_batch *b, const float *x, const float *y, const float *z, float *fx, float *fy,
                              float *fz, float *epot, int energy, BatchKick kick, int advance, bool drifted,
                              cudaStream_t s) {
    const bool centred = drifted;   // a caller's own coordinates may have crossed a face since the update
    if (!b->coul) {
        const int blocks = (b->n + B_THREADS - 1) / B_THREADS;
        if (!drifted) {
            launch_chained(k_batch_pack<false>, blocks, B_THREADS, 0, s, x, y, z, nullptr, b->sorted, b->n, b->pos_of, b->xq, b->st);
            PD_LAUNCHED();
        }
        const bool slot = b->n >= BATCH_SLOT_MIN;
        launch_batch_pairs<false>(b, fx, fy, fz, epot, energy, kick, slot ? 0 : advance, slot, centred, s);
        PD_LAUNCHED();
        if (!slot) return PD_OK;
        if (energy)
            launch_chained(k_batch_finish<true>, blocks, B_THREADS, 0, s, b->fc, b->pos_of, b->n, fx, fy, fz, epot, kick, b->st,
                                                              advance);
        else
            launch_chained(k_batch_finish<false>, blocks, B_THREADS, 0, s, b->fc, b->pos_of, b->n, fx, fy, fz, epot, kick, b->st,
                                                               advance);
        PD_LAUNCHED();
        return PD_OK;
    }
    PD_CHECK(b->mesh && b->bound && b->state.q, PD_ESTATE,
             "charged replicas need their meshes (pd_batch_set_mesh) and a bound state with charges");
    const BMeshView v = batch_mesh_view(b);
    int rc;
    if ((rc = bmesh_pack_launch(v, x, y, z, b->state.q, b->sorted, b->xq, b->st, s))) return rc;
    PD_CUDA(cudaEventRecord(b->ev_fork, s));
    PD_CUDA(cudaStreamWaitEvent(b->mesh_stream, b->ev_fork, 0));
    if ((rc = batch_mesh_transform(b, b->mesh_stream))) return rc;
    PD_CUDA(cudaEventRecord(b->ev_join, b->mesh_stream));
    BatchKick nokick = kick;
    nokick.on = 0;
    // the polynomial's coefficient bucket: the fitted force coefficients, and the energy's with energy
    if (std::max(b->coul_nf, energy ? b->coul_ne : 0) <= 14)
        launch_batch_pairs<true, 14>(b, fx, fy, fz, epot, energy, nokick, advance, true, centred, s);
    else
        launch_batch_pairs<true, BATCH_NP>(b, fx, fy, fz, epot, energy, nokick, advance, true, centred, s);
    PD_LAUNCHED();
    PD_CUDA(cudaStreamWaitEvent(s, b->ev_join, 0));
    BMeshKick mk;
    mk.vx = kick.vx;
    mk.vy = kick.vy;
    mk.vz = kick.vz;
    mk.inv_mass = kick.inv_mass;
    mk.half_dt = kick.half_dt;
    mk.on = kick.on;
    return bmesh_gather_launch(v, fx, fy, fz, epot, energy, mk, b->half_c_self, b->st, s);
}

static int batch_enqueue_step(pd_batch *b, float dt, cudaStream_t s, int cond) {
    const pd_md_state &S = b->state;
    const int blocks = batch_blocks(b), items = drift_items(blocks, b->num_sms);
    cudaGraphConditionalHandle h = 0;
    if (cond) {
        cudaStreamCaptureStatus status;
        cudaGraph_t g = nullptr;
        PD_CUDA(cudaStreamGetCaptureInfo(s, &status, nullptr, &g, nullptr, nullptr));
        PD_CUDA(cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault));
        launch_chained(k_batch_drift<true, true>, (blocks + items - 1) / items, B_THREADS, 0, s, b->n, items, S.x, S.y, S.z, S.vx, S.vy, S.vz, S.fx, S.fy, S.fz,
                                                               S.inv_mass, dt, b->rep_of, b->reps, b->ref,
                                                               b->threshold, b->coul ? nullptr : b->pos_of, b->xq,
                                                               b->rep_dmax, b->rep_flag, b->nrep,
                                                               b->st, h);
    } else {
        launch_chained(k_batch_drift<true, false>, (blocks + items - 1) / items, B_THREADS, 0, s, b->n, items, S.x, S.y, S.z, S.vx, S.vy, S.vz, S.fx, S.fy,
                                                                S.fz, S.inv_mass, dt, b->rep_of, b->reps, b->ref,
                                                                b->threshold, b->coul ? nullptr : b->pos_of, b->xq,
                                                                b->rep_dmax, b->rep_flag, b->nrep,
                                                                b->st, 0);
    }
    PD_LAUNCHED();
    int rc;
    if (cond) {
        if ((rc = capture_if_body(s, b->body, h, [&](cudaStream_t cs) {
                 return batch_rebuild_launch(b, S.x, S.y, S.z, cs);
             })))
            return rc;
    } else if ((rc = batch_rebuild_launch(b, S.x, S.y, S.z, s))) {
        return rc;
    }
    BatchKick kick;
    kick.vx = S.vx;
    kick.vy = S.vy;
    kick.vz = S.vz;
    kick.inv_mass = S.inv_mass;
    kick.half_dt = 0.5f * dt;
    kick.on = 1;
    return batch_pairs_launch(b, S.x, S.y, S.z, S.fx, S.fy, S.fz, S.epot, 0, kick, 1, true, s);
}

}  // namespace pdb

extern "C" {

int pd_batch_create(pd_batch **out, const pd_batch_replica *reps, int nrep, float skin, int cap, int lanes) {
    PD_CHECK(out && reps && nrep > 0, PD_EINVAL, "pd_batch_create: bad argument");
    PD_CHECK(cap > 0, PD_EINVAL, "pd_batch_create: row capacity must be positive");
    PD_CHECK(lanes == 1 || lanes == 2 || lanes == 4 || lanes == 8, PD_EINVAL, "pd_batch_create: lanes 1, 2, 4 or 8");
    PD_CHECK(std::isfinite(skin) && skin >= 0.f, PD_EINVAL, "pd_batch_create: skin must be finite and nonnegative");
    *out = nullptr;
    float rmax = 0.f;
    for (int r = 0; r < nrep; ++r) {
        const pd_batch_replica &R = reps[r];
        PD_CHECK(R.n > 0, PD_EINVAL, "pd_batch_create: replica %d is empty", r);
        PD_CHECK(R.kind == PD_PAIR_LJ || R.kind == PD_PAIR_WCA, PD_EINVAL, "pd_batch_create: replica %d pair model", r);
        PD_CHECK(R.rc2 > 0.f && R.eps >= 0.f && R.sigma > 0.f, PD_EINVAL, "pd_batch_create: replica %d parameters", r);
        rmax = fmaxf(rmax, sqrtf(R.rc2));
    }
    const float rl = rmax + skin;
    pd_batch *b = new pd_batch();
    b->nrep = nrep;
    b->cap = cap;
    b->lanes = lanes;
    b->rl2 = rl * rl;
    b->threshold = 0.25f * skin * skin;
    std::vector<int> rep_of, cell_rep;
    for (int r = 0; r < nrep; ++r) {
        const pd_batch_replica &R = reps[r];
        BatchRep h;
        memset(&h, 0, sizeof h);
        int ng[3];
        for (int d = 0; d < 3; ++d) {
            if (!(std::isfinite(R.box[d]) && R.box[d] > 2.0 * rl)) {
                delete b;
                set_error("pd_batch_create: replica %d box length %g is not above twice the list radius %g", r,
                          R.box[d], 2.0 * rl);
                return PD_EINVAL;
            }
            h.L[d] = (float)R.box[d];
            // cells at least r_list wide; at least three per dimension (then the stencil spans the box)
            ng[d] = std::max(3, (int)std::floor(h.L[d] / rl));
        }
        h.nx = ng[0];
        h.ny = ng[1];
        h.nz = ng[2];
        h.cell_base = b->ncell;
        h.kind = R.kind;
        h.eps = R.eps;
        h.sig2 = R.sigma * R.sigma;
        h.rc2 = R.rc2;
        h.eshift = R.eshift;
        b->hreps.push_back(h);
        b->box.insert(b->box.end(), R.box, R.box + 3);
        b->first.push_back(b->n);
        b->mean_row += (double)R.n * R.n / (R.box[0] * R.box[1] * R.box[2]) * 4.18879 * (double)rl * rl * rl;
        b->n += R.n;
        const int nc = ng[0] * ng[1] * ng[2];
        b->ncell += nc;
        rep_of.insert(rep_of.end(), R.n, r);
        cell_rep.insert(cell_rep.end(), nc, r);
    }
    int rc;
    const size_t n = (size_t)b->n;
    b->mean_row /= b->n;
    if ((rc = dalloc(&b->reps, (size_t)nrep)) || (rc = dalloc(&b->rep_of, n)) ||
        (rc = dalloc(&b->cell_rep, (size_t)b->ncell)) || (rc = dalloc(&b->st, (size_t)E_LEN)) ||
        (rc = dalloc(&b->rep_flag, (size_t)nrep)) || (rc = dalloc(&b->rep_dmax, (size_t)nrep)) ||
        (rc = dalloc(&b->cell_of, n)) || (rc = dalloc(&b->cell_count, (size_t)b->ncell)) ||
        (rc = dalloc(&b->cell_off, (size_t)b->ncell + 1)) || (rc = dalloc(&b->sorted, n)) ||
        (rc = dalloc(&b->tmp, n)) || (rc = dalloc(&b->rows, n * (size_t)cap)) || (rc = dalloc(&b->counts, n)) ||
        (rc = dalloc(&b->ref, n)) || (rc = dalloc(&b->xq, n)) || (rc = dalloc(&b->fc, n)) ||
        (rc = dalloc(&b->pos_of, n)) || (rc = dalloc(&b->scan_part, ell_scan_part_len(b->ncell)))) {
        batch_free(b);
        delete b;
        return rc;
    }
    long long init[E_LEN] = {0};
    init[E_INTERVAL] = 100;
    std::vector<int> iota(n);
    for (size_t k = 0; k < n; ++k) iota[k] = (int)k;   // a valid cell order before the first build
    if (cudaMemcpy(b->reps, b->hreps.data(), sizeof(BatchRep) * nrep, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->sorted, iota.data(), sizeof(int) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->rep_of, rep_of.data(), sizeof(int) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->cell_rep, cell_rep.data(), sizeof(int) * b->ncell, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(b->st, init, sizeof init, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(b->cell_count, 0, sizeof(int) * (size_t)b->ncell) != cudaSuccess ||
        cudaMemset(b->rep_flag, 0, sizeof(int) * (size_t)nrep) != cudaSuccess ||
        cudaMemset(b->rep_dmax, 0, sizeof(unsigned) * (size_t)nrep) != cudaSuccess ||
        cudaMemset(b->scan_part, 0, sizeof(int) * ell_scan_part_len(b->ncell)) != cudaSuccess ||
        cudaMemcpy(b->pos_of, iota.data(), sizeof(int) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(b->cell_of, 0, sizeof(int) * n) != cudaSuccess ||
        cudaMemset(b->counts, 0, sizeof(int) * n) != cudaSuccess ||
        cudaMemset(b->ref, 0, sizeof(float4) * n) != cudaSuccess ||
        cudaStreamCreateWithFlags(&b->body, cudaStreamNonBlocking) != cudaSuccess) {
        batch_free(b);
        delete b;
        set_error("pd_batch_create: device initialisation failed");
        return PD_ECUDA;
    }
    *out = b;
    return PD_OK;
}

int pd_batch_destroy(pd_batch *b) {
    if (!b) return PD_OK;
    batch_free(b);
    delete b;
    return PD_OK;
}

int pd_batch_count(pd_batch *b, int *n, int *ncell) {
    PD_CHECK(b, PD_EINVAL, "pd_batch_count: null handle");
    if (n) *n = b->n;
    if (ncell) *ncell = b->ncell;
    return PD_OK;
}

int pd_batch_set_lanes(pd_batch *b, int lanes) {
    PD_CHECK(b, PD_EINVAL, "pd_batch_set_lanes: null handle");
    PD_CHECK(lanes == 1 || lanes == 2 || lanes == 4 || lanes == 8, PD_EINVAL, "pd_batch_set_lanes: lanes 1, 2, 4 or 8");
    b->lanes = lanes;
    return PD_OK;
}

int pd_batch_update(pd_batch *b, const float *x, const float *y, const float *z, pd_stream_t sp) {
    PD_CHECK(b && x && y && z, PD_EINVAL, "pd_batch_update: null argument");
    cudaStream_t s = (cudaStream_t)sp;
    const int blocks = batch_blocks(b), items = drift_items(blocks, b->num_sms);
    launch_chained(k_batch_drift<false, false>, (blocks + items - 1) / items, B_THREADS, 0, s,
        b->n, items, const_cast<float *>(x), const_cast<float *>(y), const_cast<float *>(z), nullptr, nullptr, nullptr,
        nullptr, nullptr, nullptr, nullptr, 0.f, b->rep_of, b->reps, b->ref, b->threshold, nullptr, nullptr, b->rep_dmax,
        b->rep_flag, b->nrep, b->st, 0);
    PD_LAUNCHED();
    return batch_rebuild_launch(b, x, y, z, s);
}

int pd_batch_forces(pd_batch *b, const float *x, const float *y, const float *z, float *fx, float *fy, float *fz,
                    float *epot, int energy, pd_stream_t sp) {
    PD_CHECK(b && x && y && z && fx && fy && fz, PD_EINVAL, "pd_batch_forces: null argument");
    PD_CHECK(!energy || epot, PD_EINVAL, "pd_batch_forces: energy needs epot");
    BatchKick kick;
    memset(&kick, 0, sizeof kick);
    return batch_pairs_launch(b, x, y, z, fx, fy, fz, epot, energy, kick, 0, false, (cudaStream_t)sp);
}

int pd_batch_status(pd_batch *b, pd_ell_stats *out) {
    PD_CHECK(b && out, PD_EINVAL, "pd_batch_status: null argument");
    long long h[E_LEN];
    PD_CUDA(cudaMemcpy(h, b->st, sizeof h, cudaMemcpyDeviceToHost));
    memset(out, 0, sizeof *out);
    out->valid = h[E_VALID] != 0;
    out->error = (int)h[E_ERROR];
    out->requested = h[E_REQUEST] != 0;
    out->step = h[E_STEP];
    out->last_build = h[E_LAST_BUILD];
    out->interval = h[E_INTERVAL];
    out->checks = h[E_CHECKS];
    out->builds = h[E_BUILDS];
    out->required = h[E_REQUIRED];
    out->cap = b->cap;
    out->lanes = batch_lanes(b);
    return PD_OK;
}

int pd_batch_bind(pd_batch *b, const pd_md_state *st) {
    PD_CHECK(b && st, PD_EINVAL, "pd_batch_bind: null argument");
    PD_CHECK(st->n == b->n, PD_EINVAL, "pd_batch_bind: state has %d particles, the batch %d", st->n, b->n);
    PD_CHECK(st->x && st->y && st->z && st->vx && st->vy && st->vz && st->fx && st->fy && st->fz && st->inv_mass,
             PD_EINVAL, "pd_batch_bind: state arrays missing (per-particle inverse masses required)");
    b->state = *st;
    b->bound = true;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    return PD_OK;
}

int pd_batch_evaluate(pd_batch *b, int energy, pd_stream_t sp) {
    PD_CHECK(b && b->bound, PD_ESTATE, "pd_batch_evaluate: no state bound");
    const pd_md_state &S = b->state;
    int rc;
    if ((rc = pd_batch_update(b, S.x, S.y, S.z, sp))) return rc;
    PD_CHECK(!energy || S.epot, PD_EINVAL, "pd_batch_evaluate: energy needs epot in the state");
    return pd_batch_forces(b, S.x, S.y, S.z, S.fx, S.fy, S.fz, S.epot, energy, sp);
}

int pd_batch_step(pd_batch *b, int nsteps, float dt, int use_graph, pd_stream_t sp) {
    PD_CHECK(b && b->bound, PD_ESTATE, "pd_batch_step: no state bound");
    PD_CHECK(nsteps >= 0, PD_EINVAL, "pd_batch_step: negative step count");
    cudaStream_t s = (cudaStream_t)sp;
    for (int k = 0; k < nsteps; ++k) {
        if (!use_graph) {
            int rc = batch_enqueue_step(b, dt, s, 0);
            if (rc) return rc;
            continue;
        }
        if (!b->exec || b->exec_dt != dt || b->exec_stream != s || b->exec_lanes != b->lanes ||
            b->exec_chunk != b->mchunk * 8 + b->mtpi) {
            if (b->exec) {
                cudaGraphExecDestroy(b->exec);
                b->exec = nullptr;
            }
            PD_CHECK(s != nullptr, PD_EINVAL, "pd_batch_step: graph replay needs a non-default stream");
            for (int attempt = 0; attempt < 2 && !b->exec; ++attempt) {
                const int cond = b->cond_nodes ? 1 : 0;
                cudaGraph_t g = nullptr;
                PD_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
                const int rc = batch_enqueue_step(b, dt, s, cond);
                cudaError_t err = cudaStreamEndCapture(s, &g);
                // node priorities kept, so the charged batches' mesh branch keeps its streams' high priority
                if (rc == PD_OK && err == cudaSuccess)
                    err = cudaGraphInstantiateWithFlags(&b->exec, g, cudaGraphInstantiateFlagUseNodePriority);
                if (g) cudaGraphDestroy(g);
                if (rc == PD_OK && err == cudaSuccess) break;
                b->exec = nullptr;
                cudaGetLastError();
                if (!cond) {
                    if (rc) return rc;
                    PD_CHECK(false, PD_ECUDA, "batch step capture failed: %s", cudaGetErrorString(err));
                }
                b->cond_nodes = false;
            }
            b->exec_dt = dt;
            b->exec_stream = s;
            b->exec_lanes = b->lanes;
            b->exec_chunk = b->mchunk * 8 + b->mtpi;
        }
        PD_CUDA(cudaGraphLaunch(b->exec, s));
    }
    return PD_OK;
}

int pd_batch_set_coulomb(pd_batch *b, const pd_batch_coulomb *c) {
    PD_CHECK(b && c, PD_EINVAL, "pd_batch_set_coulomb: null argument");
    PD_CHECK(std::isfinite(c->C) && c->C > 0.f && c->rc2 > 0.f && std::isfinite(c->sx) && std::isfinite(c->selfc),
             PD_EINVAL, "pd_batch_set_coulomb: C, rc2, sx and selfc must be finite and C, rc2 positive");
    PD_CHECK(c->ne >= 1 && c->nf >= 1 && c->ne <= BATCH_NP && c->nf <= BATCH_NP, PD_EINVAL,
             "pd_batch_set_coulomb: the polynomials hold 1..%d coefficients", BATCH_NP);
    PD_CHECK(c->rc2 <= b->rl2, PD_EINVAL, "pd_batch_set_coulomb: the Coulomb cutoff exceeds the list radius %g "
             "(create the batch with a van der Waals cutoff covering it)", std::sqrt((double)b->rl2));
    BatchCoul cp{};
    cp.C = c->C;
    cp.rc2 = c->rc2;
    cp.sx = c->sx;
    cp.eshift = c->eshift;
    for (int k = 0; k < c->nf; ++k) cp.pf[k] = c->pf[k];
    for (int k = 0; k < c->ne; ++k) cp.pe[k] = c->pe[k];
    b->cp = cp;
    b->coul_ne = c->ne;
    b->coul_nf = c->nf;
    b->half_c_self = 0.5f * c->C * c->selfc;
    b->coul = true;
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    return PD_OK;
}

// Tiles of the batched meshes: replica r's cell-order positions are [first_r, first_r + N_r) (its
// cells are contiguous in the global cell order), cut into tiles of `chunk` positions; the last
// tile of a replica is padded (slot_src = -1).
static int batch_layout_chunks(pd_batch *b, int chunk) {
    batch_free_chunks(b);
    std::vector<int> crep, src;
    for (int r = 0; r < b->nrep; ++r) {
        const int first = b->first[(size_t)r];
        const int nr = (r + 1 < b->nrep ? b->first[(size_t)r + 1] : b->n) - first;
        const int nc = (nr + chunk - 1) / chunk;
        for (int c = 0; c < nc; ++c) {
            crep.push_back(r);
            for (int p = 0; p < chunk; ++p) {
                const int k = c * chunk + p;
                src.push_back(k < nr ? first + k : -1);
            }
        }
    }
    int rc;
    if ((rc = dalloc(&b->chunk_rep, crep.size())) || (rc = dalloc(&b->slot_src, src.size())) ||
        (rc = dalloc(&b->mid, src.size())) || (rc = dalloc(&b->mq, src.size())))
        return rc;
    PD_CUDA(cudaMemcpy(b->chunk_rep, crep.data(), sizeof(int) * crep.size(), cudaMemcpyHostToDevice));
    PD_CUDA(cudaMemcpy(b->slot_src, src.data(), sizeof(int) * src.size(), cudaMemcpyHostToDevice));
    PD_CUDA(cudaMemset(b->mid, 0xff, sizeof(int) * src.size()));
    PD_CUDA(cudaMemset(b->mq, 0, sizeof(float4) * src.size()));
    b->nchunk = (int)crep.size();   // only a complete layout is used
    b->mchunk = chunk;
    return PD_OK;
}

// One batched cuFFT plan per mesh size, spread over the FFT streams.
static int batch_make_plans(pd_batch *b, int prio_hi) {
    size_t wmax = 0;
    for (auto &g : b->groups) {
        int n[3] = {g.K3, g.K2, g.K1};
        const int K1h = g.K1 / 2 + 1;
        const int nn = g.K1 * g.K2 * g.K3, nm = K1h * g.K2 * g.K3;
        size_t w1 = 0, w2 = 0;
        PD_CHECK(cufftCreate(&g.fwd) == CUFFT_SUCCESS && cufftCreate(&g.bwd) == CUFFT_SUCCESS, PD_ECUFFT,
                 "batched mesh: cufftCreate failed");
        PD_CHECK(cufftSetAutoAllocation(g.fwd, 0) == CUFFT_SUCCESS && cufftSetAutoAllocation(g.bwd, 0) == CUFFT_SUCCESS,
                 PD_ECUFFT, "batched mesh: cufftSetAutoAllocation failed");
        PD_CHECK(cufftMakePlanMany(g.fwd, 3, n, nullptr, 1, nn, nullptr, 1, nm, CUFFT_R2C, g.count, &w1) ==
                         CUFFT_SUCCESS &&
                     cufftMakePlanMany(g.bwd, 3, n, nullptr, 1, nm, nullptr, 1, nn, CUFFT_C2R, g.count, &w2) ==
                         CUFFT_SUCCESS,
                 PD_ECUFFT, "batched mesh: plan of %d meshes %dx%dx%d failed", g.count, g.K1, g.K2, g.K3);
        wmax = std::max(wmax, std::max(w1, w2));
    }
    for (int k = 0; k < pd_batch::NFFT; ++k) {
        PD_CUDA(cudaMalloc(&b->fft_work[k], std::max<size_t>(wmax, 256)));
        PD_CUDA(cudaStreamCreateWithPriority(&b->fft_stream[k], cudaStreamNonBlocking, prio_hi));
        PD_CUDA(cudaEventCreateWithFlags(&b->ev_fft[k], cudaEventDisableTiming));
    }
    PD_CUDA(cudaEventCreateWithFlags(&b->ev_fft_fork, cudaEventDisableTiming));
    for (size_t gi = 0; gi < b->groups.size(); ++gi) {
        auto &g = b->groups[gi];
        void *w = b->fft_work[gi % pd_batch::NFFT];
        PD_CHECK(cufftSetWorkArea(g.fwd, w) == CUFFT_SUCCESS && cufftSetWorkArea(g.bwd, w) == CUFFT_SUCCESS,
                 PD_ECUFFT, "batched mesh: cufftSetWorkArea failed");
    }
    return PD_OK;
}

// Every replica's mesh on this library's transforms, when every mesh's planes fit in shared memory (all or none: one
// replica whose mesh does not leaves the whole batch on the cuFFT groups): the table of meshes and the work of every
// CTA, the replicas' planes largest first.
static int batch_make_transforms(pd_batch *b) {
    std::vector<FftMesh> tab((size_t)b->nrep);
    for (int r = 0; r < b->nrep; ++r) {
        const BMeshRep &R = b->hmreps[(size_t)r];
        const int K[3] = {R.K1, R.K2, R.K3};
        if (fft_route(K, &tab[(size_t)r]) != FFT_PLANES) return PD_OK;
    }
    int rc;
    if ((rc = fft_init())) return rc;
    std::vector<int> lens;
    FftBatch f{};
    std::vector<int> order((size_t)b->nrep);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int p, int q) {
        return (long long)b->hmreps[(size_t)p].K1 * b->hmreps[(size_t)p].K2 >
               (long long)b->hmreps[(size_t)q].K1 * b->hmreps[(size_t)q].K2;
    });
    std::vector<int2> planes[4], cols;
    FftBatch::Class cls[4] = {};
    for (int r : order) {
        const BMeshRep &R = b->hmreps[(size_t)r];
        FftMesh &m = tab[(size_t)r];
        for (int d = 0; d < 3; ++d) {
            const int n = m.ax[d].n;
            size_t k = 0;
            while (k < lens.size() && lens[k] != n) ++k;
            if (k == lens.size()) {
                float2 *w = nullptr;
                if ((rc = fft_twiddles(n, &w))) return rc;
                b->twiddles.push_back(w);
                lens.push_back(n);
            }
            m.ax[d].w = b->twiddles[k];
        }
        m.grid = b->gridA + R.grid;
        m.spec = b->spec + R.modes;
        m.G = b->G + R.modes;
        m.zspec[0] = m.spec;
        m.out[0] = b->gridB + R.grid;
        const int c = fft_plane_class(m);
        cls[c].inplace = c < 3;
        cls[c].threads = std::max(cls[c].threads, fft_plane_threads(m));
        cls[c].smem = std::max(cls[c].smem, fft_plane_smem(m, c < 3));
        f.line_threads = std::max(f.line_threads, fft_line_threads(m.ax[2]));
        f.line_smem = std::max(f.line_smem, fft_line_smem(m.ax[2]));
        for (int z = 0; z < R.K3; ++z) planes[c].push_back(make_int2(r, z));
        for (int k = 0; k < R.K2 * R.K1h; k += FFT_LINES_C) cols.push_back(make_int2(r, k));
    }
    std::vector<int2> all;
    for (int c = 3; c >= 0; --c) {   // the largest planes first
        if (planes[c].empty()) continue;
        cls[c].first = (int)all.size();
        cls[c].count = (int)planes[c].size();
        f.cls[f.nclass++] = cls[c];
        all.insert(all.end(), planes[c].begin(), planes[c].end());
    }
    f.ncols = (int)cols.size();
    if ((rc = dalloc(&b->fft_tab, tab.size())) || (rc = dalloc(&b->fft_planes, all.size())) ||
        (rc = dalloc(&b->fft_cols, cols.size())))
        return rc;
    PD_CUDA(cudaMemcpy(b->fft_tab, tab.data(), sizeof(FftMesh) * tab.size(), cudaMemcpyHostToDevice));
    PD_CUDA(cudaMemcpy(b->fft_planes, all.data(), sizeof(int2) * all.size(), cudaMemcpyHostToDevice));
    PD_CUDA(cudaMemcpy(b->fft_cols, cols.data(), sizeof(int2) * cols.size(), cudaMemcpyHostToDevice));
    f.tab = b->fft_tab;
    f.planes = b->fft_planes;
    f.cols = b->fft_cols;
    b->fft = f;
    return PD_OK;
}

static int batch_set_mesh(pd_batch *b, int kind, int order, double alpha, double C, const int *meshes) {
    const int nrep = b->nrep;
    std::vector<int> idx((size_t)nrep);
    std::iota(idx.begin(), idx.end(), 0);
    auto key = [&](int r) { return std::make_tuple(meshes[3 * r + 2], meshes[3 * r + 1], meshes[3 * r]); };
    std::stable_sort(idx.begin(), idx.end(), [&](int a, int c) { return key(a) < key(c); });
    b->hmreps.assign((size_t)nrep, BMeshRep{});
    long long grid = 0, modes = 0;
    for (size_t a = 0; a < idx.size();) {
        size_t e = a;
        while (e < idx.size() && key(idx[e]) == key(idx[a])) ++e;
        const int r0 = idx[a];
        pd_batch::FftGroup g{};
        g.K1 = meshes[3 * r0];
        g.K2 = meshes[3 * r0 + 1];
        g.K3 = meshes[3 * r0 + 2];
        g.count = (int)(e - a);
        grid = (grid + 63) & ~63ll;     // each group starts on a 256-byte boundary
        modes = (modes + 31) & ~31ll;
        g.grid = grid;
        g.modes = modes;
        const int K1h = g.K1 / 2 + 1;
        const long long nn = (long long)g.K1 * g.K2 * g.K3, nm = (long long)K1h * g.K2 * g.K3;
        for (size_t j = a; j < e; ++j) {
            const int r = idx[j];
            BMeshRep &R = b->hmreps[(size_t)r];
            R.K1 = g.K1;
            R.K2 = g.K2;
            R.K3 = g.K3;
            R.K1h = K1h;
            R.Lx = b->hreps[(size_t)r].L[0];
            R.Ly = b->hreps[(size_t)r].L[1];
            R.Lz = b->hreps[(size_t)r].L[2];
            R.nmodes = (int)nm;
            R.grid = grid;
            R.modes = modes;
            grid += nn;
            modes += nm;
        }
        g.fwd = g.bwd = 0;
        b->groups.push_back(g);
        a = e;
    }
    b->total_nodes = grid;
    b->total_modes = modes;
    PD_CHECK(2 * modes >= grid, PD_EINVAL, "batched mesh: the modes do not cover the grids");
    int rc;
    if ((rc = dalloc(&b->gridA, (size_t)grid)) || (rc = dalloc(&b->gridB, (size_t)grid)) ||
        (rc = dalloc(&b->spec, (size_t)modes)) || (rc = dalloc(&b->G, (size_t)modes)) ||
        (rc = dalloc(&b->mreps, (size_t)nrep)))
        return rc;
    PD_CUDA(cudaMemset(b->gridA, 0, sizeof(float) * (size_t)grid));
    PD_CUDA(cudaMemset(b->gridB, 0, sizeof(float) * (size_t)grid));
    PD_CUDA(cudaMemset(b->spec, 0, sizeof(float2) * (size_t)modes));
    PD_CUDA(cudaMemset(b->G, 0, sizeof(float) * (size_t)modes));
    PD_CUDA(cudaMemcpy(b->mreps, b->hmreps.data(), sizeof(BMeshRep) * nrep, cudaMemcpyHostToDevice));
    // every replica's influence function from the single-system mesh setup (FP64, Influence.jl)
    for (int r = 0; r < nrep; ++r) {
        const BMeshRep &R = b->hmreps[(size_t)r];
        pd_mesh_params mp;
        memset(&mp, 0, sizeof mp);
        mp.kind = kind;
        mp.order = order;
        mp.alias_order = 2;
        mp.mesh[0] = R.K1;
        mp.mesh[1] = R.K2;
        mp.mesh[2] = R.K3;
        mp.alpha = alpha;
        mp.C = C;
        const int first = b->first[(size_t)r];
        mp.nmax = std::max(1, (r + 1 < nrep ? b->first[(size_t)r + 1] : b->n) - first);
        pd_mesh *m = nullptr;
        if ((rc = pd_mesh_create(&m, &mp, &b->box[3 * (size_t)r]))) return rc;
        cudaError_t err = cudaDeviceSynchronize();
        if (err == cudaSuccess)
            err = cudaMemcpy(b->G + R.modes, m->G, sizeof(float) * (size_t)R.nmodes, cudaMemcpyDeviceToDevice);
        pd_mesh_destroy(m);
        PD_CHECK(err == cudaSuccess, PD_ECUDA, "batched mesh: influence copy failed: %s", cudaGetErrorString(err));
    }
    // the mesh branch is the longer of the two branches of the force pass: its streams get the high
    // priority, so its kernels' blocks are scheduled ahead of the pair kernel's
    int prio_lo = 0, prio_hi = 0;
    cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi);
    if ((rc = batch_make_transforms(b))) return rc;
    if (!b->fft.tab && (rc = batch_make_plans(b, prio_hi))) return rc;
    PD_CUDA(cudaStreamCreateWithPriority(&b->mesh_stream, cudaStreamNonBlocking, prio_hi));
    PD_CUDA(cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming));
    PD_CUDA(cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming));
    if ((rc = batch_layout_chunks(b, b->mchunk))) return rc;
    b->morder = order;
    b->mesh = true;
    return PD_OK;
}

int pd_batch_set_mesh(pd_batch *b, int kind, int order, double alpha, double C, const int *meshes) {
    PD_CHECK(b && meshes, PD_EINVAL, "pd_batch_set_mesh: null argument");
    PD_CHECK(b->coul, PD_ESTATE, "pd_batch_set_mesh: set the real-space Coulomb terms first (pd_batch_set_coulomb)");
    PD_CHECK(kind == PD_MESH_SPME || kind == PD_MESH_P3M_AD, PD_ENOTSUP,
             "pd_batch_set_mesh: batched meshes take SPME or P3M-AD (analytic differentiation)");
    PD_CHECK(order >= 4 && order <= 6, PD_ENOTSUP, "pd_batch_set_mesh: batched meshes take orders 4, 5 and 6");
    PD_CHECK(std::isfinite(alpha) && alpha > 0 && std::isfinite(C) && C > 0, PD_EINVAL,
             "pd_batch_set_mesh: alpha and C must be finite and positive");
    for (int r = 0; r < b->nrep; ++r)
        for (int d = 0; d < 3; ++d)
            PD_CHECK(meshes[3 * r + d] >= order && meshes[3 * r + d] <= 1024, PD_EINVAL,
                     "pd_batch_set_mesh: replica %d mesh dimension %d is %d (order %d .. 1024)", r, d,
                     meshes[3 * r + d], order);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
    batch_free_mesh(b);
    const int rc = batch_set_mesh(b, kind, order, alpha, C, meshes);
    if (rc != PD_OK) batch_free_mesh(b);
    return rc;
}

int pd_batch_set_spread_tile(pd_batch *b, int chunk, int threads_per_ion) {
    PD_CHECK(b, PD_EINVAL, "pd_batch_set_spread_tile: null handle");
    PD_CHECK(chunk == 32 || chunk == 64, PD_EINVAL, "pd_batch_set_spread_tile: 32 or 64 particles per tile");
    PD_CHECK(threads_per_ion == 2 || (threads_per_ion == 4 && chunk == 64), PD_EINVAL,
             "pd_batch_set_spread_tile: 2 threads per ion, or 4 with tiles of 64");
    b->mtpi = threads_per_ion;
    if (!b->mesh) {
        b->mchunk = chunk;
        return PD_OK;
    }
    if (chunk == b->mchunk) return PD_OK;
    const int rc = batch_layout_chunks(b, chunk);
    if (rc != PD_OK) batch_free_mesh(b);   // a batch without its tiles takes no charged step (PD_ESTATE)
    return rc;
}

int pd_batch_mesh_info(pd_batch *b, int *groups, long long *nodes, long long *modes, int *chunk, int *nchunk) {
    PD_CHECK(b, PD_EINVAL, "pd_batch_mesh_info: null handle");
    if (groups) *groups = (int)b->groups.size();
    if (nodes) *nodes = b->total_nodes;
    if (modes) *modes = b->total_modes;
    if (chunk) *chunk = b->mchunk;
    if (nchunk) *nchunk = b->nchunk;
    return PD_OK;
}

int pd_batch_rows(pd_batch *b, int **rows, int **counts, int **order) {
    PD_CHECK(b && rows && counts, PD_EINVAL, "pd_batch_rows: null argument");
    if (!b->xrows) {   // from now on every rebuild refreshes them: a captured step is captured again
        const int rc = dalloc(&b->xrows, (size_t)b->n * b->cap);
        if (rc) return rc;
        PD_CUDA(cudaMemset(b->xrows, 0xff, sizeof(int) * (size_t)b->n * b->cap));
        PD_CUDA(cudaDeviceSynchronize());   // a build may be in flight on another stream
        k_batch_export<<<(b->n + B_THREADS - 1) / B_THREADS, B_THREADS>>>(b->rows, b->counts, b->n, b->cap, b->xrows);
        PD_LAUNCHED();
        PD_CUDA(cudaDeviceSynchronize());
        if (b->exec) cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    *rows = b->xrows;
    *counts = b->counts;
    if (order) *order = b->sorted;
    return PD_OK;
}

}  // extern "C"
