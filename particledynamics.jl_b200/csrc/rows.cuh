// Neighbour rows in cell order, shared by the ELL route (ell.cu), the batched replicas (batch.cu) and the
// learned descriptors (learned.cu): the build of one cell's rows and the walk over a row.
//
// Particles are taken in cell order: position k holds particle sorted[k], its packed record is xq[k], and a
// row's entries are positions, so the records of a row's neighbours sit in a few runs of adjacent cells.
// Dense cells (ROWS_MIN_PER_CELL particles or more on average) keep a row's entries together (entry t of
// position k at k cap + t): the build appends 32 tested candidates with one coalesced store, and eight or more
// lanes walk a row through full 32-byte sectors.  Sparse cells keep the slot-major layout (t n + k) with one
// thread per row.
#pragma once

#include "common.cuh"
#include "ell_common.cuh"
#include "packed2.cuh"

namespace pdb {

constexpr int ROWS_WARPS = 4, ROWS_CAP = 512;   // 32 KB of staging per block: six blocks share an SM
constexpr int ROWS_BLOCKS = 6;
constexpr int ROWS_MIN_PER_CELL = 8;            // mean cell occupancy from which the cell-staged build is used
constexpr int ROWS_GROUP = 4;                   // particles tested against each staged candidate register

// One cell grid: its box, cells per axis and first global cell.
struct RowGrid {
    float L[3];
    int nx, ny, nz, base;
};

// Rows of the particles of local cell c (part `split` of `nsplit`), by one warp.
//
// The warp walks the stencil (z, then y offsets; x cells in range order; each cell's particles in id order,
// _kernel_neighbors3g!, DeviceNeighborCUDA.jl:510-559), stages the candidates near the bounding box of up to 32
// of the cell's particles in shared memory, and tests 32 candidates at a time (one per lane) against
// ROWS_GROUP particles: the accepted ones are appended in visiting order by ballot.  Bound by the issue of the
// tests (12 instructions per 32 candidates and particle); a lane-per-particle scan of the same stage left the
// lanes beyond the cell's particles idle and scattered its row stores (1 048 576 LJ atoms, 19 per cell: 3.34 ms
// per build, now 0.56).  Without WRAP no pair of the
// stencil crosses a periodic face: the nearest-image shift is the identity.
template <int D, bool WRAP>
__device__ __forceinline__ void rows_test(const RowGrid &g, float4 *sw, int fill, int np, float xi, float yi, float zi,
                                          int k0, float rl2, int cap, int *__restrict__ rows, int &found) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const float Lx = g.L[0], Ly = g.L[1], Lz = g.L[2], hLx = 0.5f * Lx, hLy = 0.5f * Ly, hLz = 0.5f * Lz;
    const int padded = (fill + 31) & ~31;
    if (fill + lane < padded) sw[fill + lane] = make_float4(1e30f, 1e30f, 1e30f, __int_as_float(-1));   // never near
    __syncwarp();
    for (int m0 = 0; m0 < np; m0 += ROWS_GROUP) {
        float px[ROWS_GROUP], py[ROWS_GROUP], pz[ROWS_GROUP];
        int base[ROWS_GROUP];
        int *row[ROWS_GROUP];
#pragma unroll
        for (int m = 0; m < ROWS_GROUP; ++m) {
            row[m] = rows + (size_t)(k0 + m0 + m) * cap;
            const int src = (m0 + m) & 31;
            px[m] = __shfl_sync(0xffffffffu, xi, src);
            py[m] = __shfl_sync(0xffffffffu, yi, src);
            pz[m] = __shfl_sync(0xffffffffu, zi, src);
            base[m] = __shfl_sync(0xffffffffu, found, src);
            if (m0 + m >= np) px[m] = -3e30f;   // past the group: no candidate is near
        }
        for (int t = lane; t < padded; t += 32) {
            const float4 cj = sw[t];
            const int kc = __float_as_int(cj.w);
#pragma unroll
            for (int m = 0; m < ROWS_GROUP; ++m) {
                float dx = cj.x - px[m], dy = cj.y - py[m], dz = D == 3 ? cj.z - pz[m] : 0.f;
                if (WRAP) {
                    dx = mic_fast(dx, hLx, Lx);
                    dy = mic_fast(dy, hLy, Ly);
                    if (D == 3) dz = mic_fast(dz, hLz, Lz);
                }
                const float r2 = D == 3 ? fmaf(dx, dx, fmaf(dy, dy, dz * dz)) : fmaf(dx, dx, dy * dy);
                const int k = k0 + m0 + m;
                const bool hit = r2 <= rl2 && kc != k;
                const unsigned bal = __ballot_sync(0xffffffffu, hit);
                const int at = base[m] + __popc(bal & lt);
                if (hit && at < cap) row[m][at] = kc;
                base[m] += __popc(bal);
            }
        }
#pragma unroll
        for (int m = 0; m < ROWS_GROUP; ++m)
            if (lane == m0 + m) found = base[m];
    }
    __syncwarp();
}

template <int D>
__device__ __forceinline__ unsigned cell_rows(const RowGrid &g, int c, int split, int nsplit,
                                              const float4 *__restrict__ xq, const int *__restrict__ sorted,
                                              const int *__restrict__ cell_off, float rl2, int cap,
                                              int *__restrict__ rows, int *__restrict__ counts,
                                              float4 *__restrict__ ref, float4 *sw) {
    const int lane = threadIdx.x & 31;
    const float Lx = g.L[0], Ly = g.L[1], Lz = g.L[2], hLx = 0.5f * Lx, hLy = 0.5f * Ly, hLz = 0.5f * Lz;
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const float rl = sqrtf(rl2);
    const float hx = Lx / (float)nx, hy = Ly / (float)ny, hz = Lz / (float)nz;
    const int Sx = ell_reach(rl, Lx, nx), Sy = ell_reach(rl, Ly, ny), Sz = D == 3 ? ell_reach(rl, Lz, nz) : 0;
    const int cx = c % nx, tmp = c / nx, cy = tmp % ny, cz = tmp / ny;
    // the stencil crosses no face, and its two ends (S + 1 cells apart) lie within half a box
    const bool nowrap = cx >= Sx && cx + Sx < nx && 2 * (Sx + 1) < nx && cy >= Sy && cy + Sy < ny &&
                        2 * (Sy + 1) < ny && (D == 2 || (cz >= Sz && cz + Sz < nz && 2 * (Sz + 1) < nz));
    const int pa = cell_off[g.base + c], pall = cell_off[g.base + c + 1] - pa;
    const int p0 = pa + pall * split / nsplit, pn = pa + pall * (split + 1) / nsplit - p0;
    unsigned fmax = 0;
    for (int pg = 0; pg < pn; pg += 32) {
        const int np = min(32, pn - pg), kp = p0 + pg + lane;
        const bool has = lane < np;
        const float4 me = has ? xq[kp] : make_float4(0.f, 0.f, 0.f, 0.f);
        // bounding box of the group: a candidate farther than the list radius from the box is farther from
        // every particle of the group and is not staged (a conservative margin keeps rounding from dropping
        // a candidate that the exact test accepts)
        float bl[3] = {has ? me.x : INFINITY, has ? me.y : INFINITY, has ? me.z : INFINITY};
        float bh[3] = {has ? me.x : -INFINITY, has ? me.y : -INFINITY, has ? me.z : -INFINITY};
#pragma unroll
        for (int d = 0; d < 3; ++d) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                bl[d] = fminf(bl[d], __shfl_xor_sync(0xffffffffu, bl[d], off));
                bh[d] = fmaxf(bh[d], __shfl_xor_sync(0xffffffffu, bh[d], off));
            }
        }
        const float bcx = 0.5f * (bl[0] + bh[0]), bcy = 0.5f * (bl[1] + bh[1]), bcz = 0.5f * (bl[2] + bh[2]);
        const float bhx = 0.5f * (bh[0] - bl[0]), bhy = 0.5f * (bh[1] - bl[1]), bhz = 0.5f * (bh[2] - bl[2]);
        const float rbox = rl * 1.0001f + 1e-3f, rbox2 = rbox * rbox;
        int found = 0, fill = 0;
        auto scan = [&]() {
            if (nowrap) rows_test<D, false>(g, sw, fill, np, me.x, me.y, me.z, p0 + pg, rl2, cap, rows, found);
            else rows_test<D, true>(g, sw, fill, np, me.x, me.y, me.z, p0 + pg, rl2, cap, rows, found);
            fill = 0;
        };
        // The stencil's runs of candidates (positions [ka, kb), two per (oz, oy) row at the periodic seam) are
        // looked up at once, lane 2 r + part holding one run, and then walked as one sequence: a lane's candidate
        // needs no load that waits for another run's.
        const int nrow = (2 * Sz + 1) * (2 * Sy + 1);
        for (int r0 = 0; r0 < nrow; r0 += 16) {
            int ka = 0, len = 0;
            const int r = r0 + (lane >> 1);
            if (r < nrow) {
                const int oz = r / (2 * Sy + 1) - Sz, oy = r % (2 * Sy + 1) - Sy;
                int cz2 = cz + oz, cy2 = cy + oy;
                cz2 -= cz2 >= nz ? nz : 0;
                cz2 += cz2 < 0 ? nz : 0;
                cy2 -= cy2 >= ny ? ny : 0;
                cy2 += cy2 < 0 ? ny : 0;
                const float gz = (float)max(abs(oz) - 1, 0) * hz, gy = (float)max(abs(oy) - 1, 0) * hy;
                const float g2 = fmaf(gy, gy, gz * gz);
                if (g2 <= rl2) {
                    int a1, b1, a2, b2;
                    ell_row_ranges(cx, g2, rl2, hx, Sx, nx, a1, b1, a2, b2);
                    const bool second = lane & 1;
                    if (!second || a2 <= b2) {
                        const int *off = cell_off + g.base + (cz2 * ny + cy2) * nx;
                        ka = off[second ? a2 : a1];
                        len = off[(second ? b2 : b1) + 1] - ka;
                    }
                }
            }
            int end = len;   // inclusive prefix over the runs
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += y;
            }
            const int total = __shfl_sync(0xffffffffu, end, 31);
            const int shift = ka - (end - len);   // candidate c of this run sits at position c + shift
            auto position = [&](int c) {          // of candidate c (c < total): the first run ending past it
                int run = 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const int e = __shfl_sync(0xffffffffu, end, run + o - 1);
                    run += c >= e ? o : 0;
                }
                return c + __shfl_sync(0xffffffffu, shift, run);
            };
            int kn = position(min(lane, max(total - 1, 0)));
            float4 vn = lane < total ? xq[kn] : make_float4(0.f, 0.f, 0.f, 0.f);
            for (int c0 = 0; c0 < total; c0 += 32) {
                const bool in = c0 + lane < total;
                float4 v = vn;
                const int kc = kn;
                if (c0 + 32 < total) {   // the next 32 candidates are in flight while these are tested
                    kn = position(min(c0 + 32 + lane, total - 1));
                    vn = xq[kn];
                }
                const float ex = fmaxf(fabsf(mic_fast(v.x - bcx, hLx, Lx)) - bhx, 0.f);
                const float ey = fmaxf(fabsf(mic_fast(v.y - bcy, hLy, Ly)) - bhy, 0.f);
                const float ez = D == 3 ? fmaxf(fabsf(mic_fast(v.z - bcz, hLz, Lz)) - bhz, 0.f) : 0.f;
                const bool keep = in && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= rbox2;
                const unsigned bal = __ballot_sync(0xffffffffu, keep);
                const int nk = __popc(bal);
                if (fill + nk > ROWS_CAP) scan();
                if (keep) {   // staged in the candidates' order
                    v.w = __int_as_float(kc);
                    sw[fill + __popc(bal & ((1u << lane) - 1u))] = v;
                }
                fill += nk;
            }
        }
        scan();
        if (has) {
            counts[kp] = found;
            ref[sorted[kp]] = make_float4(me.x, me.y, me.z, 0.f);
        }
        fmax = max(fmax, (unsigned)found);
    }
    return fmax;
}

// End of a row build, run by the last block: the largest row against the capacity
// (_device_commit_kernel!, DeviceNeighborCUDA.jl:345-404).
__device__ __forceinline__ void rows_commit(long long *st, int cap) {
    const long long largest = st[E_RMAX];
    st[E_RMAX] = 0;
    st[E_TICKET_R] = 0;
    st[E_REQUIRED] = largest;
    if (largest > cap) {
        st[E_ERROR] = E_ERR_CAPACITY;
        st[E_VALID] = 0;
    } else {
        st[E_VALID] = 1;
        st[E_LAST_BUILD] = st[E_STEP];
        st[E_BUILDS] += 1;
    }
}

// The row of position k walked by G lanes: entry t at row[t * stride] (UNIT: stride 1), lane's entries lane,
// lane + G, ...; f(pa, pb) runs for two records at a time (packed arithmetic).  Four entries' records and the next
// four's indices are in flight while two are evaluated; past the row's end a record is k's own, which f drops as
// a pair at distance zero.
template <int G, bool UNIT, typename F>
__device__ __forceinline__ void walk_row(const int *__restrict__ row, size_t stride, int lane, int cnt, int k,
                                         const float4 *__restrict__ xq, F &&f) {
    const int *at = row + (UNIT ? (size_t)lane : (size_t)lane * stride);
    const size_t step = UNIT ? (size_t)G : G * stride;
    int j[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) j[u] = lane + u * G < cnt ? __ldg(at + u * step) : k;
    for (int t = lane; t < cnt; t += 4 * G) {
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = __ldg(xq + j[u]);
        at += 4 * step;
#pragma unroll
        for (int u = 0; u < 4; ++u) j[u] = t + (4 + u) * G < cnt ? __ldg(at + u * step) : k;
        f(p[0], p[1]);
        if (t + 2 * G < cnt) f(p[2], p[3]);
    }
}

// Nearest-image differences of pi and pj.  WRAP: the compensated periodic difference, taken only where a
// difference exceeds half a box; without it the plain differences, which are the same values when pi keeps
// farther than the cutoff from every face: a pair that the box would wrap is then beyond the cutoff both ways.
template <int D, bool WRAP>
__device__ __forceinline__ void pair_delta(const float4 &pi, const float4 &pj, const float *L, float &dx, float &dy,
                                           float &dz) {
    dx = __fsub_rn(pi.x, pj.x);
    dy = __fsub_rn(pi.y, pj.y);
    dz = D == 3 ? __fsub_rn(pi.z, pj.z) : 0.f;
    if (WRAP) {
        const float hx = 0.5f * L[0], hy = 0.5f * L[1], hz = 0.5f * L[2];
        if (fabsf(dx) > hx || fabsf(dy) > hy || (D == 3 && fabsf(dz) > hz)) {
            dx = periodic_delta(pi.x, pj.x, hx, L[0]);
            dy = periodic_delta(pi.y, pj.y, hy, L[1]);
            if (D == 3) dz = periodic_delta(pi.z, pj.z, hz, L[2]);
        }
    }
}

// True when no pair of pi within rc can cross a periodic face.
template <int D>
__device__ __forceinline__ bool clear_of_faces(const float4 &pi, const float *L, float rc) {
    return fabsf(pi.x) + rc < 0.5f * L[0] && fabsf(pi.y) + rc < 0.5f * L[1] &&
           (D == 2 || fabsf(pi.z) + rc < 0.5f * L[2]);
}

// One row's LJ / WCA sums of two neighbours at a time: f/r = 24 eps (2 s12 - s6) / r^2 and u = 4 eps (s12 - s6) + eoff
// inside (0, rc2), which the caller tests.
struct LjRow {
    f2 sig2, eps24, eps4, eoff, two, minus1;
    float rc2;
};
__device__ __forceinline__ LjRow lj_row(float eps, float sig2, float rc2, float eoff) {
    LjRow r;
    r.sig2 = pk(sig2);
    r.eps24 = pk(24.f * eps);
    r.eps4 = pk(4.f * eps);
    r.eoff = pk(eoff);
    r.two = pk(2.f);
    r.minus1 = pk(-1.f);
    r.rc2 = rc2;
    return r;
}
template <bool ENERGY>
__device__ __forceinline__ void lj_two(const LjRow &m, f2 ir2, f2 &fr, f2 &u) {
    const f2 s2 = mul2(m.sig2, ir2);
    const f2 s6 = mul2(mul2(s2, s2), s2);
    const f2 s12 = mul2(s6, s6);
    const f2 ns6 = mul2(m.minus1, s6);
    fr = mul2(mul2(m.eps24, fma2(m.two, s12, ns6)), ir2);
    if (ENERGY) u = fma2(m.eps4, add2(s12, ns6), m.eoff);
}

}  // namespace pdb
