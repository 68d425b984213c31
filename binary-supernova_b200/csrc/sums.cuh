// sums.cuh -- the reductions of the driver's scalar results: compensated
// (double-double) grid sums, their block-parallel fixed-order merge, and the
// accrete! sums (src/sinks.jl:74-109) in the reference's sequential order.
#pragma once

#include "stage_f64.cuh"

namespace bsn {
namespace sums {

// two-sum compensated accumulator
struct DD { double hi, lo; };
__device__ __forceinline__ void dd_add(DD& s, double x) {
    double t = s.hi + x;
    double bp = t - s.hi;
    double e = (s.hi - (t - bp)) + (x - bp);
    s.hi = t;
    s.lo += e;
}
__device__ __forceinline__ DD dd_merge(DD a, DD b) {
    DD s = a;
    dd_add(s, b.hi);
    s.lo += b.lo;
    return s;
}

// Merge nblocks partial DD triples part[6 b + 2 d], part[6 b + 2 d + 1]
// (d = 0..2) with all NT threads of one block in a fixed order (thread t takes
// b = t, t + NT, ...; then a fixed shuffle tree and the warps in order), so
// the result does not depend on scheduling.  Thread 0 gets the merged pairs.
template <int NT>
__device__ void merge_partials3_pairs(const double* part, int nblocks, DD out[3]) {
    static_assert(NT % 32 == 0 && NT <= 1024, "block of whole warps");
    DD s[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (int b = threadIdx.x; b < nblocks; b += NT)
        for (int d = 0; d < 3; ++d) s[d] = dd_merge(s[d], DD{part[6 * b + 2 * d], part[6 * b + 2 * d + 1]});
    __shared__ DD red[3][NT / 32];
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            DD other = {__shfl_xor_sync(0xffffffffu, s[d].hi, o), __shfl_xor_sync(0xffffffffu, s[d].lo, o)};
            s[d] = dd_merge(s[d], other);
        }
        if ((threadIdx.x & 31) == 0) red[d][threadIdx.x >> 5] = s[d];
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) {
            DD acc = red[d][0];
            for (int w = 1; w < NT / 32; ++w) acc = dd_merge(acc, red[d][w]);
            out[d] = acc;
        }
}

// As merge_partials3_pairs; thread 0 gets out[d] = hi + lo.
template <int NT>
__device__ void merge_partials3(const double* part, int nblocks, double out[3]) {
    DD s[3];
    merge_partials3_pairs<NT>(part, nblocks, s);
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) out[d] = s[d].hi + s[d].lo;
}

// As merge_partials3_pairs; thread 0 gets out[2 d] = hi, out[2 d + 1] = lo.
template <int NT>
__device__ void merge_partials3_dd(const double* part, int nblocks, double out[6]) {
    DD s[3];
    merge_partials3_pairs<NT>(part, nblocks, s);
    if (threadIdx.x == 0)
        for (int d = 0; d < 3; ++d) { out[2 * d] = s[d].hi; out[2 * d + 1] = s[d].lo; }
}

// accrete! sums over the active-index box [ilo,ihi] x [jlo,jhi] x [klo,khi]:
// cells with |x - p| < rs and rho > rho_min add rho * rate (and m * rate).
// The block evaluates the cells in parallel, 4 NT at a time (four neighbours
// per thread), keeps the terms of those that add one in the reference's
// (k, j, i) order by a prefix sum, and four threads, one per sum, add them in
// that order.  A cell that adds nothing is left out: the sums are sequential,
// and only about a third of the box lies in the sphere.  Thread 0 gets
// out = {dm, dPx, dPy, dPz}.  (4 cells of sink radius: 43 us when one thread
// added every cell's four terms, zeros included.)
template <int NT>
__device__ void sink_sums(const double* U, int nx, int ny, int nz, double dx, double dy, double dz, double x0,
                          double y0, double z0, double px, double py, double pz, double rs, double rate,
                          double rho_min, int ilo, int ihi, int jlo, int jhi, int klo, int khi, double out[4]) {
    constexpr int CH = 4 * NT;
    __shared__ double term[4][CH];
    __shared__ int wsum[NT / 32];
    __shared__ double total4[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nI = ihi - ilo + 1, nJ = jhi - jlo + 1, nK = khi - klo + 1;
    const long long total = (nI > 0 && nJ > 0 && nK > 0) ? nI * nJ * nK : 0;
    Geom G(nx, ny, nz);
    double acc = 0.0;   // threads 0, 32, 64, 96: one sum each
    for (long long base = 0; base < total; base += CH) {
        double v[4][4];
        int n = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const long long t = base + 4 * (long long)threadIdx.x + e;
            if (t >= total) continue;
            int a = ilo + (int)(t % nI);
            long long rr = t / nI;
            int b = jlo + (int)(rr % nJ), c = klo + (int)(rr / nJ);
            double xc, yc, zc;
            f64::cell_xyz(a, b, c, x0, y0, z0, dx, dy, dz, xc, yc, zc);
            double r = sqrt(sq(xc - px) + sq(yc - py) + sq(zc - pz));
            if (r >= rs) continue;
            long long o = G.act(a, b, c);
            if (U[o] <= rho_min) continue;
            const double w[4] = {U[o] * rate, U[o + 1] * rate, U[o + 2] * rate, U[o + 3] * rate};
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == n) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[i][q] = w[q];
                }
            ++n;
        }
        int incl = n;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int at = incl - n, m = 0;
        for (int w = 0; w < NT / 32; ++w) {
            if (w < warp) at += wsum[w];
            m += wsum[w];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < n) {
#pragma unroll
                for (int q = 0; q < 4; ++q) term[q][at + i] = v[i][q];
            }
        __syncthreads();
        if (lane == 0 && warp < 4) {
            const double* tq = term[warp];
#pragma unroll 8
            for (int e = 0; e < m; ++e) acc += tq[e];
        }
        __syncthreads();
    }
    if (lane == 0 && warp < 4) total4[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int q = 0; q < 4; ++q) out[q] = total4[q];
}

}  // namespace sums
}  // namespace bsn
