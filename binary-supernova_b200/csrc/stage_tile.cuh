// stage_tile.cuh -- the fused RK3-stage kernel as a template over the stencil
// physics and the tile shape (chosen by the autotuner).  Included by the units
// that instantiate it: stage_f64_lo.cu and stage_f64_hi.cu (FP64 physics, no
// contraction), stage_fast.cu and stage_guarded.cu (FP32 stencils) and
// learned.cu (learned weights), the last three with approximate division and
// square root and every multiply-add written out.
//
// A CTA owns a TX x TY x TZ block of active cells.  It stages the block and
// the 3-cell halos of all three sweeps in shared memory once (SoA; floors
// applied in FP64 to active cells, ghost cells taken raw through the boundary
// map or from a ghost buffer, the cell pressure computed once per staged
// cell), computes every interface of the block once, a sweep at a time, and
// accumulates the flux divergence of its cells in FP64 registers.  The epilogue adds the
// source terms in the driver's order (BH gravity, self-gravity, sinks), the
// SSP-RK3 combine and the floors in FP64, stores the stage result and folds
// the next CFL speed into a device-wide max.
#pragma once

#include "stage_f64.cuh"
#include "tma.cuh"

namespace bsn {
namespace tile {

template <int TX, int TY, int TZ>
struct Shape {
    static constexpr int T[3] = {TX, TY, TZ};
    static constexpr int NCELL = TX * TY * TZ;
    static constexpr int FC0 = (TX + 1) * TY * TZ, FC1 = TX * (TY + 1) * TZ, FC2 = TX * TY * (TZ + 1);
    static constexpr int NFACE = FC0 > FC1 ? (FC0 > FC2 ? FC0 : FC2) : (FC1 > FC2 ? FC1 : FC2);
    // "cross" staging (all three sweeps from one staged region): the block,
    // then the 3-cell halos below/above it along x, y and z
    static constexpr int HX = 3 * TY * TZ, HY = 3 * TX * TZ, HZ = 3 * TX * TY;
    static constexpr int OXL = NCELL, OXH = OXL + HX, OYL = OXH + HX, OYH = OYL + HY, OZL = OYH + HY, OZH = OZL + HZ;
    static constexpr int NCROSS = OZH + HZ;
};

// Staged columns.  The stencils read rho, m_x, m_y, m_z and the cell pressure
// (c[s][0..3] and c[s][5]); E (c[s][4]) is staged only by policies whose
// epilogue reads the block's state back from shared memory (kCols = 6: E at
// column 4, P at 5).  With kCols = 5 the pressure sits in column 4.
template <int COLS>
__host__ __device__ constexpr int pcol() { return COLS - 1; }

// Physics policies --------------------------------------------------------
struct F64Physics {
    using real = double;
    static constexpr bool kDeferred = true;         // faces outside the ordinary range go to a second pass
    static constexpr bool kCenterFromSmem = true;   // smem holds the floored FP64 state
    static constexpr int kCols = 6;                 // staged columns: rho, m, E (read back by the epilogue), P
    static constexpr bool kWarpFaces = false;       // faces computed thread by thread
    static constexpr bool kQuiescentSkip = false;
    static constexpr bool kScreen = false;          // screening launch of a split stage
    __device__ static bool same(double, double) { return true; }
    static constexpr int kExtraSmem(int) { return 0; }
    __device__ static void prologue(unsigned char*, const f64::StageArgs&, int) {}
    static constexpr bool kOrdinary = true;         // faces of ordinary tiles take the shared-reciprocal code
    struct Consts { double g, gm1, igm1, gg; bool ord; };
    __device__ static Consts consts(const f64::StageArgs& A) {
        return {A.g, A.gm1, A.igm1, A.gg, f64::ordinary_gamma(A.gm1)};
    }
    // apply_floors (src/gpu_kernels.jl:26-46) on one cell, as the reference
    __device__ static void floor(double (&v)[5], const f64::StageArgs& A) {
        double P;
        f64::floor_and_pressure(v, true, A.rho_floor, A.P_floor, A.Pfl_gm1, A.gm1, &P);
    }
    // a staged cell: floors on active cells, the staged copy and its
    // pressure; whether it is ordinary (physics.cuh)
    __device__ static bool stage(double (&v)[5], bool act, const f64::StageArgs& A, const Consts& k, double (&w)[5],
                                 double& P) {
        const bool ord = f64::floor_and_pressure(v, act, A.rho_floor, A.P_floor, A.Pfl_gm1, A.gm1, &P);
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = v[q];
        return ord;
    }
    // true: the face is deferred (face_flux_f64 takes it)
    __device__ __forceinline__ static bool flux(const double (&c)[6][6], const Consts& k, int D, double F[5]) {
        return !k.ord || f64::interface_flux_ord(c, k.g, k.gm1, k.igm1, k.gg, D, F);
    }
};

// F32Physics (the fast path's policy) lives in stage_fast.cu.

__device__ __forceinline__ void load_cell(const f64::StageArgs& A, const Geom& G, int d, int a, int b, int c,
                                          double v[5], bool& active) {
    int n[3] = {G.nx, G.ny, G.nz};
    int p[3] = {a, b, c};
#pragma unroll
    for (int t = 0; t < 3; ++t)
        if (t != d) p[t] = p[t] < n[t] ? p[t] : n[t] - 1;   // partial tile: clamp (value unused)
    int pd = p[d];
    active = (pd >= 0 && pd < n[d]);
    const double* src = A.Uin;
    if (!active) {
        if (A.Gh) {
            pd = pd < -BSN_NG ? -BSN_NG : (pd > n[d] + BSN_NG - 1 ? n[d] + BSN_NG - 1 : pd);
            p[d] = pd;
            src = A.Gh;
        } else {
            p[d] = bc_map(pd, n[d], A.bc);
        }
    }
    long long off = G.act(p[0], p[1], p[2]);
#pragma unroll
    for (int q = 0; q < 5; ++q) v[q] = src[off + q];
}

// Staged values of the cross region at entry e, from active
// coordinates (a, b, c) and the axis the cell may leave the grid along.
template <int TX, int TY, int TZ>
__device__ __forceinline__ void cross_cell(int e, int a0, int b0, int c0, const Geom& G, int& a, int& b, int& c,
                                           int& d) {
    using S = Shape<TX, TY, TZ>;
    if (e < S::OXL) {
        int i = e % TX, r = e / TX, j = r % TY, kk = r / TY;
        a = a0 + i; b = b0 + j; c = c0 + kk;
        d = a >= G.nx ? 0 : (b >= G.ny ? 1 : 2);   // partial block: the axis it leaves (used only along it)
    } else if (e < S::OYL) {
        int r = e - S::OXL;
        const bool hi = r >= S::HX;
        if (hi) r -= S::HX;
        int h = r % 3, rr = r / 3, j = rr % TY, kk = rr / TY;
        a = hi ? a0 + TX + h : a0 - 3 + h; b = b0 + j; c = c0 + kk; d = 0;
    } else if (e < S::OZL) {
        int r = e - S::OYL;
        const bool hi = r >= S::HY;
        if (hi) r -= S::HY;
        int i = r % TX, rr = r / TX, h = rr % 3, kk = rr / 3;
        a = a0 + i; b = hi ? b0 + TY + h : b0 - 3 + h; c = c0 + kk; d = 1;
    } else {
        int r = e - S::OZL;
        const bool hi = r >= S::HZ;
        if (hi) r -= S::HZ;
        int i = r % TX, rr = r / TX, j = rr % TY, h = rr / TY;
        a = a0 + i; b = b0 + j; c = hi ? c0 + TZ + h : c0 - 3 + h; d = 2;
    }
}

// Density contrast of a face's six-cell stencil above which a reduced-
// precision policy computes that face in FP64: where min rho < 1e-3 max rho
// the face states reconstructed on the thin side carry the rounding of the
// dense side's values (FP32: 1e-7 of them), i.e. relative errors of 1e-4 and
// more in the thin cell, whose velocity m / rho then runs away beside sinks.
constexpr float kStiffContrast = 1e-3f;

__device__ __forceinline__ bool stiff_stencil(const float (&c)[6][6]) {
    float lo = c[0][0], hi = c[0][0];
#pragma unroll
    for (int s = 1; s < 6; ++s) { lo = fminf(lo, c[s][0]); hi = fmaxf(hi, c[s][0]); }
    return lo < kStiffContrast * hi;
}

// The FP64 flux of the face between active cells p_D - 1 and p_D along D
// (p: the face's cell on the high side), from the FP64 state as the FP64
// path stages it (boundary map, floors on active cells, pressure once):
// the same operations, so the same bits as the FP64 path's flux there.
template <int D>
__device__ __noinline__ void face_flux_f64(const f64::StageArgs& A, int a, int b, int c, double F[5]) {
    Geom G(A.nx, A.ny, A.nz);
    double cs[6][6];
    bool ord = true;
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        int p[3] = {a, b, c};
        p[D] += s - 3;
        double v[5];
        bool act;
        load_cell(A, G, D, p[0], p[1], p[2], v, act);
        ord &= f64::floor_and_pressure(v, act, A.rho_floor, A.P_floor, A.Pfl_gm1, A.gm1, &cs[s][5]);
#pragma unroll
        for (int q = 0; q < 5; ++q) cs[s][q] = v[q];
    }
    if (!(ord && f64::ordinary_gamma(A.gm1)) || f64::interface_flux_ord(cs, A.g, A.gm1, A.igm1, A.gg, D, F))
        f64::general_flux(cs, A.g, A.gm1, D, F);
}

__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_int(a) == __float_as_int(b); }
__device__ __forceinline__ bool same_bits(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b);
}

// Uniform gas: where every staged cell of a block and its halos holds the same
// bits, each direction has one flux, whatever the face, and the divergence is
// that flux minus itself: +0, the bits it has face by face, if the flux is
// finite.  Such a block skips its faces.  That covers the undisturbed
// surroundings of a blast wave and gas at rest.  Measured with a blast of
// radius 0.15-0.25 of the box at 256^3, ms per step without and with:
// FP64 22.9 and 8.3, FP32 7.2 and 3.7, learned 10.4 and 6.0 (one-step
// calls, the first flag pass included; B200).
//
// calm: the one cell's flux is certainly finite.  Its reconstructions are the
// cell to within rounding, so with density, momentum and pressure in these
// bounds and a sound speed far above the rounding of the velocity (p rho
// against m^2), the HLLC speeds are v -+ c apart and nothing overflows.  The
// FP32 bounds also keep the WENO weights' products (ratios capped at 1e18,
// squared) below the FP32 range.
__device__ __forceinline__ bool calm(const double (&w)[5]) {   // rho, m, P
    const double m2 = sq(w[1]) + sq(w[2]) + sq(w[3]);
    return w[0] >= 0x1p-90 && w[0] <= 0x1p60 && w[4] >= 0x1p-200 && w[4] <= 0x1p60 && m2 <= 0x1p120 &&
           w[4] * w[0] * 0x1p40 >= m2;
}
__device__ __forceinline__ bool calm(const float (&w)[5]) {
    const float m2 = fmaf(w[3], w[3], fmaf(w[2], w[2], w[1] * w[1]));
    return w[0] >= 0x1p-30f && w[0] <= 32.f && w[4] >= 0x1p-60f && w[4] <= 32.f && m2 <= 1024.f &&
           w[4] * w[0] * 0x1p10f >= m2;
}

// Whether a face of the block could lie on a flux register: the registers
// cover the surface of the box [lo, hi].
__device__ __forceinline__ bool touches_registers(const f64::RegFaces& R, int a0, int b0, int c0, int tx, int ty,
                                                  int tz) {
    const int o[3] = {a0, b0, c0}, t[3] = {tx, ty, tz};
    bool near = true, within = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        near = near && o[d] <= R.hi[d] && o[d] + t[d] >= R.lo[d];
        within = within && o[d] > R.lo[d] && o[d] + t[d] < R.hi[d];
    }
    return near && !within;
}

// What a face's flux feeds besides its tile's divergence: the optional flux
// arrays, the coarse flux registers, the mass ledger's boundary sum and the
// fine boundary-face buffers.  (ga, gb, gc): the face's cell on the high side;
// only the face's owning tile calls this.
template <class R, bool LED>
__device__ __forceinline__ void record_face(const f64::StageArgs& A, const Geom& G, int D, int ga, int gb, int gc,
                                            const R (&F)[5], double* sled) {
    const int gd = D == 0 ? ga : (D == 1 ? gb : gc), nd = D == 0 ? G.nx : (D == 1 ? G.ny : G.nz);
    if (A.F[D]) {
        long long ex_ = (G.nx + 2 * BSN_NG) + (D == 0), ey_ = (G.ny + 2 * BSN_NG) + (D == 1);
        long long ii = ga + BSN_NG - (D == 0), jj = gb + BSN_NG - (D == 1), kk = gc + BSN_NG - (D == 2);
        long long off = 5LL * (ii + ex_ * (jj + ey_ * kk));
#pragma unroll
        for (int q = 0; q < 5; ++q) A.F[D][off + q] = (double)F[q];
    }
    if (A.use_reg) {
        const f64::RegFaces& R_ = A.reg;
        int ta = (D == 0) ? gb : ga, tb = (D == 2) ? gb : gc;
        int ax1 = (D == 0) ? 1 : 0, ax2 = (D == 2) ? 1 : 2;
        if (ta >= R_.t0[ax1] && ta <= R_.t1[ax1] && tb >= R_.t0[ax2] && tb <= R_.t1[ax2]) {
            int n1 = R_.t1[ax1] - R_.t0[ax1] + 1;
            long long roff = 5LL * ((ta - R_.t0[ax1]) + (long long)n1 * (tb - R_.t0[ax2]));
            double* dst = nullptr;
            if (gd == R_.lo[D]) dst = R_.reg[2 * D];
            else if (gd == R_.hi[D]) dst = R_.reg[2 * D + 1];
            if (dst) {
                double fac = A.dt_dev ? A.reg.wt * *A.dt_dev : R_.fac;
#pragma unroll
                for (int q = 0; q < 5; ++q) dst[roff + q] += fac * (double)F[q];
            }
        }
    }
    if (LED && A.ledger && A.led_bnd && (gd == 0 || gd == nd)) {   // mass through the grid's boundary
        // per unit volume, as the divergence sees it (the flush multiplies by dV)
        const double inv = (D == 0) ? A.idx : (D == 1 ? A.idy : A.idz);
        atomicAdd(&sled[f64::LED_BND], (gd == 0 ? (double)F[0] : -(double)F[0]) * inv);
    }
    if (A.use_bnd && (gd == 0 || gd == nd)) {
        int ta = (D == 0) ? gb : ga, tb = (D == 2) ? gb : gc;
        int n1 = (D == 0) ? G.ny : G.nx;
        long long roff = 5LL * (ta + (long long)n1 * tb);
        double* dst = A.bnd.f[2 * D + (gd == 0 ? 0 : 1)];
#pragma unroll
        for (int q = 0; q < 5; ++q) dst[roff + q] = (double)F[q];
    }
}

template <class P, int TX, int TY, int TZ, int NT, int D, bool LED>
__device__ void sweep(const f64::StageArgs& A, const Geom& G, const typename P::Consts& k, int a0, int b0, int c0,
                      typename P::real* sC, typename P::real* sF, unsigned char* psm,
                      double (&acc)[Shape<TX, TY, TZ>::NCELL / NT][5], bool quiet_cross, bool records, bool full,
                      double* sled, unsigned int* nlist, unsigned short* list) {
    using S = Shape<TX, TY, TZ>;
    using real = typename P::real;
    constexpr int CPT = S::NCELL / NT;
    constexpr int FX = TX + (D == 0), FY = TY + (D == 1), FZ = TZ + (D == 2);
    constexpr int NF = FX * FY * FZ;
    constexpr int TD = D == 0 ? TX : (D == 1 ? TY : TZ);
    const int tid = threadIdx.x;
    const int n[3] = {G.nx, G.ny, G.nz};
    const int o[3] = {a0, b0, c0};

    const bool quiet = quiet_cross;
    __syncthreads();   // staged once by stage_block; sF free after the previous sweep's divergence
    constexpr int FSTR = S::NCROSS;   // field stride of the staged values
    // staged index of stencil cell s (0..5, cells fd-3 .. fd+2 along D) of face (fx, fy, fz)
    auto sidx = [&](int fx, int fy, int fz, int s) -> int {
        const int fd = D == 0 ? fx : (D == 1 ? fy : fz);
        const int p = fd - 3 + s;
        int cb, cs, lo, hs;
        if (D == 0) { cb = TX * (fy + TY * fz); cs = 1; lo = S::OXL + 3 * (fy + TY * fz); hs = 1; }
        else if (D == 1) { cb = fx + TX * TY * fz; cs = TX; lo = S::OYL + fx + 3 * TX * fz; hs = TX; }
        else { cb = fx + TX * fy; cs = TX * TY; lo = S::OZL + fx + TX * fy; hs = TX * TY; }
        constexpr int H = D == 0 ? S::HX : (D == 1 ? S::HY : S::HZ);
        return p < 0 ? lo + (p + 3) * hs : (p < TD ? cb + p * cs : lo + H + (p - TD) * hs);
    };
    // one face: write it to smem and, if this tile owns it, to the optional
    // flux arrays, coarse flux registers and fine boundary-face buffers
    auto emit = [&](int f, int fx, int fy, int fz, const real (&F)[5]) {
#pragma unroll
        for (int q = 0; q < 5; ++q) sF[q * S::NFACE + f] = F[q];
        if (!records) return;
        int fpos[3] = {fx, fy, fz};
        int gd = o[D] + fpos[D];
        bool owner = (fpos[D] < TD) || (gd == n[D]);
        if (!owner) return;
        record_face<real, LED>(A, G, D, o[0] + fx, o[1] + fy, o[2] + fz, F, sled);
    };
    auto face_valid = [&](int fx, int fy, int fz) {
        if (full) return true;   // the block lies within the grid
        int fpos[3] = {fx, fy, fz};
        bool valid = true;
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            int gpos = o[t] + fpos[t];
            valid = valid && (t == D ? gpos <= n[t] : gpos < n[t]);
        }
        return valid;
    };
    // thread-per-face loop (the plain stencil physics); faces that the policy
    // defers (kDeferred: FP32's stiff density stencils, FP64 operands outside
    // the ordinary range) are listed for a second pass that computes them in
    // FP64 from the state, so the main loop keeps its registers, and the
    // listed faces are spread over all threads of the block (they cluster: a
    // star's surface, a sink's surroundings)
    // (nlist, list: the block's, used by one sweep after another; the barrier
    // at a sweep's start follows every use of the sweep before)
    auto plain_faces = [&]() {
        if constexpr (P::kDeferred) {
            if (tid == 0) *nlist = 0;
            __syncthreads();
        }
        for (int f = tid; f < NF; f += NT) {
            int fx = f % FX, r = f / FX, fy = r % FY, fz = r / FY;
            if (!face_valid(fx, fy, fz)) continue;
            real c[6][6];
#pragma unroll
            for (int s = 0; s < 6; ++s) {
                const int e = sidx(fx, fy, fz, s);
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const int col = q < 4 ? q : (q == 5 ? pcol<P::kCols>() : 4);
                    c[s][q] = q == 4 ? (real)0 : sC[col * FSTR + e];
                }
            }
            real F[5];
            const bool defer = P::flux(c, k, D, F);
            if constexpr (P::kDeferred) {
                if (defer) { list[atomicAdd(nlist, 1u)] = (unsigned short)f; continue; }
            }
            emit(f, fx, fy, fz, F);
        }
        if constexpr (P::kDeferred) {
            __syncthreads();
            const int nst = (int)*nlist;   // read by every thread before the next sweep resets it
            for (int i = tid; i < nst; i += NT) {
                const int f = list[i];
                const int fx = f % FX, r = f / FX, fy = r % FY, fz = r / FY;
                double F64[5];
                face_flux_f64<D>(A, o[0] + fx, o[1] + fy, o[2] + fz, F64);
                real F[5];
#pragma unroll
                for (int q = 0; q < 5; ++q) F[q] = (real)F64[q];
                emit(f, fx, fy, fz, F);
            }
        }
    };
    if constexpr (P::kWarpFaces) {
        if (P::kQuiescentSkip && quiet) {
            plain_faces();   // uniform sweep: no per-stencil work can apply, the policy's plain flux
        } else {
            // warp-collective faces (tensor-core work inside the flux): every
            // lane of a warp takes part in every iteration, valid face or not
            const int warp = tid >> 5, lane = tid & 31;
            for (int fb = warp * 32; fb < NF; fb += NT) {
                int f = fb + lane;
                int fx = f % FX, r = f / FX, fy = r % FY, fz = r / FY;
                bool valid = f < NF && face_valid(fx, fy, fz);
                real c[6][6];
#pragma unroll
                for (int s = 0; s < 6; ++s) {
                    const int e = valid ? sidx(fx, fy, fz, s) : 0;
#pragma unroll
                    for (int q = 0; q < 6; ++q) {
                        const int col = q < 4 ? q : (q == 5 ? pcol<P::kCols>() : 4);
                        c[s][q] = (valid && (q != 4 || P::kCols == 6)) ? sC[col * FSTR + e] : (real)0;
                    }
                }
                real F[5];
                P::warp_flux(c, valid, k, F, psm, warp, quiet, D);
                if (valid) emit(f, fx, fy, fz, F);
            }
        }
    } else {
        plain_faces();
    }
    __syncthreads();

    const double inv = (D == 0) ? A.idx : (D == 1 ? A.idy : A.idz);
    constexpr int FS = (D == 0) ? 1 : (D == 1 ? FX : FX * FY);
#pragma unroll
    for (int m = 0; m < CPT; ++m) {
        int cell = tid + m * NT;
        int i = cell % TX, j = (cell / TX) % TY, kk = cell / (TX * TY);
        int fl = i + FX * (j + FY * kk);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            double dF = (double)sF[q * S::NFACE + fl + FS] - (double)sF[q * S::NFACE + fl];
            if (D == 0) acc[m][q] = -dF * inv;
            else acc[m][q] = acc[m][q] - dF * inv;
        }
    }
}

// Policy-specific shared memory (learned parameters, row buffers) after the
// staged cells and faces.
template <class P, int TX, int TY, int TZ>
__device__ __forceinline__ unsigned char* policy_smem(unsigned char* smem_raw) {
    using S = Shape<TX, TY, TZ>;
    return smem_raw + ((sizeof(typename P::real) * (P::kCols * S::NCROSS + 5 * S::NFACE) + 15) / 16) * 16;
}

// Whether active cell (a, b, c) counts in the mass ledger: outside the
// region a finer level covers (half-open [led_skip_lo, led_skip_hi)).
__device__ __forceinline__ bool led_counted(const f64::StageArgs& A, int a, int b, int c) {
    return !(a >= A.led_skip_lo[0] && a < A.led_skip_hi[0] && b >= A.led_skip_lo[1] && b < A.led_skip_hi[1] &&
             c >= A.led_skip_lo[2] && c < A.led_skip_hi[2]);
}

// TMA staging state of a CTA (stage_kernel_tma): the tensor maps, the two
// raw buffers, their mbarriers and the parity each barrier completes next.
struct TmaCtx {
    const tma::Maps* M;
    double* raw[2];
    uint64_t* bar;
    uint32_t ph[2];
};

// Raw-buffer placement of a tile: inside the face buffer when it is free
// (it is during staging) and large enough, else after the policy's smem.
// Copies of kChunkCap bytes where the dynamic smem still fits MINB CTAs per
// SM, else copies small enough for both buffers to sit in the face buffer.
template <class P, int TX, int TY, int TZ, int NT, int MINB>
struct TmaSmem {
    using S = Shape<TX, TY, TZ>;
    static constexpr int FACE_OFF = (int)sizeof(typename P::real) * P::kCols * S::NCROSS;
    static constexpr int FACE_BYTES = (int)sizeof(typename P::real) * 5 * S::NFACE;
    static constexpr int APPEND_OFF = (int)(((sizeof(typename P::real) * (P::kCols * S::NCROSS + 5 * S::NFACE) + 16) +
                                             127) / 128 * 128);
    static constexpr int in_faces(int rawb) { return FACE_BYTES >= 2 * rawb ? 2 : (FACE_BYTES >= rawb ? 1 : 0); }
    static constexpr int bytes_for(int rawb) { return APPEND_OFF + (2 - in_faces(rawb)) * rawb; }
    // per-CTA dynamic smem that keeps MINB CTAs on an SM, beside the system's
    // 1 KB, the deferred faces' list and up to 1 KB of other static smem
    static constexpr int BUDGET = 233472 / MINB - 2048 - (P::kDeferred && P::kCols == 5 ? 2 * S::NFACE : 0);
    static constexpr int CAP = bytes_for(tma::Chunks<TX, TY, TZ, tma::kChunkCap>::RAWB) <= BUDGET
                                   ? tma::kChunkCap
                                   : FACE_BYTES / 2 / 128 * 128;
    using C = tma::Chunks<TX, TY, TZ, CAP>;
    static constexpr int IN_FACES = in_faces(C::RAWB);
    static constexpr int BYTES = bytes_for(C::RAWB);   // dynamic smem of the TMA kernel
    static_assert(FACE_OFF % 128 == 0, "face buffer must start on a 128-byte boundary for TMA copies");
    // raw buffer 0 always lies in the face buffer (the layouts this path is
    // verified with); a tile whose copies fit only after the face buffer
    // keeps the plain loader
    static constexpr bool OK = IN_FACES >= 1;
};

// The cross region of block (a0, b0, c0) staged by TMA copies: each copy's
// cells converted as the plain loader converts them (P::stage, pressure),
// cells outside the active domain through the boundary map instead.  Returns
// false on every thread when a copy did not arrive within the wait bound
// (the error word is set and the copies in flight are waited for, bounded).
template <class P, int TX, int TY, int TZ, int NT, int MINB>
__device__ bool stage_cross_tma(const f64::StageArgs& A, TmaCtx& T, const Geom& G, const typename P::Consts& k,
                                int a0, int b0, int c0, typename P::real* sC, bool& odd) {
    using S = Shape<TX, TY, TZ>;
    using C = typename TmaSmem<P, TX, TY, TZ, NT, MINB>::C;
    using real = typename P::real;
    const int tid = threadIdx.x;
    const tma::Maps& M = *T.M;
    const int n[3] = {G.nx, G.ny, G.nz};
    auto issue = [&](int c, int b) {   // thread 0: copy c into buffer b
        uint32_t bytes;
        const CUtensorMap* map;
        int x, y, z;
        if (c < C::NA) {
            map = &M.a; bytes = C::BA; x = 5 * a0;
            y = b0 + 3 + (c % C::NAY) * C::AY; z = c0 + 3 + (c / C::NAY) * C::AZ;
        } else if (c < C::NA + C::NY) {
            const int r = c - C::NA, hi = r >= C::NY / 2, p = hi ? r - C::NY / 2 : r;
            map = &M.y; bytes = C::BY; x = 5 * (a0 + 2); y = hi ? b0 + TY + 3 : b0; z = c0 + 3 + p * C::YZ;
        } else {
            const int r = c - C::NA - C::NY, hi = r >= C::NZ / 2, p = hi ? r - C::NZ / 2 : r;
            map = &M.z; bytes = C::BZ; x = 5 * (a0 + 2); y = b0 + 3 + p * C::ZY; z = hi ? c0 + TZ + 3 : c0;
        }
        tma::fence_proxy_async();   // earlier generic accesses of the buffer before the copy's writes
        tma::mbar_expect_tx(&T.bar[b], bytes);
        tma::load_3d(T.raw[b], map, &T.bar[b], x, y, z);
    };
    // one staged cell: from the copy (src, 5 doubles) when it lies in the
    // active domain along axis d, else through the boundary map
    auto put = [&](int e, int a, int b, int c, int d, const double* src) {
        const int p = d == 0 ? a : (d == 1 ? b : c);
        double v[5];
        bool act = true;
        if (p >= 0 && p < n[d]) {
#pragma unroll
            for (int q = 0; q < 5; ++q) v[q] = src[q];
        } else {
            load_cell(A, G, d, a, b, c, v, act);
        }
        real w[5], pr;
        odd |= !P::stage(v, act, A, k, w, pr);
#pragma unroll
        for (int q = 0; q < 5; ++q)
            if (q < 4 || P::kCols == 6) sC[q * S::NCROSS + e] = w[q];
        sC[pcol<P::kCols>() * S::NCROSS + e] = pr;
    };
    if (tid == 0) {
        issue(0, 0);
        if (C::N > 1) issue(1, 1);
    }
    for (int c = 0; c < C::N; ++c) {
        const int b = c & 1;
        const bool got = tma::mbar_wait_bounded(&T.bar[b], T.ph[b]);
        const double* raw = T.raw[b];
        if (got) {
            if (c < C::NA) {   // block rows with their x halos: AY rows x AZ planes
                const int j0 = (c % C::NAY) * C::AY, k0 = (c / C::NAY) * C::AZ;
                for (int t = tid; t < (TX + 6) * C::AY * C::AZ; t += NT) {
                    const int ib = t % (TX + 6), r = t / (TX + 6), jb = r % C::AY, kb = r / C::AY;
                    const int j = j0 + jb, kk = k0 + kb;
                    const int e = ib < 3 ? S::OXL + ib + 3 * (j + TY * kk)
                                         : (ib >= TX + 3 ? S::OXH + (ib - TX - 3) + 3 * (j + TY * kk)
                                                         : (ib - 3) + TX * (j + TY * kk));
                    put(e, a0 - 3 + ib, b0 + j, c0 + kk, 0, raw + 5 * ib + C::RA * (jb + C::AY * kb));
                }
            } else if (c < C::NA + C::NY) {   // y halo rows
                const int r = c - C::NA, hi = r >= C::NY / 2, p = hi ? r - C::NY / 2 : r;
                for (int t = tid; t < TX * 3 * C::YZ; t += NT) {
                    const int i = t % TX, r2 = t / TX, h = r2 % 3, kb = r2 / 3, kk = p * C::YZ + kb;
                    const int e = (hi ? S::OYH : S::OYL) + i + TX * (h + 3 * kk);
                    put(e, a0 + i, hi ? b0 + TY + h : b0 - 3 + h, c0 + kk, 1, raw + 5 * (i + 1) + C::RH * (h + 3 * kb));
                }
            } else {   // z halo planes
                const int r = c - C::NA - C::NY, hi = r >= C::NZ / 2, p = hi ? r - C::NZ / 2 : r;
                for (int t = tid; t < TX * C::ZY * 3; t += NT) {
                    const int i = t % TX, r2 = t / TX, jb = r2 % C::ZY, h = r2 / C::ZY, j = p * C::ZY + jb;
                    const int e = (hi ? S::OZH : S::OZL) + i + TX * (j + TY * h);
                    put(e, a0 + i, b0 + j, hi ? c0 + TZ + h : c0 - 3 + h, 2,
                        raw + 5 * (i + 1) + C::RH * (jb + C::ZY * h));
                }
            }
        }
        // every thread is done with buffer b; one decision for the whole CTA
        const bool ok = __syncthreads_and(got);
        if (!ok) {
            if (tid == 0) {
                if (M.err) atomicOr(M.err, 1u);
                // the copies still in flight: this one and the other buffer's
                tma::mbar_wait_bounded(&T.bar[b], T.ph[b]);
                if (c + 1 < C::N) tma::mbar_wait_bounded(&T.bar[b ^ 1], T.ph[b ^ 1]);
            }
            __syncthreads();
            return false;
        }
        T.ph[b] ^= 1u;
        if (tid == 0 && c + 2 < C::N) issue(c + 2, b);
    }
    return true;
}

// The stage's base state of the cell at offset off (nothing in RHS mode).
__device__ __forceinline__ void load_un(const f64::StageArgs& A, long long off, double (&un)[5]) {
#pragma unroll
    for (int q = 0; q < 5; ++q) un[q] = A.mode == 1 ? 0.0 : A.Un[off + q];
}

// The stage's SSP-RK3 combination, before the floors.
__device__ __forceinline__ void rk_combine(const f64::StageArgs& A, double u0, double u1, double u2, double u3,
                                           double u4, const double (&un)[5], const double (&d)[5], double dt,
                                           double cdt, double (&w)[5]) {
    const double uu[5] = {u0, u1, u2, u3, u4};
    if (A.stage == 1) {
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = un[q] + dt * d[q];
    } else if (A.stage == 2) {
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = 0.75 * un[q] + 0.25 * uu[q] + cdt * d[q];
    } else {
#pragma unroll
        for (int q = 0; q < 5; ++q) w[q] = (1.0 / 3.0) * un[q] + (2.0 / 3.0) * uu[q] + cdt * d[q];
    }
}

// The end of one cell's stage from its floored input (u0..u4), base state un
// and flux divergence d: sources in the driver's order, SSP-RK3 combine, floors, the
// store, and the next CFL speed.  s_nan: the block's NaN flag; w: the result.
template <class P, bool LED>
__device__ __forceinline__ void finish_cell(const f64::StageArgs& A, const Geom& G, int a, int b, int c, double u0,
                                            double u1, double u2, double u3, double u4, const double (&un)[5],
                                            double (&d)[5], const f64::BHSrc& BH, const f64::SinkSrc& SK, double dt,
                                            double cdt, double* sled, double& smax, unsigned int& s_nan,
                                            double (&w)[5]) {
    const long long off = G.act(a, b, c);
    double xc = A.x0 + ((double)(a + 1) - 0.5) * A.dx;
    double yc = A.y0 + ((double)(b + 1) - 0.5) * A.dy;
    double zc = A.z0 + ((double)(c + 1 + A.k0) - 0.5) * A.dz;
    if (A.use_bh) {   // src/gpu_kernels.jl:199-230
        double vx = u1 / u0, vy = u2 / u0, vz = u3 / u0;
        double ax = 0.0, ay = 0.0, az = 0.0;
        for (int nb = 0; nb < BH.n; ++nb) {
            double ddx = xc - BH.px[nb], ddy = yc - BH.py[nb], ddz = zc - BH.pz[nb];
            double r2 = sq(ddx) + sq(ddy) + sq(ddz) + sq(BH.eps[nb]);
            double r3 = r2 * sqrt(r2);
            double fac = -BH.mass[nb] / r3;
            ax += fac * ddx; ay += fac * ddy; az += fac * ddz;
        }
        d[1] += u0 * ax; d[2] += u0 * ay; d[3] += u0 * az;
        d[4] += u0 * (vx * ax + vy * ay + vz * az);
    }
    if (A.use_sg) {   // src/gpu_kernels.jl:291-319
        int nx = A.nx, ny = A.ny, nz = A.nz;
        int ip = min(a + 1, nx - 1), im = max(a - 1, 0);
        int jp = min(b + 1, ny - 1), jm = max(b - 1, 0);
        int kp = min(c + 1, nz - 1), km = max(c - 1, 0);
        double fx = ip > im ? A.inv2dx : 2.0 * A.inv2dx;
        double fy = jp > jm ? A.inv2dy : 2.0 * A.inv2dy;
        double fz = kp > km ? A.inv2dz : 2.0 * A.inv2dz;
        const double* Pp = A.phi;
        long long sy = nx, sz = (long long)nx * ny;
        double gx = (Pp[ip + sy * b + sz * c] - Pp[im + sy * b + sz * c]) * fx;
        double gy = (Pp[a + sy * jp + sz * c] - Pp[a + sy * jm + sz * c]) * fy;
        double pzp = Pp[a + sy * b + sz * kp], pzm = Pp[a + sy * b + sz * km];
        if (A.phi_lo || A.phi_hi) {   // a slab's edge planes: the larger grid's central difference
            fz = A.inv2dz;
            if (c == nz - 1 && A.phi_hi) pzp = A.phi_hi[a + sy * b];
            if (c == 0 && A.phi_lo) pzm = A.phi_lo[a + sy * b];
        }
        double gz = (pzp - pzm) * fz;
        double vdotg = (u1 * gx + u2 * gy + u3 * gz) / u0;
        d[1] -= u0 * gx; d[2] -= u0 * gy; d[3] -= u0 * gz; d[4] -= u0 * vdotg;
    }
    if (A.use_sink && u0 > SK.rho_min) {   // src/gpu_kernels.jl:238-284
        for (int nb = 0; nb < SK.n; ++nb) {
            double ddx = xc - SK.px[nb], ddy = yc - SK.py[nb], ddz = zc - SK.pz[nb];
            double rr = sqrt(sq(ddx) + sq(ddy) + sq(ddz));
            if (rr < SK.rs[nb]) {
                double ts = SK.ts[nb];
                d[0] -= u0 / ts;
                if (LED && A.ledger && led_counted(A, a, b, c)) atomicAdd(&sled[f64::LED_DRAIN], u0 / ts);
                if (SK.torque_free) {
                    double rx = ddx / rr, ry = ddy / rr, rz = ddz / rr;
                    double vx = u1 / u0, vy = u2 / u0, vz = u3 / u0;
                    double vrx = vx - SK.vx[nb], vry = vy - SK.vy[nb], vrz = vz - SK.vz[nb];
                    double v_r = vrx * rx + vry * ry + vrz * rz;
                    double e_int = u4 / u0 - 0.5 * (sq(vx) + sq(vy) + sq(vz));
                    d[1] -= u0 * v_r * rx / ts;
                    d[2] -= u0 * v_r * ry / ts;
                    d[3] -= u0 * v_r * rz / ts;
                    d[4] -= (0.5 * u0 * sq(v_r) + u0 * e_int) / ts;
                } else {
                    d[1] -= u1 / ts; d[2] -= u2 / ts; d[3] -= u3 / ts; d[4] -= u4 / ts;
                }
            }
        }
    }
    if (A.use_rot) f64::rot_frame_src(d, u0, u1, u2, xc, yc, A.rot_omega);   // src/relax_ic.jl:150-176
    if (A.use_damp) f64::damp_src(d, u0, u1, u2, u3, xc, yc, A.damp_inv_td, A.damp_t, A.damp_omega);
    if (A.mode == 1) {
        // Uin is not written here: other blocks are still staging these
        // cells as halos, and a cell read while its five words were being
        // replaced by their floored values would mix the two states.  The
        // RHS entry points floor Uin in a launch of its own afterwards.
#pragma unroll
        for (int q = 0; q < 5; ++q) A.dU[off + q] = d[q];
        return;
    }
    rk_combine(A, u0, u1, u2, u3, u4, un, d, dt, cdt, w);
    const double w0 = w[0];
    P::floor(w, A);
    if (LED && A.ledger && led_counted(A, a, b, c)) {
        if (w[0] != w0) atomicAdd(&sled[f64::LED_POST], w[0] - w0);
        if (A.stage > 1) {   // the input's floors reach the combine in stages 2 and 3
            const double raw = A.Uin[off];
            if (u0 != raw) atomicAdd(&sled[f64::LED_PRE], u0 - raw);
        }
    }
#pragma unroll
    for (int q = 0; q < 5; ++q) A.Uout[off + q] = w[q];
    if (A.cfl_max) {
        double s = f64::cfl_speed(w[0], w[1], w[2], w[3], w[4], A.g, A.gm1, A.idx, A.idy, A.idz);
        if (s != s) s_nan = 1;
        else smax = fmax(smax, s);
    }
}

// One RK3 stage (or euler3d_rhs!) of the TX x TY x TZ block at active
// origin (a0, b0, c0): three sweeps, sources, combine, floors, CFL fold.
// Starts with a barrier (the first sweep's), so a CTA may call it for one
// block after another.
template <class P, int TX, int TY, int TZ, int NT, int MINB = 1, bool LED = false, bool UNI = false>
__device__ __forceinline__ bool stage_block(const f64::StageArgs& A, int a0, int b0, int c0,
                                            unsigned char* smem_raw, double* red, unsigned int& nanflag,
                                            TmaCtx* T = nullptr) {
    using S = Shape<TX, TY, TZ>;
    using real = typename P::real;
    static_assert(S::NCELL % NT == 0, "cells must divide evenly among threads");
    constexpr int CPT = S::NCELL / NT;
    real* sC = reinterpret_cast<real*>(smem_raw);
    real* sF = sC + P::kCols * S::NCROSS;

    Geom G(A.nx, A.ny, A.nz);
    const int tid = threadIdx.x;
    if (tid == 0) nanflag = 0;
    typename P::Consts k = P::consts(A);
    unsigned char* psm = policy_smem<P, TX, TY, TZ>(smem_raw);
    double acc[CPT][5];
    // this block's mass-ledger sums (LED kernels with A.ledger set; the other
    // kernels carry no ledger code at all)
    __shared__ double sled[LED ? f64::LED_TERMS : 1];
    if (LED && A.ledger && tid < f64::LED_TERMS) sled[tid] = 0.0;   // ordered before use by the staging barriers

    // UNI (the launches over listed tiles): uniform, calm gas in the block and
    // its halos, with no use for its fluxes besides the divergence, skips the
    // faces; found while staging.  The other launches carry no test: it costs
    // 2-5 % where no block is uniform.
    const bool rim = a0 == 0 || b0 == 0 || c0 == 0 || a0 + TX >= A.nx || b0 + TY >= A.ny || c0 + TZ >= A.nz;
    // fluxes used by more than the divergence
    const bool face_out = A.F[0] || A.F[1] || A.F[2] || (rim && (A.use_bnd || (LED && A.ledger && A.led_bnd))) ||
                         (A.use_reg && touches_registers(A.reg, a0, b0, c0, TX, TY, TZ));
    bool uniform = false;
    __syncthreads();   // the previous block of a persistent CTA is done with smem
    {
        // the block and the halos of all three sweeps, staged once (floors in
        // FP64 on active cells, ghosts raw, pressure once per cell)
        bool odd = false;               // a staged cell outside the policy's ordinary range
        bool differs = false;           // staged cells that are not all the same
        real w0[5];
        if (T) {
            if (!stage_cross_tma<P, TX, TY, TZ, NT, MINB>(A, *T, G, k, a0, b0, c0, sC, odd)) return false;
        } else {
            for (int e = tid; e < S::NCROSS; e += NT) {
                int a, b, c, d;
                cross_cell<TX, TY, TZ>(e, a0, b0, c0, G, a, b, c, d);
                double v[5];
                bool act;
                load_cell(A, G, d, a, b, c, v, act);
                real w[5], pr;
                odd |= !P::stage(v, act, A, k, w, pr);
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (q < 4 || P::kCols == 6) sC[q * S::NCROSS + e] = w[q];
                sC[pcol<P::kCols>() * S::NCROSS + e] = pr;
                if constexpr (UNI) {
                    w[4] = pr;
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        if (e == tid) w0[q] = w[q];
                        differs |= !same_bits(w[q], w0[q]);
                    }
                }
            }
        }
        if constexpr (P::kOrdinary) k.ord = !__syncthreads_or(odd || !k.ord);
        else if constexpr (UNI) __syncthreads();
        if (UNI && !face_out) {
            static_assert(S::NCROSS >= NT, "a staged entry per thread");
            if (!differs) {
                differs = !calm(w0);
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    differs |= !same_bits(w0[q], sC[(q < 4 ? q : pcol<P::kCols>()) * S::NCROSS]);
            }
            uniform = !__syncthreads_or(differs);
        }
    }
    // policies with per-stencil work that only non-uniform data can need (the
    // learned weights' fallback test) learn here, per sweep, whether every
    // value the sweep's stencils read (the block and that sweep's halos)
    // equals the block's first cell within the policy's margin
    bool quiet[3] = {false, false, false};
    if (P::kQuiescentSkip && !uniform) {
        if constexpr (!UNI && !P::kOrdinary) __syncthreads();
        unsigned varied = 0u;   // bit 0: block, bits 1-3: x, y, z halos
        for (int e = tid; e < S::NCROSS; e += NT) {
            bool v = false;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const int col = q < 4 ? q : pcol<P::kCols>();
                v |= !P::same(sC[col * S::NCROSS + e], sC[col * S::NCROSS]);
            }
            if (v) varied |= e < S::OXL ? 1u : (e < S::OYL ? 2u : (e < S::OZL ? 4u : 8u));
        }
        const bool vb = __syncthreads_or(varied & 1u), vx = __syncthreads_or(varied & 2u),
                   vy = __syncthreads_or(varied & 4u), vz = __syncthreads_or(varied & 8u);
        quiet[0] = !(vb || vx);
        quiet[1] = !(vb || vy);
        quiet[2] = !(vb || vz);
        if constexpr (P::kScreen) {
            // a block with a non-uniform sweep is left to the split stage's
            // other launch: listed, nothing written here (the test is uniform
            // over the CTA, so every thread returns)
            if (!(quiet[0] && quiet[1] && quiet[2])) {
                if (tid == 0) {
                    const int gx = (A.nx + TX - 1) / TX, gy = (A.ny + TY - 1) / TY;
                    const int t = a0 / TX + gx * (b0 / TY + gy * (c0 / TZ));
                    A.split_list[atomicAdd(A.split_count, 1u)] = t;
                    if (UNI) A.uni_out[t] = 0;   // its result is no more uniform than its input
                }
                return true;
            }
        }
    }
    const bool full = a0 + TX <= A.nx && b0 + TY <= A.ny && c0 + TZ <= A.nz;
    static_assert(S::NFACE <= 65536, "face indices of 16 bits");
    // Faces deferred to a sweep's second pass.  Where their list would cost a
    // CTA per SM (FP64 16x8x4 at two: 880 bytes are left) it lies in the staged
    // column of E, whose halo cells nothing reads.
    constexpr int kDyn = (P::kCols * S::NCROSS + 5 * S::NFACE) * (int)sizeof(real) + 16, kRest = 1024 + 512;
    constexpr bool kListInHalo = P::kDeferred && P::kCols == 6 && (kDyn + kRest) * MINB <= 233472 &&
                                 (kDyn + kRest + 2 * S::NFACE) * MINB > 233472;
    static_assert(!kListInHalo || sizeof(real) * (S::NCROSS - S::NCELL) >= 2 * S::NFACE, "the halos hold the list");
    __shared__ unsigned int nlist;
    __shared__ unsigned short slist[P::kDeferred && !kListInHalo ? S::NFACE : 1];
    unsigned short* list = kListInHalo ? reinterpret_cast<unsigned short*>(sC + 4 * S::NCROSS + S::NCELL) : slist;
    if (uniform) {
        // -(F - F) / dx - (F - F) / dy - (F - F) / dz of finite fluxes
        const double none = (-(0.0) * A.idx - 0.0 * A.idy) - 0.0 * A.idz;
#pragma unroll
        for (int m = 0; m < CPT; ++m)
#pragma unroll
            for (int q = 0; q < 5; ++q) acc[m][q] = none;
    } else {
        sweep<P, TX, TY, TZ, NT, 0, LED>(A, G, k, a0, b0, c0, sC, sF, psm, acc, quiet[0], face_out, full, sled, &nlist, list);
        sweep<P, TX, TY, TZ, NT, 1, LED>(A, G, k, a0, b0, c0, sC, sF, psm, acc, quiet[1], face_out, full, sled, &nlist, list);
        sweep<P, TX, TY, TZ, NT, 2, LED>(A, G, k, a0, b0, c0, sC, sF, psm, acc, quiet[2], face_out, full, sled, &nlist, list);
    }

    const double dt = A.dt_dev ? *A.dt_dev : A.dt;
    const f64::BHSrc& BH = A.bh_dev ? *A.bh_dev : A.bh;     // kernel parameters are __grid_constant__
    const f64::SinkSrc& SK = A.sk_dev ? *A.sk_dev : A.sk;
    const double cdt = A.stage == 2 ? 0.25 * dt : (A.stage == 3 ? (2.0 / 3.0) * dt : dt);
    double smax = 0.0;
    double wref[UNI ? 5 : 1];
    bool have = false, mixed = false;   // whether wref is set; results that differ from it
    __shared__ double s_w[UNI ? 5 : 1];
#pragma unroll
    for (int m = 0; m < CPT; ++m) {
        int idx = tid + m * NT;
        int i = idx % TX, j = (idx / TX) % TY, kk = idx / (TX * TY);
        int a = a0 + i, b = b0 + j, c = c0 + kk;
        if (a >= A.nx || b >= A.ny || c >= A.nz) continue;
        long long off = G.act(a, b, c);
        double u[5], un[5], w[5];
        if (P::kCenterFromSmem) {
            constexpr int FS = S::NCROSS;   // the block's cells: the cross region's first part
            int e = i + TX * (j + TY * kk);
#pragma unroll
            for (int q = 0; q < 5; ++q) u[q] = (double)sC[q * FS + e];
        } else {
#pragma unroll
            for (int q = 0; q < 5; ++q) u[q] = A.Uin[off + q];
            P::floor(u, A);
        }
        load_un(A, off, un);
        finish_cell<P, LED>(A, G, a, b, c, u[0], u[1], u[2], u[3], u[4], un, acc[m], BH, SK, dt, cdt, sled, smax,
                            nanflag, w);
        if constexpr (UNI) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                if (!have) wref[q] = w[q];
                else mixed |= !same_bits(w[q], wref[q]);
            }
            have = true;
            if (m == 0 && tid == 0) {   // the tile's first cell is always an active one
#pragma unroll
                for (int q = 0; q < 5; ++q) s_w[q] = w[q];
            }
        }
    }
    if constexpr (UNI) {
        __syncthreads();
        if (have) {
#pragma unroll
            for (int q = 0; q < 5; ++q) mixed |= !same_bits(wref[q], s_w[q]);
        }
        const bool uni = !__syncthreads_or(mixed);
        const int gx = (A.nx + TX - 1) / TX, gy = (A.ny + TY - 1) / TY;
        if (tid == 0) A.uni_out[a0 / TX + gx * (b0 / TY + (long long)gy * (c0 / TZ))] = uni;
    }
    if (A.cfl_max) {
        for (int o = 16; o > 0; o >>= 1) smax = fmax(smax, __shfl_xor_sync(0xffffffffu, smax, o));
        if ((tid & 31) == 0) red[tid >> 5] = smax;
        __syncthreads();
        if (tid == 0) {
            double m = 0.0;
            for (int w = 0; w < NT / 32; ++w) m = fmax(m, red[w]);
            atomicMax(A.cfl_max, (unsigned long long)__double_as_longlong(m));
            if (nanflag) atomicOr(A.cfl_nan, 1u);
        }
    }
    if (LED && A.ledger) {
        __syncthreads();   // every cell's and face's contribution is in sled
        if (tid < f64::LED_TERMS && sled[tid] != 0.0) atomicAdd(&A.ledger[tid], sled[tid] * (A.dx * A.dy * A.dz));
    }
    return true;
}

// One launch per stage on one grid: CTA (x, y, z) owns block (x, y, z).
// LED: the instantiation that keeps the mass ledger (A.ledger) -- the driver
// loops' launches; the others compile no ledger code.
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool LED = false>
__global__ void __launch_bounds__(NT, MINB) stage_kernel(const __grid_constant__ f64::StageArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red[NT / 32];
    __shared__ unsigned int nanflag;
    if (A.done_dev && *A.done_dev) return;   // device time loop already reached t_end
    P::prologue(policy_smem<P, TX, TY, TZ>(smem_raw), A, NT);   // visible after the first barrier
    stage_block<P, TX, TY, TZ, NT, MINB, LED>(A, blockIdx.x * TX, blockIdx.y * TY, blockIdx.z * TZ, smem_raw, red,
                                              nanflag);
}

// stage_kernel with the cross region staged by TMA copies (tma.cuh): one
// block per CTA, as stage_kernel.  Launched only where build_maps accepted
// the grid (uniform grid, tile dividing it, even nx, no ghost buffer).
template <class P, int TX, int TY, int TZ, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
    stage_kernel_tma(const __grid_constant__ f64::StageArgs A, const __grid_constant__ tma::Maps M) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red[NT / 32];
    __shared__ unsigned int nanflag;
    __shared__ __align__(8) uint64_t bar[2];
    if (A.done_dev && *A.done_dev) return;
    using TS = TmaSmem<P, TX, TY, TZ, NT, MINB>;
    using C = typename TS::C;
    // a copy's destination must lie on a 128-byte boundary: the dynamic shared
    // memory starts where the static part ends, at the alignment of its
    // declaration -- the strictest one that a unit's kernels give the name must
    // be the first, so all of them say 128
    if (tma::smem_u32(smem_raw) & 127u) {
        if (threadIdx.x == 0 && M.err) atomicOr(M.err, 1u);
        return;
    }
    P::prologue(policy_smem<P, TX, TY, TZ>(smem_raw), A, NT);
    if (threadIdx.x == 0) {
        tma::mbar_init(&bar[0], 1);
        tma::mbar_init(&bar[1], 1);
        tma::fence_barrier_init();
    }
    __syncthreads();
    unsigned char* face = smem_raw + TS::FACE_OFF;
    unsigned char* app = smem_raw + TS::APPEND_OFF;
    TmaCtx T;
    T.M = &M;
    T.raw[0] = reinterpret_cast<double*>(TS::IN_FACES >= 1 ? face : app);
    T.raw[1] = reinterpret_cast<double*>(TS::IN_FACES == 2 ? face + C::RAWB
                                                             : (TS::IN_FACES == 1 ? app : app + C::RAWB));
    T.bar = bar;
    T.ph[0] = T.ph[1] = 0u;
    stage_block<P, TX, TY, TZ, NT, MINB>(A, blockIdx.x * TX, blockIdx.y * TY, blockIdx.z * TZ, smem_raw, red, nanflag,
                                         &T);
}

// The listed blocks of a stage (written by the launch before it on the same
// stream), walked by a persistent grid: each CTA takes its first block by its
// index, then draws the next from a queue counter (list_count[1], zeroed with
// the count), so CTAs whose blocks take longer take fewer.  UNI: the list is
// uniform_stage_kernel's, so its tiles may still be uniform, and their results'
// flags are kept.  A learned screen's list holds no such tile, and there the
// test cost 5 %: a learned 256^3 step without uniform gas 32.9 ms without it
// and 34.4 with it, 128x96x80 2.39 and 2.49.
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool UNI>
__global__ void __launch_bounds__(NT, MINB) stage_kernel_list(const __grid_constant__ f64::StageArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red[NT / 32];
    __shared__ unsigned int nanflag;
    __shared__ int next;
    if (A.done_dev && *A.done_dev) return;
    const int n = (int)*A.list_count;
    if ((int)blockIdx.x >= n) return;
    P::prologue(policy_smem<P, TX, TY, TZ>(smem_raw), A, NT);   // visible after the first barrier
    const int gx = (A.nx + TX - 1) / TX, gy = (A.ny + TY - 1) / TY;
    for (int t = blockIdx.x; t < n;) {
        const int b = A.list[t];
        stage_block<P, TX, TY, TZ, NT, MINB, false, UNI>(A, (b % gx) * TX, ((b / gx) % gy) * TY, (b / (gx * gy)) * TZ,
                                                         smem_raw, red, nanflag);
        // the block's barriers order every thread's reads of `next` before this write
        if (threadIdx.x == 0) next = (int)gridDim.x + (int)atomicAdd(A.list_count + 1, 1u);
        __syncthreads();
        t = next;
    }
}

// The tiles of a stage whose result is one cell: uniform in the input and the
// base state, with the same cell in the six neighbouring tiles, calm, above the
// floors, and no sources (the host's condition).  Nothing is staged and one cell is read and
// combined per tile; the others are listed for the stage kernel, whose CTAs
// (registers for the faces, two or three per SM) a quiet tile would only hold.
// Bound by its stores; 128 threads per tile and few registers keep some 2,000
// tiles in flight.  A warp per row, here and in uniform_tiles_kernel, instead
// of divisions per word: two FP32 256^3 steps 6.56 -> 6.06 ms, one FP64 step
// 7.97 -> 7.49, two learned steps 10.9 -> 10.3.
template <class P>
__global__ void __launch_bounds__(128, 8) uniform_stage_kernel(const __grid_constant__ f64::StageArgs A, int tx, int ty,
                                                                int tz) {
    if (A.done_dev && *A.done_dev) return;
    const int tid = threadIdx.x, gx = gridDim.x, gy = gridDim.y, gz = gridDim.z;
    const int nb[3] = {(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z};
    const long long tile = nb[0] + gx * (nb[1] + (long long)gy * nb[2]);
    if (tile == 0 && tid < 2) A.list_zero[tid] = 0u;
    const Geom G(A.nx, A.ny, A.nz);
    bool one = A.uni_in[tile] && (A.Un == A.Uin || A.uni_un[tile]);   // the same for every thread
    double un[5], u[5];
    if (one) {
        const long long o0 = G.act(nb[0] * tx, nb[1] * ty, nb[2] * tz);
        load_un(A, o0, un);   // before the vote: the result may be stored over it
#pragma unroll
        for (int q = 0; q < 5; ++q) u[q] = A.Uin[o0 + q];
        bool same = true;
        if (tid < 6) {   // the tile through face tid; beyond an outflow boundary this tile's own cells continue
            const int d = tid >> 1, n = d == 0 ? gx : (d == 1 ? gy : gz);
            const int t = d == 0 ? tx : (d == 1 ? ty : tz), len = d == 0 ? A.nx : (d == 1 ? A.ny : A.nz);
            const int p0 = d == 0 ? nb[0] : (d == 1 ? nb[1] : nb[2]);
            int p = p0 + (tid & 1 ? 1 : -1);
            const bool periodic = A.bc == BSN_BC_PERIODIC;
            if (p < 0 || p >= n) p = periodic ? (p < 0 ? n - 1 : 0) : p0;
            const int x = d == 0 ? p : nb[0], y = d == 1 ? p : nb[1], z = d == 2 ? p : nb[2];
            // a last tile narrower than the halo, on a periodic axis: the halo reaches past it
            same = A.uni_in[x + gx * (y + (long long)gy * z)] && !(periodic && p == n - 1 && len - p * t < BSN_NG);
            const long long o = G.act(x * tx, y * ty, z * tz);
#pragma unroll
            for (int q = 0; q < 5; ++q) same = same && same_bits(A.Uin[o + q], u[q]);
        }
        // a cell that the floors change differs from the ghosts copied from it,
        // which stay raw: at the grid's boundary it is not uniform gas
        const double raw[5] = {u[0], u[1], u[2], u[3], u[4]};
        typename P::real w[5], pr;
        P::stage(u, true, A, P::consts(A), w, pr);
#pragma unroll
        for (int q = 0; q < 5; ++q) same = same && same_bits(u[q], raw[q]);
        w[4] = pr;
        one = __syncthreads_and(same && calm(w));
    }
    if (!one) {
        if (tid == 0) A.list[atomicAdd(A.list_count, 1u)] = (int)tile;
        return;
    }
    const double dt = A.dt_dev ? *A.dt_dev : A.dt;
    const double cdt = A.stage == 2 ? 0.25 * dt : (A.stage == 3 ? (2.0 / 3.0) * dt : dt);
    const double none = (-(0.0) * A.idx - 0.0 * A.idy) - 0.0 * A.idz;   // the divergence of finite equal fluxes
    const double d[5] = {none, none, none, none, none};
    double w[5];
    rk_combine(A, u[0], u[1], u[2], u[3], u[4], un, d, dt, cdt, w);
    P::floor(w, A);
    const int row = 5 * min(tx, A.nx - nb[0] * tx), rows = min(ty, A.ny - nb[1] * ty),
              planes = min(tz, A.nz - nb[2] * tz);
    double* out = A.Uout + G.act(nb[0] * tx, nb[1] * ty, nb[2] * tz);
    int b = tid >> 5, c = 0;   // a warp per row: no division per word
    while (b >= rows) b -= rows, ++c;
    while (c < planes) {
        double* o = out + G.sy * b + G.sz * c;
        for (int i = tid & 31, q = (tid & 31) % 5; i < row; i += 32, q = q < 3 ? q + 2 : q - 3)   // q = i mod 5
            o[i] = q == 0 ? w[0] : (q == 1 ? w[1] : (q == 2 ? w[2] : (q == 3 ? w[3] : w[4])));
        for (b += 4; b >= rows; b -= rows) ++c;
    }
    if (tid == 0) {
        A.uni_out[tile] = 1;
        if (A.cfl_max) {
            const double s = f64::cfl_speed(w[0], w[1], w[2], w[3], w[4], A.g, A.gm1, A.idx, A.idy, A.idz);
            if (s != s) atomicOr(A.cfl_nan, 1u);
            else {
                const unsigned long long v = (unsigned long long)__double_as_longlong(fmax(0.0, s));
                if (v > *(volatile unsigned long long*)A.cfl_max) atomicMax(A.cfl_max, v);
            }
        }
    }
}

// Several grids (mesh levels or patches of any size) in one launch: their
// blocks form one list, level l owning entries [start[l], start[l+1]); a
// persistent grid of CTAs (as many as fit at once) walks the list, drawing
// blocks from an atomic queue when one is given.  Each level keeps its own
// arguments (states, dt, flux registers, boundary capture), so every block
// computes exactly what its level's own launch would.
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool LED = false>
__global__ void __launch_bounds__(NT, MINB) stage_kernel_batch(const __grid_constant__ f64::StageBatch B) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ double red[NT / 32];
    __shared__ unsigned int nanflag;
    if (B.lv[0].done_dev && *B.lv[0].done_dev) return;
    P::prologue(policy_smem<P, TX, TY, TZ>(smem_raw), B.lv[0], NT);
    const int total = B.start[B.nlev];
    __shared__ int next;
    for (int t = blockIdx.x;; t += gridDim.x) {
        if (B.queue) {   // draw the next block; read by all before any thread draws again
            if (threadIdx.x == 0) next = (int)atomicAdd(B.queue, 1u);
            __syncthreads();
            t = next;
        }
        if (t >= total) break;
        int l = 0;
        while (l + 1 < B.nlev && t >= B.start[l + 1]) ++l;
        const f64::StageArgs& A = B.lv[l];
        const int r = t - B.start[l], gx = B.gx[l], gy = B.gy[l];
        stage_block<P, TX, TY, TZ, NT, MINB, LED>(A, (r % gx) * TX, ((r / gx) % gy) * TY, (r / (gx * gy)) * TZ,
                                                  smem_raw, red, nanflag);
    }
}

template <class P, int TX, int TY, int TZ>
constexpr int smem_bytes() {
    using S = Shape<TX, TY, TZ>;
    return (P::kCols * S::NCROSS + 5 * S::NFACE) * (int)sizeof(typename P::real) + 16;
}

// Host: launch stage_kernel_batch for the levels in B with a persistent grid
// (at most as many CTAs as fit on the device at once).
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool LED>
bsn_status launch_batch_led(bsn_ctx* ctx, f64::StageBatch B, int smem, const char* name) {
    auto fn = stage_kernel_batch<P, TX, TY, TZ, NT, MINB, LED>;
    static int occ[64] = {0}, sms[64] = {0};
    const int dev = ctx->device & 63;
    if (!occ[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return cuda_check(ctx, e, "cudaFuncSetAttribute(stage_kernel_batch)");
        int o = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fn, NT, smem);
        if (e != cudaSuccess) return cuda_check(ctx, e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, ctx->device);
        if (e != cudaSuccess) return cuda_check(ctx, e, "cudaDeviceGetAttribute");
        occ[dev] = o < 1 ? 1 : o;
    }
    if (B.nlev < 1 || B.nlev > f64::MAXLEV) return set_err(ctx, BSN_ERR_ARG, "batch of %d levels", B.nlev);
    long long total = 0;
    for (int l = 0; l < B.nlev; ++l) {
        const f64::StageArgs& A = B.lv[l];
        long long gx = (A.nx + TX - 1) / TX, gy = (A.ny + TY - 1) / TY, gz = (A.nz + TZ - 1) / TZ;
        B.gx[l] = (int)gx;
        B.gy[l] = (int)gy;
        B.start[l] = (int)total;
        total += gx * gy * gz;
    }
    if (total > 0x7fffffffLL) return set_err(ctx, BSN_ERR_UNSUPPORTED, "too many blocks in one batch");
    B.start[B.nlev] = (int)total;
    long long grid = std::min<long long>(total, (long long)occ[dev] * sms[dev]);
    prof_begin(ctx);
    fn<<<(unsigned)grid, NT, smem, ctx->stream>>>(B);
    return launch_check(ctx, name);
}

// the ledger instantiation when any level keeps a mass ledger
template <class P, int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_batch(bsn_ctx* ctx, const f64::StageBatch& B, int smem, const char* name) {
    bool led = false;
    for (int l = 0; l < B.nlev && l < f64::MAXLEV; ++l) led = led || B.lv[l].ledger;
    return led ? launch_batch_led<P, TX, TY, TZ, NT, MINB, true>(ctx, B, smem, name)
               : launch_batch_led<P, TX, TY, TZ, NT, MINB, false>(ctx, B, smem, name);
}

// Host: one stage on one grid through stage_kernel (the ledger
// instantiation when A keeps a mass ledger); smem is the dynamic smem.
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool LED>
bsn_status launch_plain_led(bsn_ctx* ctx, const f64::StageArgs& A, int smem, const char* name) {
    auto fn = stage_kernel<P, TX, TY, TZ, NT, MINB, LED>;
    static bool attr_done[64] = {false};
    const int dev = ctx->device & 63;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return cuda_check(ctx, e, "cudaFuncSetAttribute(stage_kernel)");
        attr_done[dev] = true;
    }
    dim3 grid((A.nx + TX - 1) / TX, (A.ny + TY - 1) / TY, (A.nz + TZ - 1) / TZ);
    prof_begin(ctx);
    fn<<<grid, NT, smem, ctx->stream>>>(A);
    return launch_check(ctx, name);
}
template <class P, int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_plain(bsn_ctx* ctx, const f64::StageArgs& A, int smem, const char* name) {
    return A.ledger ? launch_plain_led<P, TX, TY, TZ, NT, MINB, true>(ctx, A, smem, name)
                    : launch_plain_led<P, TX, TY, TZ, NT, MINB, false>(ctx, A, smem, name);
}

// Host: the stage kernel over the blocks in A.list (a persistent grid).
template <class P, int TX, int TY, int TZ, int NT, int MINB, bool UNI = true>
bsn_status launch_list(bsn_ctx* ctx, const f64::StageArgs& A, int smem, const char* name) {
    auto fn = stage_kernel_list<P, TX, TY, TZ, NT, MINB, UNI>;
    static int slots[64] = {0};
    const int dev = ctx->device & 63;
    if (!slots[dev]) {
        int o = 0, sms = 0;
        BSN_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        BSN_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fn, NT, smem));
        BSN_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
        slots[dev] = (o < 1 ? 1 : o) * sms;
    }
    const long long tiles = (long long)((A.nx + TX - 1) / TX) * ((A.ny + TY - 1) / TY) * ((A.nz + TZ - 1) / TZ);
    prof_begin(ctx);
    fn<<<(unsigned)std::min<long long>(tiles, slots[dev]), NT, smem, ctx->stream>>>(A);
    return launch_check(ctx, name);
}

// Host: uniform_stage_kernel, which leaves A.list.
template <class P>
bsn_status launch_uniform(bsn_ctx* ctx, const f64::StageArgs& A, int tx, int ty, int tz) {
    const dim3 grid((A.nx + tx - 1) / tx, (A.ny + ty - 1) / ty, (A.nz + tz - 1) / tz);
    prof_begin(ctx);
    uniform_stage_kernel<P><<<grid, 128, 0, ctx->stream>>>(A, tx, ty, tz);
    return launch_check(ctx, "uniform_stage_kernel");
}

// Host: one stage on one grid through stage_kernel_tma when the grid
// qualifies (tma::build_maps); *used tells whether it was launched.
template <class P, int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_tma(bsn_ctx* ctx, const f64::StageArgs& A, const char* name, bool* used) {
    using TS = TmaSmem<P, TX, TY, TZ, NT, MINB>;
    using C = typename TS::C;
    *used = false;
    if constexpr (!TS::OK) return BSN_OK;
    if (A.ledger) return BSN_OK;   // the TMA kernel keeps no mass ledger
    tma::Maps M;
    if (!tma::build_maps(ctx, A, TX, TY, TZ, C::AY, C::AZ, C::YZ, C::ZY, M)) return BSN_OK;
    auto fn = stage_kernel_tma<P, TX, TY, TZ, NT, MINB>;
    static bool attr_done[64] = {false};
    const int dev = ctx->device & 63;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, TS::BYTES);
        if (e != cudaSuccess) return cuda_check(ctx, e, "cudaFuncSetAttribute(stage_kernel_tma)");
        attr_done[dev] = true;
    }
    dim3 grid(A.nx / TX, A.ny / TY, A.nz / TZ);
    prof_begin(ctx);
    fn<<<grid, NT, TS::BYTES, ctx->stream>>>(A, M);
    *used = true;
    ctx->tma_used_last = 1;
    return launch_check(ctx, name);
}

}  // namespace tile
}  // namespace bsn
