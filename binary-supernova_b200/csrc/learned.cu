// learned.cu -- the learned WENO-weight network: sample collection from the
// method's own runs, hand-written training kernels (forward, backward, Adam),
// BF16 tensor-core inference (mma.sync m16n8k16, FP32 accumulation) used by
// the learned stencil kernel, and a standalone evaluator for tests.
//
// Tensor-core choice: the network is tiny (K = 16/32, N = 32/8) and its output
// is consumed immediately by the same thread's reconstruction.  Warp-level
// mma.sync keeps the fragments in registers, and the accumulator fragment of
// one layer is the A fragment of the next without any data movement; tcgen05
// would need the activations in shared memory and the accumulators in TMEM,
// i.e. a shared-memory/TMEM round trip per layer per 128-row tile inside the
// stencil kernel.  Built with the fast-path flags (FMA, approximate div/sqrt).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "hydro_f64.cuh"
#include "learned.cuh"
#include "physics_f32.cuh"
#include "stage_f32.cuh"
#include "stage_launch.cuh"
#include "stage_tile.cuh"

namespace bsn {
namespace learned {

// ---------------------------------------------------------------------------
// reference WENO-Z weights in FP64 (src/weno5.jl:14-61) of one side
__device__ inline void wenoz_weights64(const double v[5], int side, double w[3]) {
    const double k = 13.0 / 12.0, q = 1.0 / 4.0;
    double b0, b1, b2, d0, d1, d2;
    if (side == 0) {
        b0 = k * sq(v[0] - 2.0 * v[1] + v[2]) + q * sq(v[0] - 4.0 * v[1] + 3.0 * v[2]);
        b1 = k * sq(v[1] - 2.0 * v[2] + v[3]) + q * sq(v[1] - v[3]);
        b2 = k * sq(v[2] - 2.0 * v[3] + v[4]) + q * sq(3.0 * v[2] - 4.0 * v[3] + v[4]);
        d0 = 1.0 / 10.0; d1 = 6.0 / 10.0; d2 = 3.0 / 10.0;
    } else {
        b0 = k * sq(v[0] - 2.0 * v[1] + v[2]) + q * sq(v[0] - v[2]);
        b1 = k * sq(v[1] - 2.0 * v[2] + v[3]) + q * sq(v[1] - 4.0 * v[2] + 3.0 * v[3]);
        b2 = k * sq(v[2] - 2.0 * v[3] + v[4]) + q * sq(3.0 * v[2] - 4.0 * v[3] + v[4]);
        d0 = 3.0 / 10.0; d1 = 6.0 / 10.0; d2 = 1.0 / 10.0;
    }
    const double eps = 1e-36;
    double tau = fabs(b0 - b2);
    double a0 = d0 * (1.0 + sq(tau / (eps + b0)));
    double a1 = d1 * (1.0 + sq(tau / (eps + b1)));
    double a2 = d2 * (1.0 + sq(tau / (eps + b2)));
    double s = a0 + a1 + a2;
    w[0] = a0 / s; w[1] = a1 / s; w[2] = a2 / s;
}

__device__ __forceinline__ uint32_t mix32(uint64_t x) {
    x ^= x >> 33; x *= 0xff51afd7ed558ccdull; x ^= x >> 33; x *= 0xc4ceb9fe1a85ec53ull; x ^= x >> 33;
    return (uint32_t)x;
}

// One thread per (interface, field): left and right stencils of the six
// cells around the interface, WENO-Z weights in FP64, normalised inputs;
// smooth stencils with a spread above rounding level are kept with
// probability 1/stride.
__global__ void collect_kernel(const double* U, int nx, int ny, int nz, int bc, double gm1, int stride,
                               unsigned long long seed, float* outL, float* outR, unsigned long long* count,
                               long long cap) {
    Geom G(nx, ny, nz);
    long long nfx = (long long)(nx + 1) * ny * nz, nfy = (long long)nx * (ny + 1) * nz,
              nfz = (long long)nx * ny * (nz + 1);
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long tot = 5 * (nfx + nfy + nfz);
    if (t >= tot) return;
    int fld = (int)(t % 5);
    long long f = t / 5;
    int d;
    if (f < nfx) d = 0;
    else if ((f -= nfx) < nfy) d = 1;
    else { f -= nfy; d = 2; }
    int ex = nx + (d == 0), ey = ny + (d == 1);
    int a = (int)(f % ex), b = (int)((f / ex) % ey), c = (int)(f / ((long long)ex * ey));
    // face between cells (p-1) and p along d, p = a/b/c: cells p-3 .. p+2
    double v[6];
    for (int s = 0; s < 6; ++s) {
        int o = s - 3;
        int p[3] = {a, b, c};
        p[d] += o;
        int n[3] = {nx, ny, nz};
        for (int ax = 0; ax < 3; ++ax) p[ax] = bc_map(p[ax], n[ax], bc);
        long long off = G.act(p[0], p[1], p[2]);
        if (fld < 4) v[s] = U[off + fld];
        else v[s] = f64::cell_pressure(U[off], U[off + 1], U[off + 2], U[off + 3], U[off + 4], gm1);
    }
    for (int side = 0; side < 2; ++side) {
        if (mix32(seed ^ (uint64_t)(2 * t + side)) % (uint32_t)stride != 0) continue;
        double s5[5];
        for (int i = 0; i < 5; ++i) s5[i] = v[i + side];
        double u[5];
        if (!normalise<double>(s5, side, u)) continue;
        // Stencils whose spread is at the rounding level of their values (or
        // so small that WENO-Z's 1e-36 epsilon sets the weights) reconstruct
        // to within that spread with any weights and their normalised shape
        // is noise: no information.  Constant stencils are among them.
        double cen = side == 0 ? s5[2] : s5[1], spread = 0.0;
        for (int i = 0; i < 5; ++i) spread = fmax(spread, fabs(s5[i] - cen));
        if (!(spread > (double)SPREAD_ABS && spread > SPREAD_REL_F64 * fabs(cen))) continue;
        double w[3];
        wenoz_weights64(s5, side, w);
        unsigned long long idx = atomicAdd(&count[side], 1ull);
        if ((long long)idx >= cap) continue;
        float* o = (side == 0 ? outL : outR) + (long long)idx * SAMPLE;
        for (int i = 0; i < 5; ++i) o[i] = (float)u[i];
        for (int i = 0; i < 3; ++i) o[5 + i] = (float)w[i];
    }
}

// ---------------------------------------------------------------------------
// training: one block of TB samples computes per-sample activations and
// deltas into shared memory, then the block's weight gradients as dot
// products over its samples, accumulated into `grad` with atomics.
constexpr int TB = 128;

__device__ __forceinline__ long long pick(unsigned long long seed, long long step, long long i, long long n,
                                          int random) {
    if (!random) return i;
    return (long long)((((uint64_t)mix32(seed ^ ((uint64_t)step << 32) ^ (uint64_t)i) << 32) |
                        (uint64_t)mix32(seed * 31ull + (uint64_t)i * 977ull + (uint64_t)step)) %
                       (uint64_t)n);
}

__global__ void __launch_bounds__(TB) train_grad_kernel(const float* samples, long long n, const float* P,
                                                        float* grad, double* loss, unsigned long long seed,
                                                        long long step, long long first, int random) {
    extern __shared__ float sm[];
    float* sP = sm;                          // NPARAM
    float* sU = sP + NPARAM;                 // NIN*TB
    float* sH1 = sU + NIN * TB;              // NH*TB
    float* sH2 = sH1 + NH * TB;              // NH*TB
    float* sDZ = sH2 + NH * TB;              // NOUT*TB
    float* sD2 = sDZ + NOUT * TB;            // NH*TB
    float* sD1 = sD2 + NH * TB;              // NH*TB
    __shared__ double sloss[TB / 32];
    const int t = threadIdx.x;
    for (int i = t; i < NPARAM; i += TB) sP[i] = P[i];
    __syncthreads();
    long long gi = first + (long long)blockIdx.x * TB + t;
    bool live = random ? true : gi < n;
    float u[NIN], tg[NOUT];
    if (live) {
        long long s = pick(seed, step, gi, n, random);
        const float* x = samples + s * SAMPLE;
        for (int i = 0; i < NIN; ++i) u[i] = x[i];
        for (int i = 0; i < NOUT; ++i) tg[i] = x[NIN + i];
    } else {
        for (int i = 0; i < NIN; ++i) u[i] = 0.f;
        for (int i = 0; i < NOUT; ++i) tg[i] = 0.f;
    }
    for (int i = 0; i < NIN; ++i) sU[i * TB + t] = live ? u[i] : 0.f;
    const float* W1 = sP + OFF_W1; const float* b1 = sP + OFF_B1;
    const float* W2 = sP + OFF_W2; const float* b2 = sP + OFF_B2;
    const float* W3 = sP + OFF_W3; const float* b3 = sP + OFF_B3;
    for (int j = 0; j < NH; ++j) {
        float z = b1[j];
        for (int i = 0; i < NIN; ++i) z = fmaf(W1[j * NIN + i], u[i], z);
        sH1[j * TB + t] = fmaxf(z, 0.f);
    }
    for (int j = 0; j < NH; ++j) {
        float z = b2[j];
        for (int i = 0; i < NH; ++i) z = fmaf(W2[j * NH + i], sH1[i * TB + t], z);
        sH2[j * TB + t] = fmaxf(z, 0.f);
    }
    float zo[NOUT], om[NOUT];
    float zmax = -1e30f;
    for (int k = 0; k < NOUT; ++k) {
        float z = b3[k];
        for (int i = 0; i < NH; ++i) z = fmaf(W3[k * NH + i], sH2[i * TB + t], z);
        zo[k] = z;
        zmax = fmaxf(zmax, z);
    }
    float es = 0.f;
    for (int k = 0; k < NOUT; ++k) { om[k] = expf(zo[k] - zmax); es += om[k]; }
    float lsum = 0.f, g[NOUT], gdot = 0.f;
    for (int k = 0; k < NOUT; ++k) {
        om[k] /= es;
        float e = om[k] - tg[k];
        lsum += e * e;
        g[k] = 2.f * e;
        gdot += om[k] * g[k];
    }
    for (int k = 0; k < NOUT; ++k) sDZ[k * TB + t] = live ? om[k] * (g[k] - gdot) : 0.f;
    for (int i = 0; i < NH; ++i) {
        float s = 0.f;
        for (int k = 0; k < NOUT; ++k) s = fmaf(W3[k * NH + i], sDZ[k * TB + t], s);
        sD2[i * TB + t] = sH2[i * TB + t] > 0.f ? s : 0.f;
    }
    for (int j = 0; j < NH; ++j) {
        float s = 0.f;
        for (int i = 0; i < NH; ++i) s = fmaf(W2[i * NH + j], sD2[i * TB + t], s);
        sD1[j * TB + t] = sH1[j * TB + t] > 0.f ? s : 0.f;
    }
    // block loss
    double lv = live ? (double)lsum : 0.0;
    for (int o = 16; o > 0; o >>= 1) lv += __shfl_xor_sync(0xffffffffu, lv, o);
    if ((t & 31) == 0) sloss[t >> 5] = lv;
    __syncthreads();
    if (t == 0) {
        double s = 0.0;
        for (int w = 0; w < TB / 32; ++w) s += sloss[w];
        atomicAdd(loss, s);
    }
    // weight gradients: dot products over the block's samples
    for (int e = t; e < NPARAM; e += TB) {
        const float *x, *y;
        if (e < OFF_B1) { int j = e / NIN, i = e % NIN; x = sD1 + j * TB; y = sU + i * TB; }
        else if (e < OFF_W2) { x = sD1 + (e - OFF_B1) * TB; y = nullptr; }
        else if (e < OFF_B2) { int r = e - OFF_W2, j = r / NH, i = r % NH; x = sD2 + j * TB; y = sH1 + i * TB; }
        else if (e < OFF_W3) { x = sD2 + (e - OFF_B2) * TB; y = nullptr; }
        else if (e < OFF_B3) { int r = e - OFF_W3, k = r / NH, i = r % NH; x = sDZ + k * TB; y = sH2 + i * TB; }
        else { x = sDZ + (e - OFF_B3) * TB; y = nullptr; }
        float s = 0.f;
        if (y) for (int b = 0; b < TB; ++b) s = fmaf(x[b], y[b], s);
        else for (int b = 0; b < TB; ++b) s += x[b];
        atomicAdd(&grad[e], s);
    }
}

__global__ void adam_kernel(float* P, float* grad, float* m, float* v, float scale, float lr, float b1, float b2,
                            float eps, float bc1, float bc2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NPARAM) return;
    float g = grad[i] * scale;
    m[i] = b1 * m[i] + (1.f - b1) * g;
    v[i] = b2 * v[i] + (1.f - b2) * g * g;
    float mh = m[i] / bc1, vh = v[i] / bc2;
    P[i] -= lr * mh / (sqrtf(vh) + eps);
    grad[i] = 0.f;
}

// ---------------------------------------------------------------------------
// BF16 tensor-core inference.  Packed parameters (per side), in the order the
// MMA fragments of lane (g, tg) = (lane / 4, lane % 4) read them, so that each
// lane loads a fragment set with one 16-byte shared-memory load and the 32
// lanes of a load read consecutive 16-byte words (no bank conflicts):
//   F1[lane][j]      layer-1 B fragment of output block j (m16n8k8: one word)
//   F2[j][lane][i]   layer-2 B fragments of block j, i = (k-step, half)
//   F3[lane][i]      layer-3 B fragments, i = (k-step, half)
//   FB1[tg][j][h], FB2[tg][j][h], FB3[tg][h]   the lane's bias pairs (FP32)
// A word holds two BF16 values (the lower k in the low half); rows are output
// units, zero padded (inputs 5 -> 8 for layer 1, outputs 3 -> 8 for layer 3).
constexpr int PK_F1 = 0, PK_F2 = PK_F1 + 32 * 4 * 4, PK_F3 = PK_F2 + 32 * 16 * 4, PK_B1 = PK_F3 + 32 * 4 * 4,
              PK_B2 = PK_B1 + 32 * 4, PK_B3 = PK_B2 + 32 * 4, PK_BYTES = PK_B3 + 8 * 4;   // bytes per side
static_assert(PK_F2 % 16 == 0 && PK_F3 % 16 == 0 && PK_B1 % 16 == 0 && PK_B2 % 16 == 0 && PK_B3 % 16 == 0 &&
                  PK_BYTES % 16 == 0, "16-byte fragment loads");

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

// layer weights (row n = output unit, column k = input) with the zero padding
__device__ __forceinline__ float w1_at(const float* P, int n, int k) { return k < NIN ? P[OFF_W1 + n * NIN + k] : 0.f; }
__device__ __forceinline__ float w2_at(const float* P, int n, int k) { return P[OFF_W2 + n * NH + k]; }
__device__ __forceinline__ float w3_at(const float* P, int n, int k) { return n < NOUT ? P[OFF_W3 + n * NH + k] : 0.f; }

__global__ void pack_kernel(const float* P, unsigned char* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t* F1 = (uint32_t*)(out + PK_F1);
    uint32_t* F2 = (uint32_t*)(out + PK_F2);
    uint32_t* F3 = (uint32_t*)(out + PK_F3);
    float* B1 = (float*)(out + PK_B1);
    float* B2 = (float*)(out + PK_B2);
    float* B3 = (float*)(out + PK_B3);
    // word w of a row covers k = 2w, 2w + 1; the lane's fragment words are
    // w = tg (layer 1) and w = tg, tg + 4, tg + 8, tg + 12 (k-steps 0 and 1)
    if (i < 32 * 4) {
        const int lane = i / 4, j = i % 4, g = lane / 4, tg = lane % 4, n = 8 * j + g;
        F1[i] = pack2(w1_at(P, n, 2 * tg), w1_at(P, n, 2 * tg + 1));
    }
    if (i < 32 * 16) {
        const int j = i / 128, lane = (i / 4) % 32, q = i % 4, g = lane / 4, tg = lane % 4, n = 8 * j + g;
        const int w = tg + 4 * q;
        F2[i] = pack2(w2_at(P, n, 2 * w), w2_at(P, n, 2 * w + 1));
    }
    if (i < 32 * 4) {
        const int lane = i / 4, q = i % 4, g = lane / 4, tg = lane % 4, w = tg + 4 * q;
        F3[i] = pack2(w3_at(P, g, 2 * w), w3_at(P, g, 2 * w + 1));
    }
    if (i < 32) {
        const int tg = i / 8, j = (i / 2) % 4, h = i % 2, n = 8 * j + 2 * tg + h;
        B1[i] = P[OFF_B1 + n];
        B2[i] = P[OFF_B2 + n];
    }
    if (i < 8) {
        const int tg = i / 2, h = i % 2, n = 2 * tg + h;
        B3[i] = n < NOUT ? P[OFF_B3 + n] : 0.f;
    }
}

// max(lo, 0), max(hi, 0) rounded to BF16 and packed (lo in the low half),
// one instruction: cvt.rn.relu.bf16x2.f32 puts its first source in the high half
__device__ __forceinline__ uint32_t pack2_relu(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// D = A B + C (m16n8k16, BF16 in, FP32 accumulate); C may be other registers
// than D (a bias as the initial accumulator without copying it first)
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c0,
                                         float c1, float c2, float c3) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    mma16816(c, a, b0, b1, c[0], c[1], c[2], c[3]);
}

// D = A B + C (m16n8k8)
__device__ __forceinline__ void mma1688(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, float c0, float c1,
                                        float c2, float c3) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%8,%9,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(b0), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// Warp-collective MLP over `ntiles` tiles of 16 rows.  rows: BF16 inputs,
// 8 per row (5 used, the rest zero), 16 B per row; the first layer is one
// k = 8 MMA per 8 outputs.  Logits of row r are written to out[4*r .. 4*r+2];
// out may alias rows (a tile's rows are in registers before its logits are
// stored, and tile t's logits land below tile t+1's rows).
__device__ __noinline__ void mlp_tiles(const unsigned char* pk, const uint32_t* rows, float* out, int ntiles) {
    const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
    const uint4* F1 = (const uint4*)(pk + PK_F1) + lane;          // words j = 0..3
    const uint4* F2 = (const uint4*)(pk + PK_F2) + lane;          // F2[32 j]: (k-step 0: lo, hi, k-step 1: lo, hi)
    const uint4* F3 = (const uint4*)(pk + PK_F3) + lane;
    const float4* B1 = (const float4*)(pk + PK_B1) + 2 * tg;      // (j, h) pairs, j = 0..3
    const float4* B2 = (const float4*)(pk + PK_B2) + 2 * tg;
    const float2* B3 = (const float2*)(pk + PK_B3) + tg;
    for (int tile = 0; tile < ntiles; ++tile) {
        int r0 = tile * 16 + g, r1 = r0 + 8;
        const uint32_t a0 = rows[r0 * 4 + tg], a1 = rows[r1 * 4 + tg];
        __syncwarp();
        // layer 1: 8 (5 used) -> 32, bias as the accumulator's initial value
        const uint4 w1 = *F1;
        const float4 b1a = B1[0], b1b = B1[1];
        const float b1[8] = {b1a.x, b1a.y, b1a.z, b1a.w, b1b.x, b1b.y, b1b.z, b1b.w};
        const uint32_t w1s[4] = {w1.x, w1.y, w1.z, w1.w};
        float h[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) mma1688(h[j], a0, a1, w1s[j], b1[2 * j], b1[2 * j + 1], b1[2 * j], b1[2 * j + 1]);
        // ReLU, BF16 and the A fragments of the next layer in one instruction per pair
        uint32_t a2[2][4];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            a2[kk][0] = pack2_relu(h[2 * kk][0], h[2 * kk][1]);
            a2[kk][1] = pack2_relu(h[2 * kk][2], h[2 * kk][3]);
            a2[kk][2] = pack2_relu(h[2 * kk + 1][0], h[2 * kk + 1][1]);
            a2[kk][3] = pack2_relu(h[2 * kk + 1][2], h[2 * kk + 1][3]);
        }
        // layer 2: 32 -> 32
        const float4 b2a = B2[0], b2b = B2[1];
        const float b2[8] = {b2a.x, b2a.y, b2a.z, b2a.w, b2b.x, b2b.y, b2b.z, b2b.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 w2 = F2[32 * j];
            mma16816(h[j], a2[0], w2.x, w2.y, b2[2 * j], b2[2 * j + 1], b2[2 * j], b2[2 * j + 1]);
            mma16816(h[j], a2[1], w2.z, w2.w);
        }
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            a2[kk][0] = pack2_relu(h[2 * kk][0], h[2 * kk][1]);
            a2[kk][1] = pack2_relu(h[2 * kk][2], h[2 * kk][3]);
            a2[kk][2] = pack2_relu(h[2 * kk + 1][0], h[2 * kk + 1][1]);
            a2[kk][3] = pack2_relu(h[2 * kk + 1][2], h[2 * kk + 1][3]);
        }
        // layer 3: 32 -> 8 (3 used)
        const uint4 w3 = *F3;
        const float2 b3 = *B3;
        float o[4];
        mma16816(o, a2[0], w3.x, w3.y, b3.x, b3.y, b3.x, b3.y);
        mma16816(o, a2[1], w3.z, w3.w);
        __syncwarp();
        if (tg == 0) {
            out[4 * r0 + 0] = o[0]; out[4 * r0 + 1] = o[1];
            out[4 * r1 + 0] = o[2]; out[4 * r1 + 1] = o[3];
        } else if (tg == 1) {
            out[4 * r0 + 2] = o[0];
            out[4 * r1 + 2] = o[2];
        }
        __syncwarp();
    }
}

__device__ __forceinline__ void softmax3(const float* z, float w[3]) {
    float m = fmaxf(fmaxf(z[0], z[1]), z[2]);
    float e0 = __expf(z[0] - m), e1 = __expf(z[1] - m), e2 = __expf(z[2] - m);
    float inv = 1.0f / (e0 + e1 + e2);
    w[0] = e0 * inv; w[1] = e1 * inv; w[2] = e2 * inv;
}

// FP32 CUDA-core forward (the training kernels' arithmetic), for checking.
__device__ void mlp_fp32(const float* P, const float u[5], float w[3]) {
    float h1[NH], h2[NH], z[NOUT];
    for (int j = 0; j < NH; ++j) {
        float s = P[OFF_B1 + j];
        for (int i = 0; i < NIN; ++i) s = fmaf(P[OFF_W1 + j * NIN + i], u[i], s);
        h1[j] = fmaxf(s, 0.f);
    }
    for (int j = 0; j < NH; ++j) {
        float s = P[OFF_B2 + j];
        for (int i = 0; i < NH; ++i) s = fmaf(P[OFF_W2 + j * NH + i], h1[i], s);
        h2[j] = fmaxf(s, 0.f);
    }
    for (int k = 0; k < NOUT; ++k) {
        float s = P[OFF_B3 + k];
        for (int i = 0; i < NH; ++i) s = fmaf(P[OFF_W3 + k * NH + i], h2[i], s);
        z[k] = s;
    }
    softmax3(z, w);
}

// Standalone evaluation of n normalised stencils: tc = 0 FP32 CUDA cores,
// tc = 1 the BF16 tensor-core path of the stencil kernel.
__global__ void eval_kernel(const float* u, long long n, const float* P, const unsigned char* pk, float* w, int tc) {
    __shared__ __align__(16) uint32_t rows[4][32 * 4];     // 32 rows per warp
    __shared__ __align__(16) unsigned char spk[PK_BYTES];
    __shared__ float logits[4][32 * 4];
    for (int i = threadIdx.x; i < PK_BYTES; i += blockDim.x) spk[i] = pk[i];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float x[5] = {0, 0, 0, 0, 0};
    if (i < n) for (int k = 0; k < 5; ++k) x[k] = u[i * 5 + k];
    if (!tc) {
        if (i < n) { float o[3]; mlp_fp32(P, x, o); for (int k = 0; k < 3; ++k) w[i * 3 + k] = o[k]; }
        return;
    }
    uint32_t* R = rows[warp];
    R[lane * 4 + 0] = pack2(x[0], x[1]);
    R[lane * 4 + 1] = pack2(x[2], x[3]);
    R[lane * 4 + 2] = pack2(x[4], 0.f);
    R[lane * 4 + 3] = 0u;
    __syncwarp();
    mlp_tiles(spk, R, logits[warp], 2);
    if (i < n) { float o[3]; softmax3(&logits[warp][4 * lane], o); for (int k = 0; k < 3; ++k) w[i * 3 + k] = o[k]; }
}

struct State {
    unsigned char* packed = nullptr;   // 2 sides * PK_BYTES, device
    bool ready = false;
};

}  // namespace learned

// ---------------------------------------------------------------------------
// the learned stencil policy: FP32 stencil physics whose WENO weights come
// from the network (BF16 tensor cores) where the stencil is smooth.
namespace tile {

template <bool PACKED>
struct F32LearnedT {
    static constexpr bool kDeferred = false;   // the warp path reconstructs all faces in FP32
    using real = float;
    static constexpr bool kCenterFromSmem = false;
    static constexpr bool kWarpFaces = true;
    static constexpr int kCols = 5;         // rho, m, P: the epilogue reloads the FP64 state
    // A sweep whose staged values all lie within a quarter of the network's
    // spread thresholds of the first one cannot hold a network row (every
    // stencil spread is at most twice that): its faces skip the fallback test.
    static constexpr bool kQuiescentSkip = true;
    static constexpr bool kScreen = false;
    __device__ static bool same(float v, float ref) {
        return fabsf(v - ref) <= fmaxf(0.25f * learned::SPREAD_ABS, 0.125f * learned::SPREAD_REL_F32 * fabsf(ref));
    }
    // packed parameters of both sides + per-warp row buffers (160 rows x 16 B)
    static constexpr int kExtraSmem(int nt) { return 2 * learned::PK_BYTES + (nt / 32) * 160 * 16; }
    struct Consts { float g, gm1, inv_gm1, gg; };
    __device__ static Consts consts(const f64::StageArgs& A) {
        float g = (float)A.g;
        return {g, (float)A.gm1, 1.0f / (float)A.gm1, (g + 1.0f) / (2.0f * g)};
    }
    __device__ static float pressure(const float v[5], const Consts& k) {
        return f32::cell_pressure(v[0], v[1], v[2], v[3], v[4], k.gm1);
    }
    __device__ static void floor(double (&v)[5], const f64::StageArgs& A) {
        f32::floor_screened(v, A.rho_floor, A.P_floor, A.Pfl_gm1, A.gm1);
    }
    static constexpr bool kOrdinary = false;
    __device__ static bool stage(double (&v)[5], bool act, const f64::StageArgs& A, const Consts& k, float (&w)[5],
                                 float& P) {
        f32::stage_floored(v, act, A.rho_floor, A.P_floor, A.Pfl_gm1, A.gm1, w);
        P = pressure(w, k);
        return true;
    }
    __device__ static void prologue(unsigned char* psm, const f64::StageArgs& A, int nt) {
        static_assert(learned::PK_BYTES % 16 == 0, "16-byte copies of the packed parameters");
        const uint4* src = (const uint4*)A.mlp;   // device allocation: 256-byte aligned
        uint4* dst = (uint4*)psm;                 // policy_smem: 16-byte aligned
        for (int i = threadIdx.x; i < 2 * learned::PK_BYTES / 16; i += nt) dst[i] = src[i];
    }
    // The FP32 path's end of a face: packed, or side by side with the same bits
    // and fewer registers live around the network's tiles.  Where every block
    // of the launch is one that the screen listed, side by side is faster:
    // learned steps without uniform gas, packed and so, 128x96x80 2.39 and 2.35
    // ms, 256^3 32.9 and 32.6, 48^3 0.439 and 0.443; over all blocks of a level
    // packed is: two levels of 64^3, eight steps, 10.67 and 10.80 ms.
    __device__ __forceinline__ static void finish(const float (&c)[6][6], const Consts& k, const float (&L)[5],
                                                  const float (&Rv)[5], float (&F)[5], int D) {
        if constexpr (PACKED) f32::finish_face(c, L, Rv, k.g, k.gm1, k.inv_gm1, k.gg, D, F);
        else finish_sides(c, k, L, Rv, F, D);
    }
    __device__ static void finish_sides(const float (&c)[6][6], const Consts& k, const float (&L)[5],
                                        const float (&Rv)[5], float (&F)[5], int D) {
        const float Pm = fmaxf(fmaxf(fmaxf(c[1][5], c[2][5]), c[3][5]), c[4][5]);
        const float PL = fminf(fmaxf(L[4], 0.0f), fmaxf(c[0][5], Pm)), PR = fminf(fmaxf(Rv[4], 0.0f), fmaxf(Pm, c[5][5]));
        const float EL = f32::EL_from_P(PL, L[0], L[1], L[2], L[3], k.inv_gm1);
        const float ER = f32::EL_from_P(PR, Rv[0], Rv[1], Rv[2], Rv[3], k.inv_gm1);
        // (normal, t1, t2) = (x, y, z), (y, x, z), (z, x, y)
        float Fr[5];
        f32::hllc_normal(L[0], D == 0 ? L[1] : (D == 1 ? L[2] : L[3]), D == 0 ? L[2] : L[1], D == 2 ? L[2] : L[3], EL,
                         Rv[0], D == 0 ? Rv[1] : (D == 1 ? Rv[2] : Rv[3]), D == 0 ? Rv[2] : Rv[1],
                         D == 2 ? Rv[2] : Rv[3], ER, k.g, k.gm1, k.gg, Fr);
        F[0] = Fr[0];
        F[1] = D == 0 ? Fr[1] : Fr[2];
        F[2] = D == 0 ? Fr[2] : (D == 1 ? Fr[1] : Fr[3]);
        F[3] = D == 2 ? Fr[1] : Fr[3];
        F[4] = Fr[4];
    }
    // One interface per lane; every lane of the warp calls this (valid or not).
    // c[cell][col]: cols 0-3 rho, m_x, m_y, m_z, col 4 E, col 5 P; the
    // reconstructed fields are rho, m and P (cols 0-3 and 5), as the
    // reference's (src/gpu_kernels.jl:61-80).
    //
    // Every reconstruction first takes the FP32 WENO5-Z value (the fallback),
    // sharing candidates and smoothness indicators between the left and right
    // stencils exactly as the FP32 path does.  The network replaces it where
    // the stencil is smooth and not constant: the test tau <= THETA (min beta
    // + BETA_EPS) on the normalised stencil u = (v - v_c)/s is evaluated on
    // the raw indicators (beta scales with s^2), so only network rows pay
    // for the normalisation; the spread s must also exceed SPREAD_ABS and
    // SPREAD_REL_F32 |v_c|.  Network rows are compacted over the warp
    // (prefix sum of the lanes' counts), one side at a time, so the tensor
    // cores run ceil(rows / 16) tiles and none when the warp's stencils are
    // all quiescent or shocked.
    // Inlined into each sweep (D is a constant after inlining): an out-of-line
    // copy shrinks the kernel's code but passes the stencil and the caller's
    // live registers through local memory on every call, which costs more
    // than it saves where most sweeps are non-uniform (inside a star).
    __device__ __forceinline__ static void warp_flux(const float (&c)[6][6], bool valid, const Consts& k, float (&F)[5],
                                                     unsigned char* psm, int warp, bool quiet, int D) {
        const int lane = threadIdx.x & 31;
        uint32_t* R = (uint32_t*)(psm + 2 * learned::PK_BYTES + warp * 160 * 16);
        float* logit = (float*)R;
        const float t13 = 1.0f / 3.0f, m76 = -7.0f / 6.0f, e116 = 11.0f / 6.0f, m16 = -1.0f / 6.0f,
                    f56 = 5.0f / 6.0f;
        float L[5], Rv[5];
        unsigned need[2] = {0u, 0u};
        // the smoothness test of field q from its stencil and indicators
        auto test = [&](int q, float c0, float c1, float c2, float c3, float c4, float c5, float bA, float bB,
                        float bC, float bD, float bE) {
            // spreads about the common centre c2: left stencil c0..c4, right c1..c5
            float m14 = fmaxf(fmaxf(fabsf(c1 - c2), fabsf(c3 - c2)), fabsf(c4 - c2));
            float sL = fmaxf(m14, fabsf(c0 - c2)), sR = fmaxf(m14, fabsf(c5 - c2));
            bool smL = fabsf(bA - bC) <= learned::THETA * fmaf(learned::BETA_EPS * sL, sL, fminf(fminf(bA, bB), bC));
            bool smR = fabsf(bB - bE) <= learned::THETA * fmaf(learned::BETA_EPS * sR, sR, fminf(fminf(bB, bD), bE));
            // spreads at FP32 rounding level of the centre value (or below
            // WENO-Z's epsilon scale) carry no shape: WENO-Z stays.  This
            // also keeps the network off the 1e-30-level precursor noise that
            // upwind stencils leave ahead of a shock.
            const float smin = fmaxf(learned::SPREAD_ABS, learned::SPREAD_REL_F32 * fabsf(c2));
            need[0] |= (unsigned)(smL && sL > smin) << q;
            need[1] |= (unsigned)(smR && sR > smin) << q;
        };
        // rho, m_x and m_y, m_z in packed pairs (f32x2), P alone
#pragma unroll
        for (int q = 0; q < 4; q += 2) {
            float v[6][2];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                v[i][0] = valid ? c[i][q] : 0.f;
                v[i][1] = valid ? c[i][q + 1] : 0.f;
            }
            f32::f2 L2, R2, bA, bB, bC, bD, bE;
            f32::weno5_lr2(f32::pk2(v[0][0], v[0][1]), f32::pk2(v[1][0], v[1][1]), f32::pk2(v[2][0], v[2][1]),
                           f32::pk2(v[3][0], v[3][1]), f32::pk2(v[4][0], v[4][1]), f32::pk2(v[5][0], v[5][1]), L2,
                           R2, bA, bB, bC, bD, bE);
            f32::up2(L2, L[q], L[q + 1]);
            f32::up2(R2, Rv[q], Rv[q + 1]);
            if (quiet) continue;   // block-uniform
            float A[2], B[2], C[2], Dd[2], E[2];
            f32::up2(bA, A[0], A[1]);
            f32::up2(bB, B[0], B[1]);
            f32::up2(bC, C[0], C[1]);
            f32::up2(bD, Dd[0], Dd[1]);
            f32::up2(bE, E[0], E[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                test(q + h, v[0][h], v[1][h], v[2][h], v[3][h], v[4][h], v[5][h], A[h], B[h], C[h], Dd[h], E[h]);
        }
        {
            const int q = 4, col = 5;
            float c0 = c[0][col], c1 = c[1][col], c2 = c[2][col], c3 = c[3][col], c4 = c[4][col], c5 = c[5][col];
            if (!valid) c0 = c1 = c2 = c3 = c4 = c5 = 0.f;
            float bA, bB, bC, bD, bE;
            f32::weno5_lr(c0, c1, c2, c3, c4, c5, L[q], Rv[q], bA, bB, bC, bD, bE);
            if (!quiet) test(q, c0, c1, c2, c3, c4, c5, bA, bB, bC, bD, bE);
        }
        if (quiet) return finish(c, k, L, Rv, F, D);
        // both sides' row counts in one prefix sum (8 bits each: at most 160 rows a side)
        const int packed = __popc(need[0]) | (__popc(need[1]) << 8);
        if (!__any_sync(0xffffffffu, packed != 0)) return finish(c, k, L, Rv, F, D);   // warp-uniform
        int incl = packed;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const int tot = __shfl_sync(0xffffffffu, incl, 31), excl = incl - packed;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const int total = (tot >> (8 * side)) & 255;
            if (total == 0) continue;   // warp-uniform
            const int base = (excl >> (8 * side)) & 255;
            int r = base;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                if (!((need[side] >> q) & 1u)) continue;
                const int col = q < 4 ? q : 5;
                const float vc = c[2][col];
                float u[5], sp = 0.f;
#pragma unroll
                for (int i = 0; i < 5; ++i) {
                    u[i] = c[i + side][col] - vc;
                    sp = fmaxf(sp, fabsf(u[i]));
                }
                const float inv = 1.0f / sp;
                *reinterpret_cast<uint4*>(R + r * 4) =
                    make_uint4(learned::pack2(u[0] * inv, u[1] * inv), learned::pack2(u[2] * inv, u[3] * inv),
                               learned::pack2(u[4] * inv, 0.f), 0u);
                ++r;
            }
            const int ntiles = (total + 15) >> 4;
            for (int rr = total + lane; rr < ntiles * 16; rr += 32)
                *reinterpret_cast<uint4*>(R + rr * 4) = make_uint4(0u, 0u, 0u, 0u);
            __syncwarp();
            learned::mlp_tiles(psm + side * learned::PK_BYTES, R, logit, ntiles);
            r = base;
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                if (!((need[side] >> q) & 1u)) continue;
                const int col = q < 4 ? q : 5;
                float w[3];
                const float4 z = *reinterpret_cast<const float4*>(logit + 4 * r);
                const float zz[3] = {z.x, z.y, z.z};
                learned::softmax3(zz, w);
                ++r;
                const float v0 = c[side][col], v1 = c[side + 1][col], v2 = c[side + 2][col], v3 = c[side + 3][col],
                            v4 = c[side + 4][col];
                float qa, qb, qc;
                if (side == 0) {   // the candidate polynomials of weno5_lr (qA, qB, qC)
                    qa = fmaf(e116, v2, fmaf(m76, v1, t13 * v0));
                    qb = fmaf(t13, v3, fmaf(f56, v2, m16 * v1));
                    qc = fmaf(m16, v4, fmaf(f56, v3, t13 * v2));
                    L[q] = fmaf(w[0], qa, fmaf(w[1], qb, w[2] * qc));
                } else {           // (qB, qC, qD)
                    qa = fmaf(t13, v2, fmaf(f56, v1, m16 * v0));
                    qb = fmaf(m16, v3, fmaf(f56, v2, t13 * v1));
                    qc = fmaf(t13, v4, fmaf(m76, v3, e116 * v2));
                    Rv[q] = fmaf(w[0], qa, fmaf(w[1], qb, w[2] * qc));
                }
            }
            __syncwarp();
        }
        finish(c, k, L, Rv, F, D);
    }
    // uniform sweeps (kQuiescentSkip): no network row can occur, plain FP32 WENO5-Z + HLLC
    __device__ __forceinline__ static bool flux(const float (&c)[6][6], const Consts& k, int D, float F[5]) {
        f32::interface_flux(c, k.g, k.gm1, k.inv_gm1, k.gg, D, F);
        return false;
    }
};
using F32Learned = F32LearnedT<true>;
using F32LearnedListed = F32LearnedT<false>;

// The screening launch of the learned stage: the FP32 path's plain stencils
// for every block whose three sweeps are uniform by F32Learned's test (no
// network row can occur there, so the learned stage computes the same
// fluxes), listing the other blocks for the learned launch.
struct F32Screen : F32Physics {
    static constexpr bool kQuiescentSkip = true;
    static constexpr bool kScreen = true;
    __device__ static bool same(float v, float ref) { return F32Learned::same(v, ref); }
};

}  // namespace tile

namespace {
const TileVariant kLearnedVariants[] = {{8, 8, 8, 256, 2}, {16, 8, 4, 256, 2}, {8, 8, 8, 256, 3}, {8, 8, 4, 128, 6},
                                        {16, 16, 4, 256, 2}, {16, 8, 8, 256, 2}, {16, 16, 8, 512, 1}};

// One learned stage over every block in one launch (FMR levels and the
// coupled loops, whose grids are mostly non-uniform).
template <int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_learned_whole(bsn_ctx* ctx, const f64::StageArgs& A) {
    constexpr int smem = tile::smem_bytes<tile::F32Learned, TX, TY, TZ>() + tile::F32Learned::kExtraSmem(NT) + 16;
    return tile::launch_plain<tile::F32Learned, TX, TY, TZ, NT, MINB>(ctx, A, smem, "stage_kernel_learned");
}

// One learned stage as two launches on the context's stream: the screening
// launch over every block, then the learned launch over the blocks it listed
// (a persistent grid); 95-97 % of the Sedov blocks take the first.  Used where
// the caller asks for it (A.learned_split: the uniform-grid entry points).
template <int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_learned(bsn_ctx* ctx, const f64::StageArgs& A0) {
    if (!A0.learned_split) return launch_learned_whole<TX, TY, TZ, NT, MINB>(ctx, A0);
    constexpr int smem_s = tile::smem_bytes<tile::F32Screen, TX, TY, TZ>();
    constexpr int smem_l = tile::smem_bytes<tile::F32Learned, TX, TY, TZ>() + tile::F32Learned::kExtraSmem(NT) + 16;
    static_assert(smem_s <= 232448 && smem_l <= 232448, "tile's shared memory exceeds the per-CTA limit");
    bsn_status st;
    // sized for every variant before any graph capture (stage_autotune), so this never allocates while capturing
    unsigned int* cnt = (unsigned int*)slot(ctx, SLOT_SPLIT, learned_split_bytes(A0.nx, A0.ny, A0.nz), &st);
    BSN_TRY(st);
    f64::StageArgs A = A0;
    A.split_count = cnt;
    A.split_list = (int*)(cnt + 4);
    BSN_CUDA(ctx, cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned int), ctx->stream));   // list count, queue counter
    // the screening launch stages with the plain loader (its TMA form is not used)
    if (A.uni_in) {
        BSN_TRY(tile::launch_uniform<tile::F32Screen>(ctx, A, TX, TY, TZ));
        BSN_TRY((tile::launch_list<tile::F32Screen, TX, TY, TZ, NT, MINB>(ctx, A, smem_s, "stage_kernel_learned_screen")));
    } else {
        BSN_TRY((tile::launch_plain_led<tile::F32Screen, TX, TY, TZ, NT, MINB, false>(ctx, A, smem_s,
                                                                                     "stage_kernel_learned_screen")));
    }
    A.list = A.split_list;
    A.list_count = A.split_count;
    return tile::launch_list<tile::F32LearnedListed, TX, TY, TZ, NT, MINB, false>(ctx, A, smem_l, "stage_kernel_learned");
}
}  // namespace

int learned_variant_count() { return (int)(sizeof(kLearnedVariants) / sizeof(kLearnedVariants[0])); }
size_t learned_split_bytes(int nx, int ny, int nz) {
    long long mx = 0;
    for (const TileVariant& t : kLearnedVariants)
        mx = std::max(mx, (long long)((nx + t.tx - 1) / t.tx) * ((ny + t.ty - 1) / t.ty) * ((nz + t.tz - 1) / t.tz));
    return 16 + sizeof(int) * (size_t)mx;
}
TileVariant learned_variant(int idx) { return kLearnedVariants[idx]; }
bsn_status learned_launch_variant(bsn_ctx* ctx, int idx, const f64::StageArgs& A0) {
    learned::State* S = (learned::State*)ctx->learned_state;
    if (!S || !S->ready) return set_err(ctx, BSN_ERR_ARG, "no learned WENO weights set (bsn_learned_set_params)");
    f64::StageArgs A = A0;
    A.mlp = S->packed;
    switch (idx) {
        case 0: return launch_learned<8, 8, 8, 256, 2>(ctx, A);
        case 1: return launch_learned<16, 8, 4, 256, 2>(ctx, A);
        case 2: return launch_learned<8, 8, 8, 256, 3>(ctx, A);    // register-capped for 3 CTAs per SM
        case 3: return launch_learned<8, 8, 4, 128, 6>(ctx, A);
        case 4: return launch_learned<16, 16, 4, 256, 2>(ctx, A);
        case 5: return launch_learned<16, 8, 8, 256, 2>(ctx, A);
        case 6: return launch_learned<16, 16, 8, 512, 1>(ctx, A);
        default: return set_err(ctx, BSN_ERR_ARG, "no learned tile variant %d", idx);
    }
}

bsn_status learned_launch_batch_variant(bsn_ctx* ctx, int idx, const f64::StageBatch& B0) {
    learned::State* S = (learned::State*)ctx->learned_state;
    if (!S || !S->ready) return set_err(ctx, BSN_ERR_ARG, "no learned WENO weights set (bsn_learned_set_params)");
    f64::StageBatch B = B0;
    for (int l = 0; l < B.nlev; ++l) B.lv[l].mlp = S->packed;
    using P = tile::F32Learned;
    const char* nm = "stage_kernel_batch_learned";
    auto sm = [](int base, int nt) { return base + P::kExtraSmem(nt) + 16; };
    switch (idx) {
        case 0: return tile::launch_batch<P, 8, 8, 8, 256, 2>(ctx, B, sm(tile::smem_bytes<P, 8, 8, 8>(), 256), nm);
        case 1: return tile::launch_batch<P, 16, 8, 4, 256, 2>(ctx, B, sm(tile::smem_bytes<P, 16, 8, 4>(), 256), nm);
        case 2: return tile::launch_batch<P, 8, 8, 8, 256, 3>(ctx, B, sm(tile::smem_bytes<P, 8, 8, 8>(), 256), nm);
        case 3: return tile::launch_batch<P, 8, 8, 4, 128, 6>(ctx, B, sm(tile::smem_bytes<P, 8, 8, 4>(), 128), nm);
        case 4: return tile::launch_batch<P, 16, 16, 4, 256, 2>(ctx, B, sm(tile::smem_bytes<P, 16, 16, 4>(), 256), nm);
        case 5: return tile::launch_batch<P, 16, 8, 8, 256, 2>(ctx, B, sm(tile::smem_bytes<P, 16, 8, 8>(), 256), nm);
        case 6: return tile::launch_batch<P, 16, 16, 8, 512, 1>(ctx, B, sm(tile::smem_bytes<P, 16, 16, 8>(), 512), nm);
        default: return set_err(ctx, BSN_ERR_ARG, "no learned tile variant %d", idx);
    }
}

void learned_state_free(bsn_ctx* ctx) {
    if (!ctx->learned_state) return;
    learned::State* S = (learned::State*)ctx->learned_state;
    if (S->packed) cudaFree(S->packed);
    delete S;
    ctx->learned_state = nullptr;
}

}  // namespace bsn

using namespace bsn;
using namespace bsn::learned;

extern "C" int bsn_learned_param_count(void) { return NPARAM; }

extern "C" bsn_status bsn_learned_collect(bsn_ctx* ctx, const double* U, int nx, int ny, int nz, int bc, double gamma,
                                          int stride, unsigned long long seed, float* out_left, float* out_right,
                                          long long cap, long long counts[2]) {
    BSN_TRY(check_dims(ctx, nx, ny, nz));
    if (!U || !out_left || !out_right || !counts || stride < 1 || cap < 0)
        return set_err(ctx, BSN_ERR_ARG, "bad arguments to bsn_learned_collect");
    bsn_status st;
    unsigned long long* cnt = (unsigned long long*)slot(ctx, SLOT_RED, 64, &st); BSN_TRY(st);
    // resume counting from the caller's counts (appending to the buffers)
    unsigned long long h0[2] = {(unsigned long long)counts[0], (unsigned long long)counts[1]};
    BSN_CUDA(ctx, cudaMemcpyAsync(cnt, h0, 16, cudaMemcpyHostToDevice, ctx->stream));
    long long tot = 5LL * ((long long)(nx + 1) * ny * nz + (long long)nx * (ny + 1) * nz + (long long)nx * ny * (nz + 1));
    collect_kernel<<<grid1d(tot, 256), 256, 0, ctx->stream>>>(U, nx, ny, nz, bc, gamma - 1.0, stride, seed, out_left,
                                                              out_right, cnt, cap);
    BSN_TRY(launch_check(ctx, "collect_kernel"));
    unsigned long long h[2];
    BSN_CUDA(ctx, cudaMemcpyAsync(h, cnt, 16, cudaMemcpyDeviceToHost, ctx->stream));
    BSN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    counts[0] = (long long)h[0];   // offered; the buffers hold the first min(count, cap)
    counts[1] = (long long)h[1];
    return BSN_OK;
}

static size_t train_smem() { return sizeof(float) * (NPARAM + (NIN + 4 * NH + NOUT) * TB); }

extern "C" bsn_status bsn_learned_grad(bsn_ctx* ctx, const float* samples, long long n, const float* params,
                                       float* grad, double* loss) {
    if (!ctx || !samples || !params || !grad || !loss || n < 1) return BSN_ERR_ARG;
    bsn_status st;
    double* dl = (double*)slot(ctx, SLOT_RED, 64, &st); BSN_TRY(st);
    BSN_CUDA(ctx, cudaMemsetAsync(dl, 0, 8, ctx->stream));
    BSN_CUDA(ctx, cudaMemsetAsync(grad, 0, sizeof(float) * NPARAM, ctx->stream));
    BSN_CUDA(ctx, cudaFuncSetAttribute(train_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem()));
    train_grad_kernel<<<grid1d(n, TB), TB, train_smem(), ctx->stream>>>(samples, n, params, grad, dl, 0ull, 0, 0, 0);
    BSN_TRY(launch_check(ctx, "train_grad_kernel"));
    BSN_CUDA(ctx, cudaMemcpyAsync(loss, dl, 8, cudaMemcpyDeviceToHost, ctx->stream));
    BSN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return BSN_OK;
}

// Adam on mini-batches drawn uniformly (with replacement) from the samples,
// learning rate decayed from lr to 0 along a cosine over the steps.
extern "C" bsn_status bsn_learned_train(bsn_ctx* ctx, const float* samples, long long n, float* params, int steps,
                                        int batch, float lr, unsigned long long seed, double* last_loss) {
    if (!ctx || !samples || !params || n < 1 || steps < 0 || batch < TB || batch % TB)
        return set_err(ctx, BSN_ERR_ARG, "bad arguments to bsn_learned_train (batch must be a multiple of %d)", TB);
    bsn_status st;
    float* buf = (float*)slot(ctx, SLOT_UN, sizeof(float) * 3 * NPARAM + 64, &st); BSN_TRY(st);
    float *grad = buf, *m = buf + NPARAM, *v = buf + 2 * NPARAM;
    double* dl = (double*)slot(ctx, SLOT_RED, 64, &st); BSN_TRY(st);
    BSN_CUDA(ctx, cudaMemsetAsync(buf, 0, sizeof(float) * 3 * NPARAM, ctx->stream));
    BSN_CUDA(ctx, cudaFuncSetAttribute(train_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem()));
    const float b1 = 0.9f, b2 = 0.999f;
    double bc1 = 1.0, bc2 = 1.0;
    for (int s = 0; s < steps; ++s) {
        bool last = s == steps - 1;
        if (last) BSN_CUDA(ctx, cudaMemsetAsync(dl, 0, 8, ctx->stream));
        train_grad_kernel<<<batch / TB, TB, train_smem(), ctx->stream>>>(samples, n, params, grad, dl, seed, s, 0, 1);
        BSN_TRY(launch_check(ctx, "train_grad_kernel"));
        bc1 *= b1; bc2 *= b2;
        float lr_s = (float)(0.5 * lr * (1.0 + std::cos(3.14159265358979323846 * (double)s / (double)steps)));
        adam_kernel<<<(NPARAM + 255) / 256, 256, 0, ctx->stream>>>(params, grad, m, v, 1.0f / (float)batch, lr_s, b1,
                                                                    b2, 1e-8f, (float)(1.0 - bc1), (float)(1.0 - bc2));
        BSN_TRY(launch_check(ctx, "adam_kernel"));
    }
    if (last_loss) {
        double h = 0.0;
        BSN_CUDA(ctx, cudaMemcpyAsync(&h, dl, 8, cudaMemcpyDeviceToHost, ctx->stream));
        BSN_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        *last_loss = steps > 0 ? h / (double)batch : 0.0;
    }
    return BSN_OK;
}

// params_left/right: device FP32 parameters; packed to BF16 for the tensor cores
extern "C" bsn_status bsn_learned_set_params(bsn_ctx* ctx, const float* params_left, const float* params_right) {
    if (!ctx || !params_left || !params_right) return BSN_ERR_ARG;
    if (!ctx->learned_state) ctx->learned_state = new learned::State();
    learned::State* S = (learned::State*)ctx->learned_state;
    if (!S->packed) BSN_CUDA(ctx, cudaMalloc(&S->packed, 2 * PK_BYTES));
    pack_kernel<<<4, 256, 0, ctx->stream>>>(params_left, S->packed);
    BSN_TRY(launch_check(ctx, "pack_kernel"));
    pack_kernel<<<4, 256, 0, ctx->stream>>>(params_right, S->packed + PK_BYTES);
    BSN_TRY(launch_check(ctx, "pack_kernel"));
    S->ready = true;
    return BSN_OK;
}

extern "C" bsn_status bsn_learned_eval(bsn_ctx* ctx, const float* u, long long n, const float* params, float* w,
                                       int tensor_cores) {
    if (!ctx || !u || !params || !w || n < 0) return BSN_ERR_ARG;
    bsn_status st;
    unsigned char* pk = (unsigned char*)slot(ctx, SLOT_PHI2, PK_BYTES, &st); BSN_TRY(st);
    pack_kernel<<<4, 256, 0, ctx->stream>>>(params, pk);
    BSN_TRY(launch_check(ctx, "pack_kernel"));
    eval_kernel<<<grid1d(n, 128), 128, 0, ctx->stream>>>(u, n, params, pk, w, tensor_cores);
    return launch_check(ctx, "eval_kernel");
}
