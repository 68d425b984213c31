// hydro_f64.cuh -- internal interface of the FP64 uniform-grid path, shared by
// the coupled step, self-gravity and FMR drivers.
#pragma once

#include <cmath>
#include <cstring>
#include <algorithm>
#include <string>

#include "stage_f64.cuh"

namespace bsn {

bsn_status check_dims(bsn_ctx* ctx, int nx, int ny, int nz);
bsn_status f64_fill_ghosts(bsn_ctx* ctx, double* U, int nx, int ny, int nz, int bc);
// Cells of a half-open box [lo, hi) of active indices (lo = hi: none).
struct LedBox {
    int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    __host__ __device__ bool has(int a, int b, int c) const {
        return a >= lo[0] && a < hi[0] && b >= lo[1] && b < hi[1] && c >= lo[2] && c < hi[2];
    }
};
// apply_floors_3d! on the active cells; with led, the floors' change of the
// mass outside `skip` (rho dV, dV the cell volume) is added to *led.
bsn_status f64_floors(bsn_ctx* ctx, double* U, int nx, int ny, int nz, double rho_floor, double P_floor, double gamma,
                      const int* done_dev = nullptr, double* led = nullptr, LedBox skip = LedBox{}, double dV = 0.0);
// Fold one RK3 step's per-stage mass-ledger sums raw[3][LED_TERMS] into the
// cumulative totals tot[LEDT_COUNT] with the step's dt (hydro_f64.cu).
bsn_status f64_ledger_fold(bsn_ctx* ctx, double* raw, double* tot, const double* dt_dev, const int* done_dev);
bsn_status f64_ghost_combine(bsn_ctx* ctx, double* U, const double* S, const double* Gh, int nx, int ny, int nz,
                             int bc, double dt, const double* dt_dev = nullptr, const int* done_dev = nullptr);
void stage_args_init(f64::StageArgs& A, int nx, int ny, int nz, double dx, double dy, double dz, double gamma, int bc,
                     double rho_floor, double P_floor);
void set_stage(f64::StageArgs& A, int stage, double dt);
bsn_status f64_launch_stage(bsn_ctx* ctx, const f64::StageArgs& A);
bsn_status f64_rk3(bsn_ctx* ctx, f64::StageArgs base, double* U, double dt, const double* phi_per_stage[3],
                   unsigned long long* cfl_max, unsigned int* cfl_nan);
bsn_status f64_cfl_dt(bsn_ctx* ctx, const double* U, int nx, int ny, int nz, double dx, double dy, double dz,
                      double gamma, double cfl, double* dt_out);
bsn_status f64_cfl_fold(bsn_ctx* ctx, const double* U, int nx, int ny, int nz, double dx, double dy, double dz,
                        double gamma, unsigned long long* smax, unsigned int* nanflag);
bsn_status cfl_from_device(bsn_ctx* ctx, const unsigned long long* red, double cfl, double* dt_out);
// Replay a one-step graph up to n_steps times on ctx->stream.  With
// until_done, replays go in chunks and stop once the device flag *done_dev
// is set (each chunk's flag is read back behind it; the host waits for the
// previous chunk's flag only after queueing the next).  ev: two events,
// hflag: two pinned ints.
bsn_status graph_replay(bsn_ctx* ctx, cudaGraphExec_t exec, int kernels, int n_steps, bool until_done,
                        const int* done_dev, cudaEvent_t ev[2], volatile int* hflag);

// Steps that a first call takes as plain launches instead of capturing a
// graph.  A capture costs host time (130 us for the uniform loop, 190 for the
// coupled and two-level loops, 400 for three nested levels), and every step of
// plain launches leaves longer gaps between its kernels, so few steps are
// cheaper without and many with one.  Calls on two buffers in turn, captured
// and direct, us (B200): uniform loop, FP32 48^3, 1 / 4 / 8 / 12 steps, 267 /
// 522 / 857 / 1182 and 133 / 406 / 770 / 1131, 128^3 4 / 6 steps 2804 / 4145
// and 2819 / 4179; coupled 64^3 FP64 2 / 4 / 6 steps 1705 / 3049 / 4415 and
// 1582 / 3038 / 4494, 128^3 FP32 1 / 2 / 3 steps 2495 / 4758 / 7045 and 2450 /
// 4772 / 7110; two levels 32^3 2 / 3 / 4 steps 924 / 1248 / 1573 and 828 / 1220
// / 1600; three nested levels of the binary 64^3 1 / 2 / 3 steps 3306 / 6312 /
// 9378 and 3114 / 6314 / 9597.  A second call in a row with the same key
// (graph_key) captures whatever its steps: a program that advances one state
// by a step or two per call replays its graph from the third call on.
constexpr int kDirectUniform = 4;   // the uniform loop: some ten kernels a step
constexpr int kDirectMany = 2;      // the other loops: 40 to 120
// What a captured step holds, as bytes: the same bytes, the same step.
template <class... T>
std::string graph_key(const T&... v) {
    std::string k;
    (k.append((const char*)&v, sizeof(v)), ...);
    return k;
}
template <class F>
bsn_status launch_steps(bsn_ctx* ctx, F&& body, int n_steps) {
    const bool prof = ctx->profiling;   // as the graphs, outside the per-kernel records
    ctx->profiling = false;
    bsn_status st = BSN_OK;
    for (int i = 0; i < n_steps && st == BSN_OK; ++i) st = body();
    ctx->profiling = prof;
    return st;
}

// r_sink / t_sink of src/BinarySupernova.jl:159-171 (host FP64).
inline double bh_r_sink(const bsn_bh& b) {
    double v = 6.0 * b.mass / (b.c_code * b.c_code);
    return jmax(v, b.r_floor);
}
inline double bh_t_sink(const bsn_bh& b, double f_sink) {
    double rs = bh_r_sink(b);
    double v_ff = std::sqrt(2.0 * b.mass / rs);
    return f_sink * rs / v_ff;
}

}  // namespace bsn
