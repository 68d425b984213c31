// autotune.cu -- picks the tile shape of the fused stage kernel per grid,
// and whether its block is staged by TMA copies or by the plain loader.
//
// On the first stage of a new (precision, driver class, nx, ny, nz) the
// autotuner launches
// every tile variant on stage-1 work (reading the caller's state, writing a
// scratch array), with each staging the grid allows, times two launches of
// each with CUDA events after one warm-up, and keeps the fastest for the life
// of the context (of steps that may list uniform tiles, the fastest with and
// without a list: follow).  Every variant and staging gives bit-identical results (FP64
// by the reference's arithmetic, FP32 by its written-out multiply-adds), so
// the choice never changes a result.  The choice is stored as a code: the
// variant index plus kTmaBit when the TMA form won.
#include <algorithm>

#include "hydro_f64.cuh"
#include "stage_launch.cuh"

namespace bsn {

static int variant_count(int prec) {
    return prec == PREC_F64 ? f64_variant_count() : (prec == PREC_F32 ? f32_variant_count() : learned_variant_count());
}
static TileVariant variant(int prec, int idx) {
    return prec == PREC_F64 ? f64_variant(idx) : (prec == PREC_F32 ? f32_variant(idx) : learned_variant(idx));
}
// tile-choice code: variant index, | kTmaBit when TMA staging is chosen, or
// | kListBit when uniform tiles are done apart and the others listed
constexpr int kTmaBit = 256, kListBit = 512;

// One launch of variant `code & 255`, TMA-staged where the code asks for it
// (and the grid allows it); ctx->tma_used_last tells whether it was.
static bsn_status launch_variant(bsn_ctx* ctx, int prec, int code, const f64::StageArgs& A0) {
    f64::StageArgs A = A0;
    if (!(code & kListBit)) A.uni_in = nullptr, A.uni_un = nullptr, A.uni_out = nullptr;
    const int idx = code & (kTmaBit - 1);
    ctx->tma_now = (code & kTmaBit) ? 1 : 0;
    ctx->tma_used_last = 0;
    bsn_status st = prec == PREC_F64 ? f64_launch_variant(ctx, idx, A)
                    : prec == PREC_F32 ? f32_launch_variant(ctx, idx, A)
                                       : learned_launch_variant(ctx, idx, A);
    ctx->tma_now = 0;
    return st;
}
// the code of a forced variant: listed where A keeps uniform tiles, else TMA
// wherever the context allows it
static int forced_code(bsn_ctx* ctx, int prec, const f64::StageArgs& A) {
    const int v = ctx->forced_tile[prec] >= 0 ? ctx->forced_tile[prec] : 0;
    return v | (A.uni_in ? kListBit : (ctx->tma_on ? kTmaBit : 0));
}
static bsn_status launch_batch_variant(bsn_ctx* ctx, int prec, int idx, const f64::StageBatch& B) {
    if (prec == PREC_F64) return f64_launch_batch_variant(ctx, idx, B);
    if (prec == PREC_F32) return f32_launch_batch_variant(ctx, idx, B);
    return learned_launch_batch_variant(ctx, idx, B);
}
static bool prec_ok(int p) { return p == PREC_F64 || p == PREC_F32 || p == PREC_LEARNED; }
static std::tuple<int, int, int, int, int> tile_key(int prec, const f64::StageArgs& A) {
    return std::make_tuple(prec, A.tune_class, A.nx, A.ny, A.nz);
}
static void record(bsn_ctx* ctx, int prec, const f64::StageArgs& A, int code) {
    ctx->tile_choice[tile_key(prec, A)] = code;
    ctx->tile_last[std::make_tuple(prec, A.nx, A.ny, A.nz)] = code;
}

int tile_code(bsn_ctx* ctx, int prec, const f64::StageArgs& A) {
    auto it = ctx->tile_choice.find(tile_key(prec, A));
    return it == ctx->tile_choice.end() ? -1 : it->second;
}

// One CTA per tile: 1 where all of its active cells hold the same words.
// Bound by its loads, a warp per row (figures at uniform_stage_kernel).
__global__ void uniform_tiles_kernel(const double* U, int nx, int ny, int nz, int tx, int ty, int tz,
                                     unsigned char* out) {
    const Geom G(nx, ny, nz);
    const int a0 = blockIdx.x * tx, b0 = blockIdx.y * ty, c0 = blockIdx.z * tz;
    const int row = 5 * min(tx, nx - a0), rows = min(ty, ny - b0), planes = min(tz, nz - c0);
    __shared__ double first[5];
    if (threadIdx.x < 5) first[threadIdx.x] = U[G.act(a0, b0, c0) + threadIdx.x];
    __syncthreads();
    bool mixed = false;
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    int b = threadIdx.x >> 5, c = 0;
    while (b >= rows) b -= rows, ++c;
    while (c < planes) {
        const double* u = U + G.act(a0, b0 + b, c0 + c);
        for (int w = lane, q = lane % 5; w < row; w += 32, q = q < 3 ? q + 2 : q - 3)   // 32 words on: q + 2 mod 5
            mixed |= __double_as_longlong(u[w]) != __double_as_longlong(first[q]);
        for (b += warps; b >= rows; b -= rows) ++c;
    }
    const int any = __syncthreads_or(mixed);
    if (threadIdx.x == 0)
        out[blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z)] = !any;
}

static bsn_status find_uniform(bsn_ctx* ctx, const TileVariant& v, const f64::StageArgs& base, const double* U,
                               unsigned char* f) {
    const dim3 grid((base.nx + v.tx - 1) / v.tx, (base.ny + v.ty - 1) / v.ty, (base.nz + v.tz - 1) / v.tz);
    prof_begin(ctx);
    uniform_tiles_kernel<<<grid, 256, 0, ctx->stream>>>(U, base.nx, base.ny, base.nz, v.tx, v.ty, v.tz, f);
    return launch_check(ctx, "uniform_tiles_kernel");
}

// For uniform grids of 2^18 cells (64^3) and more with no sources.  Smaller
// ones gain nothing: with and without, ms per step with a blast, FP64 / FP32:
// 48^3 0.270 / 0.102 both ways, 64^3 0.450 / 0.172 and 0.450 / 0.177, 96^3
// 1.03 / 0.39 and 1.25 / 0.42, 128^3 1.87 / 0.67 and 2.91 / 0.93 (B200).
static bool uniform_tiles_apply(const f64::StageArgs& b) {
    if (b.mode != 0 || b.Gh || b.ledger || b.use_reg || b.use_bnd || b.F[0] || b.F[1] || b.F[2]) return false;
    if (b.use_bh | b.use_sg | b.use_sink | b.use_rot | b.use_damp) return false;
    return (long long)b.nx * b.ny * b.nz >= (1LL << 18);
}

// one block: the tiles that are not uniform, added to *listed
__global__ void count_listed_kernel(const unsigned char* uniform, int tiles, unsigned int* listed) {
    unsigned int n = 0;
    for (int i = threadIdx.x; i < tiles; i += blockDim.x) n += uniform[i] == 0;
    atomicAdd(listed, n);
}

static long long tiles_of(const TileVariant& v, const f64::StageArgs& b) {
    return (long long)((b.nx + v.tx - 1) / v.tx) * ((b.ny + v.ty - 1) / v.ty) * ((b.nz + v.tz - 1) / v.tz);
}

// Whether to list, from the share of tiles listed lately.  The timing decides
// at first; a state that then loses its uniform gas (a blast that fills the
// box), or gets some, changes sides.  Eight steps on a state without uniform
// gas after a first call on a blast, with the blast's choice kept and with this:
// FP32 128^3 9.00 and 7.29 ms, learned 47.5 and 37.7, 256^3 FP32 61.6 and 54.7.
// Listing pays for itself once it leaves out a quarter of the tiles: with 0, 20,
// 40 and 60 % of a 128^3 box in a uniform slab, us a stage, the best list and
// the best tile without, FP32 351, 331, 288, 235 and 294 throughout, FP64 959,
// 1140, 1029, 835 and 905, 1044, 1082, 1086 (the slab's neighbours are listed
// too: two tiles of its eight at 40 %).  A side that turned out wrong has to be
// exceeded by a fifth.
static void follow(bsn_ctx* ctx, int prec, const f64::StageArgs& base) {
    const auto key = tile_key(prec, base);
    auto it = ctx->list_use.find(key);
    if (it == ctx->list_use.end()) return;
    bsn_ctx::ListUse& use = it->second;
    if (use.word < 0 || use.list < 0 || use.plain < 0) return;
    volatile unsigned int* word = ctx->listed_now + use.word;
    const unsigned int n = *word;   // may arrive while the steps go on: taken at the next call then
    if (n == ~0u) return;
    *word = ~0u;
    // of a list the share of tiles it left out, else of uniform tiles (more:
    // those beside others are listed too)
    const float share = 1.f - (float)n / (float)tiles_of(variant(prec, use.list & (kTmaBit - 1)), base);
    int& code = ctx->tile_choice[key];
    const bool on = code & kListBit;
    bool want = on;
    if (on && use.left_out < 0.f) use.left_out = share;   // of the state it was timed on
    if (on && share < 0.25f && (!use.list_won || share < 0.5f * use.left_out)) {
        want = false;
        use.no_gain = std::min(std::max(share, use.taken_at), 0.6f);
    }
    if (!on && share > std::max(use.no_gain + 0.2f, 0.45f)) {
        want = true;
        use.taken_at = share;
    }
    if (want != on) {
        code = want ? use.list : use.plain;
        ctx->tile_last[std::make_tuple(prec, base.nx, base.ny, base.nz)] = code;
    }
}

bsn_status uniform_tiles_prepare(bsn_ctx* ctx, int prec, f64::StageArgs& base, UniformTiles& t) {
    t.on = uniform_tiles_apply(base);
    if (t.on && base.tune_class == TUNE_GENERIC) base.tune_class = TUNE_STEP;
    bsn_status st;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(ctx->stream, &cs);
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    if (capturing) {   // no timing and no allocation in a capture: an earlier choice and its room, or none
        const int code = tile_code(ctx, prec, base);
        t.on = t.on && code >= 0 && (code & kListBit);
    }
    if (t.on) {
        size_t tiles = 0;
        for (int v = 0; v < variant_count(prec); ++v)
            tiles = std::max(tiles, (size_t)tiles_of(variant(prec, v), base));
        tiles = (tiles + 255) / 256 * 256;
        // Room for every grid that the stage buffers have room for (per axis at
        // most 1/7 tile per stored cell of n + 6 for the longer tile edges, 1/4
        // for the shortest): it moves when they do, so a step that the caller
        // captured stays as valid as its stage buffers.
        const size_t most = ctx->slot_bytes[SLOT_A] / (5 * sizeof(double)) / 196 + 256;
        const size_t bytes = 256 + (3 + sizeof(int)) * std::max(tiles, most / 256 * 256 + 256);
        if (capturing && ctx->slot_bytes[SLOT_UNIFORM] < bytes) {
            t.on = false;
            return BSN_OK;
        }
        unsigned char* f = (unsigned char*)slot(ctx, SLOT_UNIFORM, bytes, &st);
        BSN_TRY(st);
        t.count = (unsigned int*)f;
        t.list = (int*)(f + 256);
        for (int i = 0; i < 3; ++i) t.f[i] = f + 256 + (sizeof(int) + i) * tiles;
    }
    if (capturing) return BSN_OK;
    t.able = t.on && ctx->forced_tile[prec] < 0;
    f64::StageArgs p = base;
    t.set(p, 0);
    double* scratch = nullptr;
    if (ctx->forced_tile[prec] < 0 && (tile_code(ctx, prec, base) < 0 || base.tune_class == ctx->retime_class)) {
        scratch = (double*)slot(ctx, SLOT_UN, sizeof(double) * (size_t)Geom(base.nx, base.ny, base.nz).nelem(), &st);
        BSN_TRY(st);
    }
    BSN_TRY(stage_autotune(ctx, prec, p, scratch));
    if (t.able) follow(ctx, prec, base);
    t.on = t.on && (tile_code(ctx, prec, base) & kListBit);
    return BSN_OK;
}

bsn_status uniform_tiles_note(bsn_ctx* ctx, int prec, const f64::StageArgs& base, const double* U,
                              const UniformTiles& t) {
    if (!t.able) return BSN_OK;
    auto it = ctx->list_use.find(tile_key(prec, base));
    if (it == ctx->list_use.end() || it->second.word < 0 || it->second.list < 0) return BSN_OK;
    bsn_ctx::ListUse& use = it->second;
    // listing steps know what they listed; the others look seldom: a pass over
    // the state is 1-2 % of a step
    const int every = (base.tune_class == TUNE_STEP ? 8 : 1) * (t.on ? 1 : 4);
    if (use.calls++ % every) return BSN_OK;
    if (!t.on) {
        const TileVariant v = variant(prec, use.list & (kTmaBit - 1));
        BSN_CUDA(ctx, cudaMemsetAsync(t.count, 0, 6 * sizeof(unsigned int), ctx->stream));
        BSN_TRY(find_uniform(ctx, v, base, U, t.f[0]));
        prof_begin(ctx);
        count_listed_kernel<<<1, 1024, 0, ctx->stream>>>(t.f[0], (int)tiles_of(v, base), t.count + 4);
        BSN_TRY(launch_check(ctx, "count_listed_kernel"));
    }
    BSN_CUDA(ctx, cudaMemcpyAsync(ctx->listed_now + use.word, t.count + 4, sizeof(unsigned int),
                                  cudaMemcpyDeviceToHost, ctx->stream));
    return BSN_OK;
}

bsn_status uniform_tiles_find(bsn_ctx* ctx, int prec, const f64::StageArgs& base, const double* U,
                              const UniformTiles& t) {
    if (!t.on) return BSN_OK;
    const int code = tile_code(ctx, prec, base);
    const TileVariant v = variant(prec, (code >= 0 ? code : forced_code(ctx, prec, base)) & (kTmaBit - 1));
    BSN_CUDA(ctx, cudaMemsetAsync(t.count, 0, 6 * sizeof(unsigned int), ctx->stream));
    return find_uniform(ctx, v, base, U, t.f[0]);
}

// stage-1 work of a probe, writing to scratch and recording nothing; a
// right-hand side is timed as it runs, fluxes and all (it writes the same
// values each time, and does not write its input)
static f64::StageArgs probe_args(const f64::StageArgs& probe, double* scratch) {
    f64::StageArgs a = probe;
    if (a.mode == 1) return a;
    a.Un = probe.Uin;
    a.Uout = scratch;
    a.mode = 0;
    a.stage = 1;
    a.dt = 0.0;
    a.cfl_max = nullptr;
    a.cfl_nan = nullptr;
    a.use_reg = 0;
    a.use_bnd = 0;
    a.F[0] = a.F[1] = a.F[2] = nullptr;
    a.dt_dev = nullptr;
    a.done_dev = nullptr;
    a.ledger = nullptr;
    return a;
}

// The drivers whose stages run over several grids at once: one choice for all
// of them, timed as they run, in one launch over every level.  (Timed level by
// level, levels of one size share the first one's choice: three 128^3 levels
// of the binary star took the coarse level's 8x8x8, 16.9 ms a step; timed
// without their flux registers, two FP64 levels of 64^3 took 16x8x4 in three
// calls of four, 12.08 ms for eight steps where 16x8x8 takes 11.77.)
bsn_status stage_autotune_batch(bsn_ctx* ctx, int prec, const f64::StageArgs* probes, double* const* scratch, int n) {
    if (n < 1 || n > f64::MAXLEV) return set_err(ctx, BSN_ERR_ARG, "batch of %d levels", n);
    bool known = true;
    for (int l = 0; l < n; ++l) {
        const auto key = tile_key(prec, probes[l]);
        known = known && ctx->tile_choice.count(key) &&
                (probes[l].tune_class != ctx->retime_class || ctx->retimed.count(key));
    }
    if (known) return BSN_OK;
    bsn_status st;
    unsigned int* queue = (unsigned int*)slot(ctx, SLOT_RED, 64, &st);
    BSN_TRY(st);
    f64::StageBatch B;
    B.nlev = n;
    B.queue = queue;
    for (int l = 0; l < n; ++l) {
        if (prec == PREC_LEARNED) {   // the split learned stage's block list, allocated before any capture
            slot(ctx, SLOT_SPLIT, learned_split_bytes(probes[l].nx, probes[l].ny, probes[l].nz), &st);
            BSN_TRY(st);
        }
        if (probes[l].tune_class == ctx->retime_class) ctx->retimed.insert(tile_key(prec, probes[l]));
        B.lv[l] = probe_args(probes[l], scratch[l]);
        // the fluxes that levels record, too: the loops clear the registers
        // before they use them and write the boundary faces anew
        B.lv[l].use_reg = probes[l].use_reg;
        B.lv[l].use_bnd = probes[l].use_bnd;
    }
    int best = 0;
    if (ctx->forced_tile[prec] >= 0) {
        best = forced_code(ctx, prec, B.lv[0]);
    } else {
        cudaEvent_t e0, e1;
        BSN_CUDA(ctx, cudaEventCreate(&e0));
        BSN_CUDA(ctx, cudaEventCreate(&e1));
        float best_ms = 1e30f;
        const bool prof = ctx->profiling;
        ctx->profiling = false;
        for (int v = 0; v < variant_count(prec) && st == BSN_OK; ++v)
            for (int r = 0; r < 3 && st == BSN_OK; ++r) {   // the first a warm-up
                cudaMemsetAsync(queue, 0, sizeof(unsigned int), ctx->stream);
                cudaEventRecord(e0, ctx->stream);
                st = launch_batch_variant(ctx, prec, v, B);
                cudaEventRecord(e1, ctx->stream);
                if (st == BSN_OK) st = cuda_check(ctx, cudaEventSynchronize(e1), "cudaEventSynchronize(autotune)");
                float t = 0.f;
                cudaEventElapsedTime(&t, e0, e1);
                if (r > 0 && t < best_ms) { best_ms = t; best = v; }
            }
        ctx->profiling = prof;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        BSN_TRY(st);
    }
    for (int l = 0; l < n; ++l) record(ctx, prec, probes[l], best);
    return BSN_OK;
}

bsn_status stage_autotune(bsn_ctx* ctx, int prec, const f64::StageArgs& probe, double* scratch) {
    if (prec == PREC_LEARNED) {   // the split learned stage's block list, allocated before any capture
        bsn_status st;
        slot(ctx, SLOT_SPLIT, learned_split_bytes(probe.nx, probe.ny, probe.nz), &st);
        BSN_TRY(st);
    }
    const auto key = tile_key(prec, probe);
    if (ctx->tile_choice.count(key) && (probe.tune_class != ctx->retime_class || ctx->retimed.count(key)))
        return BSN_OK;
    if (probe.tune_class == ctx->retime_class) ctx->retimed.insert(key);
    int nv = variant_count(prec);
    if (ctx->forced_tile[prec] >= 0) {
        record(ctx, prec, probe, forced_code(ctx, prec, probe));
        return BSN_OK;
    }
    const f64::StageArgs a = probe_args(probe, scratch);
    cudaEvent_t e0, e1;
    BSN_CUDA(ctx, cudaEventCreate(&e0));
    BSN_CUDA(ctx, cudaEventCreate(&e1));
    int best = 0, plain = -1, list = -1;
    float best_ms = 1e30f, plain_ms = 1e30f, list_ms = 1e30f;
    unsigned int listed = 0, mixed = 0;   // of its tiles, those listed, and those that are not uniform
    bool prof = ctx->profiling;
    ctx->profiling = false;
    bsn_status st = BSN_OK;
    auto timed = [&](auto&& f) -> float {
        cudaEventRecord(e0, ctx->stream);
        st = f();
        cudaEventRecord(e1, ctx->stream);
        st = st != BSN_OK ? st : cuda_check(ctx, cudaEventSynchronize(e1), "cudaEventSynchronize(autotune)");
        float t = 0.f;
        cudaEventElapsedTime(&t, e0, e1);
        return t;
    };
    // one code; extra: time per stage it costs besides its launches.  False:
    // failed (st), or the grid does not allow this staging
    auto try_code = [&](int code, float extra) -> bool {
        float ms = 1e30f;
        for (int r = 0; r < 3 && st == BSN_OK; ++r) {   // the first a warm-up (sets smem attributes)
            if (code & kListBit) cudaMemsetAsync(a.list_count, 0, 2 * sizeof(unsigned int), ctx->stream);
            const float t = timed([&] { return launch_variant(ctx, prec, code, a); });
            if ((code & kTmaBit) && !ctx->tma_used_last) return false;
            if (r > 0) ms = t < ms ? t : ms;
        }
        if (ms + extra < best_ms) { best_ms = ms + extra; best = code; }
        if (!(code & kListBit)) {
            if (ms < plain_ms) { plain_ms = ms; plain = code; }
        } else if (ms < list_ms && st == BSN_OK) {
            list_ms = ms;
            list = code;
            cudaMemcpyAsync(&listed, a.list_count, sizeof(listed), cudaMemcpyDeviceToHost, ctx->stream);
            cudaMemsetAsync(a.list_count, 0, sizeof(unsigned int), ctx->stream);
            count_listed_kernel<<<1, 1024, 0, ctx->stream>>>(
                a.uni_in, (int)tiles_of(variant(prec, code & (kTmaBit - 1)), a), a.list_count);
            cudaMemcpyAsync(&mixed, a.list_count, sizeof(mixed), cudaMemcpyDeviceToHost, ctx->stream);
            st = cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "cudaStreamSynchronize(autotune)");
        }
        return st == BSN_OK;
    };
    for (int v = 0; v < nv && st == BSN_OK; ++v) {
        if (try_code(v, 0.f) && ctx->tma_on) try_code(v | kTmaBit, 0.f);
        if (st == BSN_OK && a.uni_in) {   // single steps find the uniform tiles anew for their three stages
            float find = 1e30f;
            for (int r = 0; r < 3 && st == BSN_OK; ++r) {   // the first a warm-up, as in try_code
                const float t = timed([&] {
                    return find_uniform(ctx, variant(prec, v), a, a.Uin, const_cast<unsigned char*>(a.uni_in));
                });
                if (r > 0) find = std::min(find, t);
            }
            if (st == BSN_OK) try_code(v | kListBit, probe.tune_class == TUNE_STEP ? find / 3.f : 0.f);
        }
    }
    ctx->profiling = prof;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    BSN_TRY(st);
    record(ctx, prec, probe, best);
    if (list >= 0) {
        constexpr int kWords = 64;
        if (!ctx->listed_now && cudaMallocHost(&ctx->listed_now, kWords * sizeof(unsigned int)) != cudaSuccess) {
            cudaGetLastError();
            ctx->listed_now = nullptr;   // the choice stays as timed
        }
        const int next = (int)ctx->list_use.size();
        bsn_ctx::ListUse& use = ctx->list_use[key];
        if (use.word < 0 && ctx->listed_now && next < kWords) use.word = next;
        if (use.word >= 0) ctx->listed_now[use.word] = ~0u;
        use.plain = plain;
        use.list = list;
        use.list_won = best & kListBit;
        const float tiles = (float)tiles_of(variant(prec, list & (kTmaBit - 1)), probe);
        // of the timed stage; a small share may be gone by the last stage of the
        // step, and is taken from the first count then
        use.left_out = 1.f - (float)listed / tiles;
        if (use.left_out < 0.3f) use.left_out = -1.f;
        use.no_gain = use.list_won ? 0.f : 1.f - (float)mixed / tiles;
        use.taken_at = 0.f;
        use.calls = 0;
    }
    return BSN_OK;
}

bool tile_settled(bsn_ctx* ctx, int tune_class, int prec) {
    return ctx->forced_tile[prec] >= 0 || ctx->settled.count(std::make_pair(tune_class, prec)) > 0;
}

bsn_status tile_retime(bsn_ctx* ctx, int tune_class, int prec, const std::function<bsn_status()>& tune) {
    ctx->retime_class = tune_class;
    ctx->retimed.clear();
    bsn_status st = tune();
    ctx->retime_class = -1;
    ctx->retimed.clear();
    if (st == BSN_OK) ctx->settled.insert(std::make_pair(tune_class, prec));
    return st;
}

bsn_status stage_launch(bsn_ctx* ctx, int prec, const f64::StageArgs& A) {
    auto it = ctx->tile_choice.find(tile_key(prec, A));
    if (it == ctx->tile_choice.end()) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(ctx->stream, &cs);
        if (ctx->forced_tile[prec] >= 0 || cs != cudaStreamCaptureStatusNone)
            return launch_variant(ctx, prec, forced_code(ctx, prec, A), A);
        Geom G(A.nx, A.ny, A.nz);
        bsn_status st;
        double* scratch = (double*)slot(ctx, SLOT_UN, sizeof(double) * (size_t)G.nelem(), &st);
        BSN_TRY(st);
        BSN_TRY(stage_autotune(ctx, prec, A, scratch));
        it = ctx->tile_choice.find(tile_key(prec, A));
    }
    return launch_variant(ctx, prec, it->second, A);
}

// The variant of a batch is the one chosen for its last level's grid (for
// two-level FMR the fine level, the larger share of the work per step).
static bsn_status choose(bsn_ctx* ctx, int prec, const f64::StageArgs& A, int& v) {
    auto it = ctx->tile_choice.find(tile_key(prec, A));
    if (it != ctx->tile_choice.end()) { v = it->second & (kTmaBit - 1); return BSN_OK; }
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(ctx->stream, &cs);
    if (ctx->forced_tile[prec] >= 0 || cs != cudaStreamCaptureStatusNone) {
        v = ctx->forced_tile[prec] >= 0 ? ctx->forced_tile[prec] : 0;
        return BSN_OK;
    }
    Geom G(A.nx, A.ny, A.nz);
    bsn_status st;
    double* scratch = (double*)slot(ctx, SLOT_UN, sizeof(double) * (size_t)G.nelem(), &st);
    BSN_TRY(st);
    BSN_TRY(stage_autotune(ctx, prec, A, scratch));
    v = ctx->tile_choice[tile_key(prec, A)] & (kTmaBit - 1);   // several grids in one launch: the plain loader
    return BSN_OK;
}

bsn_status stage_launch_batch(bsn_ctx* ctx, int prec, const f64::StageBatch& B) {
    if (B.nlev < 1 || B.nlev > f64::MAXLEV) return set_err(ctx, BSN_ERR_ARG, "batch of %d levels", B.nlev);
    int v = 0;
    BSN_TRY(choose(ctx, prec, B.lv[B.nlev - 1], v));
    return launch_batch_variant(ctx, prec, v, B);
}

}  // namespace bsn

using namespace bsn;

extern "C" bsn_status bsn_ctx_set_tile(bsn_ctx* ctx, int precision, int variant) {
    if (!ctx) return BSN_ERR_ARG;
    if (!prec_ok(precision)) return set_err(ctx, BSN_ERR_ARG, "bad precision %d", precision);
    if (variant >= variant_count(precision)) return set_err(ctx, BSN_ERR_ARG, "no tile variant %d", variant);
    ctx->forced_tile[precision] = variant < 0 ? -1 : variant;
    for (auto it = ctx->tile_choice.begin(); it != ctx->tile_choice.end();)
        it = std::get<0>(it->first) == precision ? ctx->tile_choice.erase(it) : std::next(it);
    for (auto it = ctx->tile_last.begin(); it != ctx->tile_last.end();)
        it = std::get<0>(it->first) == precision ? ctx->tile_last.erase(it) : std::next(it);
    for (auto it = ctx->settled.begin(); it != ctx->settled.end();)
        it = it->second == precision ? ctx->settled.erase(it) : std::next(it);
    for (auto it = ctx->list_use.begin(); it != ctx->list_use.end(); ++it)   // the words stay with their grids
        if (std::get<0>(it->first) == precision) it->second.list = it->second.plain = -1;
    return BSN_OK;
}

extern "C" bsn_status bsn_ctx_get_tile(bsn_ctx* ctx, int precision, int nx, int ny, int nz, int out[5]) {
    if (!ctx || !out) return BSN_ERR_ARG;
    auto it = ctx->tile_last.find(std::make_tuple(precision, nx, ny, nz));
    if (it == ctx->tile_last.end()) return set_err(ctx, BSN_ERR_ARG, "no tile chosen yet for this grid");
    if (!prec_ok(precision)) return set_err(ctx, BSN_ERR_ARG, "bad precision %d", precision);
    TileVariant v = variant(precision, it->second & (kTmaBit - 1));
    out[0] = v.tx; out[1] = v.ty; out[2] = v.tz; out[3] = v.nt; out[4] = v.minb;
    return BSN_OK;
}

extern "C" int bsn_ctx_get_tile_tma(bsn_ctx* ctx, int precision, int nx, int ny, int nz) {
    if (!ctx) return -1;
    auto it = ctx->tile_last.find(std::make_tuple(precision, nx, ny, nz));
    if (it == ctx->tile_last.end()) return -1;
    return (it->second & kTmaBit) ? 1 : 0;
}

extern "C" int bsn_tile_variant_count(int precision) {
    return prec_ok(precision) ? variant_count(precision) : 0;
}
