// stage_f64_launch.cuh -- launches of one FP64 tile variant (stage_f64_lo.cu
// and stage_f64_hi.cu hold two variants each, to compile side by side).
#pragma once

#include "hydro_f64.cuh"
#include "stage_launch.cuh"
#include "stage_tile.cuh"

namespace bsn {
namespace {

using f64::StageArgs;
using f64::StageBatch;

template <int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_f64(bsn_ctx* ctx, const StageArgs& A) {
    if (A.uni_in) {
        BSN_TRY(tile::launch_uniform<tile::F64Physics>(ctx, A, TX, TY, TZ));
        return tile::launch_list<tile::F64Physics, TX, TY, TZ, NT, MINB>(
            ctx, A, tile::smem_bytes<tile::F64Physics, TX, TY, TZ>(), "stage_kernel");
    }
    bool tma_used = false;
    BSN_TRY((tile::launch_tma<tile::F64Physics, TX, TY, TZ, NT, MINB>(ctx, A, "stage_kernel_tma", &tma_used)));
    if (tma_used) return BSN_OK;
    return tile::launch_plain<tile::F64Physics, TX, TY, TZ, NT, MINB>(
        ctx, A, tile::smem_bytes<tile::F64Physics, TX, TY, TZ>(), "stage_kernel");
}
template <int TX, int TY, int TZ, int NT, int MINB>
bsn_status launch_f64_batch(bsn_ctx* ctx, const StageBatch& B) {
    return tile::launch_batch<tile::F64Physics, TX, TY, TZ, NT, MINB>(
        ctx, B, tile::smem_bytes<tile::F64Physics, TX, TY, TZ>(), "stage_kernel_batch");
}

}  // namespace
}  // namespace bsn
