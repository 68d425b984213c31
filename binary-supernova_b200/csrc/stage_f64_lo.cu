// stage_f64_lo.cu -- FP64 tile variants 0 and 1 of the fused stage kernel.
#include "stage_f64_launch.cuh"

namespace bsn {

bsn_status f64_launch_variant_lo(bsn_ctx* ctx, int idx, const StageArgs& A) {
    switch (idx) {
        case 0: return launch_f64<8, 8, 8, 256, 2>(ctx, A);
        case 1: return launch_f64<8, 8, 4, 128, 4>(ctx, A);
        default: return set_err(ctx, BSN_ERR_ARG, "no FP64 tile variant %d", idx);
    }
}
bsn_status f64_launch_batch_variant_lo(bsn_ctx* ctx, int idx, const StageBatch& B) {
    switch (idx) {
        case 0: return launch_f64_batch<8, 8, 8, 256, 2>(ctx, B);
        case 1: return launch_f64_batch<8, 8, 4, 128, 4>(ctx, B);
        default: return set_err(ctx, BSN_ERR_ARG, "no FP64 tile variant %d", idx);
    }
}

}  // namespace bsn
