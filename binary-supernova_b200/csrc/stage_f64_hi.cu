// stage_f64_hi.cu -- FP64 tile variants 2 and 3 of the fused stage kernel.
#include "stage_f64_launch.cuh"

namespace bsn {

bsn_status f64_launch_variant_hi(bsn_ctx* ctx, int idx, const StageArgs& A) {
    switch (idx) {
        case 2: return launch_f64<16, 8, 4, 256, 2>(ctx, A);
        case 3: return launch_f64<16, 8, 8, 512, 1>(ctx, A);
        default: return set_err(ctx, BSN_ERR_ARG, "no FP64 tile variant %d", idx);
    }
}
bsn_status f64_launch_batch_variant_hi(bsn_ctx* ctx, int idx, const StageBatch& B) {
    switch (idx) {
        case 2: return launch_f64_batch<16, 8, 4, 256, 2>(ctx, B);
        case 3: return launch_f64_batch<16, 8, 8, 512, 1>(ctx, B);
        default: return set_err(ctx, BSN_ERR_ARG, "no FP64 tile variant %d", idx);
    }
}

}  // namespace bsn
