// stage_guarded.cu -- the FP32-stencil stage kernel with stiff faces in FP64
// (F32Guarded), built as stage_fast.cu.
#include "stage_f32_launch.cuh"

namespace bsn {

bsn_status f32_guarded_launch_variant(bsn_ctx* ctx, int idx, const f64::StageArgs& A) {
    return launch_f32<tile::F32Guarded>(ctx, idx, A);
}
bsn_status f32_guarded_launch_batch_variant(bsn_ctx* ctx, int idx, const f64::StageBatch& B) {
    return launch_f32_batch<tile::F32Guarded>(ctx, idx, B);
}

}  // namespace bsn
