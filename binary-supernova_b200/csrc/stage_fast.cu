// stage_fast.cu -- FP32-stencil variants of the fused stage kernel (the fast
// path): FP32 staging, WENO5-Z, pressures and HLLC with FMA and approximate
// reciprocals/square roots; FP64 state, floors, divergence, sources, RK3
// combine and CFL.  Built with --ftz=true --prec-div=false --prec-sqrt=false.
#include "stage_f32_launch.cuh"

namespace bsn {

namespace {
// one table for both policies
const TileVariant kF32Variants[] = {{8, 8, 8, 256, 3}, {16, 8, 4, 256, 3}, {8, 8, 4, 128, 6}, {16, 8, 8, 256, 2},
                                     {16, 16, 4, 256, 2}, {16, 16, 8, 512, 1}};
}  // namespace

int f32_variant_count() { return (int)(sizeof(kF32Variants) / sizeof(kF32Variants[0])); }
TileVariant f32_variant(int idx) { return kF32Variants[idx]; }
bsn_status f32_launch_variant(bsn_ctx* ctx, int idx, const f64::StageArgs& A) {
    return A.stiff_guard ? f32_guarded_launch_variant(ctx, idx, A) : launch_f32<tile::F32Physics>(ctx, idx, A);
}

bsn_status f32_launch_batch_variant(bsn_ctx* ctx, int idx, const f64::StageBatch& B) {
    bool guard = false;
    for (int l = 0; l < B.nlev && l < f64::MAXLEV; ++l) guard = guard || B.lv[l].stiff_guard;
    return guard ? f32_guarded_launch_batch_variant(ctx, idx, B) : launch_f32_batch<tile::F32Physics>(ctx, idx, B);
}

}  // namespace bsn
