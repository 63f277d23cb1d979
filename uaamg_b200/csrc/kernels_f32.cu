// FP32 engines: plain FP32 PCG (FP64 reductions only, FP32 couplings), and the
// mixed form: FP16-stored coarse couplings, FP32 V-cycle and CG, FP64 residual
// replacement into an FP64 solution.
#include "engine.cuh"

namespace uaamg {
Engine* create_engine_f32(int mixed, int apply_only) {
    if (mixed) return new EngineT<float, __half>(true, !apply_only, apply_only != 0);
    return new EngineT<float, float>(false, !apply_only, apply_only != 0);
}
}  // namespace uaamg
