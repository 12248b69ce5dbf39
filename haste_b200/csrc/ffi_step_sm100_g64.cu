// Fused tcgen05 train step, instantiated for group size 64, fan-in 128 (the 131K- and 501K-label configurations and
// the shape the reference's Amazon-3M configuration asks for).
#include "ffi_step_sm100.cuh"

namespace haste {
int launch_train_step_sm100_g64f128(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt,
                                    float* loss, const UpdateArgs& u, int64_t B, int64_t D, int64_t L, int loss_kind, float grad_scale,
                                    int64_t ldxt, int max_ctas, cudaStream_t st, const StepDump* dump) {
  return s100::launch_step_shape<64, 128, 1>(loc, xt, tgt_ptr, tgt_ent, dxt, loss, u, B, D, L, loss_kind, grad_scale, ldxt, max_ctas, st, dump);
}
}  // namespace haste
