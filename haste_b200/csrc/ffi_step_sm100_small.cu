// Fused tcgen05 train step, instantiated for the layer shapes (64, 64), (32, 64), (32, 32) and (32, 128): the layer class's default
// group size, and the 31K-label configuration.
#include "ffi_step_sm100.cuh"

namespace haste {
int launch_train_step_sm100_small(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt,
                                  float* loss, const UpdateArgs& u, int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int loss_kind,
                                  float grad_scale, int64_t ldxt, int max_ctas, cudaStream_t st) {
  if (G == 64 && F == 64) return s100::launch_step_shape<64, 64, 1>(loc, xt, tgt_ptr, tgt_ent, dxt, loss, u, B, D, L, loss_kind, grad_scale, ldxt, max_ctas, st, nullptr);
  if (G == 32 && F == 64) return s100::launch_step_shape<32, 64, 2>(loc, xt, tgt_ptr, tgt_ent, dxt, loss, u, B, D, L, loss_kind, grad_scale, ldxt, max_ctas, st, nullptr);
  if (G == 32 && F == 128) return s100::launch_step_shape<32, 128, 1>(loc, xt, tgt_ptr, tgt_ent, dxt, loss, u, B, D, L, loss_kind, grad_scale, ldxt, max_ctas, st, nullptr);
  if (G == 32 && F == 32) return s100::launch_step_shape<32, 32, 2>(loc, xt, tgt_ptr, tgt_ent, dxt, loss, u, B, D, L, loss_kind, grad_scale, ldxt, max_ctas, st, nullptr);
  return fail(HASTE_ERR_UNSUPPORTED, "tcgen05 fused step: no kernel for group size %lld, fan-in %lld", (long long)G, (long long)F);
}
}  // namespace haste
