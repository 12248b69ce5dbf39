// Host-side launcher declarations shared between the kernel translation units and api.cu.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace haste {

// Dynamic shared memory of the kernels whose need depends on the call.  The limit that cudaFuncSetAttribute sets belongs to the
// function (per device), not to a launch, and calls come from several threads: a limit of each call's own size could be lowered by
// another thread between this thread's setting and its launch.  So every call sets the same constant, which leaves 27 KB of an
// SM's 227 for static arrays; what a launch takes is still its own size.
constexpr int DYN_SMEM_MAX = 200 * 1024;
template <class K>
int allow_dynamic_smem(K kernel) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DYN_SMEM_MAX);
  if (e != cudaSuccess) return fail(HASTE_ERR_LAUNCH, "cudaFuncSetAttribute(%d B): %s", DYN_SMEM_MAX, cudaGetErrorString(e));
  return HASTE_OK;
}


// Everything the fused weight/bias update needs.  mom_* are NULL when momentum is off.
struct UpdateArgs {
  __nv_bfloat16* w;
  __nv_bfloat16* bias;
  float* mom_w;
  float* mom_b;
  float lr, wd, mu;
  uint64_t seed;
  uint32_t step, flags;
  int64_t label0;   // global index of the shard's first label (random-bit counters are global)
};

// ldxt (here and below): row stride of xt in elements, >= B.  With a stride that is a multiple of 8, columns B .. ldxt-1 hold
// zeros and the rows are 16-byte aligned whatever B is.
// zw: writable width of a row of z, L <= zw <= ldz (columns L..zw-1 receive zeros)
int launch_forward(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t F,
                   int64_t L, int64_t G, int64_t ldz, int64_t zw, int64_t ldxt, cudaStream_t st);
bool forward_sm100_supported(const void* z, const void* xt, const void* w, int64_t B, int64_t F, int64_t L, int64_t G, int64_t ldz, int64_t ldxt);
int launch_forward_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t F,
                         int64_t L, int64_t G, int64_t ldz, int64_t zw, int64_t ldxt, cudaStream_t st);
// The label tiles a launch of the tcgen05 forward works on: every step-th tile of the layer (skip == 0), or every step-th tile but not
// every (step * skip)-th one, which an earlier launch has done (skip in 3 .. 2^12).  Tile i of the second kind is
// step * (i + i / (skip - 1) + 1); the division is a multiplication, exact for i < 2^20 * (4096 / skip).
struct TileSet {
  int step = 1, skip = 0;
  uint32_t inv = 0;                                    // 2^32 / (skip - 1), rounded up; 0 for skip == 0
  TileSet() = default;
  TileSet(int step_, int skip_) : step(step_), skip(skip_), inv(skip_ == 0 ? 0u : static_cast<uint32_t>((1ull << 32) / (skip_ - 1) + 1)) {}
  __device__ int tile(int i) const {
    return step * (i + static_cast<int>(__umulhi(static_cast<uint32_t>(i), inv)) + (skip == 0 ? 0 : 1));
  }
  int count(int n_tiles) const {
    const int with = (n_tiles + step - 1) / step;
    return skip == 0 ? with : with - (with + skip - 1) / skip;
  }
};
// Logits of the tiles of `set` only, side by side in z (label tile set.tile(i) in columns i * tile ...); z has `cols` real columns,
// rounded up to a multiple of 8 they receive zeros.
int launch_forward_tiles_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t F,
                               int64_t L, int64_t G, int64_t ldz, int64_t cols, int64_t ldxt, const TileSet& set, cudaStream_t st);
int forward_tile_labels_sm100(int64_t F, int64_t G);      // labels of a tile

// What a logit of a row has to beat: the row's k-th best (value, label) so far.  Labels before `label` win with an equal value,
// labels after it do not; .bits holds the value (bf16) in the upper half and a bf16 just below it in the lower half.
struct RowCut {
  uint32_t bits;
  int label;
};
// Forward whose epilogue keeps only the logits of the tiles of `set` that beat cut[b] (and a few more: those of a tile that
// holds cut[b].label itself may only equal it), as keys in cand[b][0 .. cap) (cnt[b] counts them all).
struct TopkFilter {
  // One counter per 128-byte line.  Side by side, the counters of 512 rows filled 16 lines, on which the 358 thousand
  // atomics of a 131 K-label launch queued: 88 us for the launch, 69 so.
  static constexpr int CNT_STRIDE = 32;
  const RowCut* cut;
  unsigned long long* cand;
  int* cnt;
  int cap, label0;
  TileSet set;
};
int launch_topk_filter_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, int64_t B, int64_t D, int64_t F, int64_t L,
                             int64_t G, int64_t ldxt, const TopkFilter& tk, cudaStream_t st);
int launch_bwd_features(const void* w, const int32_t* loc, const void* dy, float* dxt, int64_t B, int64_t D, int64_t F, int64_t L,
                        int64_t G, int64_t ldy, cudaStream_t st);
int launch_bwd_weights(const void* xt, const int32_t* loc, const void* dy, void* dw, void* dbias, const UpdateArgs* upd, int64_t B,
                       int64_t D, int64_t F, int64_t L, int64_t G, int64_t ldy, int64_t ldxt, cudaStream_t st);
int launch_train_step_mma(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt, float* loss,
                          const UpdateArgs& u, int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int loss_kind, float grad_scale,
                          int64_t ldxt, cudaStream_t st);
// Optional debug outputs of the tcgen05 fused step (tests only).
struct StepDump {
  void* z;       // bf16 [B, ldz] logits as rounded by the epilogue
  int64_t ldz;
  void* dw;      // bf16 [L,F] weight gradient consumed by the update
  void* dbias;   // bf16 [L]
};

// tcgen05 fused step: one translation unit per layer shape.  max_ctas > 0 caps the persistent grid (SMs left free for
// kernels of other streams).
int launch_train_step_sm100_g128f64(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt,
                                    float* loss, const UpdateArgs& u, int64_t B, int64_t D, int64_t L, int loss_kind, float grad_scale,
                                    int64_t ldxt, int max_ctas, cudaStream_t st, const StepDump* dump);
int launch_train_step_sm100_g64f128(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt,
                                    float* loss, const UpdateArgs& u, int64_t B, int64_t D, int64_t L, int loss_kind, float grad_scale,
                                    int64_t ldxt, int max_ctas, cudaStream_t st, const StepDump* dump);
int launch_train_step_sm100_small(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt,
                                  float* loss, const UpdateArgs& u, int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int loss_kind,
                                  float grad_scale, int64_t ldxt, int max_ctas, cudaStream_t st);
int launch_train_step(const int32_t* loc, const void* xt, const int32_t* tgt_ptr, const uint32_t* tgt_ent, float* dxt, float* loss,
                      const UpdateArgs& u, int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int loss_kind, float grad_scale,
                      int64_t ldxt, cudaStream_t st, const StepDump* dump = nullptr);
int launch_sr_round(const float* x, void* out, int64_t n, uint64_t seed, cudaStream_t st);
int launch_sgd_sr(void* w, const void* g, float* m, int64_t rows, int64_t cols, int64_t row0, float lr, float wd, float mu, uint64_t seed,
                  uint32_t step, uint32_t flags, cudaStream_t st);
// f32: dx receives the rounded values as fp32
int launch_dxt_to_dx(const float* dxt, void* dx, int64_t B, int64_t D, uint64_t seed, bool f32, cudaStream_t st);
// f32: x is fp32, rounded to bf16 on the way
int launch_transpose(const void* x, void* xt, int64_t B, int64_t D, int64_t ldxt, bool f32, cudaStream_t st);
int launch_targets_bucket(const int32_t* coo, int64_t nnz, int64_t label0, int64_t L, int64_t G, int32_t* ptr, uint32_t* ent,
                          int32_t* scratch, cudaStream_t st);
int launch_targets_bucket_noalloc(const int32_t* coo, int64_t nnz, int64_t label0, int64_t L, int64_t G, int32_t* ptr, uint32_t* ent,
                                  cudaStream_t st);
int launch_step_prepare(const void* x, void* xt, float* dxt, float* loss, const int32_t* coo, int64_t nnz, int64_t label0, int64_t L,
                        int64_t G, int32_t* ptr, uint32_t* ent, int64_t B, int64_t D, int64_t ldxt, cudaStream_t st);
bool backward_sm100_supported(const void* xt, const void* w, const void* dy, const void* dw, int64_t B, int64_t D, int64_t F, int64_t L,
                              int64_t G, int64_t ldxt);
int launch_backward_sm100(const void* xt, const void* w, const int32_t* loc, const void* dy, float* dxt, void* dw, void* dbias,
                          const UpdateArgs* upd, int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int64_t ldy, int64_t ldxt, cudaStream_t st);
int launch_pad_rows(const void* src, int64_t ld_src, void* dst, int64_t ld_dst, int64_t rows, int64_t cols, cudaStream_t st);
int launch_topk_update(const void* z, int64_t ldz, int64_t B, int64_t C, int64_t col0, int k, float* vals, int32_t* idx, cudaStream_t st);
// Whole top-k of a layer, filtered (topk.cu); scratch: topk_fused_scratch_bytes bytes, 0 = this shape takes the chunked path.
int64_t topk_fused_scratch_bytes(int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int k);
int launch_topk_fused(const int32_t* loc, const void* x, const void* w, const void* bias, void* scratch, int64_t B, int64_t D, int64_t F, int64_t L,
                      int64_t G, int k, int64_t label0, float* vals, int32_t* idx, cudaStream_t st);
int launch_check_loc(const int32_t* loc, int64_t n, int64_t D, cudaStream_t st);
// score_mode 0 mean / 1 max; prune_mode 0 threshold / 1 per-group fraction / 2 global fraction (n_prune is then the
// layer-wide count and scratch holds HASTE_REWIRE_SCRATCH_WORDS(NG, F) words)
int launch_rewire(void* w, int32_t* loc, float* mom, int64_t D, int64_t F, int64_t L, int64_t G, int64_t group0, int score_mode, int prune_mode,
                  float threshold, int64_t n_prune, int regrow_mode, int init_mode, int regroup, uint64_t seed, uint32_t step,
                  void* scratch, int32_t* changed, cudaStream_t st, uint32_t tie_base = 0);
// layer-wide selection in phases, for a layer sharded over ranks (the caller sums the histograms between the phases)
int launch_rewire_select_begin(const void* w, int64_t F, int64_t L, int64_t G, int score_mode, void* scratch, cudaStream_t st);
int launch_rewire_select_refine(int64_t F, int64_t L, int64_t G, int64_t k, void* scratch, cudaStream_t st);
int launch_rewire_select_finish(int64_t F, int64_t L, int64_t G, void* scratch, cudaStream_t st);

}  // namespace haste
