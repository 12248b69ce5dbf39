// Forward gather-GEMM of the FFI layer on tcgen05 / TMEM, for the layer shapes (group size, fan-in) = (128, 64), (64, 128),
// (64, 64), (32, 128) and, with two consecutive groups per tile, (32, 64) and (32, 32):
//     z[b, l] = sum_k xt[loc[l/G, k], b] * w[l, k] + bias[l]        (bf16 in, fp32 accumulate, bf16 out)
// This is the unfused forward of the autograd surface: it has to write the [B, L] logits, so it is bound by
// that HBM write (2*B*L bytes), not by the tensor pipe.
//
// Persistent, one CTA per SM, groups g = blockIdx.x, += gridDim.x; per group the batch is walked in 128-row
// tiles.  Same shared-memory operand layout as the fused train step (128-byte-swizzled row blocks; X tile as
// MN-major A with a row of ones under the gathered rows, W tile as K-major B, the bias as one more K step).
// Everything that moves a tile is a TMA copy: the W tile through a 2-D tensor map, the X rows by tile::gather4
// from four or eight producer warps (the gather rate grows with the number of issuing warps), and the logits leave
// through a tensor-map store from a swizzled staging tile, which also clips the ragged last group and the
// ragged last batch tile (in whole 16-byte chunks: the store's extent is the writable width rounded down to 8
// columns, and the up to 7 columns left over are written with ordinary 2-byte stores).  Warp roles (448 or 576 threads): warp 0 brings
// weights and bias, warps 2, 3, 12, 13 (to 17) gather, warp 1 issues the MMAs, warps 4-11 drain the accumulator: TMEM -> bf16 -> staging tile; one thread issues the store.
// All waits are bounded (see mbar_wait).
//
// A launch may take every n-th label tile only (TileSet), which is how top-k samples a layer.  The TOPK instantiations write no
// logits: the epilogue warps compare each logit (rounded to bf16, as it would have been
// stored) with the k-th best its row had before the launch and keep the few that beat it — expected k times the
// ratio of labels in this launch to labels before it — as keys for the merge kernel in topk.cu.  A maximum tree over 32
// logits decides per chunk whether anything passed; what did is collected in a list per warp in the shared
// memory the staging tiles would use, and flushed 32 entries at a time, so that the latency of the atomics on the
// rows' counters is paid once per flush and not once per candidate.
#include "common.cuh"
#include "launchers.h"
#include "runtime.h"
#include "sm100.cuh"

namespace haste {
namespace f100 {
using namespace sm100;

template <int GG_, int FF_, int P_>
struct Cfg {
  static constexpr int GG = GG_, FF = FF_, P = P_;     // label group, fan-in, groups per tile
  static constexpr int G = P * GG, F = P * FF, BT = 128;
  static_assert((G == 128 && F == 64) || (G == 64 && (F == 128 || F == 64)) || (G == 32 && F == 128), "tile shapes with a tcgen05 forward");
  static_assert(FF == 32 || FF % 64 == 0, "a weight row fills 64-byte or 128-byte swizzled rows");
  static constexpr int WROW = FF == 32 ? 64 : 128;    // bytes of one swizzled row of a W block
  static constexpr int FR = F + 16;                   // rows of an X block: F gathered rows, one row of ones, 15 zero rows
  static constexpr int NXS = (F == 64) ? 5 : 4;       // X ring stages
  static constexpr int XBLK = FR * 128;               // one 64-batch block of an X stage (bytes)
  static constexpr int XSTAGE = 2 * XBLK;
  static constexpr int NWB = FF == 32 ? 1 : FF / 64;  // blocks of a W stage (64 slots each, 32 at fan-in 32)
  static constexpr int WBLK = G * WROW;
  static constexpr int WSTAGE = NWB * WBLK;
  static constexpr int CROW = G == 32 ? 64 : 128;     // bytes of one swizzled row of a staging block
  static constexpr int NCB = G == 32 ? 1 : G / 64;    // blocks of a staging tile (64 labels each, 32 at G = 32)
  static constexpr int CBLK = BT * 128;
  static constexpr int CSTAGE = NCB * CBLK;
  static constexpr int BTILE = G * 32;                // bias tile: G rows x 16 bf16, no swizzle
  static constexpr int OFF_X = 0;
  static constexpr int OFF_W = OFF_X + NXS * XSTAGE;
  static constexpr int OFF_C = OFF_W + 2 * WSTAGE;
  static constexpr int OFF_BT = OFF_C + 2 * CSTAGE;
  static constexpr int OFF_BAR = OFF_BT + 2 * BTILE;
  static constexpr int OFF_MISC = OFF_BAR + 32 * 8;
  static constexpr int SMEM_BYTES = OFF_MISC + 64 + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
  static_assert(XSTAGE % 1024 == 0 && WBLK % 1024 == 0 && CBLK % 1024 == 0 && OFF_BT % 128 == 0, "tile alignment");
  static constexpr int B_XFULL = 0, B_XEMPTY = NXS, B_WFULL = 2 * NXS, B_WEMPTY = B_WFULL + 2, B_ZFULL = B_WEMPTY + 2,
                       B_ZEMPTY = B_ZFULL + 2, B_FIN = B_ZEMPTY + 2, NBAR = B_FIN + 1;
  static_assert(NBAR <= 32, "barrier space");
  static constexpr int N_EPI = 8;                     // epilogue warps: 4 TMEM lane quarters x 2 column halves
  static constexpr int EC = G / 2;                    // label columns of a tile drained by one epilogue warp
  // The products waited for their X tiles: a warp issues one gather per 100 cycles or so, and one of four producers also waited for
  // the weights' stage.  Now a warp of its own brings the weights, and two warps share a tile.  Forward of 670 K labels, 512 rows:
  // 170 -> 147 us (four warps to a tile: 158; eight producers, two to a tile: 166); 131 K labels, G=32, F=64, 256 rows, 128 slots to a tile: a layer
  // step 149 -> 138 us with eight producers, 149 with four.
  static constexpr int NPW = F == 64 ? 4 : 8;         // X producer warps: 2, 3 and those after the epilogue warps ...
  static constexpr int NSH = 2;                       // ... of which so many share a tile
  static_assert(NPW / NSH <= NXS, "a producer must not run more than one phase ahead on any stage barrier");
  static constexpr int W_EPI = 4, W_XP = W_EPI + N_EPI;
  static constexpr int NTHREADS = (W_XP + NPW - 2) * 32;
  static constexpr uint32_t TM_COLS = 2 * G;          // two accumulator stages
  // byte offset of 16-byte chunk c (8 labels) of batch row `row` in a staging tile: as the tensor map's swizzle expects it
  __device__ static __forceinline__ int c_chunk(int row, int c) {
    if (G == 32) return row * 64 + ((c ^ ((row >> 1) & 3)) << 4);
    return (c >> 3) * CBLK + row * 128 + (((c & 7) ^ (row & 7)) << 4);
  }
};

struct FwdArgs {
  const int32_t* loc;
  const __nv_bfloat16* bias;
  __nv_bfloat16* z;
  int* err;
  int64_t B, L, ldz, zw;
  int D, NG, NGR;      // NG: tiles (of G labels) of this launch; NGR: label groups of the layer
  TileSet set;
  long long wait_limit;
  // TOPK
  const RowCut* cut;           // [B] current k-th best of every row
  unsigned long long* cand;    // [B][cap] keys of the logits that beat it
  int* cnt;                    // [B] number of them, also beyond cap; TopkFilter::CNT_STRIDE apart
  int cap, label0;
};

__device__ __forceinline__ uint32_t max2(uint32_t x, uint32_t y) {      // a NaN loses against a number
  const __nv_bfloat162 v = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
  return *reinterpret_cast<const uint32_t*>(&v);
}
// 0xFFFF in each half where x > y (false for a NaN)
__device__ __forceinline__ uint32_t gt2_mask(uint32_t x, uint32_t y) {
  return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <int GG_, int FF_, int P_, bool TOPK>
__global__ void __launch_bounds__(Cfg<GG_, FF_, P_>::NTHREADS, 1)
ffi_forward_sm100_kernel(FwdArgs a, const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w,
                         const __grid_constant__ CUtensorMap tm_z) {
  using C = Cfg<GG_, FF_, P_>;
  constexpr int GG = C::GG, FF = C::FF, P = C::P;
  constexpr int G = C::G, F = C::F, BT = C::BT, NXS = C::NXS, XBLK = C::XBLK, XSTAGE = C::XSTAGE, WBLK = C::WBLK, WSTAGE = C::WSTAGE;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const uint32_t sbase = smem_u32(sm);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + C::OFF_MISC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + C::OFF_MISC + 8);
  volatile int* x_last = reinterpret_cast<volatile int*>(sm + C::OFF_MISC + 16);      // [NPW] the last tile each X producer announced
  auto bar = [&](int i) { return sbase + C::OFF_BAR + i * 8; };
  const long long WL = a.wait_limit;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int T = static_cast<int>((a.B + BT - 1) / BT);

  if (tid == 0) {
    for (int i = 0; i < NXS; ++i) { mbar_init(bar(C::B_XFULL + i), C::NSH); mbar_init(bar(C::B_XEMPTY + i), 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(C::B_WFULL + i), 1);  mbar_init(bar(C::B_WEMPTY + i), 1);
      mbar_init(bar(C::B_ZFULL + i), 1);  mbar_init(bar(C::B_ZEMPTY + i), C::N_EPI);
    }
    mbar_init(bar(C::B_FIN), 1);
    mbar_fence_init();
    *abort_flag = 0;
  }
  // rows F..F+15 of every X block: row F = ones (times the bias column = the bias), the rest zeros; written once
  for (int i = tid; i < NXS * 2 * 16 * 8; i += C::NTHREADS) {
    const int chunk = i & 7, row = (i >> 3) & 15, blk = i >> 7;
    const uint32_t v = (row == 0) ? 0x3F803F80u : 0u;
    *reinterpret_cast<uint4*>(sm + C::OFF_X + blk * XBLK + (F + row) * 128 + chunk * 16) = make_uint4(v, v, v, v);
  }
  for (int i = tid; i < 2 * C::BTILE / 16; i += C::NTHREADS) *reinterpret_cast<uint4*>(sm + C::OFF_BT + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  fence_proxy_async();
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), C::TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int n_my_groups = (a.NG > static_cast<int>(blockIdx.x)) ? (a.NG - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;

  const int prod_id = warp == 2 || warp == 3 ? warp - 2 : (warp >= C::W_XP ? 2 + warp - C::W_XP : -1);
  if (warp == 0) {
    // ================================================================ group producer: W tile (tensor map) and bias column
    int w_armed = 0;
    for (int gi = 0; gi < n_my_groups; ++gi) {
      const int g = a.set.tile(blockIdx.x + gi * gridDim.x);
      const int ws = gi & 1;
      const int64_t l0 = static_cast<int64_t>(g) * G;
      const int rows_real = static_cast<int>(imin64(G, a.L - l0));
      uint16_t bv[G / 32];
#pragma unroll
      for (int j = 0; j < G / 32; ++j) {
        const int c = lane + 32 * j;
        bv[j] = (a.bias != nullptr && c < rows_real) ? __bfloat16_as_ushort(a.bias[l0 + c]) : uint16_t(0);
      }
      const bool ok = mbar_wait(bar(C::B_WEMPTY + ws), ((gi >> 1) & 1) ^ 1, abort_flag, a.err, 21, WL, 100);
      __syncwarp();
      const bool go = __all_sync(0xffffffffu, ok && !*abort_flag);
      if (go) {
        if (lane == 0) {
          mbar_expect_tx(bar(C::B_WFULL + ws), WSTAGE);
#pragma unroll
          for (int kb = 0; kb < C::NWB; ++kb)
            tma_load_2d(sbase + C::OFF_W + ws * WSTAGE + kb * WBLK, &tm_w, kb * 64, static_cast<int>(l0), bar(C::B_WFULL + ws));
        }
        ++w_armed;
      }
#pragma unroll
      for (int j = 0; j < G / 32; ++j) {
        const int c = lane + 32 * j;
        *reinterpret_cast<uint16_t*>(sm + C::OFF_BT + ws * C::BTILE + (c >> 3) * 256 + (c & 7) * 16) = bv[j];
      }
      fence_proxy_async();
      __syncwarp();
      if (go && lane == 0) mbar_arrive(bar(C::B_WFULL + ws));
      __syncwarp();
    }
    // every copy this warp started has to land before the CTA may exit (only the most recent use of each stage: an older phase of the same
    // barrier can no longer be waited for)
    for (int j = max(0, w_armed - 2); j < w_armed; ++j) mbar_wait_final(bar(C::B_WFULL + (j & 1)), (j >> 1) & 1, WL);
  } else if (prod_id >= 0) {
    // ================================================================ X producers
    // F index rows of xt per batch tile, 256 bytes each, as gathers of four rows that land at their swizzled positions.  NSH warps share a tile,
    // one load per lane, and each announces its own bytes.
    constexpr int NLD = 2 * (F / 4) / C::NSH, STEP = C::NPW / C::NSH;            // loads per warp and tile; tiles between two of a warp
    static_assert(NLD * C::NSH == 2 * (F / 4) && NLD <= 32, "one load per lane");
    const int li = (prod_id % C::NSH) * NLD + lane, blk = li / (F / 4), r4 = li % (F / 4);
    int4 lr = make_int4(0, 0, 0, 0);
    int t = prod_id / C::NSH, gi = 0, g_have = -1, my_last = -1;
    const int n_items = n_my_groups * T;
    for (int it = t; it < n_items; it += STEP, t += STEP) {
      while (t >= T) { t -= T; ++gi; }
      if (gi != g_have) {
        g_have = gi;
        const int g = a.set.tile(blockIdx.x + gi * gridDim.x);
        const int32_t* lrow = a.loc + static_cast<int64_t>(g) * F + r4 * 4;
        // the last tile may hold one group less: its slots gather row 0 and meet zero weights
        const bool there = lane < NLD && (P == 1 || r4 * 4 < (a.NGR - g * P) * FF);
        const int top = a.D - 1;                         // clamped: never addresses outside xt
        lr.x = there ? min(max(__ldg(lrow), 0), top) : 0; lr.y = there ? min(max(__ldg(lrow + 1), 0), top) : 0;
        lr.z = there ? min(max(__ldg(lrow + 2), 0), top) : 0; lr.w = there ? min(max(__ldg(lrow + 3), 0), top) : 0;
      }
      const int xs = it % NXS;
      const bool okx = mbar_wait(bar(C::B_XEMPTY + xs), ((it / NXS) & 1) ^ 1, abort_flag, a.err, 22, WL, 100);
      __syncwarp();
      if (!__all_sync(0xffffffffu, okx && !*abort_flag)) break;          // (the flag stays up)
      const uint32_t full = bar(C::B_XFULL + xs);
      if (lane == 0) mbar_arrive_expect_tx(full, NLD * 512);
      __syncwarp();
      if (lane < NLD)
        tma_gather4(sbase + C::OFF_X + xs * XSTAGE + blk * XBLK + r4 * 512, &tm_x, t * BT + blk * 64, lr.x, lr.y, lr.z, lr.w, full);
      my_last = it;
    }
    if (lane == 0) x_last[prod_id] = my_last;
  } else if (warp == 1) {
    // ================================================================ MMA issuer
    // The warp runs its control flow converged; one elected lane issues the products and commits (descriptors stay
    // in uniform registers this way).
    constexpr uint32_t ID_FWD = make_idesc(128, GG, 1, 0);
    constexpr uint32_t ID_BIAS = make_idesc(128, G, 1, 0);
    const uint64_t D_XA = make_sdesc(sbase + C::OFF_X, XBLK, 1024);            // X tile as MN-major A
    const uint64_t D_WB = FF == 32 ? make_sdesc64(sbase + C::OFF_W, 16, 512) : make_sdesc(sbase + C::OFF_W, 16, 1024);   // W tile as K-major B
    const uint64_t D_BB = make_sdesc_noswizzle(sbase + C::OFF_BT, 128, 256);   // bias tile as K-major B (last K step)
    const uint32_t xa_lo = static_cast<uint32_t>(D_XA), xa_hi = static_cast<uint32_t>(D_XA >> 32);
    const uint32_t wb_lo = static_cast<uint32_t>(D_WB), wb_hi = static_cast<uint32_t>(D_WB >> 32);
    const uint32_t bb_lo = static_cast<uint32_t>(D_BB), bb_hi = static_cast<uint32_t>(D_BB >> 32);
    const uint32_t id_fwd = ID_FWD, id_bias = ID_BIAS;
    int it = 0, xs = 0, xph = 0;
    for (int gi = 0; gi < n_my_groups; ++gi) {
      const int ws = gi & 1;
      const bool okw = mbar_wait(bar(C::B_WFULL + ws), (gi >> 1) & 1, abort_flag, a.err, 23, WL);
      for (int t = 0; t < T; ++t, ++it) {
        const int zs = it & 1;
        bool ok = mbar_wait(bar(C::B_XFULL + xs), xph, abort_flag, a.err, 24, WL) && okw;
        ok = mbar_wait(bar(C::B_ZEMPTY + zs), ((it >> 1) & 1) ^ 1, abort_flag, a.err, 25, WL) && ok;
        tc_fence_after();
        const uint32_t xa = xa_lo + static_cast<uint32_t>(xs) * (XSTAGE >> 4), wb = wb_lo + (ws ? (WSTAGE >> 4) : 0u);
        const uint32_t bb = bb_lo + (ws ? (C::BTILE >> 4) : 0u);
        const uint32_t tz = tmem + zs * G;
        if (ok && elect_one()) {          // after an abort nothing more is issued
#pragma unroll
          for (int p = 0; p < P; ++p) {          // group p of the tile: its slots against its labels' weight rows
            const uint32_t xp = xa + ((p * FF * 128) >> 4), wp = wb + ((p * GG * C::WROW) >> 4);
            umma_bf16_lohi<false>(tz + p * GG, xp, xa_hi, wp, wb_hi, id_fwd);
#pragma unroll
            for (int ks = 1; ks < FF / 16; ++ks)
              umma_bf16_lohi<true>(tz + p * GG, xp + ((ks * 2048) >> 4), xa_hi, wp + (((ks >> 2) * WBLK + (ks & 3) * 32) >> 4), wb_hi, id_fwd);
          }
          umma_bf16_lohi<true>(tz, xa + (((F / 16) * 2048) >> 4), xa_hi, bb, bb_hi, id_bias);
          tc_commit(bar(C::B_ZFULL + zs));
          tc_commit(bar(C::B_XEMPTY + xs));
          if (t + 1 == T) tc_commit(bar(C::B_WEMPTY + ws));
        }
        __syncwarp();
        if (++xs == NXS) { xs = 0; xph ^= 1; }
      }
    }
    // every product this warp issued has completed before the CTA tears down its TMEM
    if (elect_one()) tc_commit(bar(C::B_FIN));
    __syncwarp();
    mbar_wait_final(bar(C::B_FIN), 0, WL);
  } else {
    // ================================================================ epilogue
    // TMEM -> bf16 -> staging tile (row blocks of 128 bytes, 16-byte chunk index XORed with (row & 7): the layout
    // the tensor map's 128-byte swizzle expects, and conflict-free for these row-per-thread writes) -> one TMA
    // store per 64-label block.  Two staging buffers: the store of tile i is read out of shared memory while
    // tile i + 1 is drained into the other buffer.
    const int ep = warp - C::W_EPI;
    const int q = ep & 3, h = ep >> 2;                       // TMEM lane quarter (= warp index mod 4), column half
    const int row = q * 32 + lane;
    const bool storer = (ep == 0 && lane == 0);
    int it = 0;
    if constexpr (TOPK) {
      constexpr int CAPW = 2 * C::CSTAGE / C::N_EPI / 8;     // entries of this warp's list
      static_assert(CAPW >= 32, "one entry per lane fits an empty list");
      uint2* list = reinterpret_cast<uint2*>(sm + C::OFF_C) + ep * CAPW;     // .x label, .y bf16 logit << 16 | batch row
      int count = 0;                                         // warp-uniform
      auto flush = [&]() {
        __syncwarp();
        for (int i0 = lane; i0 < count; i0 += 128) {         // four atomics per lane in flight
          uint2 e[4];
          int slot[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            slot[x] = a.cap;
            if (i0 + 32 * x < count) {
              e[x] = list[i0 + 32 * x];
              slot[x] = atomicAdd(a.cnt + static_cast<int64_t>(e[x].y & 0xFFFFu) * TopkFilter::CNT_STRIDE, 1);
            }
          }
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (slot[x] < a.cap)
              a.cand[static_cast<int64_t>(e[x].y & 0xFFFFu) * a.cap + slot[x]] = topk_key(__uint_as_float(e[x].y & 0xFFFF0000u), e[x].x);
        }
        count = 0;
        __syncwarp();
      };
      for (int gi = 0; gi < n_my_groups; ++gi) {
        const int l0 = a.set.tile(blockIdx.x + gi * gridDim.x) * G;
        const int rows_real = static_cast<int>(imin64(G, a.L - l0)), first_label = a.label0 + l0;
        for (int t = 0; t < T; ++t, ++it) {
          const int zs = it & 1;
          const int b = t * BT + row;
          const uint2 cut = b < a.B ? __ldg(reinterpret_cast<const uint2*>(a.cut) + b) : make_uint2(0x7F807F80u, 0u);   // rows beyond the batch: +inf, never passed
          const uint32_t thr2 = __byte_perm(cut.x, 0u, first_label < static_cast<int>(cut.y) ? 0x1010 : 0x3232);
          const float thr = __uint_as_float(thr2 & 0xFFFF0000u);
          const bool ok = mbar_wait(bar(C::B_ZFULL + zs), (it >> 1) & 1, abort_flag, a.err, 27, WL);
          tc_fence_after();
          const uint32_t ta = tmem + (static_cast<uint32_t>(q * 32) << 16) + zs * G + h * C::EC;
          constexpr int CW = C::EC < 32 ? C::EC : 32;            // columns per TMEM load
          // All of the tile's columns at once, so that the accumulator goes back before they are looked at (chunk by chunk: 670 K labels, 512
          // rows 280 us for the whole top-k, so 258).
          uint32_t ra[C::EC / CW][CW];
          __syncwarp();
#pragma unroll
          for (int x = 0; x < C::EC / CW; ++x) tmem_ld(ta + x * CW, ra[x]);
          tmem_ld_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar(C::B_ZEMPTY + zs));
#pragma unroll
          for (int c0 = 0; c0 < C::EC; c0 += CW) {
            const uint32_t (&r)[CW] = ra[c0 / CW];
            uint32_t p[CW / 2], m[CW / 2];
#pragma unroll
            for (int x = 0; x < CW / 2; ++x) m[x] = p[x] = pack2(__uint_as_float(r[2 * x]), __uint_as_float(r[2 * x + 1]));
#pragma unroll
            for (int w = CW / 4; w > 0; w >>= 1)
#pragma unroll
              for (int x = 0; x < w; ++x) m[x] = max2(m[x], m[x + w]);
            const float best = fmaxf(__uint_as_float(m[0] << 16), __uint_as_float(m[0] & 0xFFFF0000u));
            if (!__any_sync(0xffffffffu, best > thr)) continue;
            const int col0 = h * C::EC + c0, nvalid = rows_real - col0;      // columns of this chunk that are real labels
            // bit x: column 2x (lower half of p[x]), bit 16 + x: column 2x + 1
            uint32_t hit = 0u;
#pragma unroll
            for (int x = 0; x < CW / 2; ++x) hit |= gt2_mask(p[x], thr2) & ((1u << x) | (0x10000u << x));
            if (nvalid < CW) hit &= nvalid <= 0 ? 0u : ((1u << ((nvalid + 1) >> 1)) - 1u) | (((1u << (nvalid >> 1)) - 1u) << 16);
            if (!ok || *abort_flag) hit = 0u;
            // One entry per lane and round; nearly always one round is enough.  (523 K labels, 512 rows: 148 us with 16-column
            // loads; a prefix sum over the lanes' counts and sixteen predicated stores per lane in its place: 181 us.)
            for (unsigned any; (any = __ballot_sync(0xffffffffu, hit != 0u)) != 0u;) {
              if (count + 32 > CAPW) flush();
              if (hit != 0u) {
                const int x = __ffs(hit) - 1;
                uint32_t v = p[0];
#pragma unroll
                for (int y = 1; y < CW / 2; ++y) v = (x & 15) == y ? p[y] : v;
                const uint32_t bits = (x & 16) ? (v & 0xFFFF0000u) : (v << 16);
                list[count + __popc(any & ((1u << lane) - 1u))] =
                    make_uint2(static_cast<uint32_t>(first_label + col0 + 2 * (x & 15) + (x >> 4)), bits | static_cast<uint32_t>(b));
                hit &= hit - 1u;
              }
              count += __popc(any);
            }
          }
        }
      }
      flush();
    } else {
    for (int gi = 0; gi < n_my_groups; ++gi) {
      const int g = blockIdx.x + gi * gridDim.x;
      const int l0 = g * G;
      for (int t = 0; t < T; ++t, ++it) {
        const int zs = it & 1;
        const bool ok = mbar_wait(bar(C::B_ZFULL + zs), (it >> 1) & 1, abort_flag, a.err, 27, WL);
        tc_fence_after();
        const uint32_t ta = tmem + (static_cast<uint32_t>(q * 32) << 16) + zs * G + h * C::EC;
        // the store that last read this staging buffer (two tiles ago) has finished reading: the storing thread
        // waited for that before it arrived here
        named_bar_sync(1, C::N_EPI * 32);
        uint8_t* cst = sm + C::OFF_C + zs * C::CSTAGE;
        const int chunk0 = h * (C::EC / 8);
#pragma unroll 1
        for (int c16 = 0; c16 < C::EC; c16 += 16) {
          uint32_t r[16];
          __syncwarp();
          tmem_ld16(ta + c16, r);
          tmem_ld_wait();
#pragma unroll
          for (int e8 = 0; e8 < 16; e8 += 8) {
            const uint4 v = make_uint4(pack2(__uint_as_float(r[e8 + 0]), __uint_as_float(r[e8 + 1])),
                                       pack2(__uint_as_float(r[e8 + 2]), __uint_as_float(r[e8 + 3])),
                                       pack2(__uint_as_float(r[e8 + 4]), __uint_as_float(r[e8 + 5])),
                                       pack2(__uint_as_float(r[e8 + 6]), __uint_as_float(r[e8 + 7])));
            *reinterpret_cast<uint4*>(cst + C::c_chunk(row, chunk0 + ((c16 + e8) >> 3))) = v;
          }
        }
        tc_fence_before();
        fence_proxy_async();                                  // the staging writes become visible to the TMA store
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(C::B_ZEMPTY + zs));
        named_bar_sync(2, C::N_EPI * 32);                     // the whole staging tile is written
        if (storer) {
          if (ok && !*abort_flag) {
#pragma unroll
            for (int cb = 0; cb < C::NCB; ++cb)
              tma_store_2d(&tm_z, sbase + C::OFF_C + zs * C::CSTAGE + cb * C::CBLK, l0 + cb * 64, t * BT);
          }
          bulk_commit();
          bulk_wait_read<1>();                                // the previous tile's store has left its buffer
        }
        // The tensor-map store writes whole 16-byte chunks.  When the writable width is not a multiple of 8 columns,
        // its last columns (they lie in the last group) come out of the staging tile with 2-byte stores, one batch
        // row per thread.  The buffer is not rewritten before these threads pass the next tile's first barrier.
        const int tail0 = static_cast<int>(a.zw & ~int64_t(7)), tail_n = static_cast<int>(a.zw - tail0);
        if (tail_n > 0 && h == 0 && tail0 >= l0 && tail0 < l0 + G && ok && !*abort_flag && t * BT + row < a.B) {
          const int tc = (tail0 - l0) >> 3;                   // chunk index inside the group's row
          const uint4 v = *reinterpret_cast<const uint4*>(sm + C::OFF_C + zs * C::CSTAGE + C::c_chunk(row, tc));
          const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
          uint16_t* dst = reinterpret_cast<uint16_t*>(a.z) + (static_cast<int64_t>(t) * BT + row) * a.ldz + tail0;
#pragma unroll
          for (int i = 0; i < 7; ++i)
            if (i < tail_n) dst[i] = static_cast<uint16_t>(w4[i >> 1] >> ((i & 1) * 16));
        }
      }
    }
    if (storer) bulk_wait<0>();
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, C::TM_COLS);
  // every copy into this CTA's shared memory lands before it exits (without an abort the issuer has waited for all of them)
  if (warp == 2 && lane == 0 && *abort_flag) drain_x_ring<NXS, C::NPW, C::NSH>(bar(C::B_XFULL), x_last, WL);
}

template <int GG_, int FF_, int P_>
static int launch_shape(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t L,
                        int64_t ldz, int64_t zw, int64_t ldxt, const TileSet& set, const TopkFilter* tk, cudaStream_t st) {
  using C = Cfg<GG_, FF_, P_>;
  if (int rc = report_pending_status("tcgen05 forward")) return rc;
  int* err_dev = nullptr;
  if (int rc = device_status_word(&err_dev)) return rc;
  FwdArgs a;
  a.loc = loc; a.bias = static_cast<const __nv_bfloat16*>(bias); a.z = static_cast<__nv_bfloat16*>(z); a.err = err_dev;
  a.B = B; a.L = L; a.ldz = ldz; a.zw = zw; a.D = static_cast<int>(D); a.set = set;
  a.NG = set.count(static_cast<int>((L + C::G - 1) / C::G));
  a.NGR = static_cast<int>((L + C::GG - 1) / C::GG);
  a.wait_limit = wait_limit_cycles();
  a.cut = nullptr; a.cand = nullptr; a.cnt = nullptr; a.cap = 0; a.label0 = 0;
  if (tk) { a.cut = tk->cut; a.cand = tk->cand; a.cnt = tk->cnt; a.cap = tk->cap; a.label0 = tk->label0; }
  CUtensorMap tm_x, tm_w, tm_z;
  if (int rc = make_tmap_bf16_2d(&tm_x, xt, static_cast<uint64_t>(ldxt), static_cast<uint64_t>(D), static_cast<uint64_t>(ldxt) * 2, 64, 1)) return rc;
  if (int rc = make_tmap_bf16_2d(&tm_w, w, static_cast<uint64_t>(C::FF), static_cast<uint64_t>(L), static_cast<uint64_t>(C::FF) * 2, C::FF == 32 ? 32 : 64, C::G)) return rc;
  // the store clips at the writable width, in whole 16-byte chunks (columns L..zw-1 of the last group receive the
  // zeros its absent weight rows produce); the kernel writes the remaining zw % 8 columns itself
  if (tk) tm_z = tm_w;                          // not used
  else if (zw < 8) return fail(HASTE_ERR_UNSUPPORTED, "tcgen05 forward: writable width below 8 columns");
  else if (int rc = make_tmap_bf16_2d(&tm_z, z, static_cast<uint64_t>(zw & ~int64_t(7)), static_cast<uint64_t>(B), static_cast<uint64_t>(ldz) * 2, C::G == 32 ? 32 : 64, C::BT)) return rc;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = a.NG < sms ? a.NG : sms;
  auto k = tk ? ffi_forward_sm100_kernel<GG_, FF_, P_, true> : ffi_forward_sm100_kernel<GG_, FF_, P_, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  if (e != cudaSuccess) return fail(HASTE_ERR_LAUNCH, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  k<<<grid, C::NTHREADS, C::SMEM_BYTES, st>>>(a, tm_x, tm_w, tm_z);
  return check_launch("ffi_forward_sm100_kernel");
}

}  // namespace f100

bool forward_sm100_supported(const void* z, const void* xt, const void* w, int64_t B, int64_t F, int64_t L, int64_t G, int64_t ldz, int64_t ldxt) {
  // tensor maps need 16-byte aligned bases and row strides; coordinates are 32-bit
  const bool shape = (G == 128 && F == 64) || (G == 64 && (F == 128 || F == 64)) || (G == 32 && (F == 128 || F == 64 || F == 32));
  return shape && (ldxt % 8) == 0 && (ldz % 8) == 0 && aligned16(z) && aligned16(xt) &&
         aligned16(w) && L < (int64_t(1) << 31) && ldxt < (int64_t(1) << 31);
}

#define HASTE_F100_SHAPES(...)                                                     \
  if (G == 128 && F == 64) return f100::launch_shape<128, 64, 1>(__VA_ARGS__);    \
  if (G == 64 && F == 128) return f100::launch_shape<64, 128, 1>(__VA_ARGS__);    \
  if (G == 64 && F == 64) return f100::launch_shape<64, 64, 1>(__VA_ARGS__);      \
  if (G == 32 && F == 64) return f100::launch_shape<32, 64, 2>(__VA_ARGS__);      \
  if (G == 32 && F == 128) return f100::launch_shape<32, 128, 1>(__VA_ARGS__);    \
  if (G == 32 && F == 32) return f100::launch_shape<32, 32, 2>(__VA_ARGS__);      \
  return fail(HASTE_ERR_UNSUPPORTED, "tcgen05 forward: no kernel for group size %lld, fan-in %lld", (long long)G, (long long)F);

int launch_forward_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t F,
                         int64_t L, int64_t G, int64_t ldz, int64_t zw, int64_t ldxt, cudaStream_t st) {
  HASTE_F100_SHAPES(loc, xt, w, bias, z, B, D, L, ldz, zw, ldxt, TileSet(), nullptr, st)
}

int forward_tile_labels_sm100(int64_t F, int64_t G) { return G == 32 && F < 128 ? 64 : static_cast<int>(G); }

int launch_forward_tiles_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, void* z, int64_t B, int64_t D, int64_t F,
                               int64_t L, int64_t G, int64_t ldz, int64_t cols, int64_t ldxt, const TileSet& set, cudaStream_t st) {
  HASTE_F100_SHAPES(loc, xt, w, bias, z, B, D, L, ldz, (cols + 7) / 8 * 8, ldxt, set, nullptr, st)
}

int launch_topk_filter_sm100(const int32_t* loc, const void* xt, const void* w, const void* bias, int64_t B, int64_t D, int64_t F, int64_t L,
                             int64_t G, int64_t ldxt, const TopkFilter& tk, cudaStream_t st) {
  if (B > 65536) return fail(HASTE_ERR_UNSUPPORTED, "top-k filter: batch %lld too large", (long long)B);      // 16 bits of a list entry
  HASTE_F100_SHAPES(loc, xt, w, bias, nullptr, B, D, L, 0, 0, ldxt, tk.set, &tk, st)
}
#undef HASTE_F100_SHAPES

}  // namespace haste
