// Running per-row top-k over logits that arrive in label chunks (inference: the reference takes
// torch.topk(logits, 100) / topk(5) over the full [B,L] logits, src/evaluate.py:151-156, 219).
//
// The forward kernels produce a chunk of logits z[b, 0..C) for labels col0 .. col0+C-1 (a chunk is sized to stay
// in L2); this kernel folds it into the running top-k of every row, so the [B,L] matrix never exists.  One CTA per
// row keeps the row's current best k values (sorted, descending) and their label ids in shared memory.  A logit
// is a candidate only if it beats the current k-th value; after the first few hundred labels candidates are rare
// (about k ln(L/k) per row over the whole label set); the candidates of a range of slices are merged into the kept
// list in one step (every element computes its new position).  Equal values keep the lower label id first, which
// makes the result unique.
#include "common.cuh"
#include "launchers.h"

namespace haste {

constexpr int TK_THREADS = 128;
constexpr int TK_KMAX = 128;                 // k <= TK_THREADS: one thread per kept entry during an insertion
constexpr int TK_CAND = TK_THREADS * 8;      // candidates of one 1024-label slice
constexpr int TK_WIDE = 16;                  // slices scanned between two synchronisations once candidates are rare
constexpr int TK_BATCH = 4;                  // slices whose loads a thread has in flight at a time

__global__ void __launch_bounds__(TK_THREADS) topk_update_kernel(const uint16_t* __restrict__ z, int64_t ldz, int64_t C, int64_t col0, int k,
                                                                 float* __restrict__ vals, int32_t* __restrict__ idx) {
  __shared__ float sv[TK_KMAX];
  __shared__ int si[TK_KMAX];
  __shared__ float cv[TK_CAND];
  __shared__ int ci[TK_CAND];
  __shared__ int ncand;
  const int tid = threadIdx.x;
  const int64_t b = blockIdx.x;
  const uint16_t* zr = z + b * ldz;
  if (tid < k) { sv[tid] = vals[b * k + tid]; si[tid] = idx[b * k + tid]; }
  if (tid == 0) ncand = 0;
  __syncthreads();
  const bool vec_ok = (reinterpret_cast<uintptr_t>(zr) & 15) == 0;
  // Scans labels [c0, c0 + n_sub * 1024) of the chunk against the current k-th value and inserts what passes.  Returns
  // false, with nothing inserted, when more candidates passed than the buffer holds (only while the threshold is
  // still loose: the caller then repeats the range in 1024-label slices, which always fit).
  auto scan_and_insert = [&](int64_t c0, int n_sub) -> bool {
    const float thr = sv[k - 1];
    for (int sub0 = 0; sub0 < n_sub; sub0 += TK_BATCH) {
      // 8 consecutive labels per thread and 1024-label slice; TK_BATCH slices' loads are issued before any is looked at
      // (the scan is a stream out of L2: what it needs is bytes in flight)
      uint4 v[TK_BATCH];
      int64_t j0[TK_BATCH];
#pragma unroll
      for (int u = 0; u < TK_BATCH; ++u) {
        j0[u] = c0 + static_cast<int64_t>(sub0 + u) * TK_CAND + static_cast<int64_t>(tid) * 8;
        v[u] = make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);     // -inf: never a candidate
        if (sub0 + u < n_sub && j0[u] < C) {
          if (vec_ok && j0[u] + 8 <= C) {
            v[u] = *reinterpret_cast<const uint4*>(zr + j0[u]);
          } else {
            uint16_t t[8];
#pragma unroll
            for (int p = 0; p < 8; ++p) t[p] = (j0[u] + p < C) ? zr[j0[u] + p] : uint16_t(0xFF80);
            v[u] = make_uint4(t[0] | (uint32_t(t[1]) << 16), t[2] | (uint32_t(t[3]) << 16), t[4] | (uint32_t(t[5]) << 16), t[6] | (uint32_t(t[7]) << 16));
          }
        }
      }
#pragma unroll
      for (int u = 0; u < TK_BATCH; ++u) {
        const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int p = 0; p < 8; ++p) {
          const float e = (p & 1) ? __uint_as_float(w[p >> 1] & 0xFFFF0000u) : __uint_as_float(w[p >> 1] << 16);
          if (e > thr) {                                      // -inf never passes; a NaN logit is never selected
            const int slot = atomicAdd(&ncand, 1);
            if (slot < TK_CAND) { cv[slot] = e; ci[slot] = static_cast<int>(col0 + j0[u] + p); }
          }
        }
      }
    }
    __syncthreads();
    const int n = ncand;
    __syncthreads();
    if (tid == 0) ncand = 0;
    if (n > TK_CAND) { __syncthreads(); return false; }
    // ---- merge the candidates into the kept list, up to TK_THREADS at a time.  Every element's new position is the
    // number of elements ahead of it (larger value, or equal value and lower label id: a strict order, label ids are
    // distinct): a kept entry moves down by the candidates ahead of it, a candidate lands behind the kept entries
    // ahead of it (binary search in the sorted list) and the other candidates ahead of it.  Two barriers per batch,
    // however many candidates it holds.
    for (int base = 0; base < n; base += TK_THREADS) {
      const int m = min(TK_THREADS, n - base);
      float ov = 0.f, cvv = 0.f;
      int oi = 0, cid = 0, opos = k, cpos = k;
      if (tid < k) {
        ov = sv[tid]; oi = si[tid];
        int ahead = 0;
        for (int c = 0; c < m; ++c) {
          const float v = cv[base + c];
          ahead += (v > ov) || (v == ov && ci[base + c] < oi);
        }
        opos = tid + ahead;
      }
      if (tid < m) {
        cvv = cv[base + tid]; cid = ci[base + tid];
        int lo = 0, hi = k;                                   // first kept entry that is not ahead of the candidate
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          const bool ahead = sv[mid] > cvv || (sv[mid] == cvv && si[mid] >= 0 && si[mid] < cid);
          if (ahead) lo = mid + 1; else hi = mid;
        }
        int ahead_c = 0;
        for (int c = 0; c < m; ++c) {
          const float v = cv[base + c];
          ahead_c += (v > cvv) || (v == cvv && ci[base + c] < cid);
        }
        cpos = lo + ahead_c;
      }
      __syncthreads();
      if (opos < k) { sv[opos] = ov; si[opos] = oi; }
      if (cpos < k) { sv[cpos] = cvv; si[cpos] = cid; }
      __syncthreads();
    }
    __syncthreads();
    return true;
  };
  // Once the threshold has tightened candidates are rare (about k ln(L/k) per row over the whole label set), so the
  // chunk is walked in ranges of TK_WIDE slices with one synchronisation per range instead of one per slice.
  for (int64_t c0 = 0; c0 < C; c0 += static_cast<int64_t>(TK_WIDE) * TK_CAND) {
    const bool loose = sv[k - 1] == -INFINITY;                // fewer than k labels seen so far: every label is a candidate
    if (loose || !scan_and_insert(c0, TK_WIDE)) {
      for (int sub = 0; sub < TK_WIDE && c0 + static_cast<int64_t>(sub) * TK_CAND < C; ++sub) scan_and_insert(c0 + static_cast<int64_t>(sub) * TK_CAND, 1);
    }
  }
  if (tid < k) { vals[b * k + tid] = sv[tid]; idx[b * k + tid] = si[tid]; }
}

int launch_topk_update(const void* z, int64_t ldz, int64_t B, int64_t C, int64_t col0, int k, float* vals, int32_t* idx, cudaStream_t st) {
  if (B == 0 || C == 0) return HASTE_OK;
  topk_update_kernel<<<static_cast<unsigned>(B), TK_THREADS, 0, st>>>(static_cast<const uint16_t*>(z), ldz, C, col0, k, vals, idx);
  return check_launch("topk_update_kernel");
}


// ================================================================ whole top-k with a filtered forward
// The chunked path above writes every logit to L2 and reads it back once (670 K labels, 512 rows: 686 MB each way).  Here
// only the logits of a sample of at most TF_FIRST labels are stored, whole label tiles evenly spread over the layer; a row's k-th
// best of them is a bar that all but k * (labels of the launch / labels before it) of the other logits fail, so the forward's
// epilogue filters them in registers (TOPK instantiations of the tcgen05 forward) and a merge kernel folds the survivors in.
// Each launch covers at most TF_GROW times the labels seen before it, again evenly spread: TF_GROW * k candidates a row
// are expected, against a list of TF_CAP.  The spread makes that hold for any order of the labels: where logits rise with the
// label id at most about TF_GROW * (k + a tile) pass, where all are equal the label ids decide likewise.  (With the first 16 K
// labels as the sample, 670 K labels whose biases rise with the id took 14.2 ms for 512 rows, a masked first 16 K labels
// 5.2 ms, against 0.28 ms in random order; now 0.28 to 0.30 for all of them.)
// A row whose list overflows all the same (logits periodic in the sample's step) is computed again by the merge kernel on the
// CUDA cores, the same result up to the order of the fp32 sums: all 512 rows of 670 K labels 3.9 ms.
constexpr int TF_THREADS = 256;
constexpr int64_t TF_FIRST = 148 * 128, TF_GROW = 8;      // the sample: a tile on every SM at G = 128
constexpr int TF_CAP = 8192;
// Rows per pass over the layer: a row takes 64 KiB of candidates and up to 37 KiB of sample logits, so larger batches go through
// in slices that reuse the same 430 MB.  A slice costs one more set of launches and one more read of the weights: with 1024 rows
// 8192 rows of 670 K labels took 4,069 us, undivided (820 MB) 3,723; the chunked path takes 7,650.
constexpr int64_t TF_ROWS = 4096;
typedef unsigned long long u64;

// The keys that can be among the k best of n: all that are not below the k-th largest of the maxima of NT / lanes groups of
// `lanes` threads (a key below it has k better ones).  key(i) for i < n, 0 = no entry; non-zero keys are distinct.  At most
// k * ceil(n / NT) * lanes pass.  Ranking the maxima takes NT / lanes steps of every thread, so a small k takes few groups
// (keep_lanes).  Returns the number kept; all threads call it, and it ends with a barrier.
template <int NT, class KEY>
__device__ __forceinline__ int keep_candidates(KEY key, int n, int k, int lanes, u64* out, u64* s_max, u64* s_tau, int* s_n) {
  const int tid = threadIdx.x;
  u64 m = 0;
#pragma unroll 4
  for (int i = tid; i < n; i += NT) { const u64 v = key(i); m = v > m ? v : m; }
  for (int o = 1; o < lanes; o <<= 1) { const u64 v = __shfl_xor_sync(0xffffffffu, m, o); m = v > m ? v : m; }
  const int groups = NT / lanes;
  if (tid % lanes == 0) s_max[tid / lanes] = m;
  if (tid == 0) { *s_tau = 0; *s_n = 0; }
  __syncthreads();
  if (tid < groups) {
    const u64 mine = s_max[tid];
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < groups; ++j) rank += s_max[j] > mine;
    if (mine != 0 && rank == k - 1) *s_tau = mine;
  }
  __syncthreads();
  const u64 tau = *s_tau;
#pragma unroll 4
  for (int i = tid; i < n; i += NT) {
    const u64 v = key(i);
    if (v != 0 && v >= tau) out[atomicAdd(s_n, 1)] = v;
  }
  __syncthreads();
  return *s_n;
}
// Threads per group: the most (a power of two up to a warp) that leave 2k groups and keep the bound on what passes small.
static int keep_lanes(int64_t n, int k, int nt) {
  int lanes = 1;
  while (lanes < 32 && nt / (2 * lanes) >= (2 * k > 32 ? 2 * k : 32) && static_cast<int64_t>(k) * ((n + nt - 1) / nt) * 2 * lanes <= 2048) lanes *= 2;
  return lanes;
}
static int64_t keep_bound(int64_t n, int k, int nt) { return static_cast<int64_t>(k) * ((n + nt - 1) / nt) * keep_lanes(n, k, nt); }

// The bar that the k-th best key sets (0: fewer than k so far, any number passes).  Just below 0 stands the largest normal
// negative number: compares may flush what lies between, and what passes in addition only has to be looked at.
__device__ __forceinline__ RowCut row_cut(u64 key, int label) {
  if (key == 0) return {0xFF80FF80u, 0};
  const uint32_t v = __float_as_uint(topk_key_value(key)) >> 16;           // a bf16 above -inf, not -0
  const uint32_t below = (v & 0x8000u) ? v + 1u : v <= 0x0080u ? 0x8080u : v - 1u;
  return {(v << 16) | below, label};
}

// The k best of keys[0..s) in order, to vals / idx (label ids: label(what the keys hold); -inf / -1 where there are fewer), and the
// bar they set to *cut when cut != NULL.
struct SameLabel { __device__ int operator()(int l) const { return l; } };
template <int NT, class LABEL = SameLabel>
__device__ __forceinline__ void write_best(const u64* keys, int s, int k, float* vals, int32_t* idx, RowCut* cut, LABEL label = LABEL()) {
  const int tid = threadIdx.x;
  for (int i = tid; i < k; i += NT)
    if (i >= s) { vals[i] = -INFINITY; idx[i] = -1; }
  if (tid == 0 && cut != nullptr && s < k) *cut = row_cut(0, 0);
  for (int i = tid; i < s; i += NT) {
    const u64 v = keys[i];
    int rank = 0;
#pragma unroll 4
    for (int j = 0; j < s; ++j) rank += keys[j] > v;
    if (rank < k) {
      vals[rank] = topk_key_value(v);
      idx[rank] = label(topk_key_label(v));
      if (cut != nullptr && rank == k - 1) *cut = row_cut(v, idx[rank]);
    }
  }
}
__device__ __forceinline__ u64 logit_key(uint16_t bits, uint32_t label) {
  const float v = bf16_bits_to_float(bits);
  return v > -INFINITY ? topk_key(v, label) : 0ull;                 // -inf and NaN are never selected
}

// The sample: the k best of z[b, 0..C) (column c holds label col0 + c / tile * stride + c % tile, tile a power of two); also the
// bar they set and the row's empty candidate list.  Rows are 16-byte aligned and their length is that of whole chunks (the forward writes zeros past C, which are masked here).
// The threads' maxima are found on packed bf16 pairs, eight logits per load; equal logits around the k-th maximum may let more
// through than the list holds, and then the keys decide (which order equal logits by label).
// The kernel with keys throughout took 33 us for 512 rows.
__device__ __forceinline__ uint32_t max2u(uint32_t x, uint32_t y) {          // a NaN loses against a number
  const __nv_bfloat162 v = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float max8(const uint4& v) {
  const uint32_t m = max2u(max2u(v.x, v.y), max2u(v.z, v.w));
  return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xFFFF0000u));
}
__global__ void __launch_bounds__(TF_THREADS) topk_first_kernel(const uint16_t* __restrict__ z, int64_t ldz, int C, uint32_t col0, int tile,
                                                                uint32_t stride, int k, int cap, float* __restrict__ vals, int32_t* __restrict__ idx,
                                                                RowCut* __restrict__ row_cuts, int* __restrict__ cnt) {
  extern __shared__ __align__(16) u64 kept[];
  __shared__ u64 s_max[TF_THREADS], s_tau;
  __shared__ __align__(16) float s_val[TF_THREADS];
  __shared__ float s_cut;
  __shared__ int s_n;
  const int tid = threadIdx.x;
  const int64_t b = blockIdx.x;
  const uint16_t* zr = z + b * ldz;
  const uint4* z4 = reinterpret_cast<const uint4*>(zr);
  const int whole = C >> 3;                                                  // chunks without a masked column
  const int tile_log = __ffs(tile) - 1;
  auto label_of = [&](int c) { return static_cast<int>(col0 + static_cast<uint32_t>(c >> tile_log) * stride + static_cast<uint32_t>(c & (tile - 1))); };
  float m = -INFINITY;
#pragma unroll 4
  for (int c = tid; c < whole; c += TF_THREADS) m = fmaxf(m, max8(z4[c]));   // fmaxf drops a NaN
  for (int c = whole * 8 + tid; c < C; c += TF_THREADS) m = fmaxf(m, bf16_bits_to_float(zr[c]));
  s_val[tid] = m;
  if (tid == 0) { s_cut = -INFINITY; s_n = 0; }
  __syncthreads();
  int rank = 0;
#pragma unroll 8
  for (int j = 0; j < TF_THREADS; j += 4) {
    const float4 v = *reinterpret_cast<const float4*>(s_val + j);
    rank += (v.x > m || (v.x == m && j < tid)) + (v.y > m || (v.y == m && j + 1 < tid)) + (v.z > m || (v.z == m && j + 2 < tid)) +
            (v.w > m || (v.w == m && j + 3 < tid));
  }
  if (rank == k - 1) s_cut = m;
  __syncthreads();
  const float cut = s_cut;
  auto take = [&](uint16_t bits, int c) {
    const float v = bf16_bits_to_float(bits);
    if (v >= cut && v > -INFINITY) {
      const int slot = atomicAdd(&s_n, 1);
      if (slot < cap) kept[slot] = topk_key(v, static_cast<uint32_t>(c));
    }
  };
#pragma unroll 4
  for (int c = tid; c < whole; c += TF_THREADS) {
    const uint4 v = z4[c];
    if (max8(v) >= cut) {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) take(static_cast<uint16_t>(w[e >> 1] >> ((e & 1) * 16)), c * 8 + e);
    }
  }
  for (int c = whole * 8 + tid; c < C; c += TF_THREADS) take(zr[c], c);
  __syncthreads();
  int s = s_n;
  if (s > cap) {                                                             // uniform
    __syncthreads();
    s = keep_candidates<TF_THREADS>([&](int i) { return logit_key(zr[i], static_cast<uint32_t>(i)); }, C, k, 1, kept, s_max, &s_tau, &s_n);
  }
  write_best<TF_THREADS>(kept, s, k, vals + b * k, idx + b * k, row_cuts + b, label_of);      // the keys hold columns
  if (tid == 0) cnt[b * TopkFilter::CNT_STRIDE] = 0;
}

// Merge: the row's kept list and its candidates -> kept list, threshold; the candidate list is emptied.
constexpr int TM_LIST = 2048 + TF_THREADS;          // recomputation: running list ...
constexpr int TM_KEEP = TK_KMAX * ((TM_LIST + TF_THREADS - 1) / TF_THREADS);      // ... and what a compaction of it can keep
constexpr int TM_KEYS = TK_KMAX * ((TF_CAP + TK_KMAX + TF_THREADS - 1) / TF_THREADS);
static_assert(TM_LIST + TM_KEEP <= TM_KEYS, "the recomputation works inside the merge's buffer");

struct TopkMergeArgs {
  const int32_t* loc;
  const uint16_t *xt, *w, *bias;
  const u64* cand;
  float* vals;
  RowCut* cut;
  int32_t* idx;
  int* cnt;
  int64_t L, ldxt;
  int D, F, G, k, tile;                             // tile: labels of a tile
  TileSet set;                                      // tiles of the launch the candidates come from ...
  int n_tiles;                                      // ... and their number
  uint32_t label0;
};

__global__ void __launch_bounds__(TF_THREADS) topk_merge_kernel(TopkMergeArgs a) {
  __shared__ __align__(16) u64 keys[TM_KEYS];
  __shared__ u64 s_max[TF_THREADS], s_tau;
  __shared__ int s_n, s_list;
  const int tid = threadIdx.x, k = a.k;
  const int64_t b = blockIdx.x;
  float* vals = a.vals + b * k;
  int32_t* idx = a.idx + b * k;
  const int n = a.cnt[b * TopkFilter::CNT_STRIDE];
  if (n == 0) return;                               // uniform: nothing beat the kept list
  auto kept = [&](int i) { const int id = idx[i]; return id < 0 ? 0ull : topk_key(vals[i], static_cast<uint32_t>(id)); };
  int s;
  if (n <= TF_CAP) {
    const u64* c = a.cand + b * TF_CAP;
    s = keep_candidates<TF_THREADS>([&](int i) { return i < n ? c[i] : kept(i - n); }, n + k, k, 1, keys, s_max, &s_tau, &s_n);
  } else {
    // every logit of the launch again: 256 threads take 256 / G groups at a time, one label each
    __shared__ float xs[TF_THREADS / 16][128];      // gathered features of these groups
    u64* best = keys + TM_LIST;
    if (tid == 0) s_list = k;
    if (tid < k) keys[tid] = kept(tid);
    u64 kth = kept(k - 1);
    __syncthreads();
    const int per = TF_THREADS / a.G, gl = tid / a.G, r = tid % a.G;
    const int gpt = a.tile / a.G;                   // groups of a tile
    const int64_t NG = (a.L + a.G - 1) / a.G;       // of the layer
    const int n_groups = a.n_tiles * gpt;       // of the launch
    for (int g0 = 0; g0 < n_groups; g0 += per) {
      auto group = [&](int i) { return g0 + i < n_groups ? static_cast<int64_t>(a.set.tile((g0 + i) / gpt)) * gpt + (g0 + i) % gpt : NG; };
      for (int i = tid; i < per * a.F; i += TF_THREADS) {
        const int64_t g = group(i / a.F);
        float v = 0.f;
        if (g < NG) {
          const int d = min(max(__ldg(a.loc + g * a.F + i % a.F), 0), a.D - 1);
          v = bf16_bits_to_float(__ldg(a.xt + static_cast<int64_t>(d) * a.ldxt + b));
        }
        xs[i / a.F][i % a.F] = v;
      }
      __syncthreads();
      const int64_t l = group(gl) * a.G + r;
      if (l < a.L) {
        float acc = 0.f;
        const uint4* wr = reinterpret_cast<const uint4*>(a.w + l * a.F);
        for (int c = 0; c < a.F / 8; ++c) {
          const uint4 v = __ldg(wr + c);
          const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc = fmaf(__uint_as_float(w4[j] << 16), xs[gl][c * 8 + 2 * j], acc);
            acc = fmaf(__uint_as_float(w4[j] & 0xFFFF0000u), xs[gl][c * 8 + 2 * j + 1], acc);
          }
        }
        if (a.bias != nullptr) acc += bf16_bits_to_float(a.bias[l]);
        const float z = round_to_bf16_f(acc);
        if (z > -INFINITY) {
          const u64 key = topk_key(z, a.label0 + static_cast<uint32_t>(l));
          if (key > kth) keys[atomicAdd(&s_list, 1)] = key;
        }
      }
      __syncthreads();
      if (s_list > TM_LIST - TF_THREADS) {          // uniform; room for one more round of labels is kept
        const int m = keep_candidates<TF_THREADS>([&](int i) { return keys[i]; }, s_list, k, 1, best, s_max, &s_tau, &s_n);
        for (int i = tid; i < m; i += TF_THREADS) {
          int rank = 0;
          for (int j = 0; j < m; ++j) rank += best[j] > best[i];
          if (rank < k) { keys[rank] = best[i]; if (rank == k - 1) s_max[0] = best[i]; }
        }
        if (tid == 0) s_list = min(m, k);
        __syncthreads();
        if (m >= k) kth = s_max[0];
        __syncthreads();
      }
    }
    const int m = keep_candidates<TF_THREADS>([&](int i) { return keys[i]; }, s_list, k, 1, best, s_max, &s_tau, &s_n);
    for (int i = tid; i < m; i += TF_THREADS) keys[i] = best[i];
    __syncthreads();
    s = m;
  }
  __syncthreads();
  write_best<TF_THREADS>(keys, s, k, vals, idx, a.cut + b);
  if (tid == 0) a.cnt[b * TopkFilter::CNT_STRIDE] = 0;
}

// ================================================================ a few rows: bandwidth-bound product on the CUDA cores
// With up to TS_ROWS batch rows the layer is one read of the weights, and a 128-row tensor-core tile is nearly all padding.
// Grid: segments of whole label groups, at least two per SM where the layer is large enough.  A warp takes TS_UNIT label
// rows at a time: lane = (row of the load, 16-byte chunk), the gathered features of its 8 slots in registers, all loads of
// the unit issued before the first product.  The segment's logits stay in shared memory, where the block picks the
// k best of every batch row; topk_parts_kernel merges the segments.
constexpr int TS_ROWS = 8, TS_UNIT = 16, TS_THREADS = 256, TS_SEG = 4096, TS_MERGE = 1024;

template <int F, int NB>
__global__ void __launch_bounds__(TS_THREADS) topk_rows_kernel(const int32_t* __restrict__ loc, const uint16_t* __restrict__ x,
                                                               const uint16_t* __restrict__ w, const uint16_t* __restrict__ bias, int B, int D,
                                                               int64_t L, int G, int seg, int k, uint32_t label0, int lanes, u64* __restrict__ part) {
  constexpr int LPR = F / 8, RPL = 32 / LPR, NLD = TS_UNIT / RPL > 0 ? TS_UNIT / RPL : 1;
  static_assert(RPL <= TS_UNIT && TS_UNIT % RPL == 0, "whole loads");
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ u64 s_max[TS_THREADS], s_tau;
  __shared__ int s_n;
  uint16_t* xs = reinterpret_cast<uint16_t*>(smem);                        // [NB][D]
  uint16_t* zs = xs + (static_cast<int64_t>(NB) * D + 7) / 8 * 8;          // [NB][seg]
  u64* kept = reinterpret_cast<u64*>(zs + NB * seg);                       // seg % 16 == 0
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t l_beg = static_cast<int64_t>(blockIdx.x) * seg;
  const int n_lab = static_cast<int>(imin64(seg, L - l_beg));
  for (int i = tid; i < NB * D; i += TS_THREADS) xs[i] = i < B * D ? x[i] : uint16_t(0);
  __syncthreads();
  const int c = lane % LPR, rl = lane / LPR;
  for (int u0 = warp * TS_UNIT; u0 < n_lab; u0 += TS_THREADS / 32 * TS_UNIT) {
    const int64_t l0 = l_beg + u0;                                         // TS_UNIT divides every group size: one group per unit
    uint4 wv[NLD];
#pragma unroll
    for (int j = 0; j < NLD; ++j) {
      const int64_t l = l0 + j * RPL + rl;
      wv[j] = l < L ? __ldg(reinterpret_cast<const uint4*>(w + l * F) + c) : make_uint4(0u, 0u, 0u, 0u);
    }
    const int4* lp = reinterpret_cast<const int4*>(loc + (l0 / G) * F + c * 8);
    const int4 i0 = __ldg(lp), i1 = __ldg(lp + 1);
    const int id[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
    float xf[NB][8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int d = min(max(id[j], 0), D - 1);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) xf[nb][j] = bf16_bits_to_float(xs[nb * D + d]);
    }
#pragma unroll
    for (int j = 0; j < NLD; ++j) {
      const uint32_t w4[4] = {wv[j].x, wv[j].y, wv[j].z, wv[j].w};
      const int64_t l = l0 + j * RPL + rl;
      const float bv = (bias != nullptr && l < L) ? bf16_bits_to_float(__ldg(bias + l)) : 0.f;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        float acc = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc = fmaf(__uint_as_float(w4[e] << 16), xf[nb][2 * e], acc);
          acc = fmaf(__uint_as_float(w4[e] & 0xFFFF0000u), xf[nb][2 * e + 1], acc);
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (c == 0 && u0 + j * RPL + rl < n_lab) zs[nb * seg + u0 + j * RPL + rl] = rn_bf16_bits(acc + bv);
      }
    }
  }
  __syncthreads();
  for (int b = 0; b < B; ++b) {
    const uint16_t* zb = zs + b * seg;
    const int s = keep_candidates<TS_THREADS>([&](int i) { return logit_key(zb[i], label0 + static_cast<uint32_t>(l_beg + i)); }, n_lab, k, lanes, kept,
                                              s_max, &s_tau, &s_n);
    u64* out = part + (static_cast<int64_t>(b) * gridDim.x + blockIdx.x) * k;
    for (int i = tid; i < k; i += TS_THREADS)
      if (i >= s) out[i] = 0ull;
    for (int i = tid; i < s; i += TS_THREADS) {
      const u64 v = kept[i];
      int rank = 0;
      for (int j = 0; j < s; ++j) rank += kept[j] > v;
      if (rank < k) out[rank] = v;
    }
    __syncthreads();
  }
}

template <int NT>
__global__ void __launch_bounds__(NT) topk_parts_kernel(const u64* __restrict__ part, int n, int k, int lanes, float* __restrict__ vals,
                                                        int32_t* __restrict__ idx) {
  extern __shared__ __align__(16) u64 kept[];
  __shared__ u64 s_max[NT], s_tau;
  __shared__ int s_n;
  const int64_t b = blockIdx.x;
  const u64* p = part + b * n;
  const int s = keep_candidates<NT>([&](int i) { return p[i]; }, n, k, lanes, kept, s_max, &s_tau, &s_n);
  write_best<NT>(kept, s, k, vals + b * k, idx + b * k, nullptr);
}

// ---------------------------------------------------------------- host side
// Segment length of the few-rows kernel: whole groups, two blocks per SM, at most TS_SEG labels.
static int64_t rows_seg(int64_t L, int64_t G) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t NG = (L + G - 1) / G;
  int64_t gps = (NG + 2 * sms - 1) / (2 * sms);
  if (gps * G > TS_SEG) gps = TS_SEG / G;
  return gps * G;
}
static int64_t round16(int64_t v) { return (v + 15) / 16 * 16; }
static int pow2_rows(int64_t B) { return B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8; }
static size_t rows_smem(int64_t B, int64_t D, int64_t seg, int k) {
  const int64_t nb = pow2_rows(B);
  return static_cast<size_t>((nb * D + 7) / 8 * 16 + nb * seg * 2 + keep_bound(seg, k, TS_THREADS) * 8);
}
// Which path: 0 the chunked one (above), 1 few rows, 2 filtered forward.
// Few rows up to TS_ROWS: the filtered forward reads the same weights but pays five launches or more and a 128-row tile.  Few rows /
// filtered, us a call:  k = 5, 131 K labels (G=64, F=128): 1 row 26 / 67, 4 rows 28 / 66, 8 rows 44 / 66; 670 K labels (G=128, F=64):
// 40 / 102, 56 / 105, 83 / 105; 2.8 M labels: 115 / 289, 181 / 291, 320 / 292.  k = 100, where picking the best of every
// segment weighs more: 131 K 51 / 73, 77 / 74, 116 / 74; 670 K 72 / 110, 106 / 114, 156 / 114.  The line is drawn by the rows
// alone, so that a row's logits do not depend on k; it is right for small k and late for large.
static int topk_route(int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int k) {
  if (B <= TS_ROWS && (F == 16 || F == 32 || F == 64 || F == 128)) {
    const int64_t seg = rows_seg(L, G), parts = (L + seg - 1) / seg;
    if (rows_smem(B, D, seg, k) <= DYN_SMEM_MAX && keep_bound(parts * k, k, parts * k <= 4096 ? TS_THREADS : TS_MERGE) * 8 <= DYN_SMEM_MAX) return 1;
  }
  const bool shape = (G == 128 && F == 64) || (G == 64 && (F == 128 || F == 64)) || (G == 32 && (F == 128 || F == 64 || F == 32));
  if (shape && L < (int64_t(1) << 31) && D < (int64_t(1) << 31)) return 2;
  return 0;
}

// The launches of the filtered path: a sample (every `step`-th tile), then `launches` filter launches whose tile sets complete it,
// each TF_GROW times the labels before it at most.
struct FilterPlan {
  int tile, n_tiles, step = 1, launches = 0;
  int64_t sample;                                     // labels of the sample
  TileSet set[8];
};
static FilterPlan filter_plan(int64_t F, int64_t L, int64_t G) {
  FilterPlan p;
  p.tile = forward_tile_labels_sm100(F, G);
  p.n_tiles = static_cast<int>((L + p.tile - 1) / p.tile);
  const int first = static_cast<int>(TF_FIRST / p.tile);
  int64_t ratio = (p.n_tiles + first - 1) / first;    // at most 2^17: six launches
  for (int64_t reach = 1; reach < ratio; reach *= TF_GROW + 1) ++p.launches;
  int skip[8];
  for (int i = 0; i < p.launches; ++i) {              // factors as equal as whole numbers allow, their product is at least the ratio
    int r = 3;
    for (;; ++r) {
      int64_t reach = 1;
      for (int k = i; k < p.launches; ++k) reach *= r;
      if (reach >= ratio) break;
    }
    skip[i] = r;
    p.step *= r;
    ratio = (ratio + r - 1) / r;
  }
  for (int i = 0, step = p.step; i < p.launches; ++i) p.set[i] = TileSet(step /= skip[i], skip[i]);
  const int64_t sampled = (p.n_tiles + p.step - 1) / p.step, last = (sampled - 1) * p.step;
  p.sample = (sampled - 1) * p.tile + imin64(p.tile, L - last * p.tile);
  return p;
}

// Scratch of the filtered path, in bytes from a 16-byte aligned base: xt | logits of the sample | candidates | bars | counters
struct FusedScratch { int64_t xt, z, ldz, cand, cut, cnt, total; };
static FusedScratch fused_layout(int64_t B, int64_t D, const FilterPlan& p) {
  B = imin64(B, TF_ROWS);
  const int64_t ldxt = (B + 7) / 8 * 8;
  FusedScratch s;
  s.ldz = (p.sample + 7) / 8 * 8;
  s.xt = 0;
  s.z = round16(s.xt + D * ldxt * 2);
  s.cand = round16(s.z + B * s.ldz * 2);
  s.cut = s.cand + (p.launches > 0 ? B * TF_CAP * 8 : 0);
  s.cnt = round16(s.cut + B * static_cast<int64_t>(sizeof(RowCut)));
  s.total = round16(s.cnt + B * 4 * TopkFilter::CNT_STRIDE);
  return s;
}
int64_t topk_fused_scratch_bytes(int64_t B, int64_t D, int64_t F, int64_t L, int64_t G, int k) {
  switch (topk_route(B, D, F, L, G, k)) {
    case 1: { const int64_t seg = rows_seg(L, G); return B * ((L + seg - 1) / seg) * k * 8; }
    case 2: return fused_layout(B, D, filter_plan(F, L, G)).total;
    default: return 0;
  }
}

int launch_topk_fused(const int32_t* loc, const void* x, const void* w, const void* bias, void* scratch, int64_t B, int64_t D, int64_t F, int64_t L,
                      int64_t G, int k, int64_t label0, float* vals, int32_t* idx, cudaStream_t st) {
  const int route = topk_route(B, D, F, L, G, k);
  if (route == 1) {
    const int64_t seg = rows_seg(L, G), parts = (L + seg - 1) / seg;
    const size_t sm = rows_smem(B, D, seg, k);
    u64* part = static_cast<u64*>(scratch);
#define HASTE_TOPK_ROWS(F_, NB_)                                                                                             \
  {                                                                                                                          \
    auto kern = topk_rows_kernel<F_, NB_>;                                                                                   \
    if (int rc = allow_dynamic_smem(kern)) return rc;                                                                            \
    kern<<<static_cast<unsigned>(parts), TS_THREADS, sm, st>>>(loc, (const uint16_t*)x, (const uint16_t*)w, (const uint16_t*)bias, int(B), int(D), L, \
                                                               int(G), int(seg), k, static_cast<uint32_t>(label0), keep_lanes(seg, k, TS_THREADS), part);    \
  }
#define HASTE_TOPK_ROWS_NB(F_)                                                                                               \
  { switch (pow2_rows(B)) { case 1: HASTE_TOPK_ROWS(F_, 1) break; case 2: HASTE_TOPK_ROWS(F_, 2) break; case 4: HASTE_TOPK_ROWS(F_, 4) break; \
                            default: HASTE_TOPK_ROWS(F_, 8) } }
    if (F == 16) HASTE_TOPK_ROWS_NB(16) else if (F == 32) HASTE_TOPK_ROWS_NB(32) else if (F == 64) HASTE_TOPK_ROWS_NB(64) else HASTE_TOPK_ROWS_NB(128)
#undef HASTE_TOPK_ROWS_NB
#undef HASTE_TOPK_ROWS
    if (int rc = check_launch("topk_rows_kernel")) return rc;
    // few keys: 256 threads (their barriers and ranks cost less); many: 1024, which also keep the bound on the candidates
    const int64_t n = parts * k;
    const int nt = n <= 4096 ? TS_THREADS : TS_MERGE;
    auto merge = nt == TS_THREADS ? topk_parts_kernel<TS_THREADS> : topk_parts_kernel<TS_MERGE>;
    const size_t sm2 = static_cast<size_t>(keep_bound(n, k, nt)) * 8;
    if (int rc = allow_dynamic_smem(merge)) return rc;
    merge<<<static_cast<unsigned>(B), nt, sm2, st>>>(part, int(n), k, keep_lanes(n, k, nt), vals, idx);
    return check_launch("topk_parts_kernel");
  }
  if (route != 2) return fail(HASTE_ERR_UNSUPPORTED, "top-k: group size %lld, fan-in %lld, batch %lld take the chunked call", (long long)G, (long long)F, (long long)B);
  const FilterPlan plan = filter_plan(F, L, G);
  const FusedScratch fs = fused_layout(B, D, plan);
  char* base = static_cast<char*>(scratch);
  void* xt = base + fs.xt;
  uint16_t* z = reinterpret_cast<uint16_t*>(base + fs.z);
  RowCut* cut = reinterpret_cast<RowCut*>(base + fs.cut);
  int* cnt = reinterpret_cast<int*>(base + fs.cnt);
  u64* cand = reinterpret_cast<u64*>(base + fs.cand);
  const int cap = static_cast<int>(k * ((plan.sample + TF_THREADS - 1) / TF_THREADS));      // the bound of keep_candidates with single threads
  if (int rc = allow_dynamic_smem(topk_first_kernel)) return rc;
  for (int64_t b0 = 0; b0 < B; b0 += TF_ROWS) {
    const int64_t n = imin64(TF_ROWS, B - b0), ldxt = (n + 7) / 8 * 8;
    float* v = vals + b0 * k;
    int32_t* id = idx + b0 * k;
    if (int rc = launch_transpose(static_cast<const uint16_t*>(x) + b0 * D, xt, n, D, ldxt, false, st)) return rc;
    if (int rc = launch_forward_tiles_sm100(loc, xt, w, bias, z, n, D, F, L, G, fs.ldz, plan.sample, ldxt, TileSet(plan.step, 0), st)) return rc;
    topk_first_kernel<<<static_cast<unsigned>(n), TF_THREADS, static_cast<size_t>(cap) * 8, st>>>(
        z, fs.ldz, static_cast<int>(plan.sample), static_cast<uint32_t>(label0), plan.tile, static_cast<uint32_t>(plan.tile) * plan.step, k, cap, v, id, cut, cnt);
    if (int rc = check_launch("topk_first_kernel")) return rc;
    for (int i = 0; i < plan.launches; ++i) {
      const TopkFilter tk{cut, cand, cnt, TF_CAP, static_cast<int>(label0), plan.set[i]};
      if (int rc = launch_topk_filter_sm100(loc, xt, w, bias, n, D, F, L, G, ldxt, tk, st)) return rc;
      TopkMergeArgs a;
      a.loc = loc; a.xt = static_cast<const uint16_t*>(xt); a.w = static_cast<const uint16_t*>(w); a.bias = static_cast<const uint16_t*>(bias);
      a.cand = cand; a.vals = v; a.cut = cut; a.idx = id; a.cnt = cnt; a.L = L; a.ldxt = ldxt;
      a.D = int(D); a.F = int(F); a.G = int(G); a.k = k; a.tile = plan.tile; a.set = plan.set[i]; a.n_tiles = plan.set[i].count(plan.n_tiles);
      a.label0 = static_cast<uint32_t>(label0);
      topk_merge_kernel<<<static_cast<unsigned>(n), TF_THREADS, 0, st>>>(a);
      if (int rc = check_launch("topk_merge_kernel")) return rc;
    }
  }
  return HASTE_OK;
}

}  // namespace haste
