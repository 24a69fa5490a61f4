// Mixture-of-experts routing and token shuffling.
//   moe_route:   router logits [T, E] fp32 -> top-k weights / expert ids per token (softmax-all -> top-k -> optional
//                renormalise, or top-k -> softmax over the k, or sigmoid scores with correction and group limits), per-expert histogram, exclusive offsets and the permutation
//                that groups (token, slot) pairs by expert — one kernel launch + one small scan kernel.
//   moe_gather:  x [T, H] -> xs [T*k, H] rows in expert-grouped order (any element type).
//   moe_combine: ys [T*k, H] (expert outputs in grouped order) -> out [T, H] = sum_j w[t, j] * ys[pos(t, j)]  (fp32 sum in
//                slot order: deterministic, no atomics).
// Reference semantics: core/.../model/MixtureOfExpertsBlock.java:78-112, qwen3/Qwen3MoeFeedForward.java:107-301,
// granitemoehybrid/GraniteMoeHybridMoeFeedForward.java:112-141.
#include "common.cuh"
#include "gemm_api.h"

namespace dlv {

// Top-k of one token by one warp (E <= 1024, k <= 16): softmax statistics, k rounds of "every lane proposes its best remaining expert"
// (ties -> lower index), weights by `mode` (0: softmax over all experts, then top-k, optional renormalisation; 1: softmax over
// the k chosen; 2: sigmoid scores with a correction and group limits, see MoeRouting). Lanes store weights and expert ids, add to the histogram `counts` (global or shared memory) and, when
// `idx_copy` is given, keep a second copy of the ids there.
// best (value, index) of the warp, lower index on ties
__device__ __forceinline__ void warp_best(float& v, int& i) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, i, o);
    if (ov > v || (ov == v && oi < i)) {
      v = ov;
      i = oi;
    }
  }
}
__device__ __forceinline__ float route_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

// Groups (bit g) whose experts may be chosen: the `keep` groups with the largest sums of their two best choice scores.
__device__ __forceinline__ unsigned long long moe_kept_groups(const float* __restrict__ row, int E, const MoeRouting& r, int lane) {
  if (r.groups <= 1 || r.keep >= r.groups) return ~0ull;
  const int size = E / r.groups;
  float score[kMoeMaxGroups / 32];
#pragma unroll
  for (int j = 0; j < kMoeMaxGroups / 32; ++j) {
    const int g = lane + 32 * j;
    score[j] = -INFINITY;
    if (g >= r.groups) continue;
    float a = -INFINITY, b = -INFINITY;  // the two best
    for (int e = g * size; e < (g + 1) * size; ++e) {
      const float v = route_sigmoid(row[e]) + (r.correction != nullptr ? r.correction[e] : 0.f);
      if (v > a) {
        b = a;
        a = v;
      } else if (v > b) {
        b = v;
      }
    }
    score[j] = size > 1 ? a + b : a;
  }
  unsigned long long kept = 0ull;
  for (int n = 0; n < r.keep; ++n) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < kMoeMaxGroups / 32; ++j) {
      const int g = lane + 32 * j;
      if (g < r.groups && !((kept >> g) & 1ull) && (score[j] > bv || bi == 0x7fffffff)) {
        bv = score[j];
        bi = g;
      }
    }
    warp_best(bv, bi);
    kept |= 1ull << (bi & 63);
  }
  return kept;
}

// Order of floats as unsigned integers, -0 as 0; nothing (and what is not a number) below everything.
__device__ __forceinline__ unsigned order_key(float v) {
  const unsigned u = __float_as_uint(v + 0.f);
  return v != v ? 0u : (u & 0x80000000u ? ~u : u | 0x80000000u);
}

// NV experts per lane (expert lane + 32 j; 4, 8, 16, 24 or 32: with 32 for all beyond 256, and the half of the warps that its registers leave, one launch took 122 us for 128 tokens x 300
// experts, and 76 with 16): they stay in registers through all rounds, a round is one warp-wide maximum of their order and one minimum of the index, and
// lane r keeps what round r chose. (With the chosen ones in arrays of a thread, which a loop of run-time length puts into local memory, and five shuffles of two
// words per round, one block routed 32 tokens over 128 experts in 21.8 us and 64 over 8 in 15.3.)
template <int NV>
__device__ __forceinline__ void moe_topk_rows(const float* __restrict__ row, int E, int k, const MoeRouting& rt, int lane, float* __restrict__ w_out,
                                              int* __restrict__ idx_out, int* counts, int* idx_copy) {
  const int mode = rt.mode;
  float v[NV], mx = -INFINITY, den = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) v[j] = lane + 32 * j < E ? row[lane + 32 * j] : 0.f;
  if (mode == 2) {
    const unsigned long long kept = moe_kept_groups(row, E, rt, lane);
    const int group = rt.groups > 1 ? E / rt.groups : E;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int e = lane + 32 * j;
      if (e < E) v[j] = (kept >> (e / group)) & 1ull ? route_sigmoid(v[j]) + (rt.correction != nullptr ? rt.correction[e] : 0.f) : -INFINITY;
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (lane + 32 * j < E) mx = fmaxf(mx, v[j]);
    mx = warp_max(mx);
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (lane + 32 * j < E) den += __expf(v[j] - mx);
    den = warp_sum(den);
  }
  unsigned left = 0u;  // experts that may still be chosen
#pragma unroll
  for (int j = 0; j < NV; ++j)
    if (lane + 32 * j < E) left |= 1u << j;
  float sel_v = -INFINITY;
  int sel_i = 0;
  for (int r = 0; r < k; ++r) {
    unsigned bk = 0u;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const unsigned key = (left >> j) & 1u ? order_key(v[j]) : 0u;
      if (key > bk) {  // (of equal ones the lower index)
        bk = key;
        bv = v[j];
        bi = lane + 32 * j;
      }
    }
    const unsigned best = __reduce_max_sync(0xffffffffu, bk);
    const int i = static_cast<int>(__reduce_min_sync(0xffffffffu, bk == best && best != 0u ? static_cast<unsigned>(bi) : 0x7fffffffu));
    const float chosen = __shfl_sync(0xffffffffu, bv, i & 31);
    const int at = i < E ? i : 0;  // (not a number among the logits: stay inside the tables)
    if (lane == r) {
      sel_v = i < E ? chosen : -INFINITY;
      sel_i = at;
    }
    if ((at & 31) == lane) left &= ~(1u << (at >> 5));
  }
  // weights: lane r those of round r, summed in order
  float wt = 0.f;
  if (lane < k) {
    if (mode == 2) wt = route_sigmoid(row[sel_i]);
    else if (mode == 0) wt = __expf(sel_v - mx) / den;
  }
  if (mode == 1) {
    const float first = __shfl_sync(0xffffffffu, sel_v, 0);
    if (lane < k) wt = __expf(sel_v - first);
  }
  float s = 0.f;
  for (int r = 0; r < k; ++r) s += __shfl_sync(0xffffffffu, wt, r);
  if (mode == 2) wt = wt / (s + 1e-20f) * rt.scale;
  else if (mode == 1 || rt.renorm) wt /= s;
  if (lane < k) {
    w_out[lane] = wt;
    idx_out[lane] = sel_i;
    if (idx_copy != nullptr) idx_copy[lane] = sel_i;
    if (counts != nullptr) atomicAdd(&counts[sel_i], 1);
  }
}
// one warp per token
template <int NV>
__global__ void __launch_bounds__(256) moe_topk_kernel(const float* __restrict__ logits, int T, int E, int k, const MoeRouting rt,
                                                       float* __restrict__ w_out, int* __restrict__ idx_out, int* __restrict__ counts) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= T) return;
  moe_topk_rows<NV>(logits + static_cast<size_t>(t) * E, E, k, rt, lane, w_out + static_cast<size_t>(t) * k, idx_out + static_cast<size_t>(t) * k, counts,
                    nullptr);
}

// Routing of a decode-size batch in ONE launch of one CTA (32 warps; 24 above 512 experts and 16 above 768, whose scores take the registers): top-k per token, expert histogram and offsets, the stable
// permutation that groups (token, slot) pairs by expert, and the grouped GEMM's work list for the local experts [e0, e0 + ne)
// with `bn` rows per item. It replaces a memset and four launches (moe_topk, moe_sort, moe_items and, where the grouped GEMV reads
// token rows through `perm`, moe_gather), which cost more than the work at a few hundred pairs. Shared memory: T k + 2 E + ne + 3
// ints. Same results as the separate kernels (same tie rule, same stable order).
constexpr int kRouteSmallMaxPairs = 8192;
constexpr int kRouteSmallMaxTokens = 128;  // a warp takes every 32nd token: beyond a few tokens per warp the many-CTA kernels win
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  return v;
}
template <int NV, int THREADS>
__global__ void __launch_bounds__(THREADS) moe_route_small_kernel(const float* __restrict__ logits, int T, int E, int k, const MoeRouting rt,
                                                               float* __restrict__ w_out, int* __restrict__ idx_out, int* __restrict__ counts,
                                                               int* __restrict__ offsets, int* __restrict__ perm, int* __restrict__ pos, int e0,
                                                               int ne, int bn, int max_items, int4* __restrict__ items) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  extern __shared__ int rs[];
  const int P = T * k;
  int* idx_s = rs;              // [P] expert of every (token, slot) pair
  int* cnt_s = idx_s + P;       // [E]
  int* off_s = cnt_s + E;       // [E + 1]
  int* first_s = off_s + E + 1; // [ne + 1] first work item of every local expert
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < E; e += THREADS) cnt_s[e] = 0;
  __syncthreads();
  for (int t = warp; t < T; t += THREADS / 32)
    moe_topk_rows<NV>(logits + static_cast<size_t>(t) * E, E, k, rt, lane, w_out + static_cast<size_t>(t) * k, idx_out + static_cast<size_t>(t) * k, cnt_s,
                      idx_s + t * k);
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the histogram: lane l owns a contiguous chunk of experts
    const int chunk = (E + 31) / 32, lo = min(E, lane * chunk), hi = min(E, lo + chunk);
    int sum = 0;
    for (int e = lo; e < hi; ++e) sum += cnt_s[e];
    const int incl = warp_incl_scan(sum, lane);
    int acc = incl - sum;
    for (int e = lo; e < hi; ++e) {
      off_s[e] = acc;
      acc += cnt_s[e];
    }
    if (lane == 31) off_s[E] = incl;
  } else if (warp == 1 && items != nullptr) {  // the same over the local experts' item counts
    const int chunk = (ne + 31) / 32, lo = min(ne, lane * chunk), hi = min(ne, lo + chunk);
    int sum = 0;
    for (int e = lo; e < hi; ++e) sum += (cnt_s[e0 + e] + bn - 1) / bn;
    const int incl = warp_incl_scan(sum, lane);
    int acc = incl - sum;
    for (int e = lo; e < hi; ++e) {
      first_s[e] = acc;
      acc += (cnt_s[e0 + e] + bn - 1) / bn;
    }
    if (lane == 31) first_s[ne] = incl;
  }
  __syncthreads();
  for (int e = tid; e <= E; e += THREADS) offsets[e] = off_s[e];
  for (int e = tid; e < E; e += THREADS) counts[e] = cnt_s[e];
  // stable grouping: a warp takes an expert and walks the pairs 32 at a time (ballot + prefix count keeps ascending pair order)
  for (int e = warp; e < E; e += THREADS / 32) {
    if (cnt_s[e] == 0) continue;
    int row = off_s[e];
    for (int p0 = 0; p0 < P; p0 += 32) {
      const int p = p0 + lane;
      const bool mine = p < P && idx_s[p] == e;
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (mine) {
        const int r = row + __popc(m & ((1u << lane) - 1u));
        perm[r] = p;
        pos[p] = r;
      }
      row += __popc(m);
    }
  }
  if (items != nullptr) {
    for (int e = tid; e < ne; e += THREADS) {
      const int lo = off_s[e0 + e], hi = off_s[e0 + e + 1];
      int it = first_s[e];
      for (int r = lo; r < hi && it < max_items; r += bn, ++it) items[it] = make_int4(e, r, hi, 0);
    }
    for (int it = first_s[ne] + tid; it < max_items; it += THREADS) items[it] = make_int4(-1, 0, 0, 0);
  }
}

// single CTA: exclusive scan of counts -> offsets[E + 1]; then a stable counting sort of (token, slot) pairs by expert.
// pos[t * k + j] = row of that pair in the grouped order; perm[row] = t * k + j.
__global__ void __launch_bounds__(1024) moe_sort_kernel(const int* __restrict__ idx, const int* __restrict__ counts, int T, int E, int k,
                                                        int* __restrict__ offsets, int* __restrict__ perm, int* __restrict__ pos) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  extern __shared__ int sh[];  // E + 1 offsets
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) {
      sh[e] = acc;
      acc += counts[e];
    }
    sh[E] = acc;
  }
  __syncthreads();
  for (int e = threadIdx.x; e <= E; e += blockDim.x) offsets[e] = sh[e];
  // stable order inside an expert: ascending (token, slot). One thread per expert walks the pairs of its expert.
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int row = sh[e];
    if (counts[e] == 0) continue;
    for (int p = 0; p < T * k; ++p) {
      if (idx[p] == e) {
        perm[row] = p;
        pos[p] = row;
        ++row;
      }
    }
  }
}

// The same grouping for prefill-size batches, in parallel. The single-CTA kernel above walks all T k pairs once per expert (one
// thread each): 2.5 ms for the 65,536 pairs of an 8,192-token chunk with 128 experts, two thirds of the whole MoE block at prefill.
// Here the pairs are cut into chunks (sort_chunk): (a) every chunk counts its pairs per expert, (b) one CTA turns the expert
// histogram into offsets and the chunk counts into the first row of every (chunk, expert), (c) one warp per chunk hands out the
// rows in pair order (__match_any_sync groups the lanes of one expert; the group's first lane advances the running row). The
// order is the stable one: ascending pair index inside an expert.
// Chunks of 256 pairs spread the ranks over more warps; but one CTA scans the counts of all chunks, with fewer than four threads per expert beyond 256 experts. So those take
// chunks of 1,024 above 8,192 pairs (all of the routing, 131,072 pairs, two per token: 300 experts 194 us with 256, 106 with 1,024; 512 experts 206 and 109; 128 experts 79 and 48).
static int sort_chunk(long long pairs, int E) { return E > 256 && pairs > 8192 ? 1024 : 256; }
constexpr int kSortSerialMaxPairs = 256;  // up to here the single-CTA kernel is used (us there and in the three launches: 260 pairs of 8 experts 12.8 and 8.6, 884 pairs 36.5 and 8.6)
__global__ void __launch_bounds__(256) moe_chunk_hist_kernel(const int* __restrict__ idx, int P, int E, int chunk, int* __restrict__ chunk_hist) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  extern __shared__ int hs[];  // [E]
  for (int e = threadIdx.x; e < E; e += blockDim.x) hs[e] = 0;
  __syncthreads();
  const int p0 = blockIdx.x * chunk, p1 = min(P, p0 + chunk);
  for (int p = p0 + threadIdx.x; p < p1; p += blockDim.x) atomicAdd(&hs[idx[p]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) chunk_hist[static_cast<size_t>(blockIdx.x) * E + e] = hs[e];
}
// chunk_hist [C, E]: counts on entry, first grouped row of the (chunk, expert) on exit. Threads of neighbouring experts read a chunk's row together, and as many
// threads as there are take an expert's chunks in stretches, eight counts in flight. (One thread per expert, a load and a store behind one another for each of 64
// chunks: 11 us; a warp per expert, whose lanes read a column: 70 us at 256 chunks.)
__global__ void __launch_bounds__(1024) moe_chunk_scan_kernel(int* __restrict__ counts, int E, int C, int* __restrict__ offsets, int* __restrict__ chunk_hist) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  extern __shared__ int sh[];  // [E + 1] first rows, then [stretches][E] counts of an expert's stretches
  const int S = 1024 / E > 0 ? 1024 / E : 1, per = (C + S - 1) / S;
  int* part = sh + E + 1;
  const int st = static_cast<int>(threadIdx.x) / E, e = static_cast<int>(threadIdx.x) - st * E, c0 = st * per, c1 = min(C, c0 + per);
  int* col = chunk_hist + e;
  if (st < S) {
    int sum = 0;
#pragma unroll 8
    for (int c = c0; c < c1; ++c) sum += col[static_cast<size_t>(c) * E];
    part[st * E + e] = sum;
  }
  __syncthreads();
  if (st == 0) {
    int sum = 0;
    for (int i = 0; i < S; ++i) {  // counts of the stretches -> pairs in front of them
      const int n = part[i * E + e];
      part[i * E + e] = sum;
      sum += n;
    }
    counts[e] = sum;
    sh[e] = sum;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, chunk = (E + 31) / 32, lo = min(E, lane * chunk), hi = min(E, lo + chunk);
    int sum = 0;
    for (int i = lo; i < hi; ++i) sum += sh[i];
    const int incl = warp_incl_scan(sum, lane);
    int acc = incl - sum;
    for (int i = lo; i < hi; ++i) {
      const int n = sh[i];
      sh[i] = acc;
      acc += n;
    }
    if (lane == 31) sh[E] = incl;
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= E; i += blockDim.x) offsets[i] = sh[i];
  if (st < S) {
    int acc = sh[e] + part[st * E + e];
    for (int c = c0; c < c1; c += 8) {
      int n[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) n[i] = c + i < c1 ? col[static_cast<size_t>(c + i) * E] : 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c + i < c1) col[static_cast<size_t>(c + i) * E] = acc;
        acc += n[i];
      }
    }
  }
}
__global__ void __launch_bounds__(32) moe_chunk_rank_kernel(const int* __restrict__ idx, int P, int E, int chunk, const int* __restrict__ chunk_base,
                                                            int* __restrict__ perm, int* __restrict__ pos) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  extern __shared__ int rk[];  // [E] running row per expert, then [chunk] the chunk's expert ids
  int* run_s = rk;
  int* idx_s = rk + E;
  const int lane = threadIdx.x;
  const int p0 = blockIdx.x * chunk, n = min(P - p0, chunk);
  for (int e = lane; e < E; e += 32) run_s[e] = chunk_base[static_cast<size_t>(blockIdx.x) * E + e];
  for (int i = lane; i < n; i += 32) idx_s[i] = idx[p0 + i];
  __syncwarp();
  for (int q = 0; q < n; q += 32) {
    const int i = q + lane;
    const bool valid = i < n;
    const int e = valid ? idx_s[i] : -1 - lane;  // (lanes past the end each form a group of their own)
    const unsigned m = __match_any_sync(0xffffffffu, e);
    const int r = __popc(m & ((1u << lane) - 1u));
    const int base = valid ? run_s[e] : 0;
    __syncwarp();
    if (valid && r == 0) run_s[e] = base + __popc(m);
    __syncwarp();
    if (valid) {
      perm[base + r] = p0 + i;
      pos[p0 + i] = base + r;
    }
  }
}

__global__ void __launch_bounds__(128) moe_gather_kernel(const uint4* __restrict__ x, const int* __restrict__ perm, int k, int row_vecs,
                                                         uint4* __restrict__ xs, const int* __restrict__ offsets, int e0, int ne) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  const int row = blockIdx.x;
  if (offsets != nullptr && (row < offsets[e0] || row >= offsets[e0 + ne])) return;  // another rank's expert
  const int t = perm[row] / k;
  const uint4* src = x + static_cast<size_t>(t) * row_vecs;
  uint4* dst = xs + static_cast<size_t>(row) * row_vecs;
  for (int i = threadIdx.x; i < row_vecs; i += blockDim.x) dst[i] = src[i];
}

__global__ void __launch_bounds__(128) moe_combine_kernel(const __nv_bfloat16* __restrict__ ys, const int* __restrict__ pos,
                                                          const float* __restrict__ w, int k, int H, __nv_bfloat16* __restrict__ out,
                                                          const int* __restrict__ offsets, int e0, int ne) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  const int t = blockIdx.x;
  // rows and weights of the token's slots first, then four slots' rows at a time (one after the other, each behind its slot's row number, made the kernel 8.5 us
  // for 32 tokens of eight)
  constexpr int kSlots = 64;  // (more slots look theirs up themselves)
  __shared__ int rows[kSlots];
  __shared__ float wts[kSlots];
  auto row_at = [&](int j) {
    const int r = pos[static_cast<size_t>(t) * k + j];
    return offsets == nullptr || (r >= offsets[e0] && r < offsets[e0 + ne]) ? r : -1;  // (computed on another rank: the all-reduce adds it)
  };
  if (static_cast<int>(threadIdx.x) < min(k, kSlots)) {
    rows[threadIdx.x] = row_at(threadIdx.x);
    wts[threadIdx.x] = w[static_cast<size_t>(t) * k + threadIdx.x];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    float acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0.f;
    for (int j0 = 0; j0 < k; j0 += 4) {
      uint4 v[4];
      int r[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        r[j] = j0 + j >= k ? -1 : (j0 + j < kSlots ? rows[j0 + j] : row_at(j0 + j));
        if (r[j] >= 0) v[j] = __ldg(reinterpret_cast<const uint4*>(ys + static_cast<size_t>(r[j]) * H) + i);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (r[j] < 0) continue;
        const float wt = j0 + j < kSlots ? wts[j0 + j] : w[static_cast<size_t>(t) * k + j0 + j];
        const uint32_t vu[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = unpack_bf162(vu[e]);
          acc[2 * e] += wt * f.x;
          acc[2 * e + 1] += wt * f.y;
        }
      }
    }
    uint4 o;
    uint32_t* ou = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
    for (int e = 0; e < 4; ++e) ou[e] = pack_bf162(acc[2 * e], acc[2 * e + 1]);
    reinterpret_cast<uint4*>(out + static_cast<size_t>(t) * H)[i] = o;
  }
}

// Ints of workspace launch_moe_route needs for T tokens (0: none, the single-CTA grouping is used)
size_t moe_route_workspace_ints(int T, int E, int k) {
  const long long P = static_cast<long long>(T) * k;
  return P > kSortSerialMaxPairs ? static_cast<size_t>((P + sort_chunk(P, E) - 1) / sort_chunk(P, E)) * E : 0;
}
void launch_moe_route(const float* logits, int T, int E, int k, const MoeRouting& r, float* w, int* idx, int* counts, int* offsets,
                      int* perm, int* pos, int* ws, cudaStream_t st) {
  const bool chunks = ws != nullptr && moe_route_workspace_ints(T, E, k) > 0;
  if (!chunks) cudaMemsetAsync(counts, 0, sizeof(int) * E, st);
  if (T == 0) {
    cudaMemsetAsync(offsets, 0, sizeof(int) * (E + 1), st);
    return;
  }
  // (the chunks count their pairs themselves: 65,536 atomics on 128 counters were most of the 36 us of 8,192 tokens)
  int* histogram = chunks ? nullptr : counts;
  if (E <= 128) moe_topk_kernel<4><<<(T + 7) / 8, 256, 0, st>>>(logits, T, E, k, r, w, idx, histogram);
  else if (E <= 256) moe_topk_kernel<8><<<(T + 7) / 8, 256, 0, st>>>(logits, T, E, k, r, w, idx, histogram);
  else if (E <= 512) moe_topk_kernel<16><<<(T + 7) / 8, 256, 0, st>>>(logits, T, E, k, r, w, idx, histogram);
  else if (E <= 768) moe_topk_kernel<24><<<(T + 7) / 8, 256, 0, st>>>(logits, T, E, k, r, w, idx, histogram);
  else moe_topk_kernel<32><<<(T + 7) / 8, 256, 0, st>>>(logits, T, E, k, r, w, idx, histogram);
  const int P = T * k;
  if (chunks) {
    const int chunk = sort_chunk(P, E), C = (P + chunk - 1) / chunk;
    moe_chunk_hist_kernel<<<C, 256, sizeof(int) * E, st>>>(idx, P, E, chunk, ws);
    moe_chunk_scan_kernel<<<1, 1024, sizeof(int) * (E + 1 + 1024), st>>>(counts, E, C, offsets, ws);
    moe_chunk_rank_kernel<<<C, 32, sizeof(int) * (E + chunk), st>>>(idx, P, E, chunk, ws, perm, pos);
    return;
  }
  moe_sort_kernel<<<1, 1024, sizeof(int) * (E + 1), st>>>(idx, counts, T, E, k, offsets, perm, pos);
}
// Decode-size batches: everything of launch_moe_route + launch_moe_items in one launch. False when the batch is too large for it.
bool launch_moe_route_small(const float* logits, int T, int E, int k, const MoeRouting& r, float* w, int* idx, int* counts, int* offsets,
                            int* perm, int* pos, int e0, int ne, int bn, int max_items, int* items, cudaStream_t st) {
  if (T < 1 || T > kRouteSmallMaxTokens || T * k > kRouteSmallMaxPairs || E > 1024 || ne > 1024) return false;
  const size_t smem = sizeof(int) * (static_cast<size_t>(T) * k + 2 * E + ne + 3);
  const auto run = [&](auto kernel, int threads) {
    return launch_pdl(kernel, dim3(1), dim3(threads), smem, st, logits, T, E, k, r, w, idx, counts, offsets, perm, pos, e0, ne, bn, max_items,
                      reinterpret_cast<int4*>(items)) == cudaSuccess;
  };
  if (E <= 128) return run(moe_route_small_kernel<4, 1024>, 1024);
  if (E <= 256) return run(moe_route_small_kernel<8, 1024>, 1024);
  if (E <= 512) return run(moe_route_small_kernel<16, 1024>, 1024);
  if (E <= 768) return run(moe_route_small_kernel<24, 768>, 768);
  return run(moe_route_small_kernel<32, 512>, 512);
}
void launch_moe_gather(const void* x, const int* perm, int rows, int k, int row_bytes, void* xs, const int* offsets, int e0, int ne,
                       cudaStream_t st) {
  if (rows == 0) return;
  moe_gather_kernel<<<rows, 128, 0, st>>>(static_cast<const uint4*>(x), perm, k, row_bytes / 16, static_cast<uint4*>(xs), offsets, e0, ne);
}
void launch_moe_combine(const void* ys, const int* pos, const float* w, int T, int k, int H, void* out, const int* offsets, int e0,
                        int ne, cudaStream_t st) {
  if (T == 0) return;
  moe_combine_kernel<<<T, 128, 0, st>>>(static_cast<const __nv_bfloat16*>(ys), pos, w, k, H, static_cast<__nv_bfloat16*>(out), offsets, e0, ne);
}

// Work list of the grouped GEMM: one item {local expert, first row, end row, 0} per `bn` rows of every local expert that has
// rows, in expert order; the rest of the `max_items` slots get expert = -1. Single CTA (at most a few hundred items).
__global__ void __launch_bounds__(256) moe_items_kernel(const int* __restrict__ offsets, int e0, int ne, int bn, int max_items,
                                                        int4* __restrict__ items) {
  pdl_trigger();  // first: the next kernel may then be set up (and a GEMM prefetch its weights) while this one still waits
  pdl_wait();
  __shared__ int first[1025];
  if (ne <= 32) {  // (a lane per expert, no trip through shared memory)
    const int lane = threadIdx.x;
    if (lane < 32) {
      const int n = lane < ne ? (offsets[e0 + lane + 1] - offsets[e0 + lane] + bn - 1) / bn : 0, incl = warp_incl_scan(n, lane);
      if (lane < ne) first[lane] = incl - n;
      if (lane == 31) first[ne] = incl;
    }
  } else {
    for (int e = threadIdx.x; e < ne; e += blockDim.x) first[e] = (offsets[e0 + e + 1] - offsets[e0 + e] + bn - 1) / bn;
    __syncthreads();
  }
  if (ne > 32 && threadIdx.x < 32) {
    const int lane = threadIdx.x, chunk = (ne + 31) / 32, lo = min(ne, lane * chunk), hi = min(ne, lo + chunk);
    int sum = 0;
    for (int e = lo; e < hi; ++e) sum += first[e];
    const int incl = warp_incl_scan(sum, lane);
    int acc = incl - sum;
    for (int e = lo; e < hi; ++e) {
      const int n = first[e];
      first[e] = acc;
      acc += n;
    }
    if (lane == 31) first[ne] = incl;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ne; e += blockDim.x) {
    const int lo = offsets[e0 + e], hi = offsets[e0 + e + 1];
    int it = first[e];
    if (bn > 256) {  // wide items: an expert's rows in equal ones, since an item costs its kernel one expansion of the weights whatever its rows
      const int count = (hi - lo + bn - 1) / bn, per = count > 0 ? (hi - lo + count - 1) / count : 1;
      for (int r = lo; r < hi && it < max_items; r += per, ++it) items[it] = make_int4(e, r, min(hi, r + per), 0);
      continue;
    }
    for (int r = lo; r < hi && it < max_items; r += bn, ++it) items[it] = make_int4(e, r, hi, 0);
  }
  for (int it = first[ne] + threadIdx.x; it < max_items; it += blockDim.x) items[it] = make_int4(-1, 0, 0, 0);
}
void launch_moe_items(const int* offsets, int e0, int ne, int bn, int max_items, int* items, cudaStream_t st) {
  if (ne > 1024) return;
  moe_items_kernel<<<1, 256, 0, st>>>(offsets, e0, ne, bn, max_items, reinterpret_cast<int4*>(items));
}

}  // namespace dlv
