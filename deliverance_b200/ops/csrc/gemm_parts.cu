// GEMM  out[m, n] = sum_k X[m, k] * W[n, k]  for some dozens to some hundreds of rows, and for JQ4 experts, on pairs of SMs (tcgen05 cta_group::2),
// weights as the M operand: JQ4 out of tensor memory, bf16 out of shared memory.
//
// What bounds it: the tensor pipe for tiles of 256 tokens and more, the expansion of the weights (about 900 cycles per 128-k stage) for narrower
// ones. With 128 weight rows per CTA (gemm_tc.cuh) the activations alone ask for 64 bytes per cycle and SM, all that L2 gives, and expanding into
// shared memory (gemm_pair.cu) asks for 148 bytes per cycle of the 128 there are. Here a pair of CTAs takes 256 weight rows: each expands its own
// 128 into TENSOR MEMORY, from where the instruction reads them, and copies half of the tile's tokens (the N operand) into shared memory: at 384
// tokens 32 bytes per cycle from L2 and 84 of shared memory. A tile is up to 384 tokens wide, two instructions per 16 k, so that a weight is
// expanded once for all of them; its accumulators and two to four stages of weights fill tensor memory. Expanding is half of what the SM
// issues, so nothing else may be expensive: one commit per 128 k (each costs its thread more than a hundred cycles), and the expanding warps
// drain the accumulators themselves.
// bf16 weights come as TMA boxes in stages of 64 k beside their tokens (bound by HBM up to some 200 tokens, then by L2 and the pipe); sixteen warps only drain, and
// where a tile's accumulators fit twice the next tile runs meanwhile. Gate and up rows are fetched in turn by a five-dimensional box. Measured at gemm_parts_preferred.
//
// The tiles go to the pairs in whole waves. What is left over, or all of them where tiles are few, is cut over k into equal parts, whose fp32 sums a
// second small kernel adds up in order of k and finishes (plan_parts weighs it): 19456 x 2560 are 76 tiles on 74 pairs, 20 stages for everyone
// and 2 stages for twenty of them, not two waves of 20. No CTA waits for another pair.
//
// Roles per CTA: warps 0 and 2 copy tokens (of the first and the second instruction), warps 3 and 20 packed stages (bf16: warp 3 weights), warp 1 of the even CTA issues all
// MMAs of the pair, warp 2 owns tensor memory, warps 4-19 expand (two groups of four per 128-k stage, one per half, alternating) and drain.
// Barriers: x_full, a_full (even CTA) count both CTAs' copies and expanding warps; done (per stage: tokens and expanded weights may be overwritten)
// and acc_full are multicast commits; acc_empty (even CTA) counts both CTAs' draining warps. All waits are bounded as everywhere.
//
// Epilogues: 0 = store (+ bias); 1 = act(gate) * up: a CTA's 128 rows are 64 gate rows and the 64 up rows of the same outputs, fetched from the
// plain row order, eight of either in turn; 2 = q | k | v heads of 128 (per-head RMSNorm, rotation, paged cache write), all in the second kernel. Grouped
// mode (experts): whole tiles of the work items.
//
// It starts in ordinary stream order, as gemm_pair.cu does and for its reason.
//
// The reference multiplies prompts token by token on the CPU (native/src/main/c/simd/vector_simd.c:595).
#include <algorithm>
#include <cstdlib>
#include <stdexcept>
#include <string>

#include "divisor.h"
#include "gemm_api.h"
#include "gemm_tc.cuh"
#include "pair.cuh"

namespace dlv {

void encode_map_kchunks(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint64_t pitch_bytes, uint32_t box_rows, uint32_t chunks = 2);
void encode_map_gate_up(CUtensorMap* map, const void* base, uint64_t half, uint64_t K);

namespace {

constexpr int kMaxTokens = 384;               // accumulator columns; the rest of tensor memory holds two stages of weights
constexpr int kOneMma = 256;                  // tokens of one instruction
constexpr int kXRoom = 3 * (kMaxTokens / 2) * 256;  // one CTA's half of the tokens, 128 k: three stages of the widest tile, up to eight of others
constexpr int kMaxX = 8, kRawStages = 4, kMaxA = 4;
constexpr int kDrain = 16;                    // tokens that four draining warps turn at a time
constexpr int kDrainBytes = kDrain * (256 + 16);  // (16 bytes between rows: the eight rows of a stmatrix lie in different banks)
constexpr int kOffRaw = kXRoom;
constexpr int kOffDrain = kOffRaw + kRawStages * kQ4StageBytes;
constexpr int kOffCtrl = kOffDrain + 4 * 2 * kDrainBytes;
constexpr int kSmemBytes = kOffCtrl + 1024 + 1024;  // barriers + alignment slack
constexpr int kWStage = 128 * 128;            // bf16 weights: a CTA's 128 rows of a 64-k stage, in front of its tokens
constexpr int kStageRoom = kOffDrain;         // (they have the room of the packed stages too)
constexpr int kThreads = 672;
static_assert(kThreads == 640 + 32, "named barrier of the set-up");
static_assert(kSmemBytes <= 232448, "shared memory of an SM");

struct PartParams {
  int M, N;
  int kq;                 // stages of a tile: 128 k, bf16 weights 64 k
  int bn, box;            // tokens of a tile (a multiple of 32) and of a CTA's half of one instruction
  int x_stages;           // stages of tokens (bf16: and weights) in shared memory
  int slots;              // JQ4: stages of expanded weights in tensor memory (2 or 4); bf16: accumulators (2 where they fit)
  int n_tiles, m_tiles;   // grouped: m_tiles counts work items
  int pairs, waves;       // whole tiles: waves * pairs of them
  int parts;              // parts of each of the other tiles (0: there are none)
  int w_tiles;            // packed 128-row tiles of the weight (of one expert)
  int half;               // EPI 1: outputs per row (gate rows); the up rows follow them
  Divisor by_m, by_parts, by_group;  // m_tiles, parts, eight rows of weight tiles (grouped); the walk's divisions kept the first copies back by some 2,000 cycles
  const uint8_t* wq;
  void* out;
  int ldo, out_f32;
  int vec;                // outputs that may be stored at once: 1, 4 or 8
  const float* bias;
  float* sums;            // what the second kernel finishes: [slot][CTA][bn][128]
  const int4* items;
  int* status;
  int act_kind;
  GemmQkvArgs qkv;
};

struct Piece {
  int m0, m_lim, n_tile, expert;
  int k0, k1;   // stages
  int n1, n2;   // tokens of the first and the second instruction (multiples of 32; 0: there is no second one)
  int slot;     // where the sums go that the second kernel finishes, < 0: the drain does
};

// The pieces of a pair, in order. Every role walks them for itself. Slots: the parts of cut tiles first, then (EPI 2) whole tiles.
template <int EPI>
struct Walk {
  const PartParams& p;
  int pair, i;
  __device__ Walk(const PartParams& q, int pair_) : p(q), pair(pair_), i(-1) {}
  __device__ __forceinline__ void shape(Piece& o) {
    const int cols = (o.m_lim - o.m0 + 31) & ~31;
    o.n1 = cols <= 2 * p.box ? cols : ((cols >> 1) + 31) & ~31;
    o.n2 = cols - o.n1;
  }
  __device__ bool next(Piece& o) {
    if (p.items != nullptr) {
      // whole tiles pair, pair + pairs, ...: eight token tiles for one weight tile after the other, so that what runs at one time shares both through L2
      for (;;) {
        const int t = ++i * p.pairs + pair;
        if (t >= p.n_tiles * p.m_tiles) return false;
        constexpr int G = 8;
        const int g = p.by_group.of(t), r = t - g * G * p.n_tiles;
        const int rows = min(G, p.m_tiles - g * G);
        const int n = rows == G ? r / G : r / rows, m = g * G + (r - n * rows);
        const int4 it = p.items[m];
        if (it.x < 0) continue;
        o.m0 = it.y;
        o.m_lim = min(it.z, it.y + p.bn);
        o.n_tile = n;
        o.expert = it.x;
        o.k0 = 0;
        o.k1 = p.kq;
        o.slot = -1;
        shape(o);
        return true;
      }
    }
    int t;
    if (i < 0) {
      i = 0;
      const int cut = p.n_tiles * p.m_tiles - p.waves * p.pairs;
      if (pair < cut * p.parts) {
        const int which = p.by_parts.of(pair), part = pair - which * p.parts;
        t = p.waves * p.pairs + which;
        o.k0 = p.by_parts.of(part * p.kq);
        o.k1 = p.by_parts.of((part + 1) * p.kq);
        o.slot = EPI != 2 && p.parts == 1 ? -1 : pair;
        place(o, t);
        return true;
      }
    }
    if (i >= p.waves) return false;
    t = i++ * p.pairs + pair;
    o.k0 = 0;
    o.k1 = p.kq;
    o.slot = EPI != 2 ? -1 : (p.n_tiles * p.m_tiles - p.waves * p.pairs) * p.parts + t;
    place(o, t);
    return true;
  }
  __device__ __forceinline__ void place(Piece& o, int t) {
    o.n_tile = p.by_m.of(t);
    o.m0 = (t - o.n_tile * p.m_tiles) * p.bn;
    o.m_lim = min(p.M, o.m0 + p.bn);
    o.expert = 0;
    shape(o);
  }
};

// sixteen lanes of tensor memory x sixteen columns: lane l gets rows l / 4 and l / 4 + 8, columns 2 (l % 4) and + 1, then the same eight columns on
__device__ __forceinline__ void tmem_ld_16x256_x2(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

__device__ __forceinline__ float apply_act(int kind, float g) {
  if (kind == 2) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g)));
  // Both sides of the quotient at a quarter: __fdividef is 0 for divisors of 2^126 and more, which 1 + exp(-g) reaches in front of the end of its range. Its 2 ulp are a 2^-13th of the
  // rounding to bf16 behind the product (errors against 64 bits agree to seven digits with those of a division: 1.665046e-3, of the two kernels 3.1e-3); a division, in a drain that the
  // next tile waits for, took 4.3 us of the 38 of JQ4 19456 x 2560 with 333 rows, this multiplication 0.3 to 1.1.
  return __fdividef(0.25f * g, 0.25f + 0.25f * __expf(-g));
}

// What becomes of the sums of one token: a warp holds the token's 128 rows of a CTA's half tile, lane l rows 4 l .. + 3 (EPI 1: gate rows 2 l, 2 l + 1
// and up rows 2 l, 2 l + 1).
template <int EPI>
struct Finish {
  const PartParams& p;
  int lane, n;
  bool live;
  float add[4], nw[4];
  int head, kvh;
  bool is_q, is_k, normed, rotate;
  __device__ Finish(const PartParams& q, int n_tile, int rank, int lane_) : p(q), lane(lane_) {
    if constexpr (EPI == 1) {
      n = (n_tile * 2 + rank) * 64 + 2 * lane;
      live = n < p.half;
    } else {
      n = n_tile * 256 + rank * 128 + 4 * lane;
      live = EPI == 2 ? n_tile * 2 + rank < p.qkv.heads + 2 * p.qkv.kv_heads : n < p.N;
#pragma unroll
      for (int e = 0; e < 4; ++e) add[e] = p.bias != nullptr && n + e < p.N ? p.bias[n + e] : 0.f;
    }
    if constexpr (EPI == 2) {
      const GemmQkvArgs& a = p.qkv;
      head = n_tile * 2 + rank;
      is_q = head < a.heads;
      is_k = !is_q && head < a.heads + a.kv_heads;
      kvh = is_q ? 0 : (is_k ? head - a.heads : head - a.heads - a.kv_heads);
      const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(is_q ? a.q_norm_w : (is_k ? a.k_norm_w : nullptr));
      normed = w != nullptr;
      rotate = (is_q || is_k) && a.cos_t != nullptr;
#pragma unroll
      for (int e = 0; e < 4; ++e) nw[e] = normed && live ? bf2f(w[4 * lane + e]) + a.norm_offset : 0.f;
    }
  }
  // EPI 2: what a token's head needs beside the sums. It was there before the first kernel began, so the second one fetches it ahead of its wait.
  struct Token {
    float c[4], sn[4];
    long long slot;
  };
  __device__ void fetch(int m, Token& t) const {
    if constexpr (EPI == 2) {
      const GemmQkvArgs& a = p.qkv;
      t.slot = !is_q && a.slots != nullptr ? a.slots[m] : -1;
      if (rotate) {
        int pos = a.positions[m];
        pos = pos < 0 ? 0 : (pos >= a.max_pos ? a.max_pos - 1 : pos);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int d = ((4 * lane) & 63) + e;
          t.c[e] = d < a.rot_half ? __ldg(a.cos_t + static_cast<size_t>(pos) * a.rot_half + d) : 1.f;
          t.sn[e] = d < a.rot_half ? __ldg(a.sin_t + static_cast<size_t>(pos) * a.rot_half + d) : 0.f;
        }
      }
    }
  }
  __device__ void operator()(int m, const float (&s)[4], const Token& t) const {
    if constexpr (EPI == 0) {
      if (!live) return;
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = s[e] + add[e];
      const size_t o = static_cast<size_t>(m) * p.ldo + n;
      if (p.vec >= 4 && n + 3 < p.N) {
        if (p.out_f32) *reinterpret_cast<float4*>(static_cast<float*>(p.out) + o) = make_float4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + o) = make_uint2(pack_bf162(v[0], v[1]), pack_bf162(v[2], v[3]));
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (n + e < p.N) {
            if (p.out_f32) static_cast<float*>(p.out)[o + e] = v[e];
            else static_cast<__nv_bfloat16*>(p.out)[o + e] = f2bf(v[e]);
          }
        }
      }
    } else if constexpr (EPI == 1) {
      if (!live) return;
      const float a = apply_act(p.act_kind, s[0]) * s[2], b = apply_act(p.act_kind, s[1]) * s[3];
      __nv_bfloat16* o = static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo + n;
      *reinterpret_cast<uint32_t*>(o) = pack_bf162(a, b);
    } else {
      if (!live) return;  // (the whole warp)
      const GemmQkvArgs& a = p.qkv;
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = s[e] + add[e];
      if (normed) {
        const float inv = rsqrtf(warp_sum(v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3]) * (1.f / 128.f) + a.eps);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = bf2f(f2bf(v[e] * inv * nw[e]));  // rounded like a separate norm kernel would
      }
      if (rotate) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float other = __shfl_xor_sync(0xffffffffu, v[e], 16);  // dims d and d + 64 are 16 lanes apart
          if (((4 * lane) & 63) + e < a.rot_half) v[e] = lane < 16 ? v[e] * t.c[e] - other * t.sn[e] : v[e] * t.c[e] + other * t.sn[e];
        }
      }
      const uint2 pk = make_uint2(pack_bf162(v[0], v[1]), pack_bf162(v[2], v[3]));
      if (is_q) {
        *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo + head * 128 + 4 * lane) = pk;
      } else {
        if (t.slot >= 0) {
          const long long blk = t.slot / a.block_size, off = t.slot % a.block_size;
          __nv_bfloat16* cache = static_cast<__nv_bfloat16*>(is_k ? a.k_cache : a.v_cache);
          *reinterpret_cast<uint2*>(cache + ((blk * a.kv_heads + kvh) * a.block_size + off) * 128 + 4 * lane) = pk;
        }
      }
    }
  }
};


// the four sums of a lane out of a token's 128 (EPI 1: eight gate rows and the up rows of the same outputs in turn)
template <int EPI>
__device__ __forceinline__ void row_sums(const float* row, int lane, float (&s)[4]) {
  if constexpr (EPI == 1) {
    const float* at = row + (lane >> 2) * 16 + (2 * lane & 7);
    const float2 g = *reinterpret_cast<const float2*>(at), u = *reinterpret_cast<const float2*>(at + 8);
    s[0] = g.x; s[1] = g.y; s[2] = u.x; s[3] = u.y;
  } else {
    const float4 v = *reinterpret_cast<const float4*>(row + 4 * lane);
    s[0] = v.x; s[1] = v.y; s[2] = v.z; s[3] = v.w;
  }
}

template <bool Q4, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1) gemm_parts_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const PartParams p) {
  constexpr int NR = kRawStages;
  extern __shared__ uint8_t gr_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gr_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bar_x_full = reinterpret_cast<uint64_t*>(smem + kOffCtrl);
  uint64_t* bar_done = bar_x_full + kMaxX;
  uint64_t* bar_a_full = bar_done + kMaxX;
  uint64_t* bar_raw_full = bar_a_full + kMaxA;
  uint64_t* bar_raw_empty = bar_raw_full + NR;
  uint64_t* bar_acc_full = bar_raw_empty + NR;
  uint64_t* bar_acc_empty = bar_acc_full + 2;
  uint64_t* bar_turn = bar_acc_empty + 2;  // [4][2] sixteen tokens of a group's drain are complete in shared memory
  uint64_t* bar_last = bar_turn + 8;       // abort path: MMAs in flight have retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_last + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = __shfl_sync(0xffffffffu, static_cast<int>(cluster_ctarank()), 0);
  const int pair = static_cast<int>(blockIdx.x) >> 1;
  const int NA = p.slots, NX = p.x_stages;
  const bool two = p.bn > kOneMma;  // tiles may take a second instruction, whose tokens have a region of their own
  const int region = p.box * (Q4 ? 256 : 128), x_bytes = (two ? 2 * region : region) + (Q4 ? 0 : kWStage);  // one CTA's half of a stage
  const uint32_t NACC = Q4 ? 1 : NA;  // accumulators

  Piece pc;
  Walk<EPI> walk(p, pair);
  const bool any = walk.next(pc);
  auto copy_stage = [&](const Piece& o, int q, int s, int part, int parts) {
    // one lane copies a stage; EPI 1: four do, gate and up rows, nibbles and scales (`parts` = 2: gate or up rows by one of two warps)
    const uint32_t full = smem_u32(&bar_raw_full[s]);
    const uint8_t* src = p.wq + static_cast<size_t>(o.expert) * p.w_tiles * p.kq * kQ4StageBytes;
    uint32_t dst = 0, size = kQ4StageBytes;
    if (EPI == 1) {
      const int up = parts == 2 ? part : (lane >> 1) & 1, gates = p.half / 64, h = up * gates + min(o.n_tile * 2 + rank, gates - 1);
      const bool scales = (lane & 1) != 0;
      src += static_cast<size_t>(h >> 1) * p.kq * kQ4StageBytes + (scales ? 8192 + (h & 1) * 1024 : (h & 1) * 4096);
      dst = scales ? 8192 + up * 1024 : up * 4096;
      size = scales ? 1024 : 4096;
    } else {
      src += static_cast<size_t>(min(o.n_tile * 2 + rank, p.w_tiles - 1)) * p.kq * kQ4StageBytes;  // (past the last tile: computed and dropped)
    }
    if (lane == 0 && part == 0) mbar_expect_tx(full, kQ4StageBytes);  // (of both warps; the barrier waits for this arrival)
    __syncwarp();
    if (lane < (EPI == 1 ? 4 / parts : 1)) bulk_load_1d(smem_u32(smem + kOffRaw + s * kQ4StageBytes) + dst, src + static_cast<size_t>(q) * kQ4StageBytes, size, full);
    __syncwarp();
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kMaxX; ++s) {
      mbar_init(smem_u32(&bar_x_full[s]), 1);
      mbar_init(smem_u32(&bar_done[s]), 1);
    }
    for (int s = 0; s < kMaxA; ++s) mbar_init(smem_u32(&bar_a_full[s]), 2 * 8);
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_acc_full[b]), 1);
      mbar_init(smem_u32(&bar_acc_empty[b]), 2 * 16);
    }
    for (int s = 0; s < 8; ++s) mbar_init(smem_u32(&bar_turn[s]), 4);
    mbar_init(smem_u32(bar_last), 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_x);
    if (!Q4) tma_prefetch_desc(&map_w);
  }
  __syncwarp();
  if (Q4 && warp == 3) {
    // The first packed stages are on their way while the rest is set up: this warp only announces their barriers to the others (who find them behind the
    // cluster barrier) and copies before it waits for anyone.
    if (lane == 0) {
      for (int s = 0; s < NR; ++s) {
        mbar_init(smem_u32(&bar_raw_full[s]), 1);
        mbar_init(smem_u32(&bar_raw_empty[s]), 8);
      }
      mbar_fence_init();
    }
    __syncwarp();
    cluster_arrive_relaxed();  // (orders nothing that thread 0 has stored: barrier 2 below does, for the abort flag)
    for (int i = 0; any && i < min(pc.k1 - pc.k0, NR); ++i) copy_stage(pc, pc.k0 + i, i, 0, 1);
    asm volatile("bar.sync 2, 64;" ::: "memory");
    cluster_wait();
    __syncwarp();
  } else {
    if (Q4 && warp == 0) asm volatile("bar.arrive 2, 64;" ::: "memory");  // the abort flag is clear, before warp 3 first looks at it
    if (warp == 2) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncwarp();
    if (Q4) asm volatile("bar.sync 1, 640;" ::: "memory");  // (the other twenty warps: the address of tensor memory)
    else __syncthreads();
    cluster_meet();  // the peer's barriers exist before anything arrives on them
    tc_fence_after();
  }
  pdl_trigger();  // (behind the set-up: the next kernel's blocks are not to come between the two CTAs of a pair and their tensor memory)
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_a = tmem_base + (NA == 2 ? kMaxTokens : 256);

  if (warp == 0 || warp == 2 || (!Q4 && warp == 3)) {
    // ---------------- token copies: one per stage and instruction; bf16 weight copies ----------------
    const int mine = warp == 3 ? 2 : warp >> 1;
    if (lane == 0 && (mine != 1 || two)) {
      int g = 0, s = 0;  // stages of this pair, numbered across pieces; ring position
      uint32_t ph = 0;
      bool ok = true;
      for (bool more = any; ok && more; more = walk.next(pc)) {
        const int row = mine == 0 ? pc.m0 + rank * (pc.n1 >> 1) : pc.m0 + pc.n1 + rank * (pc.n2 >> 1);
        const int half_tile = pc.n_tile * 2 + rank;
        const uint32_t bytes = static_cast<uint32_t>((pc.n2 > 0 ? 4 * region : 2 * region) + (Q4 ? 0 : 2 * kWStage));  // of both CTAs
        for (int q = pc.k0; q < pc.k1; ++q, ++g) {
          ok = g < NX || mbar_wait(smem_u32(&bar_done[s]), ph ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (rank == 0 && mine == 0) mbar_expect_tx(smem_u32(&bar_x_full[s]), bytes);  // (for all copies; the barrier waits for this arrival)
          const uint32_t at = smem_u32(smem + s * x_bytes), full = mapa_u32(smem_u32(&bar_x_full[s]), 0);
          if (mine == 2) {
            if (EPI == 1) tma_load_5d_pair(at, &map_w, full, 0, 0, 0, half_tile * 8, q);
            else tma_load_2d_pair(at, &map_w, full, q * 64, half_tile * 128);
          } else if (mine == 0 || pc.n2 > 0) {
            tma_load_3d_pair(at + (Q4 ? 0 : kWStage) + mine * region, &map_x, full, 0, row, Q4 ? 2 * q : q);
          }
          if (++s == NX) { s = 0; ph ^= 1; }
        }
      }
      // the pair's last commits have arrived here before this CTA may leave
      for (int j = g < NX ? g : NX; ok && j > 0; --j) ok = mbar_wait(smem_u32(&bar_done[(g - j) % NX]), ((g - j) / NX) & 1, abort_flag, p.status);
    }
  } else if (Q4 && (warp == 3 || warp == 20)) {
    // ---------------- packed weight copies: alternate stages, or (EPI 1) the gate and the up rows of every stage ----------------
    const int mine = warp == 3 ? 0 : 1, ahead = any ? min(pc.k1 - pc.k0, NR) : 0;
    int g = 0;
    bool ok = true;
    for (bool more = any; ok && more; more = walk.next(pc)) {
      for (int q = pc.k0; q < pc.k1; ++q, ++g) {
        if (g < ahead || (EPI != 1 && (g & 1) != mine)) continue;  // (the first ones are under way)
        const int s = g % NR;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_raw_empty[s]), ((g / NR) & 1) ^ 1, abort_flag, p.status));
        if (!ok) break;
        copy_stage(pc, q, s, EPI == 1 ? mine : 0, EPI == 1 ? 2 : 1);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer of the pair ----------------
    if (rank == 0) {
      constexpr int KS = Q4 ? 8 : 4;  // instructions of 16 k per stage
      const uint64_t desc_w = umma_desc_k_sw128(smem_u32(smem)), desc0 = umma_desc_k_sw128(smem_u32(smem + (Q4 ? 0 : kWStage)));
      const uint64_t half_stage = static_cast<uint64_t>(region >> 5), second = static_cast<uint64_t>(region >> 4);  // JQ4: 64 k; the second instruction's tokens
      const bool leader = elect_one();
      int it = 0, sx = 0, sa = 0;
      uint32_t phx = 0, pha = 0;
      bool ok = true, ready = false;  // ready: the next stage's operands have been seen complete
      for (bool more = any; ok && more; more = walk.next(pc), ++it) {
        const int b = NACC == 2 ? it & 1 : 0;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_empty[b]), ((NACC == 2 ? it >> 1 : it) & 1) ^ 1, abort_flag, p.status));
        if (!ok) break;
        const uint32_t idesc1 = umma_idesc_bf16(256, pc.n1), idesc2 = umma_idesc_bf16(256, pc.n2), acc1 = tmem_base + b * kOneMma, acc2 = acc1 + pc.n1;
        const bool both = pc.n2 > 0;
        const int steps = pc.k1 - pc.k0;
        for (int k = 0; k < steps; ++k) {
          if (!ready) {
            ok = mbar_wait(smem_u32(&bar_x_full[sx]), phx, abort_flag, p.status);
            ok = __all_sync(0xffffffffu, ok && (!Q4 || mbar_wait(smem_u32(&bar_a_full[sa]), pha, abort_flag, p.status)));
          }
          if (!ok) break;
          tc_fence_after();
          const uint64_t at = static_cast<uint64_t>((sx * x_bytes) >> 4), db = desc0 + at, dw = desc_w + at;
          const uint32_t ta = tmem_a + sa * 64;
          auto product = [&](int j, uint32_t add) {
            const uint64_t d = db + (j < 4 ? 0 : half_stage) + (j & 3) * 2;
            if (Q4) {
              umma_bf16_pair_ts(acc1, ta + j * 8, d, idesc1, add);
              if (both) umma_bf16_pair_ts(acc2, ta + j * 8, d + second, idesc2, add);
            } else {
              umma_bf16_pair(acc1, dw + j * 2, d, idesc1, add);
              if (both) umma_bf16_pair(acc2, dw + j * 2, d + second, idesc2, add);
            }
          };
          if (leader) {
#pragma unroll
            for (int j = 0; j < KS - 1; ++j) product(j, (k > 0 || j > 0) ? 1u : 0u);
          }
          const uint32_t done = smem_u32(&bar_done[sx]);
          if (++sx == NX) { sx = 0; phx ^= 1; }
          if (Q4 && ++sa == NA) { sa = 0; pha ^= 1; }
          // look at the next stage's operands while the pipe works on these
          ready = k + 1 < steps && __all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bar_x_full[sx]), phx) && (!Q4 || mbar_try_wait(smem_u32(&bar_a_full[sa]), pha)));
          if (leader) {
            product(KS - 1, 1u);
            umma_commit_pair(done);
          }
        }
        if (!ok) break;
        if (leader) umma_commit_pair(smem_u32(&bar_acc_full[b]));
      }
      if (!ok && leader) {
        umma_commit_pair(smem_u32(bar_last));
        const unsigned long long t0 = globaltimer_ns();
        while (!mbar_try_wait(smem_u32(bar_last), 0) && globaltimer_ns() - t0 < 20000000ull) {
        }
      }
      __syncwarp();
    }
  } else if (warp >= 4 && warp < 20) {
    // ---------------- packed stage -> bf16 operand in tensor memory; accumulators -> global memory ----------------
    // Groups of four warps, (warp - 4) / 4: groups 0 and 1 expand the halves of the even 128-k stages, 2 and 3 those of the odd ones.
    const int grp = (warp - 4) >> 2, h = grp & 1, q4 = warp & 3;  // group, half of the 128-k stage, quarter of the lanes of tensor memory
    // packed row of this lane: its own, or (EPI 1) eight gate rows and the up rows of the same outputs in turn
    const int r = EPI == 1 ? ((lane >> 3) & 1) * 64 + q4 * 16 + (lane >> 4) * 8 + (lane & 7) : q4 * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(q4 * 32) << 16;
    const uint32_t lane_a = tmem_a + lanes + h * 32;  // (JQ4)
    const uint32_t remote_full = mapa_u32(smem_u32(bar_a_full), 0);
    const uint8_t* raw0 = smem + kOffRaw + r * 64 + (((2 * h) ^ ((r >> 1) & 3)) << 4);
    const uint8_t* raw1 = smem + kOffRaw + r * 64 + (((2 * h + 1) ^ ((r >> 1) & 3)) << 4);
    const uint8_t* rawsc = smem + kOffRaw + 8192 + r * 16 + h * 8;
    int j = 0, it = 0, turn = 0;  // 128-k stages of this pair, numbered across pieces; pieces; drained sixteens of this group
    const bool turned = !p.out_f32 && p.vec == 8;
    bool ok = true;
    for (bool more = any; ok && more; more = walk.next(pc), ++it) {
      for (int q = pc.k0; Q4 && q < pc.k1; ++q, ++j) {
        if ((j & 1) != (grp >> 1)) continue;
        const int sr = j % NR, sa = j & (NA - 1);
        ok = mbar_wait(smem_u32(&bar_raw_full[sr]), (j / NR) & 1, abort_flag, p.status);
        const uint4 w[2] = {*reinterpret_cast<const uint4*>(raw0 + sr * kQ4StageBytes), *reinterpret_cast<const uint4*>(raw1 + sr * kQ4StageBytes)};
        const float2 sc = *reinterpret_cast<const float2*>(rawsc + sr * kQ4StageBytes);
        uint32_t o[32];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const __nv_bfloat162 s2 = __float2bfloat162_rn(b == 0 ? sc.x : sc.y);
          const uint32_t words[4] = {w[b].x, w[b].y, w[b].z, w[b].w};
#pragma unroll
          for (int hl = 0; hl < 2; ++hl) {
#pragma unroll
            for (int wd = 0; wd < 4; ++wd) {
              const uint32_t a = (words[wd] >> (4 * hl)) & 0x0F0F0F0Fu;
              o[b * 16 + hl * 8 + wd * 2 + 0] = q4_pair_to_bf162(a, 0x4140u, s2);
              o[b * 16 + hl * 8 + wd * 2 + 1] = q4_pair_to_bf162(a, 0x4342u, s2);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bar_raw_empty[sr]));
        // The slot is free once the stage that had it, NA before this one, has retired. Stages retire in order and this warp has seen the one two
        // before that, so its barrier is at most one phase behind. (Every lane polls for itself; the stores below are warp-wide, so the warp goes
        // on or leaves as a whole.)
        const int before = j - NA;
        ok = __all_sync(0xffffffffu, ok && (before < 0 || mbar_wait(smem_u32(&bar_done[before % NX]), (before / NX) & 1, abort_flag, p.status)));
        if (!ok) break;
        tc_fence_after();
        tmem_st_x16(lane_a + sa * 64, o);
        tmem_st_x16(lane_a + sa * 64 + 16, o + 16);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(remote_full + sa * 8);
      }
      // ---- drain: the warps of a quarter take every fourth sixteen columns ----
      const int b = NACC == 2 ? it & 1 : 0;
      ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&bar_acc_full[b]), (NACC == 2 ? it >> 1 : it) & 1, abort_flag, p.status));
      if (!ok) break;
      tc_fence_after();
      const int tokens = pc.m_lim - pc.m0, cols = pc.n1 + pc.n2;
      const uint32_t acc = tmem_base + b * kOneMma + lanes;
      if (EPI == 2 || pc.slot >= 0) {
        float* dst = p.sums + static_cast<size_t>(2 * pc.slot + rank) * p.bn * 128 + q4 * 32 + lane;
        for (int c0 = grp * 16; c0 < cols; c0 += 64) {
          uint32_t v[16];
          tmem_ld_x16(acc + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) dst[static_cast<size_t>(c0 + c) * 128] = __uint_as_float(v[c]);
        }
      } else if (EPI == 0 && !turned) {
        // fp32 outputs, or rows that do not take 8 bytes at once: straight from the lanes
        const int n = pc.n_tile * 256 + rank * 128 + q4 * 32 + lane;
        const bool live = n < p.N;
        const float add = p.bias != nullptr && live ? p.bias[n] : 0.f;
        const size_t at = static_cast<size_t>(pc.m0) * p.ldo + n;
        for (int c0 = grp * kDrain; c0 < cols; c0 += 4 * kDrain) {
          uint32_t v[16];
          tmem_ld_x16(acc + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            if (live && c0 + c < tokens) {
              const float f = __uint_as_float(v[c]) + add;
              if (p.out_f32) static_cast<float*>(p.out)[at + static_cast<size_t>(c0 + c) * p.ldo] = f;
              else static_cast<__nv_bfloat16*>(p.out)[at + static_cast<size_t>(c0 + c) * p.ldo] = f2bf(f);
            }
          }
        }
      } else if constexpr (EPI != 2) {
        // Sixteen tokens at a time through shared memory, so that a warp stores whole rows (2 bytes per lane, 64 per store, took 9,700 cycles for 352
        // tokens). A thread loads rows r, r + 8, r + 16, r + 24 of its quarter and two neighbouring tokens, the form that stmatrix turns.
        // Two buffers: a warp writes one again only behind the barrier of the other, which every warp of the group reaches after it has read this one.
        constexpr int kOut = EPI == 1 ? 64 : 128, kPitch = kOut * 2 + 16;
        const int n0 = (pc.n_tile * 2 + rank) * kOut, n_lim = EPI == 1 ? p.half : p.N;
        float add[4] = {0.f, 0.f, 0.f, 0.f};
        if (EPI == 0 && p.bias != nullptr) {
#pragma unroll
          for (int i = 0; i < 4; ++i) add[i] = n0 + q4 * 32 + i * 8 + (lane >> 2) < p.N ? p.bias[n0 + q4 * 32 + i * 8 + (lane >> 2)] : 0.f;
        }
        __nv_bfloat16* out = static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(pc.m0) * p.ldo + n0;
        // this lane's row of its matrix: token (lane >> 4) * 8 + lane % 8, and eight weight rows
        const int put = (((lane >> 4) & 1) * 8 + (lane & 7)) * kPitch + (EPI == 1 ? q4 * 16 : q4 * 32) * 2 + ((lane >> 3) & 1) * 16;
        const int per = EPI == 1 ? 8 : 16, get_c = q4 * 4 + lane / per, get_e = lane % per * 8;  // tokens it stores 16 bytes of, every 32 / per
        for (int c0 = grp * kDrain; c0 < cols; c0 += 4 * kDrain, ++turn) {
          uint8_t* buf = smem + kOffDrain + (grp * 2 + (turn & 1)) * kDrainBytes;
          float v[2][8];  // [sixteen rows][token c, c + 1 of rows r and r + 8; the same of tokens + 8]
          tmem_ld_16x256_x2(acc + c0, reinterpret_cast<uint32_t*>(v[0]));
          tmem_ld_16x256_x2(acc + (16u << 16) + c0, reinterpret_cast<uint32_t*>(v[1]));
          tmem_ld_wait();
          if constexpr (EPI == 0) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const float a = add[2 * i], b = add[2 * i + 1];
              stmatrix_x4_trans(smem_u32(buf + put) + i * 32, pack_bf162(v[i][0] + a, v[i][1] + a), pack_bf162(v[i][2] + b, v[i][3] + b),
                                pack_bf162(v[i][4] + a, v[i][5] + a), pack_bf162(v[i][6] + b, v[i][7] + b));
            }
          } else {
            // (columns without a token hold zeros)
            float f[2][4];
            if (p.act_kind == 2) {
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i >> 2][i & 3] = apply_act(2, v[i >> 2][(i & 2) * 2 + (i & 1)]) * v[i >> 2][(i & 2) * 2 + (i & 1) + 2];
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) f[i >> 2][i & 3] = apply_act(1, v[i >> 2][(i & 2) * 2 + (i & 1)]) * v[i >> 2][(i & 2) * 2 + (i & 1) + 2];
            }
            stmatrix_x4_trans(smem_u32(buf + put), pack_bf162(f[0][0], f[0][1]), pack_bf162(f[1][0], f[1][1]), pack_bf162(f[0][2], f[0][3]), pack_bf162(f[1][2], f[1][3]));
          }
          __syncwarp();
          uint64_t* bar = &bar_turn[grp * 2 + (turn & 1)];
          if (lane == 0) mbar_arrive(smem_u32(bar));
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), (turn >> 1) & 1, abort_flag, p.status));
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < (EPI == 1 ? 1 : 2); ++i) {
            const int c = get_c + i * 2;
            const uint4 pk = *reinterpret_cast<const uint4*>(buf + c * kPitch + get_e * 2);
            if (c0 + c >= tokens) continue;
            __nv_bfloat16* dst = out + static_cast<size_t>(c0 + c) * p.ldo + get_e;
            if (n0 + get_e + 7 < n_lim) {
              *reinterpret_cast<uint4*>(dst) = pk;
            } else {
              const __nv_bfloat16* one = reinterpret_cast<const __nv_bfloat16*>(&pk);
              for (int k = 0; k < 8 && n0 + get_e + k < n_lim; ++k) dst[k] = one[k];
            }
          }
        }
        if (!ok) break;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(mapa_u32(smem_u32(&bar_acc_empty[b]), 0));  // the accumulator has been read
    }
  }

  // ---------------- teardown ----------------
  __syncwarp();  // single lanes ran the copy loops
  if (*abort_flag) {
    // a wait ran out: copies that are still in flight get time to land before their shared memory goes away
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 20000000ull) {
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_meet();  // no CTA leaves while the pair's MMAs or arrivals may still touch its shared memory
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
  cluster_meet();  // the release of a pair's tensor memory involves both CTAs: neither leaves before both have asked for it
}

// Second kernel: adds up the sums of cut tiles in order of k and finishes them (EPI 2: of all tiles; a tile's norms and rotations are spread over the GPU here).
// One block per half tile and 8 tokens, two tokens of a warp and four parts at a time (one token's parts in turn left the kernel waiting for L2: 25 MB of
// sums 7 us). Bound by the sums, which it finds in L2.
template <int EPI>
__global__ void __launch_bounds__(128) gemm_parts_sum_kernel(const PartParams p) {
  pdl_trigger();
  const int whole = p.waves * p.pairs, rank = blockIdx.x & 1, lane = threadIdx.x & 31;
  const int t = static_cast<int>(blockIdx.x >> 1) + (EPI == 2 ? 0 : whole);
  const int n_tile = p.by_m.of(t), m0 = (t - n_tile * p.m_tiles) * p.bn;
  const int c0 = blockIdx.y * 8 + (threadIdx.x >> 5) * 2, live = min(2, min(p.M - m0, p.bn) - c0);
  if (live <= 0) return;
  const int first = t < whole ? (p.n_tiles * p.m_tiles - whole) * p.parts + t : (t - whole) * p.parts, count = t < whole ? 1 : p.parts;
  const Finish<EPI> finish(p, n_tile, rank, lane);
  typename Finish<EPI>::Token tok[2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (j < live) finish.fetch(m0 + c0 + j, tok[j]);
  pdl_wait();
  const size_t pitch = static_cast<size_t>(2) * p.bn * 128;
  const float* part = p.sums + (static_cast<size_t>(2 * first + rank) * p.bn + c0) * 128;
  float sum[2][4] = {};
  for (int i0 = 0; i0 < count; i0 += 4) {
    float s[4][2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (i0 + i < count && j < live) row_sums<EPI>(part + (i0 + i) * pitch + j * 128, lane, s[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[j][e] += i0 + i < count && j < live ? s[i][j][e] : 0.f;
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
    if (j < live) finish(m0 + c0 + j, sum[j], tok[j]);
}

// Pairs of SMs that can hold the kernel at one time on the current GPU, within the limit that is set (as in gemm_pair.cu); 0: none.
template <bool Q4, int EPI>
int part_pairs() {
  static int caps[64];  // per GPU; 0: not asked yet, -1: none
  int dev = 0;
  if (g_gemm_pairs == 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (caps[dev] == 0) {
    cudaError_t e = cudaFuncSetAttribute(gemm_parts_kernel<Q4, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    int n = 0;
    if (e == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmemBytes;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      e = cudaOccupancyMaxActiveClusters(&n, gemm_parts_kernel<Q4, EPI>, &cfg);
    }
    if (e != cudaSuccess) (void)cudaGetLastError();  // (this query's own error; nothing was launched)
    caps[dev] = e == cudaSuccess && n > 0 ? n : -1;
  }
  const int cap = caps[dev] < 0 ? 0 : caps[dev];
  return g_gemm_pairs > 0 && g_gemm_pairs < cap ? g_gemm_pairs : cap;
}
int part_pairs_of(bool q4, int epi) {
  if (q4) return epi == 1 ? part_pairs<true, 1>() : (epi == 2 ? part_pairs<true, 2>() : part_pairs<true, 0>());
  return epi == 1 ? part_pairs<false, 1>() : (epi == 2 ? part_pairs<false, 2>() : part_pairs<false, 0>());
}
int stages_of(const GemmWeightDesc* w) { return w->is_q4 ? (w->K + 127) / 128 : w->K / 64; }

int width_of(const void* out, int ldo, bool f32) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(out) * (f32 ? 1 : 2);
  return ldo % 8 == 0 && (at & 31) == 0 && !f32 ? 8 : (ldo % 4 == 0 && (at & 15) == 0 ? 4 : 1);
}
int tiles_of(int n, int epi) { return epi == 1 ? (n / 2 + 127) / 128 : (n + 255) / 256; }

struct PartPlan {
  int bn = 0, m_tiles = 0, n_tiles = 0, pairs = 0, waves = 0, parts = 0;
  double cost = 1e30;
};
// Token tiles, whole waves and parts; in thousands of cycles. A 128-k stage takes 8 instructions of cols / 2 cycles and no less than its expansion (bf16: a 64-k stage 4,
// and no less than HBM needs for 32 KB per pair; with these constants the estimate is within a tenth of what 130 products of 64 to 2048 rows took), a piece its
// drain and the first stage that the pipe waits for (an SM stores some 30 bytes per cycle); cut tiles cost the second kernel (four parts at a time) and their sums' way back from L2.
PartPlan plan_parts(const GemmWeightDesc* w, int M, int epi) {
  PartPlan best;
  const auto up = [](int a, int b) { return (a + b - 1) / b; };
  const int n_tiles = tiles_of(w->N, epi), kq = stages_of(w), cap = part_pairs_of(w->is_q4, epi);
  if (cap <= 0) return best;
  const int few = up(M, kMaxTokens);
  for (int want = few; want <= few + 1; ++want) {
    const int bn = (up(M, want) + 31) & ~31, m_tiles = up(M, bn), tiles = n_tiles * m_tiles;
    const double stage = w->is_q4 ? std::max(0.95, bn * 4e-3) : std::max(0.6, bn * 2.1e-3), part = 0.8 + bn * 17e-3, turn = epi == 0 ? 1.0 + bn * 11.5e-3 : part;
    const int waves = tiles / cap, cut = tiles - waves * cap;
    for (int f = cut > 0 ? 1 : 0; f <= (cut > 0 ? std::min(kq, cap / cut) : 0); ++f) {
      double cost = waves * (kq * stage + turn);
      if (f > 0) cost += up(kq, f) * stage + (f > 1 ? part : turn);
      const double again = static_cast<double>(f > 1 || epi == 2 ? cut * f : 0) + (epi == 2 ? waves * cap : 0);
      if (again > 0) cost += 3.5 + up(f, 4) + again * bn * 256 * 4 / (cap * 2 * 25e3);
      if (cost < best.cost - 1e-9) {
        best.bn = bn;
        best.m_tiles = m_tiles;
        best.n_tiles = n_tiles;
        best.pairs = waves > 0 ? cap : cut * f;
        best.waves = waves;
        best.parts = f;
        best.cost = cost;
      }
    }
  }
  return best;
}
int cut_tiles(const PartPlan& q) { return q.n_tiles * q.m_tiles - q.waves * q.pairs * (q.waves > 0); }

template <bool Q4, int EPI>
void launch_parts(const GemmWeightDesc* w, const void* x, int rows, int ldx, PartParams p, cudaStream_t st) {
  if ((static_cast<long long>(p.m_tiles) + 16) * p.n_tiles + p.pairs > 0x7fffffffll) throw std::runtime_error("pair gemm (cut tiles): more tiles than the walk can number");
  CUtensorMap map_x;
  p.box = (p.bn <= kOneMma ? p.bn : (((p.bn >> 1) + 31) & ~31)) / 2;
  encode_map_kchunks(&map_x, x, static_cast<uint64_t>(rows), static_cast<uint64_t>(w->K), static_cast<uint64_t>(ldx) * 2, p.box, Q4 ? 2 : 1);
  CUtensorMap map_w = Q4 ? map_x : w->map_w64;
  if (!Q4 && EPI == 1) encode_map_gate_up(&map_w, w->data, static_cast<uint64_t>(w->N / 2), static_cast<uint64_t>(w->K));
  p.wq = static_cast<const uint8_t*>(w->data);
  p.slots = Q4 ? (p.bn <= 256 ? 4 : 2) : (p.bn <= 256 ? 2 : 1);
  p.by_m.set(p.m_tiles);
  p.by_parts.set(p.parts);
  p.by_group.set(8 * p.n_tiles);
  p.x_stages = Q4 ? std::min(kMaxX, kXRoom / (p.box * 256 * (p.bn > kOneMma ? 2 : 1))) : std::min(kMaxX, kStageRoom / (kWStage + p.box * 128 * (p.bn > kOneMma ? 2 : 1)));
  if (part_pairs<Q4, EPI>() < p.pairs || p.pairs < 1) throw std::runtime_error("pair gemm (cut tiles): no pair of SMs can hold the kernel");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * p.pairs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_parts_kernel<Q4, EPI>, map_x, map_w, p);
  const int tiles = p.n_tiles * p.m_tiles, second = EPI == 2 ? tiles : (p.parts > 1 ? tiles - p.waves * p.pairs : 0);
  if (e == cudaSuccess && p.items == nullptr && second > 0) e = launch_pdl(gemm_parts_sum_kernel<EPI>, dim3(2 * second, (p.bn + 7) / 8), dim3(128), 0, st, p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("pair gemm (cut tiles) launch: ") + cudaGetErrorString(e));
}

PartParams dense_params(const GemmWeightDesc* w, int M, int epi, float* sums, int* status) {
  const PartPlan plan = plan_parts(w, M, epi);
  PartParams p = {};
  p.M = M;
  p.N = w->N;
  p.kq = stages_of(w);
  p.bn = plan.bn;
  p.n_tiles = plan.n_tiles;
  p.m_tiles = plan.m_tiles;
  p.pairs = plan.pairs;
  p.waves = plan.waves;
  p.parts = plan.parts;
  p.w_tiles = (w->N + 127) / 128;
  p.half = w->N / 2;
  p.sums = sums;
  p.status = status;
  return p;
}

}  // namespace

// Weights and outputs the kernel takes: k in whole chunks of 64, as the token copies fetch them. `n`: rows of the weight (of one expert). EPI 1: whole
// halves of 64 rows, so that gate and up rows begin on a half tile.
bool gemm_parts_supported(const GemmWeightDesc* w, int n, const void* out, int ldo, int epi) {
  if (w->K % 64 != 0 || w->K < 64 || n < 64 || part_pairs_of(w->is_q4, epi) <= 0) return false;
  if (epi == 1) return n % (w->is_q4 ? 128 : 16) == 0 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  if (epi == 2) return ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
  return true;
}

// Whether this kernel is the faster one for M rows of a dense weight; all times in microseconds, 1.62 thousand cycles of the plan are one. It starts in ordinary order,
// some two to four microseconds behind a one-tile kernel that starts under the kernel in front, and cut tiles take a second launch; so it has to earn that. The
// comparisons are by estimates of the kernel that would run instead, where measured shapes (0.8 M to 920 M weights, 40 to 2048 rows, us here against there) fall on either side:
// JQ4, plain and heads: above 128 rows (2560 x 9728, 128 rows 15.4 against 13.0, 333 rows 22.6 against 27.2; 6144 x 2560 with heads, 128 rows 13.7 against 13.8, 333 rows 22
// against 38). Plain with at least five tiles of weights: fewer are a chain of cut tiles here and a cluster each there (1024 x 1024, 129 rows 9.3 against 7.6; 896 x 4864 13.1
// against 10.8; 1152 x 896 8.5 against 8.7, 256 rows 8.7 against 10.4), and by the one-tile kernel's estimate (2048 x 5632, 160 rows 15.0 against 14.2, 320 rows 15.7 against
// 16.4; 2560 x 4096, 160 rows 13.9 against 13.4, 320 rows 14.9 against 16.5, 768 rows 21.6 against 20.2, 1024 rows 26.3 against 34.4). That estimate does not see
// how full the token tile of 256 is: up to 224 rows it is 2 % long and then 5 % short.
// JQ4, gated: above 128 rows (0.71 to 0.95 of the other two launches). Below by the estimate, with a fourteenth to spare: expansion bounds a pair's
// 256 weight rows at 0.59 per 128 k and two one-tile CTAs at 0.35 (28672 x 4096, 40 rows 42.4 against 30.9, 128 rows 42.9 against 38.3; 7552 x 8960, 128 rows 26.5 against 22.1;
// but 19456 x 2560, whose last wave there is nearly empty, 80 rows 23.8 against 27.1, 128 rows 24.7 against 30.5).
// JQ4 from 768 rows on also by the pair kernel's estimate (behind an expansion to bf16, its drain under the next tile), which must be a seventh longer: where they are closer than that,
// prompts of several thousand rows that pull the clock down by their power ran up to a tenth longer here (19456 x 2560, 1536 rows 119 us against 143, 2048 rows 154 against 174,
// 4096 rows 332 against 322; 2560 x 9728, 2048 rows 68 against 112).
// bf16, gated: above 128 rows against the pair kernel's 1.2 estimates and 8 us (its drain takes longer than the plain one; 28672 x 3584, 384 rows 69 against 86, 896 rows 137 against 149,
// but 1280 rows 187 against 179; 18944 x 1536, 1280 rows 61 against 76; 11264 x 2048, 384 rows 22.9 against 35.5), below by the one-tile estimate too (65 to 128 rows 0.70 to 1.04; 40
// to 64 rows mostly slower: 6144 x 1024, 48 rows 9.6 against 8.3, but 23040 x 2560 29.5 against 32.4).
// bf16, heads: every sum goes through the second kernel. Up to 128 rows wide weights of 10 M and more (6144 x 4096, 65 rows 18.1 against 21.5; 6144 x 2560, 128 rows 15.1 against 18.5;
// 1536 x 13184 20.3 against 18.0, 1536 x 1024 9.8 against 8.1), to 192 rows not those of 2.3 to 6 M (2816 x 1792, 129 rows 12.8 against 12.2; on either side of them 0.68 to
// 0.95), to 256 rows where the pair kernel is not the choice there (12288 x 12544, 160 rows 71 against 107, 256 rows 94 against 82), to 384 rows always (0.59 to 0.96), then by its estimate.
// bf16, plain: from 193 rows on, against the better of the others by their estimates (3584 x 14336, 384 rows 40 against 59, 1024 rows 93 against 78; 2560 x 2048, 256 rows
// 11.5 against 12.9; 1024 x 1024, 256 rows 9.4 against 8.7). Fewer rows: the one-tile kernel reads weights at some 4.3 TB/s with 65 to 128 rows and 5.8 with 33 to 64, this one at 5.7 and
// 6.2, which pays from some 36 M and 170 M weights on, where the estimate does not say otherwise (256000 x 3584, 128 rows 323 against 424; 28672 x 8192, 65 rows 89 against 110, 48 rows 90
// against 81).
bool gemm_parts_preferred(const GemmWeightDesc* w, int M, int epi) {
  if (M <= 32 || g_gemm_persist || g_gemm_force_bn != 0) return false;  // (the last two: another kernel or tile was asked for)
  const double weights = static_cast<double>(w->N) * w->K;
  if (w->is_q4 ? (epi != 1 && M <= 128) || (epi == 0 && w->N <= 1024) : (epi == 0 && M <= 192 && weights < (M > 64 ? 36e6 : 170e6))) return false;
  if (epi == 2 && M <= 64) return false;
  const PartPlan plan = plan_parts(w, M, epi);
  if (plan.pairs == 0) return false;
  const double pair = gemm_pair_estimate(w, M, w->N), here = (w->is_q4 ? 2.5 : 3.0) + plan.cost / 1.62;
  const auto one = [&] { return gemm_tc_estimate(w, M, epi == 1); };
  if (w->is_q4) {
    if (M >= 768 && here >= 0.86 * pair) return false;
    if (epi == 1) return M > 128 || here < 0.93 * one();
    return epi == 2 || here < (M <= 224 ? 0.98 : (M <= 512 ? 1.05 : 1.0)) * one();
  }
  if (epi == 1) return M < 2048 && here < 0.95 * (1.2 * pair + 8.0) && (M > 128 || here < one());
  if (epi == 2) {
    if (M <= 128) return w->N >= 3400 && weights >= 10e6;
    if (M <= 192 && weights > 2.3e6 && weights < 6e6) return false;
    return M <= 256 ? !gemm_pair_preferred(w, M, w->N, 0) : M <= kMaxTokens || here < 0.86 * pair;
  }
  return (M <= 192 || here < (gemm_pair_preferred(w, M, w->N, 0) ? 0.95 : 1.08) * pair) && here < (M <= 64 ? 0.92 : 1.0) * one();
}

// fp32 room for the sums that the second kernel finishes (0: none)
size_t gemm_parts_room(const GemmWeightDesc* w, int M, int epi) {
  const PartPlan plan = plan_parts(w, M, epi);
  const size_t cut = static_cast<size_t>(cut_tiles(plan)), slots = cut * plan.parts + (epi == 2 ? static_cast<size_t>(plan.waves) * plan.pairs : 0);
  return epi == 2 || plan.parts > 1 ? slots * 2 * plan.bn * 128 : 0;
}

void gemm_parts_run(const GemmWeightDesc* w, const void* x, int M, int ldx, void* out, int ldo, bool out_f32, const float* bias, float* sums, int* status,
                    cudaStream_t st) {
  PartParams p = dense_params(w, M, 0, sums, status);
  p.out = out;
  p.ldo = ldo;
  p.out_f32 = out_f32 ? 1 : 0;
  p.vec = width_of(out, ldo, out_f32);
  p.bias = bias;
  if (w->is_q4) launch_parts<true, 0>(w, x, M, ldx, p, st);
  else launch_parts<false, 0>(w, x, M, ldx, p, st);
}

void gemm_parts_run_act(const GemmWeightDesc* w, const void* x, int M, int ldx, void* out, int ldo, int act, float* sums, int* status, cudaStream_t st) {
  PartParams p = dense_params(w, M, 1, sums, status);
  p.out = out;
  p.ldo = ldo;
  p.act_kind = act;
  if (w->is_q4) launch_parts<true, 1>(w, x, M, ldx, p, st);
  else launch_parts<false, 1>(w, x, M, ldx, p, st);
}

void gemm_parts_run_qkv(const GemmWeightDesc* w, const void* x, int M, int ldx, void* q_out, int ldo, const float* bias, const GemmQkvArgs* a, float* sums,
                        int* status, cudaStream_t st) {
  PartParams p = dense_params(w, M, 2, sums, status);
  p.out = q_out;
  p.ldo = ldo;
  p.bias = bias;
  p.qkv = *a;
  if (w->is_q4) launch_parts<true, 2>(w, x, M, ldx, p, st);
  else launch_parts<false, 2>(w, x, M, ldx, p, st);
}

// Experts: work items of up to `item_rows` rows (384 at most); act 0: out [rows, n], otherwise act(gate) * up: out [rows, n / 2].
void gemm_parts_run_grouped(const GemmWeightDesc* w, int n_per_expert, const void* x, int rows, int ldx, void* out, int ldo, const int* items, int max_items,
                            int item_rows, int act, int* status, cudaStream_t st) {
  if (item_rows < 1 || item_rows > kMaxTokens) throw std::runtime_error("pair gemm (cut tiles): work items of 1 to 384 rows");
  PartParams p = {};
  p.M = rows;
  p.N = n_per_expert;
  p.kq = (w->K + 127) / 128;
  p.bn = (item_rows + 31) & ~31;
  p.n_tiles = tiles_of(n_per_expert, act ? 1 : 0);
  p.m_tiles = max_items;
  p.pairs = std::min(p.n_tiles * p.m_tiles, part_pairs_of(true, act ? 1 : 0));
  p.w_tiles = (n_per_expert + 127) / 128;
  p.half = n_per_expert / 2;
  p.out = out;
  p.ldo = ldo;
  p.vec = width_of(out, ldo, false);
  p.items = reinterpret_cast<const int4*>(items);
  p.act_kind = act;
  p.status = status;
  if (act == 0) launch_parts<true, 0>(w, x, rows, ldx, p, st);
  else launch_parts<true, 1>(w, x, rows, ldx, p, st);
}

}  // namespace dlv
