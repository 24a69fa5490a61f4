// Prefill-size GEMM  out[m, n] = sum_k X[m, k] * W[n, k]  on pairs of SMs (tcgen05 cta_group::2), persistent.
//
// What bounds it: the tensor pipe. The one-tile kernel (gemm_tc.cuh) keeps it 48 % active at these sizes, because a CTA's barrier set-up,
// first copies and accumulator drain are not covered by another tile's math, and 128 x 256 per CTA needs a stage of operands every 512
// cycles. Here a pair of CTAs computes 256 tokens x 256 weight rows with M = 256 instructions (128 cycles each, so one issuing thread
// keeps ahead of the pipe), each CTA loads half of either operand, two accumulators of 256 columns fill tensor memory, and four warps
// drain one of them while the other is being accumulated. Tokens are the M operand: a thread of the drain holds one token's consecutive
// outputs, so that heads, gate / up pairs and 16-byte stores need no exchange between threads.
//
// Roles per CTA: warp 0 copies tokens, warp 3 weights (JQ4: packed stages), warp 1 of the even CTA issues all MMAs of the pair, warp 2 owns
// tensor memory, warps 4-7 drain accumulators, warps 8-23 (JQ4 only) expand packed weights into the swizzled operand tile.
// A stage is 64 k: 16 KB of tokens and 16 KB of weights per CTA. JQ4 stages arrive as one 10 KB copy per 128 k; warps 8-11 expand its
// first half, 12-15 its second, with the same arithmetic as gemm_tc.cuh ((nibble - 8) * bf16 scale).
// Barriers: `full` (even CTA) counts both CTAs' copies and expanding warps, `empty`, `acc_full` are multicast commits, `acc_empty` (even
// CTA) counts both CTAs' drain warps. All waits are bounded as everywhere; after one runs out every role leaves and the CTAs meet at the end.
//
// Epilogues: 0 = store (+ bias); 1 = act(gate) * up: the even CTA loads 128 gate rows, the odd one the up rows of the same outputs, so plain
// row order needs no interleaving; 2 = q | k | v heads of 128: per-head RMSNorm, rotation, paged cache write.
// Grouped mode (experts): a work list of (expert, first row, end row) items of 256 rows takes the place of the token tiles.
//
// It starts in ordinary stream order, behind the whole of the kernel in front, so that no role waits for that kernel; the kernel behind it may be set
// up early.
//
// 8192 x 19456 x 2560 in bf16: 516 us (590 at the power cap), the one-tile kernel 917 to 1154, cuBLAS 520 to 670 in the same runs.
//
// The reference multiplies prompts token by token on the CPU (native/src/main/c/simd/vector_simd.c:595).
#include <stdexcept>
#include <string>

#include "gemm_api.h"
#include "gemm_tc.cuh"
#include "pair.cuh"

namespace dlv {

int g_gemm_pairs = -1;

void encode_map_2d(CUtensorMap* map, int dtype_code, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows,
                   uint32_t box_cols, int swizzle_code);

namespace {

constexpr int kTokens = 256, kWRows = 256;   // tile of a pair
constexpr int kOpBytes = 128 * 128;          // one CTA's half of one operand, 64 k
constexpr int kStageBytes = 2 * kOpBytes;
constexpr int kRawBytes = kQ4StageBytes;
constexpr int kDrainBytes = 4 * 4096;        // 32 rows x 128 bytes per drain warp

template <bool Q4>
struct PairSmem {
  static constexpr int kStages = Q4 ? 5 : 6;
  static constexpr int kRaw = Q4 ? 4 : 0;
  static constexpr int kOffRaw = kStages * kStageBytes;
  static constexpr int kOffDrain = kOffRaw + kRaw * kRawBytes;
  static constexpr int kOffCtrl = kOffDrain + kDrainBytes;
  static constexpr int kBytes = kOffCtrl + 1024 + 1024;  // barriers + alignment slack
  static constexpr int kThreads = Q4 ? 768 : 256;
  static_assert(kBytes <= 232448, "shared memory of an SM");
};

struct PairParams {
  int M, N, K;       // N: weight rows (per expert in grouped mode)
  int nk;            // 64-k steps; JQ4: two for every packed stage, also where K ends in the first half of the last one (the padding holds zero
                     // scales, the copies bring zero tokens), because a group that waits for a step must also be waited for in that step
  int kq;            // JQ4: 128-k stages of a tile row
  int n_tiles, m_tiles;
  int w_rows;        // weight rows of one expert in the stacked weight (dense) / 128-row tiles of one expert (JQ4)
  int half;          // EPI 1: outputs per row (gate rows); the up rows follow them
  void* out;
  int ldo;
  const float* bias;
  const int4* items;
  int* status;
  int act_kind;
  GemmQkvArgs qkv;
};

// Packed JQ4 weight -> bf16 [N, K] in global memory, in front of a product whose rows pay for it. One block per 128 x 128 stage; 16 lanes
// write a row's 256 bytes. Bound by the 2.6 bytes per weight that it moves, most of which the product finds in L2 again.
__global__ void __launch_bounds__(256) q4_expand_kernel(const uint8_t* __restrict__ wq, __nv_bfloat16* __restrict__ out, int N, int K, int kq) {
  const int tile = blockIdx.x / kq, kb = blockIdx.x - tile * kq;
  const uint8_t* stage = wq + static_cast<size_t>(blockIdx.x) * kQ4StageBytes;
  const int c = threadIdx.x & 15, b = c >> 2, cc = c & 3;  // 8 elements: chunk cc of block b
  uint2 w[8];
  float sc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 16 + (threadIdx.x >> 4);
    w[i] = __ldg(reinterpret_cast<const uint2*>(stage + r * 64 + ((b ^ ((r >> 1) & 3)) << 4) + (cc & 1) * 8));
    sc[i] = __ldg(reinterpret_cast<const float*>(stage + 8192 + r * 16 + b * 4));
  }
  pdl_wait();  // the buffer may still be read by a product in front
  const int k = kb * 128 + c * 8;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int n = tile * 128 + i * 16 + (threadIdx.x >> 4);
    const __nv_bfloat162 s2 = __float2bfloat162_rn(sc[i]);
    const uint32_t lo = (w[i].x >> (cc >= 2 ? 4 : 0)) & 0x0F0F0F0Fu, hi = (w[i].y >> (cc >= 2 ? 4 : 0)) & 0x0F0F0F0Fu;
    if (n < N && k < K)
      *reinterpret_cast<uint4*>(out + static_cast<size_t>(n) * K + k) = make_uint4(q4_pair_to_bf162(lo, 0x4140u, s2), q4_pair_to_bf162(lo, 0x4342u, s2),
                                                                                    q4_pair_to_bf162(hi, 0x4140u, s2), q4_pair_to_bf162(hi, 0x4342u, s2));
  }
}

struct Tile {
  int m0, m_lim, n_tile, expert;  // m0 < 0: nothing to do
};

template <bool Q4, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairSmem<Q4>::kThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const PairParams p) {
  using L = PairSmem<Q4>;
  constexpr int NS = L::kStages, NR = L::kRaw > 0 ? L::kRaw : 1;
  extern __shared__ uint8_t gp_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(smem + L::kOffCtrl);
  uint64_t* bar_empty = bar_full + NS;
  uint64_t* bar_raw_full = bar_empty + NS;
  uint64_t* bar_raw_empty = bar_raw_full + NR;
  uint64_t* bar_acc_full = bar_raw_empty + NR;  // [2]
  uint64_t* bar_acc_empty = bar_acc_full + 2;   // [2]
  uint64_t* bar_last = bar_acc_empty + 2;       // abort path: MMAs in flight have retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_last + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = __shfl_sync(0xffffffffu, static_cast<int>(cluster_ctarank()), 0);
  const int pair = static_cast<int>(blockIdx.x) >> 1, pairs = static_cast<int>(gridDim.x) >> 1;
  const int total = p.n_tiles * p.m_tiles;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(smem_u32(&bar_full[s]), Q4 ? 1 + 2 * 4 : 2);  // token copies, then weight copies or the four expanding warps of each CTA
      mbar_init(smem_u32(&bar_empty[s]), 1);
    }
    for (int s = 0; s < NR; ++s) {
      mbar_init(smem_u32(&bar_raw_full[s]), 1);
      mbar_init(smem_u32(&bar_raw_empty[s]), 8);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&bar_acc_full[b]), 1);
      mbar_init(smem_u32(&bar_acc_empty[b]), 8);
    }
    mbar_init(smem_u32(bar_last), 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
  }
  __syncwarp();
  if (warp == 2) tmem_alloc_pair(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  cluster_meet();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  pdl_trigger();  // (behind the set-up: the next kernel's blocks are not to come between the two CTAs of a pair and their tensor memory)
  const uint32_t tmem_base = *tmem_slot;

  // Tiles of a pair: pair, pair + pairs, ... in an order that keeps what runs at one time within eight token tiles (work items) and a
  // few weight tiles: both are then read from L2 by several pairs.
  auto tile_of = [&](int t) -> Tile {
    constexpr int G = 8;
    const int per = G * p.n_tiles, g = t / per, r = t - g * per;
    const int rows = min(G, p.m_tiles - g * G);
    const int n = r / rows, m = g * G + (r - n * rows);
    Tile o;
    o.n_tile = n;
    o.expert = 0;
    if (p.items != nullptr) {
      const int4 it = p.items[m];
      o.expert = it.x;
      o.m0 = it.x < 0 ? -1 : it.y;
      o.m_lim = min(it.z, it.y + kTokens);
    } else {
      o.m0 = m * kTokens;
      o.m_lim = p.M;
    }
    return o;
  };

  if (warp == 0) {
    // ---------------- token copies ----------------
    if (lane == 0) {
      int g = 0;   // 64-k steps of this pair, numbered across tiles
      bool ok = true;
      for (int t = pair; t < total && ok; t += pairs) {
        const Tile tl = tile_of(t);
        if (tl.m0 < 0) continue;
        for (int k = 0; k < p.nk; ++k, ++g) {
          const int s = g % NS;
          ok = mbar_wait(smem_u32(&bar_empty[s]), ((g / NS) & 1) ^ 1, abort_flag, p.status);
          if (!ok) break;
          if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2 * kOpBytes);
          tma_load_2d_pair(smem_u32(smem + s * kStageBytes), &map_x, mapa_u32(smem_u32(&bar_full[s]), 0), k * 64, tl.m0 + rank * 128);
        }
      }
      // the pair's last commits have arrived here before this CTA may leave
      for (int j = g < NS ? g : NS; ok && j > 0; --j) ok = mbar_wait(smem_u32(&bar_empty[(g - j) % NS]), ((g - j) / NS) & 1, abort_flag, p.status);
    }
  } else if (warp == 3) {
    // ---------------- weight copies ----------------
    if (lane == 0) {
      int g = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += pairs) {
        const Tile tl = tile_of(t);
        if (tl.m0 < 0) continue;
        // first weight row of this CTA's half: half of the tile's rows, or (EPI 1) the up rows of the same outputs
        const int row = EPI == 1 ? tl.n_tile * 128 + rank * p.half : tl.n_tile * kWRows + rank * 128;
        if (Q4) {
          const int wt = tl.expert * p.w_rows + (row >> 7);
          for (int j = 0; j < p.kq; ++j, ++g) {
            const int s = g % NR;
            ok = mbar_wait(smem_u32(&bar_raw_empty[s]), ((g / NR) & 1) ^ 1, abort_flag, p.status);
            if (!ok) break;
            mbar_expect_tx(smem_u32(&bar_raw_full[s]), kRawBytes);
            tma_load_2d(smem_u32(smem + L::kOffRaw + s * kRawBytes), &map_w, smem_u32(&bar_raw_full[s]), 0, (wt * p.kq + j) * 10);
          }
        } else {
          for (int k = 0; k < p.nk; ++k, ++g) {
            const int s = g % NS;
            ok = mbar_wait(smem_u32(&bar_empty[s]), ((g / NS) & 1) ^ 1, abort_flag, p.status);
            if (!ok) break;
            if (rank == 0) mbar_expect_tx(smem_u32(&bar_full[s]), 2 * kOpBytes);
            tma_load_2d_pair(smem_u32(smem + s * kStageBytes + kOpBytes), &map_w, mapa_u32(smem_u32(&bar_full[s]), 0), k * 64, tl.expert * p.w_rows + row);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer of the pair ----------------
    if (rank == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(kTokens, kWRows);
      const uint64_t desc0 = umma_desc_k_sw128(smem_u32(smem));
      const bool leader = elect_one();
      int it = 0, s = 0;
      uint32_t ph = 0;
      bool ok = true, ready = false;  // ready: the next step's operands have been seen complete
      for (int t = pair; t < total && ok; t += pairs) {
        const Tile tl = tile_of(t);
        if (tl.m0 < 0) continue;
        const int b = it & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_empty[b]), ((it >> 1) & 1) ^ 1, abort_flag, p.status));
        if (!ok) break;
        const uint32_t acc = tmem_base + b * kWRows;
        for (int k = 0; k < p.nk; ++k) {
          if (!ready) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_full[s]), ph, abort_flag, p.status));
          if (!ok) break;
          tc_fence_after();
          const uint64_t da = desc0 + static_cast<uint64_t>((s * kStageBytes) >> 4), db = da + (kOpBytes >> 4);
          if (leader) {
#pragma unroll
            for (int j = 0; j < 3; ++j) umma_bf16_pair(acc, da + j * 2, db + j * 2, idesc, (k > 0 || j > 0) ? 1u : 0u);
          }
          const uint32_t bar_done = smem_u32(&bar_empty[s]);
          if (++s == NS) { s = 0; ph ^= 1; }
          // look at the next step's operands while the pipe works on these
          ready = k + 1 < p.nk && __all_sync(0xffffffffu, mbar_try_wait(smem_u32(&bar_full[s]), ph));
          if (leader) {
            umma_bf16_pair(acc, da + 6, db + 6, idesc, 1u);
            umma_commit_pair(bar_done);
          }
        }
        if (!ok) break;
        if (leader) umma_commit_pair(smem_u32(&bar_acc_full[b]));
        ++it;
      }
      if (!ok && leader) {
        umma_commit_pair(smem_u32(bar_last));
        const unsigned long long t0 = globaltimer_ns();
        while (!mbar_try_wait(smem_u32(bar_last), 0) && globaltimer_ns() - t0 < 20000000ull) {
        }
      }
      __syncwarp();
    }
  } else if (warp >= 8) {
    // ---------------- JQ4: packed stage -> bf16 operand tile ----------------
    if constexpr (Q4) {
      const int grp = (warp - 8) >> 2, h = grp & 1, r = threadIdx.x & 127;  // group, half of the 128-k stage, weight row
      int j = 0;   // 128-k stages of this pair, numbered across tiles
      int g0 = 0;  // 64-k step of the tile's first stage
      bool ok = true;
      for (int t = pair; t < total && ok; t += pairs) {
        const Tile tl = tile_of(t);
        if (tl.m0 < 0) continue;
        for (int q = 0; q < p.kq; ++q, ++j) {
          if ((j & 1) != (grp >> 1)) continue;
          const int sr = j % NR;
          ok = mbar_wait(smem_u32(&bar_raw_full[sr]), (j / NR) & 1, abort_flag, p.status);
          const uint8_t* raw = smem + L::kOffRaw + sr * kRawBytes;
          uint4 w[2];
          float sc[2];
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            w[b] = *reinterpret_cast<const uint4*>(raw + r * 64 + (((2 * h + b) ^ ((r >> 1) & 3)) << 4));
            sc[b] = *reinterpret_cast<const float*>(raw + 8192 + r * 16 + (2 * h + b) * 4);
          }
          // the values are formed before the operand stage is free, so that only stores stand between the pipe's release and its refill
          uint4 o[8];  // chunk 4 b + c: elements 8 c .. of block b (bytes 8 (c & 1) .., low nibbles for c < 2, then high ones)
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const __nv_bfloat162 s2 = __float2bfloat162_rn(sc[b]);
            const uint32_t words[4] = {w[b].x, w[b].y, w[b].z, w[b].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint32_t lo = (words[(c & 1) * 2] >> (c >= 2 ? 4 : 0)) & 0x0F0F0F0Fu, hi = (words[(c & 1) * 2 + 1] >> (c >= 2 ? 4 : 0)) & 0x0F0F0F0Fu;
              o[b * 4 + c] = make_uint4(q4_pair_to_bf162(lo, 0x4140u, s2), q4_pair_to_bf162(lo, 0x4342u, s2), q4_pair_to_bf162(hi, 0x4140u, s2),
                                        q4_pair_to_bf162(hi, 0x4342u, s2));
            }
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bar_raw_empty[sr]));
          const int g = g0 + 2 * q + h, s = g % NS;
          ok = __all_sync(0xffffffffu, ok && mbar_wait(smem_u32(&bar_empty[s]), ((g / NS) & 1) ^ 1, abort_flag, p.status));  // (the warp stays whole)
          if (!ok) break;
          uint8_t* dst = smem + s * kStageBytes + kOpBytes + r * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(dst + ((c ^ (r & 7)) << 4)) = o[c];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(mapa_u32(smem_u32(&bar_full[s]), 0));
        }
        g0 += p.nk;
      }
    }
  } else if (warp >= 4) {
    // ---------------- drain: accumulator -> global memory ----------------
    const int q = warp & 3;
    uint8_t* buf = smem + L::kOffDrain + q * 4096;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const int m_in = rank * 128 + q * 32 + lane;
    int it = 0;
    // chunk `c` (8 outputs) of this lane's row, in a layout whose 16-byte accesses hit all banks by rows and by chunks
    auto put = [&](int c, const float* v) {
      uint4 o;
      o.x = pack_bf162(v[0], v[1]);
      o.y = pack_bf162(v[2], v[3]);
      o.z = pack_bf162(v[4], v[5]);
      o.w = pack_bf162(v[6], v[7]);
      *reinterpret_cast<uint4*>(buf + lane * 128 + ((c ^ (lane & 7)) << 4)) = o;
    };
    // the eight chunks of 32 rows: 8 lanes per row; chunk c of a row goes to `row` + off(c) when off(c) >= 0 (elements)
    auto flush = [&](__nv_bfloat16* row, auto off) {
      __syncwarp();
      const int c = lane & 7, o = off(c);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int rr = i * 4 + (lane >> 3);
        const uint4 v = *reinterpret_cast<const uint4*>(buf + rr * 128 + ((c ^ (rr & 7)) << 4));
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(row), rr));
        if (dst != nullptr && o >= 0) *reinterpret_cast<uint4*>(dst + o) = v;
      }
      __syncwarp();
    };
    for (int t = pair; t < total; t += pairs) {
      const Tile tl = tile_of(t);
      if (tl.m0 < 0) continue;
      const int b = it & 1;
      // warp-uniform: the body holds warp-collective tensor-memory loads
      const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bar_acc_full[b]), (it >> 1) & 1, abort_flag, p.status));
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = lane_base + b * kWRows;
      const int m = tl.m0 + m_in;
      const bool live = m < tl.m_lim;
      auto release = [&] {  // the accumulator has been read
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(mapa_u32(smem_u32(&bar_acc_empty[b]), 0));
      };
      if constexpr (EPI == 0) {
        __nv_bfloat16* row = live ? static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo : nullptr;
#pragma unroll 1
        for (int c0 = 0; c0 < kWRows; c0 += 64) {
          const int n0 = tl.n_tile * kWRows + c0;
#pragma unroll 1
          for (int sub = 0; sub < 2; ++sub) {
            uint32_t v[32];
            tmem_ld_x16(acc + c0 + sub * 32, v);
            tmem_ld_x16(acc + c0 + sub * 32 + 16, v + 16);
            tmem_ld_wait();
            if (c0 + 64 == kWRows && sub == 1) release();
            float* f = reinterpret_cast<float*>(v);
            if (p.bias != nullptr) {
#pragma unroll
              for (int j = 0; j < 32; ++j) f[j] += n0 + sub * 32 + j < p.N ? __ldg(p.bias + n0 + sub * 32 + j) : 0.f;
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) put(sub * 4 + c, f + c * 8);
          }
          flush(row, [&](int c) { return n0 + c * 8 < p.N ? n0 + c * 8 : -1; });
        }
      } else if constexpr (EPI == 1) {
        __nv_bfloat16* row = live ? static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo : nullptr;
#pragma unroll 1
        for (int c0 = 0; c0 < 128; c0 += 64) {
#pragma unroll 1
          for (int sub = 0; sub < 4; ++sub) {
            uint32_t gv[16], uv[16];
            tmem_ld_x16(acc + c0 + sub * 16, gv);
            tmem_ld_x16(acc + 128 + c0 + sub * 16, uv);
            tmem_ld_wait();
            if (c0 == 64 && sub == 3) release();
            float* gf = reinterpret_cast<float*>(gv);
            const float* uf = reinterpret_cast<const float*>(uv);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              // (rows behind the last one hold zeros; a division of zero leaves the straight path for a call, for all 32 rows of the warp: 300 rows
              // of 11264 x 2048 took 69 us where 512 take 40)
              const float x = live ? gf[j] : 1.f;
              const float a = p.act_kind == 2 ? 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x))) : x / (1.f + __expf(-x));
              gf[j] = a * uf[j];
            }
            put(sub * 2, gf);
            put(sub * 2 + 1, gf + 8);
          }
          const int n0 = tl.n_tile * 128 + c0;
          flush(row, [&](int c) { return n0 + c * 8 < p.half ? n0 + c * 8 : -1; });
        }
      } else {
        const GemmQkvArgs& a = p.qkv;
        int pos = 0;
        long long slot = -1;
        if (live) {
          pos = a.positions[m];
          pos = pos < 0 ? 0 : (pos >= a.max_pos ? a.max_pos - 1 : pos);
          slot = a.slots != nullptr ? a.slots[m] : -1;
        }
        __syncwarp();
        const size_t cache_row = slot >= 0 ? static_cast<size_t>(slot / a.block_size) * a.kv_heads * a.block_size + static_cast<size_t>(slot % a.block_size) : 0;
#pragma unroll 1
        for (int hh = 0; hh < 2; ++hh) {
          const int head = tl.n_tile * 2 + hh;
          if (head >= a.heads + 2 * a.kv_heads) break;  // (uniform; the drain below still releases the accumulator)
          const bool is_q = head < a.heads, is_k = !is_q && head < a.heads + a.kv_heads;
          const __nv_bfloat16* nw = static_cast<const __nv_bfloat16*>(is_q ? a.q_norm_w : (is_k ? a.k_norm_w : nullptr));
          const bool rotate = (is_q || is_k) && a.cos_t != nullptr;
          const uint32_t hacc = acc + hh * 128;
          const float* bias = p.bias != nullptr ? p.bias + head * 128 : nullptr;
          float inv = 1.f;
          if (nw != nullptr) {
            float ss = 0.f;
#pragma unroll 1
            for (int c0 = 0; c0 < 128; c0 += 32) {
              uint32_t v[32];
              tmem_ld_x16(hacc + c0, v);
              tmem_ld_x16(hacc + c0 + 16, v + 16);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                const float x = __uint_as_float(v[j]) + (bias != nullptr ? __ldg(bias + c0 + j) : 0.f);
                ss += x * x;
              }
            }
            inv = rsqrtf(ss * (1.f / 128.f) + a.eps);
          }
          __nv_bfloat16* row = nullptr;
          if (is_q) {
            if (live) row = static_cast<__nv_bfloat16*>(p.out) + static_cast<size_t>(m) * p.ldo + head * 128;
          } else if (slot >= 0) {
            const int kvh = is_k ? head - a.heads : head - a.heads - a.kv_heads;
            row = static_cast<__nv_bfloat16*>(is_k ? a.k_cache : a.v_cache) + (cache_row + static_cast<size_t>(kvh) * a.block_size) * 128;
          }
          const float* cs = a.cos_t != nullptr ? a.cos_t + static_cast<size_t>(pos) * 64 : nullptr;
          const float* sn = a.cos_t != nullptr ? a.sin_t + static_cast<size_t>(pos) * 64 : nullptr;
#pragma unroll 1
          for (int d0 = 0; d0 < 64; d0 += 32) {  // dims d0 .. + 31 and their partners 64 above
#pragma unroll 1
            for (int sub = 0; sub < 2; ++sub) {
              const int d = d0 + sub * 16;
              uint32_t lo[16], hi[16];
              tmem_ld_x16(hacc + d, lo);
              tmem_ld_x16(hacc + 64 + d, hi);
              tmem_ld_wait();
              float* x = reinterpret_cast<float*>(lo);
              float* y = reinterpret_cast<float*>(hi);
              if (bias != nullptr) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  x[j] += __ldg(bias + d + j);
                  y[j] += __ldg(bias + 64 + d + j);
                }
              }
              if (nw != nullptr) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {  // rounded like a separate norm kernel would
                  x[j] = bf2f(f2bf(x[j] * inv * (bf2f(nw[d + j]) + a.norm_offset)));
                  y[j] = bf2f(f2bf(y[j] * inv * (bf2f(nw[64 + d + j]) + a.norm_offset)));
                }
              }
              if (rotate) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                  const float4 c4 = __ldg(reinterpret_cast<const float4*>(cs + d + j)), s4 = __ldg(reinterpret_cast<const float4*>(sn + d + j));
                  const float c[4] = {c4.x, c4.y, c4.z, c4.w}, s[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const float u = x[j + e], v = y[j + e];
                    x[j + e] = u * c[e] - v * s[e];
                    y[j + e] = v * c[e] + u * s[e];
                  }
                }
              }
              put(sub * 2, x);
              put(sub * 2 + 1, x + 8);
              put(4 + sub * 2, y);
              put(4 + sub * 2 + 1, y + 8);
            }
            flush(row, [&](int c) { return (c < 4 ? d0 + c * 8 : 64 + d0 + (c - 4) * 8); });
          }
        }
        release();
      }
      ++it;
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

// Pairs of SMs that can hold the kernel at one time on the current GPU, within the limit that is set; 0: none (a GPU or a share of one on
// which no cluster of this size fits), so that products take the one-tile kernel.
template <bool Q4, int EPI>
int pair_capacity() {
  static int caps[64];  // per GPU; 0: not asked yet, -1: none
  int dev = 0;
  if (g_gemm_pairs == 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (caps[dev] == 0) {
    using L = PairSmem<Q4>;
    cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<Q4, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes);
    int n = 0;
    if (e == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2);
      cfg.blockDim = dim3(L::kThreads);
      cfg.dynamicSmemBytes = L::kBytes;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      e = cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<Q4, EPI>, &cfg);
    }
    if (e != cudaSuccess) (void)cudaGetLastError();  // (this query's own error; nothing was launched)
    caps[dev] = e == cudaSuccess && n > 0 ? n : -1;
  }
  const int cap = caps[dev] < 0 ? 0 : caps[dev];
  return g_gemm_pairs > 0 && g_gemm_pairs < cap ? g_gemm_pairs : cap;
}

int pair_capacity_of(bool q4, int epi) {
  if (q4) return epi == 1 ? pair_capacity<true, 1>() : pair_capacity<true, 0>();
  return epi == 2 ? pair_capacity<false, 2>() : (epi == 1 ? pair_capacity<false, 1>() : pair_capacity<false, 0>());
}

// `expanded`: bf16 [N, K] room for a JQ4 weight that is expanded in front of the product (nullptr: expanded inside the kernel, stage by stage)
template <bool Q4, int EPI>
void launch_pair(const GemmWeightDesc* w, const void* x, int ldx, int rows, PairParams p, void* expanded, cudaStream_t st) {
  const int cap = pair_capacity<Q4, EPI>();
  if (cap <= 0) throw std::runtime_error("pair gemm: no pair of SMs can hold the kernel");
  CUtensorMap map_x, map_w;
  if (expanded != nullptr) {
    const int kq = (w->K + 127) / 128, stages = ((w->N + 127) / 128) * kq;
    cudaError_t e = launch_pdl(q4_expand_kernel, dim3(stages), dim3(256), 0, st, static_cast<const uint8_t*>(w->data), static_cast<__nv_bfloat16*>(expanded), w->N,
                               w->K, kq);
    if (e != cudaSuccess) throw std::runtime_error(std::string("JQ4 expansion launch: ") + cudaGetErrorString(e));
    encode_map_2d(&map_w, 0, expanded, w->N, w->K, static_cast<uint64_t>(w->K) * 2, 128, 64, 128);
  } else {
    map_w = Q4 ? w->map_w : w->map_w64;
  }
  encode_map_2d(&map_x, 0, x, static_cast<uint64_t>(rows), static_cast<uint64_t>(w->K), static_cast<uint64_t>(ldx) * 2, 128, 64, 128);
  p.K = w->K;
  p.kq = (w->K + 127) / 128;
  p.nk = Q4 ? 2 * p.kq : (w->K + 63) / 64;
  const int total = p.n_tiles * p.m_tiles;
  const int pairs = total < cap ? total : cap;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs);
  cfg.blockDim = dim3(PairSmem<Q4>::kThreads);
  cfg.dynamicSmemBytes = PairSmem<Q4>::kBytes;
  cfg.stream = st;
  // In ordinary stream order: pairs of CTAs that started under the kernel in front did not always come to an end (and a prompt-size product has
  // little to gain from its first microseconds).
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_pair_kernel<Q4, EPI>, map_w, map_x, p);
  if (e != cudaSuccess) throw std::runtime_error(std::string("pair gemm launch: ") + cudaGetErrorString(e));
}

}  // namespace

// Shapes the pair kernel takes: 16-byte output chunks, a weight of at least one tile; and a GPU that can hold a pair of it.
// `grouped`: JQ4 weights are expanded inside the kernel. `epi`: its epilogue.
bool gemm_pair_supported(const GemmWeightDesc* w, int n, const void* out, int ldo, bool grouped, int epi) {
  return n % 8 == 0 && n >= 256 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && w->K >= 64 &&
         pair_capacity_of(grouped && w->is_q4, epi) > 0;
}

// Whether the pair kernel is faster than the one-tile kernel (gemm_tc.cuh) for M rows of this weight. Both times in microseconds, by whole
// waves of tiles: a 64-k step takes 0.29 us of a 256 x 256 tile here, 0.5 us (JQ4: 0.42) of a 128 x 256 tile there, which can split k over
// up to eight CTAs where tiles are few (333 rows of 2560 x 9728: 31 us against 45). Expanding a JQ4 weight first writes 2 bytes per weight
// that push others out of L2: 36 us for 19456 x 2560. `merged`: outputs per row that the epilogue saves a later kernel from reading and writing.
// So bf16 weights come here from 192 (the gated one), 257 or 769 rows on. For 4-bit weights gemm_parts_preferred asks first and leaves prompts of a few thousand
// rows and more to this kernel.
static double waves(long long tiles, long long room) { return static_cast<double>((tiles + room - 1) / room); }
double gemm_pair_estimate(const GemmWeightDesc* w, int M, int n) {
  const double nk = (w->K + 63) / 64;
  return 5.0 + waves(static_cast<long long>((M + kTokens - 1) / kTokens) * ((n + 255) / 256), gemm_num_sms() / 2) * (nk * 0.29 + 1.0) +
         (w->is_q4 ? 2.0 + static_cast<double>(w->N) * w->K * 2.6 / 3.5e6 : 0.0);
}
bool gemm_pair_preferred(const GemmWeightDesc* w, int M, int n, int merged) {
  if (M < 192 || n < kWRows || g_gemm_persist || g_gemm_force_bn != 0) return false;  // (the last two: another kernel or tile was asked for)
  const double nk = (w->K + 63) / 64, pair = gemm_pair_estimate(w, M, n);
  const int m_tiles = (M + kTokens - 1) / kTokens, sms = gemm_num_sms();
  double one = 1e30;
  const long long tiles = static_cast<long long>((n + 127) / 128) * m_tiles;
  for (int s = 1; s <= 8 && (s == 1 || nk / s >= 4); ++s) {
    const double c = waves(tiles, sms / s) * (nk / s * (w->is_q4 ? 0.42 : 0.5) + 3.0 + (s > 1 ? 3.0 : 0.0));
    one = c < one ? c : one;
  }
  return pair < one + static_cast<double>(M) * merged * 2.0 / 5.5e6 + (merged > 0 ? 3.0 : 0.0);
}

// bytes of bf16 room that a product with this weight wants for `expanded` (0: none)
size_t gemm_pair_expanded_bytes(const GemmWeightDesc* w) { return w->is_q4 ? static_cast<size_t>(w->N) * w->K * 2 : 0; }

void gemm_pair_run(const GemmWeightDesc* w, const void* x, int M, int ldx, void* out, int ldo, const float* bias, void* expanded, int* status, cudaStream_t st) {
  PairParams p = {};
  p.M = M;
  p.N = w->N;
  p.n_tiles = (w->N + 255) / 256;
  p.m_tiles = (M + kTokens - 1) / kTokens;
  p.out = out;
  p.ldo = ldo;
  p.bias = bias;
  p.status = status;
  launch_pair<false, 0>(w, x, ldx, M, p, expanded, st);
}

// gate rows [0, N / 2) and up rows [N / 2, N) in plain order; out [M, N / 2]. JQ4 experts: whole weight tiles of either (N / 2 % 128 == 0).
bool gemm_pair_act_supported(const GemmWeightDesc* w, int n, const void* out, int ldo, bool grouped) {
  return n % 16 == 0 && (!w->is_q4 || n % 256 == 0) && gemm_pair_supported(w, n / 2, out, ldo, grouped, 1);
}

void gemm_pair_run_act(const GemmWeightDesc* w, const void* x, int M, int ldx, void* out, int ldo, int act, void* expanded, int* status, cudaStream_t st) {
  PairParams p = {};
  p.M = M;
  p.N = w->N;
  p.half = w->N / 2;
  p.n_tiles = (p.half + 127) / 128;
  p.m_tiles = (M + kTokens - 1) / kTokens;
  p.out = out;
  p.ldo = ldo;
  p.act_kind = act;
  p.status = status;
  launch_pair<false, 1>(w, x, ldx, M, p, expanded, st);
}

bool gemm_pair_qkv_supported(const GemmWeightDesc* w, const void* q_out, int ldo, const GemmQkvArgs* a) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return gemm_pair_supported(w, w->N, q_out, ldo, false, 2) && (a->cos_t == nullptr || a->rot_half == 64) && aligned(a->k_cache) && aligned(a->v_cache) && aligned(a->cos_t) &&
         aligned(a->sin_t);
}

void gemm_pair_run_qkv(const GemmWeightDesc* w, const void* x, int M, int ldx, void* q_out, int ldo, const float* bias, const GemmQkvArgs* a, void* expanded,
                       int* status, cudaStream_t st) {
  PairParams p = {};
  p.M = M;
  p.N = w->N;
  p.n_tiles = (w->N + 255) / 256;
  p.m_tiles = (M + kTokens - 1) / kTokens;
  p.out = q_out;
  p.ldo = ldo;
  p.bias = bias;
  p.status = status;
  p.qkv = *a;
  launch_pair<false, 2>(w, x, ldx, M, p, expanded, st);
}

// Experts: `items` of 256 rows; act 0: out [rows, n], otherwise act(gate) * up: out [rows, n / 2]. JQ4 experts are expanded inside the kernel:
// in front of it that would move 2.6 bytes per weight of every expert for a few hundred rows each.
void gemm_pair_run_grouped(const GemmWeightDesc* w, int n_per_expert, const void* x, int rows, int ldx, void* out, int ldo, const int* items, int max_items,
                           int act, int* status, cudaStream_t st) {
  PairParams p = {};
  p.M = rows;
  p.N = n_per_expert;
  p.half = n_per_expert / 2;
  p.n_tiles = act ? (p.half + 127) / 128 : (n_per_expert + 255) / 256;
  p.m_tiles = max_items;
  p.w_rows = w->is_q4 ? (n_per_expert + 127) / 128 : n_per_expert;
  p.out = out;
  p.ldo = ldo;
  p.act_kind = act;
  p.status = status;
  p.items = reinterpret_cast<const int4*>(items);
  if (act == 0) {
    if (w->is_q4) launch_pair<true, 0>(w, x, ldx, rows, p, nullptr, st);
    else launch_pair<false, 0>(w, x, ldx, rows, p, nullptr, st);
  } else {
    if (w->is_q4) launch_pair<true, 1>(w, x, ldx, rows, p, nullptr, st);
    else launch_pair<false, 1>(w, x, ldx, rows, p, nullptr, st);
  }
}

}  // namespace dlv
