// Persistent tcgen05 GEMM for prefill-sized problems (more than 128 tokens, from 65 on where K is not split): Y = X W^T with the same fused
// epilogues as the one-tile-per-CTA kernel (RMSNorm row scale, bias, residual, SwiGLU, sums of squares for the
// next norm), built so that the tensor cores never wait for an epilogue:
//
//   * one CTA per SM walks a list of [128 weight rows x up to 256 tokens] tiles (swap-AB: the weight tile is the MMA M
//     operand, the token tile the MMA N operand); dense matrices with sums of some length go to pairs of CTAs (cta_group::2), which share
//     [256 x up to 256] tiles: a CTA fetches its 128 weight rows and half of the tokens, 32 KB a stage instead of 48, and has six stages;
//   * the warps that fetch and multiply run their loops whole, and one elected lane issues (see elect_one in ptx.cuh). 2048 tokens, one
//     CTA with a lane of its own / elected / pairs: 4096 x 14336 210 / 210 / 174 us, 2 x 14336 x 4096 404 / 402 / 326, 300 tokens, 8192 x 8192
//     55.7 / 55.1 / 46;
//   * the fp32 accumulator is double-buffered in TMEM (2 x 256 columns): while the epilogue warps drain tile i,
//     the MMA warp already accumulates tile i+1;
//   * a TMA ring runs ahead across tile boundaries: six stages of 32 KB, four of 48 KB, or ten of 18 KB for the expert items of decode steps;
//   * two groups of four epilogue warps transpose through an 8 KB staging buffer each so that Y leaves the SM as 16-byte row chunks;
//   * grouped (MoE) form: the tiles come from a work table {expert, first row, rows, -} built on the device, an item of at most 256 (16) rows
//     each; a short item shortens the MMA and its copies (64 or 16 rows apiece) instead of fetching and multiplying rows nobody stores;
//   * SwiGLU ("dual") tiles load 64 gate rows and 64 up rows into ONE 128-row operand tile, so gate and up use the
//     same single 128x256 MMA stream as a plain GEMM; silu(gate) * up is formed when the staged rows are combined.
//
// Replaces the cuBLASLt matmul behind the reference's dense projections at prefill sizes
// (eredu-architectures/src/llama.rs:270-286,418-431; safemlx/src/ops/arithmetic.rs matmul).
#include "gemm_persistent.h"

#include <algorithm>

#include "../common/elem.cuh"
#include "../common/launch.h"
#include "../common/launch_count.h"
#include "../common/ptx.cuh"
#include "../common/tma_host.h"
#include "../common/trace.cuh"

namespace eredu {

namespace {

constexpr int kTN = 256;                         // tokens per tile (MMA N)
constexpr int kATile = 128 * 64 * 2;             // 16 KB: 128 weight rows x 64 k
constexpr int kBTile = kTN * 64 * 2;             // 32 KB: 256 tokens x 64 k
constexpr int kBand = 8;                         // token tiles that vary fastest
// Stages of the ring. BOX: grouped form, token rows of one copy - 64, or 16 for the items of a decode step (at most 16 rows): such a step
// streams the weights of nearly all experts, and what counts are the bytes on their way, 160 KB an SM with ten small stages.
// kPair: two CTAs share a tile, half of its tokens in the shared memory of each.
constexpr int kPair = 128;
template <int BOX>
struct Ring {
  static constexpr int kBoxBytes = BOX * 64 * 2;
  static constexpr int kStageBytes = kATile + (BOX == 16 ? kBoxBytes : BOX == kPair ? kBTile / 2 : kBTile);    // 18, 32 or 48 KB
  static constexpr int kStages = BOX == 16 ? 10 : BOX == kPair ? 6 : 4;
};
constexpr int kChunkCols = 16;                    // tokens of a staging pass: 16 x 128 fp32 = 8 KB
constexpr int kStagingBytes = kChunkCols * 128 * 4;
// Epilogue groups of four warps, which take every second chunk of tokens. With one, a tile of 256 tokens took ten microseconds to store: about as
// long as the products of short sums, and the end of every launch (2 x 8192 x 2048, 4096 tokens 258 -> 192 us, 300 tokens 31.0 -> 24.9; 4096 x 512,
// 2048 tokens 21.4 -> 15.2; 4096 x 4096, 300 tokens 19.2 -> 18.2).
constexpr int kGroups = 2;
constexpr int kThreads = 64 + 128 * kGroups;
constexpr int kCtrlBytes = 1024;
template <int BOX>
constexpr int kSmemBytes = 1024 + kCtrlBytes + Ring<BOX>::kStages * Ring<BOX>::kStageBytes + kGroups * kStagingBytes;

struct PGemmParams {
  void* y;
  const void* residual;
  const void* bias;
  int M, N, K;
  int ldy, ldr;
  int dual_row_offset;
  int* status;
  const float* ssq_in;
  int ssq_parts;
  float norm_eps;
  float norm_inv_dim;
  float* ssq_out;
  int out_fp32;  // plain tiles without residual and sums of squares: y is fp32
  float act_a, act_b;  // xIELU
  int act;  // plain tiles: 2 = squared ReLU before the residual, 4 = xIELU; dual tiles: 0 = silu(g) * u, 3 = relu(g) * u
  int n_tiles, m_tiles;
  int ssq_stride;  // tiles of 128 output columns
  int tn;  // token rows of a tile: 256, or fewer where that saves a round of tiles
  // grouped form: m_tiles work items, used ones first (the rest have no rows); the expert's weights start at row expert * w_rows_per_expert
  const int4* work;
  int w_rows_per_expert;
};

struct PTile {
  int tile_n, w_row0, m_base, m_cnt;
};

// Tile t of the list; false behind the last one.
template <bool GROUPED, int ROWS, bool PAIR>
__device__ __forceinline__ bool tile_at(const PGemmParams& p, int t, uint32_t crank, PTile& o) {
  int tile_m = t / p.n_tiles;
  o.tile_n = t % p.n_tiles;
  if (!GROUPED) {
    // Token tiles vary fastest, in bands of kBand: the CTAs at work share a few weight tiles and a band of token tiles (34 MB at K = 4096)
    // that stay in L2. Weight tiles first, 148 CTAs fetched 148 different ones (155 MB), and every token tile read all weights
    // from HBM again: 4.5 TB/s beside the products of a gate_up of 235 MB. That one (2 x 14336 x 4096), 2048 tokens: 447 -> 357 us,
    // 8192: 1655 -> 1385; 2 x 28672 x 8192, 4096 tokens: 3306 -> 2670. Bands of 4: 368, 1434, 2734; of 16: 353, 1367, 2839.
    const int band = t / (p.n_tiles * kBand), in = t - band * p.n_tiles * kBand;
    const int height = min(kBand, p.m_tiles - band * kBand);
    tile_m = band * kBand + in % height;
    o.tile_n = in / height;
  }
  if (PAIR) o.tile_n = 2 * o.tile_n + static_cast<int>(crank);
  o.w_row0 = o.tile_n * ROWS;
  if (GROUPED) {
    const int4 item = p.work[tile_m];
    o.w_row0 += item.x * p.w_rows_per_expert;
    o.m_base = item.y;
    o.m_cnt = min(item.z, kTN);
    return item.z > 0;
  }
  o.m_base = tile_m * p.tn;
  o.m_cnt = min(p.tn, p.M - o.m_base);
  return true;
}

__device__ __forceinline__ void epi_bar(int group) { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); }
// Barrier of all groups; whether any of their threads says so.
__device__ __forceinline__ bool epi_bar_any(bool said) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(any)
               : "r"(static_cast<uint32_t>(said)), "n"(1 + kGroups), "n"(128 * kGroups)
               : "memory");
  return any != 0;
}
__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + __expf(-x)); }

template <bool DUAL, bool GROUPED, int BOX>
__global__ void __launch_bounds__(kThreads, 1)
gemm_persistent_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, PGemmParams p) {
  constexpr int kStages = Ring<BOX>::kStages, kStageBytes = Ring<BOX>::kStageBytes, kBoxBytes = Ring<BOX>::kBoxBytes;
  pdl_launch_early();
  trace_mark(kTraceGemmPersistent, kTraceStart);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);   // [kStages]  TMA -> MMA
  uint64_t* empty_bar = full_bar + kStages;                 // [kStages]  MMA -> TMA
  uint64_t* tfull_bar = empty_bar + kStages;                // [2]        MMA -> epilogue (accumulator ready)
  uint64_t* tempty_bar = tfull_bar + 2;                     // [2]        epilogue -> MMA (accumulator drained)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  uint8_t* stages = smem + kCtrlBytes;
  uint8_t* staging = stages + kStages * kStageBytes;
  __shared__ float s_scales[2][kTN];     // of this tile and the next: a group may be a tile ahead

  const int warp = static_cast<int>(warp_uniform(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  const int kblocks = (p.K + 63) >> 6;
  const int total = p.n_tiles * p.m_tiles;
  constexpr int kRowsPerTile = DUAL ? 64 : 128;  // output columns (weight rows of the result) per tile and CTA
  // A pair walks the list together: first CTA's rows, then the second's. The first one's MMA warp issues for both.
  constexpr bool PAIR = BOX == kPair;
  const uint32_t crank = PAIR ? blockIdx.x & 1 : 0;
  const int first = PAIR ? blockIdx.x >> 1 : blockIdx.x, step = PAIR ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], (PAIR ? 2 : 1) * 128 * kGroups);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    __syncwarp();
    if (PAIR) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  // the other CTA's barriers and tensor memory are ready too
  if (PAIR) cluster_arrive_release();
  if (PAIR) cluster_wait_acquire();
  tc_fence_after_sync();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  pdl_wait();
  trace_mark(kTraceGemmPersistent, kTraceAfterWait);
  pdl_launch_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (the warp waits, one lane issues)
    // both operands are re-read by other CTAs from L2; the weights of experts, and of a single token tile, are not
    const uint64_t pol_w = GROUPED || p.m_tiles == 1 ? l2_policy_evict_first() : l2_policy_evict_last();
    const uint64_t pol_x = l2_policy_evict_last();
    const bool one = elect_one();
    int s = 0, issued = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int t = first; t < total && ok; t += step) {
      PTile tl;
      if (!tile_at<GROUPED, kRowsPerTile, PAIR>(p, t, crank, tl)) break;
      const int w_row0 = tl.w_row0;
      const int half = PAIR ? ((tl.m_cnt + 31) & ~31) >> 1 : 0;     // tokens that the MMA takes from either CTA
      const int m_base = tl.m_base + static_cast<int>(crank) * half;
      const int boxes = GROUPED ? (tl.m_cnt + BOX - 1) / BOX : 1;
      const uint32_t bytes = PAIR ? 2 * (kATile + p.tn * 64) : kATile + (GROUPED ? boxes * kBoxBytes : p.tn * 128);
      for (int kb = 0; kb < kblocks; ++kb) {
        ok = mbar_wait_warp(&empty_bar[s], ph ^ 1, p.status, kStatusSmemEmptyTimeout);
        if (!ok) break;
        uint8_t* a = stages + s * kStageBytes;
        if (one) {
          if (PAIR) {
            const uint32_t full = mapa_shared(smem_u32(&full_bar[s]), 0);
            if (crank == 0) mbar_arrive_expect_tx(&full_bar[s], bytes);
            tma_load_2d_pair_hint(a, &tmW, kb * 64, w_row0, full, pol_w);
            if (DUAL) tma_load_2d_pair_hint(a + kATile / 2, &tmW, kb * 64, p.dual_row_offset + w_row0, full, pol_w);
            tma_load_2d_pair_hint(a + kATile, &tmX, kb * 64, m_base, full, pol_x);
          } else {
            mbar_arrive_expect_tx(&full_bar[s], bytes);
            tma_load_2d_hint(a, &tmW, kb * 64, w_row0, &full_bar[s], pol_w);
            if (DUAL) tma_load_2d_hint(a + kATile / 2, &tmW, kb * 64, p.dual_row_offset + w_row0, &full_bar[s], pol_w);
            for (int i = 0; i < boxes; ++i) tma_load_2d_hint(a + kATile + i * kBoxBytes, &tmX, kb * 64, m_base + i * BOX, &full_bar[s], pol_x);
          }
        }
        ++issued;
        if (++s == kStages) {
          s = 0;
          ph ^= 1;
        }
      }
    }
    if (PAIR && ok) {  // until the MMA warp has given back every stage: it arrives on this CTA's barriers
      for (int j = max(0, issued - kStages); j < issued; ++j) mbar_wait(&empty_bar[j % kStages], (j / kStages) & 1, p.status, kStatusSmemEmptyTimeout);
    }
    if (!ok) {  // wait (bounded) for the copies still in flight before shared memory goes away
      for (int j = max(0, issued - kStages); j < issued; ++j) mbar_wait(&full_bar[j % kStages], (j / kStages) & 1, nullptr, 0);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of a pair, the first CTA's)
    if (crank == 0) {
      const bool one = elect_one();
      int s = 0, lt = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = first; t < total && ok; t += step, ++lt) {
        PTile tl;
        if (!tile_at<GROUPED, kRowsPerTile, PAIR>(p, t, crank, tl)) break;
        // the last token tile may be a short one
        const uint32_t idesc = PAIR ? umma_idesc_bf16(256, (tl.m_cnt + 31) & ~31) : umma_idesc_bf16(128, (tl.m_cnt + 15) & ~15);
        const int buf = lt & 1;
        const uint32_t bph = (lt >> 1) & 1;
        ok = mbar_wait_warp(&tempty_bar[buf], bph ^ 1, p.status, kStatusAccumTimeout);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t acc_addr = tmem_base + buf * kTN;
        for (int kb = 0; kb < kblocks; ++kb) {
          ok = mbar_wait_warp(&full_bar[s], ph, p.status, kStatusTmaFullTimeout);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a_addr = smem_u32(stages + s * kStageBytes);
          const uint64_t da = umma_desc_k_sw128(a_addr);
          const uint64_t db = umma_desc_k_sw128(a_addr + kATile);
          if (one) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (PAIR) umma_f16_pair(acc_addr, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
              else umma_f16(acc_addr, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            }
            if (PAIR) umma_commit_pair(&empty_bar[s]);
            else umma_commit(&empty_bar[s]);
          }
          if (++s == kStages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (ok && one) {
          if (PAIR) umma_commit_pair(&tfull_bar[buf]);
          else umma_commit(&tfull_bar[buf]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5 and 6..9)
    const int group = (warp - 2) >> 2;
    const int q = warp & 3;          // TMEM lane quarter this warp may read
    const int row = q * 32 + lane;   // accumulator lane = weight row inside the tile
    const int et = (threadIdx.x - 64) & 127;
    uint8_t* my_staging = staging + group * kStagingBytes;
    const __nv_bfloat16* res = static_cast<const __nv_bfloat16*>(p.residual);
    const __nv_bfloat16* bias = static_cast<const __nv_bfloat16*>(p.bias);
    __nv_bfloat16* yout = static_cast<__nv_bfloat16*>(p.y);
    int lt = 0;
    for (int t = first; t < total; t += step, ++lt) {
      PTile tl;
      if (!tile_at<GROUPED, kRowsPerTile, PAIR>(p, t, crank, tl)) break;
      const int tile_n = tl.tile_n, m_base = tl.m_base, m_cnt = tl.m_cnt;
      const int buf = lt & 1;
      const uint32_t bph = (lt >> 1) & 1;
      float* s_scale = s_scales[buf];
      if (p.ssq_in != nullptr) {
        for (int c = threadIdx.x - 64; c < kTN; c += 128 * kGroups) {
          float s = 0.f;
          if (c < m_cnt) {
            const float* src = p.ssq_in + static_cast<size_t>(m_base + c) * p.ssq_parts;
            for (int j = 0; j < p.ssq_parts; ++j) s += src[j];
          }
          s_scale[c] = rsqrtf(s * p.norm_inv_dim + p.norm_eps);
        }
      }
      // s_scale is complete behind this; all epilogue threads agree on a failure
      if (epi_bar_any(!mbar_wait(&tfull_bar[buf], bph, p.status, kStatusAccumTimeout))) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + buf * kTN + (static_cast<uint32_t>(q * 32) << 16);
      // this thread's weight row: output column n (DUAL: gate rows are lanes 0..63, up rows lanes 64..127)
      const int n = DUAL ? tile_n * 64 + (row & 63) : tile_n * 128 + row;
      const bool in_n = n < p.N;
      float b_row = 0.f;
      if (bias != nullptr && in_n) b_row = __bfloat162float(bias[DUAL && row >= 64 ? p.N + n : n]);
      const int chunks = (m_cnt + kChunkCols - 1) / kChunkCols;       // chunks past the last token are skipped
      const int last_cc = ((chunks - 1 - group) / kGroups * kGroups + group) * kChunkCols;     // this group's last one
      if (group >= chunks) {        // none: the accumulator is not waited for
        if (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[buf]), 0));
        else mbar_arrive(&tempty_bar[buf]);
      }
      for (int cc = group * kChunkCols; group < chunks && cc <= last_cc; cc += kGroups * kChunkCols) {
        // Second-pass work items of this thread (16-byte pieces of output rows); their residual is fetched now
        // so that the loads are in flight while the accumulator is read.
        constexpr int kItems = kChunkCols * kRowsPerTile / 8 / 128;
        uint4 rv[kItems];
        bool item_ok[kItems];
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
          const int id = et + 128 * i;
          const int c = DUAL ? id >> 3 : id >> 4;
          const int gn = DUAL ? tile_n * 64 + (id & 7) * 8 : tile_n * 128 + (id & 15) * 8;
          item_ok[i] = cc + c < m_cnt && gn < p.N;
          rv[i] = make_uint4(0u, 0u, 0u, 0u);
          if (item_ok[i] && res != nullptr) rv[i] = *reinterpret_cast<const uint4*>(res + static_cast<size_t>(m_base + cc + c) * p.ldr + gn);
        }
        float* stf = reinterpret_cast<float*>(my_staging);
#pragma unroll
        for (int c0 = 0; c0 < kChunkCols; c0 += 16) {
          uint32_t g[16];
          tmem_ld16(taddr + cc + c0, g);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float sc = (p.ssq_in != nullptr) ? s_scale[cc + c0 + j] : 1.f;
            stf[(c0 + j) * 128 + row] = __uint_as_float(g[j]) * sc + b_row;
          }
        }
        if (cc == last_cc) {
          // this thread has read everything it needs from TMEM: hand the accumulator back to the MMA warp
          tc_fence_before_sync();
          if (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty_bar[buf]), 0));
          else mbar_arrive(&tempty_bar[buf]);
        }
        epi_bar(group);
        const float* st = reinterpret_cast<const float*>(my_staging);
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
          const int id = et + 128 * i;
          const int c = DUAL ? id >> 3 : id >> 4;
          const int n0 = DUAL ? (id & 7) * 8 : (id & 15) * 8;
          const int m = m_base + cc + c;
          const int gn = tile_n * kRowsPerTile + n0;
          const float4 g0 = *reinterpret_cast<const float4*>(st + c * 128 + n0);
          const float4 g1 = *reinterpret_cast<const float4*>(st + c * 128 + n0 + 4);
          float v[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
          if (DUAL) {
            const float4 u0 = *reinterpret_cast<const float4*>(st + c * 128 + 64 + n0);
            const float4 u1 = *reinterpret_cast<const float4*>(st + c * 128 + 64 + n0 + 4);
            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = (p.act == 3 ? fmaxf(v[j], 0.f) : silu_f(v[j])) * u[j];
          }
          if (!DUAL && p.act == 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              v[j] = fmaxf(v[j], 0.f);
              v[j] *= v[j];
            }
          }
          if (!DUAL && p.act == 4) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = xielu<true>(v[j], p.act_a, p.act_b);
          }
          if (!DUAL && p.out_fp32) {
            if (item_ok[i]) {
              float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.y) + static_cast<size_t>(m) * p.ldy + gn);
              dst[0] = make_float4(v[0], v[1], v[2], v[3]);
              dst[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
            continue;
          }
          const uint32_t r[4] = {rv[i].x, rv[i].y, rv[i].z, rv[i].w};
          uint4 o;
          o.x = pack_bf16x2(v[0] + bf16_lo(r[0]), v[1] + bf16_hi(r[0]));
          o.y = pack_bf16x2(v[2] + bf16_lo(r[1]), v[3] + bf16_hi(r[1]));
          o.z = pack_bf16x2(v[4] + bf16_lo(r[2]), v[5] + bf16_hi(r[2]));
          o.w = pack_bf16x2(v[6] + bf16_lo(r[3]), v[7] + bf16_hi(r[3]));
          if (item_ok[i]) *reinterpret_cast<uint4*>(yout + static_cast<size_t>(m) * p.ldy + gn) = o;
          if (!DUAL && p.ssq_out != nullptr) {
            const uint32_t w[4] = {o.x, o.y, o.z, o.w};
            float sq = 0.f;
            if (item_ok[i]) {
#pragma unroll
              for (int j = 0; j < 4; ++j) sq += bf16_lo(w[j]) * bf16_lo(w[j]) + bf16_hi(w[j]) * bf16_hi(w[j]);
            }
#pragma unroll
            for (int o2 = 8; o2 > 0; o2 >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o2);
            if ((lane & 15) == 0 && cc + c < m_cnt && tile_n < p.ssq_stride) p.ssq_out[static_cast<size_t>(m) * p.ssq_stride + tile_n] = sq;
          }
        }
        epi_bar(group);  // staging may be overwritten
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) {   // neither leaves while the other's products read its shared memory, or its barriers are arrived on
    cluster_arrive_release();
    cluster_wait_acquire();
  }
  if (warp == 1) {
    __syncwarp();
    if (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
  trace_mark(kTraceGemmPersistent, kTraceEnd);
}

}  // namespace

// Token rows of a tile. A CTA (pair) walks ceil(tiles / CTAs) tiles, and with 256 rows the last of these walks is often nearly empty (1250 x 4096:
// 80 tiles on 74 pairs). Microseconds of a pair per 64 of K with 256, 224, 192, 160, 128, 96 and 64 rows: 0.40, 0.34, 0.30, 0.26, 0.25, 0.25
// and 0.24 (what it takes to fetch and issue a stage); of one CTA with 256, 128 and 64: 0.49, 0.33, 0.29 (it fetches 128 weight rows and all tokens).
// 1250 x 4096 x 14336 157 us -> 114, 1024 x 4096 x 4096 32.9 -> 28.5, 300 x 8192 x 8192 55 -> 46.
static int pick_token_tile(int M, int n_tiles, int workers, bool pair) {
  int best = kTN;
  long cost = -1;
  for (int tn = kTN; tn >= 64; tn -= pair ? 32 : 16) {
    const long tiles = static_cast<long>(n_tiles) * ((M + tn - 1) / tn);
    const int rows = std::min(tn, M);
    const long c = (tiles + workers - 1) / workers * (pair ? std::max(rows + 22, 172) : std::max(rows + 128, 220));
    if (cost < 0 || c < cost) {
      cost = c;
      best = tn;
    }
  }
  return best;
}

template <bool DUAL>
static cudaError_t launch_pair(const CUtensorMap& tmW, const CUtensorMap& tmX, const PGemmParams& p, int grid, cudaStream_t stream) {
  static bool configured[64] = {};  // the attribute is a per-device setting
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(gemm_persistent_kernel<DUAL, false, kPair>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes<kPair>);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes<kPair>;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gemm_persistent_kernel<DUAL, false, kPair>, tmW, tmX, p);
}

int launch_gemm_persistent(const void* X, const void* W, void* Y, const void* residual, const void* bias, int M, int N,
                           int K, int ldx, int ldw, int ldy, int ldr, int w_rows, int dual, int dual_row_offset,
                           int sm_count, int* status, const float* ssq_in, int ssq_parts, float norm_eps, int norm_dim,
                           float* ssq_out, int act, float act_a, float act_b, int out_fp32, cudaStream_t stream) {
  if (N % 8 != 0 || ldy % 8 != 0 || (reinterpret_cast<uintptr_t>(Y) & 15) != 0) return kPersistentUnsupported;
  if (out_fp32 && (dual || residual != nullptr || ssq_out != nullptr)) return kPersistentUnsupported;
  if (dual && (ssq_out != nullptr || N % 64 != 0 || dual_row_offset % 8 != 0)) return kPersistentUnsupported;
  if (residual != nullptr && (ldr % 8 != 0 || (reinterpret_cast<uintptr_t>(residual) & 15) != 0)) return kPersistentUnsupported;
  CUtensorMap tmW, tmX;
  int r = make_tma_2d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_rows, K, ldw, dual ? 64 : 128, 64);
  if (r != 0) return -100 + r;
  const int sms = sm_count > 0 ? sm_count : 148;
  const int n_tiles = dual ? (N + 63) / 64 : (N + 127) / 128;
  // Two CTAs to a tile: 1.1 to 1.3 times the speed wherever the products count. Sums of less than sixteen blocks are bound by the epilogue, and a
  // second CTA without rows does not help a single row tile (8192 x 2 x 768 x 768: 22.8 us with one CTA, 23.6 with two).
  const bool pair = K >= 1024 && n_tiles > 1 && sms > 1;
  const int workers = pair ? sms / 2 : sms, row_tiles = pair ? (n_tiles + 1) / 2 : n_tiles;
  const int tn = pick_token_tile(M, row_tiles, workers, pair);
  r = make_tma_2d(&tmX, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, M, K, ldx, pair ? tn / 2 : tn, 64);
  if (r != 0) return -200 + r;
  PGemmParams p = {};
  p.y = Y;
  p.residual = residual;
  p.bias = bias;
  p.M = M;
  p.N = N;
  p.K = K;
  p.ldy = ldy;
  p.ldr = ldr;
  p.dual_row_offset = dual_row_offset;
  p.status = status;
  p.ssq_in = ssq_in;
  p.ssq_parts = ssq_parts;
  p.norm_eps = norm_eps;
  p.norm_inv_dim = norm_dim > 0 ? 1.0f / static_cast<float>(norm_dim) : 0.f;
  p.ssq_out = ssq_out;
  p.act = act;
  p.act_a = act_a;
  p.act_b = act_b;
  p.out_fp32 = out_fp32;
  p.n_tiles = row_tiles;
  p.ssq_stride = n_tiles;
  p.tn = tn;
  p.m_tiles = (M + tn - 1) / tn;
  const int total = p.n_tiles * p.m_tiles;
  // equal rounds for every CTA where possible: ceil(total / rounds) CTAs, never more than the SM count
  const int rounds = (total + workers - 1) / workers;
  const int grid = (total + rounds - 1) / rounds * (pair ? 2 : 1);
  if (pair) {
    const cudaError_t e = dual ? launch_pair<true>(tmW, tmX, p, grid, stream) : launch_pair<false>(tmW, tmX, p, grid, stream);
    eredu_count_launches(1);
    return static_cast<int>(e);
  }
  auto launch = [&](auto kern) -> cudaError_t {
    static bool configured_plain = false, configured_dual = false;
    bool& configured = dual ? configured_dual : configured_plain;
    if (!configured) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes<64>);
      if (e != cudaSuccess) return e;
      configured = true;
    }
    return launch_pdl(kern, dim3(grid), dim3(kThreads), kSmemBytes<64>, stream, tmW, tmX, p);
  };
  const cudaError_t e = dual ? launch(gemm_persistent_kernel<true, false, 64>) : launch(gemm_persistent_kernel<false, false, 64>);
  eredu_count_launches(1);
  return static_cast<int>(e);
}

template <bool DUAL, int BOX>
static cudaError_t launch_grouped(const CUtensorMap& tmW, const CUtensorMap& tmX, const PGemmParams& p, int sms, cudaStream_t stream) {
  static bool configured[64] = {};  // the attribute is a per-device setting
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(gemm_persistent_kernel<DUAL, true, BOX>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes<BOX>);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int total = p.n_tiles * p.m_tiles;
  return launch_pdl(gemm_persistent_kernel<DUAL, true, BOX>, dim3(total < sms ? total : sms), dim3(kThreads), kSmemBytes<BOX>, stream, tmW, tmX, p);
}

int launch_gemm_persistent_grouped(const void* X, const void* W, void* Y, const int* work, int n_work, int item_rows, int rows_cap, int N, int K,
                                   int ldx, int ldw, int ldy, int w_rows_total, int w_rows_per_expert, int dual, int sm_count, int* status,
                                   cudaStream_t stream) {
  if (N % 8 != 0 || ldy % 8 != 0 || (reinterpret_cast<uintptr_t>(Y) & 15) != 0 || (dual && N % 64 != 0)) return kPersistentUnsupported;
  const int sms = sm_count > 0 ? sm_count : 148, box = item_rows <= 16 ? 16 : 64;
  CUtensorMap tmW, tmX;
  int r = make_tma_2d(&tmW, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w_rows_total, K, ldw, dual ? 64 : 128, 64);
  if (r != 0) return -100 + r;
  r = make_tma_2d(&tmX, X, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, rows_cap, K, ldx, box, 64);
  if (r != 0) return -200 + r;
  PGemmParams p = {};
  p.y = Y;
  p.M = rows_cap;
  p.N = N;
  p.K = K;
  p.ldy = ldy;
  p.dual_row_offset = N;
  p.status = status;
  p.n_tiles = dual ? N / 64 : (N + 127) / 128;
  p.m_tiles = n_work;
  p.work = reinterpret_cast<const int4*>(work);
  p.w_rows_per_expert = w_rows_per_expert;
  cudaError_t e;
  if (box == 16) e = dual ? launch_grouped<true, 16>(tmW, tmX, p, sms, stream) : launch_grouped<false, 16>(tmW, tmX, p, sms, stream);
  else e = dual ? launch_grouped<true, 64>(tmW, tmX, p, sms, stream) : launch_grouped<false, 64>(tmW, tmX, p, sms, stream);
  eredu_count_launches(1);
  return static_cast<int>(e);
}

}  // namespace eredu

EREDU_TRACE_INSTALLER(gemm_persistent)
