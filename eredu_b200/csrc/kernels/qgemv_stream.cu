// Persistent 4-bit decode kernel on integer tensor-core products: Y[M,N] = X[M,K] · dequant(Wq)[N,K]^T for one or two tokens, groups of 64
// or 128, matrices that give every SM more than a round of the register kernel (qgemv_mma.cu).
//
// That kernel is bound by the instructions that turn codes into bf16 operands: 85 a 16 x 64 tile, 28 of them on the half-rate integer
// pipe, and a last wave of CTAs that is nearly empty (a 57344 x 8192 gate_up has 3.03). Here a mask, and a shift and a mask, make eight u8
// operands of a word of codes (three instructions instead of seven), mma.m16n8k32 (u8 x s8 -> s32) takes twice the K of the bf16 form
// at the same rate (8.3 cycles per scheduler for either), and the CTAs are persistent.
//
// Activations as integers: within the 64 values of a token's K block, x = 2^(e-20) v with e the exponent of the largest and
// v = 65536 d2 + 256 d1 + d0, three signed bytes (21 bits and sign: a bf16 within a factor of 2^13 of the largest is represented exactly,
// smaller ones to 2^-21 of it). The products with a code (0..15) and their sums over 64 are exact in 32 bits, so what rounds is what
// rounded before: fp32 fmas per block for scale and bias,
//   sum_k (s c_k + b) x_k  =  sum_p s X_p (sum_k c_k d_pk)  +  b * sum_k x_k          X_p = 2^(e-20) 256^p
// (with the sum of the x as represented, so that what is lost of a small one is weighted with its weight and not with its code).
// The accumulators start at the bits of 1.5 * 2^23, so that their bits are the floats 1.5 * 2^23 + sum and no conversion is needed.
// A block that holds an infinity or a NaN makes its token's results NaN, as the bf16 form does (128 + code and its correction cancel there).
// Errors against 64 bits (2-norm): 1.1e-7 of normal activations (bf16 form 1.2e-6), 1.6e-6 with one of 10^4 times the others' size in each
// block (2.8e-6), 1.1e-6 to 1.5e-6 of activations over nine decades (2.3e-6 to 2.8e-6).
//
// One CTA of sixteen warps per SM (eight left the chains of a warp exposed: gate_up 69 us instead of 56 before the loops were trimmed, 45 now), or a
// cluster of ns that splits K, walks a run of 16-row tiles. The activations are turned into bytes once per CTA, in shared memory, in the
// order in which lanes meet them; every warp has a K range of its own and a private ring of bulk copies that runs on across the rounds of
// four tiles (of a gated matrix two gate and two up tiles), so that HBM does not wait for the sum over warps and CTAs at the end of a round.
// CTAs of a cluster send each other their sums (st.async) and take them a round later.
//
// With three pieces a token, three to eight tokens would need three products and their fmas; in this form as in the bf16 one (86 us of a
// gate_up with its activations in shared memory) they lost against the register kernel (72).
#include "qgemv_stream.h"

#include <algorithm>

#include "../common/launch.h"
#include "../common/launch_count.h"
#include "../common/ptx.cuh"

namespace eredu {

namespace {

constexpr int kWarps = 16, kThreads = 32 * kWarps;
constexpr int kTiles = 4;                 // row tiles of a round
constexpr int kChunk = 2;                 // K blocks of a slot
constexpr int kMaxSlots = 4;
constexpr float kMagic = 12582912.f;      // 1.5 * 2^23
constexpr uint32_t kMagicBits = 0x4B400000u;
constexpr int kMaxSmem = 226 * 1024;
constexpr int kCtrlBytes = 1024;          // [16 warps][kMaxSlots] ring barriers, [2] barriers of the exchange

// of a K block: three pieces of M tokens, then four float4 {X, X, sum, sum}
__host__ __device__ constexpr int x_block_bytes(int M) { return 3 * 64 * M + 64; }
__host__ __device__ constexpr int dq_slot_bytes(int group_shift) { return (kChunk * 64 >> group_shift) * 64; }
__host__ __device__ constexpr int slot_bytes(int group_shift) { return kTiles * (kChunk * 512 + dq_slot_bytes(group_shift)); }
__host__ __device__ constexpr int round_rows(bool gated) { return (gated ? kTiles / 2 : kTiles) * 16; }
__host__ __device__ constexpr int red_plane(bool gated, int tokens) { return (gated ? 2 : 1) * tokens * (round_rows(gated) + 4); }   // floats of a warp
__host__ __device__ constexpr int recv_floats(bool gated, int tokens) { return (gated ? 2 : 1) * tokens * round_rows(gated); }       // of a round, all ranks

__device__ __forceinline__ void store_async(uint32_t addr, float v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
               :
               : "r"(addr), "r"(__float_as_uint(v)), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_u8s8_first(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kMagicBits));
}

// Sixteen consecutive values of a block as bytes, in the order in which a word of codes falls apart under the two masks: (0,4,1,5), (2,6,3,7)
// and the same of the second eight. out[piece]: d2, d1, d0; returns the sum of the sixteen v.
__device__ __forceinline__ int split_bytes(const uint32_t (&w)[8], float inv, uint4 (&out)[3]) {
  uint32_t b[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    // + 0x8080: bytes 0 and 1 are then digits plus 128, and what is above them is rounded to fit
    b[2 * i] = __float_as_uint(fmaf(bf16_lo(w[i]), inv, kMagic + 32896.f));
    b[2 * i + 1] = __float_as_uint(fmaf(bf16_hi(w[i]), inv, kMagic + 32896.f));
  }
  uint32_t d[3][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int k = (r >> 1) * 8 + (r & 1) * 2;
    const uint32_t A = b[k], B = b[k + 4], C = b[k + 1], D = b[k + 5];
    const uint32_t ab = __byte_perm(A, B, 0x5140), cd = __byte_perm(C, D, 0x5140);
    d[2][r] = __byte_perm(ab, cd, 0x5410) ^ 0x80808080u;
    d[1][r] = __byte_perm(ab, cd, 0x7632) ^ 0x80808080u;
    // byte 2 is 64 + d2 with d2 in [-32, 32]: bit 6 flipped and copied to bit 7
    const uint32_t hi = __byte_perm(__byte_perm(A, B, 0x0062), __byte_perm(C, D, 0x0062), 0x5410) ^ 0x40404040u;
    d[0][r] = hi | ((hi & 0x40404040u) << 1);
  }
#pragma unroll
  for (int p = 0; p < 3; ++p) out[p] = make_uint4(d[p][0], d[p][1], d[p][2], d[p][3]);
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < 16; ++i) sum += b[i];
  return static_cast<int>(sum - 16u * (kMagicBits + 32896u));
}

// Column 2 p + m of a product is piece p of token m.
template <bool GATED, int TOK>
__global__ void __launch_bounds__(kThreads, 1) qgemv4_stream_kernel(const QGemvStreamParams p) {
  constexpr int S = GATED ? 2 : 1;
  constexpr int T = kTiles, RT = T / S;
  constexpr int ROWS = round_rows(GATED), LDN = ROWS + 4, PLANE = red_plane(GATED, TOK);
  constexpr int XSTRIDE = x_block_bytes(TOK);
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem);                  // [16 warps][kMaxSlots]
  uint64_t* xbars = bars + kWarps * kMaxSlots;                         // [2]
  float* red = reinterpret_cast<float*>(smem + kCtrlBytes);            // [2][16 warps][PLANE]
  float* recv = red + 2 * kWarps * PLANE;                              // [2][ns ranks][S][TOK][cols] (clusters)
  const int slot_size = slot_bytes(p.group_shift);
  uint8_t* ring = reinterpret_cast<uint8_t*>(recv + (p.ns > 1 ? 2 * recv_floats(GATED, TOK) : 0));   // [16 warps][slots]
  uint8_t* xs = ring + kWarps * p.slots * slot_size;                   // [kb_cta][XSTRIDE]

  pdl_launch_early();

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  uint32_t crank = 0;
  if (p.ns > 1) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  // the run of row tiles of this cluster, and the K blocks of this CTA and warp
  const int u0 = static_cast<int>(static_cast<long long>(blockIdx.x) * p.units / gridDim.x);
  const int u1 = static_cast<int>(static_cast<long long>(blockIdx.x + 1) * p.units / gridDim.x);
  const int rounds = (u1 - u0 + RT - 1) / RT;
  const int kbc0 = min(static_cast<int>(crank) * p.kb_cta, p.kblocks), kbc1 = min(kbc0 + p.kb_cta, p.kblocks);
  const int kb0 = min(kbc0 + warp * p.kb_warp, kbc1), kb1 = min(kb0 + p.kb_warp, kbc1);
  constexpr int C = kChunk;
  const int cols = ROWS / p.ns;                                        // output columns of a round that this CTA finishes

  uint8_t* my_ring = ring + warp * p.slots * slot_size;
  uint64_t* my_bars = bars + warp * kMaxSlots;
  if (lane == 0) {
    for (int i = 0; i < p.slots; ++i) mbar_init(&my_bars[i], 1);
    if (warp == 0 && p.ns > 1)
      for (int i = 0; i < 2; ++i) {
        mbar_init(&xbars[i], 1);
        mbar_arrive_expect_tx(&xbars[i], static_cast<uint32_t>(p.ns * S * TOK * cols * 4));
      }
    fence_mbar_init();
  }
  __syncwarp();
  if (p.ns > 1) cluster_arrive_release();

  // lane s < T copies the codes of tile s of a round, lane T + s its (scale, bias) words; the copies run on across rounds
  const bool copies_dq = lane >= T;
  const int cs = lane % T;
  const int dq_slot = dq_slot_bytes(p.group_shift);                 // of a tile
  const size_t tile_bytes = copies_dq ? (static_cast<size_t>(p.kblocks) * 64 >> p.group_shift) * 64 : static_cast<size_t>(p.kblocks) * 512;
  const uint8_t* csrc = (copies_dq ? reinterpret_cast<const uint8_t*>(p.dq) : p.wq) +
                        static_cast<size_t>(u0 + cs % RT + (cs / RT) * p.units) * tile_bytes;       // GATED: the up tiles follow the gate tiles
  const uint32_t cdst = smem_u32(my_ring) + (copies_dq ? T * C * 512 + cs * dq_slot : cs * C * 512);
  int ileft = kb1 > kb0 ? u1 - u0 : 0, ikb = kb0, islot = 0;           // tiles left, next K block, next slot
  auto issue = [&]() {   // whole warp: the next slot, if there is one
    if (ileft <= 0) return;
    const int live = min(RT, ileft), nb = min(C, kb1 - ikb);
    const uint32_t dq_bytes = max(1, (nb * 64) >> p.group_shift) * 64, code_bytes = nb * 512;
    uint64_t* bar = &my_bars[islot];
    if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(live * S) * (code_bytes + dq_bytes));
    __syncwarp();
    if (lane < 2 * T && cs % RT < live) {
      const uint32_t off = copies_dq ? static_cast<uint32_t>((ikb * 64) >> p.group_shift) * 64 : static_cast<uint32_t>(ikb) * 512;
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                   :
                   : "r"(cdst + islot * slot_size), "l"(csrc + off), "r"(copies_dq ? dq_bytes : code_bytes), "r"(smem_u32(bar))
                   : "memory");
    }
    ikb += C;
    if (ikb >= kb1) {
      ikb = kb0;
      ileft -= RT;
      csrc += RT * tile_bytes;
    }
    if (++islot == p.slots) islot = 0;
  };

  // weights do not depend on the previous kernel: the ring is full before the dependency wait
  for (int i = 0; i < p.slots; ++i) issue();

  pdl_wait();
  pdl_launch_dependents();

  // ---- activations of this CTA's K blocks: four lanes per token and block, 16 values each
  const int pairs = TOK * (kbc1 - kbc0);
  for (int q = threadIdx.x >> 2; q < ((pairs + 7) & ~7); q += kThreads / 4) {      // whole warps: eight pairs at a time
    const bool live = q < pairs;
    const int kbl = live ? q / TOK : 0, m = live ? q % TOK : 0;
    const uint4* src = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(m) * p.ldx + (kbc0 + kbl) * 64 + t * 16);
    const uint4 v0 = src[0], v1 = src[1];
    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) top = __vmaxu2(top, w[i] & 0x7FFF7FFFu);
    top = max(top >> 16, top & 0xFFFFu);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    const int raw_e = static_cast<int>(top >> 7);
    const int e = max(raw_e, 21);                       // below 2^-106 the unit stays 2^-126
    uint4 d[3];
    int sum = split_bytes(w, __uint_as_float(static_cast<uint32_t>(274 - e) << 23), d);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (live) {
      uint8_t* xb = xs + kbl * XSTRIDE;
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(xb + (i * TOK + m) * 64 + t * 16) = d[i];
      // lane t's columns 2 t + m: piece t (a fourth is empty), X = 2^(e - 127 - 20 + 8 (2 - t)); the sum goes with the top piece
      float* table = reinterpret_cast<float*>(xb + XSTRIDE - 64);
      const bool finite = raw_e < 255;
      const float nan = __uint_as_float(0x7FC00000u);
      table[t * 4 + m] = !finite ? nan : t < 3 ? __uint_as_float(static_cast<uint32_t>(e - 4 - 8 * t) << 23) : 0.f;
      table[t * 4 + 2 + m] = t > 0 ? 0.f : finite ? static_cast<float>(sum) * __uint_as_float(static_cast<uint32_t>(e - 20) << 23) : nan;
    }
  }
  if (p.ns > 1) cluster_wait_acquire();     // the peers' barriers are ready for what they are sent
  __syncthreads();

  // this lane's operands inside a block of activations (columns that do not exist read one that does: their X is 0)
  const uint32_t xoff = ((g < 6 ? g >> 1 : 0) * TOK + min(g & 1, TOK - 1)) * 64 + t * 16;
  const uint32_t toff = XSTRIDE - 64 + t * 16;
  const uint32_t code_off = g * 32 + t * 8;

  float acc[T][4];
  // one K block of the four tiles, side by side: their chains of products do not wait for one another
  auto block = [&](const uint8_t* codes, const uint32_t* dqs, const uint8_t* xb) {
    const uint4 b = *reinterpret_cast<const uint4*>(xb + xoff);
    const float4 tb = *reinterpret_cast<const float4*>(xb + toff);
    uint2 lo[T], hi[T];
#pragma unroll
    for (int s = 0; s < T; ++s) {
      lo[s] = *reinterpret_cast<const uint2*>(codes + s * C * 512);
      hi[s] = *reinterpret_cast<const uint2*>(codes + s * C * 512 + 8 * 32);
    }
    constexpr uint32_t kMask = 0x0F0F0F0Fu;
    int d[T][4];
#pragma unroll
    for (int s = 0; s < T; ++s) mma_u8s8_first(d[s], lo[s].x & kMask, hi[s].x & kMask, (lo[s].x >> 4) & kMask, (hi[s].x >> 4) & kMask, b.x, b.y);
#pragma unroll
    for (int s = 0; s < T; ++s) mma_u8s8(d[s], lo[s].y & kMask, hi[s].y & kMask, (lo[s].y >> 4) & kMask, (hi[s].y >> 4) & kMask, b.z, b.w);
#pragma unroll
    for (int s = 0; s < T; ++s) {
      const uint32_t sc_lo = dqs[s * (dq_slot / 4)], sc_hi = dqs[s * (dq_slot / 4) + 8];
      const float s_lo = __uint_as_float(sc_lo << 16), s_hi = __uint_as_float(sc_hi << 16);
      const float b_lo = __uint_as_float(sc_lo & 0xFFFF0000u), b_hi = __uint_as_float(sc_hi & 0xFFFF0000u);
      acc[s][0] = fmaf(s_lo * tb.x, __int_as_float(d[s][0]) - kMagic, fmaf(b_lo, tb.z, acc[s][0]));
      acc[s][2] = fmaf(s_hi * tb.x, __int_as_float(d[s][2]) - kMagic, fmaf(b_hi, tb.z, acc[s][2]));
      if (TOK > 1) {
        acc[s][1] = fmaf(s_lo * tb.y, __int_as_float(d[s][1]) - kMagic, fmaf(b_lo, tb.w, acc[s][1]));
        acc[s][3] = fmaf(s_hi * tb.y, __int_as_float(d[s][3]) - kMagic, fmaf(b_hi, tb.w, acc[s][3]));
      }
    }
  };

  const uint32_t recv_addr = smem_u32(recv), xbar_addr = smem_u32(xbars);
  // sum over the warps of output column cl, token m, half s of round r
  auto warps_sum = [&](int r, int s, int m, int cl) {
    const float* src = red + (r & 1) * kWarps * PLANE + (s * TOK + m) * LDN + cl;
    float part[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) part[w] = src[w * PLANE];
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += part[w];
    return sum;
  };
  auto finish = [&](int r, int m, int cl, const float (&v)[S]) {
    const int unit = u0 + r * RT, n = unit * 16 + cl;
    if (cl >= (u1 - unit) * 16 || n >= p.n_out) return;
    float out;
    if (GATED) {
      float gate = v[0], up = v[S - 1];
      if (p.bias != nullptr) {
        gate += __bfloat162float(p.bias[n]);
        up += __bfloat162float(p.bias[p.n_out + n]);
      }
      if (p.limit > 0.f) {
        gate = fminf(gate, p.limit);
        up = fminf(fmaxf(up, -p.limit), p.limit);
      }
      out = gate / (1.f + __expf(-gate)) * up;
    } else {
      out = v[0];
      if (p.bias != nullptr) out += __bfloat162float(p.bias[n]);
      if (p.residual != nullptr) out += __bfloat162float(p.residual[static_cast<size_t>(m) * p.ldr + n]);
    }
    if (p.out_fp32) static_cast<float*>(p.y)[static_cast<size_t>(m) * p.ldy + n] = out;
    else static_cast<__nv_bfloat16*>(p.y)[static_cast<size_t>(m) * p.ldy + n] = __float2bfloat16(out);
  };
  // clusters: what all CTAs of the cluster, this one too, have sent of round r, summed in rank order. A round later than it was sent, so that nobody
  // waits for it, and in front of the barrier behind which this CTA sends the next sums. A buffer is written again two rounds later, by a CTA that has
  // received all that this one sent in the round between: behind that barrier, so after these reads. For the same reason no barrier
  // completes a second phase before the first has been seen.
  const int part_floats = S * TOK * cols;
  auto finish_exchange = [&](int r) {
    if (threadIdx.x >= TOK * cols || !mbar_wait(&xbars[r & 1], (r >> 1) & 1, p.status, kStatusSmemEmptyTimeout)) return;
    if (threadIdx.x == 0 && r + 2 < rounds) mbar_arrive_expect_tx(&xbars[r & 1], static_cast<uint32_t>(p.ns * part_floats * 4));
    const float* from = recv + (r & 1) * recv_floats(GATED, TOK);
    const int m = threadIdx.x / cols, c = threadIdx.x % cols;
    float v[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
      v[s] = 0.f;
      for (int q = 0; q < p.ns; ++q) v[s] += from[q * part_floats + (s * TOK + m) * cols + c];
    }
    finish(r, m, static_cast<int>(crank) * cols + c, v);
  };

  bool ok = true;
  int slot_i = 0, parity = 0;
  for (int r = 0; r < rounds; ++r) {
#pragma unroll
    for (int s = 0; s < T; ++s)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[s][j] = 0.f;
    const uint8_t* xb = xs + (kb0 - kbc0) * XSTRIDE;
    for (int kb = kb0; kb < kb1; kb += C) {
      if (ok) ok = mbar_wait(&my_bars[slot_i], parity, p.status, kStatusTmaFullTimeout);
      if (!ok) break;
      const uint8_t* slot = my_ring + slot_i * slot_size;
      const uint32_t* dqs = reinterpret_cast<const uint32_t*>(slot + T * C * 512) + g;
      const int nb = min(C, kb1 - kb);
      block(slot + code_off, dqs, xb);
      if (nb == 2) block(slot + 512 + code_off, dqs + (64 >> p.group_shift) * 16, xb + XSTRIDE);
      xb += 2 * XSTRIDE;
      __syncwarp();                                 // every lane has read this slot
      issue();
      if (++slot_i == p.slots) {
        slot_i = 0;
        parity ^= 1;
      }
    }
    // ---- sum over warps and CTAs, and the epilogue. Of two buffers: what is read here is written again two rounds, and a barrier, later
    float* mine = red + ((r & 1) * kWarps + warp) * PLANE;
#pragma unroll
    for (int s = 0; s < T; ++s) {
      // the pieces of a token lie in the lanes of a group
#pragma unroll
      for (int j = 0; j < 4; j += TOK > 1 ? 1 : 2) {
        float v = acc[s][j];
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        if (t == 0) mine[((s / RT) * TOK + (j & 1)) * LDN + (s % RT) * 16 + g + (j >> 1) * 8] = v;
      }
    }
    if (p.ns > 1 && r > 0) finish_exchange(r - 1);
    __syncthreads();
    if (p.ns == 1) {
      if (threadIdx.x < TOK * ROWS) {
        const int m = threadIdx.x / ROWS, cl = threadIdx.x % ROWS;
        float v[S];
#pragma unroll
        for (int s = 0; s < S; ++s) v[s] = warps_sum(r, s, m, cl);
        finish(r, m, cl, v);
      }
    } else if (threadIdx.x < S * TOK * ROWS) {
      const int cl = threadIdx.x % ROWS, sm = threadIdx.x / ROWS, m = sm % TOK, s = sm / TOK;
      const float v = warps_sum(r, s, m, cl);
      const uint32_t owner = static_cast<uint32_t>(cl / cols);
      const uint32_t off = ((r & 1) * recv_floats(GATED, TOK) + static_cast<int>(crank) * part_floats + sm * cols + cl % cols) * 4;
      store_async(mapa_shared(recv_addr + off, owner), v, mapa_shared(xbar_addr + (r & 1) * 8, owner));
    }
  }
  if (p.ns > 1 && rounds > 0) finish_exchange(rounds - 1);
  if (!ok) {
    // a copy never landed (status recorded): give the other copies of this warp their bounded wait before the memory goes away
    for (int i = 0; i < p.slots; ++i) {
      mbar_wait(&my_bars[slot_i], parity, nullptr, 0);
      if (++slot_i == p.slots) {
        slot_i = 0;
        parity ^= 1;
      }
    }
  }
  if (p.ns > 1) {
    // nobody leaves while a peer may still send to it
    cluster_arrive_release();
    cluster_wait_acquire();
  }
}

int smem_bytes(const QGemvStreamParams& p, bool gated, int ns, int kb_cta, int slots) {
  return kCtrlBytes + 2 * kWarps * red_plane(gated, p.M) * 4 + (ns > 1 ? 2 * recv_floats(gated, p.M) * 4 : 0) +
         kWarps * slots * slot_bytes(p.group_shift) + kb_cta * x_block_bytes(p.M);
}

template <bool GATED, int TOK>
cudaError_t launch(const QGemvStreamParams& p, int clusters, int smem, cudaStream_t stream) {
  static bool configured[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!configured[dev]) {
    e = cudaFuncSetAttribute(qgemv4_stream_kernel<GATED, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters, p.ns, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int nattr = 0;
  if (pdl_enabled()) {
    attr[nattr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[nattr].val.programmaticStreamSerializationAllowed = 1;
    ++nattr;
  }
  if (p.ns > 1) {
    attr[nattr].id = cudaLaunchAttributeClusterDimension;
    attr[nattr].val.clusterDim.x = 1;
    attr[nattr].val.clusterDim.y = p.ns;
    attr[nattr].val.clusterDim.z = 1;
    ++nattr;
  }
  cfg.attrs = attr;
  cfg.numAttrs = nattr;
  return cudaLaunchKernelEx(&cfg, qgemv4_stream_kernel<GATED, TOK>, p);
}

}  // namespace

// Where this kernel takes a matrix, and over how many CTAs it splits K; 0: the register kernel. Turning the activations into bytes, the larger
// CTAs and their barriers cost about a microsecond, so that it takes several row tiles an SM and long rows to pay. Microseconds of one token,
// register kernel -> this one (K blocks x row tiles an SM): 57344 x 8192 gated (128 x 24) 67.5 -> 44.8, 10240 x 8192 19.3 -> 13.4, 8192 x 8192
// 11.4 -> 9.0, 28672 x 4096 gated (64 x 12) 19.7 -> 15.4, 14336 x 4096 gated (64 x 6) 10.7 -> 9.7, 8192 x 3584 (56 x 3.5) 6.6 -> 5.9, 5120 x 5120
// (80 x 2.2) 8.6 -> 6.6, 4864 x 3072 (48 x 2.1) 6.2 -> 4.8, 36864 x 2048 (32 x 16) 11.6 -> 10.5, 128256 x 2048 43 -> 29; but 4096 x 4096 (64 x 1.7)
// 4.7 / 5.2, 4736 x 5120 (80 x 2.0) 6.1 / 6.5, 12288 x 2048 (32 x 5) 6.0 / 6.1, 35520 x 1024 (16 x 15) 6.8 / 7.5.
// Two CTAs that split K: where one has no room for the activations (8192 x 28672: 35.2 -> 25.7), and where the row tiles are between one and two an
// SM and long (4096 x 11008: 10.8 -> 8.6, 2848 x 16384: 13.4 -> 9.4, 3072 x 8192: 8.0 -> 6.7; 2048 x 8192 6.4 / 6.4).
// Two tokens take more fmas: 28672 x 4096 gated 19.7 -> 17.7, 10240 x 8192 19.4 -> 15.8, 5120 x 5120 8.7 -> 7.7, 4096 x 14336 12.9 -> 11.2, 16384 x
// 4096 (64 x 7) 10.8 -> 10.6; but 14336 x 4096 gated (64 x 6) 10.7 / 11.0, 36864 x 2048 11.9 / 12.2.
static int pick_splits(const QGemvStreamParams& p, bool gated, int sms) {
  const double tiles = static_cast<double>(p.units) * (gated ? 2 : 1) / sms;
  if (tiles <= 2) return tiles >= 1.2 && p.kblocks >= 128 ? 2 : 0;
  if (smem_bytes(p, gated, 1, (p.kblocks + 1) / 2 * 2, 2) > kMaxSmem) return 2;
  if (p.kblocks >= (p.M == 1 ? 48 : 80)) return 1;
  return p.kblocks * tiles >= (p.M == 1 ? 480 : p.kblocks >= 48 ? 440 : 1000) ? 1 : 0;
}

int launch_qgemv_stream(QGemvStreamParams p, bool gated, int sm_count, cudaStream_t stream) {
  if (p.M < 1 || p.M > kQGemvStreamTokens || p.group_shift < 6 || p.group_shift > 7) return kQGemvStreamUnsupported;
  const int sms = sm_count > 0 ? sm_count : 148;
  p.units = (p.n_out + 15) / 16;
  p.ns = pick_splits(p, gated, sms);
  if (p.ns == 0) return kQGemvStreamUnsupported;
  p.kb_cta = ((p.kblocks + p.ns - 1) / p.ns + kChunk - 1) / kChunk * kChunk;          // starts on a group
  if (smem_bytes(p, gated, p.ns, p.kb_cta, 2) > kMaxSmem) return kQGemvStreamUnsupported;
  const int clusters = std::min(p.units, std::max(1, sms / p.ns));
  p.kb_warp = ((p.kb_cta + kWarps - 1) / kWarps + kChunk - 1) / kChunk * kChunk;   // a warp's slots start on a group
  p.slots = 2;
  while (p.slots < kMaxSlots && smem_bytes(p, gated, p.ns, p.kb_cta, p.slots + 1) <= kMaxSmem) ++p.slots;
  const int smem = smem_bytes(p, gated, p.ns, p.kb_cta, p.slots);
  cudaError_t e;
  if (p.M == 1) e = gated ? launch<true, 1>(p, clusters, smem, stream) : launch<false, 1>(p, clusters, smem, stream);
  else e = gated ? launch<true, 2>(p, clusters, smem, stream) : launch<false, 2>(p, clusters, smem, stream);
  eredu_count_launches(1);
  return static_cast<int>(e);
}

}  // namespace eredu
