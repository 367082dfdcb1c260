// Launcher of the persistent 4-bit decode kernel (qgemv_stream.cu), called by eredu_qgemv4. Returns a cudaError_t, or
// kQGemvStreamUnsupported where the register kernel (qgemv_mma.cu) is the faster one or the activations of a CTA do not fit in its shared memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace eredu {

constexpr int kQGemvStreamUnsupported = -7778;
constexpr int kQGemvStreamTokens = 2;

struct QGemvStreamParams {
  const __nv_bfloat16* x;
  const uint8_t* wq;    // tiles [ceil(N/16)][K/64][16 rows][32 bytes], nibble order (n0,n2,n4,n6,n1,n3,n5,n7) in each u32
  const uint32_t* dq;   // tiles [ceil(N/16)][K/group][16 rows]: bf16 scale | bf16 bias << 16
  void* y;
  const __nv_bfloat16* residual;
  const __nv_bfloat16* bias;
  int M, n_out;
  int ldx, ldy, ldr;
  int group_shift;      // 6 or 7
  int kblocks;
  int out_fp32;
  float limit;          // gated: clamp (0 = off): gate <= limit, |up| <= limit
  int* status;
  // set by the launcher
  int units;            // tiles of 16 output rows
  int kb_cta, kb_warp;  // K blocks of a CTA of the cluster, and of a warp
  int ns;               // CTAs of a cluster, which split K: one or two
  int slots;            // of a warp's ring
};

int launch_qgemv_stream(QGemvStreamParams p, bool gated, int sm_count, cudaStream_t stream);

}  // namespace eredu
