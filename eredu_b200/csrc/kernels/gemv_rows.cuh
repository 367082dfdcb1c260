// Y = X W^T for one or two tokens, included by gemm_tcgen05.cu (same parameters and epilogue as gemm_wt_kernel).
//
// A decode step of one sequence is a chain of short kernels, and what bounds the small ones is not the bytes but everything around
// them: tensor memory, barriers, the ring's first fill, the exchange between the CTAs of a K split. With so few tokens the tensor
// cores are not needed - a weight is used once or twice - so this kernel has none of it: a CTA owns 16 rows of W and all of K, a
// thread takes every 128th 16-byte piece of eight of them, in registers, and two rounds of sums (lanes, then warps) end it. Two
// pieces of every row are on their way before the dependency wait: 64 KB per CTA, which for matrices up to 19 MB is all of them, so
// that the kernel before this one hides them.
#pragma once

namespace eredu {

constexpr int kRowsThreads = 256;

__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

constexpr int kRowsPerThread = 8;                    // four warps take these rows, the other four the next
constexpr int kRowsOut = 2 * kRowsPerThread;         // output columns of a CTA

// Whole pieces of 8 along K, whole CTAs along N; M <= MT. With sums of squares the CTAs of 128 output columns are a cluster.
template <int MT>
__global__ void __launch_bounds__(kRowsThreads, 2) gemv_rows_kernel(GemmParams p, const __nv_bfloat16* x, const __nv_bfloat16* w, int ldx, int ldw) {
  constexpr int R = kRowsPerThread, V = R * MT, STEP = kRowsThreads / 2, WARPS = STEP / 32;
  __shared__ float s_red[2][WARPS][V];
  __shared__ float s_scale[MT];
  __shared__ float s_sq[MT];            // this CTA's columns
  __shared__ float s_parts[8][MT];      // cluster rank 0: of every CTA
  pdl_launch_early();
  trace_mark(kTraceGemm, kTraceStart);
  if (p.ssq_out != nullptr) cluster_arrive_relaxed();     // waited for in front of the store into CTA 0
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, side = warp / WARPS;
  const int n0 = blockIdx.x * kRowsOut;
  const int pieces = p.K >> 3;
  int at = threadIdx.x % STEP;          // piece of a row

  const int n_in = min(n0, p.N - kRowsOut);          // a CTA that only fills up its cluster reads the last columns and stores nothing
  const uint32_t pitch = static_cast<uint32_t>(ldw) * 2u;
  const uint8_t* first = reinterpret_cast<const uint8_t*>(w) + static_cast<size_t>(n_in + side * R) * pitch;
  // two batches of pieces per row: one is multiplied while the other is on its way
  uint4 wa[R], wb[R], xa[MT], xb[MT];
  auto load_w = [&](uint4 (&v)[R], int piece) {
    const uint8_t* q = first + static_cast<size_t>(piece) * 16;
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = piece < pieces ? ld_stream(q + r * static_cast<size_t>(pitch)) : make_uint4(0u, 0u, 0u, 0u);
  };
  auto load_x = [&](uint4 (&v)[MT], int piece) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
      v[m] = piece < pieces && m < p.M ? *reinterpret_cast<const uint4*>(x + static_cast<size_t>(m) * ldx + piece * 8) : make_uint4(0u, 0u, 0u, 0u);
  };
  load_w(wa, at);
  load_w(wb, at + STEP);

  pdl_wait();
  trace_mark(kTraceGemm, kTraceAfterWait);
  pdl_launch_dependents();
  load_x(xa, at);
  load_x(xb, at + STEP);
  if (p.ssq_in != nullptr && warp < MT) {
    float t = 0.f;
    if (warp < p.M)
      for (int j = lane; j < p.ssq_parts; j += 32) t += p.ssq_in[static_cast<size_t>(warp) * p.ssq_parts + j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_scale[warp] = rsqrtf(t * p.norm_inv_dim + p.norm_eps);
  }

  float v[V];
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = 0.f;
  auto multiply = [&](const uint4 (&wv)[R], const uint4 (&xv)[MT]) {
    float xf[MT][8];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint32_t u[4] = {xv[m].x, xv[m].y, xv[m].z, xv[m].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        xf[m][2 * j] = bf16_lo(u[j]);
        xf[m][2 * j + 1] = bf16_hi(u[j]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t u[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = bf16_lo(u[j]), b = bf16_hi(u[j]);
#pragma unroll
        for (int m = 0; m < MT; ++m) v[r * MT + m] = fmaf(b, xf[m][2 * j + 1], fmaf(a, xf[m][2 * j], v[r * MT + m]));
      }
    }
  };
#pragma unroll 1
  for (int base = 0; base < pieces; base += 2 * STEP) {
    multiply(wa, xa);
    at += 2 * STEP;
    load_w(wa, at);
    load_x(xa, at);
    multiply(wb, xb);
    load_w(wb, at + STEP);
    load_x(xb, at + STEP);
  }

  // lanes: every exchange halves the sums a lane carries, until it has one; then lanes that have the same one add up
  int idx = 0;
#pragma unroll
  for (int n = V / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
    idx += up ? n : 0;
  }
#pragma unroll
  for (int o = 16 / V; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  if ((lane & (32 / V - 1)) == 0) s_red[side][warp % WARPS][idx] = v[0];
  __syncthreads();

  // warps: thread m * kOut + c finishes output column c of token m
  constexpr int kItems = kRowsOut * MT;                // at most a warp
  if (warp == 0) {
    const int m = lane / kRowsOut, c = lane % kRowsOut, n = n0 + c;
    float stored = 0.f;
    if (lane < kItems && m < p.M && n < p.N) {
      float g = 0.f;
#pragma unroll
      for (int k = 0; k < WARPS; ++k) g += s_red[c / R][k][c % R * MT + m];
      const float sc = p.ssq_in != nullptr ? s_scale[m] : 1.f;
      stored = epilogue_store<false>(p, g, 0.f, m, n, sc, p.residual != nullptr ? residual_at(p, m, n) : 0.f);
    }
    if (p.ssq_out != nullptr) {
      float sq = stored * stored;
#pragma unroll
      for (int o = kRowsOut / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane < kItems && c == 0) s_sq[m] = sq;
      __syncwarp();
    }
  }
  if (p.ssq_out != nullptr) {
    // the 128 columns whose sum of squares is one number belong to the cluster's eight CTAs
    uint32_t rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    __syncwarp();
    cluster_wait_acquire();                               // CTA 0 has started: its shared memory may be written
    if (threadIdx.x < MT)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_shared(smem_u32(&s_parts[0][0]) + (rank * MT + threadIdx.x) * 4u, 0u)),
                   "f"(s_sq[threadIdx.x])
                   : "memory");
    __syncwarp();
    cluster_arrive_release();
    cluster_wait_acquire();
    if (rank == 0 && threadIdx.x < p.M) {
      float t = 0.f;
      for (int r = 0; r < 128 / kRowsOut; ++r) t += s_parts[r][threadIdx.x];
      p.ssq_out[static_cast<size_t>(threadIdx.x) * ((p.N + 127) / 128) + n0 / 128] = t;
    }
  }
  trace_mark(kTraceGemm, kTraceEnd);
}

template <int MT>
static cudaError_t launch_rows(const GemmParams& p, const void* x, const void* w, int ldx, int ldw, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  const int ctas = (p.N + kRowsOut - 1) / kRowsOut;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  constexpr int kCluster = 128 / kRowsOut;
  cfg.gridDim = dim3(p.ssq_out != nullptr ? (ctas + kCluster - 1) / kCluster * kCluster : ctas);
  if (p.ssq_out != nullptr) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = kCluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.blockDim = dim3(kRowsThreads);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, gemv_rows_kernel<MT>, p, static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), ldx, ldw);
}

}  // namespace eredu
