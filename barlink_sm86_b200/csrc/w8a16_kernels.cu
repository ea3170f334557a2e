// SPDX-License-Identifier: MIT
//
// The reference's W8A8-activation decode GEMM API, kept for callers written
// against it (torch_ext/barlink_sm86/w8a16.cu:165-212, binding.cpp:434-490):
//
//   xq, xs = w8a16_quant_act(x)              per-token int8 activations, scale amax/127
//   y = w8a16_gemm(xq, xs, wq_t, sw_t, N, K, S)
//       y[m, n] = xs[m] * sum_g sw_t[g, n] * sum_{k in group g} xq[m, k] * w[n, k]
//       wq_t int8 [K/16, N, 16] (k-chunk major), sw_t fp32 [K/128, N], M <= 16
//
// The product is bl_qlin (qlin_kernels.cu): the k-chunk-major weight layout is already an operand layout
// of the tensor core (unswizzled K-major), so a k-block is one copy and int8 x int8 products
// there, with the group scales applied per k-block.  The dp4a kernel that stood here (a thread per output
// feature, loads waiting for one another) moved 1.0 TB/s of weights: four linears of a 32B layer at 8
// tokens took 596 us, now 126 us.  A k-split is summed in a fixed order (the reference adds with
// floating-point atomics), so results are reproducible run to run.
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "bl_ops.h"
#include "heap.h"
#include "launch.h"
#include "ptx.cuh"

namespace bl {

constexpr int kQThreads = 256;
constexpr int kGroup = 128;
constexpr int kMaxM = 16;

__global__ void __launch_bounds__(kQThreads) k_quant_act(const __nv_bfloat16* __restrict__ x,
                                                          int8_t* __restrict__ xq,
                                                          float* __restrict__ xs, int K) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float s_red[kQThreads / 32];
  __shared__ float s_scale;
  const __nv_bfloat16* row = x + size_t(blockIdx.x) * K;
  float amax = 0.f;
  for (int i = threadIdx.x * 8; i < K; i += blockDim.x * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + i);
    const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z),
                 d = unpack_bf16x2(v.w);
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(b.x), fabsf(b.y))));
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fmaxf(fabsf(d.x), fabsf(d.y))));
  }
  amax = warp_max(amax);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < kQThreads / 32 ? s_red[threadIdx.x] : 0.f;
    t = warp_max(t);
    if (threadIdx.x == 0) {
      s_scale = fmaxf(t / 127.f, 1e-12f);
      xs[blockIdx.x] = s_scale;
    }
  }
  __syncthreads();
  const float inv = 1.f / s_scale;
  int8_t* out = xq + size_t(blockIdx.x) * K;
  for (int i = threadIdx.x * 8; i < K; i += blockDim.x * 8) {
    const uint4 v = *reinterpret_cast<const uint4*>(row + i);
    const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y), c = unpack_bf16x2(v.z),
                 d = unpack_bf16x2(v.w);
    const float f[8] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int q = __float2int_rn(f[j] * inv);
      q = max(-127, min(127, q));
      w[j >> 2] |= (uint32_t(q) & 0xffu) << (8 * (j & 3));
    }
    *reinterpret_cast<uint2*>(out + i) = make_uint2(w[0], w[1]);
  }
}

// The same for few tokens: a row is shared by a cluster of CL blocks, one vector a thread, read once and kept; the
// largest element passes through distributed shared memory.  One block a row and two passes over it took 7.4 us for
// 8 x 27648 in a chain of linears; this takes 4.0.
constexpr int kQaThreads = 512;
template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kQaThreads)
    k_quant_act_cluster(const __nv_bfloat16* __restrict__ x, int8_t* __restrict__ xq, float* __restrict__ xs, int K) {
  pdl_launch_dependents();
  if constexpr (CL > 1) cluster_sync_all();  // the other blocks' shared memory is there
  pdl_wait();
  __shared__ float s_red[kQaThreads / 32];
  __shared__ uint32_t s_clu[CL];
  const int row = blockIdx.x / CL, lane = threadIdx.x & 31;
  const uint32_t part = CL > 1 ? cluster_ctarank() : 0;
  const int vecs = K >> 3, per = (vecs + CL - 1) / CL, c = int(part) * per + int(threadIdx.x);
  const bool in = int(threadIdx.x) < per && c < vecs;
  const uint4 v = in ? reinterpret_cast<const uint4*>(x + size_t(row) * K)[c] : make_uint4(0, 0, 0, 0);
  const float2 p0 = unpack_bf16x2(v.x), p1 = unpack_bf16x2(v.y), p2 = unpack_bf16x2(v.z), p3 = unpack_bf16x2(v.w);
  const float f[8] = {p0.x, p0.y, p1.x, p1.y, p2.x, p2.y, p3.x, p3.y};
  float amax = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(f[j]));
  amax = warp_max(amax);
  if (lane == 0) s_red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = warp_max(s_red[lane & (kQaThreads / 32 - 1)]);
  if constexpr (CL > 1) {
    if (threadIdx.x < CL) st_cluster_u32(map_to_cta(smem_u32(&s_clu[part]), threadIdx.x), __float_as_uint(amax));
    cluster_sync_all();
#pragma unroll
    for (int q = 0; q < CL; ++q) amax = fmaxf(amax, __uint_as_float(s_clu[q]));
  }
  const float scale = fmaxf(amax / 127.f, 1e-12f);
  if (threadIdx.x == 0 && part == 0) xs[row] = scale;
  const float inv = 1.f / scale;
  if (in) {
    uint32_t w[2] = {0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      int q = __float2int_rn(f[j] * inv);
      q = max(-127, min(127, q));
      w[j >> 2] |= (uint32_t(q) & 0xffu) << (8 * (j & 3));
    }
    reinterpret_cast<uint2*>(xq + size_t(row) * K)[c] = make_uint2(w[0], w[1]);
  }
  if constexpr (CL > 1) cluster_sync_all();  // no block leaves while another may still write its word
}

}  // namespace bl

using namespace bl;

extern "C" int bl_w8a16_quant_act(const void* x, int m, int k, void* xq, void* xs, void* stream,
                                  char* err, size_t errlen) {
  if (!x || !xq || !xs || m < 1 || k < 8 || (k & 7)) {
    set_err(err, errlen, "barlink: w8a16_quant_act needs K a multiple of 8");
    return -1;
  }
  if ((reinterpret_cast<uintptr_t>(x) & 15u) || (reinterpret_cast<uintptr_t>(xq) & 7u)) {
    set_err(err, errlen, "barlink: w8a16_quant_act needs rows on 16-byte boundaries and digits on 8-byte ones");
    return -1;
  }
  auto go = [&](auto kern, int blocks, int threads) {
    return launch_k(kern, dim3(m * blocks), dim3(threads), 0, static_cast<cudaStream_t>(stream),
                    static_cast<const __nv_bfloat16*>(x), static_cast<int8_t*>(xq), static_cast<float*>(xs), k);
  };
  // Blocks of a row: one vector a thread, as long as there is an SM for every block.  Not clusters of two: rows of 5120
  // elements take them longer than one block and two passes (the reference's pair on a 32B layer, 8 tokens: 120.2 us and
  // 118.2; per-channel scales, 64 tokens: 127.2 and 126.1; group scales 277 and 267).
  const int need = (k / 8 + kQaThreads - 1) / kQaThreads, cl = need <= 1 ? 1 : need <= 4 ? 4 : 8;
  cudaError_t e;
  if (need == 2 || need > 8 || m * cl > sm_count()) e = go(k_quant_act, 1, kQThreads);
  else if (cl == 1) e = go(k_quant_act_cluster<1>, 1, kQaThreads);
  else if (cl == 4) e = go(k_quant_act_cluster<4>, 4, kQaThreads);
  else e = go(k_quant_act_cluster<8>, 8, kQaThreads);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: w8a16_quant_act launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_w8a16_gemm(const void* xq, const void* xs, const void* wq_t, const void* sw_t,
                             void* out, int m, int n, int k, int splits, void* ws, void* err_flag,
                             void* stream, char* err, size_t errlen) {
  if (m < 1 || m > kMaxM) {
    set_err(err, errlen, "barlink: w8a16_gemm is the decode kernel of the reference API: 1..%d rows (got %d)",
            kMaxM, m);
    return -2;
  }
  if (k < kGroup || k % kGroup || n < 1) {
    set_err(err, errlen, "barlink: w8a16_gemm needs K a multiple of %d", kGroup);
    return -1;
  }
  if ((reinterpret_cast<uintptr_t>(xq) | reinterpret_cast<uintptr_t>(wq_t)) & 15u) {
    set_err(err, errlen, "barlink: w8a16_gemm needs xq and wq_t on 16-byte boundaries");
    return -1;
  }
  const int G = k / kGroup;
  if (splits < 1) splits = 1;
  if (splits > G) splits = G;
  const int gper = (G + splits - 1) / splits;
  splits = (G + gper - 1) / gper;
  if (splits > 1 && !ws) {
    set_err(err, errlen, "barlink: w8a16_gemm with a k-split needs a workspace of S*M*N floats");
    return -1;
  }
  // bl_slab_finish reads 16-byte vectors
  if ((n & 7) || (reinterpret_cast<uintptr_t>(ws) & 15u)) splits = 1;
  blQlinArgs a;
  memset(&a, 0, sizeof(a));
  a.w = wq_t;
  a.src = 1;
  a.n = n;
  a.k = k;
  a.xq = xq;
  a.xs = xs;
  a.m = m;
  a.digits = 1;
  a.scale_kind = BL_QSCALE_F32_GN;
  a.scale = sw_t;
  a.group_k = kGroup;
  a.splits = splits;
  if (splits > 1) a.slabs = ws;
  a.err_flag = err_flag;
  a.out = out;
  a.ldo = n;
  if (bl_qlin(&a, stream, err, errlen) != 0) return -1;
  if (splits > 1) {
    blSlabFinishArgs f;
    memset(&f, 0, sizeof(f));
    f.slabs = ws;
    f.nsplit = splits; f.m = m; f.n = f.pitch = n;
    f.out = out;
    f.ldo = n;
    return bl_slab_finish(&f, stream, err, errlen);
  }
  return 0;
}
