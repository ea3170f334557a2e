// SPDX-License-Identifier: MIT
//
// Weight-only int4 linears for decode (1..16 tokens) on GPTQ-v1 tensors, the
// format of the reference's Triton GEMV (demos/qwen_tp/int4linear.py:5-12,
// kernel :22-44):
//
//   qweight int32 [K/8, N]   8 consecutive k per word, nibble j = k % 8
//   scales  fp16  [G, N]     one scale per (group of `group` inputs, output)
//   qzeros  int32 [G, N/8]   8 consecutive outputs per word
//   w[n, k] = (nibble - zero) * scale
//
// Groups of 128 on aligned tensors: k_w4a16_mma (below).  Other groups: k_w4a16_gemv, where
// one thread owns four adjacent outputs and reads one 16-byte vector per
// 8 inputs, so a warp reads 512 contiguous bytes; nibbles become fp16 with
// the 0x6400 exponent trick (1024 + nibble, exact), the zero point is
// subtracted in fp16 (exact) and products accumulate in fp32 per group, then
// per-group sums are scaled.  A split over k is reduced in a fixed order
// (the reference adds with floating-point atomics), so results
// repeat run to run.  More than 16 tokens: groups of 128 go to the digit kernel (qlin_kernels.cu), others
// widen the weight to bf16 once (k_w4_dequant) for a bf16 product.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "bl_ops.h"
#include "heap.h"
#include "launch.h"
#include "ptx.cuh"

namespace bl {

constexpr int kW4Threads = 128;
constexpr int kW4MaxM = 16;
constexpr int kW4MaxGroup = 128;

template <int MT>
__global__ void __launch_bounds__(kW4Threads) k_w4a16_gemv(const __nv_bfloat16* __restrict__ x,
                                                           const uint32_t* __restrict__ qw,
                                                           const __half* __restrict__ sc,
                                                           const uint32_t* __restrict__ qz,
                                                           __nv_bfloat16* __restrict__ out,
                                                           float* __restrict__ ws, int M, int N, int K,
                                                           int group, int gper) {
  // the kernels behind this one start when it ends: resident early they only took its slots (7B shape, one
  // sequence, MLP in int4: 3.22 ms a step with an early start of this kernel's dependents,
  // 2.79 ms without)
  pdl_wait();
  __shared__ float s_x[MT][kW4MaxGroup];
  const int n = (blockIdx.x * kW4Threads + threadIdx.x) * 4;
  const int G = K / group;
  const int g0 = blockIdx.y * gper, g1 = min(G, g0 + gper);
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[m][c] = 0.f;
  for (int g = g0; g < g1; ++g) {
    __syncthreads();
    for (int t = threadIdx.x; t < MT * group; t += kW4Threads) {
      const int m = t / group, k = t - m * group;
      s_x[m][k] = m < M ? __bfloat162float(x[size_t(m) * K + g * group + k]) : 0.f;
    }
    __syncthreads();
    if (n < N) {
      const uint2 sraw = *reinterpret_cast<const uint2*>(sc + size_t(g) * N + n);
      const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sraw.x));
      const float2 s23 = __half22float2(*reinterpret_cast<const __half2*>(&sraw.y));
      const float scl[4] = {s01.x, s01.y, s23.x, s23.y};
      const uint32_t zw = qz[size_t(g) * (N / 8) + (n >> 3)] >> ((n & 7) * 4);
      float part[MT][4];
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) part[m][c] = 0.f;
      const uint32_t* wp = qw + (size_t(g) * (group / 8)) * N + n;
#pragma unroll 4
      for (int kk = 0; kk < group / 8; ++kk) {
        const uint4 w4 = __ldg(reinterpret_cast<const uint4*>(wp + size_t(kk) * N));
        const uint32_t wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // 1024 + zero as fp16 in both halves
          const uint32_t zbits = 0x6400u | ((zw >> (4 * c)) & 15u);
          const __half2 z2 = __halves2half2(__ushort_as_half(zbits), __ushort_as_half(zbits));
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            // nibbles j (low half) and j + 4 (high half)
            const uint32_t bits = ((wv[c] >> (4 * j)) & 0x000F000Fu) | 0x64006400u;
            const float2 v = __half22float2(__hsub2(*reinterpret_cast<const __half2*>(&bits), z2));
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              part[m][c] = fmaf(s_x[m][kk * 8 + j], v.x, part[m][c]);
              part[m][c] = fmaf(s_x[m][kk * 8 + j + 4], v.y, part[m][c]);
            }
          }
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][c] = fmaf(part[m][c], scl[c], acc[m][c]);
    }
  }
  if (n >= N) return;
  if (gridDim.y == 1) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (m < M)
        *reinterpret_cast<uint2*>(out + size_t(m) * N + n) =
            make_uint2(pack_bf16x2(acc[m][0], acc[m][1]), pack_bf16x2(acc[m][2], acc[m][3]));
  } else {
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (m < M)
        *reinterpret_cast<float4*>(ws + (size_t(blockIdx.y) * M + m) * N + n) =
            make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
  }
}

__global__ void k_w4_reduce(const float* __restrict__ ws, __nv_bfloat16* __restrict__ out, int MN, int S) {
  pdl_wait();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= MN) return;
  float a = 0.f;
  for (int s = 0; s < S; ++s) a += ws[size_t(s) * MN + t];
  out[t] = __float2bfloat16(a);
}

// ---------------------------------------------------------------------------
// 1..16 tokens, groups of 128: mma.sync on weights expanded in registers
// ---------------------------------------------------------------------------
// The packed weight stream (37888 x 3584: 68 MB) takes 10.4 us, so a weight may cost little more than
// one instruction, and that is what bounds the kernel now (15.6 us with every load taken out; the logic pipe takes half an
// instruction a cycle, and multiplications in place of shifts were slower, 24.7 us).  8 of them are a word, 3 shifts and 4 three-input logic instructions make four bf16 pairs of
// 128 + nibble, 4 subtractions take 128 + zero off (both exact), and one mma.sync m16n8k16 multiplies 256 weights with
// 8 tokens, sums in fp32.  A warp owns 32 outputs: a lane reads 16 bytes (four outputs, eight inputs), eight lanes a
// 128-byte line, the four lanes of a quad consecutive word rows.  The order of the inputs inside a product is free, so
// a lane's words serve its own columns as they are, nibble pair (j, j + 4) by pair, and the activations are permuted
// alike.  A word's successor one group on is requested as soon as the word is used, 2 KB a warp and 48 KB an SM
// in flight.  The warps of a block take consecutive groups and are summed in order through shared memory; k-splits
// over blocks leave fp32 slabs.  (A ring in shared memory three groups deep: 26 us.)
// 37888 x 3584, us at 1 / 4 / 8 / 16 tokens: 19.7 / 19.7 / 19.7 / 28; 3584 x 18944 into slabs 12.4 / 13 / 13 / 16.6.  Before:
// an fp32 GEMV of 3.4 instructions a weight and token, words requested between two barriers of every group, up to four
// tokens, and digits on tcgen05 with words expanded in shared memory above: 28 / 51 / 40 / 40, and 21.5 / 31 / 28 / 33.
constexpr int kW4Strip = 32;
constexpr int kW4Threads1 = 768, kW4Threads2 = 512;  // threads that an SM shall hold, up to 8 tokens and above

__device__ __forceinline__ void w4_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the same onto zeros
__device__ __forceinline__ void w4_mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// nibbles j and j + 4 of a word, minus the zero point (z: 128 + zero in both halves), as a bf16 pair
// (one three-input logic instruction: written in C++ it became two)
__device__ __forceinline__ uint32_t w4_pair(uint32_t w, int j, uint32_t z) {
  uint32_t bits;  // 128 + nibble: ((w >> 4 j) & mask) | exponent
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(bits) : "r"(w >> (4 * j)), "n"(0x000F000F), "r"(0x43004300));
  const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&bits), *reinterpret_cast<const __nv_bfloat162*>(&z));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// T8: tokens in eights.  grid (strips, splits); out (bf16 [M][N], or [M][N / 2] with silu) or slabs (fp32
// [split][M][N]).
template <int T8>
__global__ void __launch_bounds__(T8 == 1 ? kW4Threads1 : kW4Threads2, 1)
    k_w4a16_mma(const __nv_bfloat16* __restrict__ x, const uint32_t* __restrict__ qw, const __half* __restrict__ sc,
                const uint32_t* __restrict__ qz, __nv_bfloat16* __restrict__ out, float* __restrict__ slabs, int M, int N,
                int K, int gper, int silu) {
  extern __shared__ float s_sum[];  // [warp][token][kW4Strip]
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int G = K >> 7;
  const int c0 = blockIdx.y * gper, c1 = min(G, c0 + gper);
  const int g0 = c0 + (c1 - c0) * warp / warps, g1 = c0 + (c1 - c0) * (warp + 1) / warps;
  // (N is a multiple of 8: the four outputs of a lane are all inside or all outside)
  int n = blockIdx.x * kW4Strip + 4 * g;
  if (n >= N) n = 0;
  // word row of this lane in step s of group gi: 16 gi + 4 s + t
  const uint32_t* wp = qw + size_t(16 * g0 + t) * N + n;
  const size_t step = size_t(4) * N;
  // before the kernels ahead have finished (they may write the weights) the first words are only asked into L2
  if (g == 0)
    for (int s = 0; s < 4 * min(g1 - g0, 2); ++s) asm volatile("prefetch.global.L2 [%0];" ::"l"(wp + s * step));
  pdl_wait();

  uint4 w[4], xv[T8];
  uint2 sraw = make_uint2(0, 0);
  uint32_t zraw = 0;
  const __nv_bfloat16* xp = x + size_t(g) * K + 128 * g0 + 8 * t;
  const __half* scp = sc + size_t(g0) * N + n;
  const uint32_t* zp = qz + size_t(g0) * (N >> 3) + (n >> 3);
  auto load_x = [&](int off) {
#pragma unroll
    for (int q = 0; q < T8; ++q)
      if (8 * q + g < M) xv[q] = __ldg(reinterpret_cast<const uint4*>(xp + size_t(8 * q) * K + off));
  };
#pragma unroll
  for (int q = 0; q < T8; ++q) xv[q] = make_uint4(0, 0, 0, 0);  // stays so for tokens beyond M
  float acc[2][T8][4];
#pragma unroll
  for (int i = 0; i < 2 * T8 * 4; ++i) (&acc[0][0][0])[i] = 0.f;
  if (g0 < g1) {
    sraw = __ldg(reinterpret_cast<const uint2*>(scp));
    zraw = __ldg(zp);
#pragma unroll
    for (int s = 0; s < 4; ++s) w[s] = __ldcs(reinterpret_cast<const uint4*>(wp + s * step));
    load_x(0);
  }
#pragma unroll 1
  for (int gi = g0; gi < g1; ++gi) {
    const bool more = gi + 1 < g1;
    wp += 4 * step;
    scp += N;
    zp += N >> 3;
    uint32_t z[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) z[c] = 0x43004300u + ((zraw >> (4 * ((n & 7) + c))) & 15u) * 0x10001u;
    const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sraw.x));
    const float2 s23 = __half22float2(*reinterpret_cast<const __half2*>(&sraw.y));
    const float scl[4] = {s01.x, s01.y, s23.x, s23.y};
    if (more) {
      sraw = __ldg(reinterpret_cast<const uint2*>(scp));
      zraw = __ldg(zp);
    }
    float d[2][T8][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      // activations 8 t .. 8 t + 7 in the order of the nibble pairs: (0,4) (1,5) (2,6) (3,7)
      uint32_t b[T8][4];
#pragma unroll
      for (int q = 0; q < T8; ++q) {
        b[q][0] = __byte_perm(xv[q].x, xv[q].z, 0x5410);
        b[q][1] = __byte_perm(xv[q].x, xv[q].z, 0x7632);
        b[q][2] = __byte_perm(xv[q].y, xv[q].w, 0x5410);
        b[q][3] = __byte_perm(xv[q].y, xv[q].w, 0x7632);
      }
      if (s < 3 || more) load_x(32 * (s + 1));
      const uint32_t wc[4] = {w[s].x, w[s].y, w[s].z, w[s].w};
#pragma unroll
      for (int r = 0; r < 2; ++r)  // rows g and g + 8 of the product: outputs n + 2 r and n + 2 r + 1
#pragma unroll
        for (int jj = 0; jj < 4; jj += 2) {
          const uint32_t a[4] = {w4_pair(wc[2 * r], jj, z[2 * r]), w4_pair(wc[2 * r + 1], jj, z[2 * r + 1]),
                                 w4_pair(wc[2 * r], jj + 1, z[2 * r]), w4_pair(wc[2 * r + 1], jj + 1, z[2 * r + 1])};
#pragma unroll
          for (int q = 0; q < T8; ++q)
            if (s == 0 && jj == 0) w4_mma0(d[r][q], a, b[q][jj], b[q][jj + 1]);
            else w4_mma(d[r][q], a, b[q][jj], b[q][jj + 1]);
        }
      if (more) w[s] = __ldcs(reinterpret_cast<const uint4*>(wp + s * step));
    }
    xp += 128;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q < T8; ++q)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][q][e] = fmaf(d[r][q][e], scl[2 * r + (e >> 1)], acc[r][q][e]);
  }
  // element e of a product: output n + 2 r + (e >> 1), token 8 q + 2 t + (e & 1)
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int q = 0; q < T8; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int m = 8 * q + 2 * t + (e & 1);
        if (m < M) s_sum[(warp * M + m) * kW4Strip + 4 * g + 2 * r + (e >> 1)] = acc[r][q][e];
      }
  __syncthreads();
  // two adjacent outputs a thread
  for (int i = threadIdx.x; i < M * (kW4Strip / 2); i += blockDim.x) {
    const int m = i / (kW4Strip / 2), c = 2 * (i % (kW4Strip / 2)), col = blockIdx.x * kW4Strip + c;
    if (col >= N) continue;
    float a = 0.f, b = 0.f;
    for (int v = 0; v < warps; ++v) {
      const float2 f = *reinterpret_cast<const float2*>(s_sum + (v * M + m) * kW4Strip + c);
      a += f.x;
      b += f.y;
    }
    if (slabs)
      __stcg(reinterpret_cast<float2*>(slabs + (size_t(blockIdx.y) * M + m) * N + col), make_float2(a, b));
    else if (silu)
      out[size_t(m) * (N >> 1) + (col >> 1)] = __float2bfloat16(a / (1.f + __expf(-a)) * b);
    else
      *reinterpret_cast<uint32_t*>(out + size_t(m) * N + col) = pack_bf16x2(a, b);
  }
}

// How a product of m tokens is dealt out: warps of a block (they share an output strip) and k-splits.  What counts is
// that the blocks fill the SMs in whole laps (37888 x 3584: 1184 strips, blocks of 3 warps, 8 an SM: one lap of 10
// groups a warp; of 4 warps it would be two of 7).
struct W4Plan {
  int warps, splits, gper;
};
static W4Plan w4_plan(int m, int n, int k, int splits, bool want_slabs) {
  const int G = k / 128, strips = (n + kW4Strip - 1) / kW4Strip, sms = sm_count();
  const int per_sm = (m <= 8 ? kW4Threads1 : kW4Threads2) / 32;  // warps that an SM holds by their registers
  const int s_lo = splits > 0 ? splits : 1, s_hi = splits > 0 ? splits : (G < 16 ? G : 16);
  W4Plan best{2, 1, G};
  int cost = 1 << 30;
  for (int s = s_lo; s <= s_hi; ++s) {
    const int gper = (G + s - 1) / s, real = (G + gper - 1) / gper;
    if (real != s && splits <= 0) continue;
    // hundredths of a group of a warp (1 us when the SM is full): the slabs and their reader; the ramp of a lap, the sums
    const int slabs = real > 1 ? (want_slabs ? 30 : 250) + 10 * real : 0;
    for (int warps : {2, 3, 4, 6, 8, 12, 16}) {
      if (warps > per_sm) break;
      const int slots = sms * (per_sm / warps), laps = (strips * real + slots - 1) / slots;
      const int c = laps * (100 * ((gper + warps - 1) / warps) + 150) + 5 * warps + slabs;
      if (c < cost) {
        cost = c;
        best = W4Plan{warps, real, gper};
      }
    }
  }
  return best;
}

// w [N, K] bf16 from the packed tensors; one thread per (8 k, 1 n) word
__global__ void k_w4_dequant(const uint32_t* __restrict__ qw, const __half* __restrict__ sc,
                             const uint32_t* __restrict__ qz, __nv_bfloat16* __restrict__ w, int N, int K,
                             int group) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= size_t(K / 8) * N) return;
  const int kw = int(t / N), n = int(t % N);
  const int g = kw * 8 / group;
  const float s = __half2float(sc[size_t(g) * N + n]);
  const int z = int((qz[size_t(g) * (N / 8) + (n >> 3)] >> ((n & 7) * 4)) & 15u);
  const uint32_t v = qw[t];
  float f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = float(int((v >> (4 * j)) & 15u) - z) * s;
  *reinterpret_cast<uint4*>(w + size_t(n) * K + kw * 8) =
      make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                 pack_bf16x2(f[6], f[7]));
}

}  // namespace bl

using namespace bl;

static int w4_check(int n, int k, int group, char* err, size_t errlen) {
  if (group < 8 || group > kW4MaxGroup || (group & 7) || k < group || k % group || n < 8 || (n & 7)) {
    set_err(err, errlen,
            "barlink: w4a16 needs group in {8..%d, multiple of 8}, K a multiple of the group and N a multiple of 8 "
            "(got N %d, K %d, group %d)", kW4MaxGroup, n, k, group);
    return -1;
  }
  return 0;
}

extern "C" int bl_w4a16_gemv(const void* x, const void* qweight, const void* scales, const void* qzeros,
                             void* out, int m, int n, int k, int group, int splits, void* ws,
                             size_t ws_bytes, void* stream, char* err, size_t errlen) {
  if (m < 1 || m > kW4MaxM) {
    set_err(err, errlen, "barlink: w4a16_gemv is the decode kernel: 1..%d rows (got %d)", kW4MaxM, m);
    return -2;
  }
  if (w4_check(n, k, group, err, errlen)) return -1;
  if ((reinterpret_cast<uintptr_t>(qweight) | reinterpret_cast<uintptr_t>(ws)) & 15u ||
      (reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(out)) & 7u) {
    set_err(err, errlen, "barlink: w4a16_gemv needs words and workspace on 16-byte boundaries, scales and output on 8-byte ones");
    return -1;
  }
  const int G = k / group;
  const int nblocks = (n / 4 + kW4Threads - 1) / kW4Threads;
  if (splits <= 0) {
    // enough blocks for every SM a few times over, every split at least two groups
    splits = (148 * 8 + nblocks - 1) / nblocks;
    if (splits > G / 2) splits = G / 2;
  }
  if (splits < 1) splits = 1;
  if (splits > G) splits = G;
  const int gper = (G + splits - 1) / splits;
  splits = (G + gper - 1) / gper;
  if (splits > 1 && (!ws || ws_bytes < size_t(splits) * m * n * sizeof(float))) {
    splits = 1;
  }
  const int gper2 = splits == 1 ? G : gper;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid(nblocks, splits);
  cudaError_t e;
#define BL_W4(MT)                                                                                      \
  e = launch_k(k_w4a16_gemv<MT>, grid, dim3(kW4Threads), 0, st, static_cast<const __nv_bfloat16*>(x),  \
               static_cast<const uint32_t*>(qweight), static_cast<const __half*>(scales),              \
               static_cast<const uint32_t*>(qzeros), static_cast<__nv_bfloat16*>(out),                 \
               static_cast<float*>(ws), m, n, k, group, gper2)
  if (m <= 1) BL_W4(1);
  else if (m <= 2) BL_W4(2);
  else if (m <= 4) BL_W4(4);
  else if (m <= 8) BL_W4(8);
  else BL_W4(16);
#undef BL_W4
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess && splits > 1) {
    e = launch_k(k_w4_reduce, dim3((m * n + 255) / 256), dim3(256), 0, st, static_cast<const float*>(ws),
                 static_cast<__nv_bfloat16*>(out), m * n, splits);
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: w4a16_gemv launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_w4a16_mma_splits(int m, int n, int k, int splits, int want_slabs) {
  if (splits > k / 128) splits = k / 128;
  return w4_plan(m, n, k, splits, want_slabs != 0).splits;
}

extern "C" int bl_w4a16_mma(const void* x, const void* qweight, const void* scales, const void* qzeros, void* out, int m,
                            int n, int k, int silu, int splits, void* slabs, void* stream, char* err, size_t errlen) {
  if (m < 1 || m > kW4MaxM) {
    set_err(err, errlen, "barlink: w4a16_mma is a decode kernel: 1..%d rows (got %d)", kW4MaxM, m);
    return -2;
  }
  if (w4_check(n, k, 128, err, errlen)) return -1;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(qweight)) & 15u ||
      reinterpret_cast<uintptr_t>(scales) & 7u || reinterpret_cast<uintptr_t>(slabs) & 15u) {
    set_err(err, errlen, "barlink: w4a16_mma needs activations, words and slabs on 16-byte boundaries and scales on 8-byte ones");
    return -1;
  }
  const int G = k / 128, gper = splits > 0 ? (G + splits - 1) / splits : 0;
  if (splits < 1 || (G + gper - 1) / gper != splits || (splits > 1 && !slabs) || (!slabs && !out) || (silu && slabs)) {
    set_err(err, errlen, "barlink: w4a16_mma: %d k-splits of %d groups (every split needs one, and plain slabs to go to)", splits, G);
    return -1;
  }
  const W4Plan p = w4_plan(m, n, k, splits, slabs != nullptr);
  const dim3 grid((n + kW4Strip - 1) / kW4Strip, splits), block(p.warps * 32);
  const size_t smem = size_t(p.warps) * m * kW4Strip * sizeof(float);
  auto go = [&](auto kern) {
    return launch_k(kern, grid, block, smem, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x),
                    static_cast<const uint32_t*>(qweight), static_cast<const __half*>(scales),
                    static_cast<const uint32_t*>(qzeros), static_cast<__nv_bfloat16*>(out), static_cast<float*>(slabs), m, n,
                    k, p.gper, silu);
  };
  cudaError_t e = m <= 8 ? go(k_w4a16_mma<1>) : go(k_w4a16_mma<2>);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: w4a16_mma launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_w4_dequant(const void* qweight, const void* scales, const void* qzeros, void* w, int n,
                             int k, int group, void* stream, char* err, size_t errlen) {
  if (w4_check(n, k, group, err, errlen)) return -1;
  const size_t total = size_t(k / 8) * n;
  cudaError_t e = launch_k(k_w4_dequant, dim3(unsigned((total + 255) / 256)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), static_cast<const uint32_t*>(qweight),
                           static_cast<const __half*>(scales), static_cast<const uint32_t*>(qzeros),
                           static_cast<__nv_bfloat16*>(w), n, k, group);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: w4 dequant launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}
