// SPDX-License-Identifier: MIT
//
// Decode linears (1..128 tokens) on quantised weights:
//   y[t, n] = xs[t] * sum_g s[n, g] * sum_{k in g} q[n, k] * X[t, k]
// on tcgen05.mma kind::i8, int8 weights against int8 digits of the activations.
//
// What bounds a decode linear is the weight stream from HBM, so nothing but that stream should cost
// time.  Widening int8 weights to bf16 on the CUDA cores did: 11 instructions per four weights held
// the kernel to 2.0-2.7 TB/s.  Here the activations are taken apart instead.  A token's bf16 row is
// scaled by a power of two so that its largest element is just below 1 and written as three base-256
// digits (k_quant_digits): a fixed-point number of 23 bits below that element, so every element down to
// 2^-15 of the largest is represented exactly and the rest to within 2^-24 of the largest.  In rows where
// that would be coarse -- more than half of the nonzero elements below 2^-13 of the scale, or an infinity -- the
// scale follows the median instead (2^12 above it), and the few elements beyond it are left out of the digits
// and added in fp32 by the epilogue (outlier_sum).  What a digit drops is thus at most 2^-24 of the largest
// and 2^-11 of the median element, whichever weights meet the outliers.  The weights go from HBM to the tensor
// core as they are, the three digit planes of all tokens are the N dimension of one MMA, sums are exact int32,
// and the epilogue puts (d0 + d1 / 2^8 + d2 / 2^16) * xs[t] together.  With activations that the caller quantised
// to int8 (one digit) the same kernel runs with a third of the N.
//
// Weight forms (SRC):
//   kRows    int8 [n][k], TMA tiles of 128 rows x 128 bytes in the 128-byte swizzle
//   kChunks  int8 [k/16][n][16] (the reference's layout, torch_ext/barlink_sm86/w8a16.cu:94-117): a
//            16-byte chunk of 128 rows is 2 KiB contiguous and already the tensor core's unswizzled
//            K-major layout, so a k-block is a plain box of eight of them
//   kNibbles int4 GPTQ-v1 (int32 [k/8][n], 8 k per word): four warps turn a raw 8 KiB tile into the
//            layout of kChunks, seven instructions per eight weights, zero point subtracted; nibbles
//            come out in the order 0 2 4 6 1 3 5 7 of each eight and k_quant_digits writes the
//            digits in that order
// Scales (SC): per output channel, applied by the epilogue; or per group of 128 (a k-block), where
// every k-block gets a TMEM accumulator of its own and the epilogue warps add acc * scale in fp32.
//
// The products of a k-block take the tensor core some 50 cycles; what a k-block costs is the instructions
// around them, in the one warp that issues them and in the one that requests the tiles.  So that warp runs
// converged with its operands in uniform registers and asks for the next stage before it issues this one's
// products (55296 x 5120, one token: 49 -> 48 us with per-row scales, 64.5 -> 54 us with group-128 scales and
// int8 activations), and a k-block of the chunk layout is one box instead of eight bulk copies (79 -> 49 us).
//
// A k-split writes fp32 slabs [split][token][n]; the consumer of the linear sums them as it reads
// (the norm, RoPE and attention kernels do), or k_slab_finish does with bias / SiLU*mul.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>
#include <string.h>

#include "bl_ops.h"
#include "heap.h"
#include "launch.h"
#include "ptx.cuh"

namespace bl {

enum { kRows = 0, kChunks = 1, kNibbles = 2 };

constexpr int kQRows = 128;      // weight rows per tile
constexpr int kQK = 128;         // weights of a row per k-block
constexpr int kQTileA = kQRows * kQK;
constexpr int kDigChunks = 128;  // marks of a token: which 256 of its activations have outliers

struct QlinShape {
  int n, m, k;
  int tiles_a, tiles_b, kblocks, splits;
  const uint32_t* zeros;         // kNibbles: int32 [groups][n/8]
  const float* xs;               // per token
  const __nv_bfloat16* x;        // three digits: the activations themselves, for rows with outliers
  int ldx;
  const void* w;
  int scale_kind;                // see blQlinArgs
  const void* scale;
  const __nv_bfloat16* row_scale;
  int groups, gk;                // scale groups of a row, k-blocks per group
  const __nv_bfloat16* bias;
  __nv_bfloat16* out;
  int ldo, silu;
  float* slabs;                  // non-null: fp32 output [split][token][n]
  uint32_t* err;
};

template <int SRC, int ND, int TB, bool GROUPED>
struct QlinCfg {
  static constexpr int BN = ND * TB;
  static constexpr int kStageA = SRC == kNibbles ? kQTileA / 2 : kQTileA;
  static constexpr int kStageB = BN * kQK;
  static constexpr int kStage = kStageA + kStageB;
  static constexpr int kA8 = SRC == kNibbles ? 4 : 0;   // expanded tiles in flight
  // as many bytes in flight as fit: the weight stream is what counts
  static constexpr int kScales = GROUPED ? 8 * kQRows * 4 : 0;   // group scales of eight k-blocks
  static constexpr int kFit = (226 * 1024 - 2048 - kScales - kA8 * kQTileA) / kStage;
  static constexpr int kStages = kFit > 10 ? 10 : kFit;
  // Barriers, then the ring on a 1024-byte boundary, and no byte more: the blocks of the kernels before and after (quantisers,
  // norms, RoPE) fit beside one of this kernel only if it leaves them 1 KB and what they declare.  With 640 bytes more the
  // stages of 32 tokens left them 1 KB: a norm that writes digits waited for an SM without such a block, and took longer
  // than norm and quantiser apart.  Norm of four slabs and product of 24 rows, us, apart / together / together now:
  // 4608 x 3584 11.2 / 11.8 / 10.6, 7168 x 5120 16.0 / 16.6 / 14.4; 5120 x 27648 alone, 20 rows, 41.7 -> 36.4.
  static constexpr int kBars = 384;
  static constexpr int kSmem = kStages * kStage + kA8 * kQTileA + kScales + kBars + 1024;
  // per-group mode hands an accumulator over every k-block: four of them where they fit
  static constexpr int kAcc = GROUPED && 4 * BN <= 512 ? 4 : 2;
  static constexpr int kCols = kAcc * BN <= 32 ? 32 : kAcc * BN <= 64 ? 64 : kAcc * BN <= 128 ? 128 : kAcc * BN <= 256 ? 256 : 512;
  static constexpr int kExpand = SRC == kNibbles ? 256 : 0;
  static constexpr int kThreads = 192 + kExpand;
  static_assert(kStages >= 3 && kAcc * BN <= 512 && kStage % 1024 == 0, "stage ring / TMEM do not fit");
  static_assert((2 * kStages + 16) * 8 + 8 <= kBars, "barriers");
  // 228 KB an SM, of which every block takes 1 KB itself; up to 256 bytes for a block beside this one
  static_assert(kSmem + 2 * 1024 + 256 <= 228 * 1024, "nothing fits beside a block");
};

// K-major tile of 16-byte chunks [chunk][row][16 B], no swizzle: eight rows of one chunk are a 128-byte
// core matrix, the next eight rows 128 bytes on (stride byte offset), the next chunk 2048 bytes on
// (leading byte offset)
__device__ __forceinline__ uint64_t umma_desc_k_chunks(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((kQRows * 16) >> 4) << 16;
  d |= static_cast<uint64_t>(128 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}

// bits (without the sign) of the smallest bf16 that the digits of a row with |x| < 2^ex cannot hold:
// 255/256 * 2^ex would round up to 128 in the first digit
__device__ __forceinline__ uint32_t digit_limit(int ex) { return (uint32_t(ex + 126) << 7) | 0x7fu; }

// The products of a token's outliers (see k_quant_digits) with weight row n, k0 <= k < k1, without what is common
// to the row.  A whole warp calls it for one token: it goes to the chunks of 256 activations that the quantiser has
// marked (16 tokens, 5120 x 27648: 36 us; with one outlier each 68 us, 189 us looking through whole rows) and deals
// with the outliers of eight neighbours together, so that a row of nothing else (all infinities: some 4000 such
// steps) still ends long before the waits of the other warps do.  Infinities come out as in any sum of products.  A
// call of its own, so that the loops around it keep their registers: such rows are rare (inlined, it cost the products
// of every other row with group scales 12 %).
template <int SRC, bool GROUPED>
__device__ __noinline__ float outlier_sum(const QlinShape& g, int m, int k0, int k1, int n) {
  const int lane = threadIdx.x & 31;
  const float xs = __ldg(g.xs + m);
  if (!(xs < 0.f)) return 0.f;
  const uint32_t limit = digit_limit(int((__float_as_uint(xs) >> 23) & 0xffu) - 120);
  const __nv_bfloat16* xr = g.x + size_t(m) * g.ldx;
  const uint8_t* marks = reinterpret_cast<const uint8_t*>(g.xs + g.m) + size_t(m) * kDigChunks;
  float sum = 0.f;
  for (int c0 = k0 >> 8; c0 << 8 < k1; c0 += 32) {
    const int c = c0 + lane;
    for (uint32_t chunks = __ballot_sync(0xffffffffu, c << 8 < k1 && marks[c]); chunks; chunks &= chunks - 1) {
      const int k8 = ((c0 + __ffs(chunks) - 1) << 8) + lane * 8;  // of this lane's eight activations
      uint32_t hit = 0;
      uint4 a = make_uint4(0, 0, 0, 0);
      if (k8 >= k0 && k8 < k1) {
        a = *reinterpret_cast<const uint4*>(xr + k8);
        const uint32_t v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (((v[j >> 1] >> (16 * (j & 1))) & 0x7fffu) >= limit) hit |= 1u << j;
      }
      for (uint32_t lanes = __ballot_sync(0xffffffffu, hit != 0); lanes; lanes &= lanes - 1) {
        const int l = __ffs(lanes) - 1, kx = __shfl_sync(0xffffffffu, k8, l), gi = kx / (kQK * g.gk);
        const uint32_t h = __shfl_sync(0xffffffffu, hit, l);
        const uint32_t v[4] = {__shfl_sync(0xffffffffu, a.x, l), __shfl_sync(0xffffffffu, a.y, l),
                               __shfl_sync(0xffffffffu, a.z, l), __shfl_sync(0xffffffffu, a.w, l)};
        uint32_t q[2] = {0, 0};  // eight weights: nibbles of q[0], or bytes
        int zero = 0;
        if constexpr (SRC == kNibbles) {
          q[0] = __ldg(static_cast<const uint32_t*>(g.w) + size_t(kx >> 3) * g.n + n);
          zero = int((__ldg(g.zeros + size_t(gi) * (g.n >> 3) + (n >> 3)) >> (4 * (n & 7))) & 15u);
        } else {
          const uint2 t = __ldg(reinterpret_cast<const uint2*>(static_cast<const signed char*>(g.w) + size_t(n) * g.k + kx));
          q[0] = t.x;
          q[1] = t.y;
        }
        float part = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float x = __uint_as_float((j & 1) ? (v[j >> 1] & 0xffff0000u) : (v[j >> 1] << 16));
          const int w = SRC == kNibbles ? int((q[0] >> (4 * j)) & 15u) - zero
                                        : int(static_cast<signed char>(q[j >> 2] >> (8 * (j & 3))));
          if ((h >> j) & 1u) part = fmaf(x, float(w), part);
        }
        float sc = 1.f;
        if constexpr (GROUPED) {
          const size_t ng = size_t(n) * g.groups + gi, gn = size_t(gi) * g.n + n;
          sc = g.scale_kind == BL_QSCALE_F32_GN    ? __ldg(static_cast<const float*>(g.scale) + gn)
               : g.scale_kind == BL_QSCALE_F16_GN  ? __half2float(static_cast<const __half*>(g.scale)[gn])
               : g.scale_kind == BL_QSCALE_BF16_NG ? __bfloat162float(static_cast<const __nv_bfloat16*>(g.scale)[ng])
                                                   : __half2float(static_cast<const __half*>(g.scale)[ng]);
        }
        sum = fmaf(part, sc, sum);
      }
    }
  }
  return sum;
}

template <int SRC, int ND, int TB, bool GROUPED>
__global__ void __launch_bounds__(QlinCfg<SRC, ND, TB, GROUPED>::kThreads, 1)
    k_qlin(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
           const __grid_constant__ QlinShape g) {
  using S = QlinCfg<SRC, ND, TB, GROUPED>;
  extern __shared__ uint8_t smem_raw[];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem_raw);
  uint64_t* empty_bar = full_bar + S::kStages;
  uint64_t* tfull_bar = empty_bar + S::kStages;
  uint64_t* tempty_bar = tfull_bar + 4;
  uint64_t* ready_bar = tempty_bar + 4;   // kNibbles: an expanded tile is ready / free again
  uint64_t* afree_bar = ready_bar + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(afree_bar + 4);
  volatile uint32_t* s_abort = tmem_slot + 1;
  const uint32_t ring = (smem_u32(smem_raw) + uint32_t(S::kBars) + 1023u) & ~1023u;
  const uint32_t ring_a8 = ring + S::kStages * S::kStage;

  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int units = g.tiles_a * g.tiles_b * g.splits;
  const int kb_per = (g.kblocks + g.splits - 1) / g.splits;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], SRC == kNibbles ? 1 + 4 : 1);  // MMAs done; int4: the raw tile is free once expanded
    }
    for (int a = 0; a < 4; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 128);
      mbar_init(&ready_bar[a], 4);   // one lane of each of the four warps of an expanding group
      mbar_init(&afree_bar[a], 1);
    }
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, S::kCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    const uint32_t leader = elect_leader();
    // in elements of the tensor map: bytes, words of eight nibbles, or (eight chunks of 128 rows) 8 bytes
    auto ax = [&](int kb, int ta) { return SRC == kRows ? kb * kQK : ta * kQRows * (SRC == kNibbles ? 1 : 2); };
    auto ay = [&](int kb, int ta) { return SRC == kRows ? ta * kQRows : kb * (kQK / (SRC == kNibbles ? 8 : 16)); };
    // Before the kernels ahead have finished, the first lap of weight tiles is asked for into L2 only: HBM keeps
    // streaming across the kernel boundary, and weights that one of those kernels writes are read as it leaves
    // them, since every copy into shared memory starts behind the wait.
    int pre = 0;
    for (int u = blockIdx.x; u < units && pre < S::kStages; u += gridDim.x) {
      const int tile = u / g.splits, sp = u - tile * g.splits, ta = tile / g.tiles_b;
      const int kb0 = sp * kb_per, kb1 = min(g.kblocks, kb0 + kb_per);
      for (int kb = kb0; kb < kb1 && pre < S::kStages; ++kb, ++pre)
        tma_prefetch_2d_warp(leader, &tmap_w, ax(kb, ta), ay(kb, ta), kHintEvictFirst);
    }
    pdl_wait();
    int stage = 0, armed = 0;
    uint32_t phase = 0;
    bool ok = true;
    bool ready = false;  // the next stage is free (asked for one stage ahead, as in the MMA warp)
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int tile = u / g.splits, sp = u - tile * g.splits;
      const int ta = tile / g.tiles_b, tb = tile - ta * g.tiles_b;
      const int kb0 = sp * kb_per, kb1 = min(g.kblocks, kb0 + kb_per);
      for (int kb = kb0; kb < kb1; ++kb) {
        const uint32_t dst = ring + stage * S::kStage;
        uint64_t* full = &full_bar[stage];
        if (!ready) ok = mbar_wait_bounded(&empty_bar[stage], phase ^ 1u, s_abort);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        mbar_expect_tx_warp(leader, full, S::kStage);
        ++armed;
        if (++stage == S::kStages) {
          stage = 0;
          phase ^= 1u;
        }
        ready = mbar_test_wait(&empty_bar[stage], phase ^ 1u);
        tma_load_2d_hint_warp(leader, dst, &tmap_w, smem_u32(full), ax(kb, ta), ay(kb, ta), kHintEvictFirst);
        tma_load_2d_hint_warp(leader, dst + S::kStageA, &tmap_x, smem_u32(full), kb * kQK, tb * S::BN, kHintEvictLast);
      }
    }
    if (!ok) {
      // copies still in flight land before the CTA goes away
      const int n = armed < S::kStages ? armed : S::kStages;
      int s = stage;
      uint32_t ph = phase;
      for (int i = 0; i < n; ++i) {
        if (--s < 0) {
          s = S::kStages - 1;
          ph ^= 1u;
        }
        for (uint32_t p = 0; p < (1u << 20); ++p)
          if (mbar_try_wait(&full_bar[s], ph)) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------
    const uint32_t leader = elect_leader();
    const uint32_t idesc = umma_idesc_i8(kQRows, S::BN);
    int stage = 0, acc = -1, a8 = 0;
    uint32_t phase = 0, a8phase = 0;
    uint32_t tphase = 1;  // of the accumulators: all are free at the start
    bool ok = true;
    // the next stage is asked for before the products of this one are issued, so that the answer is there
    // when they are
    bool ready = mbar_test_wait(&full_bar[0], 0);
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int sp = u % g.splits;
      const int kb0 = sp * kb_per, kb1 = min(g.kblocks, kb0 + kb_per);
      for (int kb = kb0; kb < kb1; ++kb) {
        if (GROUPED || kb == kb0) {
          if (++acc == S::kAcc) {
            acc = 0;
            tphase ^= 1u;
          }
          ok = mbar_wait_bounded(&tempty_bar[acc], tphase, s_abort);
        }
        // int4: the expanding threads have waited for the stage, but the digits are read here too
        if (!ready) ok = ok && mbar_wait_bounded(&full_bar[stage], phase, s_abort);
        if (SRC == kNibbles) ok = ok && mbar_wait_bounded(&ready_bar[a8], a8phase, s_abort);
        if (!__all_sync(0xffffffffu, ok)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + uint32_t(acc * S::BN);
        const uint32_t sx = ring + stage * S::kStage;
        const uint32_t sa = SRC == kNibbles ? ring_a8 + a8 * kQTileA : sx;
        uint64_t* done = &empty_bar[stage];
        if (++stage == S::kStages) {
          stage = 0;
          phase ^= 1u;
        }
        ready = mbar_test_wait(&full_bar[stage], phase);
        const uint64_t da = SRC == kRows ? umma_desc_k_sw128(sa) : umma_desc_k_chunks(sa);
        const uint64_t db = umma_desc_k_sw128(sx + S::kStageA);
        // 32 bytes along K per instruction: +2 (16-byte units) inside a swizzled row, two chunks otherwise
        constexpr int kStepA = SRC == kRows ? 2 : 2 * (kQRows * 16) / 16;
#pragma unroll
        for (int k = 0; k < kQK / 32; ++k)
          umma_i8_ss_warp(leader, d_tmem, da + uint64_t(kStepA * k), db + uint64_t(2 * k), idesc,
                          ((!GROUPED && kb > kb0) || k > 0) ? 1u : 0u);
        if (SRC == kNibbles) {
          umma_commit_warp(leader, &afree_bar[a8]);
          if (++a8 == 4) {
            a8 = 0;
            a8phase ^= 1u;
          }
        }
        umma_commit_warp(leader, done);
        if (GROUPED || kb + 1 == kb1) umma_commit_warp(leader, &tfull_bar[acc]);
      }
    }
  } else if (SRC == kNibbles && warp >= 6) {
    // ------------------------ int4 -> int8 -------------------------------
    // Two groups of 128 threads take alternate k-blocks; a thread expands one weight row: 16 words in
    // (consecutive lanes, consecutive words), eight 16-byte chunks out (consecutive lanes,
    // consecutive chunks): no bank conflicts on either side.
    pdl_wait();  // the zero points may come from a kernel ahead
    const int ct = threadIdx.x - 192, grp = ct >> 7, row = ct & 127;
    int nkb = 0;
    bool ok = true;
    // words with the zero points of this group's next kZ k-blocks, requested together and one batch ahead
    constexpr int kZ = 8;
    auto first_of = [&](int u, int before) {  // first k-block of unit u that this group expands
      const int kb0 = (u % g.splits) * kb_per;
      return kb0 + ((before & 1) != grp ? 1 : 0);
    };
    auto zero_words = [&](int u, int kb, uint32_t (&z)[kZ]) {
      const int tile = u / g.splits, kb1 = min(g.kblocks, (u - tile * g.splits + 1) * kb_per);
      const uint32_t* zp = g.zeros + (min((tile / g.tiles_b) * kQRows + row, g.n - 1) >> 3);
#pragma unroll
      for (int i = 0; i < kZ; ++i)
        z[i] = u < units && kb + 2 * i < kb1 ? __ldg(zp + size_t((kb + 2 * i) / g.gk) * (g.n >> 3)) : 0u;
    };
    uint32_t zcur[kZ], znext[kZ];
    zero_words(blockIdx.x, first_of(blockIdx.x, 0), zcur);
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int tile = u / g.splits, sp = u - tile * g.splits;
      const int kb0 = sp * kb_per, kb1 = min(g.kblocks, kb0 + kb_per);
      const int zsh = (min((tile / g.tiles_b) * kQRows + row, g.n - 1) & 7) * 4;
      // a unit of one k-block may have none for this group: on to the next unit's words
      if (first_of(u, nkb) >= kb1) zero_words(u + gridDim.x, first_of(u + gridDim.x, nkb + kb1 - kb0), zcur);
      for (int kbz = first_of(u, nkb); kbz < kb1 && ok; kbz += 2 * kZ) {
        if (kbz + 2 * kZ < kb1) zero_words(u, kbz + 2 * kZ, znext);
        else zero_words(u + gridDim.x, first_of(u + gridDim.x, nkb + kb1 - kb0), znext);
#pragma unroll
        for (int i = 0; i < kZ; ++i) {
          const int kb = kbz + 2 * i;
          if (kb >= kb1) break;
          const int b = nkb + (kb - kb0), stage = b % S::kStages;
          if (!mbar_wait_bounded_warp(&full_bar[stage], uint32_t(b / S::kStages) & 1u, s_abort) ||
              !mbar_wait_bounded_warp(&afree_bar[b & 3], (uint32_t(b >> 2) & 1u) ^ 1u, s_abort)) {
            ok = false;
            break;
          }
          const uint32_t src = ring + stage * S::kStage + row * 4;
          const uint32_t dst = ring_a8 + (b & 3) * kQTileA + row * 16;
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j)
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(w[j]) : "r"(src + j * (kQRows * 4)));
          // byte = (128 + nibble - zero) without borrow between bytes, then the sign bit flipped
          const uint32_t zz = ((zcur[i] >> zsh) & 15u) * 0x01010101u;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            uint32_t o[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t v = w[2 * c + h];
              o[2 * h] = (((v & 0x0F0F0F0Fu) | 0x80808080u) - zz) ^ 0x80808080u;
              o[2 * h + 1] = ((((v >> 4) & 0x0F0F0F0Fu) | 0x80808080u) - zz) ^ 0x80808080u;
            }
            asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst + c * (kQRows * 16)), "r"(o[0]), "r"(o[1]),
                         "r"(o[2]), "r"(o[3])
                         : "memory");
          }
          fence_proxy_async_smem();  // the tensor core reads what these threads just wrote
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&ready_bar[b & 3]);
            mbar_arrive(&empty_bar[stage]);  // raw words consumed (the MMAs' commit frees the digits)
          }
        }
#pragma unroll
        for (int i = 0; i < kZ; ++i) zcur[i] = znext[i];
      }
      nkb += kb1 - kb0;
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int q = warp & 3, row = q * 32 + lane;
    pdl_wait();
    int accs = 0;
    bool ok = true;
    // Straight-line code that runs once a tile comes at the pace of the instruction cache, not of the SM.  With
    // every loop of the epilogue unrolled, warps waited 3.5 (64 tokens, group scales) to 14 (one small tile)
    // cycles for instructions per one issued; 64 tokens took 17 us at 256 x 256 and, with group scales, 98 us at
    // 37888 x 3584.  Rolled wherever registers need no index: 8.8 and 52 us.
    // Group scales of kAhead k-blocks are requested together and one batch ahead, kept as they came and
    // turned into fp32 at their use, so that no k-block waits for a trip to HBM.  They pass through slots of
    // shared memory that only this thread touches.
    constexpr int kAhead = 8;
    uint32_t* s_sc = reinterpret_cast<uint32_t*>(smem_raw + (ring_a8 + S::kA8 * kQTileA - smem_u32(smem_raw))) + row;
    uint32_t sc_next[GROUPED ? kAhead : 1];
    auto scales_of = [&](int u, int kb) {
      const int tile = u / g.splits, kb1 = min(g.kblocks, (u - tile * g.splits + 1) * kb_per);
      const int n = (tile / g.tiles_b) * kQRows + row;
      const bool in = u < units && n < g.n;
      const uint32_t* p32 = static_cast<const uint32_t*>(g.scale);
      const unsigned short* p16 = static_cast<const unsigned short*>(g.scale);
#pragma unroll
      for (int i = 0; i < (GROUPED ? kAhead : 1); ++i) {
        const int gi = (kb + i) / g.gk;
        sc_next[i] = !in || kb + i >= kb1                    ? 0u
                     : g.scale_kind == BL_QSCALE_F32_GN ? __ldg(p32 + size_t(gi) * g.n + n)
                     : g.scale_kind == BL_QSCALE_F16_GN ? uint32_t(__ldg(p16 + size_t(gi) * g.n + n))
                                                        : uint32_t(__ldg(p16 + size_t(n) * g.groups + gi));
      }
    };
    auto scale_f32 = [&](uint32_t raw) -> float {
      return g.scale_kind == BL_QSCALE_F32_GN ? __uint_as_float(raw)
             : g.scale_kind == BL_QSCALE_BF16_NG ? __uint_as_float(raw << 16)
                                                 : __half2float(__ushort_as_half(static_cast<unsigned short>(raw)));
    };
    if constexpr (GROUPED) scales_of(blockIdx.x, (int(blockIdx.x) % g.splits) * kb_per);
    for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
      const int tile = u / g.splits, sp = u - tile * g.splits;
      const int ta = tile / g.tiles_b, tb = tile - ta * g.tiles_b;
      const int n = ta * kQRows + row, m0 = tb * TB;
      const bool nok = n < g.n;
      const int nn = nok ? n : g.n - 1;
      // one accumulator set read as fp32: columns c0 .. c0+15 of every digit plane put together
      auto read16 = [&](int acc, int c0, float (&v)[16]) {
        const uint32_t t = tmem_base + (uint32_t(q * 32) << 16) + uint32_t(acc * S::BN + c0);
        if constexpr (ND == 1) {
          uint32_t r[16];
          tmem_ld_32x16(t, r);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = float(int32_t(r[i]));
        } else {
          uint32_t r0[16], r1[16], r2[16];
          tmem_ld_32x16(t, r0);
          tmem_ld_32x16(t + TB, r1);
          tmem_ld_32x16(t + 2 * TB, r2);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i)
            v[i] = fmaf(float(int32_t(r2[i])), 1.f / 65536.f,
                        fmaf(float(int32_t(r1[i])), 1.f / 256.f, float(int32_t(r0[i]))));
        }
      };
      float rs = 1.f;  // what is left to multiply with once the sums are there
      float accf[GROUPED ? TB : 1];
      int done_acc = 0;
      if constexpr (GROUPED) {
        const int kb0 = sp * kb_per, kb1 = min(g.kblocks, kb0 + kb_per);
        if (g.row_scale) rs = __bfloat162float(g.row_scale[nn]);
#pragma unroll
        for (int i = 0; i < TB; ++i) accf[i] = 0.f;
#pragma unroll 1
        for (int kb = kb0; kb < kb1; ++kb) {
          const int i = (kb - kb0) % kAhead;
          if (i == 0) {
#pragma unroll
            for (int j = 0; j < kAhead; ++j) s_sc[j * kQRows] = sc_next[j];
            if (kb + kAhead < kb1) scales_of(u, kb + kAhead);
            else scales_of(u + gridDim.x, ((u + gridDim.x) % g.splits) * kb_per);
          }
          const float sc = scale_f32(s_sc[i * kQRows]);
          const int acc = accs % S::kAcc;
          if (!mbar_wait_bounded_warp(&tfull_bar[acc], uint32_t(accs / S::kAcc) & 1u, s_abort)) {
            ok = false;
            break;
          }
          ++accs;
          tc_fence_after_sync();
#pragma unroll
          for (int c0 = 0; c0 < TB; c0 += 16) {
            float v[16];
            read16(acc, c0, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) accf[c0 + j] = fmaf(v[j], sc, accf[c0 + j]);
          }
          tc_fence_before_sync();
          mbar_arrive(&tempty_bar[acc]);
        }
        if (!ok) break;
      } else {
        rs = __bfloat162float(static_cast<const __nv_bfloat16*>(g.scale)[nn]);
        done_acc = accs % S::kAcc;
        if (!mbar_wait_bounded_warp(&tfull_bar[done_acc], uint32_t(accs / S::kAcc) & 1u, s_abort)) break;
        ++accs;
        tc_fence_after_sync();
      }
      const float bv = (nok && g.bias && !g.slabs) ? __bfloat162float(g.bias[n]) : 0.f;
      const int m_end = min(g.m - m0, TB);  // tokens of this tile
#pragma unroll 1
      for (int c0 = 0; c0 < m_end; c0 += 16) {
        float v[16];
        if constexpr (GROUPED) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = accf[j];
          // (the next 16 sums move down: the loop body stays one)
#pragma unroll
          for (int j = 0; j + 16 < TB; ++j) accf[j] = accf[j + 16];
        } else {
          read16(done_acc, c0, v);
        }
        float xm[16];
        bool rare = false;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          xm[j] = c0 + j < m_end ? __ldg(g.xs + m0 + c0 + j) : 0.f;
          if (ND == 3) rare |= xm[j] < 0.f;
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= (ND == 3 ? fabsf(xm[j]) : xm[j]) * rs;
        if (ND == 3 && rare) {
#pragma unroll 1
          for (int t = 0; c0 + t < m_end && t < 16; ++t) {
            const float o = rs * outlier_sum<SRC, GROUPED>(g, m0 + c0 + t, sp * kb_per * kQK, min(g.k, (sp + 1) * kb_per * kQK), nn);
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (j == t) v[j] += o;
          }
        }
        const int m1 = m0 + c0, mn = nok ? min(16, m_end - c0) : 0;  // first token, tokens to store
        if (g.slabs) {
          float* o = g.slabs + (size_t(sp) * g.m + m1) * g.n + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < mn) __stcg(o + size_t(j) * g.n, v[j]);
        } else if (g.silu) {
          // even lanes hold gate rows, odd lanes the matching up rows
          __nv_bfloat16* o = g.out + size_t(m1) * g.ldo + (n >> 1);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float mine = v[j] + bv;
            const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
            if (j < mn && !(row & 1)) o[size_t(j) * g.ldo] = __float2bfloat16(mine / (1.f + __expf(-mine)) * other);
          }
        } else {
          __nv_bfloat16* o = g.out + size_t(m1) * g.ldo + n;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (j < mn) o[size_t(j) * g.ldo] = __float2bfloat16(v[j] + bv);
        }
      }
      if constexpr (!GROUPED) {
        tc_fence_before_sync();
        mbar_arrive(&tempty_bar[done_acc]);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, S::kCols);
  }
  if (threadIdx.x == 0 && *s_abort && g.err) *g.err = 1u;
}

// ---------------------------------------------------------------------------
// activations -> digits
// ---------------------------------------------------------------------------
// x [m][k] bf16 -> xq [ceil(m/tb)][3][tb][k] int8 and xs[m]: x = |xs| * (d0 + d1/2^8 + d2/2^16).  |xs| is a
// power of two chosen from the row's largest element so that d0 fits 8 bits; a negative xs says that the row
// has outliers, elements beyond the digits' range, whose digits are zero.  Behind the m words of xs lie 128 bytes a
// row, written for such rows alone: whether elements 256 c .. 256 c + 255 have outliers.  One block per token.
constexpr int kDigThreads = 512;
constexpr int kDigVec = 8;   // 16-byte vectors per thread: rows of up to 32768 elements
static_assert(kDigVec * kDigThreads / 32 <= kDigChunks, "a mark for every chunk of the longest row");
__device__ __forceinline__ uint32_t bf16x2_absmax_bits(uint32_t m, uint32_t v) {
  m = max(m, v & 0x7fffu);
  return max(m, (v >> 16) & 0x7fffu);
}
__device__ __forceinline__ uint32_t bf16x8_absmax_bits(uint32_t m, const uint4& v) {
  m = bf16x2_absmax_bits(bf16x2_absmax_bits(m, v.x), v.y);
  return bf16x2_absmax_bits(bf16x2_absmax_bits(m, v.z), v.w);
}
// The digits of a row that the blocks of a cluster (CL of them, or one) hold in registers: vector i of a thread is vector
// threadIdx.x + i * kDigThreads of its block's share, which is `vecs` long and starts at vector `first` of the row; every
// block but the last has `per` of them.  mx: the largest |x| of the thread's vectors as bf16 bits, ordered like the values,
// NaN above infinity (found while they are loaded: in a loop of its own behind the loads it cost rows of eight vectors a
// thread half as many spills again, 12.2 us for 11.6).
template <bool PERMUTE, int VPT, int CL>
__device__ __forceinline__ void digits_of_row(uint4 (&v)[VPT], uint32_t mx, int row, int rows, int first, int per, int vecs, int k, int tb,
                                              int8_t* __restrict__ xq, float* __restrict__ xs) {
  // (little shared memory: a block of these kernels fits beside one of k_qlin, which has nearly all of it)
  __shared__ uint32_t s_red[kDigThreads / 32];
  __shared__ uint32_t s_clu[2][CL];  // the words of a row's blocks, two sets in turn
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t part = CL > 1 ? cluster_ctarank() : 0;
  int turn = 0;
  // every block of the row gives a word, every thread of them finds all in s_clu[turn ^ 1]
  auto share = [&](uint32_t w) {
    if (threadIdx.x < CL) st_cluster_u32(map_to_cta(smem_u32(&s_clu[turn][part]), threadIdx.x), w);
    cluster_sync_all();
    turn ^= 1;
  };
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) s_red[warp] = mx;
  __syncthreads();
  mx = __reduce_max_sync(0xffffffffu, s_red[lane & (kDigThreads / 32 - 1)]);
  if constexpr (CL > 1) {
    share(mx);
#pragma unroll
    for (int c = 0; c < CL; ++c) mx = max(mx, s_clu[turn ^ 1][c]);
  }
  // nonzero elements below 2^(e - 127) and, in the upper half of the word, nonzero ones in all (each fits 16 bits)
  auto count = [&](int e) -> uint32_t {
    const uint32_t top = e > 0 ? uint32_t(e) << 7 : 1u;
    uint32_t n = 0;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t a = (w[j >> 1] >> (16 * (j & 1))) & 0x7fffu;
        n += (a != 0 ? 0x10000u : 0u) + (a - 1u < top - 1u ? 1u : 0u);
      }
    }
    n = __reduce_add_sync(0xffffffffu, n);
    __syncthreads();
    if (lane == 0) s_red[warp] = n;
    __syncthreads();
    n = __reduce_add_sync(0xffffffffu, lane < kDigThreads / 32 ? s_red[lane] : 0u);
    if constexpr (CL > 1) {
      share(n);
      n = 0;
#pragma unroll
      for (int c = 0; c < CL; ++c) n += s_clu[turn ^ 1][c];
    }
    return n;
  };
  // |x| < 2^ex; a largest element of 255/256 * 2^ex would round up to 128 in the first digit
  int ex = int(mx >> 7) - 126 + ((mx & 0x7fu) == 0x7fu ? 1 : 0);
  if (ex < -110) ex = -110;  // the digits of such rows reach the smallest bf16, 2^-133
  // Below 2^(ex - 13).  (What follows costs such a row 1 to 2 us in the linear, so the line lies beyond the rows that
  // products of activations give: a bf16 result is rounded to 2^-9, the median element here to 2^-11.)
  const uint32_t small = count(ex > -110 ? ex + 114 : 0);
  const bool bad = mx > 0x7f80u;  // NaN in the row: the whole row of results is NaN
  const bool split = !bad && (2 * (small & 0xffffu) > (small >> 16) || mx == 0x7f80u);
  if (split) {
    // the median's exponent: the smallest e with half of the nonzero elements below 2^(e + 1 - 127)
    int lo = 0, hi = 255;
#pragma unroll 1
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      // (keeps the compiler from holding all magnitudes in registers over this loop: the block would not fit)
#pragma unroll
      for (int i = 0; i < VPT; ++i) asm volatile("" : "+r"(v[i].x), "+r"(v[i].y), "+r"(v[i].z), "+r"(v[i].w));
      if (2 * (count(mid + 1) & 0xffffu) >= (small >> 16)) hi = mid;
      else lo = mid + 1;
    }
    ex = min(128, max(-110, lo - 126 + 12));
  }
  const uint32_t limit = digit_limit(ex);
  if (split) {
    // a warp's 32 vectors are one chunk
    uint8_t* marks = reinterpret_cast<uint8_t*>(xs + rows) + size_t(row) * kDigChunks + first / 32;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
      bool hit = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) hit |= ((w[j >> 1] >> (16 * (j & 1))) & 0x7fffu) >= limit;
      hit = __any_sync(0xffffffffu, hit);
      const int chunk = i * (kDigThreads / 32) + warp;
      if (lane == 0 && (CL == 1 || chunk * 32 < per)) marks[chunk] = hit ? 1 : 0;
    }
  }
  const float scale = bad ? 0.f : __uint_as_float(uint32_t(127 + 7 - ex) << 23);
  if (threadIdx.x == 0 && part == 0)
    xs[row] = bad ? __uint_as_float(0x7fffffffu) : __uint_as_float(uint32_t(127 - 7 + ex) << 23 | (split ? 1u << 31 : 0u));
  int8_t* base = xq + (size_t(row / tb) * 3 * tb + row % tb) * size_t(k) + size_t(first) * 8;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * kDigThreads;
    if (c >= vecs) continue;
    const uint32_t w[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    uint32_t o[3][2] = {{0, 0}, {0, 0}, {0, 0}};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t f = (j & 1) ? (w[j >> 1] & 0xffff0000u) : (w[j >> 1] << 16);
      const float y0 = bad || ((f >> 16) & 0x7fffu) >= limit ? 0.f : __uint_as_float(f) * scale;
      // every step leaves a remainder in [-128.5, 127.5) / 256, so that the next digit fits too
      const float d0 = floorf(y0 + 128.5f / 256.f);
      const float y1 = (y0 - d0) * 256.f;
      const float d1 = fminf(floorf(y1 + 128.5f / 256.f), 127.f);
      const float y2 = (y1 - d1) * 256.f;
      const float d2 = fminf(rintf(y2), 127.f);
      const int pos = PERMUTE ? ((j & 1) * 4 + (j >> 1)) : j;
      const int sh = 8 * (pos & 3);
      o[0][pos >> 2] |= (uint32_t(int(d0)) & 0xffu) << sh;
      o[1][pos >> 2] |= (uint32_t(int(d1)) & 0xffu) << sh;
      o[2][pos >> 2] |= (uint32_t(int(d2)) & 0xffu) << sh;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d)
      *reinterpret_cast<uint2*>(base + size_t(d) * tb * k + size_t(c) * 8) = make_uint2(o[d][0], o[d][1]);
  }
}

template <bool PERMUTE, int VPT, int CL>
__device__ __forceinline__ void quant_digits_body(const __nv_bfloat16* __restrict__ x, int ldx, int k, int tb,
                                                  int8_t* __restrict__ xq, float* __restrict__ xs) {
  pdl_launch_dependents();
  if constexpr (CL > 1) cluster_sync_all();  // the other blocks' shared memory is there
  pdl_wait();
  const int row = blockIdx.x / CL;
  // this block's share of the row: whole chunks of 256 elements
  const int per = CL > 1 ? ((k / 8 + CL * 32 - 1) / (CL * 32)) * 32 : k >> 3;
  const int first = CL > 1 ? int(cluster_ctarank()) * per : 0, vecs = max(0, min(per, (k >> 3) - first));
  const uint4* xr = reinterpret_cast<const uint4*>(x + size_t(row) * ldx) + first;
  uint4 v[VPT];
  uint32_t mx = 0;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * kDigThreads;
    v[i] = c < vecs ? xr[c] : make_uint4(0, 0, 0, 0);
    mx = bf16x8_absmax_bits(mx, v[i]);
  }
  digits_of_row<PERMUTE, VPT, CL>(v, mx, row, gridDim.x / CL, first, per, vecs, k, tb, xq, xs);
}
template <bool PERMUTE, int VPT>
__global__ void __launch_bounds__(kDigThreads, 2) k_quant_digits(const __nv_bfloat16* __restrict__ x, int ldx, int k, int tb,
                                                              int8_t* __restrict__ xq, float* __restrict__ xs) {
  quant_digits_body<PERMUTE, VPT, 1>(x, ldx, k, tb, xq, xs);
}
// A long row of few tokens takes one block a chain of loads, counts and conversions over eight vectors a thread (16 x 27648:
// 10 us between the linears around it, 5.0 now): a cluster of blocks shares it, one vector a thread, the row's maximum
// and counts passed through distributed shared memory.
template <bool PERMUTE, int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(kDigThreads, 2)
    k_quant_digits_cluster(const __nv_bfloat16* __restrict__ x, int ldx, int k, int tb, int8_t* __restrict__ xq,
                           float* __restrict__ xs) {
  quant_digits_body<PERMUTE, 1, CL>(x, ldx, k, tb, xq, xs);
  cluster_sync_all();  // no block leaves while another may still write its words
}

__device__ __forceinline__ void row_floats(const uint4& a, float (&f)[8]) {
  const float2 p0 = unpack_bf16x2(a.x), p1 = unpack_bf16x2(a.y), p2 = unpack_bf16x2(a.z), p3 = unpack_bf16x2(a.w);
  f[0] = p0.x; f[1] = p0.y; f[2] = p1.x; f[3] = p1.y;
  f[4] = p2.x; f[5] = p2.y; f[6] = p3.x; f[7] = p3.y;
}
__device__ __forceinline__ uint4 row_pack(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// RMSNorm (+ residual add) of one row by one block.  v: the normed row on return, vector i of a thread being vector
// threadIdx.x + i * blockDim.x.  x is the row itself, or (partials) the sum of the k-split slabs of the linear in front, rounded
// to bf16 as that linear's output would have been.  Slabs are read four at a time and rows stay packed, 64 registers a
// thread, so that a block still fits beside one of k_qlin (eight slabs at a time spilled: 14.6 us a norm instead of 7.2).
template <int VPT>
__device__ __forceinline__ void norm_row(uint4 (&v)[VPT], const uint4* __restrict__ x, const uint4* __restrict__ residual,
                                         const uint4* __restrict__ gamma, uint4* __restrict__ out,
                                         uint4* __restrict__ residual_out, int vpr, float eps,
                                         const float* __restrict__ partials, int nsplit, size_t slab) {
  __shared__ float s_part[16];
  const size_t base = size_t(blockIdx.x) * vpr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float ss = 0.f, f[8], g[8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    v[i] = make_uint4(0, 0, 0, 0);
    if (c >= vpr) continue;
    uint4 r = make_uint4(0, 0, 0, 0);
    if (residual) r = residual[base + c];
    if (partials) {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.f;
      const float* p = partials + (base + c) * 8;
#pragma unroll 1
      for (int s0 = 0; s0 < nsplit; s0 += 4) {
        float4 u[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (s0 + q < nsplit) {
            const float4* t = reinterpret_cast<const float4*>(p + size_t(s0 + q) * slab);
            u[q][0] = __ldcg(t);
            u[q][1] = __ldcg(t + 1);
          }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (s0 + q < nsplit) {
            f[0] += u[q][0].x; f[1] += u[q][0].y; f[2] += u[q][0].z; f[3] += u[q][0].w;
            f[4] += u[q][1].x; f[5] += u[q][1].y; f[6] += u[q][1].z; f[7] += u[q][1].w;
          }
      }
      v[i] = row_pack(f);
    } else {
      v[i] = x[base + c];
    }
    row_floats(v[i], f);
    if (residual) {
      row_floats(r, g);
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] += g[j];
      v[i] = row_pack(f);  // the norm sees the stored (rounded) sum
      residual_out[base + c] = v[i];
      row_floats(v[i], f);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
  }
  ss = warp_sum(ss);
  if (lane == 0) s_part[warp] = ss;
  __syncthreads();
  ss = warp_sum(lane < int(blockDim.x >> 5) ? s_part[lane] : 0.f);
  const float rstd = rsqrtf(ss / float(vpr * 8) + eps);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c >= vpr) continue;
    row_floats(v[i], f);
    row_floats(gamma[c], g);
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __bfloat162float(__float2bfloat16(f[j] * rstd)) * g[j];
    v[i] = row_pack(f);
    out[base + c] = v[i];
  }
}

// RMSNorm (+ residual) of decode rows, as k_rmsnorm does it (same sums, same bits), that leaves the digits of its result
// too: the linear behind it reads them.  16 x 5120 between the linears of a decode step: the norm and a kernel of its own
// for the digits 5.6 + 3.5 us, this 7.2.
template <int VPT>
__global__ void __launch_bounds__(kDigThreads, 2)
    k_rmsnorm_digits(const uint4* __restrict__ x, const uint4* __restrict__ residual, const uint4* __restrict__ gamma,
                     uint4* __restrict__ out, uint4* __restrict__ residual_out, int vpr, float eps,
                     const float* __restrict__ partials, int nsplit, size_t slab, int tb, int8_t* __restrict__ xq,
                     float* __restrict__ xs) {
  pdl_launch_dependents();
  pdl_wait();
  uint4 v[VPT];
  norm_row<VPT>(v, x, residual, gamma, out, residual_out, vpr, eps, partials, nsplit, slab);
  uint32_t mx = 0;
#pragma unroll
  for (int i = 0; i < VPT; ++i) mx = bf16x8_absmax_bits(mx, v[i]);
  digits_of_row<false, VPT, 1>(v, mx, blockIdx.x, gridDim.x, 0, vpr, vpr, vpr * 8, tb, xq, xs);
}

// fp32 slabs [split][m][pitch] -> bf16 [m][n]: sum in split order, then what the epilogue of the unsplit product
// does: + bias, tanh-GELU, + residual; or + bias and SiLU*mul over interleaved (gate, up) columns.  Eight columns
// per thread.  The slabs start on 16-byte boundaries and have a pitch of a multiple of 8; bias, residual and
// output are a caller's tensors, often slices of longer ones, and go element by element where their start, their
// pitch or a ragged end asks for it.
__device__ __forceinline__ void load8_any(const __nv_bfloat16* p, int cols, float (&f)[8]) {
  if (cols == 8 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
    const uint4 b = *reinterpret_cast<const uint4*>(p);
    const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y), b2 = unpack_bf16x2(b.z), b3 = unpack_bf16x2(b.w);
    f[0] = b0.x; f[1] = b0.y; f[2] = b1.x; f[3] = b1.y;
    f[4] = b2.x; f[5] = b2.y; f[6] = b3.x; f[7] = b3.y;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = j < cols ? __bfloat162float(p[j]) : 0.f;
  }
}
__global__ void __launch_bounds__(256) k_slab_finish(const blSlabFinishArgs g, size_t total8) {
  pdl_launch_dependents();
  pdl_wait();
  const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= total8) return;
  const int per = g.pitch >> 3;
  const size_t m = t / per;
  const int c = int(t - m * per) * 8, cols = min(8, g.n - c);
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, f[8];
  sum_slabs8(static_cast<const float*>(g.slabs) + m * g.pitch + c, size_t(g.m) * g.pitch, g.nsplit, a);
  if (g.bias) {
    load8_any(static_cast<const __nv_bfloat16*>(g.bias) + c, cols, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += f[j];
  }
  __nv_bfloat16* out = static_cast<__nv_bfloat16*>(g.out) + m * g.ldo + (g.silu_mul ? c >> 1 : c);
  if (g.silu_mul) {
    float o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] = a[2 * j] / (1.f + __expf(-a[2 * j])) * a[2 * j + 1];
    if (cols == 8 && (reinterpret_cast<uintptr_t>(out) & 7u) == 0) {
      *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < (cols >> 1)) out[j] = __float2bfloat16(o[j]);
    }
    return;
  }
  if (g.gelu) {
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = gelu_tanh(a[j]);
  }
  if (g.residual) {
    load8_any(static_cast<const __nv_bfloat16*>(g.residual) + m * g.ldo + c, cols, f);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] += f[j];
  }
  if (cols == 8 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
    *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]),
                                                pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7]));
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j < cols) out[j] = __float2bfloat16(a[j]);
  }
}

template <int SRC, int ND, int TB, bool GROUPED>
static int launch_qlin(const blQlinArgs& a, cudaStream_t st, char* err, size_t errlen) {
  using S = QlinCfg<SRC, ND, TB, GROUPED>;
  CUtensorMap tw, tx;
  const int tiles_b = (a.m + TB - 1) / TB;
  // digit planes are laid out tile by tile, dense; single-digit activations are plain rows
  const uint64_t xrows = ND == 1 ? uint64_t(a.m) : uint64_t(tiles_b) * S::BN;
  if (make_tmap_kmajor(a.xq, xrows, a.k, a.k, S::BN, 1, &tx, err, errlen, kQK) != 0) return -1;
  if (SRC == kRows) {
    if (make_tmap_kmajor(a.w, a.n, a.k, a.k, kQRows, 1, &tw, err, errlen, kQK) != 0) return -1;
  } else {
    // kNibbles: 16 rows of 128 packed words a k-block; kChunks: 8 rows of 128 chunks of 16 bytes, as
    // elements of 8 bytes (a box has at most 256 elements a side)
    const DriverApi* d = driver(err, errlen);
    if (!d) return -1;
    constexpr bool nib = SRC == kNibbles;
    cuuint64_t dims[2] = {cuuint64_t(a.n) * (nib ? 1 : 2), cuuint64_t(a.k / (nib ? 8 : 16))};
    cuuint64_t strides[1] = {cuuint64_t(a.n) * (nib ? 4 : 16)};
    cuuint32_t box[2] = {kQRows * (nib ? 1 : 2), kQK / (nib ? 8 : 16)}, estr[2] = {1, 1};
    if (d->cuTensorMapEncodeTiled(&tw, nib ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_INT64, 2,
                                  const_cast<void*>(a.w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
      set_err(err, errlen, "barlink: tensor map of the quantised weight failed (n %d, k %d)", a.n, a.k);
      return -1;
    }
  }
  QlinShape g;
  memset(&g, 0, sizeof(g));
  g.n = a.n;
  g.m = a.m;
  g.k = a.k;
  g.tiles_a = (a.n + kQRows - 1) / kQRows;
  g.tiles_b = tiles_b;
  g.kblocks = (a.k + kQK - 1) / kQK;
  g.splits = a.splits;
  g.zeros = static_cast<const uint32_t*>(a.zeros);
  g.xs = static_cast<const float*>(a.xs);
  g.x = static_cast<const __nv_bfloat16*>(a.x);
  g.ldx = a.ldx;
  g.w = a.w;
  g.scale_kind = a.scale_kind;
  g.scale = a.scale;
  g.row_scale = static_cast<const __nv_bfloat16*>(a.row_scale);
  g.gk = GROUPED ? a.group_k / kQK : 1;
  g.groups = GROUPED ? a.k / a.group_k : 1;
  g.bias = static_cast<const __nv_bfloat16*>(a.bias);
  g.out = static_cast<__nv_bfloat16*>(a.out);
  g.ldo = a.ldo;
  g.silu = a.silu_mul;
  g.slabs = static_cast<float*>(a.slabs);
  g.err = static_cast<uint32_t*>(a.err_flag);
  const int units = g.tiles_a * g.tiles_b * g.splits;
  const int grid = units < sm_count() ? units : sm_count();
  static bool attr[64] = {};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(k_qlin<SRC, ND, TB, GROUPED>), S::kSmem, attr);
  if (e == cudaSuccess)
    e = launch_k(k_qlin<SRC, ND, TB, GROUPED>, dim3(grid), dim3(S::kThreads), size_t(S::kSmem), st, tw, tx, g);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: quantised linear launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

// Tokens of a tile.  One int8 digit with per-channel scales takes up to 128, so that no weight tile is
// fetched twice (65 .. 128 tokens, 37888 x 3584, two tiles of 64: 55 us; one of 128: 28 us).
static int qlin_tile_tokens(int m, int digits, bool grouped) {
  return m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 || digits > 1 || grouped ? 64 : 128;
}

template <int SRC, int ND, bool GROUPED>
static int launch_qlin_tb(const blQlinArgs& a, cudaStream_t st, char* err, size_t errlen) {
  switch (qlin_tile_tokens(a.m, a.digits, GROUPED)) {
    case 16: return launch_qlin<SRC, ND, 16, GROUPED>(a, st, err, errlen);
    case 32: return launch_qlin<SRC, ND, 32, GROUPED>(a, st, err, errlen);
    case 64: return launch_qlin<SRC, ND, 64, GROUPED>(a, st, err, errlen);
    default:
      if constexpr (ND == 1 && !GROUPED) return launch_qlin<SRC, ND, 128, GROUPED>(a, st, err, errlen);
      return -1;
  }
}

}  // namespace bl

using namespace bl;

extern "C" int bl_qlin_tile_tokens(int m) { return qlin_tile_tokens(m, 3, false); }

// Work is dealt out in units of (row tile, token tile, k-split); the SMs take them lap by lap.  A lap
// costs its k-blocks plus about two of hand-over, and every split adds a slab to write and to read.
extern "C" int bl_qlin_splits(int n, int k, int m, int digits, int grouped) {
  const int tb = qlin_tile_tokens(m, digits, grouped != 0);
  const int tiles = ((n + kQRows - 1) / kQRows) * ((m + tb - 1) / tb), kb = (k + kQK - 1) / kQK, sms = sm_count();
  int best = 1;
  double cost = 1e30;
  for (int s = 1; s <= 16 && s <= kb; ++s) {
    const int per = (kb + s - 1) / s;
    if ((kb + per - 1) / per != s) continue;  // an empty split
    const int laps = (tiles * s + sms - 1) / sms;
    const double c = laps * (per + 1.0) + (s > 1 ? 2.0 + 0.25 * s : 0.0);
    if (c < cost - 1e-9) {
      cost = c;
      best = s;
    }
  }
  return best;
}

extern "C" size_t bl_quant_digits_bytes(int m, int k) {
  const int tb = bl_qlin_tile_tokens(m);
  return size_t((m + tb - 1) / tb) * 3 * tb * size_t(k);
}

extern "C" size_t bl_quant_digits_xs_bytes(int m) { return size_t(m) * (sizeof(float) + kDigChunks); }

extern "C" int bl_quant_digits(const void* x, int m, int ldx, int k, int permute, void* xq, void* xs, void* stream,
                               char* err, size_t errlen) {
  if (!x || !xq || !xs || m < 1 || k < 8 || (k & 7) || k > 8 * kDigVec * kDigThreads || (ldx & 7) ||
      (reinterpret_cast<uintptr_t>(x) & 15u)) {
    set_err(err, errlen, "barlink: quant_digits needs 16-byte aligned rows and K a multiple of 8, at most %d",
            8 * kDigVec * kDigThreads);
    return -1;
  }
  auto go = [&](auto kern, int blocks = 1) {
    return launch_k(kern, dim3(m * blocks), dim3(kDigThreads), 0, static_cast<cudaStream_t>(stream),
                    static_cast<const __nv_bfloat16*>(x), ldx, k, bl_qlin_tile_tokens(m), static_cast<int8_t*>(xq),
                    static_cast<float*>(xs));
  };
  // vectors of a thread: a row of up to 4096 elements in one, with as little code as that takes (the code of a
  // kernel this short comes from L2 or beyond on every launch)
  const int vpt = (k / 8 + kDigThreads - 1) / kDigThreads;
  cudaError_t e;
  // a cluster for a row of more than 8192 elements, as long as there is an SM for every block (a cluster of two for 5120
  // elements took 3.9 us between the linears around it, one block with two vectors a thread 3.2)
  if (vpt > 2 && m * (vpt <= 4 ? 4 : 8) <= sm_count()) {
    if (vpt <= 4) e = permute ? go(k_quant_digits_cluster<true, 4>, 4) : go(k_quant_digits_cluster<false, 4>, 4);
    else e = permute ? go(k_quant_digits_cluster<true, 8>, 8) : go(k_quant_digits_cluster<false, 8>, 8);
  } else if (vpt <= 1) e = permute ? go(k_quant_digits<true, 1>) : go(k_quant_digits<false, 1>);
  else if (vpt <= 2) e = permute ? go(k_quant_digits<true, 2>) : go(k_quant_digits<false, 2>);
  else if (vpt <= 5) e = permute ? go(k_quant_digits<true, 5>) : go(k_quant_digits<false, 5>);
  else e = permute ? go(k_quant_digits<true, kDigVec>) : go(k_quant_digits<false, kDigVec>);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: quant_digits launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_rmsnorm_digits(const void* x, const void* residual, const void* gamma, void* out, void* residual_out,
                                 int rows, int hidden, float eps, const void* partials, int nsplit, size_t slab, void* xq,
                                 void* xs, void* stream, char* err, size_t errlen) {
  const uintptr_t ends = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(residual) |
                         reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(out) |
                         reinterpret_cast<uintptr_t>(residual_out) | reinterpret_cast<uintptr_t>(partials);
  if (rows < 1 || rows > BL_QLIN_MAX_TOKENS || hidden < 8 || (hidden & 7) || hidden > 16 * kDigThreads || (!x && !partials) ||
      !gamma || !out || !xq || !xs || (ends & 15u)) {
    set_err(err, errlen, "barlink: rmsnorm_digits is for 1..%d rows of up to %d elements, a multiple of 8, on 16-byte boundaries",
            BL_QLIN_MAX_TOKENS, 16 * kDigThreads);
    return -1;
  }
  auto go = [&](auto kern) {
    return launch_k(kern, dim3(rows), dim3(kDigThreads), 0, static_cast<cudaStream_t>(stream), static_cast<const uint4*>(x),
                    static_cast<const uint4*>(residual), static_cast<const uint4*>(gamma), static_cast<uint4*>(out),
                    static_cast<uint4*>(residual_out), hidden / 8, eps, static_cast<const float*>(partials), nsplit, slab,
                    bl_qlin_tile_tokens(rows), static_cast<int8_t*>(xq), static_cast<float*>(xs));
  };
  cudaError_t e = hidden <= 8 * kDigThreads ? go(k_rmsnorm_digits<1>) : go(k_rmsnorm_digits<2>);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: rmsnorm_digits launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_slab_finish(const blSlabFinishArgs* a, void* stream, char* err, size_t errlen) {
  if (!a || !a->slabs || !a->out || a->nsplit < 1 || a->m < 1 || a->n < 1 || a->pitch < a->n || (a->pitch & 7) ||
      (reinterpret_cast<uintptr_t>(a->slabs) & 15u)) {
    set_err(err, errlen, "barlink: slab_finish needs slabs on a 16-byte boundary with a pitch of a multiple of 8 that holds n");
    return -1;
  }
  const size_t total8 = size_t(a->m) * (a->pitch / 8);
  cudaError_t e = launch_k(k_slab_finish, dim3(unsigned((total8 + 255) / 256)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), *a, total8);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: slab_finish launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}

extern "C" int bl_qlin(const blQlinArgs* a, void* stream, char* err, size_t errlen) {
  const bool grouped = a && a->scale_kind != BL_QSCALE_BF16_N;
  if (!a || !a->w || !a->xq || !a->xs || !a->scale || (!a->out && !a->slabs) || a->m < 1 || a->m > BL_QLIN_MAX_TOKENS ||
      a->n < 1 || a->k < 16 || (a->k & 15) || (a->digits != 1 && a->digits != 3)) {
    set_err(err, errlen, "barlink: qlin needs weights, activations with 1 or 3 digits, scales, an output, 1..%d tokens and K a multiple of 16",
            BL_QLIN_MAX_TOKENS);
    return -1;
  }
  if (a->digits == 3 && (!a->x || (a->ldx & 7) || (reinterpret_cast<uintptr_t>(a->x) & 15u))) {
    set_err(err, errlen, "barlink: qlin with three digits needs the 16-byte aligned rows that they were made of");
    return -1;
  }
  // 32-bit sums: |weight| <= 128, |digit| <= 128
  if (!grouped && a->k > 131072) {
    set_err(err, errlen, "barlink: qlin sums at most 131072 products per accumulator (k %d)", a->k);
    return -1;
  }
  if (grouped && (a->group_k < kQK || a->group_k % kQK || a->k % a->group_k)) {
    set_err(err, errlen, "barlink: qlin group sizes are multiples of %d that divide K", kQK);
    return -1;
  }
  if ((a->src == kChunks && (a->k % kQK || a->digits != 1 || !grouped)) ||
      (a->src == kNibbles && (a->k % kQK || a->digits != 3 || !grouped || !a->zeros || (a->n & 7)))) {
    set_err(err, errlen, "barlink: qlin: this weight form needs K a multiple of %d and group scales", kQK);
    return -1;
  }
  const int kb = (a->k + kQK - 1) / kQK;
  const int per = a->splits > 0 ? (kb + a->splits - 1) / a->splits : 0;
  if (a->splits < 1 || (kb + per - 1) / per != a->splits || (a->splits > 1 && !a->slabs)) {
    set_err(err, errlen, "barlink: qlin: %d k-splits of %d k-blocks (every split needs one, and slabs to go to)", a->splits, kb);
    return -1;
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a->src == kChunks) return launch_qlin_tb<kChunks, 1, true>(*a, st, err, errlen);
  if (a->src == kNibbles) return launch_qlin_tb<kNibbles, 3, true>(*a, st, err, errlen);
  if (grouped)
    return a->digits == 1 ? launch_qlin_tb<kRows, 1, true>(*a, st, err, errlen)
                          : launch_qlin_tb<kRows, 3, true>(*a, st, err, errlen);
  return a->digits == 1 ? launch_qlin_tb<kRows, 1, false>(*a, st, err, errlen)
                        : launch_qlin_tb<kRows, 3, false>(*a, st, err, errlen);
}
