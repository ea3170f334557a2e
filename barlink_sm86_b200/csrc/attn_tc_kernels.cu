// SPDX-License-Identifier: MIT
//
// Dense attention on the 5th-generation tensor cores (head_dim 128, bf16):
// prefill (causal, GQA) and MMDiT joint attention over packed sequences.
// The reference calls a library kernel here (flash-attn / SDPA inside
// transformers and diffusers: demos/flux2_tp/worker.py:148-160,
// demos/qwen_tp/qwen38_int8/worker.py:515-537).
//
// One CTA owns 256 query rows of one head as two 128-row tiles and walks the
// keys in tiles of 64:
//
//   warp 0      TMA producer: Q once, then a ring of K tiles and a ring of V tiles
//   warp 1      issues tcgen05.mma: S_t = Q_t K^T into TMEM (128x64 fp32, two buffers per tile),
//               O_t += P_t V into TMEM (128x128 fp32), for tiles t = 0, 1 in turn
//   warps 2-5   softmax of tile 0: every thread owns one query row (TMEM lane),
//   warps 6-9   softmax of tile 1   reads its 64 scores with tcgen05.ld, keeps the
//               running max and sum in registers, writes P (bf16) over
//               them in TMEM, from where it is the A operand of P V
//
// What bounds it: the exponentials (16 a clock and SM: 1024 cycles for 64 keys x 256 rows, as many as the
// products take) and, before S had two buffers, the chain softmax -> P V -> next S -> softmax of a tile, whose
// links added up to 2700 cycles a step.  Now S of step j + 2 is issued right behind P V of step j, so a
// tile's softmax always finds its scores; P has two buffers for the same reason, and a rescale of O waits
// for the P V before it.  S of step j + 2 goes into the columns from which P V of step j, issued just before and not waited
// for, takes P: one thread issues both, and the tensor pipe works off the products of one CTA in the order in which they are issued,
// so the scores are written behind the reads of P.  (P is written by the softmax only after s_ready of its own step, so behind
// both.)  With P in shared memory and V through a kernel that transposed it a step took the same time, so the tiles in
// shared memory do not bound it; 24 heads x 4608 tokens: 297 us with the transpose (22 of them), 269 without, 2370 cycles a step
// of an SM that always has work.  The 4096-token MMDiT forward takes 71.5 ms instead of 73.4.
// The accumulator is rescaled only when the running max has grown by more than
// 2^8 since the last rescale (the stale max is exact after the final division
// by the row sum), which takes the TMEM read-modify-write out of the loop.
//
// Every wait is bounded; a wait that runs out sets the CTA's abort word, all
// roles leave their loops, TMEM is freed and the error flag is raised.
#include <cuda_bf16.h>
#include <stdint.h>

#include "bl_ops.h"
#include "heap.h"
#include "launch.h"
#include "ptx.cuh"

namespace bl {

constexpr int kTcBM = 128;       // query rows per tile
constexpr int kTcTiles = 2;      // tiles per CTA
constexpr int kTcBKV = 64;       // keys per step
constexpr int kTcHD = 128;
constexpr int kTcStages = 4;     // K tiles and V tiles in flight, a ring each
constexpr int kTcThreads = 320;
constexpr uint32_t kTcQBytes = kTcBM * kTcHD * 2;          // 32 KiB per query tile
constexpr uint32_t kTcKBytes = kTcBKV * kTcHD * 2;         // 16 KiB
constexpr uint32_t kTcVBytes = kTcHD * kTcBKV * 2;         // 16 KiB
constexpr uint32_t kTcOffK = kTcTiles * kTcQBytes;
constexpr uint32_t kTcOffV = kTcOffK + kTcStages * kTcKBytes;
constexpr uint32_t kTcOffBar = kTcOffV + kTcStages * kTcVBytes;
constexpr uint32_t kTcSmem = kTcOffBar + 256 + 1024;       // barriers + alignment slack
static_assert(kTcSmem <= 232448, "attention tiles do not fit the shared memory of one CTA");
constexpr uint32_t kTcTmemCols = 512;                      // S of tile t, step parity p: 128 t + 64 p, P in its first half; O of tile t: 256 + 128 t
constexpr int kTcLastRowsFirst = 2;                        // in `causal`, beside 1
constexpr float kTcRescale = 8.f;                          // log2 units

__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]),
      "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]),
      "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 operations in one instruction, each rounded as its scalar form
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

// B operand of P V as V lies in memory: [key][64 columns of the head], 128-byte rows in the 128-byte swizzle, so the
// columns (N) are contiguous: eight keys are 1024 bytes (stride byte offset), the other 64 columns half a tile on
// (leading byte offset); 16 keys of a product are 2048 bytes.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t half_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(half_bytes >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
constexpr uint32_t kUmmaBMajorN = 1u << 16;  // instruction descriptor: B is N-major
// A from TMEM: a lane a row, a 32-bit column two neighbours along K
__device__ __forceinline__ void umma_f16_ts_warp(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(leader)
      : "memory");
}

__global__ void __launch_bounds__(kTcThreads, 1)
    k_attn_tc(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
              const __grid_constant__ CUtensorMap tmap_v, __nv_bfloat16* __restrict__ out,
              const int* __restrict__ cu_q, const int* __restrict__ cu_k, int nq, int nkv, int o_stride,
              float scale_log2, int causal, uint32_t* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  uint64_t* bars = reinterpret_cast<uint64_t*>(gen + kTcOffBar);
  uint64_t* q_full = bars;             // 1
  uint64_t* k_full = bars + 1;         // kTcStages each
  uint64_t* k_empty = k_full + kTcStages;
  uint64_t* v_full = k_empty + kTcStages;
  uint64_t* v_empty = v_full + kTcStages;
  uint64_t* s_ready = v_empty + kTcStages;  // [tile][step parity]
  uint64_t* p_ready = s_ready + 4;     // [tile][step parity]
  uint64_t* pv_done = p_ready + 4;     // [tile], one phase per step
  uint64_t* o_final = pv_done + 2;     // [tile]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_final + 2);
  volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(o_final + 3);
  static_assert((1 + 4 * kTcStages + 14) * 8 <= 256, "barriers");

  // cu_q / cu_k may come from the kernel just before this one
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Causal: the later rows have more keys, so their blocks are dealt out first, over all heads and sequences
  // (8 x 1024, 28 heads on 4: 126.7 -> 123.7 us).
  const bool last_first = causal & kTcLastRowsFirst;
  const int b = last_first ? blockIdx.y : blockIdx.z, head = last_first ? blockIdx.x : blockIdx.y, kvh = head / (nq / nkv);
  const int rblock = last_first ? int(gridDim.z - 1 - blockIdx.z) : int(blockIdx.x);
  const int q0 = cu_q[b], lq = cu_q[b + 1] - q0;
  const int k0 = cu_k[b], lk = cu_k[b + 1] - k0;
  const int row0 = rblock * (kTcTiles * kTcBM);   // first query row of this CTA in its sequence
  if (row0 >= lq) return;
  const int off = lk - lq;                             // causal: key j visible to query i iff j <= i + off
  int kv_end = lk;
  if (causal) {
    const int last = min(lq, row0 + kTcTiles * kTcBM) - 1;
    kv_end = max(0, min(lk, last + off + 1));
  }
  const int n_steps = (kv_end + kTcBKV - 1) / kTcBKV;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    for (int t = 0; t < kTcTiles; ++t) {
      for (int p = 0; p < 2; ++p) {
        mbar_init(&s_ready[2 * t + p], 1);
        mbar_init(&p_ready[2 * t + p], kTcBM);
      }
      mbar_init(&pv_done[t], 1);
      mbar_init(&o_final[t], 1);
    }
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTcTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (lane == 0 && n_steps > 0) {
      mbar_expect_tx(q_full, kTcTiles * kTcQBytes);
      for (int t = 0; t < kTcTiles; ++t)
        for (int h = 0; h < 2; ++h)
          tma_load_2d_hint_s(base + t * kTcQBytes + h * (kTcQBytes / 2), &tmap_q, smem_u32(q_full),
                             head * kTcHD + h * 64, q0 + row0 + t * kTcBM, kHintEvictFirst);
      int stage = 0;
      uint32_t phase = 0;
      int k_issued = 0, v_issued = 0;
      for (int j = 0; j < n_steps; ++j) {
        if (!mbar_wait_bounded(&k_empty[stage], phase ^ 1u, s_abort)) break;
        mbar_expect_tx(&k_full[stage], kTcKBytes);
        for (int h = 0; h < 2; ++h)
          tma_load_2d_hint_s(base + kTcOffK + stage * kTcKBytes + h * (kTcKBytes / 2), &tmap_k, smem_u32(&k_full[stage]),
                             kvh * kTcHD + h * 64, k0 + j * kTcBKV, kHintEvictLast);
        ++k_issued;
        if (!mbar_wait_bounded(&v_empty[stage], phase ^ 1u, s_abort)) break;
        mbar_expect_tx(&v_full[stage], kTcVBytes);
        for (int h = 0; h < 2; ++h)
          tma_load_2d_hint_s(base + kTcOffV + stage * kTcVBytes + h * (kTcVBytes / 2), &tmap_v, smem_u32(&v_full[stage]),
                             kvh * kTcHD + h * 64, k0 + j * kTcBKV, kHintEvictLast);
        ++v_issued;
        if (++stage == kTcStages) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (*s_abort) {
        // leaving early: let the copies still in flight land before the CTA exits
        auto drain = [&](uint64_t* full, int issued) {
          for (int j = max(0, issued - kTcStages); j < issued; ++j)
            for (uint32_t p = 0; p < (1u << 20); ++p)
              if (mbar_try_wait(&full[j % kTcStages], uint32_t(j / kTcStages) & 1u)) break;
        };
        drain(k_full, k_issued);
        drain(v_full, v_issued);
        for (uint32_t p = 0; p < (1u << 20); ++p)
          if (mbar_try_wait(q_full, 0)) break;
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------
    if (n_steps > 0) {
      const uint32_t leader = elect_leader();
      const uint32_t idesc_s = umma_idesc_f16(kTcBM, kTcBKV, 1);
      const uint32_t idesc_o = umma_idesc_f16(kTcBM, kTcHD, 1) | kUmmaBMajorN;
      // S of a step with parity p, from K stage ks0
      auto issue_s = [&](int t, int p, int kst) {
        const uint64_t dq = umma_desc_k_sw128(base + t * kTcQBytes), dk = umma_desc_k_sw128(base + kTcOffK + kst * kTcKBytes);
#pragma unroll
        for (int ks = 0; ks < kTcHD / 16; ++ks)
          umma_f16_ss_warp(leader, tmem_base + uint32_t(t * 128 + p * kTcBKV),
                           dq + uint64_t((ks >> 2) * (kTcQBytes / 32) + 2 * (ks & 3)),
                           dk + uint64_t((ks >> 2) * (kTcKBytes / 32) + 2 * (ks & 3)), idesc_s, ks > 0 ? 1u : 0u);
        umma_commit_warp(leader, &s_ready[2 * t + p]);
      };
      auto issue_pv = [&](int t, int p, int vst, bool acc) {
        const uint64_t dv = umma_desc_mn_sw128(base + kTcOffV + vst * kTcVBytes, kTcVBytes / 2);
#pragma unroll
        for (int ks = 0; ks < kTcBKV / 16; ++ks)
          umma_f16_ts_warp(leader, tmem_base + 256u + uint32_t(t * kTcHD), tmem_base + uint32_t(t * 128 + p * kTcBKV + 8 * ks),
                           dv + uint64_t(128 * ks), idesc_o, (acc || ks > 0) ? 1u : 0u);
        umma_commit_warp(leader, &pv_done[t]);
      };
      bool ok = mbar_wait_bounded_warp(q_full, 0, s_abort);
      // scores of the first two steps
      int kst = 0, vst = 0;
      uint32_t kphase = 0, vphase = 0;
      for (int j = 0; j < min(2, n_steps) && ok; ++j) {
        ok = mbar_wait_bounded_warp(&k_full[kst], kphase, s_abort);
        if (!ok) break;
        tc_fence_after_sync();
        issue_s(0, j, kst);
        issue_s(1, j, kst);
        umma_commit_warp(leader, &k_empty[kst]);
        ++kst;
      }
      for (int j = 0; j < n_steps && ok; ++j) {
        const int p = j & 1;
        const bool more = j + 2 < n_steps;
#pragma unroll
        for (int t = 0; t < kTcTiles; ++t) {
          bool here = mbar_wait_bounded(&p_ready[2 * t + p], uint32_t(j >> 1) & 1u, s_abort);
          // the next tiles are there long before the probabilities
          if (t == 0) {
            here = here && mbar_wait_bounded(&v_full[vst], vphase, s_abort);
            if (more) here = here && mbar_wait_bounded(&k_full[kst], kphase, s_abort);
          }
          ok = __all_sync(0xffffffffu, here);
          if (!ok) break;
          if (t == 0 && (j + 1) * kTcBKV > lk) {
            // rows beyond the sequence are another's: their probabilities are zero, their values may be infinite
            for (int i = lane + (lk - j * kTcBKV) * 16; i < kTcBKV * 16; i += 32)
              asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(base + kTcOffV + vst * kTcVBytes +
                                                                        ((i >> 3) & 1) * (kTcVBytes / 2) + (i >> 4) * 128 + (i & 7) * 16),
                           "r"(0)
                           : "memory");
            fence_proxy_async_smem();
            __syncwarp();
          }
          tc_fence_after_sync();
          issue_pv(t, p, vst, j > 0);
          if (more) issue_s(t, p, kst);
          // (a wait for the last phase of pv_done could be answered by the last but two)
          if (j + 1 == n_steps) umma_commit_warp(leader, &o_final[t]);
        }
        if (!ok) break;
        umma_commit_warp(leader, &v_empty[vst]);
        if (++vst == kTcStages) {
          vst = 0;
          vphase ^= 1u;
        }
        if (more) {
          umma_commit_warp(leader, &k_empty[kst]);
          if (++kst == kTcStages) {
            kst = 0;
            kphase ^= 1u;
          }
        }
      }
    }
  } else {
    // ------------------------------ softmax -------------------------------
    const int t = (warp - 2) >> 2;                 // tile of this warp group
    const int quarter = warp & 3;                  // TMEM lanes this warp may touch
    const int row = quarter * 32 + lane;           // row inside the tile
    const int qi = row0 + t * kTcBM + row;         // query index inside the sequence
    const uint32_t lane_addr = tmem_base + (uint32_t(quarter * 32) << 16);
    const uint32_t s_tile = lane_addr + uint32_t(t * 128);
    const uint32_t o_addr = lane_addr + 256u + uint32_t(t * kTcHD);
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n_steps; ++j) {
      const int p = j & 1;
      if (!mbar_wait_bounded_warp(&s_ready[2 * t + p], uint32_t(j >> 1) & 1u, s_abort)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      const uint32_t s_addr = s_tile + uint32_t(p * kTcBKV);
      float s[kTcBKV];
      {
        uint32_t r0[32], r1[32];
        tmem_ld_32x32(s_addr, r0);
        tmem_ld_32x32(s_addr + 32, r1);
        tmem_ld_wait();
        const float2 sl = make_float2(scale_log2, scale_log2);
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          const float2 a = mul2(make_float2(__uint_as_float(r0[c]), __uint_as_float(r0[c + 1])), sl);
          const float2 b = mul2(make_float2(__uint_as_float(r1[c]), __uint_as_float(r1[c + 1])), sl);
          s[c] = a.x;
          s[c + 1] = a.y;
          s[c + 32] = b.x;
          s[c + 33] = b.y;
        }
      }
      const int kbase = j * kTcBKV;
      const int lim = causal ? min(lk, qi + off + 1) : lk;   // keys [0, lim) are visible to this row
      if (kbase + kTcBKV > lim) {
#pragma unroll
        for (int c = 0; c < kTcBKV; ++c)
          if (kbase + c >= lim) s[c] = -INFINITY;
      }
      // four chains: the maximum is on the way from the scores to everything else
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int c = 4; c < kTcBKV; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], s[c]);
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const float m_new = fmaxf(m_used, mx);
      const bool grow = m_new > m_used + kTcRescale;          // also true on the first finite max
      if (__any_sync(0xffffffffu, grow)) {
        const float alpha = (m_new == -INFINITY) ? 1.f : ex2_approx(m_used - m_new);
        if (j > 0) {
          // P V of the previous step may still be running.  Parity tells its phase, j - 1, apart from its
          // neighbours: phase j needs this warp's own P; phase j - 2 is over and its arrival made, since the arrival
          // for S of step j, which this warp has seen, was committed behind it by the same thread, to the same
          // tensor pipe, which completes in order, with the products of S in between.  (A barrier for each step
          // parity, which would need less of that, cost 1 % at 24 heads x 4608 tokens.)
          if (!mbar_wait_bounded_warp(&pv_done[t], uint32_t(j - 1) & 1u, s_abort)) {
            ok = false;
            break;
          }
          tc_fence_after_sync();
#pragma unroll 1
          for (int c0 = 0; c0 < kTcHD; c0 += 32) {
            uint32_t r[32];
            tmem_ld_32x32(o_addr + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; ++c) r[c] = __float_as_uint(__uint_as_float(r[c]) * alpha);
            tmem_st_32x32(o_addr + c0, r);
          }
          tmem_st_wait();
        }
        l *= alpha;
        m_used = m_new;
      }
      const float mref = (m_used == -INFINITY) ? 0.f : m_used;
      const float2 neg = make_float2(-mref, -mref);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      uint32_t pk[kTcBKV / 2];
#pragma unroll
      for (int c = 0; c < kTcBKV; c += 2) {
        const float2 x = add2(make_float2(s[c], s[c + 1]), neg);
        const float2 e = make_float2(ex2_approx(x.x), ex2_approx(x.y));
        sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], e);
        pk[c >> 1] = pack_bf16x2(e.x, e.y);
      }
      sum[0] = add2(sum[0], sum[1]);
      l += sum[0].x + sum[0].y;
      tmem_st_32x32(s_addr, pk);  // over the scores that it was made of
      tmem_st_wait();
      tc_fence_before_sync();
      mbar_arrive(&p_ready[2 * t + p]);
    }
    // ------------------------------ output --------------------------------
    const bool valid = qi < lq;
    __nv_bfloat16* orow = out + size_t(q0 + qi) * o_stride + head * kTcHD;
    if (n_steps == 0) {
      if (valid)
        for (int c = 0; c < kTcHD; c += 8) *reinterpret_cast<uint4*>(orow + c) = make_uint4(0, 0, 0, 0);
    } else if (ok && mbar_wait_bounded_warp(&o_final[t], 0, s_abort)) {
      tc_fence_after_sync();
      const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
      for (int c0 = 0; c0 < kTcHD; c0 += 32) {
        uint32_t r[32];
        tmem_ld_32x32(o_addr + c0, r);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            *reinterpret_cast<uint4*>(orow + c0 + c) = make_uint4(
                pack_bf16x2(__uint_as_float(r[c]) * inv, __uint_as_float(r[c + 1]) * inv),
                pack_bf16x2(__uint_as_float(r[c + 2]) * inv, __uint_as_float(r[c + 3]) * inv),
                pack_bf16x2(__uint_as_float(r[c + 4]) * inv, __uint_as_float(r[c + 5]) * inv),
                pack_bf16x2(__uint_as_float(r[c + 6]) * inv, __uint_as_float(r[c + 7]) * inv));
          }
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, kTcTmemCols);
  }
  if (threadIdx.x == 0 && *s_abort && err) *err = 1u;
}

}  // namespace bl

using namespace bl;

extern "C" size_t bl_attn_tc_scratch_bytes(int, int, int) { return 0; }

// Tensor-core dense attention.  `total_q`: rows of q; `total_k`: rows that k and v have (at least cu_k[batch]).
extern "C" int bl_attn_fwd_tc(const void* q, const void* k, const void* v, void* out, const int* cu_q,
                              const int* cu_k, int batch, int max_q, int max_k, int total_q, int total_k,
                              int nq, int nkv, int hd, int q_stride, int k_stride, int v_stride,
                              int o_stride, float scale, int causal, void* /* vt */, void* err_flag, void* stream,
                              char* err, size_t errlen) {
  if (hd != kTcHD || nkv < 1 || nq % nkv) {
    set_err(err, errlen, "barlink: tensor-core attention is built for head_dim %d and nq %% nkv == 0", kTcHD);
    return -1;
  }
  if ((q_stride | k_stride | v_stride | o_stride) & 7) {
    set_err(err, errlen, "barlink: attention needs token strides that are multiples of 8 elements");
    return -1;
  }
  if (batch < 1 || max_q < 1 || max_k < 1) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CUtensorMap tq, tk, tv;
  if (make_tmap_kmajor(q, uint64_t(total_q), uint64_t(nq) * kTcHD, uint64_t(q_stride), kTcBM, 2, &tq, err, errlen) ||
      make_tmap_kmajor(k, uint64_t(total_k), uint64_t(nkv) * kTcHD, uint64_t(k_stride), kTcBKV, 2, &tk, err, errlen) ||
      make_tmap_kmajor(v, uint64_t(total_k), uint64_t(nkv) * kTcHD, uint64_t(v_stride), kTcBKV, 2, &tv, err, errlen))
    return -1;
  static bool attr[64] = {};
  cudaError_t e = allow_smem(reinterpret_cast<const void*>(k_attn_tc), int(kTcSmem), attr);
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: tensor-core attention shared memory opt-in failed: %s", cudaGetErrorString(e));
    return -1;
  }
  const unsigned rblocks = unsigned((max_q + kTcTiles * kTcBM - 1) / (kTcTiles * kTcBM));
  // (a grid has at most 65535 blocks along y and z, and max_q may be any bound of the lengths)
  const bool last_first = causal && rblocks <= 65535;
  const dim3 grid = last_first ? dim3(nq, batch, rblocks) : dim3(rblocks, nq, batch);
  e = launch_k(k_attn_tc, grid, dim3(kTcThreads), kTcSmem, st, tq, tk, tv, static_cast<__nv_bfloat16*>(out), cu_q, cu_k, nq,
               nkv, o_stride, scale * 1.4426950408889634f, causal ? (last_first ? 1 | kTcLastRowsFirst : 1) : 0,
               static_cast<uint32_t*>(err_flag));
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_err(err, errlen, "barlink: tensor-core attention launch failed: %s", cudaGetErrorString(e));
    return -1;
  }
  return 0;
}
