// SPDX-License-Identifier: MIT
//
// Second half of the `_C` binding: single-process forms of the collectives
// (ranks that share a GPU), dense attention, W8A16 and the fused
// GEMM+collective tensor-parallel linears.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/extension.h>

#include <algorithm>
#include <map>

#include "backend.h"
#include "bl_core.h"
#include "bl_ops.h"
#include "heap.h"

namespace py = pybind11;

// (Numbers go into the messages of TORCH_CHECK as text, std::to_string: put into a stream by an extension, an integer
// crashes the process where the toolchain's C++ library and the one that torch brings differ.)

namespace {

constexpr size_t kErr = 512;
#define BL_CHECK(expr)                                                 \
  do {                                                                 \
    char _e[kErr] = {0};                                               \
    char* err = _e;                                                    \
    size_t errlen = kErr;                                              \
    (void)err; (void)errlen;                                           \
    int _rc = (expr);                                                  \
    TORCH_CHECK(_rc == 0, _e[0] ? _e : "barlink: call failed: " #expr); \
  } while (0)

blCtx* ctx_or_throw() {
  blCtx* c = blpg::global_ctx();
  TORCH_CHECK(c != nullptr, "barlink: not initialised -- call init(devices, pool_mb) or init_peer(...) first");
  return c;
}

int kind_code(const std::string& k) {
  if (k == "allreduce") return 0;
  if (k == "reduce_scatter") return 1;
  if (k == "allgather") return 2;
  if (k == "broadcast") return 3;
  if (k == "allreduce_rmsnorm") return 4;
  if (k == "barrier") return 5;
  TORCH_CHECK(false, "barlink: unknown collective '", k, "'");
}
int algo_code2(const std::string& a) {
  if (a == "oneshot") return BL_ALGO_ONESHOT;
  if (a == "twoshot") return BL_ALGO_TWOSHOT;
  if (a == "nvls") return BL_ALGO_NVLS;
  return BL_ALGO_AUTO;
}

// one tensor per rank in every list; lists may be empty when the collective
// does not use them
void sp_collective(const std::string& kind, std::vector<at::Tensor> ins, std::vector<at::Tensor> outs,
                   std::vector<at::Tensor> aux_in, std::vector<at::Tensor> aux_out,
                   std::vector<at::Tensor> gamma, const std::string& algo, int root, double eps) {
  blCtx* c = ctx_or_throw();
  const int world = bl_world(c);
  const int k = kind_code(kind);
  auto ptrs = [&](std::vector<at::Tensor>& v, const char* name) {
    std::vector<void*> p;
    if (v.empty()) return p;
    TORCH_CHECK(int(v.size()) == world, "barlink: ", name, " needs one tensor per rank (",
                std::to_string(world), ")");
    for (auto& t : v) {
      TORCH_CHECK(t.is_cuda() && t.is_contiguous(), "barlink: ", name, " tensors must be contiguous CUDA tensors");
      p.push_back(t.data_ptr());
    }
    return p;
  };
  std::vector<void*> pi = ptrs(ins, "ins"), po = ptrs(outs, "outs"), pai = ptrs(aux_in, "aux_in"),
                     pao = ptrs(aux_out, "aux_out"), pg = ptrs(gamma, "gamma");
  std::vector<void*> streams(world, nullptr);
  int dtype = BL_DTYPE_U8;
  size_t bytes = 0;
  int rows = 0, hidden = 0;
  if (k != 5) {
    TORCH_CHECK(!ins.empty() && !outs.empty(), "barlink: ins and outs are required");
    dtype = blpg::dtype_code(ins[0].scalar_type());
    TORCH_CHECK(dtype >= 0, "barlink: unsupported dtype ", ins[0].scalar_type());
    bytes = (k == 1) ? outs[0].nbytes() : ins[0].nbytes();
    if (k == 4) {
      hidden = int(ins[0].size(-1));
      rows = int(ins[0].numel() / hidden);
    }
    for (int r = 0; r < world; ++r)
      streams[r] = at::cuda::getCurrentCUDAStream(ins[r].device().index()).stream();
  } else {
    for (int r = 0; r < world; ++r) streams[r] = at::cuda::getCurrentCUDAStream().stream();
  }
  py::gil_scoped_release nogil;
  BL_CHECK(bl_sp_collective(c, k, pi.empty() ? nullptr : pi.data(), po.empty() ? nullptr : po.data(),
                            pai.empty() ? nullptr : pai.data(), pao.empty() ? nullptr : pao.data(),
                            pg.empty() ? nullptr : pg.data(), bytes, dtype, algo_code2(algo), root,
                            rows, hidden, float(eps), streams.data(), err, errlen));
}

void sp_sendrecv(int src, int dst, const at::Tensor& in, const at::Tensor& out) {
  blCtx* c = ctx_or_throw();
  TORCH_CHECK(in.is_cuda() && out.is_cuda() && in.is_contiguous() && out.is_contiguous() &&
                  in.nbytes() == out.nbytes(),
              "barlink: sp_sendrecv needs contiguous CUDA tensors of equal size");
  void* st = at::cuda::getCurrentCUDAStream(in.device().index()).stream();
  py::gil_scoped_release nogil;
  BL_CHECK(bl_sp_sendrecv(c, src, dst, in.data_ptr(), out.data_ptr(), in.nbytes(), st, err, errlen));
}

// q [T, nq, hd], k / v [Tk, nkv, hd] (token stride free, heads and dims dense)
at::Tensor& attn_err(int dev) {
  static std::map<int, at::Tensor> m;
  auto it = m.find(dev);
  if (it != m.end()) return it->second;
  return m.emplace(dev, at::zeros({4}, at::TensorOptions().device(at::kCUDA, dev).dtype(at::kInt))).first->second;
}
int attn_error_flag(int dev) { return attn_err(dev).cpu()[0].item<int>(); }

// max_k > 0 (longest key sequence) selects the tcgen05 kernel; BL_ATTN_TC=0 keeps the mma.sync kernel
at::Tensor attn_fwd(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v,
                    const at::Tensor& cu_q, const at::Tensor& cu_k, int max_q, double scale,
                    bool causal, int max_k) {
  auto chk = [](const at::Tensor& t, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 3 && t.stride(2) == 1 &&
                    t.stride(1) == t.size(2),
                "barlink: ", name, " must be a bfloat16 CUDA tensor [tokens, heads, head_dim] with dense heads");
  };
  chk(q, "q");
  chk(k, "k");
  chk(v, "v");
  TORCH_CHECK(cu_q.is_cuda() && cu_q.scalar_type() == at::kInt && cu_k.is_cuda() &&
                  cu_k.scalar_type() == at::kInt && cu_q.numel() == cu_k.numel() && cu_q.numel() >= 2,
              "barlink: cu_q / cu_k must be int32 CUDA tensors of batch + 1 entries");
  const int batch = int(cu_q.numel()) - 1;
  const int nq = int(q.size(1)), nkv = int(k.size(1)), hd = int(q.size(2));
  TORCH_CHECK(k.size(2) == hd && v.size(2) == hd && v.size(1) >= nkv,
              "barlink: k and v must have q's head_dim, and v a head for each of k's");
  at::Tensor out = at::empty({q.size(0), nq, hd}, q.options());
  c10::cuda::CUDAGuard guard(q.device());
  void* st = at::cuda::getCurrentCUDAStream(q.device().index()).stream();
  static const bool tc_on = [] {
    const char* e = getenv("BL_ATTN_TC");
    return !(e && e[0] == '0');
  }();
  if (q.size(0) > 0 && tc_on && max_k > 0 && hd == 128 && v.size(0) > 0) {
    // K and V are fetched in boxes of 64 rows whose last one reaches beyond its sequence, so the tensor maps end with the
    // shorter of the two (K may be a longer preallocated buffer).  A map knows no rows that lie on one another, and the
    // stride of a single row says nothing.
    const int rows = int(std::min(k.size(0), v.size(0)));
    const at::Tensor vm = v.size(0) > 1 && v.stride(0) == 0 ? v.contiguous() : v;
    const int v_stride = int(v.size(0) > 1 ? vm.stride(0) : vm.size(1) * hd);
    BL_CHECK(bl_attn_fwd_tc(q.data_ptr(), k.data_ptr(), vm.data_ptr(), out.data_ptr(), cu_q.data_ptr<int>(),
                            cu_k.data_ptr<int>(), batch, max_q, max_k, int(q.size(0)), rows, nq, nkv,
                            hd, int(q.stride(0)), int(k.stride(0)), v_stride, nq * hd, float(scale),
                            causal ? 1 : 0, nullptr, attn_err(q.device().index()).data_ptr(), st, err,
                            errlen));
    return out;
  }
  if (q.size(0) > 0)
    BL_CHECK(bl_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(),
                         cu_q.data_ptr<int>(), cu_k.data_ptr<int>(), batch, max_q, nq, nkv, hd,
                         int(q.stride(0)), int(k.stride(0)), int(v.stride(0)), nq * hd, float(scale),
                         causal ? 1 : 0, st, err, errlen));
  return out;
}

void check_bf16x(const at::Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.is_contiguous() && t.scalar_type() == at::kBFloat16, "barlink: ", name,
              " must be a contiguous bfloat16 CUDA tensor");
}

// kernels that read whole vectors: a tensor that starts between two of them (a view) is copied
at::Tensor on_16_bytes(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0 ? t : t.clone(); }

struct W8Scratch {
  at::Tensor ws, counters, err_flag;
};
W8Scratch& w8_scratch(int dev) {
  static std::map<int, W8Scratch> m;
  auto it = m.find(dev);
  if (it != m.end()) return it->second;
  auto o = at::TensorOptions().device(at::kCUDA, dev);
  W8Scratch s;
  s.ws = at::empty({int64_t(64) << 20}, o.dtype(at::kByte));
  s.counters = at::zeros({16384}, o.dtype(at::kInt));
  s.err_flag = at::zeros({4}, o.dtype(at::kInt));
  return m.emplace(dev, s).first->second;
}

// y = x @ (wq * scale[:, None]).T (+ bias): bf16 activations, int8 per-channel
// weights widened to bf16 inside the tcgen05 main loop (<= 256 tokens); more
// tokens widen the weight once and use the bf16 GEMM.
// bf16 group scales [n, groups] -> (row_max bf16 [n], rel fp16 [n, groups]): done once per weight
std::tuple<at::Tensor, at::Tensor> w8_group_scales(const at::Tensor& scales) {
  check_bf16x(scales, "scales");
  TORCH_CHECK(scales.dim() == 2, "barlink: group scales must be [n, groups]");
  const int n = int(scales.size(0)), groups = int(scales.size(1));
  at::Tensor row = at::empty({n}, scales.options());
  at::Tensor rel = at::empty({n, groups}, scales.options().dtype(at::kHalf));
  c10::cuda::CUDAGuard guard(scales.device());
  void* st = at::cuda::getCurrentCUDAStream(scales.device().index()).stream();
  BL_CHECK(bl_w8_group_scales(scales.data_ptr(), n, groups, row.data_ptr(), rel.data_ptr(), st, err, errlen));
  return {row, rel};
}

// ---- decode linears on quantised weights: int8 weights against int8 digits of the activations ----
struct QWeight {
  const void* w;
  int src, n, k;
  int scale_kind;
  const void* scale;
  const void* row_scale = nullptr;
  int group_k = 0;
  const void* zeros = nullptr;
  // digits that the norm in front has left (bl_rmsnorm_digits), both or neither
  c10::optional<at::Tensor> xq, xs;
};
// digits that a caller hands in for x; `used`: the product reads digits
void check_digits(const at::Tensor& x, int k, bool used, const c10::optional<at::Tensor>& xq, const c10::optional<at::Tensor>& xs) {
  if (!xq && !xs) return;
  TORCH_CHECK(used, "barlink: digits are for bf16 activations of 1..", std::to_string(BL_QLIN_MAX_TOKENS),
              " 16-byte aligned rows of at most 32768 elements");
  const int m = int(x.size(0));
  auto ok = [&](const c10::optional<at::Tensor>& t, at::ScalarType type, size_t bytes) {
    return t && t->device() == x.device() && t->scalar_type() == type && t->is_contiguous() && t->nbytes() == bytes;
  };
  TORCH_CHECK(ok(xq, at::kChar, bl_quant_digits_bytes(m, k)) && ok(xs, at::kFloat, bl_quant_digits_xs_bytes(m)) &&
                  (reinterpret_cast<uintptr_t>(xq->data_ptr()) & 15u) == 0,
              "barlink: digits do not belong to these activations (see rmsnorm_digits)");
}
// a shape that bl_qlin takes and (three digits) bf16 rows that bl_quant_digits can read; per-channel sums are
// 32-bit over all of K
bool qlin_takes(const at::Tensor& x, int k, bool act_int8, bool grouped = false) {
  if (x.size(0) < 1 || x.size(0) > BL_QLIN_MAX_TOKENS || k % 16 != 0) return false;
  return act_int8 ? grouped || k <= 131072
                  : k <= 32768 && x.stride(0) % 8 == 0 && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15u) == 0;
}
// y = activations (xq, xs: int8 rows, or three digit planes) times q.  want_slabs: fp32 [splits, m, n]
// when the shape wants a k-split (bias is then the consumer's), else bf16 [m, n].  like: options of x.
// x: the bf16 activations (three digit planes are made of them).
at::Tensor qlin_product(const at::Tensor& x, const at::Tensor& xq, const at::Tensor& xs, int m, int digits, const QWeight& q,
                        const c10::optional<at::Tensor>& bias, bool silu_mul, int splits, bool want_slabs,
                        const at::TensorOptions& like, void* err_flag, void* st) {
  if (bias) {
    check_bf16x(*bias, "bias");
    TORCH_CHECK(bias->numel() == q.n, "barlink: bias must have n entries");
  }
  if (splits <= 0) splits = bl_qlin_splits(q.n, q.k, m, digits, q.scale_kind != BL_QSCALE_BF16_N);
  // bl_slab_finish reads slabs whose pitch is a multiple of 8
  if (!want_slabs && q.n % 8 != 0) splits = 1;
  const int kb = (q.k + 127) / 128, per = (kb + splits - 1) / splits;
  splits = (kb + per - 1) / per;
  blQlinArgs a;
  memset(&a, 0, sizeof(a));
  a.w = q.w; a.src = q.src; a.n = q.n; a.k = q.k;
  a.xq = xq.data_ptr(); a.xs = xs.data_ptr();
  a.m = m; a.digits = digits;
  a.x = x.data_ptr();
  a.ldx = int(x.stride(0));
  a.scale_kind = q.scale_kind; a.scale = q.scale; a.row_scale = q.row_scale; a.group_k = q.group_k; a.zeros = q.zeros;
  a.splits = splits;
  a.err_flag = err_flag;
  at::Tensor slabs, out;
  if (splits > 1) {
    slabs = at::empty({splits, m, q.n}, like.dtype(at::kFloat));
    a.slabs = slabs.data_ptr();
  } else {
    out = at::empty({m, silu_mul ? q.n / 2 : q.n}, like);
    a.out = out.data_ptr();
    a.ldo = int(out.size(1));
    a.bias = bias ? bias->data_ptr() : nullptr;
    a.silu_mul = silu_mul ? 1 : 0;
  }
  BL_CHECK(bl_qlin(&a, st, err, errlen));
  if (splits == 1) return out;
  if (want_slabs) return slabs;
  out = at::empty({m, silu_mul ? q.n / 2 : q.n}, like);
  blSlabFinishArgs f;
  memset(&f, 0, sizeof(f));
  f.slabs = slabs.data_ptr();
  f.nsplit = splits; f.m = m; f.n = f.pitch = q.n;
  f.bias = bias ? bias->data_ptr() : nullptr;
  f.silu_mul = silu_mul ? 1 : 0;
  f.out = out.data_ptr();
  f.ldo = int(out.size(1));
  BL_CHECK(bl_slab_finish(&f, st, err, errlen));
  return out;
}
// digits = 3: x as it is; digits = 1: x quantised to int8 per token.  Callers let go of the GIL first: a
// launch waits when the queue is full.
at::Tensor qlin_run(const at::Tensor& x, int digits, const QWeight& q, const c10::optional<at::Tensor>& bias,
                    bool silu_mul, int splits, bool want_slabs, void* err_flag, void* st) {
  const int m = int(x.size(0));
  at::Tensor xq, xs;
  if (q.xq) {
    xq = *q.xq;
    xs = *q.xs;
  } else if (digits == 3) {
    xs = at::empty({int64_t(bl_quant_digits_xs_bytes(m) / sizeof(float))}, x.options().dtype(at::kFloat));
    xq = at::empty({int64_t(bl_quant_digits_bytes(m, q.k))}, x.options().dtype(at::kChar));
    BL_CHECK(bl_quant_digits(x.data_ptr(), m, int(x.stride(0)), q.k, q.src == 2 ? 1 : 0, xq.data_ptr(), xs.data_ptr(), st,
                             err, errlen));
  } else {
    const at::Tensor xc = on_16_bytes(x.contiguous());
    xs = at::empty({m}, x.options().dtype(at::kFloat));
    xq = at::empty({m, q.k}, x.options().dtype(at::kChar));
    BL_CHECK(bl_w8a16_quant_act(xc.data_ptr(), m, q.k, xq.data_ptr(), xs.data_ptr(), st, err, errlen));
  }
  return qlin_product(x, xq, xs, m, digits, q, bias, silu_mul, splits, want_slabs, x.options(), err_flag, st);
}

// RMSNorm (+ residual, updated in place) of 1..128 decode rows or of the k-split slabs of the linear before, and the digits of
// the result for the linears behind it: (normed, residual, xq, xs).
std::tuple<at::Tensor, at::Tensor, at::Tensor, at::Tensor> rmsnorm_digits(const at::Tensor& x, const at::Tensor& gamma, double eps,
                                                                          const c10::optional<at::Tensor>& residual) {
  check_bf16x(gamma, "gamma");
  const bool slabs = x.scalar_type() == at::kFloat;
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && (slabs ? x.dim() == 3 : x.scalar_type() == at::kBFloat16 && x.dim() == 2),
              "barlink: rmsnorm_digits takes contiguous bfloat16 rows or float32 [splits, rows, hidden] slabs");
  const int hidden = int(x.size(-1)), rows = int(x.size(-2)), nsplit = slabs ? int(x.size(0)) : 0;
  TORCH_CHECK(gamma.numel() == hidden && rows >= 1 && rows <= BL_QLIN_MAX_TOKENS && (!slabs || nsplit >= 1),
              "barlink: gamma must have hidden elements, and rmsnorm_digits takes 1..", std::to_string(BL_QLIN_MAX_TOKENS), " rows");
  const auto like = x.options().dtype(at::kBFloat16);
  at::Tensor out = at::empty({rows, hidden}, like), res;
  if (residual) {
    check_bf16x(*residual, "residual");
    TORCH_CHECK(residual->numel() == int64_t(rows) * hidden, "barlink: residual must match x");
    res = *residual;
  }
  at::Tensor xs = at::empty({int64_t(bl_quant_digits_xs_bytes(rows) / sizeof(float))}, like.dtype(at::kFloat));
  at::Tensor xq = at::empty({int64_t(bl_quant_digits_bytes(rows, hidden))}, like.dtype(at::kChar));
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(x.device().index()).stream();
  py::gil_scoped_release nogil;
  BL_CHECK(bl_rmsnorm_digits(slabs ? nullptr : x.data_ptr(), residual ? res.data_ptr() : nullptr, gamma.data_ptr(), out.data_ptr(),
                             residual ? res.data_ptr() : nullptr, rows, hidden, float(eps), slabs ? x.data_ptr() : nullptr, nsplit,
                             size_t(rows) * hidden, xq.data_ptr(), xs.data_ptr(), st, err, errlen));
  return {out, res, xq, xs};
}

// Decode form of w8a16_linear without a reduction: fp32 slabs [splits, m, n] (scaled, no bias) for the
// kernel that reads them next, or the bf16 result when the shape wants no k-split.
at::Tensor w8a16_linear_split(const at::Tensor& x, const at::Tensor& wq, const at::Tensor& scale,
                              const c10::optional<at::Tensor>& bias, bool act_int8,
                              const c10::optional<at::Tensor>& xq, const c10::optional<at::Tensor>& xs) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1,
              "barlink: x must be a 2-D bfloat16 CUDA tensor with unit inner stride");
  TORCH_CHECK(wq.is_cuda() && wq.is_contiguous() && wq.scalar_type() == at::kChar && wq.dim() == 2 &&
                  wq.size(1) == x.size(1),
              "barlink: wq must be a contiguous int8 [n, k] CUDA tensor with k = x.shape[1]");
  check_bf16x(scale, "scale");
  const int k = int(x.size(1)), n = int(wq.size(0)), dev = x.device().index();
  TORCH_CHECK(scale.numel() == n, "barlink: scale must have one entry per output channel");
  TORCH_CHECK(qlin_takes(x, k, act_int8), "barlink: w8a16_linear_split is for 1..", std::to_string(BL_QLIN_MAX_TOKENS),
              " 16-byte aligned rows, K % 16 == 0");
  check_digits(x, k, !act_int8, xq, xs);
  c10::cuda::CUDAGuard guard(x.device());
  void* flag = w8_scratch(dev).err_flag.data_ptr();
  py::gil_scoped_release nogil;
  QWeight q{wq.data_ptr(), 0, n, k, BL_QSCALE_BF16_N, scale.data_ptr()};
  q.xq = xq;
  q.xs = xs;
  return qlin_run(x, act_int8 ? 1 : 3, q, bias, false, 0, true, flag, at::cuda::getCurrentCUDAStream(dev).stream());
}

at::Tensor w8a16_linear(const at::Tensor& x, const at::Tensor& wq, const at::Tensor& scale,
                        const c10::optional<at::Tensor>& bias, bool silu_mul, int splits,
                        const c10::optional<at::Tensor>& group_rel, bool act_int8,
                        const c10::optional<at::Tensor>& group_scale, const c10::optional<at::Tensor>& xq_in,
                        const c10::optional<at::Tensor>& xs_in) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1,
              "barlink: x must be a 2-D bfloat16 CUDA tensor with unit inner stride");
  TORCH_CHECK(wq.is_cuda() && wq.is_contiguous() && wq.scalar_type() == at::kChar && wq.dim() == 2 &&
                  wq.size(1) == x.size(1),
              "barlink: wq must be a contiguous int8 [n, k] CUDA tensor with k = x.shape[1]");
  check_bf16x(scale, "scale");
  const int m = int(x.size(0)), k = int(x.size(1)), n = int(wq.size(0));
  TORCH_CHECK(group_scale || scale.numel() == n, "barlink: scale must have one entry per output channel");
  if (group_scale) {
    TORCH_CHECK(act_int8 && !group_rel && m <= 64, "barlink: group_scale goes with act_int8 and at most 64 tokens");
    TORCH_CHECK(group_scale->is_cuda() && group_scale->is_contiguous() && group_scale->scalar_type() == at::kBFloat16 &&
                    group_scale->dim() == 2 && group_scale->size(0) == n && k % group_scale->size(1) == 0 &&
                    (k / group_scale->size(1)) % 128 == 0,
                "barlink: group_scale must be contiguous bfloat16 [n, k / group] with a group size that is a multiple of 128");
  }
  const int dev = x.device().index();
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  if (m == 0) return at::empty({0, silu_mul ? n / 2 : n}, x.options());
  if (group_rel) {
    TORCH_CHECK(group_rel->is_cuda() && group_rel->is_contiguous() && group_rel->scalar_type() == at::kHalf &&
                    group_rel->dim() == 2 && group_rel->size(0) == n && k % group_rel->size(1) == 0,
                "barlink: group_rel must be contiguous float16 [n, k / group] (see w8_group_scales)");
    TORCH_CHECK(m <= 256, "barlink: in-kernel group scales take at most 256 tokens");
  }
  TORCH_CHECK(!(act_int8 && group_rel), "barlink: int8 activations go with per-channel or group_scale weight scales");
  // 1..128 tokens: the weights go to the tensor cores as they are (qlin_kernels.cu).  Group scales need
  // groups of whole 128-wide k-blocks.
  const bool by_qlin = qlin_takes(x, k, act_int8, bool(group_scale)) && (!group_rel || (k / group_rel->size(1)) % 128 == 0);
  check_digits(x, k, by_qlin && !act_int8, xq_in, xs_in);
  if (by_qlin) {
    QWeight q{wq.data_ptr(), 0, n, k, BL_QSCALE_BF16_N, scale.data_ptr()};
    q.xq = xq_in;
    q.xs = xs_in;
    if (group_scale) {
      q.scale_kind = BL_QSCALE_BF16_NG;
      q.scale = group_scale->data_ptr();
      q.group_k = k / int(group_scale->size(1));
    } else if (group_rel) {
      q.scale_kind = BL_QSCALE_F16_NG;
      q.scale = group_rel->data_ptr();
      q.row_scale = scale.data_ptr();
      q.group_k = k / int(group_rel->size(1));
    }
    void* flag = w8_scratch(dev).err_flag.data_ptr();
    py::gil_scoped_release nogil;
    return qlin_run(x, act_int8 ? 1 : 3, q, bias, silu_mul, splits, false, flag, st);
  }
  at::Tensor out = at::empty({m, silu_mul ? n / 2 : n}, x.options());
  if (act_int8) {
    // the reference's numerics (w8a16.cu:37-92 there quantises the activations per token and
    // multiplies int8 by int8): both operands go to the tensor cores as int8
    TORCH_CHECK(k % 16 == 0, "barlink: int8 activations need K % 16 == 0");
    const at::Tensor xc = on_16_bytes(x.contiguous());
    at::Tensor xq = at::empty({m, k}, x.options().dtype(at::kChar));
    at::Tensor xs = at::empty({m}, x.options().dtype(at::kFloat));
    BL_CHECK(bl_w8a16_quant_act(xc.data_ptr(), m, k, xq.data_ptr(), xs.data_ptr(), st, err, errlen));
    W8Scratch& s = w8_scratch(dev);
    if (bias) {
      check_bf16x(*bias, "bias");
      TORCH_CHECK(bias->numel() == n, "barlink: bias must have n entries");
    }
    if (m <= 256) {
      blW8A16Args a;
      memset(&a, 0, sizeof(a));
      a.xq = xq.data_ptr();
      a.xs = xs.data_ptr();
      a.m = m;
      a.ldx = k;
      a.wq = wq.data_ptr();
      a.n = n;
      a.k = k;
      a.scale = scale.data_ptr();
      a.bias = bias ? bias->data_ptr() : nullptr;
      a.out = out.data_ptr();
      a.ldo = silu_mul ? n / 2 : n;
      a.silu_mul = silu_mul ? 1 : 0;
      a.splits = splits;
      a.ws = s.ws.data_ptr();
      a.ws_bytes = size_t(s.ws.nbytes());
      a.counters = s.counters.data_ptr();
      a.n_counters = int(s.counters.numel());
      a.err_flag = s.err_flag.data_ptr();
      py::gil_scoped_release nogil;
      BL_CHECK(bl_w8a16_linear(&a, st, err, errlen));
    } else {
      // prefill: token-major tiles
      blGemmArgs g;
      memset(&g, 0, sizeof(g));
      g.a = xq.data_ptr(); g.ra = m; g.lda = k;
      g.b = wq.data_ptr(); g.rb = n; g.ldb = k;
      g.k = k;
      g.out = out.data_ptr();
      g.ldo = silu_mul ? n / 2 : n;
      g.bias = bias ? bias->data_ptr() : nullptr;
      g.silu_mul = silu_mul ? 1 : 0;
      g.splits = 1;
      g.err_flag = s.err_flag.data_ptr();
      g.i8 = 1;
      g.feat_scale = scale.data_ptr();
      g.tok_scale = xs.data_ptr();
      py::gil_scoped_release nogil;
      BL_CHECK(bl_gemm_bf16(&g, st, err, errlen));
    }
    return out;
  }
  if (m > 256) {
    at::Tensor w = at::empty({n, k}, x.options());
    const at::Tensor wa = (reinterpret_cast<uintptr_t>(wq.data_ptr()) & 7u) == 0 ? wq : wq.clone();  // (read 8 bytes at a time)
    BL_CHECK(bl_w8_dequant(wa.data_ptr(), scale.data_ptr(), w.data_ptr(), n, k, st, err, errlen));
    py::object lin = py::module_::import("barlink_sm86_b200").attr("load_extension")().attr("linear");
    // `w` was written by the kernel just launched: the GEMM must not fetch weight tiles ahead of
    // that kernel's completion (its producer otherwise requests them before griddepcontrol.wait)
    using namespace pybind11::literals;
    return lin(x, w, bias ? py::cast(*bias) : py::none(), py::none(), silu_mul, "dynamic_weights"_a = true)
        .cast<at::Tensor>();
  }
  W8Scratch& s = w8_scratch(dev);
  blW8A16Args a;
  memset(&a, 0, sizeof(a));
  a.x = x.data_ptr();
  a.m = m;
  a.ldx = int(x.stride(0));
  a.wq = wq.data_ptr();
  a.n = n;
  a.k = k;
  a.scale = scale.data_ptr();
  if (group_rel) {
    a.group_rel = group_rel->data_ptr();
    a.group_k = k / int(group_rel->size(1));
  }
  if (bias) {
    check_bf16x(*bias, "bias");
    TORCH_CHECK(bias->numel() == n, "barlink: bias must have n entries");
    a.bias = bias->data_ptr();
  }
  a.out = out.data_ptr();
  a.ldo = silu_mul ? n / 2 : n;
  a.silu_mul = silu_mul ? 1 : 0;
  a.splits = splits;
  a.ws = s.ws.data_ptr();
  a.ws_bytes = size_t(s.ws.nbytes());
  a.counters = s.counters.data_ptr();
  a.n_counters = int(s.counters.numel());
  a.err_flag = s.err_flag.data_ptr();
  {
    py::gil_scoped_release nogil;
    BL_CHECK(bl_w8a16_linear(&a, st, err, errlen));
  }
  return out;
}

int w8_error_flag(int dev) { return w8_scratch(dev).err_flag.cpu()[0].item<int>(); }

// the reference's pair (binding.cpp:434-490 there)
std::vector<at::Tensor> w8a16_quant_act(const at::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && x.dim() == 2 && x.scalar_type() == at::kBFloat16,
              "barlink w8a16_quant_act: x must be a contiguous 2-D bfloat16 CUDA tensor");
  const int m = int(x.size(0)), k = int(x.size(1));
  TORCH_CHECK(k % 8 == 0, "barlink w8a16_quant_act: K % 8 must be 0");
  c10::cuda::CUDAGuard guard(x.device());
  const at::Tensor xa = on_16_bytes(x);
  at::Tensor xq = at::empty({m, k}, x.options().dtype(at::kChar));
  at::Tensor xs = at::empty({m}, x.options().dtype(at::kFloat));
  void* st = at::cuda::getCurrentCUDAStream(x.device().index()).stream();
  if (m > 0) BL_CHECK(bl_w8a16_quant_act(xa.data_ptr(), m, k, xq.data_ptr(), xs.data_ptr(), st, err, errlen));
  return {xq, xs};
}

at::Tensor w8a16_gemm(const at::Tensor& xq, const at::Tensor& xs, const at::Tensor& wq_t,
                      const at::Tensor& sw_t, int64_t N, int64_t K, int64_t S, int splits) {
  TORCH_CHECK(xq.is_cuda() && xq.is_contiguous() && xq.dim() == 2 && xq.scalar_type() == at::kChar,
              "barlink w8a16_gemm: xq must be contiguous int8 [M, K]");
  const int m = int(xq.size(0));
  TORCH_CHECK(xq.size(1) == K && K % 128 == 0, "barlink w8a16_gemm: K must match xq and be a multiple of 128");
  TORCH_CHECK(wq_t.is_contiguous() && wq_t.scalar_type() == at::kChar && wq_t.numel() == N * K &&
                  sw_t.is_contiguous() && sw_t.scalar_type() == at::kFloat && sw_t.numel() == (K / 128) * N,
              "barlink w8a16_gemm: wq_t int8 [K/16, N, 16] and sw_t float32 [K/128, N], contiguous");
  TORCH_CHECK(xs.is_contiguous() && xs.scalar_type() == at::kFloat && xs.numel() == m,
              "barlink w8a16_gemm: xs must be float32 [M]");
  TORCH_CHECK(m <= 16, "barlink w8a16_gemm: M > 16 is not supported by this decode kernel (use w8a16_linear)");
  c10::cuda::CUDAGuard guard(xq.device());
  const int dev = xq.device().index();
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  const auto like = xq.options().dtype(at::kBFloat16);
  if (m == 0) return at::empty({0, N}, like);
  // S is the caller's k-split for the reference's kernel; here the shape decides, or `splits`
  (void)S;
  if (splits <= 0) splits = bl_qlin_splits(int(N), int(K), m, 1, 1);
  if (splits > K / 128) splits = int(K / 128);
  void* flag = w8_scratch(dev).err_flag.data_ptr();
  py::gil_scoped_release nogil;
  const at::Tensor xa = on_16_bytes(xq);
  at::Tensor out = at::empty({m, N}, like), ws;
  if (splits > 1) ws = at::empty({splits, m, N}, like.dtype(at::kFloat));
  BL_CHECK(bl_w8a16_gemm(xa.data_ptr(), xs.data_ptr(), wq_t.data_ptr(), sw_t.data_ptr(), out.data_ptr(), m, int(N), int(K),
                         splits, splits > 1 ? ws.data_ptr() : nullptr, flag, st, err, errlen));
  return out;
}

// GPTQ-v1 int4 linear.  Groups of 128: up to 16 rows expanded in registers for mma.sync (w4a16_kernels.cu), up to 128 rows
// int8 digits of the activations (qlin_kernels.cu); else the GEMV up to 16 rows; else widen the weight and use the bf16 GEMM.
// silu_mul: SiLU(gate) * up over interleaved (gate, up) columns.  want_slabs: see qlin_product.
at::Tensor w4a16_linear(const at::Tensor& x, const at::Tensor& qweight, const at::Tensor& scales,
                        const at::Tensor& qzeros, int group, int splits, bool silu_mul, bool want_slabs) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.is_contiguous(),
              "barlink: x must be a contiguous 2-D bfloat16 CUDA tensor");
  TORCH_CHECK(qweight.is_cuda() && qweight.is_contiguous() && qweight.scalar_type() == at::kInt &&
                  qweight.dim() == 2 && qweight.size(0) * 8 == x.size(1),
              "barlink: qweight must be a contiguous int32 [K/8, N] CUDA tensor with K = x.shape[1]");
  const int m = int(x.size(0)), k = int(x.size(1)), n = int(qweight.size(1));
  TORCH_CHECK(group > 0 && k % group == 0, "barlink: K must be a multiple of the group size");
  TORCH_CHECK(scales.is_cuda() && scales.is_contiguous() && scales.scalar_type() == at::kHalf &&
                  scales.dim() == 2 && scales.size(0) == k / group && scales.size(1) == n,
              "barlink: scales must be a contiguous float16 [K/group, N] CUDA tensor");
  TORCH_CHECK(qzeros.is_cuda() && qzeros.is_contiguous() && qzeros.scalar_type() == at::kInt &&
                  qzeros.dim() == 2 && qzeros.size(0) == k / group && qzeros.size(1) * 8 == n,
              "barlink: qzeros must be a contiguous int32 [K/group, N/8] CUDA tensor");
  const int dev = x.device().index();
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  TORCH_CHECK(!silu_mul || n % 16 == 0, "barlink: SiLU*mul of an int4 linear needs N a multiple of 16");
  if (m == 0) return at::empty({0, silu_mul ? n / 2 : n}, x.options());
  W8Scratch& s = w8_scratch(dev);
  const bool aligned = ((reinterpret_cast<uintptr_t>(x.data_ptr()) | reinterpret_cast<uintptr_t>(qweight.data_ptr())) & 15u) == 0;
  // (37888 x 3584, us: GEMV 28 / 51 / 176 at 1 / 4 / 16 rows, digits 39 to 40, this 19.7 / 19.7 / 28)
  if (group == 128 && m <= 16 && n % 8 == 0 && aligned && (reinterpret_cast<uintptr_t>(scales.data_ptr()) & 7u) == 0) {
    py::gil_scoped_release nogil;
    const int s4 = bl_w4a16_mma_splits(m, n, k, splits, want_slabs ? 1 : 0);
    const int n_out = silu_mul ? n / 2 : n;
    at::Tensor out, slabs;
    if (s4 > 1) slabs = at::empty({s4, m, n}, x.options().dtype(at::kFloat));
    else out = at::empty({m, n_out}, x.options());
    BL_CHECK(bl_w4a16_mma(x.data_ptr(), qweight.data_ptr(), scales.data_ptr(), qzeros.data_ptr(),
                          s4 > 1 ? nullptr : out.data_ptr(), m, n, k, s4 > 1 ? 0 : silu_mul, s4,
                          s4 > 1 ? slabs.data_ptr() : nullptr, st, err, errlen));
    if (s4 == 1) return out;
    if (want_slabs) return slabs;
    out = at::empty({m, n_out}, x.options());
    blSlabFinishArgs f;
    memset(&f, 0, sizeof(f));
    f.slabs = slabs.data_ptr();
    f.nsplit = s4; f.m = m; f.n = f.pitch = n;
    f.silu_mul = silu_mul ? 1 : 0;
    f.out = out.data_ptr();
    f.ldo = n_out;
    BL_CHECK(bl_slab_finish(&f, st, err, errlen));
    return out;
  }
  // Above 16 rows the digit kernel; the other way is to widen the weight for a bf16 product: 64 rows, 296 and 143 us
  // (37888 x 3584, 3584 x 18944) against 70 and 45; faster only for small weights (2048 x 2048 10 against 17), whose
  // values it rounds to bf16.
  if (group == 128 && m <= BL_QLIN_MAX_TOKENS && k <= 32768 && n % 8 == 0 && aligned) {
    QWeight q{qweight.data_ptr(), 2, n, k, BL_QSCALE_F16_GN, scales.data_ptr()};
    q.group_k = group;
    q.zeros = qzeros.data_ptr();
    py::gil_scoped_release nogil;
    return qlin_run(x, 3, q, c10::nullopt, silu_mul, splits > k / 128 ? k / 128 : splits, want_slabs,
                    s.err_flag.data_ptr(), st);
  }
  auto finish = [&](const at::Tensor& y) {
    if (!silu_mul) return y;
    at::Tensor o = at::empty({m, n / 2}, x.options());
    BL_CHECK(bl_silu_mul(y.data_ptr(), o.data_ptr(), m, n / 2, 1, st, err, errlen));
    return o;
  };
  if (m > 16) {
    at::Tensor w = at::empty({n, k}, x.options());
    BL_CHECK(bl_w4_dequant(qweight.data_ptr(), scales.data_ptr(), qzeros.data_ptr(), w.data_ptr(), n, k, group,
                           st, err, errlen));
    return finish(at::matmul(x, w.t()));  // prefill path, not the decode hot path
  }
  at::Tensor out = at::empty({m, n}, x.options());
  const at::Tensor words = on_16_bytes(qweight), sc = on_16_bytes(scales);
  BL_CHECK(bl_w4a16_gemv(x.data_ptr(), words.data_ptr(), sc.data_ptr(), qzeros.data_ptr(), out.data_ptr(),
                         m, n, k, group, splits, s.ws.data_ptr(), size_t(s.ws.nbytes()), st, err, errlen));
  return finish(out);
}

at::Tensor w4_dequant(const at::Tensor& qweight, const at::Tensor& scales, const at::Tensor& qzeros, int group) {
  TORCH_CHECK(qweight.is_cuda() && qweight.is_contiguous() && qweight.scalar_type() == at::kInt &&
                  scales.is_cuda() && scales.is_contiguous() && scales.scalar_type() == at::kHalf &&
                  qzeros.is_cuda() && qzeros.is_contiguous() && qzeros.scalar_type() == at::kInt,
              "barlink: w4_dequant needs contiguous CUDA qweight (int32), scales (float16), qzeros (int32)");
  const int k = int(qweight.size(0)) * 8, n = int(qweight.size(1));
  c10::cuda::CUDAGuard guard(qweight.device());
  at::Tensor w = at::empty({n, k}, scales.options().dtype(at::kBFloat16));
  BL_CHECK(bl_w4_dequant(qweight.data_ptr(), scales.data_ptr(), qzeros.data_ptr(), w.data_ptr(), n, k, group,
                         at::cuda::getCurrentCUDAStream(qweight.device().index()).stream(), err, errlen));
  return w;
}

void qknorm_rope(const at::Tensor& qkv, const c10::optional<at::Tensor>& gq,
                 const c10::optional<at::Tensor>& gk, const at::Tensor& positions, int heads, double eps,
                 double theta, int axes) {
  TORCH_CHECK(qkv.is_cuda() && qkv.scalar_type() == at::kBFloat16 && qkv.dim() == 2 && qkv.stride(1) == 1 &&
                  qkv.size(1) >= int64_t(2 * heads) * 128,
              "barlink: qknorm_rope needs a 2-D bfloat16 CUDA tensor whose rows start with the q and k heads");
  TORCH_CHECK(positions.is_cuda() && positions.scalar_type() == at::kInt && positions.is_contiguous() &&
                  positions.numel() == qkv.size(0) * axes,
              "barlink: positions must be int32 [rows, axes]");
  if (gq) check_bf16x(*gq, "gq");
  if (gk) check_bf16x(*gk, "gk");
  c10::cuda::CUDAGuard guard(qkv.device());
  void* st = at::cuda::getCurrentCUDAStream(qkv.device().index()).stream();
  if (qkv.size(0) > 0)
    BL_CHECK(bl_qknorm_rope(qkv.data_ptr(), gq ? gq->data_ptr() : nullptr, gk ? gk->data_ptr() : nullptr,
                            positions.data_ptr<int>(), int(qkv.size(0)), heads, 128, int(qkv.stride(0)),
                            float(eps), float(theta), axes, st, err, errlen));
}

at::Tensor layernorm_modulate(const at::Tensor& x, const at::Tensor& shift, const at::Tensor& scale,
                              int rows_per_batch, double eps) {
  check_bf16x(x, "x");
  TORCH_CHECK(shift.is_cuda() && scale.is_cuda() && shift.scalar_type() == at::kBFloat16 &&
                  scale.scalar_type() == at::kBFloat16 && shift.dim() == 2 && scale.dim() == 2 &&
                  shift.stride(1) == 1 && scale.stride(1) == 1 && shift.stride(0) == scale.stride(0),
              "barlink: shift/scale must be bfloat16 [batch, hidden] views with the same pitch");
  const int hidden = int(x.size(-1));
  const int rows = int(x.numel() / hidden);
  at::Tensor out = at::empty_like(x);
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(x.device().index()).stream();
  if (rows > 0)
    BL_CHECK(bl_layernorm_modulate(x.data_ptr(), shift.data_ptr(), scale.data_ptr(), out.data_ptr(), rows,
                                   hidden, rows_per_batch, int(shift.stride(0)), float(eps), st, err, errlen));
  return out;
}

void gate_residual(const at::Tensor& x, const at::Tensor& y, const at::Tensor& gate, int rows_per_batch) {
  check_bf16x(x, "x");
  check_bf16x(y, "y");
  TORCH_CHECK(gate.is_cuda() && gate.scalar_type() == at::kBFloat16 && gate.dim() == 2 && gate.stride(1) == 1 &&
                  x.sizes() == y.sizes(),
              "barlink: gate must be a bfloat16 [batch, hidden] view and y must match x");
  const int hidden = int(x.size(-1));
  const int rows = int(x.numel() / hidden);
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(x.device().index()).stream();
  if (rows > 0)
    BL_CHECK(bl_gate_residual(x.data_ptr(), y.data_ptr(), gate.data_ptr(), rows, hidden, rows_per_batch,
                              int(gate.stride(0)), st, err, errlen));
}

// ---- host-only internals, exposed so that they can be unit-tested without a GPU ----

// ---- decode linears with the collective folded in (dlin_kernels.cu) ----------------------
struct DlinScratch {
  at::Tensor sync, err_flag;
};
DlinScratch& dlin_scratch(int dev) {
  static std::map<int, DlinScratch> m;
  auto it = m.find(dev);
  if (it != m.end()) return it->second;
  auto o = at::TensorOptions().device(at::kCUDA, dev).dtype(at::kInt);
  DlinScratch s;
  s.sync = at::zeros({16 + 64 * 8}, o);  // counters, then the segment sums of the gather prologue
  s.err_flag = at::zeros({4}, o);
  return m.emplace(dev, s).first->second;
}
int dlin_error_flag(int dev) { return dlin_scratch(dev).err_flag.cpu()[0].item<int>(); }

// a one-rank stand-in for the link in ordinary device memory (single-GPU runs of the same kernels)
at::Tensor dlin_local_link(int tokens, int hidden, int dev) {
  c10::cuda::CUDAGuard guard(c10::Device(at::kCUDA, dev));
  at::Tensor buf = at::empty({int64_t(bl_dlin_local_link_bytes(tokens, hidden))},
                             at::TensorOptions().device(at::kCUDA, dev).dtype(at::kByte));
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  BL_CHECK(bl_dlin_local_link_init(buf.data_ptr(), tokens, hidden, st, err, errlen));
  return buf;
}

void dlin_fill_common(blDlinArgs& a, const at::Tensor& x, int hidden, const c10::optional<at::Tensor>& link,
                      int dev) {
  a.x = x.data_ptr();
  a.tokens = int(x.size(0));
  a.ldx = int(x.stride(0));
  a.hidden = hidden;
  if (link) {
    TORCH_CHECK(link->is_cuda() && link->is_contiguous() &&
                    size_t(link->nbytes()) >= bl_dlin_local_link_bytes(a.tokens, hidden),
                "barlink: the local link buffer is too small for ", std::to_string(a.tokens), " x ", std::to_string(hidden));
    a.local_link = link->data_ptr();
  }
  a.err_flag = dlin_scratch(dev).err_flag.data_ptr();
}

// pro: "none" | "gather_norm";  epi: "store" | "silu_mul" | "push"
// gather_norm: x is written first (RMSNorm(residual + all-reduced rows) * gamma), residual is
// updated in place.  push: returns nothing useful (the rows are in every rank's inbox).
at::Tensor dlin(const at::Tensor& x, const at::Tensor& w, const std::string& pro, const std::string& epi,
                const c10::optional<at::Tensor>& out_opt, const c10::optional<at::Tensor>& bias,
                const c10::optional<at::Tensor>& residual, const c10::optional<at::Tensor>& gamma, double eps,
                int hidden, const c10::optional<at::Tensor>& link, int cluster, bool first,
                const c10::optional<at::Tensor>& trace) {
  check_bf16x(w, "weight");
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1 &&
                  w.dim() == 2 && w.stride(1) == 1 && w.size(1) == x.size(1),
              "barlink: dlin needs bf16 x [tokens, k] and w [n, k] with unit inner strides");
  const int dev = x.device().index();
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  blDlinArgs a;
  memset(&a, 0, sizeof(a));
  a.w = w.data_ptr();
  a.n = int(w.size(0));
  a.k = int(w.size(1));
  a.ldw = int(w.stride(0));
  a.pro = pro == "gather_norm" ? 1 : 0;
  TORCH_CHECK(a.pro == 1 || pro == "none", "barlink: dlin prologue must be none or gather_norm");
  a.epi = epi == "store" ? 0 : epi == "silu_mul" ? 1 : epi == "push" ? 2 : -1;
  TORCH_CHECK(a.epi >= 0, "barlink: dlin epilogue must be store, silu_mul or push");
  dlin_fill_common(a, x, hidden > 0 ? hidden : a.k, link, dev);
  if (a.pro == 1) {
    TORCH_CHECK(residual && gamma, "barlink: gather_norm needs residual and gamma");
    check_bf16x(*residual, "residual");
    check_bf16x(*gamma, "gamma");
    TORCH_CHECK(residual->numel() == x.numel() && x.is_contiguous() && gamma->numel() == a.k,
                "barlink: residual must match x, gamma must have k entries");
    a.residual_in = first ? nullptr : residual->data_ptr();
    a.residual_out = residual->data_ptr();
    a.gamma = gamma->data_ptr();
    a.eps = float(eps);
    a.sync = dlin_scratch(dev).sync.data_ptr();
  }
  at::Tensor out;
  if (a.epi != 2) {
    const int64_t cols = a.epi == 1 ? a.n / 2 : a.n;
    out = out_opt ? *out_opt : at::empty({x.size(0), cols}, x.options());
    TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kBFloat16 && out.dim() == 2 && out.size(0) == x.size(0) &&
                    out.size(1) == cols && out.stride(1) == 1,
                "barlink: dlin out must be bf16 [tokens, ", std::to_string(cols), "]");
    a.out = out.data_ptr();
    a.ldo = int(out.stride(0));
    if (bias) {
      check_bf16x(*bias, "bias");
      TORCH_CHECK(bias->numel() == a.n, "barlink: bias must have n entries");
      a.bias = bias->data_ptr();
    }
  }
  a.cluster = cluster;
  if (trace) {
    TORCH_CHECK(trace->is_cuda() && trace->scalar_type() == at::kLong && trace->is_contiguous() &&
                    trace->numel() >= 12 * 8 * ((a.n + 127) / 128),
                "barlink: trace must be a contiguous int64 CUDA tensor of 12 words per CTA");
    a.trace = trace->data_ptr();
  }
  blCtx* c = link ? nullptr : blpg::global_ctx();
  {
    py::gil_scoped_release nogil;
    BL_CHECK(bl_dlin(c, &a, st, err, errlen));
  }
  return a.epi == 2 ? x : out;
}

// x = RMSNorm(residual + all-reduced inbox rows) * gamma, residual updated in place
void gather_norm(const at::Tensor& x, const at::Tensor& residual, const at::Tensor& gamma, double eps,
                 const c10::optional<at::Tensor>& link, bool first) {
  check_bf16x(residual, "residual");
  check_bf16x(gamma, "gamma");
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.is_contiguous() &&
                  residual.numel() == x.numel() && gamma.numel() == x.size(1),
              "barlink: gather_norm needs contiguous bf16 x [tokens, hidden], residual of that shape, gamma [hidden]");
  const int dev = x.device().index();
  c10::cuda::CUDAGuard guard(x.device());
  void* st = at::cuda::getCurrentCUDAStream(dev).stream();
  blDlinArgs a;
  memset(&a, 0, sizeof(a));
  dlin_fill_common(a, x, int(x.size(1)), link, dev);
  a.residual_in = first ? nullptr : residual.data_ptr();
  a.residual_out = residual.data_ptr();
  a.gamma = gamma.data_ptr();
  a.eps = float(eps);
  blCtx* c = link ? nullptr : blpg::global_ctx();
  py::gil_scoped_release nogil;
  BL_CHECK(bl_gather_norm(c, &a, st, err, errlen));
}

py::dict layout_of(size_t pool_bytes, int world) {
  const bl::Layout L = bl::compute_layout(pool_bytes, world);
  py::dict d;
  d["pool_bytes"] = L.pool_bytes;
  d["user_bytes"] = L.user_bytes;
  d["stage_off"] = L.stage_off;
  d["stage_slice"] = L.stage_slice;
  d["lamport_off"] = L.lamport_off;
  d["lamport_slice"] = L.lamport_slice;
  d["p2p_off"] = L.p2p_off;
  d["p2p_slice"] = L.p2p_slice;
  d["sig_off"] = L.sig_off;
  return d;
}

// ops: ("alloc", bytes) -> offset or -1; ("free", offset, bytes) -> 1 / 0
std::vector<int64_t> arena_replay(size_t user_bytes, const std::vector<py::tuple>& ops) {
  bl::Arena a;
  std::vector<int64_t> out;
  for (const auto& op : ops) {
    const std::string kind = op[0].cast<std::string>();
    if (kind == "alloc") out.push_back(bl::arena_alloc(a, user_bytes, op[1].cast<size_t>()));
    else out.push_back(bl::arena_free(a, op[1].cast<size_t>(), op[2].cast<size_t>()) ? 1 : 0);
  }
  return out;
}

}  // namespace

void bind_extra(py::module_& m) {
  m.def("layout_of", &layout_of, py::arg("pool_bytes"), py::arg("world"));
  m.def("arena_replay", &arena_replay, py::arg("user_bytes"), py::arg("ops"));
  m.def("algo_for", [](size_t bytes, int world, const std::string& dtype, bool multicast, size_t pool_bytes,
                       const std::string& algo) {
    const int dt = dtype == "bf16" ? BL_DTYPE_BF16 : dtype == "fp16" ? BL_DTYPE_FP16 : dtype == "fp32" ? BL_DTYPE_FP32
                 : dtype == "fp64" ? BL_DTYPE_FP64 : BL_DTYPE_U8;
    const int al = algo == "oneshot" ? BL_ALGO_ONESHOT : algo == "twoshot" ? BL_ALGO_TWOSHOT
                 : algo == "nvls" ? BL_ALGO_NVLS : BL_ALGO_AUTO;
    static const char* names[] = {"auto", "oneshot", "twoshot", "nvls"};
    return std::string(names[bl_algo_for(bytes, world, dt, multicast ? 1 : 0, pool_bytes, al)]);
  }, py::arg("bytes"), py::arg("world"), py::arg("dtype") = "bf16", py::arg("multicast") = false,
        py::arg("pool_bytes") = size_t(1) << 30, py::arg("algo") = "auto");
  m.def("pick_splits", [](int tiles, int kblocks, int sms, int want) { return bl::pick_splits(tiles, kblocks, sms, want); },
        py::arg("tiles"), py::arg("kblocks"), py::arg("sms") = 148, py::arg("want") = 0);
  m.def("w4a16_linear", &w4a16_linear, py::arg("x"), py::arg("qweight"), py::arg("scales"), py::arg("qzeros"),
        py::arg("group") = 128, py::arg("splits") = 0, py::arg("silu_mul") = false, py::arg("want_slabs") = false);
  m.def("w4_dequant", &w4_dequant, py::arg("qweight"), py::arg("scales"), py::arg("qzeros"), py::arg("group") = 128);
  m.def("qknorm_rope", &qknorm_rope, py::arg("qkv"), py::arg("gq"), py::arg("gk"), py::arg("positions"),
        py::arg("heads"), py::arg("eps") = 1e-6, py::arg("theta") = 1e4, py::arg("axes") = 2);
  m.def("layernorm_modulate", &layernorm_modulate, py::arg("x"), py::arg("shift"), py::arg("scale"),
        py::arg("rows_per_batch"), py::arg("eps") = 1e-6);
  m.def("gate_residual", &gate_residual, py::arg("x"), py::arg("y"), py::arg("gate"),
        py::arg("rows_per_batch"));
  m.def("w8a16_linear", &w8a16_linear, py::arg("x"), py::arg("wq"), py::arg("scale"),
        py::arg("bias") = py::none(), py::arg("silu_mul") = false, py::arg("splits") = 0,
        py::arg("group_rel") = py::none(), py::arg("act_int8") = false, py::arg("group_scale") = py::none(),
        py::arg("xq") = py::none(), py::arg("xs") = py::none());
  m.def("w8a16_linear_split", &w8a16_linear_split, py::arg("x"), py::arg("wq"), py::arg("scale"),
        py::arg("bias") = py::none(), py::arg("act_int8") = false, py::arg("xq") = py::none(), py::arg("xs") = py::none());
  m.def("w4a16_splits", [](int m_, int n, int k) { return bl_w4a16_mma_splits(m_, n, k, 0, 0); }, py::arg("m"), py::arg("n"),
        py::arg("k"));
  m.def("rmsnorm_digits", &rmsnorm_digits, py::arg("x"), py::arg("gamma"), py::arg("eps"), py::arg("residual") = py::none());
  m.def("w8_group_scales", &w8_group_scales, py::arg("scales"));
  m.def("w8_error_flag", &w8_error_flag, py::arg("device") = 0);
  m.def("dlin", &dlin, py::arg("x"), py::arg("weight"), py::arg("pro") = "none", py::arg("epi") = "store",
        py::arg("out") = py::none(), py::arg("bias") = py::none(), py::arg("residual") = py::none(),
        py::arg("gamma") = py::none(), py::arg("eps") = 1e-6, py::arg("hidden") = 0, py::arg("link") = py::none(),
        py::arg("cluster") = 0, py::arg("first") = false, py::arg("trace") = py::none());
  m.def("gather_norm", &gather_norm, py::arg("x"), py::arg("residual"), py::arg("gamma"), py::arg("eps") = 1e-6,
        py::arg("link") = py::none(), py::arg("first") = false);
  m.def("dlin_local_link", &dlin_local_link, py::arg("tokens"), py::arg("hidden"), py::arg("device") = 0);
  m.def("dlin_error_flag", &dlin_error_flag, py::arg("device") = 0);
  m.def("dlin_cluster", [](int n, int k, int tokens, int want) { return bl_dlin_cluster(n, k, tokens, want); },
        py::arg("n"), py::arg("k"), py::arg("tokens") = 64, py::arg("want") = 0);
  m.def("w8a16_quant_act", &w8a16_quant_act);
  m.def("w8a16_gemm", &w8a16_gemm, py::arg("xq"), py::arg("xs"), py::arg("wq_t"), py::arg("sw_t"),
        py::arg("N"), py::arg("K"), py::arg("S"), py::arg("splits") = 0);
  m.def("attn_fwd", &attn_fwd, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("cu_q"),
        py::arg("cu_k"), py::arg("max_q"), py::arg("scale"), py::arg("causal"), py::arg("max_k") = 0);
  m.def("attn_error_flag", &attn_error_flag, py::arg("device") = 0);
  m.def("sp_collective", &sp_collective, py::arg("kind"), py::arg("ins") = std::vector<at::Tensor>{},
        py::arg("outs") = std::vector<at::Tensor>{}, py::arg("aux_in") = std::vector<at::Tensor>{},
        py::arg("aux_out") = std::vector<at::Tensor>{}, py::arg("gamma") = std::vector<at::Tensor>{},
        py::arg("algo") = "auto", py::arg("root") = 0, py::arg("eps") = 1e-6);
  m.def("sp_sendrecv", &sp_sendrecv, py::arg("src"), py::arg("dst"), py::arg("inp"), py::arg("out"));
}
