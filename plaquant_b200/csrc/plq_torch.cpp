// PyTorch front end of the calls that a forward pass makes most often: the pack, a whole quantised linear, a whole decoder
// layer.
// The kernels are those of libplq_b200.so, launched one after the other on the current stream; this file only allocates
// and forwards.  Called operator by operator from Python a linear is two foreign calls and nine allocations (~40 us of
// host time against 8 - 15 us on the device for up to a few hundred rows), a layer nine foreign calls and ~30.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <dlfcn.h>

#include <optional>
#include <tuple>

#include "../../include/plq.h"

namespace {

using at::Tensor;

// The C entry points, out of the library that _lib has loaded (init).
struct Api {
  decltype(&::plq_pack) pack;
  decltype(&::plq_rmsnorm_pack) rmsnorm_pack;
  decltype(&::plq_add_rmsnorm_pack) add_rmsnorm_pack;
  decltype(&::plq_silu_mul_pack) silu_mul_pack;
  decltype(&::plq_gemv_tc) gemv_tc;
  decltype(&::plq_mixed_gemm) mixed_gemm;
  decltype(&::plq_mixed_gemm_silu_mul) mixed_gemm_silu_mul;
  decltype(&::plq_rope_kv_append) rope_kv_append;
  decltype(&::plq_rope_kv_append_nvfp4_values) rope_kv_append_nvfp4_values;
  decltype(&::plq_sf_tiled_bytes) sf_tiled_bytes;
} api;

void init(const std::string& path) {
  void* lib = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!lib) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
  auto find = [&](auto& fn, const char* name) {
    void* at = dlsym(lib, name);
    if (!at) throw std::runtime_error(path + " has no " + name);
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(at);
  };
  find(api.pack, "plq_pack");
  find(api.rmsnorm_pack, "plq_rmsnorm_pack");
  find(api.add_rmsnorm_pack, "plq_add_rmsnorm_pack");
  find(api.silu_mul_pack, "plq_silu_mul_pack");
  find(api.gemv_tc, "plq_gemv_tc");
  find(api.mixed_gemm, "plq_mixed_gemm");
  find(api.mixed_gemm_silu_mul, "plq_mixed_gemm_silu_mul");
  find(api.rope_kv_append, "plq_rope_kv_append");
  find(api.rope_kv_append_nvfp4_values, "plq_rope_kv_append_nvfp4_values");
  find(api.sf_tiled_bytes, "plq_sf_tiled_bytes");
}

// Raises the package's PlqError for a non-zero status.
void check(int status) {
  if (status != PLQ_OK) {
    pybind11::gil_scoped_acquire gil;
    pybind11::module_::import("plaquant_b200._lib").attr("check")(status);
  }
}

int64_t up256(int64_t b) { return (b + 255) / 256 * 256; }

const void* ptr(const Tensor& t) { return t.numel() == 0 ? nullptr : t.const_data_ptr(); }

// A packed [rows, k_lo + k_hi] operand with tiled scales, laid out at `base`.
struct PackedAt {
  uint8_t *lo, *lo_sf, *hi, *hi_sf;
  int64_t bytes;
  PackedAt(void* base, int64_t rows, int64_t k_lo, int64_t k_hi) {
    uint8_t* at = static_cast<uint8_t*>(base);
    const int64_t n[4] = {up256(rows * (k_lo / 2)), up256(api.sf_tiled_bytes(rows, k_lo / 16)), up256(rows * k_hi),
                          up256(api.sf_tiled_bytes(rows, k_hi / 32))};
    lo = at; lo_sf = lo + n[0]; hi = lo_sf + n[1]; hi_sf = hi + n[2];
    bytes = n[0] + n[1] + n[2] + n[3];
  }
};

Tensor checked_gamma(const Tensor& gamma, int64_t k) {
  if (!gamma.is_cuda()) throw std::runtime_error("gamma must be a CUDA tensor: plaquant_b200 has no CPU path");
  if (gamma.scalar_type() != at::kBFloat16 || gamma.numel() != k) throw pybind11::type_error("gamma must be bfloat16 [K]");
  return gamma.contiguous();
}

// [RMSNorm] -> [Hadamard] -> pack of bf16 CUDA x[..., K] into new buffers: (lo_codes, lo_sf, hi_codes, hi_sf).
std::tuple<Tensor, Tensor, Tensor, Tensor> pack(const Tensor& x, int64_t k_hi, bool hadamard, bool tiled,
                                                const std::optional<Tensor>& gamma, double eps) {
  const int64_t k = x.size(-1), k_lo = k - k_hi;
  const Tensor g = gamma ? checked_gamma(*gamma, k) : Tensor();
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor x2 = x.reshape({-1, k}).contiguous();
  const int64_t rows = x2.size(0);
  const auto u8 = x.options().dtype(at::kByte);
  Tensor lo = at::empty({rows, k_lo / 2}, u8), hi = at::empty({rows, k_hi}, u8), lo_sf, hi_sf;
  if (tiled) {
    lo_sf = at::empty({api.sf_tiled_bytes(rows, k_lo / 16)}, u8);
    hi_sf = at::empty({api.sf_tiled_bytes(rows, k_hi / 32)}, u8);
  } else {
    lo_sf = at::empty({rows, k_lo / 16}, u8);
    hi_sf = at::empty({rows, k_hi / 32}, u8);
  }
  auto at = [](const Tensor& t) { return t.numel() == 0 ? nullptr : t.data_ptr(); };
  const int layout = tiled ? PLQ_SF_TILED : PLQ_SF_ROWMAJOR;
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  check(gamma ? api.rmsnorm_pack(ptr(x2), g.const_data_ptr(), static_cast<float>(eps), rows, k, k_hi, hadamard, at(lo), at(lo_sf),
                                 at(hi), at(hi_sf), layout, stream)
              : api.pack(ptr(x2), rows, k, k_hi, hadamard, at(lo), at(lo_sf), at(hi), at(hi_sf), layout, stream));
  return {lo, lo_sf, hi, hi_sf};
}

// A packed weight: B operand of the products, and the status word their kernels report to.
struct Linear {
  Tensor lo, lo_sf, hi, hi_sf, status;
  int64_t n, k_lo, k_hi;
  int64_t k() const { return k_lo + k_hi; }
  int64_t packed_bytes(int64_t rows) const { return PackedAt(nullptr, rows, k_lo, k_hi).bytes; }

  // `like`: the choice of kernel for another number of rows (the two sum K in different orders).
  int product(const PackedAt& a, int64_t rows, void* y, int64_t ldy, void* stream, int64_t like = 0) const {
    int32_t* st = status.data_ptr<int32_t>();
    if (std::max(rows, like) <= 16)      // decode: stream the weights once; every product here has a pack in front of it
      return api.gemv_tc(a.lo, a.lo_sf, a.hi, a.hi_sf, ptr(lo), ptr(lo_sf), ptr(hi), ptr(hi_sf), rows, n, k_lo, k_hi, y, ldy, st,
                         PLQ_GEMV_STATIC_B | PLQ_GEMV_INTERLEAVED, stream);
    return api.mixed_gemm(a.lo, a.lo_sf, a.hi, a.hi_sf, ptr(lo), ptr(lo_sf), ptr(hi), ptr(hi_sf), rows, n, k_lo, k_hi, y, ldy, st,
                          stream);
  }

  // [RMSNorm] -> [Hadamard] -> pack -> product of x[..., K]; nullopt for an input that the Python path has to look at
  // (another dtype, device or K, no rows): it raises what it always raised.
  std::optional<Tensor> forward(const Tensor& x, bool hadamard, const std::optional<Tensor>& gamma, double eps,
                                const std::optional<Tensor>& out) const {
    if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.size(-1) != k() || x.device() != lo.device() ||
        x.numel() == 0)
      return std::nullopt;
    const Tensor g = gamma ? checked_gamma(*gamma, k()) : Tensor();
    pybind11::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = x.contiguous();
    const int64_t rows = x.numel() / k();
    const Tensor ws = at::empty({packed_bytes(rows)}, x.options().dtype(at::kByte));
    Tensor y = out ? *out : at::empty({rows, n}, x.options());
    void* stream = c10::cuda::getCurrentCUDAStream().stream();
    const PackedAt p(ws.data_ptr(), rows, k_lo, k_hi);
    check(gamma ? api.rmsnorm_pack(x2.const_data_ptr(), g.const_data_ptr(), static_cast<float>(eps), rows, k(), k_hi, hadamard, p.lo,
                                   p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream)
                : api.pack(x2.const_data_ptr(), rows, k(), k_hi, hadamard, p.lo, p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    check(product(p, rows, y.data_ptr(), y.stride(0), stream));
    if (x.dim() == 2 && !out) return y;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = n;
    return y.view(shape);
  }
};

Tensor heads_first(const Tensor& t) { return t.transpose(1, 2); }

// One decoder layer on one GPU: h + delta -> RMSNorm(ln1) -> qkv -> RoPE, cache append -> attention -> o_proj -> residual,
// RMSNorm(ln2) -> gate_up -> SiLU * up -> down_proj.  Returns (residual stream, down_proj's output not added to it yet).
// k_view / v_view: the first `ctx` positions of caches allocated for `cap`; the new rows go to `pos` (or *pos_dev).
// More than one position per sequence: all of them (a causal mask over the positions themselves) or with a mask.
// Packed caches (uint8) need `had`, the float32 Hadamard of the queries.  With `last_only` everything behind the attention
// runs for the last position of each sequence alone, results [B, 1, hidden] (the same bits: rows are independent).
std::tuple<Tensor, Tensor> decoder_layer(const Linear& qkv, const Linear& o, const Linear& gate_up, const Linear& down,
                                         const Tensor& ln1, const Tensor& ln2, int64_t heads, int64_t kv_heads, double eps_,
                                         const Tensor& h, const std::optional<Tensor>& delta, const Tensor& cos,
                                         const Tensor& sin, const Tensor& k_view, const Tensor& v_view, int64_t cap, int64_t pos,
                                         const std::optional<Tensor>& pos_dev, const std::optional<Tensor>& mask,
                                         const std::optional<Tensor>& had, bool last_only) {
  pybind11::gil_scoped_release nogil;
  const c10::cuda::CUDAGuard guard(h.device());
  const int64_t b = h.size(0), t = h.size(1), hidden = h.size(2), rows = b * t, ctx = k_view.size(1);
  const int64_t nq = (heads + 2 * kv_heads) * 128, ffn = down.k(), attn_width = heads * 128;
  TORCH_CHECK(h.is_contiguous() && h.scalar_type() == at::kBFloat16 && (!delta || (delta->is_contiguous() && delta->sizes() == h.sizes())),
              "h and delta must be contiguous bfloat16 [B, T, hidden]");
  TORCH_CHECK(qkv.n == nq && qkv.k() == hidden && o.k() == attn_width && o.n == hidden && gate_up.k() == hidden &&
                  gate_up.n == 2 * ffn && down.n == hidden && ffn % 128 == 0,
              "the layer's linears do not fit together");
  TORCH_CHECK(cos.numel() == t * 128 && sin.numel() == t * 128 && cos.is_contiguous() && sin.is_contiguous(), "cos / sin: one row per new position");
  const bool packed = k_view.scalar_type() == at::kByte;
  const int64_t width = packed ? 72 : 128;
  for (const Tensor* c : {&k_view, &v_view})
    TORCH_CHECK(c->size(0) == b && c->size(1) == ctx && c->size(2) == kv_heads && c->size(3) == width && ctx <= cap &&
                    c->scalar_type() == k_view.scalar_type() && (b == 1 || c->stride(0) == cap * kv_heads * width) &&
                    c->stride(1) == kv_heads * width && c->stride(2) == width && c->stride(3) == 1,
                "the caches must be the leading positions of contiguous allocations");
  TORCH_CHECK(t == 1 || mask || t == ctx, "a chunk behind a prompt needs a mask");
  int64_t packed_bytes = 0;
  for (const Linear* l : {&qkv, &o, &gate_up, &down}) packed_bytes = std::max(packed_bytes, l->packed_bytes(rows));
  const auto opts = h.options();
  // Workspace: the packed operand of the linear that runs, then its output; qkv's is dead before o's is written, and the
  // attention's operands have storage of their own.
  const bool gated = rows > 16;                        // the GEMM applies SiLU(gate) * up itself: one column per pair
  const int64_t out0 = up256(2 * rows * hidden);
  const Tensor ws = at::empty({packed_bytes + std::max(2 * rows * nq, out0 + (gated ? 2 : 4) * rows * ffn)}, opts.dtype(at::kByte));
  uint8_t* act = static_cast<uint8_t*>(ws.data_ptr()) + packed_bytes;
  void* stream = c10::cuda::getCurrentCUDAStream().stream();
  int32_t* status = qkv.status.data_ptr<int32_t>();
  const float eps = static_cast<float>(eps_);

  Tensor h1 = h;
  {
    const PackedAt p(ws.data_ptr(), rows, qkv.k_lo, qkv.k_hi);
    if (delta) {
      h1 = at::empty_like(h);
      check(api.add_rmsnorm_pack(delta->const_data_ptr(), h.const_data_ptr(), h1.data_ptr(), ln1.const_data_ptr(), eps, rows, hidden,
                                 qkv.k_hi, 1, p.lo, p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    } else {
      check(api.rmsnorm_pack(h.const_data_ptr(), ln1.const_data_ptr(), eps, rows, hidden, qkv.k_hi, 1, p.lo, p.lo_sf, p.hi, p.hi_sf,
                             PLQ_SF_TILED, stream));
    }
    check(qkv.product(p, rows, act, nq, stream));
  }
  Tensor q = at::empty({b, t, heads, 128}, packed ? opts.dtype(at::kFloat) : opts), kk = k_view, vv = v_view;
  const int64_t* at_pos = pos_dev ? pos_dev->const_data_ptr<int64_t>() : nullptr;
  if (packed) {
    kk = at::empty({b, ctx, kv_heads, 128}, opts);
    vv = at::empty_like(kk);
    check(api.rope_kv_append_nvfp4_values(act, nq, cos.const_data_ptr(), sin.const_data_ptr(), b, t, heads, kv_heads, 128, q.data_ptr(),
                                          k_view.data_ptr(), v_view.data_ptr(), cap, at_pos, pos, ctx, kk.data_ptr(), vv.data_ptr(),
                                          status, stream));
    q = at::matmul(q, *had).to(at::kBFloat16);
  } else {
    check(api.rope_kv_append(act, nq, cos.const_data_ptr(), sin.const_data_ptr(), b, t, heads, kv_heads, 128, q.data_ptr(),
                             k_view.data_ptr(), v_view.data_ptr(), cap, at_pos, pos, status, stream));
  }
  Tensor attn = heads_first(at::scaled_dot_product_attention(heads_first(q), heads_first(kk), heads_first(vv), mask, 0.0,
                                                                   !mask && t > 1, std::nullopt, true))
                          .contiguous();

  const int64_t like = rows;
  if (last_only) {
    attn = attn.slice(1, t - 1).contiguous();
    h1 = h1.slice(1, t - 1).contiguous();
  }
  const int64_t out_rows = last_only ? b : rows;
  Tensor h2 = at::empty_like(h1), delta2 = at::empty_like(h1);
  uint8_t* gu = act + out0;
  {
    const PackedAt p(ws.data_ptr(), out_rows, o.k_lo, o.k_hi);
    check(api.pack(attn.const_data_ptr(), out_rows, attn_width, o.k_hi, 1, p.lo, p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    check(o.product(p, out_rows, act, hidden, stream, like));
  }
  {
    const PackedAt p(ws.data_ptr(), out_rows, gate_up.k_lo, gate_up.k_hi);
    check(api.add_rmsnorm_pack(act, h1.const_data_ptr(), h2.data_ptr(), ln2.const_data_ptr(), eps, out_rows, hidden, gate_up.k_hi, 1, p.lo,
                               p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    if (gated)
      check(api.mixed_gemm_silu_mul(p.lo, p.lo_sf, p.hi, p.hi_sf, ptr(gate_up.lo), ptr(gate_up.lo_sf), ptr(gate_up.hi), ptr(gate_up.hi_sf),
                                    out_rows, ffn, gate_up.k_lo, gate_up.k_hi, gu, ffn, status, stream));
    else
      check(gate_up.product(p, out_rows, gu, 2 * ffn, stream, like));
  }
  {
    const PackedAt p(ws.data_ptr(), out_rows, down.k_lo, down.k_hi);
    if (gated)
      check(api.pack(gu, out_rows, ffn, down.k_hi, 1, p.lo, p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    else
      check(api.silu_mul_pack(gu, gu + 2 * ffn, 2 * ffn, out_rows, ffn, down.k_hi, 1, p.lo, p.lo_sf, p.hi, p.hi_sf, PLQ_SF_TILED, stream));
    check(down.product(p, out_rows, delta2.data_ptr(), hidden, stream, like));
  }
  return {h2, delta2};
}

// Does nothing else share the memory of a or of b?  (The base that a view keeps alive does not count.)
bool alone(const Tensor& a, const Tensor& b) {
  auto one = [](const Tensor& t) { return t.storage().use_count() == (t.is_view() ? 2u : 1u); };
  return one(a) && one(b);
}

}  // namespace

PYBIND11_MODULE(_plq_torch, m) {
  pybind11::class_<Linear>(m, "Linear")
      .def(pybind11::init([](Tensor lo, Tensor lo_sf, Tensor hi, Tensor hi_sf, Tensor status, int64_t n, int64_t k_lo, int64_t k_hi) {
        return Linear{lo, lo_sf, hi, hi_sf, status, n, k_lo, k_hi};
      }))
      .def("forward", &Linear::forward);
  m.def("init", &init);
  m.def("pack", &pack);
  m.def("alone", &alone);
  m.def("decoder_layer", &decoder_layer);
}
