// Host path of the operators: argument checks, output and scratch allocation, stride handling and the
// calls into the C ABI, in one native call per operator.
//
// What bounds it: nothing but host instructions.  Driving the C ABI from Python through ctypes cost
// 15-25 us per launch (about thirty argument conversions, a data_ptr / stride call for each, three to
// eight torch.empty calls, the stream and device look-ups); a decode step of three launches spent 68 us
// on the host for 14 us of GPU work.  Here an operator costs its launches (2.1 us each, its C entry included), its
// allocations (0.55 us each, release included), 0.3 to 1.6 us of guards, checks and views, and 1.2 to 1.6 us of argument
// parsing in the interpreter: a decode step 6.5 + 1.1 + 1.7 + 4.3 = 13.6 us, a short prompt with its cache
// 5.9 + 3.9 + 1.9 + 3.4 = 15.1.  The GIL is released for the whole of a call.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <array>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../../include/nvfp4_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int64_t kKeyTile = 128;

struct AssertionFailure : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct UnsupportedType : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct NotImplemented : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline void require(bool ok, const char* msg) {
  if (__builtin_expect(!ok, 0)) throw AssertionFailure(msg);
}

// An operand of another number of dimensions is a ValueError, as it is where a shape is unpacked.
inline void require_dims(const Tensor& t, int64_t n, const char* msg) {
  if (__builtin_expect(t.dim() != n, 0)) throw std::invalid_argument(msg);
}

inline int64_t next_mult(int64_t n, int64_t m) { return (n + m - 1) / m * m; }

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return NVFP4_DT_BF16;
    case at::kHalf: return NVFP4_DT_FP16;
    case at::kFloat: return NVFP4_DT_FP32;
    default:
      throw UnsupportedType(std::string("unsupported dtype torch.") + c10::toString(t) +
                            "; expected bfloat16, float16 or float32");
  }
}

void require_cuda(const Tensor& t, const char* name) {
  if (__builtin_expect(!t.is_cuda(), 0))
    throw std::runtime_error(std::string(name) + " must be a CUDA tensor: sageattention_b200 has no CPU path (got device " +
                             t.device().str() + ")");
}

// ---------------------------------------------------------------- device, stream, status word
// One int32 per device that kernels write when a bounded wait expires; allocated on first use.
std::mutex g_status_mutex;
std::vector<Tensor>& status_words() {
  static auto* v = new std::vector<Tensor>(64);      // never destroyed: CUDA may be gone at exit
  return *v;
}
Tensor status_word(int64_t index) {
  std::lock_guard<std::mutex> lock(g_status_mutex);
  auto& v = status_words();
  if (index >= (int64_t)v.size()) v.resize(index + 1);
  if (!v[index].defined())
    v[index] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, (c10::DeviceIndex)index));
  return v[index];
}

// The device of a call made current, its stream, the status word and the check of return codes.
struct Call {
  at::Device dev;
  c10::cuda::CUDAGuard guard;
  c10::NoGradGuard no_grad;
  cudaStream_t stream;
  int* status;

  explicit Call(const Tensor& t)
      : dev(t.device()), guard(dev), stream(c10::cuda::getCurrentCUDAStream(dev.index()).stream()),
        status(status_word(dev.index()).data_ptr<int>()) {}

  void same(const Tensor& t) const {
    if (__builtin_expect(t.device() == dev, 1)) return;
    if (!t.is_cuda())
      throw std::runtime_error("operands must be CUDA tensors: sageattention_b200 has no CPU path (got device " +
                               t.device().str() + ")");
    throw std::runtime_error("operands live on different devices: " + dev.str() + " and " + t.device().str());
  }
  void same(const OptTensor& t) const {
    if (t.has_value()) same(*t);
  }

  void done(int rc, const char* what) const {
    if (__builtin_expect(rc != 0, 0))
      throw std::runtime_error(std::string(what) + " failed (code " + std::to_string(rc) + "): " + nvfp4_last_error());
    const char* e = std::getenv("NVFP4_CHECK_STATUS");
    if (__builtin_expect(e != nullptr && std::strcmp(e, "1") == 0, 0)) {
      Tensor w = status_word(dev.index());
      const int st = w.item<int>();                  // synchronising read, debug mode only
      if (st) {
        w.zero_();
        char msg[160];
        std::snprintf(msg, sizeof msg, "%s: a bounded in-kernel wait expired (status 0x%x: site %d); outputs of this call are undefined",
                      what, st, st & 0xFF);
        throw std::runtime_error(msg);
      }
    }
  }

  Tensor empty(at::IntArrayRef sizes, at::ScalarType t) const {
    return at::detail::empty_cuda(sizes, t, dev, std::nullopt);
  }
};

inline uint8_t* u8(const Tensor& t) { return static_cast<uint8_t*>(t.data_ptr()); }
template <typename T = void>
inline T* opt_ptr(const OptTensor& t) { return t.has_value() ? static_cast<T*>(t->data_ptr()) : nullptr; }

// [B1, B2, S, D] seen as [B1*B2, S, D] rows: base pointer and strides, `keep` owning a copy where the
// two batch axes do not collapse.
struct Rows {
  Tensor keep;
  const void* p;
  int64_t b, r, k, sb, sr, sk;
};
Rows rows_of(const Tensor& t) {
  if (t.dim() == 3) return {t, t.data_ptr(), t.size(0), t.size(1), t.size(2), t.stride(0), t.stride(1), t.stride(2)};
  require(t.dim() == 4, "expected a [Z, H, S, D] tensor");
  const auto sz = t.sizes();
  const auto st = t.strides();
  const int64_t b = sz[0] * sz[1];
  if (sz[0] == 1 || sz[1] == 1 || st[0] == sz[1] * st[1]) {
    const int64_t sb = sz[1] == 1 ? st[0] : st[1];
    return {t, t.data_ptr(), b, sz[2], sz[3], sb, st[2], st[3]};
  }
  Tensor c = t.contiguous();
  return {c, c.data_ptr(), b, sz[2], sz[3], sz[2] * sz[3], sz[3], 1};
}

// A [Z, H, S, D] operand of known extents: as it is, or (any other shape of as many elements) reshaped to
// [Z*H, S, D] rows.  Throws where the elements do not make up the extents: the kernels take their sizes from
// one operand and would read past the end of another.
Tensor as_rows(const Tensor& t, int64_t b, int64_t s, int64_t d) {
  if (t.dim() == 4 && t.size(0) * t.size(1) == b && t.size(2) == s && t.size(3) == d) return t;
  return t.reshape({b, s, d});
}

// ---------------------------------------------------------------- packers
void pack_rows_call(const Call& c, const Rows& x, int dt, int64_t r, int64_t k_read, int64_t kp, int64_t sxr, int64_t sxk,
                    uint8_t* nib, int64_t snb, int64_t snr, uint8_t* sc, int64_t ssb, int64_t ssr) {
  if (x.b * r * kp == 0) return;
  c.done(nvfp4_pack(x.p, dt, x.b, r, k_read, kp, x.sb, sxr, sxk, nib, snb, snr, sc, ssb, ssr, c.stream), "nvfp4_pack");
}

void pack_into(const Tensor& x, const Tensor& nib, const Tensor& sc, bool transpose, std::optional<int64_t> k_pad) {
  require_cuda(x, "x");
  Call c(x);
  c.same(nib);
  c.same(sc);
  require_dims(x, 3, "x must be three-dimensional");
  const Rows xr = rows_of(x);
  const int64_t r = transpose ? xr.k : xr.r, k_read = transpose ? xr.r : xr.k;
  const int64_t sxr = transpose ? xr.sk : xr.sr, sxk = transpose ? xr.sr : xr.sk;
  const int64_t kp = k_pad.value_or(k_read);
  require(kp % 16 == 0, "padded contraction dim must be a multiple of 16");
  require(kp >= k_read, "k_pad must cover the contraction axis");
  require(nib.dim() == 3 && sc.dim() == 3 && nib.size(0) == xr.b && nib.size(1) == r && nib.size(2) == kp / 2 &&
              sc.size(0) == xr.b && sc.size(1) == r && sc.size(2) == kp / 16,
          "output view shape mismatch");
  require(nib.stride(2) == 1 && sc.stride(2) == 1, "output rows must be contiguous");
  pack_rows_call(c, xr, dtype_code(x.scalar_type()), r, k_read, kp, sxr, sxk, u8(nib), nib.stride(0), nib.stride(1),
                 u8(sc), sc.stride(0), sc.stride(1));
}

struct Pack {
  Tensor nib, sc;
};

Pack quant_rows(const Call& c, const Rows& x, at::ScalarType t, bool transpose, std::optional<int64_t> k_pad) {
  const int64_t r = transpose ? x.k : x.r, k_read = transpose ? x.r : x.k;
  const int64_t kp = k_pad.value_or(k_read);
  require(kp % 16 == 0, "padded contraction dim must be a multiple of 16");
  require(kp >= k_read, "k_pad must cover the contraction axis");
  Pack p{c.empty({x.b, r, kp / 2}, at::kByte), c.empty({x.b, r, kp / 16}, at::kFloat8_e4m3fn)};
  pack_rows_call(c, x, dtype_code(t), r, k_read, kp, transpose ? x.sk : x.sr, transpose ? x.sr : x.sk, u8(p.nib),
                 r * (kp / 2), kp / 2, u8(p.sc), r * (kp / 16), kp / 16);
  return p;
}

std::tuple<Tensor, Tensor> quant(const Tensor& x, bool transpose, std::optional<int64_t> k_pad) {
  require_cuda(x, "x");
  require_dims(x, 3, "x must be three-dimensional");
  Call c(x);
  Pack p = quant_rows(c, rows_of(x), x.scalar_type(), transpose, k_pad);
  return {p.nib, p.sc};
}

std::tuple<Tensor, Tensor> rope_quant(const Tensor& x, const Tensor& cos, const Tensor& sin, const OptTensor& positions,
                                      int64_t pos0) {
  require_cuda(x, "x");
  Call c(x);
  require_dims(x, 3, "x must be [B, R, D]");
  const int64_t b = x.size(0), r = x.size(1), d = x.size(2);
  require(x.stride(2) == 1, "rows must be contiguous along D");
  require(cos.size(-1) == d / 2 && sin.sizes() == cos.sizes() && cos.scalar_type() == at::kFloat,
          "cos / sin must be fp32 [P, D/2]");
  const Tensor cs = cos.contiguous(), sn = sin.contiguous();
  c.same(cs);
  c.same(sn);
  OptTensor pos;
  if (positions.has_value()) {
    pos = positions->to(x.device(), at::kInt).contiguous();
    require(pos->numel() == r, "one position per row");
  }
  Tensor nib = c.empty({b, r, d / 2}, at::kByte), sc = c.empty({b, r, d / 16}, at::kFloat8_e4m3fn);
  c.done(nvfp4_rope_pack(x.data_ptr(), dtype_code(x.scalar_type()), b, r, (int)d, x.stride(0), x.stride(1),
                         cs.data_ptr<float>(), sn.data_ptr<float>(), opt_ptr<int32_t>(pos), pos0, u8(nib), r * (d / 2), d / 2,
                         u8(sc), r * (d / 16), d / 16, c.stream),
         "nvfp4_rope_pack");
  return {nib, sc};
}

std::tuple<Tensor, Tensor> quant_mxfp8_t(const Tensor& x_in, int64_t s_pad, const OptTensor& amax) {
  require_cuda(x_in, "x");
  Call c(x_in);
  require_dims(x_in, 3, "x must be [B, S, D]");
  const int64_t b = x_in.size(0), s = x_in.size(1), d = x_in.size(2);
  require(s_pad % 32 == 0 && s_pad >= s, "s_pad must be a multiple of 32 covering S");
  const Tensor x = x_in.stride(2) == 1 ? x_in : x_in.contiguous();
  Tensor out = c.empty({b, d, s_pad}, at::kByte), sc = c.empty({b, d, s_pad / 32}, at::kByte);
  if (b * s_pad > 0)
    c.done(nvfp4_pack_mx8_t(x.data_ptr(), dtype_code(x.scalar_type()), b, s, (int)d, s_pad, x.stride(0), x.stride(1),
                            opt_ptr<float>(amax), u8(out), u8(sc), c.stream),
           "nvfp4_pack_mx8_t");
  return {out, sc};
}

std::tuple<Tensor, Tensor, OptTensor> vproj_quant(const Tensor& x_in, const Tensor& weight_in, const OptTensor& bias_in,
                                                  int64_t hk, int64_t d, std::optional<int64_t> s_pad, bool return_value) {
  require_cuda(x_in, "x");
  Call c(x_in);
  require_dims(x_in, 3, "x must be [Z, S, hidden]");
  const int64_t z = x_in.size(0), s = x_in.size(1), hidden = x_in.size(2), feats = hk * d;
  require(weight_in.dim() == 2 && weight_in.size(0) == feats && weight_in.size(1) == hidden, "weight must be [Hk*D, hidden]");
  const auto t = x_in.scalar_type();
  require((t == at::kBFloat16 || t == at::kHalf) && weight_in.scalar_type() == t, "operands must be bf16 or fp16");
  require(hidden % 8 == 0 && d % 16 == 0, "hidden must be a multiple of 8 and head_dim of 16");
  const Tensor x = (x_in.stride(2) != 1 || x_in.stride(0) % 8 || x_in.stride(1) % 8) ? x_in.contiguous() : x_in;
  const Tensor w = weight_in.contiguous();
  c.same(w);
  OptTensor bias;
  if (bias_in.has_value()) {
    c.same(*bias_in);
    bias = bias_in->to(t).contiguous();
    require(bias->numel() == feats, "bias must have Hk*D elements");
  }
  const int64_t sp = s_pad.value_or(next_mult(s, kKeyTile));
  require(sp % 16 == 0 && sp >= s, "s_pad must be a multiple of 16 covering S");
  Tensor vnv = c.empty({z * hk, d, sp / 2}, at::kByte), vsc = c.empty({z * hk, d, sp / 16}, at::kFloat8_e4m3fn);
  OptTensor v;
  if (return_value) v = c.empty({z, s, hk, d}, t);
  c.done(nvfp4_vproj_pack(x.data_ptr(), w.data_ptr(), opt_ptr<>(bias), dtype_code(t), z, s, hidden, hk, (int)d, x.stride(0),
                          x.stride(1), sp, u8(vnv), u8(vsc), opt_ptr<>(v), return_value ? s * feats : 0,
                          return_value ? feats : 0, c.status, c.stream),
         "nvfp4_vproj_pack");
  if (return_value) v = v->permute({0, 2, 1, 3});
  return {vnv, vsc, v};
}

struct Dual {
  Tensor dn, ds, tn, ts;
};
Dual quant_dual_rows(const Call& c, const Rows& x, at::ScalarType t, int64_t sp, const float* amax, int sr, uint32_t seed) {
  require(sp % 16 == 0 && sp >= x.r, "s_pad must be a multiple of 16 covering S");
  require(x.k % 16 == 0, "D must be a multiple of 16");
  Dual o{c.empty({x.b, x.r, x.k / 2}, at::kByte), c.empty({x.b, x.r, x.k / 16}, at::kFloat8_e4m3fn),
         c.empty({x.b, x.k, sp / 2}, at::kByte), c.empty({x.b, x.k, sp / 16}, at::kFloat8_e4m3fn)};
  if (x.b * sp > 0)
    c.done(nvfp4_pack_dual(x.p, dtype_code(t), x.b, x.r, (int)x.k, sp, x.sb, x.sr, amax, sr, seed, u8(o.dn), u8(o.ds), u8(o.tn),
                           u8(o.ts), c.stream),
           "nvfp4_pack_dual");
  return o;
}

Rows unit_rows(const Tensor& t) {      // rows with unit stride along D
  Rows r = rows_of(t);
  if (r.sk == 1) return r;
  return rows_of(t.contiguous());
}

std::tuple<Tensor, Tensor, Tensor, Tensor> quant_dual(const Tensor& x, std::optional<int64_t> s_pad, const OptTensor& amax,
                                                      bool sr_d, bool sr_s, int64_t seed) {
  require_cuda(x, "x");
  require_dims(x, 3, "x must be [B, S, D]");
  Call c(x);
  Dual o = quant_dual_rows(c, unit_rows(x), x.scalar_type(), s_pad.value_or(next_mult(x.size(1), 16)), opt_ptr<float>(amax),
                           (sr_d ? 1 : 0) | (sr_s ? 2 : 0), (uint32_t)(seed & 0xFFFFFFFF));
  return {o.dn, o.ds, o.tn, o.ts};
}

// The six packs of a forward: Q, K along D and V along the keys.
struct FwdPacks {
  Tensor qn, qs, kn, ks, vn, vs;
};
bool qkv_fusable(const Rows& q, const Rows& k, const Rows& v, bool same_dtype, int64_t s_pad) {
  return same_dtype && q.sk == 1 && k.sk == 1 && v.sk == 1 && v.b == k.b && v.r == k.r && v.k == k.k && k.k == q.k &&
         (q.k == 64 || q.k == 128 || q.k == 256) && s_pad % 16 == 0 && q.b * q.r * k.b * k.r > 0;
}
FwdPacks quant_qkv_rows(const Call& c, const Tensor& qt, const Tensor& kt, const Tensor& vt, const Rows& q, const Rows& k,
                        const Rows& v, int64_t s_pad) {
  const auto t = qt.scalar_type();
  FwdPacks o;
  if (!qkv_fusable(q, k, v, kt.scalar_type() == t && vt.scalar_type() == t, s_pad)) {
    Pack a = quant_rows(c, q, t, false, std::nullopt), b = quant_rows(c, k, kt.scalar_type(), false, std::nullopt);
    Pack e = quant_rows(c, v, vt.scalar_type(), true, s_pad);
    return {a.nib, a.sc, b.nib, b.sc, e.nib, e.sc};
  }
  const int64_t d = q.k;
  o.qn = c.empty({q.b, q.r, d / 2}, at::kByte);
  o.qs = c.empty({q.b, q.r, d / 16}, at::kFloat8_e4m3fn);
  o.kn = c.empty({k.b, k.r, d / 2}, at::kByte);
  o.ks = c.empty({k.b, k.r, d / 16}, at::kFloat8_e4m3fn);
  o.vn = c.empty({k.b, d, s_pad / 2}, at::kByte);
  o.vs = c.empty({k.b, d, s_pad / 16}, at::kFloat8_e4m3fn);
  c.done(nvfp4_pack_qkv(q.p, k.p, v.p, dtype_code(t), q.b, k.b, q.r, k.r, s_pad, (int)d, q.sb, q.sr, k.sb, k.sr, v.sb, v.sr,
                        u8(o.qn), u8(o.qs), u8(o.kn), u8(o.ks), u8(o.vn), u8(o.vs), c.stream),
         "nvfp4_pack_qkv");
  return o;
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> quant_qkv(const Tensor& q, const Tensor& k, const Tensor& v,
                                                                     int64_t s_pad) {
  require_cuda(q, "q");
  Call c(q);
  c.same(k);
  c.same(v);
  FwdPacks o = quant_qkv_rows(c, q, k, v, rows_of(q), rows_of(k), rows_of(v), s_pad);
  return {o.qn, o.qs, o.kn, o.ks, o.vn, o.vs};
}

// ---------------------------------------------------------------- forward
OptTensor checked_bias(const Call& c, const OptTensor& bias, int64_t z, int64_t s_kv) {
  if (!bias.has_value()) return std::nullopt;
  OptTensor b = (bias->scalar_type() == at::kFloat && bias->device() == c.dev) ? bias->contiguous()
                                                                               : bias->to(c.dev, at::kFloat).contiguous();
  require(b->dim() == 2 && b->size(0) == z && b->size(1) == s_kv, "key_pad_bias must be [Z, Skv]");
  return b;
}

struct FwdOut {
  Tensor out;
  OptTensor lse;
};
FwdOut run_fwd(const Call& c, const FwdPacks& p, int64_t z, int64_t h, int64_t hk, int64_t s_q, int64_t s_kv, int64_t d,
               double scaling, at::ScalarType out_dtype, bool causal, const OptTensor& bias_in, const OptTensor& seq_id,
               const OptTensor& seq_start, bool zshd, bool want_lse) {
  require(d == 128 || d == 256, "D must be 128 or 256");
  const int64_t s_pad = p.vn.size(-1) * 2;
  require(s_pad % kKeyTile == 0 && s_pad >= s_kv, "V^T key axis must be padded to a multiple of the key tile (128)");
  const OptTensor bias = checked_bias(c, bias_in, z, s_kv);
  c.same(seq_id);
  c.same(seq_start);
  FwdOut o;
  int64_t so_z, so_h, so_s;
  if (zshd) {
    o.out = c.empty({z, s_q, h, d}, out_dtype);
    so_z = s_q * h * d; so_s = h * d; so_h = d;
  } else {
    o.out = c.empty({z, h, s_q, d}, out_dtype);
    so_z = h * s_q * d; so_h = s_q * d; so_s = d;
  }
  if (want_lse) o.lse = c.empty({z * h, s_q}, at::kFloat);
  c.done(nvfp4_fwd(u8(p.qn), u8(p.qs), u8(p.kn), u8(p.ks), u8(p.vn), u8(p.vs), opt_ptr<float>(bias), opt_ptr<int32_t>(seq_id),
                   opt_ptr<int32_t>(seq_start), o.out.data_ptr(), dtype_code(out_dtype), so_z, so_h, so_s,
                   opt_ptr<float>(o.lse), z, h, hk, s_q, s_kv, s_pad, (int)d, (float)scaling, causal ? NVFP4_FWD_CAUSAL : 0,
                   c.status, c.stream),
         "nvfp4_fwd");
  return o;
}

FwdPacks dense_packs(const Call& c, const Tensor& qn, const Tensor& qs, const Tensor& kn, const Tensor& ks, const Tensor& vn,
                     const Tensor& vs) {
  FwdPacks p{qn.contiguous(), qs.contiguous(), kn.contiguous(), ks.contiguous(), vn.contiguous(), vs.contiguous()};
  for (const Tensor* t : {&p.qn, &p.qs, &p.kn, &p.ks, &p.vn, &p.vs}) c.same(*t);
  return p;
}

std::tuple<Tensor, OptTensor> flash_packed(const Tensor& qn, const Tensor& qs, const Tensor& kn, const Tensor& ks,
                                           const Tensor& vn, const Tensor& vs, int64_t z, int64_t h, int64_t hk, int64_t s_q,
                                           int64_t s_kv, int64_t d, double scaling, at::ScalarType out_dtype, bool causal,
                                           const OptTensor& bias, const OptTensor& seq_id, const OptTensor& seq_start,
                                           bool zshd, bool want_lse) {
  require_cuda(qn, "qnv");
  Call c(qn);
  FwdOut o = run_fwd(c, dense_packs(c, qn, qs, kn, ks, vn, vs), z, h, hk, s_q, s_kv, d, scaling, out_dtype, causal, bias,
                     seq_id, seq_start, zshd, want_lse);
  return {o.out, o.lse};
}

void check_packs(const Tensor& nv, const Tensor& sc, int64_t b, int64_t r, int64_t k, const char* msg) {
  require(nv.dim() == 3 && sc.dim() == 3 && nv.size(0) == b && nv.size(1) == r && nv.size(2) == k / 2 && sc.size(0) == b &&
              sc.size(1) == r && sc.size(2) == k / 16,
          msg);
}

// Pack (unless the caller did) and attend; returns (out, lse | None, packs | ()).
std::tuple<Tensor, OptTensor, std::vector<Tensor>> flash_attention(
    const Tensor& query, const Tensor& key, const Tensor& value, double scaling, bool causal, int64_t g, const OptTensor& bias,
    bool varlen, const OptTensor& seq_id, const OptTensor& seq_start, bool zshd, bool want_lse, bool want_packs,
    const OptTensor& qnv, const OptTensor& qsc, const OptTensor& knv, const OptTensor& ksc) {
  require_cuda(query, "query");
  for (const Tensor* t : {&query, &key}) require_dims(*t, 4, "query and key must be [Z, H, S, D]");
  const int64_t z = query.size(0), h = query.size(1), s_q = query.size(2), d = query.size(3);
  const int64_t hk = key.size(1), s_kv = key.size(2);
  require(h == hk * g, "num_key_value_groups must equal H // Hk");
  require(d == 128 || d == 256, "D must be 128 or 256");
  if (causal && !varlen) require(s_kv >= s_q, "causal attention requires Skv >= Sq (bottom-right aligned mask)");
  if (varlen || seq_id.has_value()) {
    require(z == 1, "cu_seqlens varlen requires Z must be 1 (one packed row)");
    require(s_q == s_kv, "cu_seqlens varlen requires Sq == Skv");
  }
  if (varlen) require(causal, "cu_seqlens varlen is block-diagonal causal: pass causal=True");
  Call c(query);
  c.same(key);
  c.same(value);
  const int64_t s_pad = next_mult(s_kv, kKeyTile);
  const Rows q = rows_of(query), k = rows_of(as_rows(key, z * hk, s_kv, d)), v = rows_of(as_rows(value, z * hk, s_kv, d));
  FwdPacks p;
  if (!qnv.has_value() && !knv.has_value()) {
    p = quant_qkv_rows(c, query, key, value, q, k, v, s_pad);       // one launch
  } else {
    Pack a, b;
    if (qnv.has_value()) {
      a = {*qnv, qsc.value()};
      check_packs(a.nib, a.sc, z * h, s_q, d, "q_packs layout mismatch: expected along-D packs of the query rows");
    } else {
      a = quant_rows(c, q, query.scalar_type(), false, std::nullopt);
    }
    if (knv.has_value()) {
      b = {*knv, ksc.value()};
      check_packs(b.nib, b.sc, z * hk, s_kv, d, "k_packs layout mismatch: expected along-D packs of the key rows");
    } else {
      b = quant_rows(c, k, key.scalar_type(), false, std::nullopt);
    }
    Pack e = quant_rows(c, v, value.scalar_type(), true, s_pad);
    p = {a.nib, a.sc, b.nib, b.sc, e.nib, e.sc};
  }
  const bool external = qnv.has_value() || knv.has_value();
  FwdOut o = run_fwd(c, external ? dense_packs(c, p.qn, p.qs, p.kn, p.ks, p.vn, p.vs) : p, z, h, hk, s_q, s_kv, d, scaling,
                     query.scalar_type(), causal, bias, seq_id, seq_start, zshd, want_lse);
  std::vector<Tensor> packs;
  if (want_packs) packs = {p.qn, p.qs, p.kn, p.ks, p.vn, p.vs};
  return {o.out, o.lse, std::move(packs)};
}

// ---------------------------------------------------------------- decode
struct DecodeArgs {
  int64_t z, h, hk, d;
  const Tensor *knv, *ksc, *vnv, *vsc;
  int64_t s_kv;
  double scaling;
  int64_t g;
};

struct Window {                        // the high-precision side of a hybrid decode
  const Tensor *rk, *rv;
  int64_t ring_cap, first, count;
  int pieces;
};

// Split-K decode over the packed cache, plus (hybrid) the window's partials merged by the same combine.
std::tuple<Tensor, OptTensor> decode_core(const Call& c, const Tensor& query, const DecodeArgs& a, bool want_lse,
                                          std::optional<int64_t> split_in, const Window* win) {
  require(a.d % 16 == 0 && (a.d == 128 || a.d == 256), "D must be 128 or 256");
  const int64_t zhk = a.knv->size(0);
  require(zhk % a.z == 0, "packed KV batch must be a multiple of Z");
  const int64_t hk = zhk / a.z;
  require(a.h % hk == 0 && a.h / hk == a.g, "G mismatch vs packed KV");
  if (a.g > 16) throw AssertionFailure("GQA group " + std::to_string(a.g) + " must be <= 16");
  require(a.s_kv >= 1, "decode needs at least one key");
  const Tensor q = query.stride(3) == 1 ? query : query.contiguous();
  for (const Tensor* t : {a.knv, a.ksc, a.vnv, a.vsc}) {
    c.same(*t);
    require(t->stride(-1) == 1, "packed cache rows must be contiguous");
  }
  require(a.knv->stride(1) == a.d / 2 && a.ksc->stride(1) == a.d / 16, "K rows must be dense");
  const int64_t slot_bytes = (16 * a.d + 32) * 4;
  const int sms = at::cuda::getDeviceProperties(c.dev.index())->multiProcessorCount;
  int nsplit = 0;
  int64_t split_kv = 0;
  size_t wbytes = 0;
  if (!split_in.has_value()) {
    c.done(nvfp4_decode_plan(a.s_kv, zhk, (int)a.d, sms, &nsplit, &split_kv, &wbytes), "nvfp4_decode_plan");
  } else if (*split_in == 0) {
    // the balanced decomposition (every CTA streams an equal share of all key tiles), forced
    const int64_t tiles = (a.s_kv + 127) / 128, total = zhk * tiles;
    const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>(sms, std::max<int64_t>(total / 4, 1)));
    const int64_t per = (total + ctas - 1) / ctas;
    wbytes = (size_t)(ctas * ((per + tiles - 2) / tiles + 1) * slot_bytes);
  } else {
    split_kv = *split_in;
    require(split_kv % 128 == 0, "split_kv must be a multiple of 128");
    nsplit = (int)((a.s_kv + split_kv - 1) / split_kv);
    wbytes = (size_t)(zhk * nsplit * slot_bytes);
  }
  wbytes += (size_t)(win ? zhk * win->pieces * slot_bytes : 0);       // the window's partials behind the decode's own
  Tensor ws = c.empty({(int64_t)wbytes}, at::kByte);
  Tensor out = c.empty({a.z, a.h, 1, a.d}, q.scalar_type());
  OptTensor lse;
  if (want_lse) lse = c.empty({a.z, a.h}, at::kFloat);
  auto run = [&](auto entry, const char* what, auto... window) {
    c.done(entry(q.data_ptr(), dtype_code(q.scalar_type()), q.stride(0), q.stride(1), u8(*a.knv), a.knv->stride(0), u8(*a.ksc),
                 a.ksc->stride(0), u8(*a.vnv), a.vnv->stride(0), a.vnv->stride(1), u8(*a.vsc), a.vsc->stride(0),
                 a.vsc->stride(1), a.z, hk, (int)a.g, (int)a.d, a.s_kv, (float)a.scaling, out.data_ptr(), opt_ptr<float>(lse),
                 ws.data_ptr(), wbytes, nsplit, split_kv, window..., c.status, c.stream),
           what);
  };
  if (win)
    run(nvfp4_decode_window, "nvfp4_decode_window", win->rk->data_ptr(), win->rv->data_ptr(), win->ring_cap, win->first,
        win->count, win->pieces);
  else
    run(nvfp4_decode, "nvfp4_decode");
  return {out, lse};
}

std::tuple<Tensor, OptTensor> decode(const Tensor& query, const Tensor& knv, const Tensor& ksc, const Tensor& vnv,
                                     const Tensor& vsc, int64_t s_kv, double scaling, int64_t g, bool want_lse,
                                     std::optional<int64_t> split_kv) {
  require_cuda(query, "query");
  require_dims(query, 4, "query must be [Z, H, 1, D]");
  require(query.size(2) == 1, "nvfp4_flash_decode is for seqlen_q == 1 (decode)");
  Call c(query);
  const DecodeArgs a{query.size(0), query.size(1), 0, query.size(3), &knv, &ksc, &vnv, &vsc, s_kv, scaling, g};
  return decode_core(c, query, a, want_lse, split_kv, nullptr);
}

Tensor hybrid_decode(const Tensor& query, const Tensor& knv, const Tensor& ksc, const Tensor& vnv, const Tensor& vsc,
                     const Tensor& rk, const Tensor& rv, int64_t length, int64_t recent_window, double scaling, int64_t g) {
  require_cuda(query, "query");
  require_dims(query, 4, "query must be [Z, H, 1, D]");
  require(query.size(2) == 1, "nvfp4_flash_decode is for seqlen_q == 1 (decode)");
  Call c(query);
  c.same(rk);
  c.same(rv);
  const int64_t z = query.size(0), h = query.size(1), d = query.size(3), hk = rk.size(1), cap = rk.size(2);
  require(rk.dim() == 4 && rk.size(0) == z && rk.size(3) == d && h == hk * g, "query does not fit the window's rings");
  const int64_t cut = std::max<int64_t>(0, length - recent_window) / 16 * 16, count = length - cut;
  Tensor q = query.stride(3) == 1 ? query : query.contiguous();
  if (q.scalar_type() != rk.scalar_type()) q = q.to(rk.scalar_type());
  Tensor out;
  if (cut == 0) {
    // everything is still inside the window: exact attention over the ring alone
    out = c.empty({z, h, 1, d}, at::kFloat);
    Tensor lse = c.empty({z, h}, at::kFloat);
    c.done(nvfp4_window_attention(q.data_ptr(), dtype_code(q.scalar_type()), q.stride(0), q.stride(1), rk.data_ptr(),
                                  rv.data_ptr(), z, hk, (int)g, (int)d, cap, cut, count, (float)scaling,
                                  out.data_ptr<float>(), lse.data_ptr<float>(), c.stream),
           "nvfp4_window_attention");
  } else {
    // The window is cut into a few key ranges per (batch, kv head), pieces of at most 144 keys; each
    // block writes an un-normalised split-K partial behind the FP4 decode's own, and the decode's
    // combine merges prefix and window in one pass.
    const int pieces = (int)std::max<int64_t>(1, std::min<int64_t>(64, (count + 143) / 144));
    const Window w{&rk, &rv, cap, cut, count, pieces};
    const DecodeArgs a{z, h, hk, d, &knv, &ksc, &vnv, &vsc, cut, scaling, g};
    out = std::get<0>(decode_core(c, q, a, false, std::nullopt, &w));
  }
  return out.scalar_type() == query.scalar_type() ? out : out.to(query.scalar_type());
}

// Views of the first `cut` tokens of a cache, the V^T axis up to `s_pad` keys.
std::tuple<Tensor, Tensor, Tensor, Tensor> packed_views(const Tensor& knv, const Tensor& ksc, const Tensor& vnv,
                                                        const Tensor& vsc, int64_t cut, int64_t s_pad) {
  // Plain strided views of buffers that never take part in autograd, made without a trip through the
  // dispatcher (four narrow() calls cost a decode step as much as a kernel launch).
  auto prefix = [](const Tensor& t, int64_t axis, int64_t n) {
    require(t.dim() == 3 && n >= 0 && n <= t.size(axis), "view exceeds the cache");
    Tensor v = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(t.storage()), t.key_set(), t.dtype());
    int64_t sizes[3] = {t.size(0), t.size(1), t.size(2)};
    sizes[axis] = n;
    v.unsafeGetTensorImpl()->set_sizes_and_strides(at::IntArrayRef(sizes, 3), t.strides(), t.storage_offset());
    return v;
  };
  return {prefix(knv, 1, cut), prefix(ksc, 1, cut), prefix(vnv, 2, s_pad / 2), prefix(vsc, 2, s_pad / 16)};
}

void append_token(const Tensor& key_new, const Tensor& value_new, const Tensor& knv, const Tensor& ksc, const Tensor& vnv,
                  const Tensor& vsc, const Tensor& v_partial, const OptTensor& rk, const OptTensor& rv, int64_t pos) {
  require_cuda(key_new, "key_new");
  Call c(knv);
  c.same(key_new);
  c.same(value_new);
  const int64_t zhk = knv.size(0), d = knv.size(2) * 2;
  const auto t = v_partial.scalar_type();
  require(key_new.numel() == zhk * d && value_new.numel() == zhk * d, "one token per (batch, kv head) unit");
  // one row per (batch, kv head) unit: [Z, Hk, 1, D] or [Z*Hk, D] is read in place; any other shape of as many
  // elements ([Z, 1, Hk, D], say) is brought to rows first
  auto rows = [&](const Tensor& x, int64_t& stride) -> Tensor {
    if (x.scalar_type() == t && x.stride(-1) == 1 && x.size(-1) == d) {
      if (x.dim() == 2) { stride = x.stride(0); return x; }
      if (x.dim() == 4 && x.size(2) == 1 && (x.size(0) == 1 || x.size(1) == 1 || x.stride(0) == x.size(1) * x.stride(1))) {
        stride = x.size(1) == 1 ? x.stride(0) : x.stride(1);
        return x;
      }
    }
    stride = d;
    return x.reshape({zhk, d}).to(t).contiguous();
  };
  int64_t sk = 0, sv = 0;
  Tensor kn = rows(key_new, sk), vn = rows(value_new, sv);
  if (sk != sv) {
    kn = kn.reshape({zhk, d}).contiguous();
    vn = vn.reshape({zhk, d}).contiguous();
    sk = d;
  }
  c.done(nvfp4_kv_append(kn.data_ptr(), vn.data_ptr(), dtype_code(t), sk, zhk, (int)d, pos, u8(knv), knv.stride(0), u8(ksc),
                         ksc.stride(0), u8(vnv), vnv.stride(0), vnv.stride(1), u8(vsc), vsc.stride(0), vsc.stride(1),
                         v_partial.data_ptr(), opt_ptr<>(rk), opt_ptr<>(rv), rk.has_value() ? rk->size(2) : 0, c.stream),
         "nvfp4_kv_append");
}

// A prompt into the cache buffers in one launch; false when the operands need the general path (another
// dtype than the cache's, or rows that are not contiguous along D).
bool kv_prefill(const Tensor& key, const Tensor& value, const Tensor& knv, const Tensor& ksc, const Tensor& vnv,
                const Tensor& vsc, const Tensor& v_partial, const OptTensor& rk, const OptTensor& rv) {
  require_cuda(key, "key");
  require(key.dim() == 4, "key must be [Z, Hk, S, D]");
  Call c(knv);
  c.same(key);
  c.same(value);
  const auto t = v_partial.scalar_type();
  if (key.scalar_type() != t || value.scalar_type() != t) return false;
  const Rows k = rows_of(key), v = rows_of(as_rows(value, key.size(0) * key.size(1), key.size(2), key.size(3)));
  if (k.sk != 1 || v.sk != 1) return false;
  require(k.b == knv.size(0) && k.k == knv.size(2) * 2, "key must be [Z, Hk, S, D] of the cache");
  require(k.r <= knv.size(1), "prefill exceeds capacity");
  c.done(nvfp4_kv_prefill(k.p, v.p, dtype_code(t), k.b, k.r, (int)k.k, k.sb, k.sr, v.sb, v.sr, u8(knv), knv.stride(0), u8(ksc),
                          ksc.stride(0), u8(vnv), vnv.stride(0), vnv.stride(1), u8(vsc), vsc.stride(0), vsc.stride(1),
                          v_partial.data_ptr(), opt_ptr<>(rk), opt_ptr<>(rv), rk.has_value() ? rk->size(2) : 0, c.stream),
         "nvfp4_kv_prefill");
  return true;
}

// ---------------------------------------------------------------- backward
struct Prep {
  OptTensor copy, delta, amax;
};
Prep bwd_prep_call(const Call& c, const Tensor& x_in, const OptTensor& y_in, bool want_copy, bool want_amax) {
  const Tensor x = x_in.stride(3) == 1 ? x_in : x_in.contiguous();
  const int64_t b1 = x.size(0), b2 = x.size(1), s = x.size(2), d = x.size(3);
  Prep p;
  if (want_copy) p.copy = c.empty({b1 * b2, s, d}, at::kBFloat16);
  if (y_in.has_value()) p.delta = c.empty({b1 * b2, s}, at::kFloat);
  if (want_amax) p.amax = at::zeros({1}, at::TensorOptions().dtype(at::kFloat).device(c.dev));
  Tensor y;
  if (y_in.has_value()) {
    c.same(*y_in);
    y = y_in->scalar_type() == x.scalar_type() ? *y_in : y_in->to(x.scalar_type());
    if (y.stride(3) != 1) y = y.contiguous();
  }
  const bool has_y = y.defined();
  c.done(nvfp4_bwd_prep(x.data_ptr(), dtype_code(x.scalar_type()), x.stride(0), x.stride(1), x.stride(2), b1, b2,
                        has_y ? y.data_ptr() : nullptr, has_y ? y.stride(0) : 0, has_y ? y.stride(1) : 0,
                        has_y ? y.stride(2) : 0, s, (int)d, opt_ptr<>(p.copy), opt_ptr<float>(p.delta), opt_ptr<float>(p.amax),
                        c.stream),
         "nvfp4_bwd_prep");
  return p;
}

std::tuple<OptTensor, OptTensor, OptTensor> bwd_prep(const Tensor& x, const OptTensor& y, bool want_copy, bool want_amax) {
  require_cuda(x, "x");
  Call c(x);
  Prep p = bwd_prep_call(c, x, y, want_copy, want_amax);
  return {p.copy, p.delta, p.amax};
}

// [B1, B2, S, D] as contiguous bf16 rows; no copy when it already is that
Tensor bf16_rows_call(const Call& c, const Tensor& x) {
  if (x.scalar_type() == at::kBFloat16 && x.is_contiguous()) return x;
  return *bwd_prep_call(c, x, std::nullopt, true, false).copy;
}
// The same for Q, K and V: those that need a copy in one launch where their rows allow it.
std::array<Tensor, 3> bf16_rows3(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v) {
  const Tensor* in[3] = {&q, &k, &v};
  std::array<Tensor, 3> r;
  const void* x[3];
  void* out[3];
  int64_t strides[9], extents[9];
  int n = 0;
  bool one = true;
  for (int i = 0; i < 3; ++i) {
    const Tensor& t = *in[i];
    if (t.scalar_type() == at::kBFloat16 && t.is_contiguous()) { r[i] = t; continue; }
    one = one && t.stride(3) == 1 && t.element_size() == 2 && t.scalar_type() == q.scalar_type() &&
          ((reinterpret_cast<uintptr_t>(t.data_ptr()) | (uint64_t)(t.stride(0) * 2) | (uint64_t)(t.stride(1) * 2) |
            (uint64_t)(t.stride(2) * 2)) & 31) == 0 && t.numel() > 0 && t.size(0) * t.size(1) * t.size(2) < (1LL << 31);
    x[n] = t.data_ptr();
    for (int e = 0; e < 3; ++e) { strides[3 * n + e] = t.stride(e); extents[3 * n + e] = t.size(e); }
    ++n;
  }
  if (n < 2 || !one) return {bf16_rows_call(c, q), bf16_rows_call(c, k), bf16_rows_call(c, v)};
  n = 0;
  for (int i = 0; i < 3; ++i)
    if (!r[i].defined()) {
      r[i] = c.empty(in[i]->sizes(), at::kBFloat16);
      out[n++] = r[i].data_ptr();
    }
  c.done(nvfp4_bf16_copies(n, x, out, dtype_code(q.scalar_type()), strides, extents, (int)q.size(3), c.stream),
         "nvfp4_bf16_copies");
  return r;
}
Tensor bf16_rows(const Tensor& x) {
  require_cuda(x, "x");
  Call c(x);
  return bf16_rows_call(c, x).reshape({x.size(0) * x.size(1), x.size(2), x.size(3)});
}

// packs handed in by the caller may be strided views: the kernels' tensor maps assume dense rows
Pack given_or_quant(const Call& c, const OptTensor& nv, const OptTensor& sc, const Rows& x, at::ScalarType t, const char* msg) {
  if (!nv.has_value()) return quant_rows(c, x, t, false, std::nullopt);
  check_packs(*nv, sc.value(), x.b, x.r, x.k, msg);
  Pack p{nv->contiguous(), sc->contiguous()};
  c.same(p.nib);
  c.same(p.sc);
  return p;
}
// The kernels take Z, H, Sq, D from q and Hk, Skv from k; every other operand has to have as many rows.
void check_bwd_operands(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse,
                        const Tensor& dout) {
  auto rows = [](const Tensor& t, int64_t b, int64_t s, int64_t d) {
    return (t.dim() == 4 ? t.size(0) * t.size(1) == b : t.dim() == 3 && t.size(0) == b) && t.size(-2) == s && t.size(-1) == d;
  };
  const int64_t b = q.size(0) * q.size(1), bk = q.size(0) * k.size(1), s = q.size(2), d = q.size(3);
  if (!rows(q, b, s, d) || !rows(k, bk, k.size(2), d) || !rows(v, bk, k.size(2), d) || !rows(out, b, s, d) ||
      !rows(dout, b, s, d) || lse.numel() != b * s)
    throw std::runtime_error("backward operands: shape mismatch between q, k, v, out, lse and the gradient of out");
}
constexpr const char* kQPacks = "q_packs layout mismatch: expected along-D packs of the query rows";
constexpr const char* kKPacks = "k_packs layout mismatch: expected along-D packs of the key rows";

std::tuple<Tensor, Tensor, Tensor> bwd_hp(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out_in,
                                          const Tensor& lse_in, const Tensor& dout_in, double scaling, bool causal,
                                          const OptTensor& seq_start, const OptTensor& seq_end, bool zshd,
                                          const OptTensor& qnv_in, const OptTensor& qsc_in, const OptTensor& knv_in,
                                          const OptTensor& ksc_in, const OptTensor& bias_in) {
  require_cuda(q, "q");
  Call c(q);
  for (const Tensor* t : {&k, &v, &out_in, &lse_in, &dout_in}) c.same(*t);
  const int64_t z = q.size(0), h = q.size(1), s_q = q.size(2), d = q.size(3), hk = k.size(1), s_kv = k.size(2);
  require(d == 128 || d == 256, "D must be 128 or 256");
  const Tensor out = zshd ? out_in.transpose(1, 2) : out_in, dout = zshd ? dout_in.transpose(1, 2) : dout_in;
  check_bwd_operands(q, k, v, out, lse_in, dout);
  const auto gdt = dout.scalar_type();
  const bool need_copy = !(gdt == at::kBFloat16 && dout.is_contiguous());
  Prep pp = bwd_prep_call(c, dout, out, need_copy, false);
  const Tensor doc = need_copy ? *pp.copy : dout;
  const auto [qc, kc, vc] = bf16_rows3(c, q, k, v);
  Pack qp = given_or_quant(c, qnv_in, qsc_in, rows_of(q), q.scalar_type(), kQPacks);
  Pack kp = given_or_quant(c, knv_in, ksc_in, rows_of(k), k.scalar_type(), kKPacks);
  Tensor dq = c.empty({z, h, s_q, d}, gdt), dk = c.empty({z, hk, s_kv, d}, gdt), dv = c.empty({z, hk, s_kv, d}, gdt);
  const Tensor lse = lse_in.contiguous();
  const OptTensor bias = checked_bias(c, bias_in, z, s_kv);
  c.same(seq_start);
  c.same(seq_end);
  c.done(nvfp4_bwd_hp(u8(qp.nib), u8(qp.sc), u8(kp.nib), u8(kp.sc), qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), doc.data_ptr(),
                      lse.data_ptr<float>(), pp.delta->data_ptr<float>(), opt_ptr<float>(bias), opt_ptr<int32_t>(seq_start),
                      opt_ptr<int32_t>(seq_end), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dtype_code(gdt), z, h, hk, s_q,
                      s_kv, (int)d, (float)scaling, causal ? 1 : 0, c.status, c.stream),
         "nvfp4_bwd_hp");
  return {dq, dk, dv};
}

std::tuple<Tensor, Tensor, Tensor> bwd_fp4(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out_in,
                                           const Tensor& lse_in, const Tensor& dout_in, double scaling, bool causal,
                                           const OptTensor& seq_start, const OptTensor& seq_end, bool zshd, bool fp8,
                                           const OptTensor& qnv_in, const OptTensor& qsc_in, const OptTensor& knv_in,
                                           const OptTensor& ksc_in, const OptTensor& qtnv_in, const OptTensor& qtsc_in,
                                           const OptTensor& ktnv_in, const OptTensor& ktsc_in, const OptTensor& vdnv_in,
                                           const OptTensor& vdsc_in, const OptTensor& bias_in, bool sr, bool sr_p_dv,
                                           bool sr_dot_dv, bool sr_ds_dq, int64_t seed) {
  require_cuda(q, "q");
  Call c(q);
  for (const Tensor* t : {&k, &v, &out_in, &lse_in, &dout_in}) c.same(*t);
  const int64_t z = q.size(0), h = q.size(1), s_q = q.size(2), d = q.size(3), hk = k.size(1), s_kv = k.size(2);
  require(d == 128 || d == 256, "D must be 128 or 256");
  const Tensor out = zshd ? out_in.transpose(1, 2) : out_in, dout = zshd ? dout_in.transpose(1, 2) : dout_in;
  check_bwd_operands(q, k, v, out, lse_in, dout);
  const auto gdt = dout.scalar_type();
  Prep pp = bwd_prep_call(c, dout, out, false, true);          // strided reads: no copy for the pre-pass
  const float* amax = pp.amax->data_ptr<float>();
  const Rows dor = unit_rows(dout);
  const int64_t sq_pad = next_mult(s_q, kKeyTile), skv_pad = next_mult(s_kv, kKeyTile);
  Dual dd = quant_dual_rows(c, dor, gdt, sq_pad, amax, (sr ? 1 : 0) | (sr_dot_dv ? 2 : 0), (uint32_t)(seed & 0xFFFFFFFF));
  const Rows qr = unit_rows(q), kr = unit_rows(k), vr = rows_of(v);
  Pack qp, kp;
  Tensor dot_n = dd.tn, dot_s = dd.ts, qt_n, qt_s, kt_n, kt_s;
  auto mx8 = [&](const Rows& x, at::ScalarType t, int64_t sp, const float* am, Tensor& n, Tensor& s) {
    n = c.empty({x.b, x.k, sp}, at::kByte);
    s = c.empty({x.b, x.k, sp / 32}, at::kByte);
    c.done(nvfp4_pack_mx8_t(x.p, dtype_code(t), x.b, x.r, (int)x.k, sp, x.sb, x.sr, am, u8(n), u8(s), c.stream),
           "nvfp4_pack_mx8_t");
  };
  if (fp8) {
    require(!qtnv_in.has_value() && !ktnv_in.has_value(),
            "fp8_rownorm repacks Q^T/K^T as MXFP8; incompatible with saved FP4 transposed packs");
    mx8(dor, gdt, sq_pad, amax, dot_n, dot_s);
    qp = given_or_quant(c, qnv_in, qsc_in, qr, q.scalar_type(), kQPacks);
    kp = given_or_quant(c, knv_in, ksc_in, kr, k.scalar_type(), kKPacks);
    mx8(qr, q.scalar_type(), sq_pad, nullptr, qt_n, qt_s);
    mx8(kr, k.scalar_type(), skv_pad, nullptr, kt_n, kt_s);
  } else {
    // both layouts of an operand from one read, or only the transposed one when the caller has the other
    auto both = [&](const OptTensor& nv, const OptTensor& sc, const OptTensor& tn, const OptTensor& ts, const Rows& x,
                    at::ScalarType t, int64_t sp, const char* msg, Pack& p, Tensor& on, Tensor& os) {
      if (!nv.has_value()) {
        Dual o = quant_dual_rows(c, x, t, sp, nullptr, 0, 0);
        p = {o.dn, o.ds};
        on = o.tn;
        os = o.ts;
        return;
      }
      p = given_or_quant(c, nv, sc, x, t, msg);
      if (tn.has_value()) {
        on = *tn;
        os = ts.value();
      } else {
        Pack e = quant_rows(c, x, t, true, sp);
        on = e.nib;
        os = e.sc;
      }
    };
    both(qnv_in, qsc_in, qtnv_in, qtsc_in, qr, q.scalar_type(), sq_pad, kQPacks, qp, qt_n, qt_s);
    both(knv_in, ksc_in, ktnv_in, ktsc_in, kr, k.scalar_type(), skv_pad, kKPacks, kp, kt_n, kt_s);
  }
  const int64_t tb = fp8 ? 1 : 2;            // elements per byte of a transposed pack
  require(qt_n.dim() == 3 && qt_n.size(0) == z * h && qt_n.size(1) == d && qt_n.size(2) == sq_pad / tb && kt_n.dim() == 3 &&
              kt_n.size(0) == z * hk && kt_n.size(1) == d && kt_n.size(2) == skv_pad / tb,
          "transposed pack layout");
  Pack vd = vdnv_in.has_value() ? Pack{*vdnv_in, vdsc_in.value()} : quant_rows(c, vr, v.scalar_type(), false, std::nullopt);
  Tensor dq = c.empty({z, h, s_q, d}, gdt), dk = c.empty({z, hk, s_kv, d}, gdt), dv = c.empty({z, hk, s_kv, d}, gdt);
  const Tensor lse = lse_in.contiguous();
  const OptTensor bias = checked_bias(c, bias_in, z, s_kv);
  c.same(seq_start);
  c.same(seq_end);
  const int flags = (causal ? 1 : 0) | (sr ? NVFP4_BWD_SR_DS_DK : 0) | (sr_p_dv ? NVFP4_BWD_SR_P_DV : 0) |
                    (sr_ds_dq ? NVFP4_BWD_SR_DS_DQ : 0) | (fp8 ? NVFP4_BWD_MXFP8 : 0);
  c.done(nvfp4_bwd_fp4(u8(qp.nib), u8(qp.sc), u8(kp.nib), u8(kp.sc), u8(vd.nib), u8(vd.sc), u8(dd.dn), u8(dd.ds), u8(dot_n),
                       u8(dot_s), u8(qt_n), u8(qt_s), u8(kt_n), u8(kt_s), lse.data_ptr<float>(), pp.delta->data_ptr<float>(),
                       amax, opt_ptr<float>(bias), opt_ptr<int32_t>(seq_start), opt_ptr<int32_t>(seq_end), dq.data_ptr(),
                       dk.data_ptr(), dv.data_ptr(), dtype_code(gdt), z, h, hk, s_q, s_kv, sq_pad, skv_pad, (int)d,
                       (float)scaling, flags, (uint32_t)((uint64_t)seed * 2654435761ull + 1ull), c.status, c.stream),
         "nvfp4_bwd_fp4");
  return {dq, dk, dv};
}

// ---------------------------------------------------------------- autograd
// The differentiable attention as a graph node of its own: a Python autograd.Function with the
// operator's 26 arguments costs ~55 us per forward and backward before any kernel is launched, more than
// the kernels of a short training step.  The node keeps the operands.  Backward with bf16 gradient products
// calls bwd_hp above without entering the interpreter; the block-scaled modes go through flash._attention_backward
// (stochastic-rounding defaults and seed).  The node's name states the mode.
PyObject* g_backward = nullptr;        // set once; never released

void set_backward(py::object fn) { g_backward = fn.release().ptr(); }

struct AttentionBackward : torch::autograd::Node {
  torch::autograd::SavedVariable q, k, v, out, lse, qnv, qsc, knv, ksc, bias, seq_id, seq_start, seq_end;
  double scaling = 0.0;
  bool causal = false, zshd = false, sr = false;
  int64_t g = 1;
  std::string mode;
  std::optional<bool> sr_p_dv, sr_dot_dv, sr_ds_dq;

  std::string name() const override { return "NVFP4AttentionBackward[" + mode + "]"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto* x : {&q, &k, &v, &out, &lse, &qnv, &qsc, &knv, &ksc, &bias, &seq_id, &seq_start, &seq_end}) x->reset_data();
  }
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    if (!grads[0].defined()) return torch::autograd::variable_list(3);
    Tensor qt, kt, vt, ot, lt;
    OptTensor o[8];
    {   // not held while waiting for the interpreter's lock
      std::lock_guard<std::mutex> lock(mutex_);
      qt = q.unpack(), kt = k.unpack(), vt = v.unpack(), ot = out.unpack(shared_from_this()), lt = lse.unpack();
      const torch::autograd::SavedVariable* saved[8] = {&seq_id, &seq_start, &seq_end, &qnv, &qsc, &knv, &ksc, &bias};
      for (int i = 0; i < 8; ++i)
        if (Tensor t = saved[i]->unpack(); t.defined()) o[i] = t;
    }
    if (mode == "bf16") {
      auto [dq, dk, dv] = bwd_hp(qt, kt, vt, ot, lt, grads[0], scaling, causal, o[1], o[2], zshd, o[3], o[4], o[5], o[6], o[7]);
      return {dq, dk, dv};
    }
    py::gil_scoped_acquire gil;
    py::object r = py::reinterpret_borrow<py::object>(g_backward)(
        qt, kt, vt, ot, lt, grads[0], scaling, causal, g, o[0], o[1], o[2], zshd, mode, o[3], o[4], o[5], o[6], o[7], sr,
        sr_p_dv, sr_dot_dv, sr_ds_dq);
    auto t = r.cast<std::tuple<Tensor, Tensor, Tensor>>();
    return {std::get<0>(t), std::get<1>(t), std::get<2>(t)};
  }
};

Tensor attention(const Tensor& query, const Tensor& key, const Tensor& value, double scaling, bool causal, int64_t g,
                 const OptTensor& bias, const OptTensor& seq_id, const OptTensor& seq_start, const OptTensor& seq_end, bool zshd,
                 const OptTensor& qnv, const OptTensor& qsc, const OptTensor& knv, const OptTensor& ksc, const std::string& mode,
                 bool sr, std::optional<bool> sr_p_dv, std::optional<bool> sr_dot_dv, std::optional<bool> sr_ds_dq) {
  // A node made here has no rule for tangents, and the kernels would drop them without a word.
  auto dual = [](const Tensor& t) { return t._fw_grad(0).defined(); };
  if (dual(query) || dual(key) || dual(value) || (bias.has_value() && dual(*bias)))
    throw NotImplemented("nvfp4_flash_attn_func does not implement forward-mode AD (no jvp)");
  // A bias that requires a gradient gets none, but it makes the output part of the graph.
  const bool record = c10::GradMode::is_enabled() && (query.requires_grad() || key.requires_grad() || value.requires_grad() ||
                                                      (bias.has_value() && bias->requires_grad()));
  c10::AutoGradMode no_grad(false);
  auto [out, lse, packs] = flash_attention(query, key, value, scaling, causal, g, bias, false, seq_id, seq_start, zshd, true,
                                           record, qnv, qsc, knv, ksc);
  if (!record) return out;
  std::shared_ptr<AttentionBackward> node(new AttentionBackward(), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(query, key, value));
  using torch::autograd::SavedVariable;
  auto keep = [](const OptTensor& t) { return SavedVariable(t.has_value() ? *t : Tensor(), false); };
  node->q = SavedVariable(query, false);
  node->k = SavedVariable(key, false);
  node->v = SavedVariable(value, false);
  node->lse = SavedVariable(*lse, false);
  node->qnv = SavedVariable(packs[0], false);
  node->qsc = SavedVariable(packs[1], false);
  node->knv = SavedVariable(packs[2], false);
  node->ksc = SavedVariable(packs[3], false);
  node->bias = keep(bias);
  node->seq_id = keep(seq_id);
  node->seq_start = keep(seq_start);
  node->seq_end = keep(seq_end);
  node->scaling = scaling; node->causal = causal; node->zshd = zshd; node->g = g; node->mode = mode;
  node->sr = sr; node->sr_p_dv = sr_p_dv; node->sr_dot_dv = sr_dot_dv; node->sr_ds_dq = sr_ds_dq;
  torch::autograd::set_history(out, node);
  node->out = SavedVariable(out, true);
  return out;
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  m.doc() = "native host path of the NVFP4 operators";
  py::register_exception_translator([](std::exception_ptr e) {
    try {
      if (e) std::rethrow_exception(e);
    } catch (const AssertionFailure& x) {
      PyErr_SetString(PyExc_AssertionError, x.what());
    } catch (const UnsupportedType& x) {
      PyErr_SetString(PyExc_TypeError, x.what());
    } catch (const NotImplemented& x) {
      PyErr_SetString(PyExc_NotImplementedError, x.what());
    }
  });
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("status_word", &status_word, nogil());
  m.def("pack_into", &pack_into, nogil());
  m.def("quant", &quant, nogil());
  m.def("rope_quant", &rope_quant, nogil());
  m.def("quant_mxfp8_t", &quant_mxfp8_t, nogil());
  m.def("vproj_quant", &vproj_quant, nogil());
  m.def("quant_dual", &quant_dual, nogil());
  m.def("quant_qkv", &quant_qkv, nogil());
  m.def("flash_packed", &flash_packed, nogil());
  m.def("flash_attention", &flash_attention, nogil());
  m.def("decode", &decode, nogil());
  m.def("hybrid_decode", &hybrid_decode, nogil());
  m.def("packed_views", &packed_views, nogil());
  m.def("append_token", &append_token, nogil());
  m.def("kv_prefill", &kv_prefill, nogil());
  m.def("bwd_prep", &bwd_prep, nogil());
  m.def("bf16_rows", &bf16_rows, nogil());
  m.def("bwd_hp", &bwd_hp, nogil());
  m.def("bwd_fp4", &bwd_fp4, nogil());
  m.def("set_backward", &set_backward);
  m.def("attention", &attention, nogil());
}
