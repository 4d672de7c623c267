// Native form of the per-call host work of the operators in ops.py: argument checks, output allocation and the C-ABI
// calls, without a Python view, attribute access or ctypes conversion per buffer.  A decode step issues one prepare and
// one GEMM per linear, a few microseconds of GPU work each; as Python this host work took 30 to 40 us per linear, several
// times the kernels it launched (see ops.py for the operators and their meaning; the checks and messages are those).
//
// Tensors are borrowed; outputs come from the torch caching allocator on the current stream of the input's device.
#include <torch/csrc/utils/pybind.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContextLight.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cstdint>
#include <optional>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/sharq_b200.h"

namespace py = pybind11;

namespace {

using at::Tensor;

[[noreturn]] void fail(const std::string &msg) { throw std::runtime_error(msg); }

inline void need(bool ok, const char *msg) {
  if (!ok) fail(msg);
}

// A non-zero status of an entry point; becomes sharq_b200._lib.SharqError.
struct LibraryError : std::runtime_error {
  using std::runtime_error::runtime_error;
};

inline void check(int status) {
  if (status != 0) throw LibraryError(sharq_last_error());
}

inline void *ptr(const Tensor &t) { return t.data_ptr(); }
inline void *stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

inline Tensor empty_like_on(const Tensor &ref, at::IntArrayRef sizes, at::ScalarType type) {
  return at::empty(sizes, ref.options().dtype(type).layout(at::kStrided).requires_grad(false));
}

inline bool is_plain(const Tensor &t, at::ScalarType type) { return t.is_cuda() && t.scalar_type() == type && t.is_contiguous(); }

inline int64_t round256(int64_t n) { return (n + 255) & ~int64_t(255); }
inline int64_t sf_bytes(int64_t rows, int64_t k) { return (rows / 128 + 1) * 128 * k / 16; }

void check_x(const Tensor &x) {
  need(x.is_cuda(), "X must be a CUDA tensor");
  need(x.is_contiguous(), "X must be contiguous");
  need(x.scalar_type() == at::kBFloat16, "X must be torch.bfloat16");
  need(x.dim() == 2, "X must be shaped [M, K]");
}

void check_k128(const char *op, const char *verb, int64_t k) {
  if (k % 128 != 0) fail(std::string(op) + " " + verb + " K to be a multiple of 128, got " + std::to_string(k));
}

// The five prepare outputs and `extra` trailing bytes in one allocation, at 256-byte aligned offsets.
struct Prepared {
  Tensor buf;
  int64_t m, k, sa, se, ssf, sq, o_e, o_sfa, o_q, o_sf, o_tail;
  uint8_t *base;

  Prepared(const Tensor &ref, int64_t m_, int64_t k_, int64_t extra) : m(m_), k(k_) {
    const int64_t k256 = (k + 255) / 256 * 256;
    sa = m * k256 / 4;
    se = ((m + 127) / 128 * 128) * k256 / 16;
    ssf = sf_bytes(m, k);
    sq = m * (k / 2);
    o_e = round256(sa);
    o_sfa = o_e + round256(se);
    o_q = o_sfa + round256(ssf);
    o_sf = o_q + round256(sq);
    o_tail = o_sf + round256(ssf);
    buf = empty_like_on(ref, {o_tail + extra}, at::kByte);
    base = static_cast<uint8_t *>(buf.data_ptr());
  }
  uint8_t *a_comp() const { return base; }
  uint8_t *e() const { return base + o_e; }
  uint8_t *sfa() const { return base + o_sfa; }
  uint8_t *q_res() const { return base + o_q; }
  uint8_t *sf_res() const { return base + o_sf; }
  uint8_t *tail() const { return base + o_tail; }
  // A contiguous tensor in the allocation, `offset` bytes into it, made without the dispatcher: with as_strided and view the six to eight
  // outputs of a prepare were 5 of its 12 us on the host.
  Tensor part(int64_t offset, at::IntArrayRef sizes, at::ScalarType type) const {
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf.storage()), buf.key_set(), c10::scalarTypeToTypeMeta(type));
    c10::TensorImpl *impl = t.unsafeGetTensorImpl();
    impl->set_storage_offset(offset / (int64_t)c10::elementSize(type));
    impl->set_sizes_contiguous(sizes);
    return t;
  }
  Tensor view(int64_t offset, int64_t n) const { return part(offset, {n}, at::kByte); }
  // a 0-dim float32 view at `offset` bytes behind the tail
  Tensor scalar(int64_t offset) const { return part(o_tail + offset, {}, at::kFloat); }
  std::vector<Tensor> outputs() const {
    return {view(0, sa), view(o_e, se), view(o_sfa, ssf), part(o_q, {m, k / 2}, at::kByte), view(o_sf, ssf)};
  }
};

// Scaled (RMSNorm-fused when gamma is given) prepare; workspace and scale live in the tail of the outputs.
struct Scaled {
  Prepared p;
  int64_t ws_bytes, scale_at;
  Tensor total;

  Scaled(const Tensor &x, const std::optional<Tensor> &gamma, double eps, int64_t n, const std::optional<Tensor> &residual)
      : p(x, x.size(0), x.size(1), round256((int64_t)sharq_prepare_workspace_best_bytes((int)x.size(0))) + 256) {
    ws_bytes = (int64_t)sharq_prepare_workspace_best_bytes((int)p.m);
    scale_at = round256(ws_bytes);
    const int m = (int)p.m, k = (int)p.k;
    c10::cuda::OptionalCUDAGuard guard(x.device());
    float *scale = reinterpret_cast<float *>(p.tail() + scale_at);
    if (residual) {
      total = at::empty_like(x);
      check(sharq_fused_add_rmsnorm_sparse_residual_quantize_x(ptr(x), ptr(*residual), ptr(total), ptr(*gamma), (float)eps, m,
                                                               (int)n, k, p.tail(), (size_t)ws_bytes, p.a_comp(), p.e(), p.sfa(),
                                                               p.q_res(), p.sf_res(), scale, stream_of(x)));
    } else if (gamma) {
      check(sharq_fused_rmsnorm_sparse_residual_quantize_x(ptr(x), ptr(*gamma), (float)eps, m, (int)n, k, p.tail(),
                                                           (size_t)ws_bytes, p.a_comp(), p.e(), p.sfa(), p.q_res(), p.sf_res(),
                                                           scale, stream_of(x)));
    } else {
      check(sharq_scaled_sparse_residual_quantize_x(ptr(x), m, (int)n, k, p.tail(), (size_t)ws_bytes, p.a_comp(), p.e(),
                                                    p.sfa(), p.q_res(), p.sf_res(), scale, stream_of(x)));
    }
  }
};

std::vector<Tensor> scaled_prepare(const Tensor &x, const std::optional<Tensor> &gamma, double eps, int64_t n,
                         const std::optional<Tensor> &residual, bool return_workspace) {
  check_x(x);
  const int64_t k = x.size(1);
  const char *op = residual ? "fused_add_rmsnorm_sparse_residual_quantize_x"
                            : (gamma ? "fused_rmsnorm_sparse_residual_quantize_x" : "scaled_sparse_residual_quantize_x");
  if (residual)
    need(is_plain(*residual, at::kBFloat16) && residual->sizes() == x.sizes() && residual->device() == x.device(),
         "residual must be a contiguous CUDA bfloat16 tensor shaped like X on the same device");
  if (gamma) {
    const Tensor &w = *gamma;
    if (residual) {
      need(is_plain(w, at::kBFloat16) && w.dim() == 1 && w.size(0) == k && w.device() == x.device(),
           "rmsnorm_weight must be a contiguous CUDA bfloat16 tensor shaped [K] on X's device");
    } else {
      need(w.is_cuda(), "rmsnorm_weight must be a CUDA tensor");
      need(w.is_contiguous(), "rmsnorm_weight must be contiguous");
      need(w.scalar_type() == at::kBFloat16, "rmsnorm_weight must be torch.bfloat16");
      need(w.dim() == 1, "rmsnorm_weight must be shaped [K]");
      need(w.device() == x.device(), "rmsnorm_weight must be on the same device as X");
      if (w.size(0) != k)
        fail("rmsnorm_weight size mismatch: expected " + std::to_string(k) + ", got " + std::to_string(w.size(0)));
    }
  }
  check_k128(op, gamma && !residual ? "currently requires" : "requires", k);
  if (gamma && k / 32 > 1024) fail(std::string(op) + " requires K/32 <= 1024, got " + std::to_string(k / 32));
  Scaled s(x, gamma, eps, n, residual);
  std::vector<Tensor> out = s.p.outputs();
  out.push_back(s.p.scalar(s.scale_at));
  if (residual)
    out.push_back(s.total);
  else if (return_workspace)
    out.push_back(s.p.view(s.p.o_tail, 256 + 4 * s.p.m));
  return out;
}

std::vector<Tensor> swiglu_prepare(const Tensor &gate_up, int64_t n) {
  need(is_plain(gate_up, at::kBFloat16) && gate_up.dim() == 2, "gate_up must be a contiguous CUDA bfloat16 matrix");
  const int64_t m = gate_up.size(0), f2 = gate_up.size(1), k = f2 / 2;
  if (f2 % 2 != 0 || k % 128 != 0)
    fail("swiglu_sparse_residual_quantize_x requires K to be a multiple of 128, got " + std::to_string(k));
  const int64_t h_bytes = m * k * 2;
  constexpr int64_t kWs = 256 + 8192;  // with a word for the maximum of every CTA of the SwiGLU kernel
  Prepared p(gate_up, m, k, kWs + 256 + h_bytes);
  c10::cuda::OptionalCUDAGuard guard(gate_up.device());
  check(sharq_swiglu_sparse_residual_quantize_x(ptr(gate_up), (int)m, (int)n, (int)k, p.tail() + kWs + 256, p.tail(), (size_t)kWs, p.a_comp(),
                                                p.e(), p.sfa(), p.q_res(), p.sf_res(),
                                                reinterpret_cast<float *>(p.tail() + kWs), stream_of(gate_up)));
  std::vector<Tensor> out = p.outputs();
  out.push_back(p.scalar(kWs));
  return out;
}

void check_u8(const Tensor &t, const at::Device &dev, int64_t want, const char *name) {
  if (!(t.is_cuda() && t.device() == dev && t.scalar_type() == at::kByte && t.is_contiguous()))
    fail(std::string(name) + " must be a contiguous CUDA uint8 tensor on the device of Q_res");
  if (t.numel() != want)
    fail(std::string(name) + ".numel() mismatch: expected " + std::to_string(want) + ", got " + std::to_string(t.numel()));
}

const float *scale_ptr(const Tensor &scale, const at::Device &dev, const char *name) {
  const std::string n(name);
  if (!scale.is_cuda()) fail(n + " must be a CUDA tensor");
  if (!scale.is_contiguous()) fail(n + " must be contiguous");
  if (scale.scalar_type() != at::kFloat) fail(n + " must be torch.float32");
  if (scale.numel() != 1) fail(n + " must contain exactly one element");
  if (scale.device() != dev) fail(n + " must be on the same device as the inputs");
  return static_cast<const float *>(scale.data_ptr());
}

Tensor output(const Tensor &ref, int64_t m, int64_t n, const std::optional<Tensor> &out) {
  if (!out) return empty_like_on(ref, {m, n}, at::kBFloat16);
  need(out->is_cuda() && out->device() == ref.device() && out->scalar_type() == at::kBFloat16 && out->is_contiguous() &&
           out->dim() == 2 && out->size(0) == m && out->size(1) == n,
       "out must be a contiguous CUDA bfloat16 tensor shaped [M, N]");
  return *out;
}

void check_bias(const std::optional<Tensor> &bias, int64_t n, const at::Device &dev) {
  if (!bias) return;
  need(is_plain(*bias, at::kBFloat16) && bias->numel() == n, "bias must be a contiguous CUDA bfloat16 tensor with N elements");
  need(bias->device() == dev, "bias must be on the same device as the inputs");
}

void check_weight(const Tensor &qw, const Tensor &sfs, const Tensor &sfd, const at::Device &dev, int64_t n, int64_t k) {
  check_u8(qw, dev, n * (k / 2), "QW");
  check_u8(sfs, dev, sf_bytes(n, k), "SFW_sparse");
  check_u8(sfd, dev, sf_bytes(n, k), "SFW_dense");
}

// flag: the device's error flag; with split_k it also stands for the GEMM's (unwritten) workspace.
Tensor linear_gemm(const Tensor &a_comp, const Tensor &e, const Tensor &sfa, const Tensor &q_res, const Tensor &sf_res,
                   const Tensor &qw, const Tensor &sfs, const Tensor &sfd, const std::optional<Tensor> &alpha_t, double alpha,
                   const std::optional<Tensor> &bias, const std::optional<Tensor> &out, const std::optional<Tensor> &residual,
                   const Tensor &flag, bool split_k) {
  const int64_t m = q_res.size(0), k = q_res.size(1) * 2, n = qw.size(0);
  const at::Device dev = q_res.device();
  const int64_t k256 = (k + 255) / 256 * 256;
  check_u8(a_comp, dev, m * k256 / 4, "A_comp");
  check_u8(e, dev, ((m + 127) / 128 * 128) * k256 / 16, "E");
  check_u8(sfa, dev, sf_bytes(m, k), "SFA_sparse");
  check_u8(q_res, dev, m * (k / 2), "Q_res");
  check_u8(sf_res, dev, sf_bytes(m, k), "SF_res");
  check_weight(qw, sfs, sfd, dev, n, k);
  check_bias(bias, n, dev);
  if (residual)
    need(is_plain(*residual, at::kBFloat16) && residual->device() == dev && residual->numel() == m * n,
         "residual must be a contiguous CUDA bfloat16 tensor with M * N elements on the device of Q_res");
  Tensor d = output(q_res, m, n, out);
  const float *alpha_dev = alpha_t ? scale_ptr(*alpha_t, dev, "alpha") : nullptr;
  c10::cuda::OptionalCUDAGuard guard(dev);
  check(sharq_linear_gemm_residual(ptr(a_comp), ptr(e), ptr(sfa), ptr(q_res), ptr(sf_res), ptr(qw), ptr(sfs), ptr(sfd), (int)m,
                                   (int)n, (int)k, (float)alpha, alpha_dev, bias ? ptr(*bias) : nullptr,
                                   residual ? ptr(*residual) : nullptr, ptr(d), split_k ? ptr(flag) : nullptr, split_k ? 16 : 0,
                                   static_cast<int *>(ptr(flag)), stream_of(q_res)));
  return d;
}

// Prepare and fused GEMM of a whole linear in one call.
Tensor linear_forward(const Tensor &x, const Tensor &qw, const Tensor &sfs, const Tensor &sfd, double weight_scale,
                      const std::optional<Tensor> &bias, const Tensor &flag, bool split_k) {
  check_x(x);
  const int64_t m = x.size(0), k = x.size(1), n = qw.size(0);
  check_k128("scaled_sparse_residual_quantize_x", "requires", k);
  check_weight(qw, sfs, sfd, x.device(), n, k);
  check_bias(bias, n, x.device());
  Scaled s(x, std::nullopt, 0.0, n, std::nullopt);
  Tensor d = empty_like_on(x, {m, n}, at::kBFloat16);
  c10::cuda::OptionalCUDAGuard guard(x.device());
  check(sharq_linear_gemm_ws(s.p.a_comp(), s.p.e(), s.p.sfa(), s.p.q_res(), s.p.sf_res(), ptr(qw), ptr(sfs), ptr(sfd), (int)m,
                             (int)n, (int)k, (float)weight_scale, reinterpret_cast<float *>(s.p.tail() + s.scale_at),
                             bias ? ptr(*bias) : nullptr, ptr(d), split_k ? ptr(flag) : nullptr, split_k ? 16 : 0,
                             static_cast<int *>(ptr(flag)), stream_of(x)));
  return d;
}

Tensor dense_gemm(const Tensor &a, const Tensor &b, const Tensor &sfa, const Tensor &sfb, double alpha,
                  const std::optional<Tensor> &alpha_t, const std::optional<Tensor> &c_in, double beta,
                  const std::optional<Tensor> &bias, const std::optional<Tensor> &out, const Tensor &flag, bool split_k) {
  need(a.is_cuda() && b.is_cuda() && sfa.is_cuda() && sfb.is_cuda(), "A, B, SFA and SFB must be CUDA tensors");
  const int64_t m = a.size(0), n = b.size(0), k = a.size(1) * 2;
  const at::Device dev = a.device();
  check_bias(bias, n, dev);
  Tensor d = output(a, m, n, out);
  const float *alpha_dev = alpha_t ? scale_ptr(*alpha_t, dev, "scale") : nullptr;
  c10::cuda::OptionalCUDAGuard guard(dev);
  check(sharq_matmul_bias_ws(ptr(a), ptr(b), ptr(sfa), ptr(sfb), (int)m, (int)n, (int)k, (float)alpha, alpha_dev,
                             c_in ? ptr(*c_in) : nullptr, (float)beta, bias ? ptr(*bias) : nullptr, ptr(d),
                             split_k ? ptr(flag) : nullptr, split_k ? 16 : 0, static_cast<int *>(ptr(flag)), stream_of(a)));
  return d;
}

Tensor sparse_gemm(const std::string &name, const Tensor &a_comp, const Tensor &b, const Tensor &e, const Tensor &sfa,
                   const Tensor &sfb, int64_t m, int64_t n, int64_t k, double alpha, const std::optional<Tensor> &alpha_t,
                   double beta, const Tensor &flag, bool split_k) {
  need(m > 0 && n > 0 && k > 0, "M, N, K must be positive");
  if (beta != 0.0) fail(name + " currently requires beta == 0");
  const Tensor *ts[5] = {&a_comp, &b, &e, &sfa, &sfb};
  const char *names[5] = {"A_comp", "B", "E", "SFA", "SFB"};
  for (const Tensor *t : ts)
    if (!t->is_cuda()) fail(name + " inputs must be CUDA tensors");
  for (const Tensor *t : ts)
    if (!t->is_contiguous()) fail(name + " inputs must be contiguous");
  for (int i = 0; i < 5; ++i)
    if (ts[i]->scalar_type() != at::kByte) fail(std::string(names[i]) + " must be torch.uint8");
  for (const Tensor *t : ts)
    if (t->device() != a_comp.device()) fail(name + " inputs must be on the same device");
  int64_t want[4];
  check(sharq_get_sparse_nvfp4_buffer_sizes((int)m, (int)n, (int)k, want));
  const Tensor *sized[4] = {&a_comp, &e, &sfa, &sfb};
  const char *sized_names[4] = {"A_comp", "E", "SFA", "SFB"};
  for (int i = 0; i < 4; ++i)
    if (sized[i]->numel() != want[i])
      fail(std::string(sized_names[i]) + ".numel() mismatch: expected " + std::to_string(want[i]) + ", got " +
           std::to_string(sized[i]->numel()));
  need(b.dim() == 2, "B must be a 2D tensor shaped [N, K/2]");
  if (b.size(0) != n) fail("B.size(0) mismatch: expected " + std::to_string(n) + ", got " + std::to_string(b.size(0)));
  if (b.size(1) != k / 2) fail("B.size(1) mismatch: expected " + std::to_string(k / 2) + ", got " + std::to_string(b.size(1)));
  Tensor d = empty_like_on(a_comp, {m, n}, at::kBFloat16);
  const float *alpha_dev = alpha_t ? scale_ptr(*alpha_t, a_comp.device(), "alpha") : nullptr;
  c10::cuda::OptionalCUDAGuard guard(a_comp.device());
  check(sharq_sparse_matmul_ws(ptr(a_comp), ptr(b), ptr(e), ptr(sfa), ptr(sfb), (int)m, (int)n, (int)k, (float)alpha, alpha_dev,
                               (float)beta, ptr(d), split_k ? ptr(flag) : nullptr, split_k ? 16 : 0,
                               static_cast<int *>(ptr(flag)), stream_of(a_comp)));
  return d;
}

// x: a 16-byte aligned contiguous CUDA bf16 matrix (ops._scaled_quantize_input)
std::vector<Tensor> scaled_quantize(const Tensor &x, bool shared) {
  const int64_t rows = x.size(0), k = x.size(1);
  const size_t ws_bytes = sharq_scaled_quantize_workspace_bytes();
  Tensor q = empty_like_on(x, {rows, k / 2}, at::kByte), sf = empty_like_on(x, {sf_bytes(rows, k)}, at::kByte);
  Tensor ws = empty_like_on(x, {(int64_t)ws_bytes}, at::kByte), scale = empty_like_on(x, {}, at::kFloat);
  c10::cuda::OptionalCUDAGuard guard(x.device());
  if (!shared) {
    check(sharq_scaled_quantize_nvfp4(ptr(x), (int)rows, (int)k, ptr(ws), ws_bytes, ptr(q), ptr(sf),
                                      static_cast<float *>(ptr(scale)), stream_of(x)));
    return {q, sf, scale};
  }
  Tensor sf2 = empty_like_on(x, {sf_bytes(rows, k)}, at::kByte);
  check(sharq_scaled_quantize_w32_shared(ptr(x), (int)rows, (int)k, ptr(ws), ws_bytes, ptr(q), ptr(sf), ptr(sf2),
                                         static_cast<float *>(ptr(scale)), stream_of(x)));
  return {q, sf, sf2, scale};
}

// Fused GEMM of a merged gate_up weight with SwiGLU in its epilogue -> (h, bits of max|h|)
std::vector<Tensor> linear_gemm_swiglu(const Tensor &a_comp, const Tensor &e, const Tensor &sfa, const Tensor &q_res,
                                       const Tensor &sf_res, const Tensor &qw, const Tensor &sfs, const Tensor &sfd,
                                       const Tensor &alpha_t, double alpha, const Tensor &flag) {
  const int64_t m = q_res.size(0), k = q_res.size(1) * 2, n = qw.size(0);
  const at::Device dev = q_res.device();
  if (n % 256 != 0) fail("the merged gate_up weight must have a multiple of 256 rows, got " + std::to_string(n));
  const int64_t k256 = (k + 255) / 256 * 256;
  check_u8(a_comp, dev, m * k256 / 4, "A_comp");
  check_u8(e, dev, ((m + 127) / 128 * 128) * k256 / 16, "E");
  check_u8(sfa, dev, sf_bytes(m, k), "SFA_sparse");
  check_u8(q_res, dev, m * (k / 2), "Q_res");
  check_u8(sf_res, dev, sf_bytes(m, k), "SF_res");
  check_weight(qw, sfs, sfd, dev, n, k);
  c10::cuda::OptionalCUDAGuard guard(dev);
  Tensor h = empty_like_on(q_res, {m, n / 2}, at::kBFloat16);
  Tensor amax = empty_like_on(q_res, {sharq_gemm_swiglu_absmax_words((int)m, (int)(n / 2))}, at::kInt);
  check(sharq_linear_gemm_swiglu(ptr(a_comp), ptr(e), ptr(sfa), ptr(q_res), ptr(sf_res), ptr(qw), ptr(sfs), ptr(sfd), (int)m,
                                 (int)(n / 2), (int)k, (float)alpha, scale_ptr(alpha_t, dev, "alpha"), ptr(h), ptr(amax),
                                 static_cast<int *>(ptr(flag)), stream_of(q_res)));
  return {h, amax};
}

std::vector<Tensor> absmax_prepare(const Tensor &x, int64_t n, const Tensor &amax_bits) {
  check_x(x);
  check_k128("absmax_sparse_residual_quantize_x", "requires", x.size(1));
  need(amax_bits.is_cuda() && amax_bits.device() == x.device() && amax_bits.scalar_type() == at::kInt && amax_bits.is_contiguous() &&
           amax_bits.numel() >= 1,
       "amax_bits must be a contiguous CUDA int32 vector on X's device");
  Prepared p(x, x.size(0), x.size(1), 256);
  c10::cuda::OptionalCUDAGuard guard(x.device());
  check(sharq_absmax_sparse_residual_quantize_x(ptr(x), (int)p.m, (int)n, (int)p.k, ptr(amax_bits), (int)amax_bits.numel(), p.a_comp(), p.e(), p.sfa(),
                                                p.q_res(), p.sf_res(), reinterpret_cast<float *>(p.tail()), stream_of(x)));
  std::vector<Tensor> out = p.outputs();
  out.push_back(p.scalar(0));
  return out;
}

void rope_inplace(const Tensor &qkv, int64_t heads, int64_t head_dim, const Tensor &cos, const Tensor &sin, int64_t seq_len) {
  need(qkv.is_cuda() && qkv.scalar_type() == at::kBFloat16 && qkv.dim() == 2 && qkv.stride(1) == 1,
       "qkv must be a CUDA bfloat16 matrix with unit column stride");
  const Tensor *tables[2] = {&cos, &sin};
  for (int i = 0; i < 2; ++i)
    if (!(is_plain(*tables[i], at::kBFloat16) && tables[i]->dim() == 2 && tables[i]->size(0) == seq_len &&
          tables[i]->size(1) == head_dim))
      fail(std::string(i == 0 ? "cos" : "sin") + " must be a contiguous CUDA bfloat16 tensor shaped [seq_len, head_dim]");
  need(heads * head_dim <= qkv.size(1), "heads * head_dim exceeds the row width");
  c10::cuda::OptionalCUDAGuard guard(qkv.device());
  check(sharq_rope_inplace(ptr(qkv), (int)qkv.size(0), (int)qkv.stride(0), (int)seq_len, (int)heads, (int)head_dim, ptr(cos),
                           ptr(sin), stream_of(qkv)));
}

// The GIL is released while a call allocates and launches (a launch waits when the queue of the GPU is full).
template <typename... Args>
auto as_tuple(std::vector<Tensor> (*fn)(Args...)) {
  return [fn](Args... args) {
    std::vector<Tensor> v;
    {
      py::gil_scoped_release nogil;
      v = fn(args...);
    }
    py::tuple t(v.size());
    for (size_t i = 0; i < v.size(); ++i) t[i] = std::move(v[i]);
    return t;
  };
}

}  // namespace

PYBIND11_MODULE(sharq_native, m) {
  static py::object sharq_error = py::module_::import("sharq_b200._lib").attr("SharqError");
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const LibraryError &e) {
      PyErr_SetString(sharq_error.ptr(), e.what());
    }
  });
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("scaled_prepare", as_tuple(&scaled_prepare));
  m.def("swiglu_prepare", as_tuple(&swiglu_prepare));
  m.def("scaled_quantize", as_tuple(&scaled_quantize));
  m.def("linear_gemm_swiglu", as_tuple(&linear_gemm_swiglu));
  m.def("absmax_prepare", as_tuple(&absmax_prepare));
  m.def("rope_inplace", &rope_inplace, nogil());
  m.def("linear_gemm", &linear_gemm, nogil());
  m.def("linear_forward", &linear_forward, nogil());
  m.def("dense_gemm", &dense_gemm, nogil());
  m.def("sparse_gemm", &sparse_gemm, nogil());
}
