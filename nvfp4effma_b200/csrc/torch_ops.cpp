// CUDA kernels of the torch operators that sit on the hot paths (torch.ops.nvfp4effma.*; schemas and Meta kernels are in _ops.py): argument
// checks, layout fix-ups, output allocation and ONE call of the C ABI, in C++.  Through ctypes the same steps took 15-25 us of host time per
// operator (struct building, attribute lookups, 5 us for the current stream alone) -- several times what the decode kernels run.
//
// Exceptions are those of the C ABI's status mapping: TypeError (dtype), ValueError (shape, INVALID_VALUE), NotImplementedError
// (NOT_SUPPORTED), RuntimeError (CUDA).
#include <map>
#include <mutex>
#include <tuple>
#include <vector>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>
#include "../../include/nvfp4effma.h"
#include "../../include/nvfp4effma_b200.h"

namespace {

using at::ScalarType;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

void check(nvfp4a_status st) {
  if (st == NVFP4A_OK) return;
  const char *m = nvfp4a_last_error();
  if (!m || !*m) m = nvfp4a_status_string(st);
  TORCH_CHECK_NOT_IMPLEMENTED(st != NVFP4A_NOT_SUPPORTED, m);
  TORCH_CHECK_VALUE(st != NVFP4A_INVALID_VALUE, m);
  TORCH_CHECK(false, m);
}

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// the element type as Python spells it
const char *dtype_name(ScalarType t) {
  switch (t) {
    case at::kByte: return "uint8";
    case at::kChar: return "int8";
    case at::kShort: return "int16";
    case at::kInt: return "int32";
    case at::kLong: return "int64";
    case at::kHalf: return "float16";
    case at::kBFloat16: return "bfloat16";
    case at::kFloat: return "float32";
    case at::kDouble: return "float64";
    case at::kBool: return "bool";
    default: return c10::toString(t);
  }
}
nvfp4a_dtype dense_code(ScalarType t) {
  if (t == at::kBFloat16) return NVFP4A_BF16;
  if (t == at::kHalf) return NVFP4A_FP16;
  TORCH_CHECK_TYPE(t == at::kFloat, "torch.", dtype_name(t), " is not one of the dense element types (bfloat16, float16, float32)");
  return NVFP4A_FP32;
}
bool is_dense(ScalarType t) { return t == at::kBFloat16 || t == at::kHalf || t == at::kFloat; }

bool misaligned(const Tensor &t, uintptr_t mask) { return ((uintptr_t)t.data_ptr() & mask) != 0; }
// the address of a tensor that a kernel will use: one of host memory would fault on the GPU (pinned memory is mapped there)
void *device_ptr(const Tensor &t, const char *name) {
  TORCH_CHECK_VALUE(t.is_cuda() || t.is_pinned(), name, " lives on ", t.device(), "; the library works on CUDA memory only");
  return t.data_ptr();
}
void *addr(const OptTensor &t, const char *name) { return t ? device_ptr(*t, name) : nullptr; }

// a 2-D matrix the library can address: unit stride along rows, a pitch that is a multiple of `mult` and not below the row length, a
// 16-byte aligned base; anything else is copied once
Tensor matrix(const Tensor &t, int64_t mult, const char *name) {
  TORCH_CHECK_VALUE(t.dim() == 2, name, ": expected a matrix, got ", t.dim(), " dimensions");
  const int64_t pitch = t.stride(0);
  return t.stride(1) != 1 || pitch < t.size(1) || pitch % mult || misaligned(t, 15) ? t.contiguous() : t;
}

nvfp4a_tensor dense_tensor(const Tensor &t, const char *name, const OptTensor &amax = std::nullopt) {
  nvfp4a_tensor r = {};
  r.data = device_ptr(t, name);
  r.dtype = dense_code(t.scalar_type());
  r.amax = (float *)addr(amax, "amax");
  return r;
}

Tensor empty(at::IntArrayRef shape, ScalarType t, const Tensor &like) { return at::empty(shape, like.options().dtype(t)); }
Tensor zeros(at::IntArrayRef shape, ScalarType t, const Tensor &like) { return at::zeros(shape, like.options().dtype(t)); }

// an operand with what keeps its buffers alive until the launch is enqueued
struct Operand {
  nvfp4a_tensor t = {};
  int64_t ld = 0;
  Tensor data, scales;
};

// block-scale rows whose pitch has to be a multiple of 4 entries
Tensor padded_rows(const Tensor &s) {
  Tensor wide = zeros({s.size(0), (s.size(1) + 3) / 4 * 4}, s.scalar_type(), s);
  wide.narrow(1, 0, s.size(1)).copy_(s);
  return wide;
}

Operand fp4_operand(const Tensor &data, const Tensor &scales, const OptTensor &glob, int64_t flags, int64_t smax) {
  Operand o;
  o.data = matrix(data, 32, "NVFP4 data");
  o.scales = scales;
  if (!(flags & NVFP4A_SCALES_SWIZZLED)) {
    if (o.scales.stride(-1) != 1 || o.scales.stride(0) % 4 || misaligned(o.scales, 3)) {
      o.scales = o.scales.contiguous();
      if (o.scales.stride(0) % 4) o.scales = padded_rows(o.scales);
    }
    o.t.ld_scale = (int)o.scales.stride(0);
  }
  o.t.data = device_ptr(o.data, "NVFP4 data");
  o.t.dtype = NVFP4A_NVFP4;
  o.t.block_scale = device_ptr(o.scales, "block scales");
  o.t.global_scale = (const float *)addr(glob, "global");
  o.t.flags = (unsigned)flags;
  o.t.scale_max = (int)smax;
  o.ld = 2 * o.data.stride(0);
  return o;
}

// uint8 = NVFP4, int8 = INT8 + FP32 scales, else dense
Operand activation(const Tensor &x, const OptTensor &scales, const OptTensor &glob, int64_t flags, int64_t smax) {
  if (x.scalar_type() == at::kByte) {
    TORCH_CHECK_VALUE(scales.has_value(), "NVFP4 activations come with block scales");
    return fp4_operand(x, *scales, glob, flags, smax);
  }
  Operand o;
  if (x.scalar_type() == at::kChar) {
    TORCH_CHECK_VALUE(scales.has_value(), "int8 activations come with block scales");
    o.data = matrix(x, 64, "int8 activations");
    o.scales = scales->contiguous();
    if (misaligned(o.scales, 15) || o.scales.stride(0) % 4) o.scales = padded_rows(o.scales);
    o.t.data = device_ptr(o.data, "int8 activations");
    o.t.dtype = NVFP4A_INT8;
    o.t.block_scale = device_ptr(o.scales, "block scales");
    o.t.ld_scale = (int)o.scales.stride(0);
  } else {
    o.data = matrix(x, 64, "activations");
    o.t = dense_tensor(o.data, "x");
  }
  o.ld = o.data.stride(0);
  return o;
}

ScalarType result_dtype(const Tensor &x, std::optional<ScalarType> want) {
  return want ? *want : is_dense(x.scalar_type()) ? x.scalar_type() : at::kBFloat16;
}
void check_out(const Tensor &out, int64_t T, int64_t N) {
  TORCH_CHECK_VALUE(out.dim() == 2 && out.size(0) == T && out.size(1) == N && out.stride(1) == 1, "out must be a [", T, ", ", N,
                    "] matrix with unit stride along its rows, got ", out.sizes(), " / strides ", out.strides());
  dense_code(out.scalar_type());
}
OptTensor amax_buffer(bool want, const Tensor &like) { return want ? OptTensor(zeros({1}, at::kFloat, like)) : std::nullopt; }

struct Bias {
  nvfp4a_tensor t = {};
  Tensor keep;
  const nvfp4a_tensor *p = nullptr;
  Bias(const OptTensor &b, int64_t n) {
    if (!b) return;
    TORCH_CHECK_VALUE(b->numel() == n, "bias has ", b->numel(), " elements for ", n, " output features");
    keep = b->contiguous();
    t = dense_tensor(keep, "bias");
    p = &t;
  }
};
void check_k(int64_t k) { TORCH_CHECK_VALUE(k % 64 == 0, "k = ", k, ": the reduction length must be a multiple of 64"); }

// The scratch of one GEMM call comes from torch's allocator: no second pool beside it, and a captured call leaves no allocation in the graph and
// does what it does outside.  Of the current device (the output may be pinned host memory).  Freed when the call is enqueued, to be used again in the
// order of its stream like any tensor.  An allocator that the thread has set for itself is back afterwards.
struct CallScratch {
  std::vector<Tensor> held;
  void *(*old)(void *, size_t) = nullptr;
  void *old_ctx = nullptr;
  CallScratch() {
    nvfp4a_b200_get_scratch_alloc(&old, &old_ctx);
    nvfp4a_b200_set_scratch_alloc(&alloc, this);
  }
  ~CallScratch() { nvfp4a_b200_set_scratch_alloc(old, old_ctx); }
  CallScratch(const CallScratch &) = delete;
  static void *alloc(void *ctx, size_t bytes) {
    CallScratch *const self = (CallScratch *)ctx;
    try {
      self->held.push_back(at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA)));
      return self->held.back().data_ptr();
    } catch (...) {   // out of memory: the library does without
      return nullptr;
    }
  }
};

// ---- linear -----------------------------------------------------------------------------------------------------------------------
// One nvfp4a_gemm (or nvfp4a_gemv_tc on the weight's image up to 8 tokens) writing `out`; the amax tensor or none.
OptTensor gemm_into(const Tensor &out, const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &w, const Tensor &ws,
                    const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, const OptTensor &bias, double alpha, double beta, bool want_amax,
                    const OptTensor &w_img) {
  check_k(k);
  const int64_t T = x.size(0), N = w.size(0);
  check_out(out, T, N);
  const OptTensor amax = amax_buffer(want_amax, out);
  const Operand b = activation(x, xs, xg, xf, xm);
  const nvfp4a_tensor d = dense_tensor(out, "out", amax);
  const Bias bi(bias, N);
  const int ldd = (int)out.stride(0);
  const nvfp4a_tensor *c = beta != 0.0 ? &d : nullptr;   // beta accumulates into out itself
  const int ldc = beta != 0.0 ? ldd : 0;
  if (w_img && T <= 8) {
    nvfp4a_tensor a = {};
    a.data = device_ptr(*w_img, "the weight's image");
    a.dtype = NVFP4A_NVFP4;
    a.global_scale = (const float *)addr(wg, "global");
    a.flags = (unsigned)wf;
    a.scale_max = (int)wm;
    check(nvfp4a_gemv_tc((int)N, (int)T, (int)k, (float)alpha, &a, &b.t, (int)b.ld, (float)beta, c, ldc, &d, ldd, bi.p, stream()));
  } else {
    const Operand a = fp4_operand(w, ws, wg, wf, wm);
    CallScratch scratch;
    check(nvfp4a_gemm((int)N, (int)T, (int)k, (float)alpha, &a.t, (int)a.ld, &b.t, (int)b.ld, (float)beta, c, ldc, &d, ldd, bi.p, stream()));
  }
  return amax;
}

std::tuple<Tensor, OptTensor> linear(const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &w, const Tensor &ws,
                                     const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, const OptTensor &bias, std::optional<ScalarType> out_dtype,
                                     double alpha, bool want_amax, const OptTensor &w_img) {
  const c10::cuda::CUDAGuard guard(w.device());
  const Tensor out = empty({x.size(0), w.size(0)}, result_dtype(x, out_dtype), w);
  return {out, gemm_into(out, x, xs, xg, xf, xm, w, ws, wg, wf, wm, k, bias, alpha, 0.0, want_amax, w_img)};
}
OptTensor linear_out(const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &w, const Tensor &ws,
                     const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, const OptTensor &bias, Tensor out, double alpha, double beta, bool want_amax,
                     const OptTensor &w_img) {
  const c10::cuda::CUDAGuard guard(w.device());
  return gemm_into(out, x, xs, xg, xf, xm, w, ws, wg, wf, wm, k, bias, alpha, beta, want_amax, w_img);
}

// ---- grouped linear (mixture of experts) ---------------------------------------------------------------------------------------------
OptTensor grouped_into(const Tensor &out, const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &seg,
                       const Tensor &w, const Tensor &ws, const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, int64_t groups, const OptTensor &bias,
                       double alpha, double beta, bool want_amax) {
  check_k(k);
  TORCH_CHECK_VALUE(groups >= 1 && w.size(0) % groups == 0, w.size(0), " weight rows do not split into ", groups, " groups");
  TORCH_CHECK_VALUE(seg.scalar_type() == at::kInt && seg.numel() == groups + 1, "seg must hold ", groups + 1, " int32 row offsets");
  const int64_t T = x.size(0), N = w.size(0) / groups;
  check_out(out, T, N);
  const OptTensor amax = amax_buffer(want_amax, out);
  const Operand b = activation(x, xs, xg, xf, xm), a = fp4_operand(w, ws, wg, wf, wm);
  const nvfp4a_tensor d = dense_tensor(out, "out", amax);
  const Bias bi(bias, w.size(0));
  const int ldd = (int)out.stride(0);
  const Tensor sg = seg.contiguous();
  CallScratch scratch;
  check(nvfp4a_gemm_grouped((int)groups, (int)N, (int)k, (int)T, (float)alpha, &a.t, (int)a.ld, &b.t, (int)b.ld, (float)beta, beta != 0.0 ? &d : nullptr,
                            beta != 0.0 ? ldd : 0, &d, ldd, bi.p, (const int *)device_ptr(sg, "seg"), stream()));
  return amax;
}
std::tuple<Tensor, OptTensor> grouped_linear(const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &seg,
                                             const Tensor &w, const Tensor &ws, const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, int64_t groups,
                                             const OptTensor &bias, std::optional<ScalarType> out_dtype, double alpha, bool want_amax) {
  const c10::cuda::CUDAGuard guard(w.device());
  // rows of x past seg[groups] belong to no group: the library leaves their outputs alone, so they read zero
  const Tensor out = zeros({x.size(0), w.size(0) / std::max<int64_t>(groups, 1)}, result_dtype(x, out_dtype), w);
  return {out, grouped_into(out, x, xs, xg, xf, xm, seg, w, ws, wg, wf, wm, k, groups, bias, alpha, 0.0, want_amax)};
}
OptTensor grouped_linear_out(const Tensor &x, const OptTensor &xs, const OptTensor &xg, int64_t xf, int64_t xm, const Tensor &seg, const Tensor &w,
                             const Tensor &ws, const OptTensor &wg, int64_t wf, int64_t wm, int64_t k, int64_t groups, const OptTensor &bias, Tensor out,
                             double alpha, double beta, bool want_amax) {
  const c10::cuda::CUDAGuard guard(w.device());
  return grouped_into(out, x, xs, xg, xf, xm, seg, w, ws, wg, wf, wm, k, groups, bias, alpha, beta, want_amax);
}

// ---- images and the image GEMM -------------------------------------------------------------------------------------------------------
Tensor tc_image(int64_t operand, const Tensor &x, const OptTensor &scales, int64_t flags, int64_t k) {
  const c10::cuda::CUDAGuard guard(x.device());
  const Operand s = activation(x, scales, std::nullopt, flags & (NVFP4A_SCALES_SWIZZLED | NVFP4A_SCALES_UE5M3), 0);
  const size_t size = nvfp4a_tc_image_bytes((int)operand, s.t.dtype, (int)x.size(0), (int)k);
  TORCH_CHECK_NOT_IMPLEMENTED(size != 0, "no image of kind ", operand, " for a torch.", dtype_name(x.scalar_type()), " operand with k = ", k);
  const Tensor image = empty({(int64_t)size}, at::kByte, x);
  check(nvfp4a_tc_image((int)operand, &s.t, (int)s.ld, (int)x.size(0), (int)k, image.data_ptr(), stream()));
  return image;
}

// The zeroed scratch buffer of the `_tc` entries, one per (device, stream): calls on one stream are ordered, and every call leaves the
// buffer zeroed.  (Never destroyed: the CUDA context may be gone before static destructors run.)
void *workspace(const Tensor &like, cudaStream_t s) {
  static std::mutex lock;
  static auto *buffers = new std::map<std::pair<int, cudaStream_t>, Tensor>;
  const std::lock_guard<std::mutex> hold(lock);
  Tensor &b = (*buffers)[{like.device().index(), s}];
  if (!b.defined()) b = zeros({(int64_t)nvfp4a_tc_workspace_bytes()}, at::kByte, like);
  return b.data_ptr();
}

OptTensor image_gemm_into(const Tensor &out, const Tensor &x_img, int64_t x_dtype, const OptTensor &xg, int64_t xf, int64_t xm, int64_t T, const Tensor &w_img,
                          const OptTensor &wg, int64_t wf, int64_t wm, int64_t N, int64_t K, const OptTensor &bias, double alpha, double beta, bool want_amax) {
  TORCH_CHECK_VALUE(x_dtype >= 0 && x_dtype < 3, "x_dtype = ", x_dtype, ": 0 NVFP4, 1 int8, 2 bfloat16");
  check_out(out, T, N);
  const OptTensor amax = amax_buffer(want_amax, out);
  nvfp4a_tensor a = {}, b = {};
  a.data = device_ptr(w_img, "the weight's image");
  a.dtype = NVFP4A_NVFP4;
  a.global_scale = (const float *)addr(wg, "global");
  a.flags = (unsigned)wf;
  a.scale_max = (int)wm;
  b.data = device_ptr(x_img, "the activations' image");
  b.dtype = x_dtype == 0 ? NVFP4A_NVFP4 : x_dtype == 1 ? NVFP4A_INT8 : NVFP4A_BF16;
  if (x_dtype == 0) {
    b.global_scale = (const float *)addr(xg, "global");
    b.flags = (unsigned)xf;
    b.scale_max = (int)xm;
  }
  const nvfp4a_tensor d = dense_tensor(out, "out", amax);
  const Bias bi(bias, N);
  const int ldd = (int)out.stride(0);
  const cudaStream_t s = stream();
  CallScratch scratch;
  check(nvfp4a_gemm_tc((int)N, (int)T, (int)K, (float)alpha, &a, &b, (float)beta, beta != 0.0 ? &d : nullptr, beta != 0.0 ? ldd : 0, &d, ldd, bi.p,
                       workspace(w_img, s), s));
  return amax;
}
std::tuple<Tensor, OptTensor> linear_tc(const Tensor &x_img, int64_t x_dtype, const OptTensor &xg, int64_t xf, int64_t xm, int64_t T, const Tensor &w_img,
                                        const OptTensor &wg, int64_t wf, int64_t wm, int64_t N, int64_t K, const OptTensor &bias, ScalarType out_dtype,
                                        double alpha, bool want_amax) {
  const c10::cuda::CUDAGuard guard(w_img.device());
  const Tensor out = empty({T, N}, out_dtype, w_img);
  return {out, image_gemm_into(out, x_img, x_dtype, xg, xf, xm, T, w_img, wg, wf, wm, N, K, bias, alpha, 0.0, want_amax)};
}
OptTensor linear_tc_out(const Tensor &x_img, int64_t x_dtype, const OptTensor &xg, int64_t xf, int64_t xm, int64_t T, const Tensor &w_img,
                        const OptTensor &wg, int64_t wf, int64_t wm, int64_t N, int64_t K, const OptTensor &bias, Tensor out, double alpha, double beta,
                        bool want_amax) {
  const c10::cuda::CUDAGuard guard(w_img.device());
  return image_gemm_into(out, x_img, x_dtype, xg, xf, xm, T, w_img, wg, wf, wm, N, K, bias, alpha, beta, want_amax);
}

// ---- quantization ---------------------------------------------------------------------------------------------------------------------
void check_matrix16(const Tensor &x, const char *fn) {
  TORCH_CHECK_VALUE(x.dim() == 2, fn, " takes a matrix, got shape ", x.sizes());
  dense_code(x.scalar_type());
  TORCH_CHECK_VALUE(x.size(1) % 16 == 0, x.size(1), " values per row: NVFP4 / INT8 blocks hold 16, so the last dimension must be a multiple of 16");
}
// block scales of a [rows, cols] matrix; entries no kernel writes (the swizzled layout's padding) read zero
Tensor scale_buffer(int64_t rows, int64_t cols, int64_t flags, const Tensor &like) {
  if (!(flags & NVFP4A_SCALES_SWIZZLED)) return empty({rows, cols / 16}, at::kByte, like);
  const int64_t r = (rows + 127) / 128 * 128, c = (cols / 16 + 3) / 4 * 4;
  return r != rows || c != cols / 16 ? zeros({r, c}, at::kByte, like) : empty({r, c}, at::kByte, like);
}

using Quantized = std::tuple<OptTensor, OptTensor, OptTensor, OptTensor, OptTensor, OptTensor, OptTensor>;
// nvfp4a_quantize_ex.  With compute_amax the globals are computed here and returned in positions 4 / 5 (g_row / g_col are not used);
// otherwise the given decode factors are applied and those positions are empty.  A column-wise half describes the transpose
// [cols, rows padded to 16].
Quantized quantize_ex(const Tensor &x0, bool rowwise, bool columnwise, const OptTensor &g_row, const OptTensor &g_col, int64_t flags, int64_t smax,
                      int64_t tile_rows, int64_t fos, bool compute_amax, bool want_amax) {
  check_matrix16(x0, "quantize_ex");
  const c10::cuda::CUDAGuard guard(x0.device());
  const int64_t rows = x0.size(0), cols = x0.size(1), rows16 = (rows + 15) / 16 * 16;
  OptTensor out[7];
  auto global = [&](int64_t n) { return rows * cols ? empty({n}, at::kFloat, x0) : zeros({n}, at::kFloat, x0); };   // (stored by the call)
  if (rowwise) {
    out[0] = empty({rows, cols / 2}, at::kByte, x0);
    out[1] = scale_buffer(rows, cols, flags, x0);
    if (compute_amax) out[4] = global(flags & NVFP4A_GLOBAL_PER_ROW ? rows : 1);
  }
  if (columnwise) {
    out[2] = rows16 != rows ? zeros({cols, rows16 / 2}, at::kByte, x0) : empty({cols, rows16 / 2}, at::kByte, x0);
    out[3] = scale_buffer(cols, rows16, flags, x0);
    if (compute_amax) out[5] = global(1);
  }
  if (want_amax) out[6] = zeros({1}, at::kFloat, x0);
  const Tensor x = matrix(x0, 16, "x");
  const nvfp4a_tensor src = dense_tensor(x, "x");
  nvfp4a_tensor half[2] = {};
  for (int h = 0; h < 2; ++h) {
    if (!out[2 * h]) continue;
    half[h].data = out[2 * h]->data_ptr();
    half[h].dtype = NVFP4A_NVFP4;
    half[h].block_scale = out[2 * h + 1]->data_ptr();
    half[h].global_scale = (const float *)addr(compute_amax ? out[4 + h] : h ? g_col : g_row, "global");
    half[h].amax = (float *)addr(out[6], "amax");
    half[h].flags = (unsigned)(h ? flags & ~(int64_t)NVFP4A_GLOBAL_PER_ROW : flags);
    half[h].scale_max = (int)smax;
  }
  nvfp4a_quant_config cfg = {(int)tile_rows, (nvfp4a_4over6)fos, compute_amax ? 1 : 0};
  check(nvfp4a_quantize_ex(&src, (int)x.stride(0), (int)rows, (int)cols, out[0] ? &half[0] : nullptr, (int)cols, out[2] ? &half[1] : nullptr, (int)rows16,
                           &cfg, stream()));
  return {out[0], out[1], out[2], out[3], out[4], out[5], out[6]};
}

std::tuple<Tensor, Tensor> quantize_int8(const Tensor &x0) {
  check_matrix16(x0, "quantize_int8");
  const c10::cuda::CUDAGuard guard(x0.device());
  const int64_t rows = x0.size(0), cols = x0.size(1);
  const Tensor q = empty({rows, cols}, at::kChar, x0), s = empty({rows, cols / 16}, at::kFloat, x0), x = matrix(x0, 16, "x");
  const nvfp4a_tensor src = dense_tensor(x, "x");
  nvfp4a_tensor dst = {};
  dst.data = q.data_ptr();
  dst.dtype = NVFP4A_INT8;
  dst.block_scale = s.data_ptr();
  check(nvfp4a_quantize(&src, (int)x.stride(0), &dst, (int)cols, (int)rows, (int)cols, stream()));
  return {q, s};
}

// quantize_int8 and linear in one call: up to 8 tokens in one kernel too, which makes the activations INT8 itself (the same bytes)
std::tuple<Tensor, OptTensor> linear_w4a8(const Tensor &x0, const Tensor &w, const Tensor &ws, const OptTensor &wg, int64_t wf, int64_t wm, int64_t k,
                                          const OptTensor &bias, std::optional<ScalarType> out_dtype, double alpha, bool want_amax, const OptTensor &w_img) {
  check_matrix16(x0, "linear_w4a8");
  check_k(k);
  const int64_t T = x0.size(0), N = w.size(0);
  if (T >= 1 && T <= 8 && T * k <= NVFP4A_B200_GEMV_W4A8_VALUES && x0.size(1) == k && x0.device() == w.device()) {
    const c10::cuda::CUDAGuard guard(w.device());
    const Tensor x = matrix(x0, 16, "x");
    if (x.stride(0) % 64 == 0) {
      const nvfp4a_tensor b = dense_tensor(x, "x");
      const Tensor out = empty({T, N}, result_dtype(x0, out_dtype), w);
      const OptTensor amax = amax_buffer(want_amax, out);
      const nvfp4a_tensor d = dense_tensor(out, "out", amax);
      const Bias bi(bias, N);
      Operand a;
      if (w_img) {
        a.t.data = device_ptr(*w_img, "the weight's image");
        a.t.dtype = NVFP4A_NVFP4;
        a.t.global_scale = (const float *)addr(wg, "global");
        a.t.flags = (unsigned)wf;
        a.t.scale_max = (int)wm;
      } else {
        a = fp4_operand(w, ws, wg, wf, wm);
      }
      const nvfp4a_status st = nvfp4a_b200_gemv_w4a8((int)N, (int)T, (int)k, (float)alpha, &a.t, (int)a.ld, w_img ? 1 : 0, &b, (int)x.stride(0), 0.f, nullptr, 0, &d,
                                                     (int)out.stride(0), bi.p, stream());
      if (st != NVFP4A_NOT_SUPPORTED) {
        check(st);
        return {out, amax};
      }
    }
  }
  const auto [q, s] = quantize_int8(x0);
  const c10::cuda::CUDAGuard guard(w.device());
  const Tensor out = empty({T, N}, result_dtype(x0, out_dtype), w);
  return {out, gemm_into(out, q, s, std::nullopt, 0, 0, w, ws, wg, wf, wm, k, bias, alpha, 0.0, want_amax, w_img)};
}

Tensor dequantize(const Tensor &data, const Tensor &scales, const OptTensor &glob, int64_t flags, int64_t smax, int64_t cols, ScalarType dtype) {
  dense_code(dtype);
  const c10::cuda::CUDAGuard guard(data.device());
  const Tensor out = empty({data.size(0), cols}, dtype, data);
  const Operand s = fp4_operand(data, scales, glob, flags, smax);
  const nvfp4a_tensor d = dense_tensor(out, "out");
  check(nvfp4a_dequantize(&s.t, (int)s.ld, &d, (int)cols, (int)data.size(0), (int)cols, stream()));
  return out;
}

}  // namespace

TORCH_LIBRARY_IMPL(nvfp4effma, CUDA, m) {
  m.impl("quantize_ex", &quantize_ex);
  m.impl("quantize_int8", &quantize_int8);
  m.impl("dequantize", &dequantize);
  m.impl("linear", &linear);
  m.impl("linear_out", &linear_out);
  m.impl("linear_w4a8", &linear_w4a8);
  m.impl("grouped_linear", &grouped_linear);
  m.impl("grouped_linear_out", &grouped_linear_out);
  m.impl("tc_image", &tc_image);
  m.impl("linear_tc", &linear_tc);
  m.impl("linear_tc_out", &linear_tc_out);
}
