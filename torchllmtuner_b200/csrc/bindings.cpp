// Python bindings: thin tensor -> pointer adapters over the C entry points in kernels.h. All checks that can be
// done on the host (dtype, device, contiguity, alignment) are done here so the kernels can assume them.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include <atomic>

#include "kernels.h"

namespace {

using torch::Tensor;

inline cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

inline void check_bf16(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(t.scalar_type() == at::kBFloat16, name, " must be bfloat16");
}
// Number of kernels of this library launched so far (the caller-side count; each binding adds what it enqueues). Atomic: the C++
// autograd nodes run their backward in autograd's thread without the GIL, beside launches of Python threads.
static std::atomic<int64_t> g_launches{0};
inline void check_rc(int rc, const char* what, int launches = 1) {
  TORCH_CHECK(rc == 0, what, " failed with code ", rc);
  g_launches.fetch_add(launches, std::memory_order_relaxed);
}

Tensor& status_word() {
  static Tensor s;
  if (!s.defined()) s = torch::zeros({8}, torch::dtype(torch::kInt32).device(torch::kCUDA));
  return s;
}
inline int* status_ptr() { return status_word().data_ptr<int>(); }

// Row-major 2-D view description of a tensor whose last dim is contiguous.
struct Mat {
  const void* ptr;
  int64_t rows, cols, ld;
};
inline Mat as_mat(const Tensor& t, const char* name) {
  check_bf16(t, name);
  TORCH_CHECK(t.dim() == 2 && t.stride(1) == 1, name, " must be 2-D with a contiguous last dim");
  return Mat{t.data_ptr(), t.size(0), t.size(1), t.stride(0)};
}

// A slice of a peer-memory collective handed to a kernel's comm warps (see csrc/comm.cuh). Pointers are raw device
// addresses (peers' symmetric buffers are not torch tensors on this rank).
struct PySideJob {
  int64_t kind = 0;                 // 0 none, 1 copy, 2 reduce
  std::vector<int64_t> src;         // device addresses
  int64_t dst = 0;
  int64_t n = 0;                    // copy: bytes; reduce: elements
  bool accumulate = false;
  int64_t wait_flags = 0;           // device address of the local flag array, 0 = no wait
  int64_t n_wait = 0;
  int64_t wait_value = 0;
};

// out[M,N] (+)= op(a) * op(b); layouts as in llmt_gemm_bf16. a_mn / b_mn say that the stored matrix is [K][M] / [K][N].
void gemm(const Tensor& a, const Tensor& b, Tensor& out, bool a_mn, bool b_mn, bool accumulate, int64_t max_ctas,
          const c10::optional<PySideJob>& side) {
  c10::cuda::CUDAGuard guard(a.device());
  const Mat A = as_mat(a, "a"), B = as_mat(b, "b");
  TORCH_CHECK(out.is_cuda() && out.dim() == 2 && out.stride(1) == 1, "out must be 2-D CUDA with contiguous last dim");
  const bool f32 = out.scalar_type() == at::kFloat;
  TORCH_CHECK(f32 || out.scalar_type() == at::kBFloat16, "out must be float32 or bfloat16");
  const int64_t M = a_mn ? A.cols : A.rows, K = a_mn ? A.rows : A.cols;
  const int64_t N = b_mn ? B.cols : B.rows, Kb = b_mn ? B.rows : B.cols;
  TORCH_CHECK(K == Kb, "inner dimensions differ: ", K, " vs ", Kb);
  TORCH_CHECK(out.size(0) == M && out.size(1) == N, "out has the wrong shape");
  if (side.has_value() && side->kind != 0) {
    const void* src[8] = {nullptr};
    TORCH_CHECK(side->src.size() >= 1 && side->src.size() <= 8, "side job needs 1..8 sources");
    for (size_t i = 0; i < side->src.size(); ++i) src[i] = reinterpret_cast<const void*>(side->src[i]);
    check_rc(llmt_gemm_bf16_fused(A.ptr, B.ptr, out.data_ptr(), (int)M, (int)N, (int)K, A.ld, B.ld, out.stride(0), a_mn, b_mn, f32,
                                  accumulate, (int)side->kind, (int)side->src.size(), src, reinterpret_cast<void*>(side->dst),
                                  (long long)side->n, side->accumulate, reinterpret_cast<const uint32_t*>(side->wait_flags),
                                  (int)side->n_wait, (uint32_t)side->wait_value, status_ptr(), cur_stream()),
             "llmt_gemm_bf16_fused");
    return;
  }
  const int rc = llmt_gemm_bf16(A.ptr, B.ptr, out.data_ptr(), (int)M, (int)N, (int)K, A.ld, B.ld, out.stride(0), a_mn, b_mn, f32,
                                accumulate, status_ptr(), (int)max_ctas, cur_stream());
  TORCH_CHECK(rc == 0, "llmt_gemm_bf16 failed with code ", rc, " (M=", M, " N=", N, " K=", K, " lda=", A.ld, " ldb=", B.ld,
              " ldc=", out.stride(0), " a_mn=", a_mn, " b_mn=", b_mn, " a%16=", reinterpret_cast<uintptr_t>(A.ptr) % 16,
              " b%16=", reinterpret_cast<uintptr_t>(B.ptr) % 16, ")");
  g_launches.fetch_add(1, std::memory_order_relaxed);
}

// GEMM fused with a tensor-parallel row collective over peer memory (csrc/comm.cuh). mode 1: `a` is the local gathered
// matrix [M,K] that the kernel fills from `peer_src` (each rank's [M/world, K] chunk) while it multiplies; mode 2: `c` is
// this rank's symmetric partial matrix [M,N], `out` [M/world, N] receives the reduced rows (+ residual).
void gemm_tp(const Tensor& a, const Tensor& b, Tensor& c, bool b_mn, bool accumulate, int64_t mode, int64_t world, int64_t rank, int64_t epoch,
             const std::vector<int64_t>& peer_src, int64_t flags, const std::vector<int64_t>& peer_flags, Tensor& counters,
             const c10::optional<Tensor>& acc, const c10::optional<Tensor>& out, const c10::optional<Tensor>& residual) {
  c10::cuda::CUDAGuard guard(a.device());
  const Mat A = as_mat(a, "a"), B = as_mat(b, "b");
  check_bf16(c, "c");
  TORCH_CHECK(c.dim() == 2 && c.stride(1) == 1);
  const int64_t M = A.rows, K = A.cols, N = b_mn ? B.cols : B.rows, Kb = b_mn ? B.rows : B.cols;
  TORCH_CHECK(K == Kb && c.size(0) == M && c.size(1) == N, "gemm_tp: shapes do not match");
  TORCH_CHECK(!accumulate || b_mn, "gemm_tp: accumulate is only built for the [K][N] layout of b");
  TORCH_CHECK((int64_t)peer_src.size() == world && (int64_t)peer_flags.size() == world && world <= 8);
  TORCH_CHECK(counters.is_cuda() && counters.scalar_type() == at::kInt && counters.numel() >= 3 * world);
  const void* ps[8] = {nullptr};
  uint32_t* pf[8] = {nullptr};
  for (int64_t i = 0; i < world; ++i) {
    ps[i] = reinterpret_cast<const void*>(peer_src[i]);
    pf[i] = reinterpret_cast<uint32_t*>(peer_flags[i]);
  }
  float* accp = nullptr;
  void* outp = nullptr;
  const void* resp = nullptr;
  if (mode == 2) {
    TORCH_CHECK(acc.has_value() && out.has_value(), "reduce-scatter form needs acc and out");
    TORCH_CHECK(acc->scalar_type() == at::kFloat && acc->is_contiguous() && acc->numel() >= M / world * N);
    check_bf16(*out, "out");
    TORCH_CHECK(out->is_contiguous() && out->numel() == M / world * N);
    accp = acc->data_ptr<float>();
    outp = out->data_ptr();
    if (residual.has_value()) {
      check_bf16(*residual, "residual");
      TORCH_CHECK(residual->is_contiguous() && residual->numel() == out->numel());
      resp = residual->data_ptr();
    }
  }
  check_rc(llmt_gemm_bf16_tp(A.ptr, B.ptr, c.data_ptr(), (int)M, (int)N, (int)K, A.ld, B.ld, c.stride(0), b_mn, accumulate, (int)mode, (int)world,
                             (int)rank, (uint32_t)epoch, ps, reinterpret_cast<const uint32_t*>(flags), pf,
                             reinterpret_cast<uint32_t*>(counters.data_ptr<int>()), accp, outp, resp, status_ptr(), cur_stream()),
           "llmt_gemm_bf16_tp");
}

// ---- expert-parallel exchange over peer memory (csrc/ep_comm.cu). Peer buffers are raw device addresses.
static void fill_ptrs(const std::vector<int64_t>& v, void** out) {
  TORCH_CHECK(v.size() >= 1 && v.size() <= 8, "1..8 peers");
  for (size_t i = 0; i < 8; ++i) out[i] = i < v.size() ? reinterpret_cast<void*>(v[i]) : nullptr;
}
inline void check_i32(const Tensor& t, const char* n) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kInt && t.is_contiguous(), n, " must be a contiguous CUDA int32 tensor");
}

// Returns (seg_offsets [E/R + 1], totals [E/R], send_off [E]) as int32 device tensors.
std::vector<Tensor> ep_exchange(const Tensor& flat, int64_t E, int64_t me, const std::vector<int64_t>& tables,
                                const std::vector<int64_t>& flags, int64_t epoch, int64_t cap) {
  c10::cuda::CUDAGuard guard(flat.device());
  TORCH_CHECK(flat.is_cuda() && flat.scalar_type() == at::kLong && flat.is_contiguous());
  const int64_t R = (int64_t)tables.size();
  void *tp[8], *fp[8];
  fill_ptrs(tables, tp);
  fill_ptrs(flags, fp);
  auto o = torch::dtype(torch::kInt32).device(flat.device());
  Tensor seg = torch::empty({E / R + 1}, o), tot = torch::empty({E / R}, o), off = torch::empty({E}, o);
  check_rc(llmt_ep_exchange(flat.data_ptr<int64_t>(), flat.numel(), (int)E, (int)R, (int)me, tp, fp, (uint32_t)epoch, (int)cap,
                            seg.data_ptr<int>(), tot.data_ptr<int>(), off.data_ptr<int>(), status_ptr(), cur_stream()),
           "llmt_ep_exchange");
  return {seg, tot, off};
}

// (drank, drow) int32 [ncopies]: owner rank and row of every token copy (stable order inside each expert's run).
std::vector<Tensor> ep_plan(const Tensor& flat, int64_t E, int64_t R, const Tensor& send_off) {
  c10::cuda::CUDAGuard guard(flat.device());
  TORCH_CHECK(flat.is_cuda() && flat.scalar_type() == at::kLong && flat.is_contiguous());
  check_i32(send_off, "send_off");
  auto o = torch::dtype(torch::kInt32).device(flat.device());
  Tensor drank = torch::empty({flat.numel()}, o), drow = torch::empty({flat.numel()}, o);
  check_rc(llmt_ep_plan(flat.data_ptr<int64_t>(), flat.numel(), (int)E, (int)R, send_off.data_ptr<int>(), drank.data_ptr<int>(),
                        drow.data_ptr<int>(), cur_stream()),
           "llmt_ep_plan");
  return {drank, drow};
}

// peers[drank[c]][drow[c]] = scale[c] * src[c / k]; returns dot[c] = <src[c / k], other[c]> when `other` is given.
c10::optional<Tensor> ep_push_rows(const Tensor& src, const c10::optional<Tensor>& scale, const Tensor& drank, const Tensor& drow,
                                   const std::vector<int64_t>& bufs, int64_t cap, int64_t k, const c10::optional<Tensor>& other) {
  c10::cuda::CUDAGuard guard(src.device());
  check_bf16(src, "src");
  TORCH_CHECK(src.dim() == 2 && src.is_contiguous());
  check_i32(drank, "drank");
  check_i32(drow, "drow");
  const int64_t n = drank.numel(), D = src.size(1);
  TORCH_CHECK(drow.numel() == n && n == src.size(0) * k, "one destination per token copy");
  void* bp[8];
  fill_ptrs(bufs, bp);
  const float* sp = nullptr;
  if (scale.has_value()) {
    TORCH_CHECK(scale->scalar_type() == at::kFloat && scale->is_contiguous() && scale->numel() == n);
    sp = scale->data_ptr<float>();
  }
  c10::optional<Tensor> dot;
  const void* op = nullptr;
  float* dp = nullptr;
  if (other.has_value()) {
    check_bf16(*other, "other");
    TORCH_CHECK(other->is_contiguous() && other->numel() == n * D);
    dot = torch::empty({n}, torch::dtype(torch::kFloat32).device(src.device()));
    op = other->data_ptr();
    dp = dot->data_ptr<float>();
  }
  check_rc(llmt_ep_push_rows(src.data_ptr(), sp, drank.data_ptr<int>(), drow.data_ptr<int>(), bp, (int)bufs.size(), (int)cap, n, (int)k,
                             (int)D, op, dp, status_ptr(), cur_stream()),
           "llmt_ep_push_rows");
  return dot;
}

// out[t] = sum_j w[t, j] * peers[drank][drow]; returns (out, raw rows [T*k, D] when keep).
std::vector<Tensor> ep_pull_rows(const std::vector<int64_t>& bufs, const Tensor& drank, const Tensor& drow,
                                 const c10::optional<Tensor>& w, int64_t cap, int64_t T, int64_t k, int64_t D, bool keep) {
  c10::cuda::CUDAGuard guard(drank.device());
  check_i32(drank, "drank");
  check_i32(drow, "drow");
  TORCH_CHECK(drank.numel() == T * k && drow.numel() == T * k);
  void* bp[8];
  fill_ptrs(bufs, bp);
  auto o = torch::dtype(torch::kBFloat16).device(drank.device());
  Tensor out = torch::empty({T, D}, o);
  Tensor kp = keep ? torch::empty({T * k, D}, o) : Tensor();
  const float* wp = nullptr;
  if (w.has_value()) {
    TORCH_CHECK(w->scalar_type() == at::kFloat && w->is_contiguous() && w->numel() == T * k);
    wp = w->data_ptr<float>();
  }
  check_rc(llmt_ep_pull_rows(bp, (int)bufs.size(), drank.data_ptr<int>(), drow.data_ptr<int>(), wp, out.data_ptr(),
                             keep ? kp.data_ptr() : nullptr, (int)cap, (int)T, (int)k, (int)D, cur_stream()),
           "llmt_ep_pull_rows");
  if (keep) return {out, kp};
  return {out};
}

// dst rows below seg_offsets[-1] = live rows of src (address), alignment padding zeroed when zero_pad.
void ep_clone_rows(int64_t src, Tensor& dst, const Tensor& seg_offsets, const Tensor& totals, bool zero_pad) {
  c10::cuda::CUDAGuard guard(dst.device());
  check_bf16(dst, "dst");
  TORCH_CHECK(dst.dim() == 2 && dst.is_contiguous());
  check_i32(seg_offsets, "seg_offsets");
  check_i32(totals, "totals");
  check_rc(llmt_ep_clone_rows(reinterpret_cast<const void*>(src), dst.data_ptr(), seg_offsets.data_ptr<int>(), totals.data_ptr<int>(),
                              (int)totals.numel(), (int)dst.size(1), zero_pad, cur_stream()),
           "llmt_ep_clone_rows");
}

void side_job(const PySideJob& j, int64_t ctas) {
  const void* src[8] = {nullptr};
  TORCH_CHECK(j.src.size() >= 1 && j.src.size() <= 8, "side job needs 1..8 sources");
  for (size_t i = 0; i < j.src.size(); ++i) src[i] = reinterpret_cast<const void*>(j.src[i]);
  check_rc(llmt_side_job((int)j.kind, (int)j.src.size(), src, reinterpret_cast<void*>(j.dst), (long long)j.n, j.accumulate,
                         reinterpret_cast<const uint32_t*>(j.wait_flags), (int)j.n_wait, (uint32_t)j.wait_value, (int)ctas,
                         status_ptr(), cur_stream()),
           "llmt_side_job");
}

void signal_peers(const std::vector<int64_t>& peer_flag_ptrs, int64_t slot, int64_t value) {
  uint32_t* p[8] = {nullptr};
  TORCH_CHECK(peer_flag_ptrs.size() >= 1 && peer_flag_ptrs.size() <= 8);
  for (size_t i = 0; i < peer_flag_ptrs.size(); ++i) p[i] = reinterpret_cast<uint32_t*>(peer_flag_ptrs[i]);
  check_rc(llmt_signal_peers(p, (int)peer_flag_ptrs.size(), (int)slot, (uint32_t)value, cur_stream()), "llmt_signal_peers");
}

// max_polls == 0: the library's default limit (seconds); tests pass a small limit to see a wait expire quickly.
void wait_flags(int64_t flags_ptr, int64_t n, int64_t value, int64_t site, int64_t max_polls) {
  check_rc(llmt_wait_flags(reinterpret_cast<const uint32_t*>(flags_ptr), (int)n, (uint32_t)value, (int)site, (uint32_t)max_polls,
                           status_ptr(), cur_stream()),
           "llmt_wait_flags");
}

void grouped_gemm(const Tensor& a, const Tensor& b, Tensor& out, const Tensor& seg_offsets, bool b_mn, bool accumulate) {
  c10::cuda::CUDAGuard guard(a.device());
  const Mat A = as_mat(a, "a");
  check_bf16(b, "b");
  check_bf16(out, "out");
  TORCH_CHECK(b.dim() == 3 && b.is_contiguous(), "b must be contiguous [G, N, K] or [G, K, N]");
  TORCH_CHECK(seg_offsets.is_cuda() && seg_offsets.scalar_type() == at::kInt && seg_offsets.is_contiguous());
  const int G = (int)b.size(0);
  TORCH_CHECK(seg_offsets.numel() == G + 1);
  const int64_t N = b_mn ? b.size(2) : b.size(1), K = b_mn ? b.size(1) : b.size(2);
  TORCH_CHECK(A.cols == K && out.size(0) == A.rows && out.size(1) == N && out.stride(1) == 1);
  check_rc(llmt_grouped_gemm_bf16(A.ptr, b.data_ptr(), out.data_ptr(), seg_offsets.data_ptr<int>(), G, (int)A.rows, (int)N,
                                  (int)K, A.ld, out.stride(0), b_mn, 0, accumulate, status_ptr(), cur_stream()),
           "llmt_grouped_gemm_bf16");
}

// out[G, M, N] (+)= a_g^T b_g ; a [rows, M], b [rows, N]
void grouped_wgrad(const Tensor& a, const Tensor& b, Tensor& out, const Tensor& seg_offsets, bool accumulate) {
  c10::cuda::CUDAGuard guard(a.device());
  const Mat A = as_mat(a, "a"), B = as_mat(b, "b");
  TORCH_CHECK(out.dim() == 3 && out.is_contiguous() && out.is_cuda());
  const bool f32 = out.scalar_type() == at::kFloat;
  const int G = (int)out.size(0);
  TORCH_CHECK(seg_offsets.numel() == G + 1 && A.rows == B.rows && out.size(1) == A.cols && out.size(2) == B.cols);
  check_rc(llmt_grouped_wgrad_bf16(A.ptr, B.ptr, out.data_ptr(), seg_offsets.data_ptr<int>(), G, (int)A.rows, (int)A.cols,
                                   (int)B.cols, A.ld, B.ld, f32, accumulate, status_ptr(), cur_stream()),
           "llmt_grouped_wgrad_bf16");
}

std::vector<Tensor> rmsnorm_fwd(const Tensor& x, const c10::optional<Tensor>& res, const Tensor& w, double eps) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(x, "x");
  check_bf16(w, "w");
  TORCH_CHECK(x.is_contiguous() && w.is_contiguous());
  const int64_t D = x.size(-1), T = x.numel() / D;
  Tensor y = torch::empty_like(x);
  Tensor rstd = torch::empty({T}, x.options().dtype(torch::kFloat));
  Tensor s;
  const void* rp = nullptr;
  void* sp = nullptr;
  if (res.has_value()) {
    check_bf16(*res, "res");
    TORCH_CHECK(res->is_contiguous() && res->numel() == x.numel());
    s = torch::empty_like(x);
    rp = res->data_ptr();
    sp = s.data_ptr();
  }
  check_rc(llmt_rmsnorm_fwd(x.data_ptr(), rp, w.data_ptr(), y.data_ptr(), sp, rstd.data_ptr<float>(), (int)T, (int)D,
                            (float)eps, cur_stream()),
           "llmt_rmsnorm_fwd");
  if (res.has_value()) return {y, rstd, s};
  return {y, rstd};
}

// Returns (dx, dw [D], fp32 or, with `dw_bf16`, rounded to bf16 by the kernel that sums it). `x` is the tensor that was
// normalised (the sum when a residual was added).
std::vector<Tensor> rmsnorm_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& rstd,
                                const c10::optional<Tensor>& dres, bool dw_bf16) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(dy, "dy");
  check_bf16(x, "x");
  TORCH_CHECK(dy.is_contiguous() && x.is_contiguous());
  const int64_t D = x.size(-1), T = x.numel() / D;
  Tensor dx = torch::empty_like(x);
  Tensor dw = T > 0 ? torch::empty({D}, x.options().dtype(dw_bf16 ? at::kBFloat16 : at::kFloat))
                    : torch::zeros({D}, x.options().dtype(dw_bf16 ? at::kBFloat16 : at::kFloat));
  Tensor part = torch::empty({llmt_rmsnorm_bwd_partials((int)T), D}, x.options().dtype(torch::kFloat));
  const void* dr = nullptr;
  if (dres.has_value()) {
    check_bf16(*dres, "dres");
    TORCH_CHECK(dres->is_contiguous());
    dr = dres->data_ptr();
  }
  check_rc(llmt_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(), dr, dx.data_ptr(),
                            part.data_ptr<float>(), dw_bf16 ? nullptr : dw.data_ptr<float>(), dw_bf16 ? dw.data_ptr() : nullptr, 0,
                            (int)T, (int)D, cur_stream()),
           "llmt_rmsnorm_bwd", 2);
  return {dx, dw};
}

// x [T, H, HD] with arbitrary token stride (stride(1) == HD, stride(2) == 1). w may be undefined (no norm).
std::vector<Tensor> qk_norm_rope_fwd(const Tensor& x, const c10::optional<Tensor>& w, const Tensor& cosb, const Tensor& sinb,
                                     double eps) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(x, "x");
  TORCH_CHECK(x.dim() == 3 && x.stride(2) == 1 && x.stride(1) == x.size(2), "x must be [T, H, HD] with packed heads");
  TORCH_CHECK(cosb.scalar_type() == at::kFloat && sinb.scalar_type() == at::kFloat && cosb.is_contiguous() && sinb.is_contiguous());
  const int T = (int)x.size(0), H = (int)x.size(1), HD = (int)x.size(2);
  TORCH_CHECK(cosb.size(0) == T && cosb.size(1) == HD / 2);
  Tensor y = torch::empty({T, H, HD}, x.options());
  Tensor rstd = torch::empty({(int64_t)T * H}, x.options().dtype(torch::kFloat));
  const void* wp = w.has_value() ? w->data_ptr() : nullptr;
  check_rc(llmt_qk_norm_rope_fwd(x.data_ptr(), x.stride(0), wp, cosb.data_ptr<float>(), sinb.data_ptr<float>(), y.data_ptr(),
                                 y.stride(0), rstd.data_ptr<float>(), T, H, HD, (float)eps, cur_stream()),
           "llmt_qk_norm_rope_fwd");
  return {y, rstd};
}

std::vector<Tensor> qk_norm_rope_bwd(const Tensor& dy, const Tensor& x, const c10::optional<Tensor>& w, const Tensor& cosb,
                                     const Tensor& sinb, const Tensor& rstd, bool dw_bf16) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(dy, "dy");
  TORCH_CHECK(dy.dim() == 3 && dy.stride(2) == 1 && dy.stride(1) == dy.size(2));
  TORCH_CHECK(x.dim() == 3 && x.stride(2) == 1 && x.stride(1) == x.size(2));
  const int T = (int)x.size(0), H = (int)x.size(1), HD = (int)x.size(2);
  Tensor dx = torch::empty({T, H, HD}, x.options());
  Tensor dw, part;
  const void* wp = nullptr;
  float *pp = nullptr, *dwp = nullptr;
  void* dw16 = nullptr;
  if (w.has_value()) {
    wp = w->data_ptr();
    dw = torch::empty({HD}, x.options().dtype(dw_bf16 ? at::kBFloat16 : at::kFloat));
    part = torch::empty({llmt_qk_norm_rope_bwd_partials(T, H), HD}, x.options().dtype(torch::kFloat));
    pp = part.data_ptr<float>();
    if (dw_bf16) dw16 = dw.data_ptr();
    else dwp = dw.data_ptr<float>();
  }
  check_rc(llmt_qk_norm_rope_bwd(dy.data_ptr(), dy.stride(0), x.data_ptr(), x.stride(0), wp, cosb.data_ptr<float>(),
                                 sinb.data_ptr<float>(), rstd.data_ptr<float>(), dx.data_ptr(), dx.stride(0), pp, dwp, dw16,
                                 0, T, H, HD, cur_stream()),
           "llmt_qk_norm_rope_bwd", w.has_value() ? 2 : 1);
  if (w.has_value()) return {dx, dw};
  return {dx};
}

inline int64_t row_stride_2d(const Tensor& t) {
  TORCH_CHECK(t.dim() == 2 && t.stride(1) == 1, "expected a 2-D tensor with a contiguous last dim");
  return t.stride(0);
}

static const int* limit_ptr(const c10::optional<Tensor>& row_limit) {
  if (!row_limit.has_value()) return nullptr;
  TORCH_CHECK(row_limit->is_cuda() && row_limit->scalar_type() == at::kInt && row_limit->numel() >= 1, "row_limit must be a CUDA int32 tensor");
  return row_limit->data_ptr<int>();
}

// s fp32 [B, R, C] contiguous, lse fp32 with B * R elements -> P bf16 [B, R, C]; row r is query (r % n) of its chunk.
Tensor attn_rows_probs(const Tensor& s, const Tensor& lse, int64_t n, int64_t diag, double scale, bool causal) {
  c10::cuda::CUDAGuard guard(s.device());
  TORCH_CHECK(s.is_cuda() && s.scalar_type() == at::kFloat && s.is_contiguous() && s.dim() == 3, "s must be a contiguous fp32 [B, R, C]");
  TORCH_CHECK(lse.is_cuda() && lse.scalar_type() == at::kFloat && lse.is_contiguous() && lse.numel() == s.size(0) * s.size(1));
  TORCH_CHECK(n > 0 && s.size(1) % n == 0, "rows per batch must be a multiple of the chunk length");
  Tensor p = torch::empty(s.sizes(), s.options().dtype(at::kBFloat16));
  check_rc(llmt_attn_rows_probs(s.data_ptr<float>(), lse.data_ptr<float>(), p.data_ptr(), s.size(0) * s.size(1), (int)s.size(2), (int)n,
                                (int)diag, (float)scale, causal ? 1 : 0, cur_stream()),
           "llmt_attn_rows_probs");
  return p;
}
Tensor attn_rows_ds(const Tensor& dp, const Tensor& p, const Tensor& delta) {
  c10::cuda::CUDAGuard guard(dp.device());
  TORCH_CHECK(dp.is_cuda() && dp.scalar_type() == at::kFloat && dp.is_contiguous() && dp.dim() == 3);
  TORCH_CHECK(p.is_cuda() && p.scalar_type() == at::kBFloat16 && p.is_contiguous() && p.sizes() == dp.sizes());
  TORCH_CHECK(delta.is_cuda() && delta.scalar_type() == at::kFloat && delta.is_contiguous() && delta.numel() == dp.size(0) * dp.size(1));
  Tensor ds = torch::empty(dp.sizes(), p.options());
  check_rc(llmt_attn_rows_ds(dp.data_ptr<float>(), p.data_ptr(), delta.data_ptr<float>(), ds.data_ptr(), dp.size(0) * dp.size(1),
                             (int)dp.size(2), cur_stream()),
           "llmt_attn_rows_ds");
  return ds;
}

// row_limit (optional int32 device scalar): rows at or beyond it are neither read nor written.
Tensor swiglu_fwd(const Tensor& gate, const Tensor& up, const c10::optional<Tensor>& row_limit) {
  c10::cuda::CUDAGuard guard(gate.device());
  check_bf16(gate, "gate");
  check_bf16(up, "up");
  TORCH_CHECK(row_stride_2d(gate) == row_stride_2d(up) && gate.sizes() == up.sizes());
  Tensor out = torch::empty({gate.size(0), gate.size(1)}, gate.options());
  check_rc(llmt_swiglu_fwd(gate.data_ptr(), up.data_ptr(), out.data_ptr(), gate.size(0), (int)gate.size(1), gate.stride(0),
                           out.stride(0), limit_ptr(row_limit), cur_stream()),
           "llmt_swiglu_fwd");
  return out;
}

// dgate/dup are written into `dgate_out` / `dup_out` (same row stride), which lets them be the two halves of one buffer.
void swiglu_bwd(const Tensor& dout, const Tensor& gate, const Tensor& up, Tensor& dgate_out, Tensor& dup_out,
                const c10::optional<Tensor>& row_limit) {
  c10::cuda::CUDAGuard guard(gate.device());
  check_bf16(dout, "dout");
  TORCH_CHECK(row_stride_2d(gate) == row_stride_2d(up) && row_stride_2d(dgate_out) == row_stride_2d(dup_out));
  check_rc(llmt_swiglu_bwd(dout.data_ptr(), gate.data_ptr(), up.data_ptr(), dgate_out.data_ptr(), dup_out.data_ptr(),
                           gate.size(0), (int)gate.size(1), gate.stride(0), row_stride_2d(dout), dgate_out.stride(0),
                           limit_ptr(row_limit), cur_stream()),
           "llmt_swiglu_bwd");
}

// In place: logits become d(sum CE)/d(logits) * grad_scale. Returns (row_loss fp32 [rows], row_lse fp32 [rows]).
std::vector<Tensor> ce_fwd_bwd(Tensor& logits, const Tensor& labels, double grad_scale, const c10::optional<Tensor>& scale_t,
                               int64_t ignore_index, bool write_grad) {
  c10::cuda::CUDAGuard guard(logits.device());
  check_bf16(logits, "logits");
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1);
  TORCH_CHECK(labels.is_cuda() && labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == logits.size(0));
  const int rows = (int)logits.size(0), V = (int)logits.size(1);
  Tensor loss = torch::empty({rows}, logits.options().dtype(torch::kFloat));
  Tensor lse = torch::empty({rows}, logits.options().dtype(torch::kFloat));
  const float* sp = scale_t.has_value() ? scale_t->data_ptr<float>() : nullptr;
  check_rc(llmt_ce_fwd_bwd(logits.data_ptr(), labels.data_ptr<int64_t>(), loss.data_ptr<float>(), lse.data_ptr<float>(), rows,
                           V, logits.stride(0), sp, (float)grad_scale, (int)ignore_index, write_grad, cur_stream()),
           "llmt_ce_fwd_bwd");
  return {loss, lse};
}

// bf16(x * scale) in a new tensor; x contiguous fp32 or bf16, scale one fp32 value on the device.
Tensor scale_to_bf16(const Tensor& x, const Tensor& scale) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_cuda() && x.is_contiguous() && (x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16),
              "x must be a contiguous fp32 or bf16 CUDA tensor");
  TORCH_CHECK(scale.is_cuda() && scale.scalar_type() == at::kFloat && scale.numel() == 1, "scale must be one fp32 value on the device");
  Tensor out = torch::empty(x.sizes(), x.options().dtype(at::kBFloat16));
  check_rc(llmt_scale_to_bf16(x.data_ptr(), x.scalar_type() == at::kBFloat16, scale.data_ptr<float>(), out.data_ptr(), x.numel(), cur_stream()),
           "llmt_scale_to_bf16");
  return out;
}

// Vocabulary-parallel cross-entropy over one shard of the logits [rows, V/R] (in place: the shard becomes its gradient);
// `stats` / `flags` are every rank's statistics and flag tables in symmetric memory (device addresses).
Tensor ce_vocab_parallel(Tensor& logits, const Tensor& labels, int64_t vocab_start, int64_t me, const std::vector<int64_t>& stats,
                         const std::vector<int64_t>& flags, int64_t cap, int64_t epoch, double grad_scale, int64_t ignore_index,
                         bool write_grad) {
  c10::cuda::CUDAGuard guard(logits.device());
  check_bf16(logits, "logits");
  TORCH_CHECK(logits.dim() == 2 && logits.stride(1) == 1);
  TORCH_CHECK(labels.is_cuda() && labels.scalar_type() == at::kLong && labels.is_contiguous() && labels.numel() == logits.size(0));
  TORCH_CHECK(stats.size() == flags.size() && stats.size() >= 1 && stats.size() <= 8);
  const int rows = (int)logits.size(0), V = (int)logits.size(1), R = (int)stats.size();
  void* sp[8] = {nullptr};
  void* fp[8] = {nullptr};
  for (int i = 0; i < R; ++i) { sp[i] = reinterpret_cast<void*>(stats[i]); fp[i] = reinterpret_cast<void*>(flags[i]); }
  Tensor loss = torch::empty({rows}, logits.options().dtype(torch::kFloat));
  check_rc(llmt_ce_vocab_parallel(logits.data_ptr(), labels.data_ptr<int64_t>(), loss.data_ptr<float>(), rows, V, logits.stride(0),
                                  vocab_start, R, (int)me, sp, fp, (int)cap, (uint32_t)epoch, (float)grad_scale, (int)ignore_index,
                                  write_grad, status_ptr(), cur_stream()),
           "llmt_ce_vocab_parallel");
  return loss;
}

// Table rows of the ids this rank owns, stored into the output shard of the rank that owns each token.
void vp_embed_scatter(const Tensor& ids, const Tensor& w, int64_t vstart, int64_t vend, const std::vector<int64_t>& out, int64_t chunk) {
  c10::cuda::CUDAGuard guard(w.device());
  check_bf16(w, "weight");
  TORCH_CHECK(w.dim() == 2 && w.is_contiguous() && ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous());
  TORCH_CHECK(out.size() >= 1 && out.size() <= 8);
  void* op[8] = {nullptr};
  for (size_t i = 0; i < out.size(); ++i) op[i] = reinterpret_cast<void*>(out[i]);
  check_rc(llmt_vp_embed_scatter(ids.data_ptr<int64_t>(), w.data_ptr(), vstart, vend, op, (int)out.size(), (int)ids.numel(), (int)chunk,
                                 (int)w.size(1), cur_stream()),
           "llmt_vp_embed_scatter");
}

void adamw(Tensor& p32, const c10::optional<Tensor>& p16, const Tensor& g, Tensor& m, Tensor& v, double lr, double b1,
           double b2, double eps, double wd, int64_t step, const c10::optional<Tensor>& clip_coef, double grad_scale,
           bool decoupled) {
  c10::cuda::CUDAGuard guard(p32.device());
  TORCH_CHECK(p32.scalar_type() == at::kFloat && m.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat);
  TORCH_CHECK(p32.is_contiguous() && g.is_contiguous() && m.is_contiguous() && v.is_contiguous());
  const int64_t n = p32.numel();
  TORCH_CHECK(g.numel() == n && m.numel() == n && v.numel() == n);
  const bool gb = g.scalar_type() == at::kBFloat16;
  TORCH_CHECK(gb || g.scalar_type() == at::kFloat, "grad must be bf16 or fp32");
  void* p16p = nullptr;
  if (p16.has_value()) {
    check_bf16(*p16, "p16");
    TORCH_CHECK(p16->is_contiguous() && p16->numel() == n);
    p16p = p16->data_ptr();
  }
  const float* cc = clip_coef.has_value() ? clip_coef->data_ptr<float>() : nullptr;
  check_rc(llmt_adamw(p32.data_ptr<float>(), p16p, g.data_ptr(), gb, m.data_ptr<float>(), v.data_ptr<float>(), n, (float)lr,
                      (float)b1, (float)b2, (float)eps, (float)wd, (int)step, cc, (float)grad_scale, decoupled, cur_stream()),
           "llmt_adamw");
}

// out[0] (+)= sum(x^2), deterministic. scratch: fp32 >= sqnorm_scratch_floats().
void sqnorm(const Tensor& x, Tensor& scratch, Tensor& out, bool accumulate) {
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK(x.is_contiguous() && scratch.scalar_type() == at::kFloat && out.scalar_type() == at::kFloat);
  TORCH_CHECK(scratch.numel() >= llmt_sqnorm_scratch_floats());
  const bool b = x.scalar_type() == at::kBFloat16;
  TORCH_CHECK(b || x.scalar_type() == at::kFloat);
  check_rc(llmt_sqnorm(x.data_ptr(), b, x.numel(), scratch.data_ptr<float>(), out.data_ptr<float>(), accumulate, cur_stream()),
           "llmt_sqnorm", 2);
}
int64_t sqnorm_scratch_floats() { return llmt_sqnorm_scratch_floats(); }

void clip_coef(const Tensor& total_sq, double max_norm, Tensor& coef, Tensor& norm_out, Tensor& finite) {
  c10::cuda::CUDAGuard guard(total_sq.device());
  check_rc(llmt_clip_coef(total_sq.data_ptr<float>(), (float)max_norm, coef.data_ptr<float>(), norm_out.data_ptr<float>(),
                          finite.data_ptr<int>(), cur_stream()),
           "llmt_clip_coef");
}

std::vector<Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& tiles, double scale, bool causal) {
  c10::cuda::CUDAGuard guard(q.device());
  check_bf16(q, "q"); check_bf16(k, "k"); check_bf16(v, "v");
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.dim() == 3);
  TORCH_CHECK(q.stride(2) == 1 && q.stride(1) == q.size(2) && k.stride(2) == 1 && k.stride(1) == k.size(2) &&
              v.stride(2) == 1 && v.stride(1) == v.size(2), "q/k/v need packed heads [T, H, HD]");
  TORCH_CHECK(tiles.is_cuda() && tiles.scalar_type() == at::kInt && tiles.is_contiguous() && tiles.size(1) == 8);
  const int Tq = (int)q.size(0), Hq = (int)q.size(1), HD = (int)q.size(2), Tk = (int)k.size(0), Hkv = (int)k.size(1);
  Tensor o = torch::empty({Tq, Hq, HD}, q.options());
  Tensor lse = torch::empty({Hq, Tq}, q.options().dtype(torch::kFloat));
  check_rc(llmt_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr<float>(), tiles.data_ptr<int>(),
                         (int)tiles.size(0), Tq, Tk, Hq, Hkv, HD, q.stride(0), k.stride(0), v.stride(0), o.stride(0),
                         (float)scale, causal, status_ptr(), cur_stream()),
           "llmt_attn_fwd");
  return {o, lse};
}

// k_tile_passes: the dK/dV kernel runs once per pass; passes after the first accumulate (pieces that share keys).
std::vector<Tensor> attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& dout,
                             const Tensor& lse, const Tensor& q_tiles, const std::vector<Tensor>& k_tile_passes, double scale,
                             bool causal, bool zero_init, bool fused) {
  c10::cuda::CUDAGuard guard(q.device());
  check_bf16(dout, "dout");
  TORCH_CHECK(dout.dim() == 3 && dout.stride(2) == 1 && dout.stride(1) == dout.size(2) && o.is_contiguous());
  const int Tq = (int)q.size(0), Hq = (int)q.size(1), HD = (int)q.size(2), Tk = (int)k.size(0), Hkv = (int)k.size(1);
  Tensor dq = (zero_init && !fused) ? torch::zeros({Tq, Hq, HD}, q.options()) : torch::empty({Tq, Hq, HD}, q.options());
  Tensor dk = zero_init ? torch::zeros({Tk, Hkv, HD}, k.options()) : torch::empty({Tk, Hkv, HD}, k.options());
  Tensor dv = zero_init ? torch::zeros({Tk, Hkv, HD}, v.options()) : torch::empty({Tk, Hkv, HD}, v.options());
  Tensor delta = torch::empty({Hq, Tq}, q.options().dtype(torch::kFloat));
  const int npass = (int)k_tile_passes.size();
  if (fused) {
    // one walk per key tile yields dK, dV and that tile's share of dQ, which is summed in an fp32 accumulator
    Tensor acc = torch::empty({Tq, Hq, HD}, q.options().dtype(torch::kFloat));
    const int n = npass > 0 ? npass : 1;
    for (int p = 0; p < n; ++p) {
      const int* kt = npass > 0 ? k_tile_passes[p].data_ptr<int>() : nullptr;
      const int nkt = npass > 0 ? (int)k_tile_passes[p].size(0) : 0;
      check_rc(llmt_attn_bwd_fused(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dout.data_ptr(), lse.data_ptr<float>(),
                                   delta.data_ptr<float>(), acc.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), kt,
                                   nkt, Tq, Tk, Hq, Hkv, HD, q.stride(0), k.stride(0), v.stride(0), o.stride(0), dout.stride(0),
                                   dq.stride(0), dk.stride(0), dv.stride(0), (float)scale, causal, p == 0, p == n - 1,
                                   status_ptr(), cur_stream()),
               "llmt_attn_bwd_fused", (p == 0 ? 1 : 0) + (nkt > 0 ? 1 : 0) + (p == n - 1 ? 1 : 0));
    }
    return {dq, dk, dv};
  }
  for (int p = 0; p < (npass > 0 ? npass : 1); ++p) {
    const int* kt = npass > 0 ? k_tile_passes[p].data_ptr<int>() : nullptr;
    const int nkt = npass > 0 ? (int)k_tile_passes[p].size(0) : 0;
    check_rc(llmt_attn_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dout.data_ptr(), lse.data_ptr<float>(),
                           delta.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), q_tiles.data_ptr<int>(),
                           p == 0 ? (int)q_tiles.size(0) : 0, kt, nkt, Tq, Tk, Hq, Hkv, HD, q.stride(0), k.stride(0), v.stride(0),
                           o.stride(0), dout.stride(0), dq.stride(0), dk.stride(0), dv.stride(0), (float)scale, causal,
                           /*pass=*/p, status_ptr(), cur_stream()),
             "llmt_attn_bwd", p == 0 ? 3 : 1);
  }
  return {dq, dk, dv};
}

// Head size 256. `zero_init`: some query or key row belongs to no tile and its gradient is zero.
std::vector<Tensor> attn_bwd_wide(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& dout, const Tensor& lse,
                                  const Tensor& q_tiles, const Tensor& k_tiles, double scale, bool causal, bool zero_init) {
  c10::cuda::CUDAGuard guard(q.device());
  check_bf16(q, "q"); check_bf16(k, "k"); check_bf16(v, "v"); check_bf16(dout, "dout");
  for (const Tensor* t : {&q, &k, &v, &dout})
    TORCH_CHECK(t->dim() == 3 && t->size(2) == 256 && t->stride(2) == 1 && t->stride(1) == 256, "operands need packed heads [T, H, 256]");
  for (const Tensor* t : {&q_tiles, &k_tiles})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kInt && t->is_contiguous() && t->size(1) == 8, "tile tables must be int32 [n, 8]");
  TORCH_CHECK(o.is_contiguous() && lse.is_contiguous() && dout.size(0) == q.size(0) && dout.size(1) == q.size(1));
  const int Tq = (int)q.size(0), Hq = (int)q.size(1), Tk = (int)k.size(0), Hkv = (int)k.size(1);
  auto make = [&](const Tensor& t) { return zero_init ? torch::zeros(t.sizes(), t.options()) : torch::empty(t.sizes(), t.options()); };
  Tensor dq = make(q), dk = make(k), dv = make(v);
  Tensor delta = torch::empty({Hq, Tq}, q.options().dtype(torch::kFloat));
  const int nq = (int)q_tiles.size(0), nk = (int)k_tiles.size(0);
  const int nsplit = zero_init ? 1 : llmt_attn_bwd_wide_splits(nk, Hq, Hkv);
  Tensor part;
  if (nsplit > 1) part = torch::empty({2, nsplit, Tk, Hkv, 256}, delta.options());
  check_rc(llmt_attn_bwd_wide(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), dout.data_ptr(), lse.data_ptr<float>(),
                              delta.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), nsplit > 1 ? part.data_ptr<float>() : nullptr,
                              nsplit, q_tiles.data_ptr<int>(), nq, k_tiles.data_ptr<int>(), nk, Tq, Tk, Hq, Hkv, q.stride(0), k.stride(0),
                              v.stride(0), o.stride(0), dout.stride(0), dq.stride(0), dk.stride(0), dv.stride(0), (float)scale, causal,
                              status_ptr(), cur_stream()),
           "llmt_attn_bwd_wide", nsplit > 1 ? 3 : 2);
  return {dq, dk, dv};
}

// ---- MoE
std::vector<Tensor> router_topk(const Tensor& logits, const c10::optional<Tensor>& bias, int64_t k, int64_t score_fn, bool renorm,
                                double route_scale) {
  c10::cuda::CUDAGuard guard(logits.device());
  TORCH_CHECK(logits.is_cuda() && logits.scalar_type() == at::kFloat && logits.dim() == 2 && logits.is_contiguous());
  const int T = (int)logits.size(0), E = (int)logits.size(1);
  Tensor w = torch::empty({T, k}, logits.options());
  Tensor idx = torch::empty({T, k}, logits.options().dtype(torch::kLong));
  Tensor counts = torch::zeros({E}, logits.options());
  Tensor denom = torch::empty({T}, logits.options());
  const float* bp = bias.has_value() ? bias->data_ptr<float>() : nullptr;
  check_rc(llmt_router_topk(logits.data_ptr<float>(), bp, w.data_ptr<float>(), idx.data_ptr<int64_t>(), counts.data_ptr<float>(),
                            denom.data_ptr<float>(), T, E, (int)k, (int)score_fn, renorm, (float)route_scale, cur_stream()),
           "llmt_router_topk");
  return {w, idx, counts, denom};
}
Tensor router_topk_bwd(const Tensor& logits, const Tensor& dw, const Tensor& idx, const Tensor& denom, int64_t score_fn, bool renorm,
                       double route_scale) {
  c10::cuda::CUDAGuard guard(logits.device());
  Tensor dl = torch::zeros_like(logits);
  Tensor dwc = dw.contiguous();
  check_rc(llmt_router_topk_bwd(logits.data_ptr<float>(), dwc.data_ptr<float>(), idx.data_ptr<int64_t>(), denom.data_ptr<float>(),
                                dl.data_ptr<float>(), (int)logits.size(0), (int)logits.size(1), (int)idx.size(1), (int)score_fn, renorm,
                                (float)route_scale, cur_stream()),
           "llmt_router_topk_bwd");
  return dl;
}
// flat [n] int64 expert ids -> (dest [n] int64 row of every copy, seg [E + 1] int32, counts [E] int64); copies of one expert
// keep their order, every segment starts on a multiple of `align` rows.
std::vector<Tensor> moe_plan(const Tensor& flat, int64_t E, int64_t align) {
  c10::cuda::CUDAGuard guard(flat.device());
  TORCH_CHECK(flat.is_cuda() && flat.scalar_type() == at::kLong && flat.is_contiguous(), "flat must be a contiguous int64 CUDA tensor");
  const int64_t n = flat.numel();
  Tensor dest = torch::empty({n}, flat.options()), counts = torch::empty({E}, flat.options());
  Tensor ints = torch::empty({E + 1 + llmt_moe_plan_scratch_ints(n, (int)E)}, flat.options().dtype(torch::kInt));
  Tensor seg = torch::empty({E + 1}, ints.options());
  check_rc(llmt_moe_plan(flat.data_ptr<int64_t>(), n, (int)E, (int)align, ints.data_ptr<int>(), dest.data_ptr<int64_t>(), seg.data_ptr<int>(),
                         counts.data_ptr<int64_t>(), status_ptr(), cur_stream()),
           "llmt_moe_plan", 3);
  return {dest, seg, counts};
}
struct Padding {
  const int* seg = nullptr;
  const int64_t* counts = nullptr;
  int E = 0;
};
static Padding padding_of(const c10::optional<Tensor>& seg, const c10::optional<Tensor>& counts) {
  if (!seg.has_value()) return {};
  TORCH_CHECK(counts.has_value() && seg->is_cuda() && seg->scalar_type() == at::kInt && seg->is_contiguous() && counts->is_cuda() &&
                  counts->scalar_type() == at::kLong && counts->is_contiguous() && seg->numel() == counts->numel() + 1,
              "seg must be int32 [E + 1] and counts int64 [E]");
  return {seg->data_ptr<int>(), counts->data_ptr<int64_t>(), (int)counts->numel()};
}
// Without seg / counts the rows must be zero-initialised by the caller; with them the padding rows are zeroed here.
void permute_rows(const Tensor& x, const Tensor& dest, Tensor& rows, int64_t k, const c10::optional<Tensor>& seg,
                  const c10::optional<Tensor>& counts) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(x, "x");
  check_bf16(rows, "rows");
  TORCH_CHECK(x.is_contiguous() && rows.is_contiguous() && dest.scalar_type() == at::kLong && dest.is_contiguous());
  const Padding pad = padding_of(seg, counts);
  check_rc(llmt_permute_rows(x.data_ptr(), dest.data_ptr<int64_t>(), rows.data_ptr(), dest.numel(), (int)k, (int)x.size(1), pad.seg, pad.counts,
                             pad.E, cur_stream()),
           "llmt_permute_rows");
}
Tensor combine_rows(const Tensor& y, const Tensor& dest, const c10::optional<Tensor>& w, int64_t T, int64_t k) {
  c10::cuda::CUDAGuard guard(y.device());
  check_bf16(y, "y");
  TORCH_CHECK(y.is_contiguous() && dest.is_contiguous());
  Tensor out = torch::empty({T, y.size(1)}, y.options());
  const float* wp = w.has_value() ? w->data_ptr<float>() : nullptr;
  check_rc(llmt_combine_rows(y.data_ptr(), dest.data_ptr<int64_t>(), wp, out.data_ptr(), (int)T, (int)k, (int)y.size(1), cur_stream()),
           "llmt_combine_rows");
  return out;
}
std::vector<Tensor> combine_bwd(const Tensor& dout, const Tensor& y, const Tensor& dest, const Tensor& w, int64_t k,
                                const c10::optional<Tensor>& seg, const c10::optional<Tensor>& counts) {
  c10::cuda::CUDAGuard guard(y.device());
  const Padding pad = padding_of(seg, counts);
  Tensor dy = pad.seg != nullptr && dest.numel() > 0 ? torch::empty_like(y) : torch::zeros_like(y);
  Tensor dw = torch::empty({dest.numel()}, y.options().dtype(torch::kFloat));
  Tensor d = dout.contiguous();
  check_rc(llmt_combine_bwd(d.data_ptr(), y.data_ptr(), dest.data_ptr<int64_t>(), w.data_ptr<float>(), dy.data_ptr(), dw.data_ptr<float>(),
                            dest.numel(), (int)k, (int)y.size(1), pad.seg, pad.counts, pad.E, cur_stream()),
           "llmt_combine_bwd");
  return {dy, dw};
}

// ---- around the gated delta rule
static void check_conv(const Tensor& x, const Tensor& w, const Tensor& pos) {
  check_bf16(x, "x");
  check_bf16(w, "w");
  TORCH_CHECK(x.dim() == 2 && x.stride(1) == 1 && w.dim() == 2 && w.is_contiguous() && w.size(0) == x.size(1), "x [T, C], w [C, K]");
  TORCH_CHECK(pos.is_cuda() && pos.scalar_type() == at::kLong && pos.is_contiguous() && pos.numel() == x.size(0), "positions must be int64 [T]");
}
Tensor conv_silu_fwd(const Tensor& x, const Tensor& w, const Tensor& pos) {
  c10::cuda::CUDAGuard guard(x.device());
  check_conv(x, w, pos);
  Tensor y = torch::empty(x.sizes(), x.options());
  check_rc(llmt_conv_silu_fwd(x.data_ptr(), x.stride(0), w.data_ptr(), pos.data_ptr<int64_t>(), y.data_ptr(), (int)x.size(0), (int)x.size(1),
                              (int)w.size(1), cur_stream()),
           "llmt_conv_silu_fwd");
  return y;
}
std::vector<Tensor> conv_silu_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& pos) {
  c10::cuda::CUDAGuard guard(x.device());
  check_conv(x, w, pos);
  check_bf16(dy, "dy");
  TORCH_CHECK(dy.sizes() == x.sizes() && dy.stride(1) == 1);
  const int T = (int)x.size(0), C = (int)x.size(1), K = (int)w.size(1);
  Tensor dx = torch::empty(x.sizes(), x.options()), dw = T > 0 ? torch::empty(w.sizes(), w.options()) : torch::zeros(w.sizes(), w.options());
  Tensor part = torch::empty({llmt_conv_silu_blocks(T), C, K}, x.options().dtype(at::kFloat));
  check_rc(llmt_conv_silu_bwd(dy.data_ptr(), dy.stride(0), x.data_ptr(), x.stride(0), w.data_ptr(), pos.data_ptr<int64_t>(), dx.data_ptr(),
                              part.data_ptr<float>(), dw.data_ptr(), T, C, K, cur_stream()),
           "llmt_conv_silu_bwd", 2);
  return {dx, dw};
}
// mixed [T, (2 Hk + Hv) d] -> q, k [T, Hv, d], v [T, Hv, d] fp32
std::vector<Tensor> delta_qkv_fwd(const Tensor& mixed, int64_t Hk, int64_t Hv, double qscale, double eps) {
  c10::cuda::CUDAGuard guard(mixed.device());
  check_bf16(mixed, "mixed");
  TORCH_CHECK(mixed.dim() == 2 && mixed.is_contiguous() && Hk > 0 && mixed.size(1) % (2 * Hk + Hv) == 0);
  const int64_t T = mixed.size(0), d = mixed.size(1) / (2 * Hk + Hv);
  auto o = mixed.options().dtype(at::kFloat);
  Tensor q = torch::empty({T, Hv, d}, o), k = torch::empty({T, Hv, d}, o), v = torch::empty({T, Hv, d}, o);
  check_rc(llmt_delta_qkv_fwd(mixed.data_ptr(), q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), (int)T, (int)Hk, (int)Hv, (int)d,
                              (float)qscale, (float)eps, cur_stream()),
           "llmt_delta_qkv_fwd");
  return {q, k, v};
}
Tensor delta_qkv_bwd(const Tensor& dq, const Tensor& dk, const Tensor& dv, const Tensor& mixed, int64_t Hk, int64_t Hv, double qscale, double eps) {
  c10::cuda::CUDAGuard guard(mixed.device());
  for (const Tensor* t : {&dq, &dk, &dv}) TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && t->sizes() == dq.sizes());
  Tensor dm = torch::empty_like(mixed);
  check_rc(llmt_delta_qkv_bwd(dq.data_ptr<float>(), dk.data_ptr<float>(), dv.data_ptr<float>(), mixed.data_ptr(), dm.data_ptr(), (int)mixed.size(0),
                              (int)Hk, (int)Hv, (int)dq.size(2), (float)qscale, (float)eps, cur_stream()),
           "llmt_delta_qkv_bwd");
  return dm;
}
Tensor gated_norm_fwd(const Tensor& x, const Tensor& gate, const Tensor& w, double eps) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(x, "x"); check_bf16(gate, "gate"); check_bf16(w, "w");
  TORCH_CHECK(x.is_contiguous() && gate.is_contiguous() && w.is_contiguous() && x.sizes() == gate.sizes() && x.size(-1) == w.numel());
  Tensor y = torch::empty_like(x);
  check_rc(llmt_gated_norm_fwd(x.data_ptr(), gate.data_ptr(), w.data_ptr(), y.data_ptr(), x.numel() / x.size(-1), (int)x.size(-1), (float)eps,
                               cur_stream()),
           "llmt_gated_norm_fwd");
  return y;
}
std::vector<Tensor> gated_norm_bwd(const Tensor& dy, const Tensor& x, const Tensor& gate, const Tensor& w, double eps) {
  c10::cuda::CUDAGuard guard(x.device());
  check_bf16(dy, "dy");
  TORCH_CHECK(dy.is_contiguous() && dy.sizes() == x.sizes());
  const int64_t D = x.size(-1), R = x.numel() / D;
  Tensor dx = torch::empty_like(x), dg = torch::empty_like(x), dw = R > 0 ? torch::empty_like(w) : torch::zeros_like(w);
  Tensor part = torch::empty({llmt_gated_norm_bwd_blocks(R, (int)D), D}, x.options().dtype(at::kFloat));
  check_rc(llmt_gated_norm_bwd(dy.data_ptr(), x.data_ptr(), gate.data_ptr(), w.data_ptr(), dx.data_ptr(), dg.data_ptr(), part.data_ptr<float>(),
                               dw.data_ptr(), R, (int)D, (float)eps, cur_stream()),
           "llmt_gated_norm_bwd", 2);
  return {dx, dg, dw};
}

// q, k, v [T, H, D], beta, g [T, H] fp32 -> (o [T, H, D], what the backward needs: G, W1, W2, P, inv, S, U).
static void check_delta(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta) {
  for (const Tensor* t : {&q, &k, &v, &beta})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() && reinterpret_cast<uintptr_t>(t->data_ptr()) % 16 == 0,
                "delta rule operands must be contiguous fp32 CUDA tensors on 16-byte boundaries");
  TORCH_CHECK(q.dim() == 3 && k.sizes() == q.sizes() && v.sizes() == q.sizes() && beta.numel() == q.size(0) * q.size(1), "q, k, v [T, H, D], beta [T, H]");
}
std::vector<Tensor> delta_rule_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& g, bool keep) {
  c10::cuda::CUDAGuard guard(q.device());
  check_delta(q, k, v, beta);
  TORCH_CHECK(g.is_cuda() && g.scalar_type() == at::kFloat && g.is_contiguous() && g.numel() == beta.numel());
  const int64_t T = q.size(0), H = q.size(1), D = q.size(2), N = (T + 63) / 64;
  auto o = q.options();
  Tensor out = torch::empty(q.sizes(), o), G = torch::empty({N, H, 64}, o.dtype(at::kDouble)), W1 = torch::empty({N, H, 64, D}, o), W2 = torch::empty({N, H, 64, D}, o),
         P = torch::empty({N, H, 64, 64}, o), inv, S, U;
  if (keep) {
    inv = torch::empty({2, N, H, 64, 64}, o);
    S = torch::empty({N, H, D, D}, o);
    U = torch::empty(q.sizes(), o);
  }
  check_rc(llmt_delta_rule_fwd(q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), beta.data_ptr<float>(), g.data_ptr<float>(),
                               G.data_ptr<double>(), W1.data_ptr<float>(), W2.data_ptr<float>(), P.data_ptr<float>(),
                               keep ? inv.data_ptr<float>() : nullptr, keep ? S.data_ptr<float>() : nullptr, keep ? U.data_ptr<float>() : nullptr,
                               out.data_ptr<float>(), (int)T, (int)H, (int)D, cur_stream()),
           "llmt_delta_rule_fwd", 2);
  if (!keep) return {out};
  return {out, G, W1, W2, P, inv, S, U};
}
std::vector<Tensor> delta_rule_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& G,
                                   const Tensor& W1, const Tensor& W2, const Tensor& P, const Tensor& inv, const Tensor& S, const Tensor& U) {
  c10::cuda::CUDAGuard guard(q.device());
  check_delta(q, k, v, beta);
  TORCH_CHECK(dout.scalar_type() == at::kFloat && dout.is_contiguous() && dout.sizes() == q.sizes() && reinterpret_cast<uintptr_t>(dout.data_ptr()) % 16 == 0);
  TORCH_CHECK(G.is_cuda() && G.scalar_type() == at::kDouble && G.is_contiguous());
  for (const Tensor* t : {&W1, &W2, &P, &inv, &S, &U}) TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous());
  Tensor dS = torch::empty_like(S), dU = torch::empty_like(U), dq = torch::empty_like(q), dk = torch::empty_like(q), dv = torch::empty_like(q),
         db = torch::empty_like(beta), dg = torch::empty_like(beta);
  check_rc(llmt_delta_rule_bwd(dout.data_ptr<float>(), q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), beta.data_ptr<float>(),
                               G.data_ptr<double>(), W1.data_ptr<float>(), W2.data_ptr<float>(), P.data_ptr<float>(), inv.data_ptr<float>(),
                               S.data_ptr<float>(), U.data_ptr<float>(), dS.data_ptr<float>(), dU.data_ptr<float>(), dq.data_ptr<float>(),
                               dk.data_ptr<float>(), dv.data_ptr<float>(), db.data_ptr<float>(), dg.data_ptr<float>(), (int)q.size(0),
                               (int)q.size(1), (int)q.size(2), cur_stream()),
           "llmt_delta_rule_bwd", 2);
  return {dq, dk, dv, db, dg};
}

// ---- autograd nodes of the small hot ops
// A launch of a small training step takes the device a few microseconds and took the host 20 to 27: the Python frames of
// apply() and backward(), reshapes, allocations and attribute look-ups around one kernel call. These nodes do the same with the
// same kernels in C++. What needs Python stays there: a pending peer-memory collective (it rides on the product, so the
// queue decides) and weights whose gradient accumulates into an owner's buffer (`main_grad`) hand the whole backward to
// `functional._linears_backward`. Saved tensors go through the usual hooks (activation checkpointing, offload).
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;

struct PyHooks {
  PyObject* symm = nullptr;               // module that holds the active collective queue (`_ACTIVE`)
  PyObject* linears_backward = nullptr;   // functional._linears_backward(x2, ws, dys, need_x, need_ws)
};
PyHooks& py_hooks() {
  static PyHooks h;                       // references are kept for the life of the process
  return h;
}
void set_autograd_hooks(const py::object& symm, const py::object& linears_backward) {
  PyHooks& h = py_hooks();
  py::object a = symm, b = linears_backward;
  Py_XDECREF(h.symm);
  Py_XDECREF(h.linears_backward);
  h.symm = a.release().ptr();
  h.linears_backward = b.release().ptr();
}
// With the GIL held: is a collective queue active, or does one of the weights own a gradient buffer?
bool python_takes_backward(const variable_list& ws) {
  const PyHooks& h = py_hooks();
  TORCH_CHECK(h.symm != nullptr && h.linears_backward != nullptr, "set_autograd_hooks was not called");
  py::object active = py::reinterpret_steal<py::object>(PyObject_GetAttrString(h.symm, "_ACTIVE"));
  if (!active) throw py::error_already_set();
  if (!active.is_none()) return true;
  for (const Tensor& w : ws) {
    py::object pw = py::reinterpret_steal<py::object>(THPVariable_Wrap(w));
    if (!pw) throw py::error_already_set();
    if (!PyObject_HasAttrString(pw.ptr(), "main_grad")) continue;
    if (!py::object(pw.attr("main_grad")).is_none()) return true;
  }
  return false;
}

Tensor rows_2d(const Tensor& t) {
  Tensor r = t.dim() == 2 ? t : t.reshape({-1, t.size(-1)});
  return r.stride(1) == 1 ? r : r.contiguous();
}
Tensor like_rows(const Tensor& x, int64_t n) {         // empty tensor of x's shape with the last dimension replaced
  auto sz = x.sizes().vec();
  sz.back() = n;
  return torch::empty(sz, x.options());
}

// y_i = x W_i^T for one to three weights that read the same rows. dx is summed by the products' epilogues.
struct NativeLinears : public torch::autograd::Function<NativeLinears> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w0, const OptTensor& w1, const OptTensor& w2) {
    Tensor x2 = rows_2d(x);
    variable_list saved{x2, w0}, ys;
    if (w1.has_value()) saved.push_back(*w1);
    if (w2.has_value()) saved.push_back(*w2);
    for (size_t i = 1; i < saved.size(); ++i) {
      Tensor y = like_rows(x, saved[i].size(0)), y2 = y.view({-1, saved[i].size(0)});
      gemm(x2, saved[i], y2, false, false, false, 0, c10::nullopt);
      ys.push_back(y);
    }
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->save_for_backward(saved);
    return ys;
  }
  static variable_list backward(AutogradContext* ctx, variable_list dys) {
    variable_list saved = ctx->get_saved_variables();
    const Tensor x2 = saved[0];
    const variable_list ws(saved.begin() + 1, saved.end());
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector();
    variable_list out(4);
    const bool need_x = ctx->needs_input_grad(0);
    variable_list d2;
    for (const Tensor& d : dys) d2.push_back(rows_2d(d));
    {
      py::gil_scoped_acquire gil;
      try {
        if (python_takes_backward(ws)) {
          std::vector<bool> need_w;
          for (size_t i = 0; i < ws.size(); ++i) need_w.push_back(ctx->needs_input_grad(1 + i));
          py::object fn = py::reinterpret_borrow<py::object>(py_hooks().linears_backward);
          auto r = fn(x2, ws, d2, need_x, need_w).cast<std::vector<OptTensor>>();
          for (size_t i = 0; i < r.size() && i < out.size(); ++i)
            if (r[i].has_value()) out[i] = i == 0 ? r[i]->reshape(shape) : *r[i];
          return out;
        }
      } catch (py::error_already_set& e) {
        e.restore();                      // the engine carries a python_error, type and all, to the thread that called backward
        throw python_error();
      }
    }
    for (size_t i = 0; i < ws.size(); ++i) {
      if (need_x) {
        if (i == 0) out[0] = torch::empty(shape, x2.options());
        Tensor dx = out[0].view({-1, x2.size(1)});
        gemm(d2[i], ws[i], dx, false, true, i > 0, 0, c10::nullopt);               // dy [M,N] @ W [N,K]
      }
      if (ctx->needs_input_grad(1 + i)) {
        out[1 + i] = torch::empty(ws[i].sizes(), ws[i].options());
        gemm(d2[i], x2, out[1 + i], true, true, false, 0, c10::nullopt);           // dy^T [N,M] @ x [M,K]
      }
    }
    return out;
  }
};
variable_list linears_node(const Tensor& x, const variable_list& ws) {
  TORCH_CHECK(ws.size() >= 1 && ws.size() <= 3, "one to three weights");
  return NativeLinears::apply(x, ws[0], ws.size() > 1 ? OptTensor(ws[1]) : OptTensor(), ws.size() > 2 ? OptTensor(ws[2]) : OptTensor());
}

struct NativeSwiGLU : public torch::autograd::Function<NativeSwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gate, const Tensor& up, const OptTensor& row_limit) {
    Tensor g2 = rows_2d(gate), u2 = rows_2d(up);
    if (g2.stride(0) != u2.stride(0)) { g2 = g2.contiguous(); u2 = u2.contiguous(); }
    ctx->save_for_backward({g2, u2, row_limit.has_value() ? *row_limit : Tensor()});
    ctx->saved_data["shape"] = gate.sizes().vec();
    return swiglu_fwd(g2, u2, row_limit).view(gate.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list d) {
    variable_list s = ctx->get_saved_variables();
    const Tensor &g2 = s[0], &u2 = s[1];
    const std::vector<int64_t> shape = ctx->saved_data["shape"].toIntVector();
    const int64_t F = g2.size(1);
    Tensor both = torch::empty({g2.size(0), 2 * F}, g2.options());
    Tensor dg = both.narrow(1, 0, F), du = both.narrow(1, F, F);
    swiglu_bwd(rows_2d(d[0]), g2, u2, dg, du, s[2].defined() ? OptTensor(s[2]) : OptTensor());
    return {shape.size() == 2 ? dg : dg.reshape(shape), shape.size() == 2 ? du : du.reshape(shape), Tensor()};
  }
};

struct NativeRMSNorm : public torch::autograd::Function<NativeRMSNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    Tensor xc = x.contiguous();
    auto r = rmsnorm_fwd(xc, c10::nullopt, w, eps);
    ctx->save_for_backward({xc, w, r[1]});
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list d) {
    variable_list s = ctx->get_saved_variables();
    auto r = rmsnorm_bwd(d[0].contiguous(), s[0], s[1], s[2], c10::nullopt, true);
    return {r[0], r[1], Tensor()};
  }
};
struct NativeAddRMSNorm : public torch::autograd::Function<NativeAddRMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& res, const Tensor& w, double eps) {
    auto r = rmsnorm_fwd(x.contiguous(), res.contiguous(), w, eps);
    ctx->save_for_backward({r[2], w, r[1]});
    return {r[0], r[2]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list d) {
    variable_list s = ctx->get_saved_variables();
    auto r = rmsnorm_bwd(d[0].contiguous(), s[0], s[1], s[2], d[1].contiguous(), true);
    return {r[0], r[0], r[1], Tensor()};
  }
};

// One node for q and one for k: either output can be differentiated (and its graph freed) without the other.
struct NativeQKNormRope : public torch::autograd::Function<NativeQKNormRope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& w, const Tensor& cosb, const Tensor& sinb, double eps) {
    auto r = qk_norm_rope_fwd(x, w, cosb, sinb, eps);
    ctx->save_for_backward({x, w.has_value() ? *w : Tensor(), cosb, sinb, r[1]});
    return r[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list d) {
    variable_list s = ctx->get_saved_variables(), out(5);
    Tensor dy = d[0];
    if (dy.stride(2) != 1 || dy.stride(1) != dy.size(2)) dy = dy.contiguous();
    const Tensor& w = s[1];
    const bool w16 = w.defined() && w.scalar_type() == at::kBFloat16;
    auto r = qk_norm_rope_bwd(dy, s[0], w.defined() ? OptTensor(w) : OptTensor(), s[2], s[3], s[4], w16);
    out[0] = r[0];
    if (w.defined()) out[1] = w16 ? r[1] : r[1].to(w.scalar_type());
    return out;
  }
};
Tensor swiglu_node(const Tensor& g, const Tensor& u, const OptTensor& row_limit) { return NativeSwiGLU::apply(g, u, row_limit); }
Tensor rmsnorm_node(const Tensor& x, const Tensor& w, double eps) { return NativeRMSNorm::apply(x, w, eps); }
variable_list add_rmsnorm_node(const Tensor& x, const Tensor& r, const Tensor& w, double eps) { return NativeAddRMSNorm::apply(x, r, w, eps); }
variable_list qk_norm_rope_node(const Tensor& q, const Tensor& k, const OptTensor& qw, const OptTensor& kw, const Tensor& cosb, const Tensor& sinb, double eps) {
  return {NativeQKNormRope::apply(q, qw, cosb, sinb, eps), NativeQKNormRope::apply(k, kw, cosb, sinb, eps)};
}

// Reads the status word (synchronises the current stream) and clears it. Returns {code, site, block, extra}.
std::vector<int64_t> read_status(bool clear) {
  Tensor h = status_word().cpu();
  std::vector<int64_t> r{h[0].item<int64_t>(), h[1].item<int64_t>(), h[2].item<int64_t>(), h[3].item<int64_t>()};
  if (clear && r[0] != 0) status_word().zero_();
  return r;
}
Tensor status_tensor() { return status_word(); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<PySideJob>(m, "SideJob")
      .def(py::init<>())
      .def_readwrite("kind", &PySideJob::kind)
      .def_readwrite("src", &PySideJob::src)
      .def_readwrite("dst", &PySideJob::dst)
      .def_readwrite("n", &PySideJob::n)
      .def_readwrite("accumulate", &PySideJob::accumulate)
      .def_readwrite("wait_flags", &PySideJob::wait_flags)
      .def_readwrite("n_wait", &PySideJob::n_wait)
      .def_readwrite("wait_value", &PySideJob::wait_value);
  m.def("gemm", &gemm, "bf16 tcgen05 GEMM", py::arg("a"), py::arg("b"), py::arg("out"), py::arg("a_mn"), py::arg("b_mn"),
        py::arg("accumulate") = false, py::arg("max_ctas") = 0, py::arg("side") = py::none());
  m.def("delta_rule_fwd", &delta_rule_fwd);
  m.def("delta_rule_bwd", &delta_rule_bwd);
  m.def("conv_silu_fwd", &conv_silu_fwd);
  m.def("conv_silu_bwd", &conv_silu_bwd);
  m.def("delta_qkv_fwd", &delta_qkv_fwd);
  m.def("delta_qkv_bwd", &delta_qkv_bwd);
  m.def("gated_norm_fwd", &gated_norm_fwd);
  m.def("gated_norm_bwd", &gated_norm_bwd);
  m.def("set_autograd_hooks", &set_autograd_hooks);
  m.def("linears_node", &linears_node);
  m.def("swiglu_node", &swiglu_node);
  m.def("rmsnorm_node", &rmsnorm_node);
  m.def("add_rmsnorm_node", &add_rmsnorm_node);
  m.def("qk_norm_rope_node", &qk_norm_rope_node);
  m.def("router_topk", &router_topk);
  m.def("router_topk_bwd", &router_topk_bwd);
  m.def("moe_plan", &moe_plan);
  m.def("permute_rows", &permute_rows, py::arg("x"), py::arg("dest"), py::arg("rows"), py::arg("k"), py::arg("seg") = py::none(),
        py::arg("counts") = py::none());
  m.def("combine_rows", &combine_rows);
  m.def("combine_bwd", &combine_bwd, py::arg("dout"), py::arg("y"), py::arg("dest"), py::arg("w"), py::arg("k"), py::arg("seg") = py::none(),
        py::arg("counts") = py::none());
  m.def("gemm_tp", &gemm_tp, py::arg("a"), py::arg("b"), py::arg("c"), py::arg("b_mn"), py::arg("accumulate"), py::arg("mode"), py::arg("world"),
        py::arg("rank"), py::arg("epoch"), py::arg("peer_src"), py::arg("flags"), py::arg("peer_flags"), py::arg("counters"),
        py::arg("acc") = py::none(), py::arg("out") = py::none(), py::arg("residual") = py::none());
  m.def("ep_exchange", &ep_exchange);
  m.def("ep_plan", &ep_plan);
  m.def("ep_push_rows", &ep_push_rows);
  m.def("ep_pull_rows", &ep_pull_rows);
  m.def("ep_clone_rows", &ep_clone_rows);
  m.def("side_job", &side_job);
  m.def("signal_peers", &signal_peers);
  m.def("wait_flags", &wait_flags, py::arg("flags_ptr"), py::arg("n"), py::arg("value"), py::arg("site"), py::arg("max_polls") = 0);
  m.def("grouped_gemm", &grouped_gemm, py::arg("a"), py::arg("b"), py::arg("out"), py::arg("seg_offsets"), py::arg("b_mn"),
        py::arg("accumulate") = false);
  m.def("grouped_wgrad", &grouped_wgrad);
  m.def("rmsnorm_fwd", &rmsnorm_fwd);
  m.def("rmsnorm_bwd", &rmsnorm_bwd, py::arg("dy"), py::arg("x"), py::arg("w"), py::arg("rstd"), py::arg("dres"), py::arg("dw_bf16") = false);
  m.def("qk_norm_rope_fwd", &qk_norm_rope_fwd);
  m.def("qk_norm_rope_bwd", &qk_norm_rope_bwd, py::arg("dy"), py::arg("x"), py::arg("w"), py::arg("cos"), py::arg("sin"), py::arg("rstd"),
        py::arg("dw_bf16") = false);
  m.def("attn_rows_probs", &attn_rows_probs);
  m.def("attn_rows_ds", &attn_rows_ds);
  m.def("swiglu_fwd", &swiglu_fwd, py::arg("gate"), py::arg("up"), py::arg("row_limit") = py::none());
  m.def("swiglu_bwd", &swiglu_bwd, py::arg("dout"), py::arg("gate"), py::arg("up"), py::arg("dgate_out"), py::arg("dup_out"),
        py::arg("row_limit") = py::none());
  m.def("ce_fwd_bwd", &ce_fwd_bwd);
  m.def("scale_to_bf16", &scale_to_bf16);
  m.def("ce_vocab_parallel", &ce_vocab_parallel);
  m.def("vp_embed_scatter", &vp_embed_scatter);
  m.def("adamw", &adamw);
  m.def("sqnorm", &sqnorm);
  m.def("sqnorm_scratch_floats", &sqnorm_scratch_floats);
  m.def("clip_coef", &clip_coef);
  m.def("attn_fwd", &attn_fwd, py::arg("q"), py::arg("k"), py::arg("v"), py::arg("tiles"), py::arg("scale"), py::arg("causal"));
  m.def("attn_bwd", &attn_bwd);
  m.def("attn_bwd_wide", &attn_bwd_wide);
  m.def("read_status", &read_status, py::arg("clear") = true);
  m.def("status_tensor", &status_tensor);
  m.def("launch_count", &launch_count);
}
