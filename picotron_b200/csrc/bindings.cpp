// Python bindings of the sm_100a kernels (module picotron_b200._C).
// This file contains no device code: it validates tensors, allocates outputs through the PyTorch
// caching allocator and calls the C launch API of the .cu files on the current CUDA stream.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <algorithm>
#include <vector>

using torch::Tensor;

extern "C" {
int pt_gemm_bf16(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
                 long long ldd, int a_mn, int b_mn, int out_mode, int num_sms, cudaStream_t stream);
void pt_gemm_set_pair(int on);
int pt_gemm_get_pair();
int pt_gemm_bf16_fused(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd,
                       int epi, void* H, long long ldh, int inter, const float* cosT, const float* sinT, int seq, int rot_heads,
                       int head_dim, void* status, cudaStream_t stream);
int pt_gemm_bf16_ce(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd,
                    const long long* targets, long long vocab_start, void* part, float* tgt, void* status, cudaStream_t stream);
int pt_ce_finish(void* logits, const void* part, int tiles, const long long* targets, const float* tgt, float* terms, long long T,
                 int V, long long ld, float scale, long long vocab_start, cudaStream_t st);
int pt_ce_combine(const void* part, float* rowmax, float* sumexp, long long T, int tiles, cudaStream_t st);
void* pt_status_word();
void pt_attention_set_profile(unsigned long long* counters);
void pt_gemm_set_group_m(int g);
void pt_gemm_set_tile_n(int n);
int pt_gemm_tile_columns(int M, int n_cols, int K, int f32, int b_mn, int has_192);
int pt_gemm_parts(int M, int N, int K, int kind, int add, int* tile_n);
void pt_gemm_set_cluster(int n);
int pt_gemm_bf16_cluster(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd, int b_mn, const void* res,
                          long long ldr, void* status, cudaStream_t stream);
long long pt_gemm_split_elems(int M, int N, int K, int kind, int parts);
void pt_gemm_set_split_k(int on);
int pt_gemm_bf16_split(const void* A, const void* B, void* D, float* ws, int M, int N, int K, long long lda, long long ldb,
                       long long ldd, int kind, int parts, int tile_n, const void* res, long long ldr, void* status, cudaStream_t stream);
int pt_gemm_get_group_m();
void pt_gemm_set_tma_epilogue(int on);
int pt_gemm_get_tma_epilogue();
unsigned int pt_kernel_status_fetch_and_clear();
unsigned long long pt_launch_count();
void pt_count_launches(int n);
int pt_rmsnorm_fwd(const void* x, const void* delta, const void* w, void* x_new, void* y, float* rstd, int T, int H,
                   float eps, cudaStream_t st);
int pt_rmsnorm_bwd_partial_rows(int T, int num_sms);
int pt_rmsnorm_bwd(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                   float* dw, float* partial, int T, int H, int num_sms, cudaStream_t st);
int pt_rmsnorm_bwd_acc(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                       float* dw_acc, int T, int H, int num_sms, cudaStream_t st);
int pt_rope(void* qkv, const float* cosT, const float* sinT, long long T, int n_rot, int d, int S,
            long long row_stride, int inverse, cudaStream_t st);
int pt_swiglu_fwd(const void* gu, void* out, long long T, int I, cudaStream_t st);
int pt_swiglu_bwd(const void* gu, const void* da, void* dgu, long long T, int I, cudaStream_t st);
int pt_embedding_fwd(const long long* ids, const void* w, void* out, long long T, int H, long long rows,
                     long long vocab_start, cudaStream_t st);
int pt_embedding_bwd(const long long* ids, const void* dy, float* dw, long long T, int H, long long rows,
                     long long vocab_start, cudaStream_t st);
int pt_ce_stats(const void* logits, const long long* targets, float* rowmax, float* sumexp, float* tgt, long long T,
                int V, long long ld, long long vocab_start, cudaStream_t st);
int pt_ce_grad(void* logits, const long long* targets, const float* lse, long long T, int V, long long ld, float scale,
               long long vocab_start, cudaStream_t st);
int pt_accumulate(float* acc, const void* g, long long n, int g_is_f32, cudaStream_t st);
int pt_add(const void* a, const void* b, void* out, long long n, cudaStream_t st);
int pt_scale(float* x, const float* coef, long long n, cudaStream_t st);
int pt_adamw_multi(void** params, const float** grads, float** ms, float** vs, float** masters,
                   const long long* numels, int count, int param_is_bf16, int step, float lr, float beta1, float beta2,
                   float eps, float wd, cudaStream_t st);
int pt_merge_attention(float* out, float* lse, const void* bo, const float* bl, int B, int S, int h, int d,
                       cudaStream_t st);
int pt_allreduce_symm(void* const* buf_ptrs, void* const* flag_ptrs, void* mc_ptr, long long offset_elems, long long n,
                      int is_bf16, float scale, int rank, int world, int num_blocks, long long staging_off_bytes, cudaStream_t st);
void pt_set_wait_limit_ns(unsigned long long ns);
int pt_pdl_enabled();
void pt_set_pdl(int on);
void pt_chain_begin();
void pt_chain_end();
void pt_next_launch_waits();
unsigned long long pt_get_wait_limit_ns();
int pt_gemm_allreduce_bf16(const void* A, const void* B, void* const* buf_ptrs, void* const* flag_ptrs, void* mc_ptr,
                           long long d_offset,
                           int M, int N, int K, long long lda, long long ldb, long long ldd, int a_mn, int b_mn, int rank,
                           int world, int clusters_cap, cudaStream_t stream);
int pt_symm_barrier(void* const* flag_ptrs, int rank, int world, cudaStream_t st);
int pt_ce_stats_combine_peers(void* const* buf_ptrs, long long offset_bytes, int world, long long n, float* lse, float* tgt,
                              cudaStream_t st);
int pt_embedding_gather_peers(const long long* ids, void* const* shard_ptrs, int world, long long rows_per_rank, long long T, int H,
                              void* out, cudaStream_t st);
int pt_gather_peer(void* dst, const void* const* src_ptrs, int n_src, long long bytes_each, cudaStream_t st);
int pt_reduce_dkv_symm(void* const* buf_ptrs, long long offset_elems, int me, int world, long long tokens, int width,
                       void* dk, void* dv, long long dk_row, long long dv_row, cudaStream_t st);
void pt_attention_set_clusters(int largest);
int pt_attention_bwd_parts(int B, int Sq, int Sk, int hq, int hkv, int d, int causal, int n_segs, int sms, int pairs, int triples);
int pt_attention_fwd_segs(const void* q, const void* const* k_ptrs, const void* const* v_ptrs, int n_segs, void* o,
                          float* lse, int B, int Sq, int Sk, int hq, int hkv, int d, long long q_row, long long k_row,
                          long long v_row, int causal, float scale, cudaStream_t st);
int pt_attention_bwd_segs(const void* dout, const void* q, const void* const* k_ptrs, const void* const* v_ptrs, int n_segs,
                          const void* o, const float* lse, const float* delta_in, float* delta_ws, float* dq_ws, void* dq,
                          void* dk, void* dv, int out_f32, long long seg_stride, int B, int Sq, int Sk, int hq, int hkv,
                          int d, long long q_row, long long k_row, long long v_row, long long dq_row, long long dk_row,
                          long long dv_row, int causal, float scale, cudaStream_t st);
int pt_attention_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int Sq, int Sk, int hq,
                     int hkv, int d, long long q_row, long long k_row, long long v_row, int causal, float scale,
                     cudaStream_t st);
int pt_attention_bwd(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse,
                     const float* delta_in, float* delta_ws, float* dq_ws, void* dq, void* dk, void* dv, int B, int Sq,
                     int Sk, int hq, int hkv, int d, long long q_row, long long k_row, long long v_row,
                     long long dq_row, long long dk_row, long long dv_row, int causal, float scale, cudaStream_t st);
int pt_attention_bwd_rope(const void* dout, const void* q, const void* k, const void* v, const void* o, const float* lse,
                          const float* delta_in, float* delta_ws, float* dq_ws, void* dq, void* dk, void* dv, int B, int Sq,
                          int Sk, int hq, int hkv, int d, long long q_row, long long k_row, long long v_row, long long dq_row,
                          long long dk_row, long long dv_row, int causal, float scale, const float* cosT, const float* sinT,
                          int rope_seq, cudaStream_t st);
}

namespace {

inline cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }
inline int num_sms() { return at::cuda::getCurrentDeviceProperties()->multiProcessorCount; }

#define PT_CHECK_RC(rc, what) TORCH_CHECK((rc) == 0, what, " failed with code ", (rc))
// (-6: the attention backward was compiled with another register count than its warpgroups share out)
#define PT_CHECK_BWD_RC(rc, what)                                                                                              \
  do {                                                                                                                         \
    const int rc_ = (rc);                                                                                                      \
    TORCH_CHECK(rc_ != -6, what, ": this build of the kernel has another number of registers per thread than its warpgroups "  \
                "share out; rebuild with python -m picotron_b200.build");                                                      \
    PT_CHECK_RC(rc_, what);                                                                                                    \
  } while (0)
#define PT_CHECK_BF16(t) TORCH_CHECK((t).is_cuda() && (t).scalar_type() == at::kBFloat16, #t " must be a CUDA bf16 tensor")
#define PT_CHECK_F32(t) TORCH_CHECK((t).is_cuda() && (t).scalar_type() == at::kFloat, #t " must be a CUDA fp32 tensor")

// rows x cols view of a 2-D tensor whose rows are contiguous; returns the row stride in elements
inline long long row_stride_2d(const Tensor& t, const char* name) {
  TORCH_CHECK(t.dim() == 2 && (t.size(1) == 1 || t.stride(1) == 1), name, " must be 2-D with contiguous rows");
  return t.size(0) == 1 ? t.size(1) : t.stride(0);
}

std::vector<Tensor> rmsnorm_fwd(const Tensor& x, const Tensor& w, double eps) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w);
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && w.is_contiguous() && w.numel() == x.size(1));
  c10::cuda::CUDAGuard guard(x.device());
  auto y = torch::empty_like(x);
  auto rstd = torch::empty({x.size(0)}, x.options().dtype(at::kFloat));
  PT_CHECK_RC(pt_rmsnorm_fwd(x.data_ptr(), nullptr, w.data_ptr(), nullptr, y.data_ptr(), rstd.data_ptr<float>(),
                             (int)x.size(0), (int)x.size(1), (float)eps, stream()), "rmsnorm_fwd");
  return {y, rstd};
}

std::vector<Tensor> add_rmsnorm_fwd(const Tensor& x, const Tensor& delta, const Tensor& w, double eps) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(delta); PT_CHECK_BF16(w);
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && delta.is_contiguous() && delta.sizes() == x.sizes() &&
              w.numel() == x.size(1));
  c10::cuda::CUDAGuard guard(x.device());
  auto x_new = torch::empty_like(x);
  auto y = torch::empty_like(x);
  auto rstd = torch::empty({x.size(0)}, x.options().dtype(at::kFloat));
  PT_CHECK_RC(pt_rmsnorm_fwd(x.data_ptr(), delta.data_ptr(), w.data_ptr(), x_new.data_ptr(), y.data_ptr(),
                             rstd.data_ptr<float>(), (int)x.size(0), (int)x.size(1), (float)eps, stream()),
              "add_rmsnorm_fwd");
  return {x_new, y, rstd};
}

// Returns {dx, dw}. With `dw_acc` (fp32 [H]) the weight gradient is ADDED to it and returned as the second element.
std::vector<Tensor> rmsnorm_bwd(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& rstd,
                                const c10::optional<Tensor>& dres, const c10::optional<Tensor>& dw_acc) {
  PT_CHECK_BF16(dy); PT_CHECK_BF16(x); PT_CHECK_BF16(w); PT_CHECK_F32(rstd);
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && dy.is_contiguous() && dy.sizes() == x.sizes());
  if (dres.has_value()) { PT_CHECK_BF16(*dres); TORCH_CHECK(dres->is_contiguous() && dres->sizes() == x.sizes()); }
  c10::cuda::CUDAGuard guard(x.device());
  const int T = (int)x.size(0), H = (int)x.size(1);
  if (dw_acc.has_value()) {
    PT_CHECK_F32(*dw_acc);
    TORCH_CHECK(dw_acc->is_contiguous() && dw_acc->numel() == H, "rmsnorm_bwd: dw_acc must be a contiguous fp32 [H] tensor");
  }
  auto dx = torch::empty_like(x);
  // one kernel that adds dw with vector reductions (shapes it covers), else partials + a second kernel
  Tensor dw = dw_acc.has_value() ? *dw_acc : torch::zeros({H}, x.options().dtype(at::kFloat));
  const int rc = pt_rmsnorm_bwd_acc(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(),
                                    dres.has_value() ? dres->data_ptr() : nullptr, dx.data_ptr(), dw.data_ptr<float>(), T, H,
                                    num_sms(), stream());
  if (rc == 0) return {dx, dw};
  TORCH_CHECK(rc == 1, "rmsnorm_bwd failed with code ", rc);
  auto dw_new = torch::empty({H}, x.options().dtype(at::kFloat));
  auto partial = torch::empty({pt_rmsnorm_bwd_partial_rows(T, num_sms()), H}, x.options().dtype(at::kFloat));
  PT_CHECK_RC(pt_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr<float>(),
                             dres.has_value() ? dres->data_ptr() : nullptr, dx.data_ptr(), dw_new.data_ptr<float>(),
                             partial.data_ptr<float>(), T, H, num_sms(), stream()), "rmsnorm_bwd");
  if (dw_acc.has_value()) {
    dw.add_(dw_new);
    return {dx, dw};
  }
  return {dx, dw_new};
}

void rope_(Tensor& qkv, const Tensor& cosT, const Tensor& sinT, int64_t n_rot, int64_t d, int64_t S, bool inverse) {
  PT_CHECK_BF16(qkv); PT_CHECK_F32(cosT); PT_CHECK_F32(sinT);
  TORCH_CHECK(cosT.is_contiguous() && sinT.is_contiguous() && cosT.size(0) >= S && cosT.size(1) == d / 2);
  const long long rs = row_stride_2d(qkv, "qkv");
  TORCH_CHECK(n_rot * d <= qkv.size(1));
  c10::cuda::CUDAGuard guard(qkv.device());
  PT_CHECK_RC(pt_rope(qkv.data_ptr(), cosT.data_ptr<float>(), sinT.data_ptr<float>(), qkv.size(0), (int)n_rot, (int)d,
                      (int)S, rs, inverse ? 1 : 0, stream()), "rope");
}

Tensor swiglu_fwd(const Tensor& gu) {
  PT_CHECK_BF16(gu);
  TORCH_CHECK(gu.dim() == 2 && gu.is_contiguous() && gu.size(1) % 2 == 0);
  c10::cuda::CUDAGuard guard(gu.device());
  auto out = torch::empty({gu.size(0), gu.size(1) / 2}, gu.options());
  PT_CHECK_RC(pt_swiglu_fwd(gu.data_ptr(), out.data_ptr(), gu.size(0), (int)(gu.size(1) / 2), stream()), "swiglu_fwd");
  return out;
}

Tensor swiglu_bwd(const Tensor& gu, const Tensor& da) {
  PT_CHECK_BF16(gu); PT_CHECK_BF16(da);
  TORCH_CHECK(gu.dim() == 2 && gu.is_contiguous() && da.is_contiguous() && da.size(0) == gu.size(0) &&
              da.size(1) * 2 == gu.size(1));
  c10::cuda::CUDAGuard guard(gu.device());
  auto dgu = torch::empty_like(gu);
  PT_CHECK_RC(pt_swiglu_bwd(gu.data_ptr(), da.data_ptr(), dgu.data_ptr(), gu.size(0), (int)da.size(1), stream()),
              "swiglu_bwd");
  return dgu;
}

// A GEMM with few output tiles, K in parts (pt_gemm_parts) through a workspace from the caching allocator; kind 0: D = A B,
// 1: D += A^T B (fp32), 2: D = A B^T (+ res). False (nothing launched) where it would not pay or the operands do not allow it.
bool gemm_split_into(const void* a, const void* b, void* d, int64_t M, int64_t N, int64_t K, long long lda, long long ldb, long long ldd,
                     int kind, const void* res, long long ldr, const at::TensorOptions& on) {
  if (!pt_gemm_get_pair() || !pt_gemm_get_tma_epilogue() || lda % 8 || ldb % 8 || ldd % (kind == 1 ? 4 : 8) || ldr % 8 ||
      (((uintptr_t)a | (uintptr_t)b | (uintptr_t)d | (uintptr_t)res) & 15))
    return false;
  int tile_n = 256;
  const int parts = pt_gemm_parts((int)M, (int)N, (int)K, kind, res != nullptr, &tile_n);
  if (parts < 0) {
    const int rc = pt_gemm_bf16_cluster(a, b, d, (int)M, (int)N, (int)K, lda, ldb, ldd, kind == 0, res, ldr, pt_status_word(), stream());
    if (rc == -5) return false;
    TORCH_CHECK(rc == 0, "gemm (cluster) failed with code ", rc);
    return true;
  }
  if (parts <= 1) return false;
  auto ws = torch::empty({pt_gemm_split_elems((int)M, (int)N, (int)K, kind, parts)}, on.dtype(at::kFloat));
  const int rc = pt_gemm_bf16_split(a, b, d, ws.data_ptr<float>(), (int)M, (int)N, (int)K, lda, ldb, ldd, kind, parts, tile_n, res, ldr,
                                    pt_status_word(), stream());
  if (rc == -5) return false;                            // (CTA pairs cannot be scheduled: the general path)
  TORCH_CHECK(rc == 0, "gemm (split) failed with code ", rc);
  return true;
}

// gu[T, 2I] = x w_gu^T and h[T, I] = silu(gate) * up from ONE GEMM (SwiGLU epilogue). Returns {} when the fused kernel does
// not cover the case (CTA pairs or the TMA epilogue unavailable, I % 128 != 0): the caller then runs GEMM + activation kernel.
std::vector<Tensor> gemm_swiglu(const Tensor& x, const Tensor& w_gu) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w_gu);
  const long long lda = row_stride_2d(x, "x"), ldb = row_stride_2d(w_gu, "w_gu");
  const int64_t M = x.size(0), K = x.size(1), N2 = w_gu.size(0);
  TORCH_CHECK(w_gu.size(1) == K && N2 % 2 == 0, "gemm_swiglu: shape mismatch");
  if (!pt_gemm_get_pair() || (N2 / 2) % 128 != 0) return {};
  c10::cuda::CUDAGuard guard(x.device());
  auto gu = torch::empty({M, N2}, x.options());
  auto h = torch::empty({M, N2 / 2}, x.options());
  const int rc = pt_gemm_bf16_fused(x.data_ptr(), w_gu.data_ptr(), gu.data_ptr(), (int)M, (int)N2, (int)K, lda, ldb, N2, 1,
                                    h.data_ptr(), N2 / 2, (int)(N2 / 2), nullptr, nullptr, 0, 0, 0, pt_status_word(), stream());
  if (rc == 1 || rc == -5) return {};
  TORCH_CHECK(rc == 0, "gemm_swiglu failed with code ", rc);
  return {gu, h};
}

// qkv[T, N] = x w^T with RoPE applied to the first `n_rot` heads in the GEMM epilogue. Returns an undefined tensor when
// the fused kernel does not cover the case.
Tensor gemm_rope(const Tensor& x, const Tensor& w, const Tensor& cosT, const Tensor& sinT, int64_t n_rot, int64_t d, int64_t S) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w); PT_CHECK_F32(cosT); PT_CHECK_F32(sinT);
  const long long lda = row_stride_2d(x, "x"), ldb = row_stride_2d(w, "w");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K, "gemm_rope: shape mismatch");
  TORCH_CHECK(cosT.is_contiguous() && sinT.is_contiguous() && cosT.size(0) >= S && cosT.size(1) == d / 2 && sinT.sizes() == cosT.sizes());
  if (!pt_gemm_get_pair() || N % 8 != 0) return Tensor();
  c10::cuda::CUDAGuard guard(x.device());
  auto qkv = torch::empty({M, N}, x.options());
  const int rc = pt_gemm_bf16_fused(x.data_ptr(), w.data_ptr(), qkv.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, N, 2, nullptr, 0,
                                    0, cosT.data_ptr<float>(), sinT.data_ptr<float>(), (int)S, (int)n_rot, (int)d,
                                    pt_status_word(), stream());
  if (rc == 1 || rc == -5) return Tensor();
  TORCH_CHECK(rc == 0, "gemm_rope failed with code ", rc);
  return qkv;
}

// y[T, N] = x w^T + res (res: bf16 [T, N], the residual stream) from one GEMM whose epilogue fetches the residual tile with
// TMA and adds it before the single rounding to bf16. Returns an undefined tensor when the fused kernel does not cover the case.
Tensor gemm_add(const Tensor& x, const Tensor& w, const Tensor& res) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w); PT_CHECK_BF16(res);
  const long long lda = row_stride_2d(x, "x"), ldb = row_stride_2d(w, "w"), ldh = row_stride_2d(res, "res");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K && res.size(0) == M && res.size(1) == N, "gemm_add: shape mismatch");
  if (!pt_gemm_get_pair() || N % 8 != 0) return Tensor();
  c10::cuda::CUDAGuard guard(x.device());
  auto y = torch::empty({M, N}, x.options());
  if (gemm_split_into(x.data_ptr(), w.data_ptr(), y.data_ptr(), M, N, K, lda, ldb, N, 2, res.data_ptr(), ldh, x.options())) return y;
  const int rc = pt_gemm_bf16_fused(x.data_ptr(), w.data_ptr(), y.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, N, 4,
                                    res.data_ptr(), ldh, 0, nullptr, nullptr, 0, 0, 0, pt_status_word(), stream());
  if (rc == 1 || rc == -5) return Tensor();
  TORCH_CHECK(rc == 0, "gemm_add failed with code ", rc);
  return y;
}

// dgu[T, 2I] = SwiGLU backward of (dy w) against the packed pre-activations gu[T, 2I], all in the dgrad GEMM's epilogue
// (dy: [T, H], w: the down-projection weight [H, I]). Returns an undefined tensor when the fused kernel does not cover the case.
Tensor gemm_dgrad_swiglu_bwd(const Tensor& dy, const Tensor& w, const Tensor& gu) {
  PT_CHECK_BF16(dy); PT_CHECK_BF16(w); PT_CHECK_BF16(gu);
  const long long lda = row_stride_2d(dy, "dy"), ldb = row_stride_2d(w, "w"), ldh = row_stride_2d(gu, "gu");
  const int64_t M = dy.size(0), K = dy.size(1), I = w.size(1);
  TORCH_CHECK(w.size(0) == K && gu.size(0) == M && gu.size(1) == 2 * I, "gemm_dgrad_swiglu_bwd: shape mismatch");
  if (!pt_gemm_get_pair() || I % 64 != 0) return Tensor();
  c10::cuda::CUDAGuard guard(dy.device());
  auto dgu = torch::empty({M, 2 * I}, dy.options());
  const int rc = pt_gemm_bf16_fused(dy.data_ptr(), w.data_ptr(), dgu.data_ptr(), (int)M, (int)I, (int)K, lda, ldb, 2 * I, 5,
                                    gu.data_ptr(), ldh, (int)I, nullptr, nullptr, 0, 0, 0, pt_status_word(), stream());
  if (rc == 1 || rc == -5) return Tensor();
  TORCH_CHECK(rc == 0, "gemm_dgrad_swiglu_bwd failed with code ", rc);
  return dgu;
}

// D = op(A) op(B) on raw operands (pt_gemm_bf16).
void gemm_into(const void* a, const void* b, void* d, int64_t M, int64_t N, int64_t K, long long lda, long long ldb, long long ldd,
               bool trans_a, bool trans_b, int mode, const at::TensorOptions& on) {
  const int kind = mode == 0 && !trans_a ? (trans_b ? 0 : 2) : (mode == 1 && trans_a && trans_b) ? 1 : -1;
  if (kind >= 0 && gemm_split_into(a, b, d, M, N, K, lda, ldb, ldd, kind, nullptr, 0, on)) return;
  const int rc = pt_gemm_bf16(a, b, d, (int)M, (int)N, (int)K, lda, ldb, ldd, trans_a ? 1 : 0, trans_b ? 1 : 0, mode, num_sms(), stream());
  TORCH_CHECK(rc == 0, "gemm failed with code ", rc, " (M=", M, " N=", N, " K=", K, " lda=", lda, " ldb=", ldb, " ldd=", ldd,
              " trans_a=", trans_a, " trans_b=", trans_b, " mode=", mode, " a%16=", (uintptr_t)a % 16, " b%16=", (uintptr_t)b % 16,
              " d%16=", (uintptr_t)d % 16, ")");
}

// D = op(a) op(b); see pt_gemm_bf16. trans_a: a is [K,M]; trans_b: b is [K,N] (else [N,K]).
Tensor gemm(const Tensor& a, const Tensor& b, bool trans_a, bool trans_b, const c10::optional<Tensor>& out,
            bool accumulate) {
  PT_CHECK_BF16(a); PT_CHECK_BF16(b);
  const long long lda = row_stride_2d(a, "a"), ldb = row_stride_2d(b, "b");
  const int64_t M = trans_a ? a.size(1) : a.size(0), K = trans_a ? a.size(0) : a.size(1);
  const int64_t N = trans_b ? b.size(1) : b.size(0), Kb = trans_b ? b.size(0) : b.size(1);
  TORCH_CHECK(K == Kb, "gemm: reduction dims differ (", K, " vs ", Kb, ")");
  c10::cuda::CUDAGuard guard(a.device());
  Tensor d;
  int mode;
  if (out.has_value()) {
    d = *out;
    TORCH_CHECK(d.is_cuda() && d.dim() == 2 && d.size(0) == M && d.size(1) == N, "gemm: bad out shape");
    if (d.scalar_type() == at::kFloat) mode = accumulate ? 1 : 2;
    else { TORCH_CHECK(d.scalar_type() == at::kBFloat16 && !accumulate, "gemm: accumulate needs an fp32 out"); mode = 0; }
  } else {
    TORCH_CHECK(!accumulate, "gemm: accumulate needs out");
    d = torch::empty({M, N}, a.options());
    mode = 0;
  }
  if (K == 0) return mode == 1 ? d : d.zero_();          // (the weight gradient of no tokens: the GEMM writes nothing)
  gemm_into(a.data_ptr(), b.data_ptr(), d.data_ptr(), M, N, K, lda, ldb, row_stride_2d(d, "out"), trans_a, trans_b, mode, a.options());
  return d;
}

Tensor embedding_fwd(const Tensor& ids, const Tensor& w, int64_t vocab_start) {
  PT_CHECK_BF16(w);
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous() && w.is_contiguous());
  c10::cuda::CUDAGuard guard(w.device());
  auto out = torch::empty({ids.numel(), w.size(1)}, w.options());
  PT_CHECK_RC(pt_embedding_fwd((const long long*)ids.data_ptr<int64_t>(), w.data_ptr(), out.data_ptr(), ids.numel(),
                               (int)w.size(1), w.size(0), vocab_start, stream()), "embedding_fwd");
  return out;
}

void embedding_bwd(const Tensor& ids, const Tensor& dy, Tensor& dw, int64_t vocab_start) {
  PT_CHECK_BF16(dy); PT_CHECK_F32(dw);
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous() && dy.is_contiguous() &&
              dw.is_contiguous() && dy.size(0) == ids.numel() && dy.size(1) == dw.size(1));
  c10::cuda::CUDAGuard guard(dw.device());
  PT_CHECK_RC(pt_embedding_bwd((const long long*)ids.data_ptr<int64_t>(), dy.data_ptr(), dw.data_ptr<float>(),
                               ids.numel(), (int)dw.size(1), dw.size(0), vocab_start, stream()), "embedding_bwd");
}

std::vector<Tensor> ce_stats(const Tensor& logits, const Tensor& targets, int64_t vocab_start) {
  PT_CHECK_BF16(logits);
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous() &&
              targets.numel() == logits.size(0));
  const long long ld = row_stride_2d(logits, "logits");
  c10::cuda::CUDAGuard guard(logits.device());
  auto f = logits.options().dtype(at::kFloat);
  auto rowmax = torch::empty({logits.size(0)}, f), sumexp = torch::empty({logits.size(0)}, f),
       tgt = torch::empty({logits.size(0)}, f);
  PT_CHECK_RC(pt_ce_stats(logits.data_ptr(), (const long long*)targets.data_ptr<int64_t>(), rowmax.data_ptr<float>(),
                          sumexp.data_ptr<float>(), tgt.data_ptr<float>(), logits.size(0), (int)logits.size(1), ld,
                          vocab_start, stream()), "ce_stats");
  return {rowmax, sumexp, tgt};
}

// logits[T, V] = x w^T together with the cross-entropy row statistics, which the GEMM's epilogue computes tile by tile:
// returns {logits, rowmax, sumexp, target_logit} (the contract of ce_stats), or {} when the fused kernel does not apply.
std::vector<Tensor> gemm_ce_stats(const Tensor& x, const Tensor& w, const Tensor& targets, int64_t vocab_start) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w);
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous() && targets.numel() == x.size(0));
  const long long lda = row_stride_2d(x, "x"), ldb = row_stride_2d(w, "w");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K, "gemm_ce_stats: shape mismatch");
  if (!pt_gemm_get_pair() || N % 8 != 0) return {};
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t tiles = (N + 255) / 256;
  auto f = x.options().dtype(at::kFloat);
  auto logits = torch::empty({M, N}, x.options());
  auto part = torch::empty({M, tiles, 2}, f);
  auto tgt = torch::zeros({M}, f);
  const int rc = pt_gemm_bf16_ce(x.data_ptr(), w.data_ptr(), logits.data_ptr(), (int)M, (int)N, (int)K, lda, ldb, N,
                                 (const long long*)targets.data_ptr<int64_t>(), vocab_start, part.data_ptr(),
                                 tgt.data_ptr<float>(), pt_status_word(), stream());
  if (rc == 1 || rc == -5) return {};
  TORCH_CHECK(rc == 0, "gemm_ce_stats failed with code ", rc);
  auto rowmax = torch::empty({M}, f), sumexp = torch::empty({M}, f);
  PT_CHECK_RC(pt_ce_combine(part.data_ptr(), rowmax.data_ptr<float>(), sumexp.data_ptr<float>(), M, (int)tiles, stream()),
              "ce_combine");
  return {logits, rowmax, sumexp, tgt};
}

// LM head and cross entropy of a chunk of tokens on one GPU: loss terms (lse - target logit) -> terms[T] (fp32) and, with
// `need_grad`, the gradient of the logits, (softmax - onehot) * scale, as the returned bf16 [T, V] tensor (without it the logits
// are never written and the result is an empty tensor). Undefined when the fused kernel does not apply (nothing is written then).
Tensor gemm_ce_loss(const Tensor& x, const Tensor& w, const Tensor& targets, int64_t vocab_start, double scale, Tensor& terms,
                    bool need_grad) {
  PT_CHECK_BF16(x); PT_CHECK_BF16(w); PT_CHECK_F32(terms);
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous() && targets.numel() == x.size(0));
  TORCH_CHECK(terms.is_contiguous() && terms.numel() == x.size(0), "gemm_ce_loss: terms must be a contiguous fp32 [T] tensor");
  const long long lda = row_stride_2d(x, "x"), ldb = row_stride_2d(w, "w");
  const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K, "gemm_ce_loss: shape mismatch");
  if (!pt_gemm_get_pair() || N % 8 != 0) return Tensor();
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t tiles = (N + 255) / 256;
  auto f = x.options().dtype(at::kFloat);
  auto logits = torch::empty({need_grad ? M : 0, N}, x.options());
  void* lp = need_grad ? logits.data_ptr() : nullptr;
  auto part = torch::empty({M * tiles * 2 + M}, f);                      // tile pairs, then the target logits
  float* tgt = part.data_ptr<float>() + M * tiles * 2;
  const long long* tg = (const long long*)targets.data_ptr<int64_t>();
  const int rc = pt_gemm_bf16_ce(x.data_ptr(), w.data_ptr(), lp, (int)M, (int)N, (int)K, lda, ldb, N, tg, vocab_start, part.data_ptr(),
                                 tgt, pt_status_word(), stream());
  if (rc == 1 || rc == -5) return Tensor();
  TORCH_CHECK(rc == 0, "gemm_ce_loss failed with code ", rc);
  PT_CHECK_RC(pt_ce_finish(lp, part.data_ptr(), (int)tiles, tg, tgt, terms.data_ptr<float>(), M, (int)N, N, (float)scale, vocab_start,
                           stream()), "ce_finish");
  return logits;
}

void ce_grad_(Tensor& logits, const Tensor& targets, const Tensor& lse, double scale, int64_t vocab_start) {
  PT_CHECK_BF16(logits); PT_CHECK_F32(lse);
  TORCH_CHECK(targets.is_cuda() && targets.scalar_type() == at::kLong && targets.is_contiguous() &&
              lse.is_contiguous() && lse.numel() == logits.size(0));
  const long long ld = row_stride_2d(logits, "logits");
  c10::cuda::CUDAGuard guard(logits.device());
  PT_CHECK_RC(pt_ce_grad(logits.data_ptr(), (const long long*)targets.data_ptr<int64_t>(), lse.data_ptr<float>(),
                         logits.size(0), (int)logits.size(1), ld, (float)scale, vocab_start, stream()), "ce_grad");
}

void accumulate_(Tensor& acc, const Tensor& g) {
  PT_CHECK_F32(acc);
  TORCH_CHECK(g.is_cuda() && acc.is_contiguous() && g.is_contiguous() && acc.numel() == g.numel());
  TORCH_CHECK(g.scalar_type() == at::kBFloat16 || g.scalar_type() == at::kFloat);
  c10::cuda::CUDAGuard guard(acc.device());
  PT_CHECK_RC(pt_accumulate(acc.data_ptr<float>(), g.data_ptr(), acc.numel(), g.scalar_type() == at::kFloat, stream()),
              "accumulate");
}

Tensor add(const Tensor& a, const Tensor& b) {
  PT_CHECK_BF16(a); PT_CHECK_BF16(b);
  TORCH_CHECK(a.is_contiguous() && b.is_contiguous() && a.sizes() == b.sizes());
  c10::cuda::CUDAGuard guard(a.device());
  auto out = torch::empty_like(a);
  PT_CHECK_RC(pt_add(a.data_ptr(), b.data_ptr(), out.data_ptr(), a.numel(), stream()), "add");
  return out;
}

void adamw_multi_(std::vector<Tensor> params, std::vector<Tensor> grads, std::vector<Tensor> ms, std::vector<Tensor> vs,
                  std::vector<c10::optional<Tensor>> masters, int64_t step, double lr, double beta1, double beta2,
                  double eps, double wd) {
  const size_t n = params.size();
  TORCH_CHECK(grads.size() == n && ms.size() == n && vs.size() == n && masters.size() == n);
  if (n == 0) return;
  c10::cuda::CUDAGuard guard(params[0].device());
  // group by parameter dtype (bf16 / fp32); everything else must be fp32 and contiguous
  for (int pass = 0; pass < 2; ++pass) {
    const auto want = pass == 0 ? at::kBFloat16 : at::kFloat;
    std::vector<void*> p; std::vector<const float*> g; std::vector<float*> m, v, mw; std::vector<long long> numel;
    for (size_t i = 0; i < n; ++i) {
      if (params[i].scalar_type() != want) continue;
      TORCH_CHECK(params[i].is_cuda() && params[i].is_contiguous() && grads[i].is_contiguous() &&
                  ms[i].is_contiguous() && vs[i].is_contiguous(), "adamw: tensors must be contiguous CUDA tensors");
      PT_CHECK_F32(grads[i]); PT_CHECK_F32(ms[i]); PT_CHECK_F32(vs[i]);
      TORCH_CHECK(grads[i].numel() == params[i].numel() && ms[i].numel() == params[i].numel() &&
                  vs[i].numel() == params[i].numel());
      p.push_back(params[i].data_ptr()); g.push_back(grads[i].data_ptr<float>());
      m.push_back(ms[i].data_ptr<float>()); v.push_back(vs[i].data_ptr<float>());
      if (masters[i].has_value()) { PT_CHECK_F32(*masters[i]); mw.push_back(masters[i]->data_ptr<float>()); }
      else mw.push_back(nullptr);
      numel.push_back(params[i].numel());
    }
    if (p.empty()) continue;
    PT_CHECK_RC(pt_adamw_multi(p.data(), g.data(), m.data(), v.data(), mw.data(), numel.data(), (int)p.size(),
                               pass == 0 ? 1 : 0, (int)step, (float)lr, (float)beta1, (float)beta2, (float)eps,
                               (float)wd, stream()), "adamw_multi");
  }
  for (size_t i = 0; i < n; ++i)
    TORCH_CHECK(params[i].scalar_type() == at::kBFloat16 || params[i].scalar_type() == at::kFloat,
                "adamw: parameters must be bf16 or fp32");
}

void scale_(Tensor& x, const Tensor& coef) {
  PT_CHECK_F32(x); PT_CHECK_F32(coef);
  TORCH_CHECK(x.is_contiguous() && coef.numel() == 1 && coef.device() == x.device(),
              "scale_: a contiguous tensor and one coefficient on its device");
  c10::cuda::CUDAGuard guard(x.device());
  PT_CHECK_RC(pt_scale(x.data_ptr<float>(), coef.data_ptr<float>(), x.numel(), stream()), "scale_");
}

void merge_attention_(Tensor& out, Tensor& lse, const Tensor& bo, const Tensor& bl) {
  PT_CHECK_F32(out); PT_CHECK_F32(lse); PT_CHECK_BF16(bo); PT_CHECK_F32(bl);
  TORCH_CHECK(out.dim() == 4 && out.is_contiguous() && bo.is_contiguous() && bo.sizes() == out.sizes() &&
              lse.is_contiguous() && bl.is_contiguous() && lse.sizes() == bl.sizes());
  c10::cuda::CUDAGuard guard(out.device());
  PT_CHECK_RC(pt_merge_attention(out.data_ptr<float>(), lse.data_ptr<float>(), bo.data_ptr(), bl.data_ptr<float>(),
                                 (int)out.size(0), (int)out.size(1), (int)out.size(2), (int)out.size(3), stream()),
              "merge_attention");
}

// q [B,Sq,hq,d], k/v [B,Sk,hkv,d]: last two dims contiguous, token stride arbitrary (slices of packed qkv).
inline long long token_stride(const Tensor& t, const char* name) {
  TORCH_CHECK(t.dim() == 4 && t.stride(3) == 1 && t.stride(2) == t.size(3), name, ": head/feature dims must be packed");
  TORCH_CHECK(t.size(0) == 1 || t.stride(0) == t.stride(1) * t.size(1), name, ": batch and sequence must be collapsible");
  return t.stride(1);
}

std::vector<Tensor> attention_fwd(const Tensor& q, const Tensor& k, const Tensor& v, bool causal, double scale) {
  PT_CHECK_BF16(q); PT_CHECK_BF16(k); PT_CHECK_BF16(v);
  const int B = (int)q.size(0), Sq = (int)q.size(1), hq = (int)q.size(2), d = (int)q.size(3);
  const int Sk = (int)k.size(1), hkv = (int)k.size(2);
  TORCH_CHECK(k.size(0) == B && v.size(0) == B && v.size(1) == Sk && v.size(2) == hkv && k.size(3) == d &&
              v.size(3) == d && hq % hkv == 0);
  c10::cuda::CUDAGuard guard(q.device());
  auto o = torch::empty({B, Sq, hq, d}, q.options());
  auto lse = torch::empty({B, hq, Sq}, q.options().dtype(at::kFloat));
  PT_CHECK_RC(pt_attention_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr<float>(), B, Sq, Sk,
                               hq, hkv, d, token_stride(q, "q"), token_stride(k, "k"), token_stride(v, "v"),
                               causal ? 1 : 0, (float)scale, stream()), "attention_fwd");
  return {o, lse};
}

// With `rope_cos` / `rope_sin` (fp32 [S, d/2]) the inverse rotation of RoPE is applied to dq and dk before they are written
// (query / key i at position i % S), i.e. the gradients are those of the un-rotated q and k.
std::vector<Tensor> attention_bwd(const Tensor& dout, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
                                  const Tensor& lse, bool causal, double scale, const c10::optional<Tensor>& delta,
                                  const c10::optional<std::vector<Tensor>>& outs, const c10::optional<Tensor>& rope_cos,
                                  const c10::optional<Tensor>& rope_sin) {
  PT_CHECK_BF16(dout); PT_CHECK_BF16(q); PT_CHECK_BF16(k); PT_CHECK_BF16(v); PT_CHECK_BF16(o); PT_CHECK_F32(lse);
  const int B = (int)q.size(0), Sq = (int)q.size(1), hq = (int)q.size(2), d = (int)q.size(3);
  const int Sk = (int)k.size(1), hkv = (int)k.size(2);
  TORCH_CHECK(dout.is_contiguous() && o.is_contiguous() && lse.is_contiguous());
  c10::cuda::CUDAGuard guard(q.device());
  Tensor dq, dk, dv;
  if (outs.has_value()) {
    TORCH_CHECK(outs->size() == 3);
    dq = (*outs)[0]; dk = (*outs)[1]; dv = (*outs)[2];
    PT_CHECK_BF16(dq); PT_CHECK_BF16(dk); PT_CHECK_BF16(dv);
  } else {
    dq = torch::empty({B, Sq, hq, d}, q.options());
    dk = torch::empty({B, Sk, hkv, d}, q.options());
    dv = torch::empty({B, Sk, hkv, d}, q.options());
  }
  auto f = q.options().dtype(at::kFloat);
  Tensor delta_ws = torch::empty({B, hq, Sq}, f);
  Tensor dq_ws = delta.has_value() ? torch::zeros({B, Sq, hq, d}, f) : torch::empty({B, Sq, hq, d}, f);
  if (delta.has_value()) { PT_CHECK_F32(*delta); TORCH_CHECK(delta->is_contiguous() && delta->numel() == delta_ws.numel()); }
  const float* cosp = nullptr;
  const float* sinp = nullptr;
  int rope_seq = 0;
  if (rope_cos.has_value()) {
    TORCH_CHECK(rope_sin.has_value(), "attention_bwd: rope_cos without rope_sin");
    PT_CHECK_F32(*rope_cos); PT_CHECK_F32(*rope_sin);
    TORCH_CHECK(rope_cos->is_contiguous() && rope_sin->is_contiguous() && rope_cos->dim() == 2 && rope_cos->size(1) == d / 2 &&
                rope_sin->sizes() == rope_cos->sizes() && rope_cos->size(0) >= Sq && rope_cos->size(0) >= Sk,
                "attention_bwd: rope tables must be fp32 [S, d/2] with S >= the sequence lengths");
    cosp = rope_cos->data_ptr<float>();
    sinp = rope_sin->data_ptr<float>();
    TORCH_CHECK(Sq == Sk, "attention_bwd: rope fusion needs self-attention (Sq == Sk)");
    rope_seq = Sq;                       // row b*Sq + i of the flattened tokens is at position i
  }
  PT_CHECK_BWD_RC(pt_attention_bwd_rope(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                                    lse.data_ptr<float>(), delta.has_value() ? delta->data_ptr<float>() : nullptr,
                                    delta_ws.data_ptr<float>(), dq_ws.data_ptr<float>(), dq.data_ptr(), dk.data_ptr(),
                                    dv.data_ptr(), B, Sq, Sk, hq, hkv, d, token_stride(q, "q"), token_stride(k, "k"),
                                    token_stride(v, "v"), token_stride(dq, "dq"), token_stride(dk, "dk"),
                                    token_stride(dv, "dv"), causal ? 1 : 0, (float)scale, cosp, sinp, rope_seq, stream()),
              "attention_bwd");
  return {dq, dk, dv};
}

// ---------------------------------------------------------------------------------------------
// A decoder layer's launches in one call (one GPU per layer: no tensor, sequence or context parallelism). Small models and
// short sequences are bound by the host: from Python every launch costs 12 to 20 us, more than most of their kernels take, and a
// tensor object per operand costs again: the native call of a forward layer took 43 us with one and takes 26 as it is. So what the
// backward needs lies in TWO allocations (bf16 and fp32), addressed by offsets. The kernels, their order and the fallbacks are those of
// the layer node's Python path.
// ---------------------------------------------------------------------------------------------
struct LayerDims {
  int64_t B, S, H, I, hq, hkv, d;
  int64_t T() const { return B * S; }
  int64_t O() const { return hq * d; }                   // columns of the attention output
  int64_t Q() const { return (hq + 2 * hkv) * d; }       // columns of the packed qkv activation
};

// Element offsets of the parts of a layer's saved activations, each on a 256-byte (bf16) boundary.
struct LayerSaved {
  int64_t h1, qkv, o, x_mid, h2, gu, a, total, rstd1, rstd2, lse, total32;
  explicit LayerSaved(const LayerDims& n) {
    int64_t at = 0;
    auto take = [&at](int64_t elems) { const int64_t here = at; at += (elems + 127) / 128 * 128; return here; };
    const int64_t T = n.T();
    h1 = take(T * n.H); qkv = take(T * n.Q()); o = take(T * n.O()); x_mid = take(T * n.H); h2 = take(T * n.H); gu = take(T * 2 * n.I);
    a = take(T * n.I); total = at;
    at = 0;
    rstd1 = take(T); rstd2 = take(T); lse = take(T * n.hq); total32 = at;
  }
};

// The saved activations of decoder_layer_fwd_packed as tensors {rstd1, h1, qkv, o, lse, x_mid, rstd2, h2, gu, a} (views; for callers that
// work on tensors).
std::vector<Tensor> decoder_layer_saved(const Tensor& s16, const Tensor& s32, int64_t B, int64_t S, int64_t H, int64_t I, int64_t hq,
                                        int64_t hkv, int64_t d) {
  const LayerDims n{B, S, H, I, hq, hkv, d};
  const LayerSaved at(n);
  TORCH_CHECK(s16.numel() == at.total && s32.numel() == at.total32, "decoder_layer_saved: sizes do not match");
  const int64_t T = n.T();
  auto part = [T](const Tensor& t, int64_t off, int64_t cols) { return t.narrow(0, off, T * cols).view({T, cols}); };
  return {s32.narrow(0, at.rstd1, T), part(s16, at.h1, H), part(s16, at.qkv, n.Q()), part(s16, at.o, n.O()),
          s32.narrow(0, at.lse, T * hq).view({B, hq, S}), part(s16, at.x_mid, H), s32.narrow(0, at.rstd2, T), part(s16, at.h2, H),
          part(s16, at.gu, 2 * I), part(s16, at.a, I)};
}

bool all_bf16_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (!t->is_cuda() || t->scalar_type() != at::kBFloat16) return false;
  return true;
}

// Weights and tables of a layer: shapes and layouts that the kernels rely on.
void check_layer(const LayerDims& n, const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT, const Tensor& sinT, const Tensor& wo,
                 const Tensor& ln2, const Tensor& w_gu, const Tensor& wd) {
  auto matrix = [](const Tensor& t, int64_t rows, int64_t cols) {
    return t.dim() == 2 && t.size(0) == rows && t.size(1) == cols && (cols == 1 || t.stride(1) == 1);
  };
  TORCH_CHECK(matrix(w_qkv, n.Q(), n.H) && matrix(wo, n.H, n.O()) && matrix(w_gu, 2 * n.I, n.H) && matrix(wd, n.H, n.I) &&
              ln1.numel() == n.H && ln2.numel() == n.H && ln1.is_contiguous() && ln2.is_contiguous(), "decoder layer: weight shapes");
  PT_CHECK_F32(cosT); PT_CHECK_F32(sinT);
  TORCH_CHECK(cosT.is_contiguous() && cosT.dim() == 2 && cosT.size(0) >= n.S && cosT.size(1) == n.d / 2 && sinT.is_contiguous() &&
              sinT.sizes() == cosT.sizes(), "decoder layer: rope tables must be fp32 [S, d/2] with S >= the sequence length");
}

using bf16_t = at::BFloat16;
inline bf16_t* bf16_ptr(const Tensor& t) { return reinterpret_cast<bf16_t*>(t.data_ptr()); }
inline bool fused_gemm(int rc, const char* what) {          // false: not covered, nothing launched
  if (rc == 1 || rc == -5) return false;
  TORCH_CHECK(rc == 0, what, " failed with code ", rc);
  return true;
}

// A layer's weights and tables as the launches take them; q|k|v and gate|up are one matrix each.
struct LayerPointers {
  const void *ln1, *w_qkv, *wo, *ln2, *w_gu, *wd;
  long long ld_qkv, ld_o, ld_gu, ld_d;
  const float *cosp, *sinp;
};
LayerPointers layer_pointers(const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT, const Tensor& sinT, const Tensor& wo, const Tensor& ln2,
                             const Tensor& w_gu, const Tensor& wd) {
  return {ln1.data_ptr(), w_qkv.data_ptr(), wo.data_ptr(), ln2.data_ptr(), w_gu.data_ptr(), wd.data_ptr(), row_stride_2d(w_qkv, "w_qkv"),
          row_stride_2d(wo, "wo"), row_stride_2d(w_gu, "w_gu"), row_stride_2d(wd, "wd"), cosT.data_ptr<float>(), sinT.data_ptr<float>()};
}

// The launches of a layer's forward: x [T, H] -> out [T, H], the activations to `b` and `f` (LayerSaved).
void layer_fwd(const LayerDims& n, const void* x, const LayerPointers& w, double eps, double scale, bf16_t* const b, float* const f, void* out,
               const at::TensorOptions& on) {
  const LayerSaved at(n);
  const int64_t T = n.T(), H = n.H, I = n.I, O = n.O(), Q = n.Q(), B = n.B, S = n.S, hq = n.hq, hkv = n.hkv, d = n.d;
  bf16_t *const h1 = b + at.h1, *const qkv = b + at.qkv, *const o = b + at.o, *const x_mid = b + at.x_mid, *const h2 = b + at.h2,
         *const gu = b + at.gu, *const a = b + at.a;
  const cudaStream_t st = stream();
  const bool pair = pt_gemm_get_pair();
  void* const status = pt_status_word();
  PT_CHECK_RC(pt_rmsnorm_fwd(x, nullptr, w.ln1, nullptr, h1, f + at.rstd1, (int)T, (int)H, (float)eps, st), "rmsnorm_fwd");
  if (!(pair && Q % 8 == 0 &&
        fused_gemm(pt_gemm_bf16_fused(h1, w.w_qkv, qkv, (int)T, (int)Q, (int)H, H, w.ld_qkv, Q, 2, nullptr, 0, 0, w.cosp, w.sinp, (int)S,
                                      (int)(hq + hkv), (int)d, status, st), "gemm_rope"))) {
    gemm_into(h1, w.w_qkv, qkv, T, Q, H, H, w.ld_qkv, Q, false, false, 0, on);
    PT_CHECK_RC(pt_rope(qkv, w.cosp, w.sinp, T, (int)(hq + hkv), (int)d, (int)S, Q, 0, st), "rope");
  }
  PT_CHECK_RC(pt_attention_fwd(qkv, qkv + O, qkv + O + hkv * d, o, f + at.lse, (int)B, (int)S, (int)S, (int)hq, (int)hkv, (int)d, Q, Q, Q, 1,
                               (float)scale, st), "attention_fwd");
  gemm_into(o, w.wo, out, T, H, O, O, w.ld_o, H, false, false, 0, on);     // (`out` is free until the down projection)
  PT_CHECK_RC(pt_rmsnorm_fwd(x, out, w.ln2, x_mid, h2, f + at.rstd2, (int)T, (int)H, (float)eps, st), "add_rmsnorm_fwd");
  if (!(pair && I % 128 == 0 &&
        fused_gemm(pt_gemm_bf16_fused(h2, w.w_gu, gu, (int)T, (int)(2 * I), (int)H, H, w.ld_gu, 2 * I, 1, a, I, (int)I, nullptr, nullptr,
                                      0, 0, 0, status, st), "gemm_swiglu"))) {
    gemm_into(h2, w.w_gu, gu, T, 2 * I, H, H, w.ld_gu, 2 * I, false, false, 0, on);
    PT_CHECK_RC(pt_swiglu_fwd(gu, a, T, (int)I, st), "swiglu_fwd");
  }
  if (!(pair && H % 8 == 0 && gemm_split_into(a, w.wd, out, T, H, I, I, w.ld_d, H, 2, x_mid, H, on)) &&
      !(pair && H % 8 == 0 &&
        fused_gemm(pt_gemm_bf16_fused(a, w.wd, out, (int)T, (int)H, (int)I, I, w.ld_d, H, 4, x_mid, H, 0, nullptr, nullptr, 0,
                                      0, 0, status, st), "gemm_add"))) {
    Tensor y = torch::empty({T, H}, on);
    gemm_into(a, w.wd, y.data_ptr(), T, H, I, I, w.ld_d, H, false, false, 0, on);
    PT_CHECK_RC(pt_add(x_mid, y.data_ptr(), out, T * H, st), "add");
  }
}

// Returns {x_out, saved bf16, saved fp32} (LayerSaved), or {} (nothing launched) for operands that are not bf16.
std::vector<Tensor> decoder_layer_fwd_packed(const Tensor& x, const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT, const Tensor& sinT,
                                             const Tensor& wo, const Tensor& ln2, const Tensor& w_gu, const Tensor& wd, double eps, int64_t B,
                                             int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale) {
  if (!all_bf16_cuda({&x, &ln1, &w_qkv, &wo, &ln2, &w_gu, &wd})) return {};
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.size(0) == B * S && w_gu.dim() == 2 && hq % hkv == 0);
  const LayerDims n{B, S, x.size(1), w_gu.size(0) / 2, hq, hkv, d};
  check_layer(n, ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd);
  const LayerSaved at(n);
  c10::cuda::CUDAGuard guard(x.device());
  const auto on = x.options();
  Tensor s16 = torch::empty({at.total}, on), s32 = torch::empty({at.total32}, on.dtype(at::kFloat)), out = torch::empty({n.T(), n.H}, on);
  layer_fwd(n, x.data_ptr(), layer_pointers(ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd), eps, scale, bf16_ptr(s16), s32.data_ptr<float>(),
            out.data_ptr(), on);
  return {out, s16, s32};
}

// ---------------------------------------------------------------------------------------------
// All layers of a model in one call each way. A layer of its own costs the host 25 us (forward) and 85 (backward) in Python and autograd on top
// of its launches, which small models and short prompts do not hide. `params`: nine tensors a layer (q, k, v, out, gate, up, down, norm 1,
// norm 2), `tables`: two (cosines, sines).
// ---------------------------------------------------------------------------------------------
constexpr int LAYER_PARAMS = 9;
// The layers' launches are a chain (pt_chain_begin): the GEMMs' B operands are weights and, in the backward, activations of the forward, none of
// which it writes; nor the second operand of the SwiGLU backward.
struct Chain {
  Chain() { pt_chain_begin(); }
  ~Chain() { pt_chain_end(); }
};

// Matrices that lie back to back in one storage, [rows, cols] together: their address, or nullptr.
const void* adjacent(const std::vector<Tensor>& ts, size_t first, int count, int64_t rows, int64_t cols) {
  int64_t seen = 0;
  const char* const base = reinterpret_cast<const char*>(ts[first].data_ptr());
  for (size_t i = first; i < first + count; ++i) {
    const Tensor& t = ts[i];
    if (t.dim() != 2 || t.size(1) != cols || !t.is_contiguous() || base + seen * cols * 2 != t.data_ptr() ||
        t.storage().data() != ts[first].storage().data())
      return nullptr;
    seen += t.size(0);
  }
  return seen == rows ? base : nullptr;
}

// The layers' operands, or {} where one is not a contiguous bf16 tensor of the expected shape on x's device or its q|k|v or gate|up do not lie
// back to back (the single layers' calls say what is wrong, or put them together).
std::vector<LayerPointers> stack_pointers(const LayerDims& n, const Tensor& x, const std::vector<Tensor>& params, const std::vector<Tensor>& tables) {
  const size_t layers = tables.size() / 2;
  if (layers == 0 || params.size() != layers * LAYER_PARAMS || tables.size() != 2 * layers) return {};
  std::vector<LayerPointers> out(layers);
  for (const Tensor& t : params)
    if (t.scalar_type() != at::kBFloat16 || !t.is_contiguous() || t.device() != x.device()) return {};
  for (const Tensor& t : tables)
    if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.device() != x.device() || t.dim() != 2 || t.size(0) < n.S || t.size(1) != n.d / 2)
      return {};
  for (size_t i = 0; i < layers; ++i) {
    const size_t p = i * LAYER_PARAMS;
    LayerPointers& w = out[i];
    w.w_qkv = adjacent(params, p, 3, n.Q(), n.H);
    w.wo = adjacent(params, p + 3, 1, n.H, n.O());
    w.w_gu = adjacent(params, p + 4, 2, 2 * n.I, n.H);
    w.wd = adjacent(params, p + 6, 1, n.H, n.I);
    if (!w.w_qkv || !w.wo || !w.w_gu || !w.wd || params[p + 7].numel() != n.H || params[p + 8].numel() != n.H) return {};
    w.ln1 = params[p + 7].data_ptr();
    w.ln2 = params[p + 8].data_ptr();
    w.ld_qkv = w.ld_gu = n.H;
    w.ld_o = n.O();
    w.ld_d = n.I;
    w.cosp = tables[2 * i].data_ptr<float>();
    w.sinp = tables[2 * i + 1].data_ptr<float>();
  }
  return out;
}
LayerDims stack_dims(const Tensor& x, const std::vector<Tensor>& params, int64_t B, int64_t S, int64_t hq, int64_t hkv, int64_t d) {
  return LayerDims{B, S, x.size(1), params.size() < LAYER_PARAMS || params[6].dim() != 2 ? 0 : params[6].size(1), hq, hkv, d};
}

// x [T, H] through all layers: {x_out, then per layer its saved bf16, saved fp32 and output} (LayerSaved; the output of the last one is
// x_out), or with save = false {x_out} alone, the activations of all layers in one place. {} (nothing launched) where an operand is not as
// stack_pointers wants it.
std::vector<Tensor> decoder_stack_fwd(const Tensor& x, const std::vector<Tensor>& params, const std::vector<Tensor>& tables, double eps, int64_t B,
                                      int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale, bool save) {
  if (!all_bf16_cuda({&x}) || x.dim() != 2 || !x.is_contiguous() || x.size(0) != B * S || x.size(0) == 0 || hq % hkv) return {};
  const LayerDims n = stack_dims(x, params, B, S, hq, hkv, d);
  const auto w = stack_pointers(n, x, params, tables);
  if (w.empty()) return {};
  const LayerSaved at(n);
  c10::cuda::CUDAGuard guard(x.device());
  const auto on = x.options();
  std::vector<Tensor> r(1);
  Tensor in = x, s16, s32, free;
  const Chain chain;
  for (size_t i = 0; i < w.size(); ++i) {
    if (save || i == 0) {
      s16 = torch::empty({at.total}, on);
      s32 = torch::empty({at.total32}, on.dtype(at::kFloat));
    }
    // (without saving, two outputs are used in turn; the caller's x is not one of them)
    Tensor out = !save && i >= 2 ? free : torch::empty({n.T(), n.H}, on);
    layer_fwd(n, in.data_ptr(), w[i], eps, scale, bf16_ptr(s16), s32.data_ptr<float>(), out.data_ptr(), on);
    if (save) {
      r.push_back(s16);
      r.push_back(s32);
      r.push_back(out);
    }
    free = in;
    in = out;
  }
  r[0] = in;
  return r;
}

// The same with the activations as tensors of their own (views): {x_out, h1, rstd1, qkv, o, lse, x_mid, rstd2, h2, gu, a}, or {}.
std::vector<Tensor> decoder_layer_fwd(const Tensor& x, const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT, const Tensor& sinT,
                                      const Tensor& wo, const Tensor& ln2, const Tensor& w_gu, const Tensor& wd, double eps, int64_t B,
                                      int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale) {
  auto r = decoder_layer_fwd_packed(x, ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd, eps, B, S, hq, hkv, d, scale);
  if (r.empty()) return {};
  auto v = decoder_layer_saved(r[1], r[2], B, S, x.size(1), w_gu.size(0) / 2, hq, hkv, d);
  return {r[0], v[1], v[0], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9]};
}

// The fp32 regions of parameters that one GEMM accumulates into together, as one [rows, cols] region: its address, or nullptr unless
// they are adjacent in one storage.
float* packed_region(const std::vector<Tensor>& mg, int first, int count, int64_t rows, int64_t cols) {
  const Tensor& f = mg[first];
  int64_t seen = 0;
  for (int i = first; i < first + count; ++i) {
    const Tensor& t = mg[i];
    if (t.dim() != 2 || !t.is_contiguous() || t.size(1) != cols || t.scalar_type() != at::kFloat || !t.is_cuda() ||
        t.storage().data() != f.storage().data() || t.storage_offset() != f.storage_offset() + seen * cols)
      return nullptr;
    seen += t.size(0);
  }
  TORCH_CHECK(seen == rows, "decoder layer: shape of a gradient region");
  return f.data_ptr<float>();
}

// dx of an RMSNorm (+ dres); the weight gradient is added to dw (fp32 [H]).
void rmsnorm_bwd_into(const void* dy, const void* x, const Tensor& w, const float* rstd, const void* dres, void* dx, const Tensor& dw,
                      int64_t T, int64_t H, const at::TensorOptions& on) {
  const int rc = pt_rmsnorm_bwd_acc(dy, x, w.data_ptr(), rstd, dres, dx, dw.data_ptr<float>(), (int)T, (int)H, num_sms(), stream());
  if (rc == 0) return;
  TORCH_CHECK(rc == 1, "rmsnorm_bwd failed with code ", rc);
  auto dw_new = torch::empty({H}, on.dtype(at::kFloat));
  auto partial = torch::empty({pt_rmsnorm_bwd_partial_rows((int)T, num_sms()), H}, on.dtype(at::kFloat));
  PT_CHECK_RC(pt_rmsnorm_bwd(dy, x, w.data_ptr(), rstd, dres, dx, dw_new.data_ptr<float>(), partial.data_ptr<float>(), (int)T, (int)H,
                             num_sms(), stream()), "rmsnorm_bwd");
  PT_CHECK_RC(pt_accumulate(dw.data_ptr<float>(), dw_new.data_ptr(), H, 1, stream()), "accumulate");
}

// What a layer's backward reads of its forward.
struct LayerActivations {
  const bf16_t *h1, *qkv, *o, *x_mid, *h2, *gu, *a;
  const float *rstd1, *rstd2, *lse;
};

// A second stream beside the current one. It goes on (`go`) from where the current one was at the last `mark`; `done` notes how far it has got and
// `join` makes the current stream wait for that (two notes, so that one may be a layer old). The allocator keeps memory that is allocated on it
// apart.
struct SideStream {
  c10::cuda::CUDAStream stream;
  cudaEvent_t marked, noted[2];
  void mark(cudaStream_t at) { C10_CUDA_CHECK(cudaEventRecord(marked, at)); }
  void go() {
    C10_CUDA_CHECK(cudaStreamWaitEvent(stream, marked, 0));
    pt_next_launch_waits();
  }
  void done(int i) { C10_CUDA_CHECK(cudaEventRecord(noted[i & 1], stream)); }
  void join(cudaStream_t waits, int i) {
    C10_CUDA_CHECK(cudaStreamWaitEvent(waits, noted[i & 1], 0));
    pt_next_launch_waits();
  }
};
// The one beside `current` on its device (the current one), or nullptr where there is none. A thread has up to four a device, for the streams that it used last,
// made at the first use and given back with the thread. (Autograd runs the backward passes of all threads on one thread a device: one side stream
// for all of them would put the weight gradients of one caller behind those of another.) One that is part of a graph capture other than the current
// stream's is left alone: to make it wait for work outside of its capture is an error and ends that capture.
SideStream* side_stream(cudaStream_t current) {
  struct Streams {
    struct Slot {
      cudaStream_t beside = nullptr;
      uint64_t used = 0;
      std::unique_ptr<SideStream> side;
    } slots[4];
    ~Streams() {
      for (auto& slot : slots)
        if (SideStream* s = slot.side.get()) {       // (errors: the process may be past its CUDA context)
          for (cudaEvent_t e : {s->marked, s->noted[0], s->noted[1]}) cudaEventDestroy(e);
          cudaStreamDestroy(s->stream);
        }
    }
  };
  static thread_local std::vector<std::unique_ptr<Streams>> of;
  static thread_local uint64_t uses = 0;
  const int device = c10::cuda::current_device();
  if ((size_t)device >= of.size()) of.resize(device + 1);
  if (!of[device]) of[device] = std::make_unique<Streams>();
  auto* const slots = of[device]->slots;
  auto* slot = &slots[0];
  for (auto* s = slots; s != slots + 4; ++s) {
    if (s->side && s->beside == current) {
      slot = s;
      break;
    }
    if (s->used < slot->used) slot = s;              // (never used: 0)
  }
  if (!slot->side) {
    cudaStream_t raw = nullptr;
    cudaEvent_t e[3] = {};
    bool made = cudaStreamCreateWithFlags(&raw, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t& ev : e) made = made && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess;
    if (!made) {
      for (cudaEvent_t ev : e)
        if (ev != nullptr) cudaEventDestroy(ev);
      if (raw != nullptr) cudaStreamDestroy(raw);
      cudaGetLastError();
      return nullptr;
    }
    slot->side.reset(new SideStream{c10::cuda::getStreamFromExternal(raw, (c10::DeviceIndex)device), e[0], {e[1], e[2]}});
  }
  cudaStreamCaptureStatus here = cudaStreamCaptureStatusNone, there = here;
  unsigned long long here_id = 0, there_id = 0;
  if (cudaStreamGetCaptureInfo(current, &here, &here_id) != cudaSuccess || cudaStreamGetCaptureInfo(slot->side->stream, &there, &there_id) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (there != cudaStreamCaptureStatusNone && (there != here || there_id != here_id)) return nullptr;
  slot->beside = current;
  slot->used = ++uses;
  return slot->side.get();
}

// Where a layer's weight gradients are added (fp32).
struct LayerGrads {
  float *qkv, *o, *gu, *d;
  const Tensor *ln1, *ln2;
};
// The regions of the nine parameters from mg[first] on; false unless they are as the launches take them.
bool layer_grads(const LayerDims& n, const std::vector<Tensor>& mg, size_t first, LayerGrads& g) {
  g.qkv = packed_region(mg, (int)first, 3, n.Q(), n.H);
  g.o = packed_region(mg, (int)first + 3, 1, n.H, n.O());
  g.gu = packed_region(mg, (int)first + 4, 2, 2 * n.I, n.H);
  g.d = packed_region(mg, (int)first + 6, 1, n.H, n.I);
  if (g.qkv == nullptr || g.o == nullptr || g.gu == nullptr || g.d == nullptr) return false;
  for (size_t i = first + 7; i < first + 9; ++i)
    if (!mg[i].is_cuda() || mg[i].scalar_type() != at::kFloat || !mg[i].is_contiguous() || mg[i].numel() != n.H) return false;
  g.ln1 = &mg[first + 7];
  g.ln2 = &mg[first + 8];
  return true;
}

// Scratch of a layer's backward (bytes): dgu, whose place the attention's gradients take when it is done with, or, beside a second stream that may
// still read it, not; the normed inputs' gradients (dh); dx_mid.
struct LayerScratch {
  int64_t dO, dqkv, dq, delta, dh, dx_mid, total;
  LayerScratch(const LayerDims& n, bool two_streams) {
    auto up = [](int64_t bytes) { return (bytes + 255) / 256 * 256; };
    const int64_t T = n.T(), b_h = up(2 * T * n.H), b_dgu = up(4 * T * n.I);
    dO = two_streams ? b_dgu : 0;
    dqkv = dO + up(2 * T * n.O());
    dq = dqkv + up(2 * T * n.Q());
    delta = dq + up(4 * T * n.O());
    dh = std::max(b_dgu, delta + up(4 * T * n.hq));
    dx_mid = dh + b_h;
    total = dx_mid + b_h;
  }
};

// The launches of a layer's backward. x: the forward's input; ln1, ln2: the norms' weights; s: LayerScratch bytes.
void layer_bwd_launches(const LayerDims& n, const void* dout, const void* x, const LayerActivations& acts, const LayerPointers& w, const Tensor& ln1,
                        const Tensor& ln2, const LayerGrads& g, char* const s, void* dx, double scale, const at::TensorOptions& on, SideStream* side = nullptr) {
  const LayerScratch at(n, side != nullptr);
  const int64_t T = n.T(), H = n.H, I = n.I, O = n.O(), Q = n.Q(), B = n.B, S = n.S, hq = n.hq, hkv = n.hkv, d = n.d;
  const bf16_t *const h1 = acts.h1, *const qkv = acts.qkv, *const o = acts.o, *const x_mid = acts.x_mid, *const h2 = acts.h2,
               *const gu = acts.gu, *const a = acts.a;
  void *const dgu = s, *const dO = s + at.dO, *const dq_ws = s + at.dq, *const delta = s + at.delta;
  bf16_t* const dqkv = reinterpret_cast<bf16_t*>(s + at.dqkv);
  void *const dh = s + at.dh, *const dx_mid = s + at.dx_mid;
  const cudaStream_t st = stream();
  // The weight gradients are nobody's input: on a stream beside the layer's own they fill the SMs that its kernels leave idle. Each is given to the
  // device after the kernel of the layer that needs the same gradient, so that the layer's goes first.
  auto mark = [&] {
    if (side != nullptr) side->mark(st);
  };
  auto weight_grad = [&](auto launch) {
    if (side == nullptr) return launch();
    side->go();
    const c10::cuda::CUDAStreamGuard on_side(side->stream);
    launch();
  };

  mark();
  if (!(pt_gemm_get_pair() && I % 64 == 0 &&
        fused_gemm(pt_gemm_bf16_fused(dout, w.wd, dgu, (int)T, (int)I, (int)H, H, w.ld_d, 2 * I, 5, const_cast<bf16_t*>(gu), 2 * I,
                                      (int)I, nullptr, nullptr, 0, 0, 0, pt_status_word(), st), "gemm_dgrad_swiglu_bwd"))) {
    Tensor da = torch::empty({T, I}, on);
    gemm_into(dout, w.wd, da.data_ptr(), T, I, H, H, w.ld_d, I, false, true, 0, on);
    PT_CHECK_RC(pt_swiglu_bwd(gu, da.data_ptr(), dgu, T, (int)I, st), "swiglu_bwd");
  }
  weight_grad([&] { gemm_into(dout, a, g.d, H, I, T, H, I, I, true, true, 1, on); });
  mark();
  gemm_into(dgu, w.w_gu, dh, T, H, 2 * I, 2 * I, w.ld_gu, H, false, true, 0, on);
  weight_grad([&] { gemm_into(dgu, h2, g.gu, 2 * I, H, T, 2 * I, H, H, true, true, 1, on); });
  rmsnorm_bwd_into(dh, x_mid, ln2, acts.rstd2, dout, dx_mid, *g.ln2, T, H, on);
  mark();
  gemm_into(dx_mid, w.wo, dO, T, O, H, H, w.ld_o, O, false, true, 0, on);             // dL/d(attention output)
  PT_CHECK_BWD_RC(pt_attention_bwd_rope(dO, qkv, qkv + O, qkv + O + hkv * d, o, acts.lse, nullptr, reinterpret_cast<float*>(delta),
                                        reinterpret_cast<float*>(dq_ws), dqkv, dqkv + O, dqkv + O + hkv * d, (int)B, (int)S, (int)S, (int)hq,
                                        (int)hkv, (int)d, Q, Q, Q, Q, Q, Q, 1, (float)scale, w.cosp, w.sinp, (int)S, st), "attention_bwd");
  weight_grad([&] { gemm_into(dx_mid, o, g.o, H, O, T, H, O, O, true, true, 1, on); });
  mark();
  gemm_into(dqkv, w.w_qkv, dh, T, H, Q, Q, w.ld_qkv, H, false, true, 0, on);
  weight_grad([&] { gemm_into(dqkv, h1, g.qkv, Q, H, T, Q, H, H, true, true, 1, on); });
  rmsnorm_bwd_into(dh, x, ln1, acts.rstd1, dx_mid, dx, *g.ln1, T, H, on);
}

LayerActivations saved_activations(const LayerDims& n, const Tensor& s16, const Tensor& s32) {
  const LayerSaved at(n);
  const bf16_t* const b = bf16_ptr(s16);
  const float* const f = s32.data_ptr<float>();
  return LayerActivations{b + at.h1, b + at.qkv, b + at.o, b + at.x_mid, b + at.h2, b + at.gu, b + at.a, f + at.rstd1, f + at.rstd2, f + at.lse};
}

// Backward of a layer; the weight gradients are added to the fp32 regions `mg` (q, k, v, out, gate, up, down, norm 1, norm 2). x: the
// forward's input; `saved_by(dims)` gives its activations once the dimensions are known. Returns dx, or an undefined tensor (nothing
// launched).
template <class SavedBy>
Tensor layer_bwd(const Tensor& dout, const Tensor& x, SavedBy saved_by, const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT,
                 const Tensor& sinT, const Tensor& wo, const Tensor& ln2, const Tensor& w_gu, const Tensor& wd, const std::vector<Tensor>& mg,
                 int64_t B, int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale) {
  TORCH_CHECK(mg.size() == 9);
  if (!all_bf16_cuda({&dout, &x, &ln1, &w_qkv, &wo, &ln2, &w_gu, &wd})) return Tensor();
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous() && x.size(0) == B * S && dout.is_contiguous() && dout.sizes() == x.sizes() &&
              w_gu.dim() == 2 && hq % hkv == 0);
  const LayerDims n{B, S, x.size(1), w_gu.size(0) / 2, hq, hkv, d};
  LayerGrads g;
  if (!layer_grads(n, mg, 0, g)) return Tensor();
  check_layer(n, ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd);
  const LayerActivations acts = saved_by(n);
  c10::cuda::CUDAGuard guard(x.device());
  const auto on = x.options();
  Tensor scratch = torch::empty({LayerScratch(n, false).total}, on.dtype(at::kByte)), dx = torch::empty({n.T(), n.H}, on);
  layer_bwd_launches(n, dout.data_ptr(), x.data_ptr(), acts, layer_pointers(ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd), ln1, ln2, g,
                     reinterpret_cast<char*>(scratch.data_ptr()), dx.data_ptr(), scale, on);
  return dx;
}

// Backward of decoder_stack_fwd (with save): xs, s16, s32 are the layers' inputs and saved activations, mg the fp32 regions of `params`.
// Returns dx, or an undefined tensor (nothing launched).
Tensor decoder_stack_bwd(const Tensor& dout, const std::vector<Tensor>& xs, const std::vector<Tensor>& s16, const std::vector<Tensor>& s32,
                         const std::vector<Tensor>& params, const std::vector<Tensor>& tables, const std::vector<Tensor>& mg, int64_t B, int64_t S,
                         int64_t hq, int64_t hkv, int64_t d, double scale) {
  const size_t layers = xs.size();
  if (layers == 0 || !all_bf16_cuda({&dout}) || dout.dim() != 2 || !dout.is_contiguous() || dout.size(0) != B * S || dout.size(0) == 0 || hq % hkv ||
      s16.size() != layers || s32.size() != layers || mg.size() != params.size())
    return Tensor();
  const LayerDims n = stack_dims(dout, params, B, S, hq, hkv, d);
  const auto w = stack_pointers(n, dout, params, tables);
  if (w.size() != layers) return Tensor();
  const LayerSaved at(n);
  std::vector<LayerGrads> g(layers);
  for (size_t i = 0; i < layers; ++i) {
    if (!layer_grads(n, mg, i * LAYER_PARAMS, g[i])) return Tensor();
    for (const Tensor* t : {&xs[i], &s16[i], &s32[i]})
      if (t->device() != dout.device() || !t->is_contiguous() || t->scalar_type() != (t == &s32[i] ? at::kFloat : at::kBFloat16)) return Tensor();
    if (xs[i].sizes() != dout.sizes() || s16[i].numel() != at.total || s32[i].numel() != at.total32) return Tensor();
  }
  c10::cuda::CUDAGuard guard(dout.device());
  const auto on = dout.options();
  // Two streams where a layer keeps the device busier than the host (8 us a layer for the second): at least 12 GFLOP. Passes in turn, 12 to 24 pairs,
  // us one / two and the middle half of the gains: 16 layers of the 135M shape, 3 x 601 tokens 3,323 / 3,129 (6.1 to 6.3 %), 8 x 1024 8,044 / 7,939
  // (1.0 to 1.7); 16 of the 360M shape, 4 x 1024 7,972 / 7,671 (3.3 to 4.5); 5 layers of the 1.7B shape, 2 x 4 x 128 4,620 / 4,503 (2.2 to 3.1), 15
  // layers, 4 x 1024 27,493 / 26,929 (1.4 to 2.7; on another box 0.1 to 2.0); 4 of the 7B shape, 1 x 1024 6,693 / 6,522 (1.4 to 3.0), 4 x 1024 21,323 /
  // 21,005 (0.8 to 2.3); no difference beyond what the power cap does from run to run at 3 of the 8B shape, 8192 tokens 55,321 / 55,412 (-1.0 to 0.6)
  // and 4 of the 1B shape, 32768 tokens 173,197 / 172,975 (-1.4 to 2.0). 2 layers of width 512, 512 tokens lose: 795 / 817.
  const double gflop = 4e-9 * n.T() * (double)(n.H * (n.Q() + n.O() + 3 * n.I));
  const cudaStream_t st = stream();
  SideStream* side = gflop >= 12 ? side_stream(st) : nullptr;
  // The second stream may be a layer behind, so layers take two scratch areas in turn (up to 1 GB for both) and a layer's incoming gradient is kept
  // for one layer more; a larger one is used again as soon as the second stream is done with it. One stream needs the least: where the device is
  // too full for more, it has to do.
  int64_t bytes = LayerScratch(n, side != nullptr).total;
  bool late = side != nullptr && layers > 1 && bytes <= (512 << 20);
  Tensor scratch, grad = dout, kept[2];
  try {
    scratch = torch::empty({late ? 2 * bytes : bytes}, on.dtype(at::kByte));
  } catch (const c10::OutOfMemoryError&) {
    if (side == nullptr) throw;
    side = nullptr;
    late = false;
    bytes = LayerScratch(n, false).total;
    scratch = torch::empty({bytes}, on.dtype(at::kByte));
  }
  struct Joined {                                                        // whatever happens, memory is not given back before it is done with
    SideStream* side;
    cudaStream_t st;
    ~Joined() {
      if (side == nullptr) return;
      cudaEventRecord(side->noted[0], side->stream);
      cudaStreamWaitEvent(st, side->noted[0], 0);
    }
  } joined{side, st};
  const Chain chain;
  for (size_t i = layers; i-- > 0;) {
    if (late && i + 2 < layers) {
      side->join(st, (int)i);                                            // (what layer i + 2 noted)
      kept[i & 1] = Tensor();
    }
    Tensor dx = torch::empty({n.T(), n.H}, on);
    layer_bwd_launches(n, grad.data_ptr(), xs[i].data_ptr(), saved_activations(n, s16[i], s32[i]), w[i], params[i * LAYER_PARAMS + 7],
                       params[i * LAYER_PARAMS + 8], g[i], reinterpret_cast<char*>(scratch.data_ptr()) + (late ? (int64_t)(i & 1) * bytes : 0),
                       dx.data_ptr(), scale, on, side);
    if (side != nullptr) {
      side->done((int)i);
      if (late) kept[i & 1] = grad;
      else side->join(st, (int)i);
    }
    grad = dx;
  }
  return grad;
}

// `s16`, `s32`: what decoder_layer_fwd_packed saved.
Tensor decoder_layer_bwd_packed(const Tensor& dout, const Tensor& x, const Tensor& s16, const Tensor& s32, const Tensor& ln1, const Tensor& w_qkv,
                                const Tensor& cosT, const Tensor& sinT, const Tensor& wo, const Tensor& ln2, const Tensor& w_gu,
                                const Tensor& wd, const std::vector<Tensor>& mg, int64_t B, int64_t S, int64_t hq, int64_t hkv, int64_t d,
                                double scale) {
  if (!all_bf16_cuda({&s16})) return Tensor();
  auto saved_by = [&](const LayerDims& n) {
    const LayerSaved at(n);
    PT_CHECK_F32(s32);
    TORCH_CHECK(s16.is_contiguous() && s16.numel() == at.total && s32.is_contiguous() && s32.numel() == at.total32,
                "decoder layer: saved activations of another shape");
    return saved_activations(n, s16, s32);
  };
  return layer_bwd(dout, x, saved_by, ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd, mg, B, S, hq, hkv, d, scale);
}

// `saved` = {x, rstd1, h1, qkv, o, lse, x_mid, rstd2, h2, gu, a}, tensors wherever they lie.
Tensor decoder_layer_bwd(const Tensor& dout, const std::vector<Tensor>& saved, const Tensor& ln1, const Tensor& w_qkv, const Tensor& cosT,
                         const Tensor& sinT, const Tensor& wo, const Tensor& ln2, const Tensor& w_gu, const Tensor& wd,
                         const std::vector<Tensor>& mg, int64_t B, int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale) {
  TORCH_CHECK(saved.size() == 11);
  auto saved_by = [&](const LayerDims& n) {
    auto bf16 = [&](int i, int64_t cols) {
      PT_CHECK_BF16(saved[i]);
      TORCH_CHECK(saved[i].is_contiguous() && saved[i].numel() == n.T() * cols, "decoder layer: saved activation ", i, " of another shape");
      return (const bf16_t*)bf16_ptr(saved[i]);
    };
    auto f32 = [&](int i, int64_t cols) {
      PT_CHECK_F32(saved[i]);
      TORCH_CHECK(saved[i].is_contiguous() && saved[i].numel() == n.T() * cols, "decoder layer: saved statistic ", i, " of another shape");
      return (const float*)saved[i].data_ptr<float>();
    };
    return LayerActivations{bf16(2, n.H), bf16(3, n.Q()), bf16(4, n.O()), bf16(6, n.H), bf16(8, n.H), bf16(9, 2 * n.I), bf16(10, n.I),
                            f32(1, 1), f32(7, 1), f32(5, n.hq)};
  };
  return layer_bwd(dout, saved[0], saved_by, ln1, w_qkv, cosT, sinT, wo, ln2, w_gu, wd, mg, B, S, hq, hkv, d, scale);
}

void allreduce_symm(std::vector<int64_t> buf_ptrs, std::vector<int64_t> flag_ptrs, int64_t mc_ptr, int64_t offset_elems,
                    int64_t n, bool is_bf16, double scale, int64_t rank, int64_t world, int64_t num_blocks,
                    int64_t staging_off_bytes) {
  TORCH_CHECK((int64_t)buf_ptrs.size() == world && (int64_t)flag_ptrs.size() == world && world <= 8);
  void* b[8]; void* f[8];
  for (int i = 0; i < world; ++i) { b[i] = reinterpret_cast<void*>(buf_ptrs[i]); f[i] = reinterpret_cast<void*>(flag_ptrs[i]); }
  PT_CHECK_RC(pt_allreduce_symm(b, f, reinterpret_cast<void*>(mc_ptr), offset_elems, n, is_bf16 ? 1 : 0, (float)scale,
                                (int)rank, (int)world, (int)num_blocks, staging_off_bytes, stream()), "allreduce_symm");
}

// Attention of local queries over K/V segments given by raw (possibly peer-mapped) pointers: segment i is a
// [B, Sk, hkv, d] bf16 tensor with token stride kv_row at k_ptrs[i] / v_ptrs[i]; causal masks inside the last segment.
std::vector<Tensor> attention_fwd_segs(const Tensor& q, std::vector<int64_t> k_ptrs, std::vector<int64_t> v_ptrs, int64_t Sk,
                                       int64_t hkv, int64_t kv_row, bool causal, double scale) {
  PT_CHECK_BF16(q);
  const int B = (int)q.size(0), Sq = (int)q.size(1), hq = (int)q.size(2), d = (int)q.size(3);
  const int n = (int)k_ptrs.size();
  TORCH_CHECK(n >= 1 && n <= 8 && (int)v_ptrs.size() == n);
  c10::cuda::CUDAGuard guard(q.device());
  const void* kp[8]; const void* vp[8];
  for (int i = 0; i < n; ++i) { kp[i] = reinterpret_cast<const void*>(k_ptrs[i]); vp[i] = reinterpret_cast<const void*>(v_ptrs[i]); }
  auto o = torch::empty({B, Sq, hq, d}, q.options());
  auto lse = torch::empty({B, hq, Sq}, q.options().dtype(at::kFloat));
  PT_CHECK_RC(pt_attention_fwd_segs(q.data_ptr(), kp, vp, n, o.data_ptr(), lse.data_ptr<float>(), B, Sq, (int)Sk, hq, (int)hkv,
                                    d, token_stride(q, "q"), kv_row, kv_row, causal ? 1 : 0, (float)scale, stream()),
              "attention_fwd_segs");
  return {o, lse};
}

// Backward of attention_fwd_segs. Returns dq (bf16, contiguous). The fp32 dk/dv partials of segment i are written to
// partial_ptr + i*seg_stride (dk) and + i*seg_stride + B*Sk*hkv*d (dv), token stride hkv*d.
Tensor attention_bwd_segs(const Tensor& dout, const Tensor& q, std::vector<int64_t> k_ptrs, std::vector<int64_t> v_ptrs,
                          int64_t Sk, int64_t hkv, int64_t kv_row, const Tensor& o, const Tensor& lse,
                          const c10::optional<Tensor>& delta, int64_t partial_ptr, int64_t seg_stride, bool causal,
                          double scale) {
  PT_CHECK_BF16(dout); PT_CHECK_BF16(q); PT_CHECK_BF16(o); PT_CHECK_F32(lse);
  if (delta.has_value()) { PT_CHECK_F32(*delta); }
  const int B = (int)q.size(0), Sq = (int)q.size(1), hq = (int)q.size(2), d = (int)q.size(3);
  const int n = (int)k_ptrs.size();
  TORCH_CHECK(n >= 1 && n <= 8 && (int)v_ptrs.size() == n && dout.is_contiguous() && o.is_contiguous());
  c10::cuda::CUDAGuard guard(q.device());
  const void* kp[8]; const void* vp[8];
  for (int i = 0; i < n; ++i) { kp[i] = reinterpret_cast<const void*>(k_ptrs[i]); vp[i] = reinterpret_cast<const void*>(v_ptrs[i]); }
  auto dq = torch::empty({B, Sq, hq, d}, q.options());
  const auto f32 = q.options().dtype(at::kFloat);
  auto dq_ws = delta.has_value() ? torch::zeros({B, Sq, hq, d}, f32) : torch::empty({B, Sq, hq, d}, f32);
  auto delta_ws = torch::empty({B, hq, Sq}, q.options().dtype(at::kFloat));
  float* part = reinterpret_cast<float*>(partial_ptr);
  const long long per = (long long)B * Sk * hkv * d;
  PT_CHECK_BWD_RC(pt_attention_bwd_segs(dout.data_ptr(), q.data_ptr(), kp, vp, n, o.data_ptr(), lse.data_ptr<float>(),
                                    delta.has_value() ? delta->data_ptr<float>() : nullptr, delta_ws.data_ptr<float>(),
                                    dq_ws.data_ptr<float>(), dq.data_ptr(), part, part + per,
                                    1, seg_stride, B, Sq, (int)Sk, hq, (int)hkv, d, token_stride(q, "q"), kv_row, kv_row,
                                    (long long)hq * d, (long long)hkv * d, (long long)hkv * d, causal ? 1 : 0, (float)scale,
                                    stream()), "attention_bwd_segs");
  return dq;
}

// out (2-D bf16 inside the symmetric data region, element offset d_offset) = sum over ranks of op(a) op(b)
void gemm_allreduce(const Tensor& a, const Tensor& b, bool trans_a, bool trans_b, Tensor& out, std::vector<int64_t> buf_ptrs,
                    std::vector<int64_t> flag_ptrs, int64_t mc_ptr, int64_t d_offset, int64_t rank, int64_t world,
                    int64_t clusters_cap) {
  PT_CHECK_BF16(a); PT_CHECK_BF16(b); PT_CHECK_BF16(out);
  const long long lda = row_stride_2d(a, "a"), ldb = row_stride_2d(b, "b"), ldd = row_stride_2d(out, "out");
  const int64_t M = trans_a ? a.size(1) : a.size(0), K = trans_a ? a.size(0) : a.size(1);
  const int64_t N = trans_b ? b.size(1) : b.size(0), Kb = trans_b ? b.size(0) : b.size(1);
  TORCH_CHECK(K == Kb && out.size(0) == M && out.size(1) == N, "gemm_allreduce: shape mismatch");
  TORCH_CHECK((int64_t)buf_ptrs.size() == world && (int64_t)flag_ptrs.size() == world && world <= 8);
  c10::cuda::CUDAGuard guard(a.device());
  void* bp[8]; void* fp[8];
  for (int i = 0; i < world; ++i) { bp[i] = reinterpret_cast<void*>(buf_ptrs[i]); fp[i] = reinterpret_cast<void*>(flag_ptrs[i]); }
  const int rc = pt_gemm_allreduce_bf16(a.data_ptr(), b.data_ptr(), bp, fp, reinterpret_cast<void*>(mc_ptr), d_offset, (int)M, (int)N, (int)K, lda, ldb, ldd,
                                        trans_a ? 1 : 0, trans_b ? 1 : 0, (int)rank, (int)world,
                                        (int)clusters_cap, stream());
  TORCH_CHECK(rc == 0, "gemm_allreduce failed with code ", rc, " (M=", M, " N=", N, " K=", K, ")");
}

// number of CTA pairs of the fused GEMM+all-reduce kernel that fit on the current device
int64_t gemm_allreduce_max_clusters() {
  static const uint16_t dummy[64] = {0};
  void* none[1] = {nullptr};
  const int rc = pt_gemm_allreduce_bf16(dummy, dummy, none, none, nullptr, 0, 256, 256, 64, 64, 64, 256, 0, 0, 0, 1, 0, stream());
  return rc;
}

void symm_barrier(std::vector<int64_t> flag_ptrs, int64_t rank, int64_t world) {
  TORCH_CHECK((int64_t)flag_ptrs.size() == world && world <= 8);
  void* f[8];
  for (int i = 0; i < world; ++i) f[i] = reinterpret_cast<void*>(flag_ptrs[i]);
  PT_CHECK_RC(pt_symm_barrier(f, (int)rank, (int)world, stream()), "symm_barrier");
}

void reduce_dkv_symm(std::vector<int64_t> buf_ptrs, int64_t offset_elems, int64_t me, int64_t world, Tensor& dk, Tensor& dv) {
  PT_CHECK_BF16(dk); PT_CHECK_BF16(dv);
  TORCH_CHECK((int64_t)buf_ptrs.size() == world && world <= 8 && dk.dim() == 4 && dk.sizes() == dv.sizes());
  c10::cuda::CUDAGuard guard(dk.device());
  void* b[8];
  for (int i = 0; i < world; ++i) b[i] = reinterpret_cast<void*>(buf_ptrs[i]);
  const long long tokens = dk.size(0) * dk.size(1);
  const int width = (int)(dk.size(2) * dk.size(3));
  PT_CHECK_RC(pt_reduce_dkv_symm(b, offset_elems, (int)me, (int)world, tokens, width, dk.data_ptr(), dv.data_ptr(),
                                 token_stride(dk, "dk"), token_stride(dv, "dv"), stream()), "reduce_dkv_symm");
}

// out[T, H] (bf16): row ids[t] of a vocabulary-parallel embedding whose shards ([rows_per_rank, H] each) are at shard_ptrs
Tensor embedding_gather_peers(const Tensor& ids, std::vector<int64_t> shard_ptrs, int64_t rows_per_rank, int64_t H, const Tensor& like) {
  PT_CHECK_BF16(like);
  TORCH_CHECK(ids.is_cuda() && ids.scalar_type() == at::kLong && ids.is_contiguous() && shard_ptrs.size() >= 1 && shard_ptrs.size() <= 8);
  c10::cuda::CUDAGuard guard(like.device());
  void* b[8];
  for (size_t i = 0; i < shard_ptrs.size(); ++i) b[i] = reinterpret_cast<void*>(shard_ptrs[i]);
  auto out = torch::empty({ids.numel(), H}, like.options());
  PT_CHECK_RC(pt_embedding_gather_peers((const long long*)ids.data_ptr<int64_t>(), b, (int)shard_ptrs.size(), rows_per_rank,
                                        ids.numel(), (int)H, out.data_ptr(), stream()), "embedding_gather_peers");
  return out;
}

// {lse, target_logit} of n rows from the per-shard statistics every rank of the group left at `offset_bytes` of its buffer
std::vector<Tensor> ce_stats_combine_peers(std::vector<int64_t> buf_ptrs, int64_t offset_bytes, int64_t n, const Tensor& like) {
  TORCH_CHECK(buf_ptrs.size() >= 1 && buf_ptrs.size() <= 8 && like.is_cuda());
  c10::cuda::CUDAGuard guard(like.device());
  void* b[8];
  for (size_t i = 0; i < buf_ptrs.size(); ++i) b[i] = reinterpret_cast<void*>(buf_ptrs[i]);
  auto f = like.options().dtype(at::kFloat);
  auto lse = torch::empty({n}, f), tgt = torch::empty({n}, f);
  PT_CHECK_RC(pt_ce_stats_combine_peers(b, offset_bytes, (int)buf_ptrs.size(), n, lse.data_ptr<float>(), tgt.data_ptr<float>(),
                                        stream()), "ce_stats_combine_peers");
  return {lse, tgt};
}

// dst (contiguous, n blocks of bytes_each) <- the blocks at src_ptrs (raw, possibly peer-mapped device pointers)
void gather_peer(Tensor& dst, std::vector<int64_t> src_ptrs, int64_t bytes_each) {
  TORCH_CHECK(dst.is_cuda() && dst.is_contiguous() && src_ptrs.size() <= 8);
  TORCH_CHECK((int64_t)(dst.numel() * dst.element_size()) >= bytes_each * (int64_t)src_ptrs.size(), "gather_peer: dst too small");
  c10::cuda::CUDAGuard guard(dst.device());
  const void* p[8];
  for (size_t i = 0; i < src_ptrs.size(); ++i) p[i] = reinterpret_cast<const void*>(src_ptrs[i]);
  PT_CHECK_RC(pt_gather_peer(dst.data_ptr(), p, (int)src_ptrs.size(), bytes_each, stream()), "gather_peer");
}

int64_t kernel_status() { return (int64_t)pt_kernel_status_fetch_and_clear(); }
int64_t launch_count() { return (int64_t)pt_launch_count(); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("rmsnorm_fwd", &rmsnorm_fwd);
  m.def("add_rmsnorm_fwd", &add_rmsnorm_fwd);
  m.def("rmsnorm_bwd", &rmsnorm_bwd, py::arg("dy"), py::arg("x"), py::arg("w"), py::arg("rstd"), py::arg("dres") = py::none(),
        py::arg("dw_acc") = py::none());
  m.def("rope_", &rope_);
  m.def("swiglu_fwd", &swiglu_fwd);
  m.def("swiglu_bwd", &swiglu_bwd);
  m.def("gemm", &gemm, py::arg("a"), py::arg("b"), py::arg("trans_a"), py::arg("trans_b"), py::arg("out") = py::none(),
        py::arg("accumulate") = false);
  m.def("gemm_swiglu", &gemm_swiglu, "x w_gu^T with the SwiGLU activation fused into the GEMM epilogue: returns [gu, h] or [].");
  m.def("gemm_rope", &gemm_rope, "x w_qkv^T with RoPE of the first n_rot heads fused into the GEMM epilogue (None if not covered).");
  m.def("gemm_add", &gemm_add, "x w^T + res with the residual add fused into the GEMM epilogue (None if not covered).");
  m.def("gemm_dgrad_swiglu_bwd", &gemm_dgrad_swiglu_bwd,
        "SwiGLU backward fused into the epilogue of the down-projection dgrad GEMM: returns the packed [T, 2I] gradient (None if not covered).");
  m.def("embedding_fwd", &embedding_fwd);
  m.def("embedding_bwd", &embedding_bwd);
  m.def("ce_stats", &ce_stats);
  m.def("gemm_ce_loss", &gemm_ce_loss,
        "LM-head GEMM + cross entropy: loss terms into `terms`, gradient of the logits returned (None if not covered).");
  m.def("gemm_ce_stats", &gemm_ce_stats,
        "LM-head GEMM whose epilogue also produces the cross-entropy row statistics: [logits, rowmax, sumexp, target_logit] or [].");
  m.def("ce_grad_", &ce_grad_);
  m.def("accumulate_", &accumulate_);
  m.def("add", &add);
  m.def("adamw_multi_", &adamw_multi_);
  m.def("decoder_layer_fwd", &decoder_layer_fwd);
  m.def("decoder_layer_bwd", &decoder_layer_bwd);
  m.def("decoder_layer_fwd_packed", &decoder_layer_fwd_packed, "decoder_layer_fwd with the saved activations in two allocations.");
  m.def("decoder_layer_saved", &decoder_layer_saved, "The saved activations of decoder_layer_fwd_packed as tensors (views).");
  m.def("decoder_layer_bwd_packed", &decoder_layer_bwd_packed);
  m.def("decoder_stack_fwd", &decoder_stack_fwd, "All layers' forward in one call; [] where an operand is not as it has to be.");
  m.def("decoder_stack_bwd", [](const Tensor& dout, const std::vector<Tensor>& xs, const std::vector<Tensor>& s16, const std::vector<Tensor>& s32,
                                const std::vector<Tensor>& params, const std::vector<Tensor>& tables, const std::vector<Tensor>& mg, int64_t B,
                                int64_t S, int64_t hq, int64_t hkv, int64_t d, double scale) -> c10::optional<Tensor> {
    Tensor dx = decoder_stack_bwd(dout, xs, s16, s32, params, tables, mg, B, S, hq, hkv, d, scale);
    return dx.defined() ? c10::optional<Tensor>(dx) : c10::nullopt;
  }, "All layers' backward in one call; None where an operand is not as it has to be.");
  m.def("scale_", &scale_);
  m.def("merge_attention_", &merge_attention_);
  m.def("attention_fwd", &attention_fwd);
  m.def("attention_bwd", &attention_bwd, py::arg("dout"), py::arg("q"), py::arg("k"), py::arg("v"), py::arg("o"),
        py::arg("lse"), py::arg("causal"), py::arg("scale"), py::arg("delta") = py::none(), py::arg("outs") = py::none(),
        py::arg("rope_cos") = py::none(), py::arg("rope_sin") = py::none());
  m.def("set_gemm_pair", [](bool on) { pt_gemm_set_pair(on ? 1 : 0); },
        "Use 256x256 tiles on CTA pairs (tcgen05 cta_group::2) for GEMMs (default) or 128x256 single-CTA tiles.");
  m.def("get_gemm_pair", []() { return pt_gemm_get_pair() != 0; });
  m.def("set_gemm_tma_epilogue", [](bool on) { pt_gemm_set_tma_epilogue(on ? 1 : 0); },
        "CTA-pair GEMM epilogue through shared memory and TMA store / reduce-add (default) or per-thread 16-byte stores.");
  m.def("get_gemm_tma_epilogue", []() { return pt_gemm_get_tma_epilogue() != 0; });
  m.def("set_gemm_group_m", [](int64_t g) { pt_gemm_set_group_m((int)g); },
        "CTA-pair GEMM tile numbering: rows of 256-row tiles per group (L2 locality of concurrently running tiles; default 8).");
  m.def("set_gemm_split_dgrad", [](bool on) { pt_gemm_set_split_k(on ? 1 : 0); },
        "GEMMs with few output tiles (forward, with a residual, input and weight gradients): K split over idle CTA pairs (default on; for the "
         "calling thread)");
  m.def("set_gemm_split_parts", [](int64_t n) { pt_gemm_set_split_k(n > 1 ? (int)n : 1); },
        "GEMMs that may be split over K are always cut into n parts by this thread (tests, measurements); 0 or 1: the rule.");
  m.def("set_gemm_cluster", [](int64_t n) { pt_gemm_set_cluster((int)n); },
        "GEMMs X W^T (+ residual) and dY W share K between the pairs of a cluster: 0 by the rule, 1 never, 2 wherever it can be (this thread).");
  m.def("gemm_plan", [](const std::string& kind, int64_t M, int64_t N, int64_t K) {
          const int splits = kind == "dgrad" ? 0 : kind == "wgrad" ? 1 : kind == "fwd" || kind == "add" ? 2 : -1;
          TORCH_CHECK(splits >= 0 || kind == "rope" || kind == "swiglu" || kind == "swiglu_bwd", "gemm_plan: ", kind);
          int tile_n = 256;
          const int parts = splits >= 0 ? pt_gemm_parts((int)M, (int)N, (int)K, splits, kind == "add", &tile_n) : 1;
          if (parts < 0) return std::pair<int64_t, int64_t>(128, -2);
          if (parts <= 1) tile_n = pt_gemm_tile_columns((int)M, (int)N, (int)K, splits == 1, splits == 0 || splits == 1 || kind == "swiglu_bwd",
                                                       splits >= 0 || kind == "swiglu_bwd");
          return std::pair<int64_t, int64_t>(tile_n, parts);
        }, "(columns of a tile, parts of K) that the rule gives a GEMM with output [M, N]: kind fwd, add, dgrad, wgrad, rope, swiglu (N = 2I) or\n"
           "swiglu_bwd (N = I). (128, -2): K is shared by the two pairs of a cluster.");
  m.def("set_gemm_tile_n", [](int64_t n) { pt_gemm_set_tile_n((int)n); },
        "columns of the GEMM output tiles: 128, 192 (where the epilogue has it), 256, or 0 for the choice by shape (for the calling thread). "
         "With a given width K is not split, unless set_gemm_split_parts says so.");
  m.def("get_gemm_group_m", []() { return (int64_t)pt_gemm_get_group_m(); });
  m.def("attention_set_profile", [](const c10::optional<Tensor>& counters) {
          if (!counters.has_value()) { pt_attention_set_profile(nullptr); return; }
          TORCH_CHECK(counters->is_cuda() && counters->scalar_type() == at::kLong && counters->is_contiguous() &&
                      counters->numel() >= 16, "attention_set_profile: need a contiguous CUDA int64 tensor of >= 16 elements");
          pt_attention_set_profile(reinterpret_cast<unsigned long long*>(counters->data_ptr<int64_t>()));
        }, py::arg("counters") = py::none(),
        "Phase profiling of the attention kernels: later forward/backward launches add their per-phase SM-cycle counts to "
        "`counters` (layout in csrc/attention_tcgen05.cu); None switches it off. The caller keeps the tensor alive.");
  m.def("attention_set_clusters", [](int64_t largest) { pt_attention_set_clusters((int)largest); },
        "Largest cluster of CTAs that share a key block's query heads in the attention backward: 3 by default, 1: none (this thread).");
  m.def("attention_bwd_parts", [](int64_t B, int64_t Sq, int64_t Sk, int64_t hq, int64_t hkv, int64_t d, bool causal, int64_t n_segs, int64_t sms,
                                  int64_t pairs, int64_t triples) {
    return pt_attention_bwd_parts((int)B, (int)Sq, (int)Sk, (int)hq, (int)hkv, (int)d, causal, (int)n_segs, (int)sms, (int)pairs, (int)triples);
  }, "CTAs that share a key block's query heads in the attention backward of a device with `sms` SMs and room for `pairs` clusters of two\n"
     "or `triples` clusters of three CTAs.");
  m.def("attention_fwd_segs", &attention_fwd_segs);
  m.def("attention_bwd_segs", &attention_bwd_segs);
  m.def("gemm_allreduce", &gemm_allreduce,
        "GEMM whose output tiles are all-reduced over peer memory inside the same kernel (csrc/gemm_allreduce_tcgen05.cu).");
  m.def("gemm_allreduce_max_clusters", &gemm_allreduce_max_clusters);
  m.def("symm_barrier", &symm_barrier);
  m.def("reduce_dkv_symm", &reduce_dkv_symm);
  m.def("embedding_gather_peers", &embedding_gather_peers,
        "Vocabulary-parallel embedding lookup that reads every row from its owner's shard in symmetric memory (no reduction).");
  m.def("ce_stats_combine_peers", &ce_stats_combine_peers,
        "Vocabulary-parallel cross entropy: combine the per-shard (max, sum-exp, target logit) triples of all ranks (csrc/comm.cu).");
  m.def("gather_peer", &gather_peer, "Copy equally sized blocks out of peers' memory into one local buffer (csrc/comm.cu).");
  m.def("allreduce_symm", &allreduce_symm,
        "In-place all-reduce of a region of a symmetric buffer over peer memory (see csrc/comm.cu).");
  m.def("set_pdl", [](bool on) { pt_set_pdl(on ? 1 : 0); },
        "Programmatic dependent launch of the step's kernels (prologues overlap the previous kernel's tail); default on, "
        "PICOTRON_PDL=0 switches it off.");
  m.def("get_pdl", []() { return pt_pdl_enabled() != 0; });
  m.def("set_wait_limit_ns", [](int64_t ns) { pt_set_wait_limit_ns((unsigned long long)(ns > 0 ? ns : 0)); },
        "Limit (ns of the GPU global timer) of every cross-rank wait inside the peer-memory kernels; 0 restores the default (4 s). "
        "A wait that runs out makes the kernel return early and leaves a code in the status word (kernel_status).");
  m.def("get_wait_limit_ns", []() { return (int64_t)pt_get_wait_limit_ns(); });
  m.def("count_launches", [](int64_t n) { pt_count_launches((int)n); },
        "Add n to the launch counter (kernels replayed from a CUDA graph are launched without passing through this library).");
  m.def("launch_count", &launch_count, "Number of kernels this library has launched in this process.");
  m.def("kernel_status", &kernel_status,
        "Fetch-and-clear the device status word: 0 if no kernel gave up a bounded wait, else an encoded site.");
}
