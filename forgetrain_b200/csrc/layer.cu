// One decoder block per call: the launch sequence of the forward pass and of the two halves of the
// backward pass, without tensor parallelism. Host code only; every kernel is an entry point of its
// own that can also be called by itself (gemm_sm100.cu, attn_*.cu, elementwise.cu).
//
// Why: launched one by one from Python, an op costs its caller 24 us (argument checks, wrapping,
// allocation, stream look-up) and a 0.5B step of one micro-batch has 580 launches: 17 ms of host
// time for 9 ms of GPU work at 512 tokens, 6 ms with the blocks launched from here. That step 14.2 -> 8.1
// ms, the tiny model at 2 x 256 tokens 2.57 -> 0.85 ms, logits of 256 tokens 3.92 -> 1.69 ms.
//
// Structure mirrors exports/train_engine_0.5B/src/training_engine_tensor/forward.py:81-217 and
// backward.py:125-393 of the reference; the same sequence op by op, with the collectives of tensor
// parallelism, is MiniCPM4.layer_forward / layer_backward.
#include <cuda_runtime.h>
#include <stdint.h>

#include "layer.h"

extern "C" {
int ft_add_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, void*, int, int, float,
                       cudaStream_t);
int ft_rmsnorm_bwd(const void*, const void*, const void*, const void*, const void*, void*, void*,
                   void*, int, int, int, cudaStream_t);
int ft_rope(void*, const void*, const void*, const void*, long, int, int, int, int, int, int,
            cudaStream_t);
int ft_attn_fwd(const void*, void*, void*, int, int, int, int, int, int, int, float, int*,
                cudaStream_t);
int ft_attn_bwd(const void*, const void*, const void*, const void*, void*, void*, void*, int, int,
                int, int, int, int, int, int, float, int, const void*, const void*, const void*,
                int*, cudaStream_t);
int ft_gemm_bf16(const void*, const void*, void*, int, int, int, int, int, int, int, int, int, int,
                 float, int, int, int, int*, cudaStream_t);
int ft_gemm_swiglu_bf16(const void*, const void*, void*, void*, int, int, int, int, int, int, int,
                        float, int, int*, cudaStream_t);
int ft_gemm_swiglu_bwd_bf16(const void*, const void*, const void*, void*, int, int, int, int, int,
                            int, int, float, int, int*, cudaStream_t);
}

namespace {

#define FT_TRY(call)            \
  do {                          \
    const int rc_ = (call);     \
    if (rc_) return rc_;        \
  } while (0)

// y[T][N] = alpha * x[T][K] w[N][K]^T
int linear(const void* x, const void* w, void* y, int T, int N, int K, float alpha, int* status,
           cudaStream_t st) {
  return ft_gemm_bf16(x, w, y, T, N, K, K, K, N, 0, 0, 0, 0, alpha, 0, 0, 0, status, st);
}
// dx[T][K] = alpha * dy[T][N] w[N][K]
int dgrad(const void* dy, const void* w, void* dx, int T, int N, int K, float alpha, int* status,
          cudaStream_t st) {
  return ft_gemm_bf16(dy, w, dx, T, K, N, N, K, K, 0, 1, 0, 0, alpha, 0, 0, 0, status, st);
}

// Weight-gradient GEMMs on a stream of their own (or in line when there is none): each starts
// behind an event of the main stream, `join` makes the main stream wait for the last one issued.
// What they read may be freed once the main stream has been joined.
class SideStream {
 public:
  SideStream(cudaStream_t main, cudaStream_t side) : main_(main), side_(side) {}
  ~SideStream() { join(); }   // also on the way out of a call that failed half-way
  // dw[N][K] (+)= alpha * dy[T][N]^T x[T][K]
  int wgrad(const void* dy, const void* x, void* dw, int T, int N, int K, float alpha,
            int accumulate, int* status) {
    if (side_ != nullptr) FT_TRY(order(main_, side_));
    pending_ = side_ != nullptr;
    return ft_gemm_bf16(dy, x, dw, N, K, T, N, K, K, 1, 1, 1, accumulate, alpha, 0, 0, 0, status,
                        side_ != nullptr ? side_ : main_);
  }
  int join() {
    if (!pending_) return 0;
    pending_ = false;
    return order(side_, main_);
  }

 private:
  static int order(cudaStream_t first, cudaStream_t then) {
    cudaEvent_t ev;
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) return -11;
    const bool ok = cudaEventRecord(ev, first) == cudaSuccess &&
                    cudaStreamWaitEvent(then, ev, 0) == cudaSuccess;
    cudaEventDestroy(ev);   // released by the driver when the wait has passed
    return ok ? 0 : -11;
  }
  cudaStream_t main_, side_;
  bool pending_ = false;
};

}  // namespace

extern "C" int ft_layer_fwd(const FtLayerFwd* a, cudaStream_t st) {
  const int nq = a->n_groups * a->g * a->D, nqkv = a->n_groups * (a->g + 2) * a->D;
  const void* h_in = a->res != nullptr ? a->h_in : a->x;
  FT_TRY(ft_add_rmsnorm_fwd(a->res, a->x, a->w_an, a->h_in, a->n1, a->rs1, a->T, a->H, a->eps, st));
  FT_TRY(linear(a->n1, a->w_qkv, a->qkv, a->T, nqkv, a->H, 1.f, a->status, st));
  FT_TRY(ft_rope(a->qkv, a->cos, a->sin, a->pos, a->T, a->S, a->n_groups, a->g, a->D, nqkv, 0, st));
  FT_TRY(ft_attn_fwd(a->qkv, a->attn, a->lse, a->T / a->S, a->S, a->n_groups, a->g, a->D, nqkv, nq,
                     a->scale, a->status, st));
  FT_TRY(linear(a->attn, a->w_o, a->o, a->T, a->H, nq, a->r, a->status, st));
  FT_TRY(ft_add_rmsnorm_fwd(h_in, a->o, a->w_fn, a->h_mid, a->n2, a->rs2, a->T, a->H, a->eps, st));
  FT_TRY(ft_gemm_swiglu_bf16(a->n2, a->w_fc1, a->y1, a->act, a->T, a->F, a->H, a->H, a->H, 2 * a->F,
                             a->F, 1.f, 0, a->status, st));
  return linear(a->act, a->w_2, a->f, a->T, a->H, a->F, a->r, a->status, st);
}

extern "C" int ft_layer_bwd_ffn(const FtLayerBwdFfn* a, cudaStream_t side_stream, cudaStream_t st) {
  SideStream side(st, side_stream);
  FT_TRY(ft_gemm_swiglu_bwd_bf16(a->dh, a->w_2, a->y1, a->dy1, a->T, a->F, a->H, a->H, a->F,
                                 2 * a->F, 2 * a->F, a->r, 0, a->status, st));
  FT_TRY(side.wgrad(a->dh, a->act, a->g_2, a->T, a->H, a->F, a->r, a->accumulate, a->status));
  FT_TRY(side.wgrad(a->dy1, a->n2, a->g_fc1, a->T, 2 * a->F, a->H, 1.f, a->accumulate, a->status));
  FT_TRY(dgrad(a->dy1, a->w_fc1, a->dn2, a->T, 2 * a->F, a->H, 1.f, a->status, st));
  FT_TRY(side.join());   // dh, which the FC2 weight gradient reads, is overwritten next
  return ft_rmsnorm_bwd(a->dn2, a->h_mid, a->w_fn, a->rs2, a->dh, a->dh, a->partial, a->g_fn,
                        a->accumulate, a->T, a->H, st);
}

extern "C" int ft_layer_bwd_attn(const FtLayerBwdAttn* a, cudaStream_t side_stream,
                                 cudaStream_t st) {
  const int nq = a->n_groups * a->g * a->D, nqkv = a->n_groups * (a->g + 2) * a->D;
  SideStream side(st, side_stream);
  FT_TRY(dgrad(a->dh, a->w_o, a->dattn, a->T, a->H, nq, a->r, a->status, st));
  FT_TRY(side.wgrad(a->dh, a->attn, a->g_o, a->T, a->H, nq, a->r, a->accumulate, a->status));
  FT_TRY(ft_attn_bwd(a->dattn, a->qkv, a->attn, a->lse, a->dqkv, a->acc, a->delta, a->T / a->S, a->S,
                     a->n_groups, a->g, a->D, nqkv, nq, nq, a->scale, 0, a->cos, a->sin, a->pos,
                     a->status, st));
  FT_TRY(side.wgrad(a->dqkv, a->n1, a->g_qkv, a->T, nqkv, a->H, 1.f, a->accumulate, a->status));
  FT_TRY(dgrad(a->dqkv, a->w_qkv, a->dn1, a->T, nqkv, a->H, 1.f, a->status, st));
  FT_TRY(side.join());   // dh, which the output-projection weight gradient reads, is overwritten next
  return ft_rmsnorm_bwd(a->dn1, a->h_in, a->w_an, a->rs1, a->dh, a->dh, a->partial, a->g_an,
                        a->accumulate, a->T, a->H, st);
}
