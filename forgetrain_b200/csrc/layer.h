// Arguments of the one-block calls (layer.cu); the ctypes mirrors are in ops/layer.py. All matrices
// are contiguous, activations and weights bf16, statistics and gradients of weights fp32. T tokens =
// sequences of S; H hidden size, n_groups KV groups of g query heads each, head dimension D, F feed-
// forward width. r: muP residual multiplier; scale: softmax scale; pos: int32 [T] or null.
#pragma once

struct FtLayerFwd {
  // block input = res + x (res null: x alone, and h_in is not written)
  const void *res, *x, *w_an, *w_qkv, *w_o, *w_fn, *w_fc1, *w_2, *cos, *sin, *pos;
  void *h_in, *n1, *rs1, *qkv, *attn, *lse, *o, *h_mid, *n2, *rs2, *y1, *act, *f;
  int* status;
  int T, S, H, n_groups, g, D, F;
  float eps, r, scale;
};

// Feed-forward half of the backward: dh (gradient of the block output) becomes the gradient of the
// block's middle. Scratch: dy1 [T][2F], dn2 [T][H], partial (ft_rmsnorm_bwd).
struct FtLayerBwdFfn {
  void* dh;
  const void *y1, *act, *n2, *h_mid, *rs2, *w_2, *w_fc1, *w_fn;
  void *g_2, *g_fc1, *g_fn, *dy1, *dn2, *partial;
  int* status;
  int T, H, F, accumulate;
  float r;
};

// Attention half: dh becomes the gradient of the block input. Scratch: dattn [T][n_groups g D], dqkv
// [T][n_groups (g + 2) D], acc and delta (ft_attn_bwd), dn1 [T][H], partial (ft_rmsnorm_bwd).
struct FtLayerBwdAttn {
  void* dh;
  const void *attn, *lse, *qkv, *n1, *h_in, *rs1, *w_o, *w_qkv, *w_an, *cos, *sin, *pos;
  void *g_o, *g_qkv, *g_an, *dattn, *dqkv, *acc, *delta, *dn1, *partial;
  int* status;
  int T, S, H, n_groups, g, D, accumulate;
  float r, scale;
};
