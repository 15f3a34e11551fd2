// Launch interface of the training-step kernels: what surrounds the GEMMs and the attention of a transformer block,
// the language-model loss, and the optimizer. 16-bit element types only unless noted; every accumulation is fp32.
#pragma once
#include <cuda_runtime.h>

#include "core/core.h"

namespace hl {
namespace train {

constexpr int kMaxNormWidth = 1024;   // the ring of the backward pass holds whole rows, a lane the sums of its columns
constexpr int64_t kMaxRows = 65535 * 128;   // of the strip kernels: their row ranges are the grid's second dimension

// Column sums end in two steps: the kernels that walk the rows write one fp32 partial per CTA and column, one later
// launch adds up the partials of several of them. `src` is [rows][width], `dst` has the element type of the call.
struct ColSegment {
  const float* src;
  void* dst;
  int rows, width;
};
constexpr int kMaxColSegments = 8;

// dx = residual + gradient of the layer norm at x for the output gradient dh (residual may be null).
// partials: [3][layerNormPartials(rows)][width]: dgamma, dbeta, and (dx_sums) the column sums of dx as stored.
int layerNormPartials(int64_t rows);
hlResult_t layerNormBackward(int dt, const void* dh, const void* x, const float* mean, const float* rstd, const void* gamma,
                             const void* residual, void* dx, bool dx_sums, float* partials, int64_t rows, int width, cudaStream_t s);

// out = gelu(u), tanh form.
hlResult_t geluForward(int dt, const void* u, void* out, int64_t count, cudaStream_t s);
// Rows a strip kernel gives to one CTA: its partials are [stripPartials(rows)][width].
int stripPartials(int64_t rows);
// du = dg * gelu'(u), and column-sum partials of du (unless null). width a multiple of 8.
hlResult_t geluBackward(int dt, const void* dg, const void* u, void* du, float* partials, int64_t rows, int width, cudaStream_t s);
// Column-sum partials of a [rows][width] matrix.
hlResult_t columnSums(int dt, const void* src, float* partials, int64_t rows, int width, cudaStream_t s);
// The gradients of the three attention operands, each [batch, heads, seq, head_dim] by strides (head_dim contiguous),
// written side by side as [batch * seq][3 * heads * head_dim], with column-sum partials.
struct Strided4 {
  const void* p;
  int64_t sb, sh, st;
};
hlResult_t packQkvGradient(int dt, const Strided4 grads[3], void* dqkv, float* partials, int64_t batch, int64_t seq, int heads, int head_dim,
                           cudaStream_t s);
hlResult_t finishColumns(int dt, const ColSegment* segs, int n, cudaStream_t s);

// Cross entropy over the rows of `logits` ([rows] of `vocab` elements, `stride` apart, stride a multiple of 8):
// lse[row]; loss[0] = mean over the rows whose target is not ignore_index, loss[1] = how many those are.
// scratch: 2 floats per row.
hlResult_t crossEntropyForward(int dt, const void* logits, int64_t stride, const int64_t* targets, int64_t rows, int vocab, int64_t ignore_index,
                               float* lse, float* row_loss, float* loss, cudaStream_t s);
// dlogits (same layout; the padding behind `vocab` becomes zero) for the gradient *grad of the mean loss.
hlResult_t crossEntropyBackward(int dt, const void* logits, int64_t stride, const int64_t* targets, int64_t rows, int vocab, int64_t ignore_index,
                                const float* lse, const float* loss, const float* grad, void* dlogits, cudaStream_t s);

// One AdamW update of `count` elements (a multiple of 8). The gradient is a sum over `ranks`; `keep` = 1 - lr * decay,
// `rest1` = 1 - beta1 and `rest2` = 1 - beta2 (not to be taken in fp32: 1 - 0.999f is 5e-5 off), `step` =
// lr / (1 - beta1^t), `correction2` = 1 - beta2^t. master: fp32 copy of 16-bit weights, or null.
struct AdamWArgs {
  float ranks, keep, beta1, rest1, beta2, rest2, step, correction2, eps;
};
hlResult_t shardedAdamW(int dt, const void* grad, void* weight, float* master, float* m, float* v, int64_t count, const AdamWArgs& a,
                        cudaStream_t s);

// One AdamW step on several 16-bit or fp32 tensors at once, moments of the weights' type, arithmetic in fp32. `step` is
// each tensor's own step count, already advanced.
struct AdamWTensor {
  void *weight, *m, *v;
  const void* grad;
  const float* step;
  int64_t count;
};
constexpr int kMaxAdamWTensors = 480;
hlResult_t multiAdamW(int dt, const AdamWTensor* tensors, int n, double lr, double beta1, double beta2, double decay, double eps, cudaStream_t s);

// Mixture of experts (moe.cu). row_of: [tokens], row of the dispatch buffer or -1; token_of: [experts * capacity]; count: [experts], rows in use.
hlResult_t moeRoute(int dt, const void* logits, int tokens, int experts, int capacity, int* expert, float* gate, int* row_of, int* token_of,
                    int* count, cudaStream_t s);
hlResult_t moeGather(const void* src, const int* index, void* dst, int rows, int width, cudaStream_t s);
hlResult_t moeCombine(int dt, const void* x, const float* gate, const void* rows, const int* row_of, void* y, int tokens, int width, cudaStream_t s);
hlResult_t moeRowGradient(int dt, const void* dy, const float* gate, const void* rows, const int* token_of, void* drows, float* dgate, int n_rows,
                          int width, cudaStream_t s);
// Whether moeTokenGradient adds the router's share to dx itself (else the caller adds dlogits * router). dy may be null.
bool moeRouterFits(int experts);
hlResult_t moeTokenGradient(int dt, const void* dy, const void* drows, const int* row_of, const void* logits, const int* expert, const float* gate,
                            const float* dgate, const void* router, void* dx, void* dlogits, int tokens, int width, int experts, cudaStream_t s);

// The same, and partials of the router's gradient ([moeRouterPartials(tokens)][experts * width], to be finished by finishColumns), in
// one pass; for as many experts as fit.
bool moeTokensAndRouterFits(int experts);
int moeRouterPartials(int tokens);
hlResult_t moeTokensAndRouter(int dt, const void* dy, const void* drows, const int* row_of, const void* logits, const int* expert, const float* gate,
                              const float* dgate, const void* router, const void* x, void* dx, float* partials, int tokens, int width, int experts,
                              cudaStream_t s);

// Products of groups of matrices (expert_gemm.cu): out[g][n][m] = sum over k of A[g][m][k] B[g][n][k]. a_mn / b_mn: the operand is
// stored [g][k][m] / [g][k][n] instead. All are contiguous and start on 16-byte boundaries, inner dimensions are multiples of 8.
// With `counts`, a group's n (kGemmRaggedN) or k (kGemmRaggedK) ends at counts[g], rounded up to 32 rows, one at least;
// operand rows between the two are zeros, and rows of `out` behind them are not written.
enum GemmRagged { kGemmWhole = 0, kGemmRaggedN = 1, kGemmRaggedK = 2 };
// What follows: nothing; aux = gelu(out); out = product * gelu'(aux). The product is rounded before it goes on.
enum GemmEpilogue { kGemmStore = 0, kGemmGelu = 1, kGemmGeluGradient = 2 };
struct GemmSpec {
  const void *a, *b;
  void *out, *aux;
  int m, n, k;
  bool a_mn, b_mn;
  int ragged, epilogue;
  const void* bias = nullptr;    // [m], added before the product is rounded; not with kGemmGeluGradient
  float* columns = nullptr;      // kGemmGeluGradient: partials of the sums of `out` over n: [gemmPartials(n)][m]; one group, without counts
};
inline int gemmPartials(int64_t n) { return 2 * (int)((n + 255) / 256); }
// Whether it runs on the current device: a GPU and a driver that it is made for, page-locked memory for its status, and not switched
// off (HYLINK_OWN_PRODUCTS=0). Where it does not, the library's products are taken.
bool gemmRuns(int dt);
// Whether experts of this width and hidden width, with this many rows in all, go through it; `captured`: into a CUDA graph.
bool expertGemmPays(int64_t rows, int64_t width, int64_t hidden, bool captured);
// The same for the first product of a transformer block's MLP, and the gradient of what follows it.
bool mlpGemmPays(int64_t rows, int64_t width, int64_t hidden);
// One launch of `n` products, two at most. `limit_ns` ends every wait inside it (0: two seconds); without `loads` operands never
// arrive, for tests of that.
hlResult_t expertGemm(int dt, const GemmSpec* specs, int n, int groups, const int* counts, cudaStream_t s, uint64_t limit_ns = 0, bool loads = true);
// An error once a wait inside a product on `device` (-1: the current one) has run out, until it is asked with `clear`. Launches ask
// without. The results of that product and of what came after it are not valid; to be asked where the host has waited for them.
hlResult_t gemmStatus(int device, bool clear);

}  // namespace train
}  // namespace hl
