// The block-FP8 layer as two host calls: the forward pass after the router GEMM, and the backward
// pass up to the router's own gradient.  Each enqueues the same kernels, through the same entry
// points, as a caller that makes the calls one by one; what goes is the host work between them.
// From Python the forward pass took 273 us of host time (eight wrapper calls and five
// [experts]-sized tensor operations, against 88 us of kernels for one decoded token) and takes 130,
// the backward pass 366 us and takes 172.
//
// No step reads device memory on the host or allocates: the caller hands over every result and
// scratch buffer (sizes beside the declarations in include/b200moe.h).
#include <cstdlib>
#include <cstring>
#include <initializer_list>

#include <nvtx3/nvToolsExt.h>

#include "common.cuh"
#include "host_util.h"
#include "../../include/b200moe.h"

namespace b200 {

// The frequencies the auxiliary loss's gradient needs, from the sort's offsets (bit for bit what torch
// gives for the quotients: it multiplies by the rounded reciprocal of the number of assignments).
__global__ void frequency_kernel(const int* __restrict__ offsets, int experts, float per_assignment, int sigmoid,
                                 float* __restrict__ frequency) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= experts) return;
  const float count = (float)(offsets[e + 1] - offsets[e]);
  frequency[e] = (sigmoid ? count * (float)experts : count) * per_assignment;
}

// Pieces of a workspace, each on a 256-byte boundary.
struct Pieces {
  char* base;
  long long used;
  template <typename T>
  T* take(long long count) {
    T* at = reinterpret_cast<T*>(base + used);
    used += (count * (long long)sizeof(T) + 255) / 256 * 256;
    return at;
  }
};

struct ForwardScratch {
  float *x_scale, *act_scale;
  void *sort, *statistics;
  long long bytes;
  ForwardScratch(char* base, long long tokens, int width, int inner, int experts, int top_k) {
    const long long rows = tokens * top_k;
    Pieces p = {base, 0};
    x_scale = p.take<float>(rows * (width / 128));
    act_scale = p.take<float>(rows * (inner / 128));
    sort = p.take<char>(b200moe_sort_assignments_workspace_bytes(rows, experts));
    statistics = p.take<char>(b200moe_routing_probability_sum_workspace_bytes(tokens, experts));
    bytes = p.used;
  }
};

struct BackwardScratch {
  float *dy_scale, *gh_scale, *dscore, *grad_route_weights, *frequency;
  long long bytes;
  BackwardScratch(char* base, long long tokens, int width, int inner, int experts, int top_k) {
    const long long rows = tokens * top_k;
    Pieces p = {base, 0};
    dy_scale = p.take<float>(rows * (width / 128));
    gh_scale = p.take<float>(rows * (2 * inner / 128));
    dscore = p.take<float>(rows);
    grad_route_weights = p.take<float>(rows);
    frequency = p.take<float>(experts);
    bytes = p.used;
  }
};

static bool sizes_ok(long long tokens, int width, int inner, int experts, int top_k) {
  return tokens > 0 && width > 0 && inner > 0 && width % 128 == 0 && inner % 128 == 0 && experts > 0 &&
         experts <= 1024 && top_k > 0 && top_k <= 32 && top_k <= experts && tokens * top_k <= 0x7fffffffLL;
}

static bool mode_ok(int mode) { return mode >= B200MOE_ROUTE_TOPK_THEN_SOFTMAX && mode <= B200MOE_ROUTE_SIGMOID_NOAUX_TC; }

// The pointers of a call are looked at before its first launch: a missing or misaligned one must not
// show up when part of the work is on the stream already.
static bool all_given(std::initializer_list<const void*> pointers) {
  for (const void* p : pointers)
    if (p == nullptr) return false;
  return true;
}

static bool all_aligned(uintptr_t bytes, std::initializer_list<const void*> pointers) {  // (NULL is aligned)
  for (const void* p : pointers)
    if ((uintptr_t)p % bytes) return false;
  return true;
}

// B200MOE_NVTX=1: a range around each step's launches, as the Python wrappers have around theirs.
struct Range {
  explicit Range(const char* name) {
    if (wanted()) nvtxRangePushA(name);
  }
  ~Range() {
    if (wanted()) nvtxRangePop();
  }
  static bool wanted() {
    static const bool on = [] {
      const char* v = getenv("B200MOE_NVTX");
      return v != nullptr && strcmp(v, "1") == 0;
    }();
    return on;
  }
};

}  // namespace b200

using namespace b200;

// One step through its entry point, in an NVTX range of the wrapper's name where ranges are wanted.
#define B200_STEP(name, ...)                         \
  do {                                               \
    const Range range_("b200moe." #name);            \
    const int code_ = b200moe_##name(__VA_ARGS__);   \
    if (code_ != B200MOE_OK) return code_;           \
  } while (0)

extern "C" long long b200moe_forward_workspace_bytes(long long tokens, int width, int inner, int experts, int top_k) {
  if (!sizes_ok(tokens, width, inner, experts, top_k)) return -1;
  return ForwardScratch(nullptr, tokens, width, inner, experts, top_k).bytes;
}

extern "C" int b200moe_forward_fp8(const b200moe_forward_args* a, void* stream) {
  if (a == nullptr || !sizes_ok(a->tokens, a->width, a->inner, a->experts, a->top_k) || !mode_ok(a->mode))
    return B200MOE_ERR_ARG;
  if (!all_given({a->x, a->residual, a->logits, a->w13, a->w13_scale, a->w2, a->w2_scale, a->route_weights, a->ids,
                  a->order, a->offsets, a->slots, a->counts, a->h13, a->output, a->aux, a->probability_sum, a->x_q,
                  a->act_q, a->expert_rows, a->workspace, a->status}))
    return B200MOE_ERR_ARG;
  if (!all_aligned(16, {a->x, a->residual, a->w13, a->w2, a->h13, a->output, a->x_q, a->act_q, a->expert_rows}) ||
      !all_aligned(256, {a->workspace}))
    return B200MOE_ERR_ALIGN;
  const int D = a->width, F = a->inner, E = a->experts, K = a->top_k;
  const long long T = a->tokens, R = T * K;
  const ForwardScratch s((char*)a->workspace, T, D, F, E, K);
  B200_STEP(route_topk, a->logits, E, (int)T, E, K, a->mode, a->bias, a->n_group, a->topk_group,
            a->routed_scaling, a->route_weights, a->ids, stream);
  B200_STEP(sort_assignments, a->ids, R, E, a->order, a->offsets, a->slots, a->counts, s.sort, a->status,
            stream);
  // scales are stored block-major, [width / 128][rows]
  B200_STEP(quantize_rows_scatter, a->x, D, T, a->slots, K, R, D, a->x_q, D, s.x_scale, 1, R, nullptr, D,
            a->status, stream);
  B200_STEP(grouped_gemm_fp8, a->x_q, D, s.x_scale, 1, R, a->w13, a->w13_scale, a->h13, 2LL * F, nullptr, 0,
            a->offsets, E, E, R, 2 * F, D, 0, 256, a->status, stream);
  B200_STEP(swiglu_quantize, a->h13, 2LL * F, R, F, a->act_q, F, s.act_scale, 1, R, nullptr, F, a->limit,
            a->limited, stream);
  B200_STEP(grouped_gemm_fp8, a->act_q, F, s.act_scale, 1, R, a->w2, a->w2_scale, a->expert_rows, D, nullptr, 0,
            a->offsets, E, E, R, D, F, 0, 256, a->status, stream);
  B200_STEP(combine, a->expert_rows, D, R, a->slots, a->route_weights, a->residual, D, a->output, D, T, D, K,
            stream);
  const Range range("b200moe.routing_statistics");
  return launch_routing_statistics(a->logits, E, T, E, a->mode, s.statistics, a->probability_sum, a->counts, K, a->aux,
                                   reinterpret_cast<cudaStream_t>(stream));
}

extern "C" long long b200moe_backward_workspace_bytes(long long tokens, int width, int inner, int experts, int top_k) {
  if (!sizes_ok(tokens, width, inner, experts, top_k)) return -1;
  return BackwardScratch(nullptr, tokens, width, inner, experts, top_k).bytes;
}

extern "C" int b200moe_backward_fp8(const b200moe_backward_args* a, void* stream) {
  if (a == nullptr || !sizes_ok(a->tokens, a->width, a->inner, a->experts, a->top_k) || !mode_ok(a->mode))
    return B200MOE_ERR_ARG;
  if (!all_given({a->grad_output, a->x, a->w13, a->w13_scale, a->w2, a->w2_scale, a->logits, a->route_weights, a->ids,
                  a->order, a->offsets, a->slots, a->h13, a->grad_x, a->grad_logits, a->grad_logits_high,
                  a->grad_logits_low, a->dy_q, a->rows, a->r, a->gh_q, a->workspace, a->status}) ||
      (a->grad_w13 != nullptr && a->gh == nullptr))
    return B200MOE_ERR_ARG;
  if (!all_aligned(16, {a->grad_output, a->x, a->w13, a->w2, a->h13, a->grad_x, a->grad_w13, a->grad_w2, a->dy_q,
                        a->rows, a->r, a->gh_q, a->gh}) ||
      !all_aligned(256, {a->workspace}))
    return B200MOE_ERR_ALIGN;
  const int D = a->width, F = a->inner, E = a->experts, K = a->top_k;
  const long long T = a->tokens, R = T * K;
  const BackwardScratch s((char*)a->workspace, T, D, F, E, K);
  cudaStream_t cuda_stream = reinterpret_cast<cudaStream_t>(stream);
  // `rows` holds in turn: dy and x in expert order (operands of the weight gradients), the input
  // gradient's rows.  `r` becomes the down weight's second operand in place.
  void* dy_rows = a->grad_w2 != nullptr ? a->rows : nullptr;
  B200_STEP(quantize_rows_scatter, a->grad_output, D, T, a->slots, K, R, D, a->dy_q, D, s.dy_scale, 1, R,
            dy_rows, D, a->status, stream);
  B200_STEP(grouped_gemm_fp8, a->dy_q, D, s.dy_scale, 1, R, a->w2, a->w2_scale, a->r, F, nullptr, 0, a->offsets,
            E, E, R, F, D, 1, 256, a->status, stream);
  B200_STEP(dswiglu_routed, a->h13, 2LL * F, a->r, F, a->route_weights, R, a->order, R, F, s.dscore, a->gh_q,
            2LL * F, s.gh_scale, 1, R, a->gh, 2LL * F, a->grad_w2 != nullptr ? a->r : nullptr, F,
            a->limit, a->limited, a->status, stream);
  B200_STEP(gather_scalar, s.dscore, R, a->slots, R, s.grad_route_weights, a->status, stream);
  if (a->grad_w2 != nullptr)
    B200_STEP(grouped_wgrad_bf16, a->rows, D, a->r, F, a->offsets, E, 1, R, D, F, a->grad_w2,
              a->weight_gradients_fp32, a->status, stream);
  if (a->grad_w13 != nullptr) {
    B200_STEP(scatter_rows, a->x, D, T, a->slots, K, R, D, a->rows, D, a->status, stream);
    B200_STEP(grouped_wgrad_bf16, a->gh, 2LL * F, a->rows, D, a->offsets, E, 1, R, 2 * F, D, a->grad_w13,
              a->weight_gradients_fp32, a->status, stream);
  }
  B200_STEP(grouped_gemm_fp8, a->gh_q, 2LL * F, s.gh_scale, 1, R, a->w13, a->w13_scale, a->rows, D, nullptr, 0,
            a->offsets, E, E, R, D, 2 * F, 1, 256, a->status, stream);
  B200_STEP(combine, a->rows, D, R, a->slots, nullptr, nullptr, 0, a->grad_x, D, T, D, K, stream);
  const bool sigmoid = a->mode == B200MOE_ROUTE_SIGMOID_NOAUX_TC;
  const Range range("b200moe.routing_gradient");
  if (a->grad_aux != nullptr) {
    frequency_kernel<<<(E + 255) / 256, 256, 0, cuda_stream>>>(a->offsets, E, 1.0f / (float)R, sigmoid, s.frequency);
    const int code = launch_status();
    if (code != B200MOE_OK) return code;
  }
  return launch_routing_gradient(a->logits, E, T, E, K, a->mode, a->ids, a->route_weights, s.grad_route_weights,
                                 a->grad_aux, a->grad_aux != nullptr ? s.frequency : nullptr,
                                 (float)((sigmoid ? 1.0 : (double)E) / (double)T), a->grad_probability_sum,
                                 a->grad_logits, E, a->grad_logits_high, a->grad_logits_low, cuda_stream);
}
