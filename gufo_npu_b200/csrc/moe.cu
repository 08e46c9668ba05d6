// The routed-expert FFN of the MoE models on the device: the router's top-k
// (Route, src/models/qwen35/moe.cpp:16-41 in the reference), the shared
// expert's gate (SharedExpertScale, :43-46), the experts' SwiGLU FFN as grouped
// products over the stacked expert tensors (GgufProjections::ApplyExpert,
// src/models/qwen35/gguf_projections.cpp:218-237) and the weighted sum of
// Decoder::MoeFfn (src/models/qwen35/decoder.cpp:535-557).
//
// The chosen experts stay in device memory from the router kernel to the
// grouped products, so a step never waits for the host. Bytes per token and
// layer: the chosen experts' rows (k * (2 * expert_ffn * hidden + hidden *
// expert_ffn) weights at their GGUF size) plus the router rows; HBM-bound.
#include "moe.cuh"

#include <cfloat>

namespace gufo {

namespace {

constexpr int kRouteThreads = 256;
constexpr int kRouteMaxExperts = 1024;
// The smallest positive normal fp16: the floor of the top-k probability mass
// (moe.cpp:12).
constexpr double kWeightSumFloor = 6.103515625e-5;

// One block per token. Probabilities are exp(logit - max) in double as in the
// reference, computed by all threads; warp 0 then holds experts l, l + 32, ...
// (PER_LANE of them) in lane l. Their sum is a shuffle tree instead of the
// reference's index-order loop, which can move a weight by the last bit of its fp32
// value. The arg-max rounds order (probability, id) exactly as the reference does
// (moe.cpp:28-32): the bits of positive doubles order as integers, so a round is
// three warp-wide integer reductions (high words, low words, ids) where doubles
// passed through shuffles took fifteen dependent steps. Bound by latency: an L2
// round trip, then dependent steps.
// The dependents may start once the wait has returned: they find every kernel
// before this one complete (EnqueueMoeFfn relies on it).
template <int PER_LANE>
__global__ void __launch_bounds__(kRouteThreads)
RouteKernel(const float* __restrict__ logits, int stride, int experts, int k,
            int* __restrict__ chosen, float* __restrict__ weights, float* __restrict__ shared_scale) {
  constexpr int kEach = PER_LANE * 32 / kRouteThreads;
  extern __shared__ double shared_prob[];   // [experts], then [k] the chosen ones in slot order
  __shared__ float warp_top[kRouteThreads / 32];
  double* picked = shared_prob + experts;
  const int token = blockIdx.x;
  const float* row = logits + static_cast<size_t>(token) * stride;
  const int lane = threadIdx.x & 31;
  GridDependencyWait();
  GridLaunchDependents();
  float v[kEach];
  float top = -FLT_MAX;
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int e = threadIdx.x + kRouteThreads * j;
    v[j] = e < experts ? row[e] : -FLT_MAX;
    top = fmaxf(top, v[j]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
  }
  if (lane == 0) {
    warp_top[threadIdx.x >> 5] = top;
  }
  if (threadIdx.x == kRouteThreads - 32 && shared_scale != nullptr) {
    shared_scale[token] = static_cast<float>(1.0 / (1.0 + exp(-static_cast<double>(row[experts]))));
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kRouteThreads / 32; ++w) {
    top = fmaxf(top, warp_top[w]);
  }
  const double max_logit = static_cast<double>(top);
#pragma unroll
  for (int j = 0; j < kEach; ++j) {
    const int e = threadIdx.x + kRouteThreads * j;
    if (e < experts) {
      shared_prob[e] = exp(static_cast<double>(v[j]) - max_logit);
    }
  }
  __syncthreads();
  if (threadIdx.x >= 32) {
    return;
  }
  unsigned long long key[PER_LANE];
  unsigned left = 0;   // which of the lane's entries can still win a round
  double total = 0;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int e = lane + 32 * j;
    const double prob = e < experts ? shared_prob[e] : 0.0;
    total += prob;
    // A NaN (of a NaN or an infinite logit) ranks with the zeros: the ids stay below
    // `experts` whatever the logits, as the products that follow address by them. The
    // row's total is NaN then, and so is every weight.
    key[j] = prob >= 0.0 ? static_cast<unsigned long long>(__double_as_longlong(prob)) : 0ull;
    left |= e < experts ? 1u << j : 0u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    total += __shfl_xor_sync(0xFFFFFFFFu, total, o);
  }
  for (int slot = 0; slot < k; ++slot) {
    unsigned long long best = 0;
    int at = 0x7FFFFFFF;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      // Ascending j is ascending id, so a strict compare keeps the lower id.
      if ((left >> j & 1u) != 0 && (at == 0x7FFFFFFF || key[j] > best)) {
        best = key[j];
        at = lane + 32 * j;
      }
    }
    const unsigned high = static_cast<unsigned>(best >> 32), low = static_cast<unsigned>(best);
    const unsigned top_high = __reduce_max_sync(0xFFFFFFFFu, high);
    const unsigned top_low = __reduce_max_sync(0xFFFFFFFFu, high == top_high ? low : 0u);
    const int winner = __reduce_min_sync(0xFFFFFFFFu, high == top_high && low == top_low ? at : 0x7FFFFFFF);
    if (winner == at && at != 0x7FFFFFFF) {
      left &= ~(1u << (at >> 5));
    }
    if (lane == 0) {
      picked[slot] = __longlong_as_double(static_cast<long long>(static_cast<unsigned long long>(top_high) << 32 | top_low));
      chosen[static_cast<size_t>(token) * k + slot] = winner;
    }
  }
  __syncwarp();
  // The slot-order sum of the chosen probabilities (moe.cpp:33-36).
  double mass = 0;
  for (int first = 0; first < k; first += 32) {
    const double mine = first + lane < k ? picked[first + lane] / total : 0.0;
    for (int s = 0; s < 32 && first + s < k; ++s) {
      mass += __shfl_sync(0xFFFFFFFFu, mine, s);
    }
  }
  mass = mass > kWeightSumFloor ? mass : kWeightSumFloor;
  for (int slot = lane; slot < k; slot += 32) {
    weights[static_cast<size_t>(token) * k + slot] = static_cast<float>(picked[slot] / total / mass);
  }
}

// out[t][i] = shared[t][i] * scale[t] + sum over slots, in slot order, of
// weights[t][slot] * expert_out[t][slot][i] (decoder.cpp:541-556). `out` may be
// `shared`.
__global__ void __launch_bounds__(256)
CombineKernel(const float* shared, const float* __restrict__ scale,
              const float* __restrict__ weights, const float* __restrict__ expert_out, int k,
              int hidden, float* out) {
  GridDependencyWait();
  const int token = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= hidden) {
    return;
  }
  float v = shared[static_cast<size_t>(token) * hidden + i] * scale[token];
  for (int slot = 0; slot < k; ++slot) {
    v = fmaf(weights[static_cast<size_t>(token) * k + slot],
             expert_out[(static_cast<size_t>(token) * k + slot) * hidden + i], v);
  }
  out[static_cast<size_t>(token) * hidden + i] = v;
}

}  // namespace

int EnqueueRoute(gufo_cuda_ctx* ctx, const float* logits, int stride, int tokens, int experts, int k,
                 int* chosen, float* weights, float* shared_scale) {
  if (tokens <= 0 || experts <= 0 || k <= 0 || k > experts || experts > kRouteMaxExperts || stride < experts) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "route: 1 <= k <= experts <= 1024, stride >= experts");
  }
  const size_t smem = static_cast<size_t>(experts + k) * sizeof(double);
  if (experts <= 256) {
    GUFO_CUDA_TRY(LaunchOverlapped(RouteKernel<8>, dim3(tokens), dim3(kRouteThreads), smem, ctx->stream, 1, logits,
                                   stride, experts, k, chosen, weights, shared_scale));
  } else {
    GUFO_CUDA_TRY(LaunchOverlapped(RouteKernel<32>, dim3(tokens), dim3(kRouteThreads), smem, ctx->stream, 1, logits,
                                   stride, experts, k, chosen, weights, shared_scale));
  }
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

int BuildExpertBank(gufo_cuda_ctx* ctx, const gufo_cuda_expert_bank& bank, ExpertBank* out) {
  if (bank.experts <= 0 || bank.expert_ffn <= 0 || bank.hidden <= 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert bank: counts must be positive");
  }
  const struct {
    gufo_cuda_matrix handle;
    int64_t rows, cols;
    const char* name;
  } want[3] = {{bank.gate_exps, bank.expert_ffn, bank.hidden, "ffn_gate_exps"},
               {bank.up_exps, bank.expert_ffn, bank.hidden, "ffn_up_exps"},
               {bank.down_exps, bank.hidden, bank.expert_ffn, "ffn_down_exps"}};
  GemvPart parts[3];
  for (int i = 0; i < 3; ++i) {
    const Matrix* m = ctx->FindMatrix(want[i].handle);
    if (m == nullptr) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, std::string("expert bank: no matrix for ") + want[i].name);
    }
    // Experts are stacked along the rows: [cols, rows, experts] in GGUF terms
    // (gguf_projections.cpp:132-139).
    if (m->cols != want[i].cols || m->rows != want[i].rows * bank.experts) {
      return Fail(GUFO_CUDA_SHAPE, std::string("expert bank: ") + want[i].name + " has shape [" +
                                       std::to_string(m->cols) + ", " + std::to_string(m->rows) +
                                       "], expected [" + std::to_string(want[i].cols) + ", " +
                                       std::to_string(want[i].rows * bank.experts) + "]");
    }
    parts[i] = {m->data, static_cast<int>(want[i].rows), 0, m->type, static_cast<int>(m->row_bytes)};
  }
  out->experts = bank.experts;
  out->expert_ffn = bank.expert_ffn;
  out->hidden = bank.hidden;
  out->in = GemvArgs{};
  out->in.parts[0] = parts[0];
  out->in.parts[1] = parts[1];
  out->in.parts[1].out_offset = bank.expert_ffn;
  out->in.nparts = 2;
  out->in.total_rows = 2 * bank.expert_ffn;
  out->in.y_stride = 2 * bank.expert_ffn;
  out->in.cols = bank.hidden;
  out->down = GemvArgs{};
  out->down.parts[0] = parts[2];
  out->down.nparts = 1;
  out->down.total_rows = bank.hidden;
  out->down.y_stride = bank.hidden;
  out->down.cols = bank.expert_ffn;
  return GUFO_CUDA_OK;
}

namespace {

// The down rows of `groups` inputs, each with k chosen experts (FastGemvArgs::mix_*).
int LaunchDown(gufo_cuda_ctx* ctx, const ExpertBank& bank, const int* ids, const float* weights, const float* scale,
               const float* shared, int groups, int k, const float* act, float* out) {
  FastGemvArgs args{};
  args.parts[0] = {bank.down.parts[0].data, bank.down.parts[0].rows, 0};
  args.cols = k * bank.down.cols;
  args.row_bytes = bank.down.parts[0].row_bytes;
  args.x = act;
  args.y = out;
  args.y_stride = bank.hidden;
  args.tokens = 1;
  args.groups = groups;
  args.mix_ids = ids;
  args.mix_weights = weights;
  args.mix_experts = k;
  args.mix_blocks = bank.down.cols / kSuperBlock;
  args.mix_base = shared;
  args.mix_scale = scale;
  return LaunchGemvMixture(ctx, args);
}

// Whether the mixture kernel takes the down rows of k experts at a time.
bool DownFits(const gufo_cuda_ctx* ctx, const ExpertBank& bank, int k, const float* act) {
  return !ctx->force_general && bank.down.parts[0].type == GUFO_CUDA_Q4_K && bank.down.cols % kSuperBlock == 0 &&
         MixtureFits(k * bank.down.cols) && (reinterpret_cast<uintptr_t>(act) & 15) == 0;
}

}  // namespace

int EnqueueExpertFfn(gufo_cuda_ctx* ctx, const ExpertBank& bank, const int* ids, int pairs, const float* x,
                     int x_stride, int pairs_per_input, float* ffn, float* act, float* y) {
  if (pairs <= 0 || ids == nullptr || x == nullptr || ffn == nullptr || y == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert ffn: null pointer or no pairs");
  }
  GemvArgs in = bank.in;
  in.x = x;
  in.y = ffn;
  in.group_ids = ids;
  in.groups = pairs;
  in.x_group_stride = x_stride;
  in.x_group_div = pairs_per_input > 1 ? pairs_per_input : 1;
  in.y_group_stride = 2 * bank.expert_ffn;
  GemvArgs down = bank.down;
  down.y = y;
  down.group_ids = ids;
  down.groups = pairs;
  down.y_group_stride = bank.hidden;
  if (act != nullptr && GroupedSwiGluInProduct(ctx, in)) {
    // A block multiplies a gate tile and the up tile of the same rows and stores
    // silu(gate) * up; the down product starts from plain rows.
    in.y = act;
    in.y_group_stride = bank.expert_ffn;
    const int rc = LaunchGemvGrouped(ctx, in, kProloguePlain, nullptr, true);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
    down.x = act;
    down.x_group_stride = bank.expert_ffn;
    return DownFits(ctx, bank, 1, act) ? LaunchDown(ctx, bank, ids, nullptr, nullptr, nullptr, pairs, 1, act, y)
                                       : LaunchGemvGrouped(ctx, down, kProloguePlain, nullptr);
  }
  int rc = LaunchGemvGrouped(ctx, in, kProloguePlain, nullptr);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  down.x = ffn;
  down.x_group_stride = 2 * bank.expert_ffn;
  return LaunchGemvGrouped(ctx, down, kPrologueSwiGlu, act);
}

int EnqueueMoeCombine(gufo_cuda_ctx* ctx, const float* shared, const float* scale, const float* weights,
                      const float* expert_out, int tokens, int k, int hidden, float* out) {
  if (tokens <= 0 || k <= 0 || hidden <= 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe combine: counts must be positive");
  }
  GUFO_CUDA_TRY(LaunchOverlapped(CombineKernel, dim3((hidden + 255) / 256, tokens), dim3(256), 0, ctx->stream, 1,
                                 shared, scale, weights, expert_out, k, hidden, out));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

int EnqueueMoeFfn(gufo_cuda_ctx* ctx, const ExpertBank& bank, const int* ids, const float* weights,
                  const float* scale, int tokens, int k, const float* x, int x_stride, const float* shared,
                  float* ffn, float* act, float* expert_out, float* out, bool behind_route) {
  if (tokens <= 0 || k <= 0 || ids == nullptr || weights == nullptr || scale == nullptr || x == nullptr ||
      shared == nullptr || ffn == nullptr || act == nullptr || expert_out == nullptr || out == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe ffn: null pointer or no tokens");
  }
  GemvArgs in = bank.in;
  in.x = x;
  in.y = act;
  in.group_ids = ids;
  in.groups = tokens * k;
  in.x_group_stride = x_stride;
  in.x_group_div = k;
  in.y_group_stride = bank.expert_ffn;
  if (DownFits(ctx, bank, k, act) && GroupedSwiGluInProduct(ctx, in)) {
    // Two launches: gate / up with the SwiGLU in its epilogue, then the down rows of a
    // token's experts side by side with the weighted sum. Directly behind the router's
    // top-k the inputs are complete once the first of them runs (RouteKernel), and its
    // image is built while the top-k is being found. It lets the second start only once
    // the ids are complete.
    in.early_input = behind_route ? 1 : 0;
    const int rc = LaunchGemvGrouped(ctx, in, kProloguePlain, nullptr, true);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
    return LaunchDown(ctx, bank, ids, weights, scale, shared, tokens, k, act, out);
  }
  const int rc = EnqueueExpertFfn(ctx, bank, ids, tokens * k, x, x_stride, k, ffn, act, expert_out);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  return EnqueueMoeCombine(ctx, shared, scale, weights, expert_out, tokens, k, bank.hidden, out);
}

}  // namespace gufo

using gufo::Fail;

extern "C" {

int gufo_cuda_route_device(gufo_cuda_ctx* ctx, const float* router, int stride, int tokens, int experts, int k,
                           int* chosen, float* weights, float* shared_scale) {
  if (ctx == nullptr || router == nullptr || chosen == nullptr || weights == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "route: null pointer");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  if (shared_scale != nullptr && stride < experts + 1) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "route: the shared expert's logit follows the experts'");
  }
  return gufo::EnqueueRoute(ctx, router, stride, tokens, experts, k, chosen, weights, shared_scale);
}

int gufo_cuda_expert_ffn_device(gufo_cuda_ctx* ctx, const gufo_cuda_expert_bank* bank, const int* ids, int pairs,
                                const float* x, int64_t x_stride, int pairs_per_input, float* ffn, float* act,
                                float* y) {
  if (ctx == nullptr || bank == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert ffn: null pointer");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  gufo::ExpertBank built;
  const int rc = gufo::BuildExpertBank(ctx, *bank, &built);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  if (x_stride != 0 && x_stride < bank->hidden) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert ffn: x_stride is 0 (shared input) or at least hidden");
  }
  if (act == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert ffn: null scratch");
  }
  if (pairs_per_input < 1) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "expert ffn: pairs_per_input is at least 1");
  }
  return gufo::EnqueueExpertFfn(ctx, built, ids, pairs, x, static_cast<int>(x_stride), pairs_per_input, ffn, act, y);
}

int gufo_cuda_moe_ffn_device(gufo_cuda_ctx* ctx, const gufo_cuda_expert_bank* bank, const int* ids,
                             const float* weights, const float* scale, int tokens, int k, const float* x,
                             int64_t x_stride, const float* shared, float* ffn, float* act, float* expert_out,
                             float* out) {
  if (ctx == nullptr || bank == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe ffn: null pointer");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  gufo::ExpertBank built;
  const int rc = gufo::BuildExpertBank(ctx, *bank, &built);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  if (x_stride != 0 && x_stride < bank->hidden) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe ffn: x_stride is 0 (shared input) or at least hidden");
  }
  return gufo::EnqueueMoeFfn(ctx, built, ids, weights, scale, tokens, k, x, static_cast<int>(x_stride), shared, ffn,
                             act, expert_out, out, false);
}

int gufo_cuda_moe_layer_device(gufo_cuda_ctx* ctx, const gufo_cuda_expert_bank* bank, const float* router, int stride,
                               int tokens, int k, int* chosen, float* weights, float* scale, const float* x,
                               int64_t x_stride, const float* shared, float* ffn, float* act, float* expert_out,
                               float* out) {
  if (ctx == nullptr || bank == nullptr || router == nullptr || chosen == nullptr || weights == nullptr ||
      scale == nullptr || x == nullptr || shared == nullptr || ffn == nullptr || act == nullptr ||
      expert_out == nullptr || out == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe layer: null pointer");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  gufo::ExpertBank built;
  int rc = gufo::BuildExpertBank(ctx, *bank, &built);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  if (stride < bank->experts + 1) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe layer: the shared expert's logit follows the experts'");
  }
  if (x_stride != 0 && x_stride < bank->hidden) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe layer: x_stride is 0 (shared input) or at least hidden");
  }
  rc = gufo::EnqueueRoute(ctx, router, stride, tokens, bank->experts, k, chosen, weights, scale);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  return gufo::EnqueueMoeFfn(ctx, built, chosen, weights, scale, tokens, k, x, static_cast<int>(x_stride), shared, ffn,
                             act, expert_out, out, true);
}

int gufo_cuda_moe_combine_device(gufo_cuda_ctx* ctx, const float* shared, const float* scale, const float* weights,
                                 const float* expert_out, int tokens, int k, int hidden, float* out) {
  if (ctx == nullptr || shared == nullptr || scale == nullptr || weights == nullptr || expert_out == nullptr ||
      out == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "moe combine: null pointer");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  return gufo::EnqueueMoeCombine(ctx, shared, scale, weights, expert_out, tokens, k, hidden, out);
}

}  // extern "C"
