// The Gated DeltaNet decode step (Mixer::Linear,
// src/models/qwen35/decoder.cpp:161-265 in the reference; its delta rule,
// lines 234-257, restated blockwise in src/models/qwen35_2b/deltanet.cpp:56-82).
//
// Per value head the fp32 state S[i (key)][j (value)] is read from HBM once,
// kept on chip across the retrieval pass (u = (decay S)^T k), the rank-1 update
// (S' = decay S + k delta^T) and the readout (y = S'^T q), and written once:
// algorithmic traffic is 2 * dk * dk * 4 bytes per head, the HBM roofline of
// this kernel. Columns of S evolve independently
// (src/models/qwen35/prefill_mixer.cpp:662-667), so one thread block takes one
// (sequence, value head) and each of its warps one tile of 32 columns.
//
// Warp layout: lane = 8 * ig + jq; jq owns four adjacent columns (one float4),
// ig owns rows ig, ig + 4, ..., so one load instruction of a warp covers four
// 128-byte row segments. A lane keeps its dk / 4 float4 of S (128 registers at
// dk = 128) from the loads to the stores: all of a tile's state is requested
// from HBM at once, the column sums of the two passes need only two shuffle
// steps, and the block meets just once, for the gated RMSNorm over the head's
// dk outputs.
#include "common.cuh"

#include <vector>

namespace gufo {

constexpr int kMaxHeadDim = 128;
constexpr int kDeltaThreads = kMaxHeadDim;            // one thread per column
constexpr int kMaxSeqs = 64;                          // descriptors per launch
constexpr int kMaxRunTokens = 4;                      // tokens of a sequence per launch

struct DeltaRuleArgs {
  gufo_cuda_delta_seq seq[kMaxSeqs];
  int key_heads;
  int value_heads;
  int head_dim;
  int early_state;   // as in LinearArgs below
};

struct LinearShape {
  int key_heads;
  int value_heads;
  int head_dim;
  int conv_kernel;
  float rms_eps;
  const float* conv;
  const float* ssm_a;
  const float* dt_bias;
  const float* ssm_norm;
  // When the caller knows that no kernel shortly before this one in the stream
  // wrote the states, their loads may start ahead of the dependency wait.
  int early_state;
  // Non-null alpha_w: the gates come from these rows instead of the input row.
  DeltaNetGateRows gate_rows;
};

// A launch of up to SEQS sequences (a decode step's one travels light).
template <int SEQS>
struct LinearArgs {
  LinearShape shape;
  DeltaNetSeq seq[SEQS];
};

namespace {

// A warp's tile of COLS (8 or 16) adjacent columns of a head's state: a lane
// holds rows ig, ig + 32 / G, ... (ig = lane / G, G = COLS / 4) of four adjacent
// columns (4 * (lane % G)). Narrow tiles mean many warps per head.
template <int COLS>
struct NarrowTile {
  static constexpr int kGroups = COLS / 4;                 // lanes across the columns
  static constexpr int kRowGroups = 32 / kGroups;
  static constexpr int kRowsPerLane = kMaxHeadDim / kRowGroups;
  float4 s[kRowsPerLane];
};

template <int COLS>
__device__ __forceinline__ void LoadNarrowTile(NarrowTile<COLS>& tile, const float* __restrict__ src, int dk,
                                               int tile_index) {
  using T = NarrowTile<COLS>;
  const int lane = threadIdx.x & 31;
  const int col = tile_index * COLS + 4 * (lane % T::kGroups);
  const int ig = lane / T::kGroups;
  const int rows = dk / T::kRowGroups;
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      tile.s[r] = *reinterpret_cast<const float4*>(src + static_cast<size_t>(r * T::kRowGroups + ig) * dk + col);
    }
  }
}

// Sum over the warp's row groups; every lane gets its columns' totals.
template <int COLS>
__device__ __forceinline__ float4 NarrowColumnSum(float4 v) {
#pragma unroll
  for (int o = NarrowTile<COLS>::kGroups; o <= 16; o <<= 1) {
    v.x += __shfl_xor_sync(0xFFFFFFFFu, v.x, o);
    v.y += __shfl_xor_sync(0xFFFFFFFFu, v.y, o);
    v.z += __shfl_xor_sync(0xFFFFFFFFu, v.z, o);
    v.w += __shfl_xor_sync(0xFFFFFFFFu, v.w, o);
  }
  return v;
}

// The delta rule on this warp's column tile, which becomes S'. Writes S' to dst
// (may be null) and the tile's outputs to out (no barrier); with `squares`, lane 0
// also leaves the sum of the squares of the tile's outputs there. q, k, v: the
// head's vectors in shared memory.
template <int COLS>
__device__ __forceinline__ void NarrowDeltaTile(NarrowTile<COLS>& tile, float* __restrict__ dst, int dk,
                                                int tile_index, const float* q, const float* k, const float* v_in,
                                                float decay, float beta, float* out, float* squares = nullptr) {
  using T = NarrowTile<COLS>;
  const int lane = threadIdx.x & 31;
  const int col = tile_index * COLS + 4 * (lane % T::kGroups);
  const int ig = lane / T::kGroups;
  const int rows = dk / T::kRowGroups;
  float4 (&s)[T::kRowsPerLane] = tile.s;
  // Pass 1: u_j = sum_i S_ij * (k_i * decay).
  float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      const float ki = k[r * T::kRowGroups + ig] * decay;
      u.x = fmaf(s[r].x, ki, u.x);
      u.y = fmaf(s[r].y, ki, u.y);
      u.z = fmaf(s[r].z, ki, u.z);
      u.w = fmaf(s[r].w, ki, u.w);
    }
  }
  u = NarrowColumnSum<COLS>(u);
  const float4 v = *reinterpret_cast<const float4*>(&v_in[col]);
  float4 delta;
  delta.x = beta * (v.x - u.x);
  delta.y = beta * (v.y - u.y);
  delta.z = beta * (v.z - u.z);
  delta.w = beta * (v.w - u.w);
  // Pass 2: S'_ij = S_ij * decay + k_i * delta_j; y_j = sum_i S'_ij * q_i.
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      const int i = r * T::kRowGroups + ig;
      const float ki = k[i];
      const float qi = q[i];
      float4 n;
      n.x = fmaf(s[r].x, decay, ki * delta.x);
      n.y = fmaf(s[r].y, decay, ki * delta.y);
      n.z = fmaf(s[r].z, decay, ki * delta.z);
      n.w = fmaf(s[r].w, decay, ki * delta.w);
      if (dst != nullptr) {
        *reinterpret_cast<float4*>(dst + static_cast<size_t>(i) * dk + col) = n;
      }
      s[r] = n;
      y.x = fmaf(n.x, qi, y.x);
      y.y = fmaf(n.y, qi, y.y);
      y.z = fmaf(n.z, qi, y.z);
      y.w = fmaf(n.w, qi, y.w);
    }
  }
  y = NarrowColumnSum<COLS>(y);
  if (ig == 0) {
    *reinterpret_cast<float4*>(&out[col]) = y;
  }
  if (squares != nullptr) {
    // Lanes 0 .. kGroups - 1 hold the tile's COLS outputs.
    float sq = ig == 0 ? y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w : 0.f;
#pragma unroll
    for (int o = T::kGroups / 2; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
    }
    if (lane == 0) {
      *squares = sq;
    }
  }
}

constexpr int kStepCols = 16;   // columns per warp in the decode step's kernel
constexpr int kRuleCols = 16;   // and in the stand-alone delta rule (8: 4.9 us for config 3, 16: 4.1, 32: 4.6)

// Gates given: one warp per thread block, grid = (dk / 16, value_heads,
// sequences). The tiles of a head need nothing from one another here, and
// many small blocks per SM let one tile's stores overlap another's loads
// (16-column tiles: 1024 warps for eight sequences of sixteen heads).
__global__ void __launch_bounds__(32)
DeltaRuleKernel(const __grid_constant__ DeltaRuleArgs args) {
  __shared__ __align__(16) float q[kMaxHeadDim], k[kMaxHeadDim], v[kMaxHeadDim], y[kMaxHeadDim];
  const gufo_cuda_delta_seq& seq = args.seq[blockIdx.z];
  const int head = blockIdx.y;
  const int tile = blockIdx.x;
  const int dk = args.head_dim;
  const int kh = head % args.key_heads;
  const int lane = threadIdx.x;
  const size_t state_at = static_cast<size_t>(head) * dk * dk;
  NarrowTile<kRuleCols> state;
  GridLaunchDependents();
  if (args.early_state) {
    LoadNarrowTile(state, seq.state + state_at, dk, tile);
  }
  GridDependencyWait();
  if (!args.early_state) {
    LoadNarrowTile(state, seq.state + state_at, dk, tile);
  }
  for (int i = lane; i < dk; i += 32) {
    q[i] = seq.q[kh * dk + i];
    k[i] = seq.k[kh * dk + i];
  }
  if (lane < kRuleCols) {
    v[tile * kRuleCols + lane] = seq.v[head * dk + tile * kRuleCols + lane];
  }
  const float decay = seq.decay[head], beta = seq.beta[head];
  __syncwarp();
  float* dst = (seq.state_out != nullptr ? seq.state_out : seq.state) + state_at;
  NarrowDeltaTile(state, dst, dk, tile, q, k, v, decay, beta, y);
  __syncwarp();
  if (lane < kRuleCols) {
    seq.y[head * dk + tile * kRuleCols + lane] = y[tile * kRuleCols + lane];
  }
}

__device__ __forceinline__ float Sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float Silu(float x) { return x * Sigmoid(x); }
__device__ __forceinline__ float Softplus(float x) {
  return x > 20.0f ? x : log1pf(expf(x));
}

// Mixer::Linear for one (sequence, value head), up to TOK tokens. grid =
// (value_heads, sequences), 2 * dk threads: thread t < dk owns channel t of the
// head's q and k and output t of the epilogue, thread dk + t channel t of v; warp w
// owns columns 16 w .. 16 w + 15 of the state. (With dk threads and 32 columns per
// warp the kernel spent 6.5 us per layer of the decode step on four warps' worth of
// dependent instructions.)
//
// All that does not need the state - convolutions, gates, norms of every token -
// is done first, for all tokens at once and under the state's load; the tokens then
// follow one another on the state in registers with no block barrier between them
// (a warp's columns need nothing from the others'), and the gated norms of all
// tokens close the block. The state is read once and written once (a draft's once
// more) whatever the tokens: as a launch per token index, 32 sequences of 32 heads
// with one to four tokens took 110 us and moved the states up to eight times.
template <int TOK>
struct LinearShared {
  float q[TOK][kMaxHeadDim];
  float k[TOK][kMaxHeadDim];
  float v[TOK][kMaxHeadDim];
  float y[TOK][kMaxHeadDim];
  float gate[TOK][2];                                  // decay, beta
  float scratch[(2 * kDeltaThreads / 32) * 5 * TOK];   // five sums a token and warp
};

template <int TOK, int WIN, int SEQS>
__global__ void __launch_bounds__(2 * kDeltaThreads, SEQS > 2 ? 2 : 1)
DeltaNetLinearKernel(const __grid_constant__ LinearArgs<SEQS> args) {
  __shared__ __align__(16) LinearShared<TOK> sh;
  const LinearShape& a = args.shape;
  const DeltaNetSeq& seq = args.seq[blockIdx.y];
  const int n = TOK == 1 ? 1 : seq.tokens;
  const int head = blockIdx.x;
  const int hk = a.key_heads;
  const int hv = a.value_heads;
  const int dk = a.head_dim;
  const int threads = 2 * dk;
  const int warps = threads / 32;
  const int key_dim = hk * dk;
  const int value_dim = hv * dk;
  const int channels = 2 * key_dim + value_dim;
  const int kernel = a.conv_kernel;
  const int window = kernel - 1;      // at most WIN
  const int kh = head % hk;
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const bool lower = tid < dk;        // q and k channels, the epilogue
  const int ch = lower ? tid : tid - dk;
  const size_t state_at = static_cast<size_t>(head) * dk * dk;
  NarrowTile<kStepCols> state_tile;
  // Causal depthwise conv + SiLU of a channel; its window moves on in registers.
  // All loads of a thread's channels are issued before the first store, so they
  // overlap.
  struct Taps {
    float old[WIN];
    float w[WIN + 1];
  };
  // The layer's weights never depend on the kernels before this one.
  auto fetch_weights = [&](int c, Taps& taps) {
    const float* kw = a.conv + static_cast<size_t>(c) * kernel;
#pragma unroll
    for (int t = 0; t < WIN; ++t) {
      taps.w[t] = t < window ? kw[t] : 0.f;
    }
    taps.w[WIN] = kw[window];
  };
  // The window is state: written a step ago (early_state) or by the launch
  // just before this one.
  auto fetch_window = [&](int c, Taps& taps) {
#pragma unroll
    for (int t = 0; t < WIN; ++t) {
      taps.old[t] = t < window ? seq.conv_in[static_cast<size_t>(t) * channels + c] : 0.f;
    }
  };
  auto conv = [&](Taps& taps, float cur) -> float {
    float acc = taps.w[WIN] * cur;
#pragma unroll
    for (int t = 0; t < WIN; ++t) {
      if (t < window) {
        acc = fmaf(taps.w[t], taps.old[t], acc);
      }
    }
#pragma unroll
    for (int t = 0; t < WIN; ++t) {
      taps.old[t] = t == window - 1 ? cur : (t + 1 < WIN ? taps.old[t + 1] : cur);
    }
    return Silu(acc);
  };
  auto store_window = [&](float* to, int c, const Taps& taps) {
#pragma unroll
    for (int t = 0; t < WIN; ++t) {
      if (t < window) {
        to[static_cast<size_t>(t) * channels + c] = taps.old[t];
      }
    }
  };
  // The window of the key head's q and k channels is advanced by the first
  // value head that reads the key head; every head advances its own v.
  // A lower thread convolves q (ta) and k (tb) of its channel, an upper one v (ta).
  const int ch_a = lower ? kh * dk + ch : 2 * key_dim + head * dk + ch;
  const int ch_b = key_dim + kh * dk + ch;
  const bool owner = !lower || head < hk;
  Taps ta, tb;
  // The first passes of the head's alpha and beta rows (weights as well).
  constexpr int kGateAhead = 2;
  const DeltaNetGateRows& g = a.gate_rows;
  const bool gate_rows = g.alpha_w != nullptr;
  const float4* wa = reinterpret_cast<const float4*>(g.alpha_w + static_cast<size_t>(head) * g.cols);
  const float4* wb = reinterpret_cast<const float4*>(g.beta_w + static_cast<size_t>(head) * g.cols);
  const float4* norm = reinterpret_cast<const float4*>(g.norm_w);
  const float4 one4 = make_float4(1.f, 1.f, 1.f, 1.f);
  float4 wa_ahead[kGateAhead], wb_ahead[kGateAhead], nw_ahead[kGateAhead];
  GridLaunchDependents();
  if (a.early_state) {
    LoadNarrowTile(state_tile, seq.ssm_in + state_at, dk, warp);
    fetch_window(ch_a, ta);
    if (lower) {
      fetch_window(ch_b, tb);
    }
  }
  fetch_weights(ch_a, ta);
  if (lower) {
    fetch_weights(ch_b, tb);
  }
  if (gate_rows) {
#pragma unroll
    for (int j = 0; j < kGateAhead; ++j) {
      const int i = tid + j * threads;
      if (i < g.cols / 4) {
        wa_ahead[j] = wa[i];
        wb_ahead[j] = wb[i];
        nw_ahead[j] = norm != nullptr ? norm[i] : one4;
      }
    }
  }
  const float norm_w = lower ? a.ssm_norm[ch] : 0.f;
  const float ssm_a = a.ssm_a[head], dt_bias = a.dt_bias[head];
  GridDependencyWait();
  if (!a.early_state) {
    LoadNarrowTile(state_tile, seq.ssm_in + state_at, dk, warp);
    fetch_window(ch_a, ta);
    if (lower) {
      fetch_window(ch_b, tb);
    }
  }
  // What the tokens bring, the epilogue's z included, requested at once.
  float cur_a[TOK], cur_b[TOK], z[TOK];
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    cur_a[t] = cur_b[t] = z[t] = 0.f;
    if (t < n) {
      const float* in = seq.in + t * seq.in_stride;
      cur_a[t] = in[ch_a];
      if (lower) {
        cur_b[t] = in[ch_b];
        z[t] = in[channels + head * dk + ch];
      }
    }
  }
  // Five sums a token: the gate input's squares, the two gate dots, the q and k
  // norms' squares; one block-wide reduction for all of them.
  float sums[TOK][5];
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      sums[t][i] = 0.f;
    }
  }
  if (gate_rows) {
    // The head's alpha and beta rows against the normed input, one float4 per
    // thread and pass (GgufProjections serves these F32 rows through its own
    // dot, src/models/qwen35/gguf_projections.cpp:162-170). With norm weights
    // the input is the residual stream and the RMS norm is applied on the way
    // (DeltaNetStep::Run, src/models/qwen35_2b/deltanet.cpp:358-392): the dots are
    // taken against x * w and scaled by the norm's 1 / rms afterwards (a scalar).
    auto pass = [&](int i, const float4& nw, const float4& av, const float4& bv) {
      float4 xv[TOK];
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        xv[t] = t < n ? *(reinterpret_cast<const float4*>(seq.x + t * seq.x_stride) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        sums[t][0] += xv[t].x * xv[t].x + xv[t].y * xv[t].y + xv[t].z * xv[t].z + xv[t].w * xv[t].w;
        const float4 x = make_float4(xv[t].x * nw.x, xv[t].y * nw.y, xv[t].z * nw.z, xv[t].w * nw.w);
        sums[t][1] += av.x * x.x + av.y * x.y + av.z * x.z + av.w * x.w;
        sums[t][2] += bv.x * x.x + bv.y * x.y + bv.z * x.z + bv.w * x.w;
      }
    };
#pragma unroll
    for (int j = 0; j < kGateAhead; ++j) {
      const int i = tid + j * threads;
      if (i < g.cols / 4) {
        pass(i, nw_ahead[j], wa_ahead[j], wb_ahead[j]);
      }
    }
    for (int i = tid + kGateAhead * threads; i < g.cols / 4; i += threads) {
      pass(i, norm != nullptr ? norm[i] : one4, wa[i], wb[i]);
    }
  }
  float qv[TOK], kv[TOK];
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    qv[t] = kv[t] = 0.f;
    if (t < n) {
      const float first = conv(ta, cur_a[t]);
      if (lower) {
        qv[t] = first;
        kv[t] = conv(tb, cur_b[t]);
      } else {
        sh.v[t][ch] = first;
      }
      if (owner && t >= n - 2) {
        float* to = t == n - 1 ? seq.conv_out : seq.conv_saved;
        store_window(to, ch_a, ta);
        if (lower) {
          store_window(to, ch_b, tb);
        }
      }
      sums[t][3] = qv[t] * qv[t];
      sums[t][4] = kv[t] * kv[t];
    }
  }
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    if (t < n) {
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const float total = WarpSum(sums[t][i]);
        if (lane == 0) {
          sh.scratch[(warp * TOK + t) * 5 + i] = total;
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    if (t < n) {
      // Every thread needs its token's q / k sums, the gates' lanes the others.
      float qq = 0.f, kk = 0.f;
      for (int w = 0; w < warps; ++w) {
        qq += sh.scratch[(w * TOK + t) * 5 + 3];
        kk += sh.scratch[(w * TOK + t) * 5 + 4];
      }
      // L2 norms (+1e-6 under the root); q also takes 1/sqrt(dk).
      if (lower) {
        sh.q[t][ch] = qv[t] * ((1.0f / sqrtf(qq + 1e-6f)) * (1.0f / sqrtf(static_cast<float>(dk))));
        sh.k[t][ch] = kv[t] * (1.0f / sqrtf(kk + 1e-6f));
      }
    }
  }
  // The gates by lanes of the first upper warp: token tid / 2, decay and beta.
  if (!lower && ch < 2 * n) {
    const int t = ch >> 1, which = ch & 1;
    float dot;
    if (gate_rows) {
      float sq = 0.f;
      dot = 0.f;
      for (int w = 0; w < warps; ++w) {
        sq += sh.scratch[(w * TOK + t) * 5];
        dot += sh.scratch[(w * TOK + t) * 5 + 1 + which];
      }
      if (norm != nullptr) {
        dot *= 1.0f / sqrtf(sq / static_cast<float>(g.cols) + g.eps);
      }
    } else {
      dot = seq.in[t * seq.in_stride + channels + value_dim + which * hv + head];   // alpha | beta follow z
    }
    sh.gate[t][which] = which == 0 ? expf(ssm_a * Softplus(dot + dt_bias)) : Sigmoid(dot);
  }
  __syncthreads();
  // (The scratch's last readers passed the barrier above.)
#pragma unroll
  for (int t = 0; t < TOK; ++t) {
    if (t < n) {
      float* dst = t == n - 1 ? seq.ssm_last + state_at : (t == n - 2 ? seq.ssm + state_at : nullptr);
      NarrowDeltaTile(state_tile, dst, dk, warp, sh.q[t], sh.k[t], sh.v[t], sh.gate[t][0], sh.gate[t][1], sh.y[t],
                      &sh.scratch[t * warps + warp]);
    }
  }
  // Gated RMSNorm over the head's dk outputs: RMS(o) * w * silu(z); the warps'
  // tiles left their outputs' squares, so one barrier serves both.
  __syncthreads();
  if (lower) {
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      if (t < n) {
        float total = 0.f;
        for (int w = 0; w < warps; ++w) {
          total += sh.scratch[t * warps + w];
        }
        const float inv = 1.0f / sqrtf(total / static_cast<float>(dk) + a.rms_eps);
        seq.y[t * seq.y_stride + head * dk + ch] = sh.y[t][ch] * inv * norm_w * Silu(z[t]);
      }
    }
  }
}

int CheckHeads(int key_heads, int value_heads, int head_dim) {
  if (key_heads <= 0 || value_heads <= 0 || value_heads % key_heads != 0) {
    return Fail(GUFO_CUDA_SHAPE, "deltanet: value heads must tile the key heads");
  }
  if (head_dim <= 0 || head_dim > kMaxHeadDim || head_dim % 32 != 0) {
    return Fail(GUFO_CUDA_SHAPE,
                "deltanet: unsupported head dim " + std::to_string(head_dim) +
                    " (multiples of 32 up to 128)");
  }
  return GUFO_CUDA_OK;
}

}  // namespace
}  // namespace gufo

using gufo::Fail;

extern "C" {

int gufo_cuda_delta_rule_device(gufo_cuda_ctx* ctx,
                                const gufo_cuda_delta_seq* seqs, int nseq,
                                int key_heads, int value_heads, int head_dim) {
  if (ctx == nullptr || (seqs == nullptr && nseq > 0)) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "delta_rule: null pointer");
  }
  if (nseq < 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "delta_rule: negative sequence count");
  }
  int rc = gufo::CheckHeads(key_heads, value_heads, head_dim);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  for (int s = 0; s < nseq; ++s) {
    const gufo_cuda_delta_seq& q = seqs[s];
    if (q.state == nullptr || q.q == nullptr || q.k == nullptr || q.v == nullptr ||
        q.decay == nullptr || q.beta == nullptr || q.y == nullptr) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "delta_rule: null pointer in a sequence");
    }
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  for (int s0 = 0; s0 < nseq; s0 += gufo::kMaxSeqs) {
    const int n = nseq - s0 < gufo::kMaxSeqs ? nseq - s0 : gufo::kMaxSeqs;
    gufo::DeltaRuleArgs args{};
    for (int s = 0; s < n; ++s) {
      args.seq[s] = seqs[s0 + s];
    }
    args.key_heads = key_heads;
    args.value_heads = value_heads;
    args.head_dim = head_dim;
    args.early_state = ctx->early_state ? 1 : 0;
    const dim3 grid(head_dim / gufo::kRuleCols, value_heads, n);
    GUFO_CUDA_TRY(gufo::LaunchOverlapped(gufo::DeltaRuleKernel, grid, dim3(32), 0,
                                         ctx->stream, 1, args));
    ctx->launches.fetch_add(1);
  }
  return GUFO_CUDA_OK;
}

int gufo_cuda_deltanet_layer_create(gufo_cuda_ctx* ctx,
                                    const gufo_cuda_deltanet_params* p,
                                    gufo_cuda_deltanet_layer* out) {
  if (ctx == nullptr || p == nullptr || out == nullptr || p->conv == nullptr ||
      p->ssm_a == nullptr || p->dt_bias == nullptr || p->ssm_norm == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_layer_create: null pointer");
  }
  int rc = gufo::CheckHeads(p->key_heads, p->value_heads, p->head_dim);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  if (p->conv_kernel < 2 || p->conv_kernel > 8) {
    return Fail(GUFO_CUDA_SHAPE, "deltanet: conv kernel must be 2..8 taps");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  gufo::DeltaNetLayer layer;
  layer.key_heads = p->key_heads;
  layer.value_heads = p->value_heads;
  layer.head_dim = p->head_dim;
  layer.conv_kernel = p->conv_kernel;
  layer.rms_eps = p->rms_eps;
  const size_t channels =
      static_cast<size_t>(2 * p->key_heads + p->value_heads) * p->head_dim;
  struct Copy {
    float** dst;
    const float* src;
    size_t n;
  } copies[] = {{&layer.conv, p->conv, channels * p->conv_kernel},
                {&layer.ssm_a, p->ssm_a, static_cast<size_t>(p->value_heads)},
                {&layer.dt_bias, p->dt_bias, static_cast<size_t>(p->value_heads)},
                {&layer.ssm_norm, p->ssm_norm, static_cast<size_t>(p->head_dim)}};
  for (auto& c : copies) {
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(c.dst), c.n * 4);
    if (e == cudaSuccess) {
      e = cudaMemcpyAsync(*c.dst, c.src, c.n * 4, cudaMemcpyHostToDevice, ctx->stream);
    }
    if (e != cudaSuccess) {
      cudaFree(layer.conv);
      cudaFree(layer.ssm_a);
      cudaFree(layer.dt_bias);
      cudaFree(layer.ssm_norm);
      return gufo::CudaFail(e, "deltanet_layer_create");
    }
  }
  GUFO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  const int64_t id = ctx->next_id++;
  ctx->deltanet_layers.emplace(id, layer);
  *out = id;
  return GUFO_CUDA_OK;
}

int gufo_cuda_deltanet_layer_free(gufo_cuda_ctx* ctx,
                                  gufo_cuda_deltanet_layer layer) {
  if (ctx == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_layer_free: ctx is null");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  auto it = ctx->deltanet_layers.find(layer);
  if (it == ctx->deltanet_layers.end()) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_layer_free: unknown handle");
  }
  GUFO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  cudaFree(it->second.conv);
  cudaFree(it->second.ssm_a);
  cudaFree(it->second.dt_bias);
  cudaFree(it->second.ssm_norm);
  ctx->deltanet_layers.erase(it);
  return GUFO_CUDA_OK;
}

int gufo_cuda_deltanet_linear_device(gufo_cuda_ctx* ctx,
                                     gufo_cuda_deltanet_layer layer,
                                     const gufo_cuda_linear_seq* seqs, int nseq) {
  if (ctx == nullptr || (seqs == nullptr && nseq > 0)) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_linear: null pointer");
  }
  if (nseq < 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_linear: negative sequence count");
  }
  for (int s = 0; s < nseq; ++s) {
    const gufo_cuda_linear_seq& q = seqs[s];
    if (q.in == nullptr || q.conv_in == nullptr || q.conv_out == nullptr ||
        q.ssm == nullptr || q.y == nullptr) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_linear: null pointer in a sequence");
    }
    if (q.conv_in == q.conv_out) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT,
                  "deltanet_linear: conv_in and conv_out must be distinct buffers");
    }
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  auto it = ctx->deltanet_layers.find(layer);
  if (it == ctx->deltanet_layers.end()) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_linear: unknown layer handle");
  }
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  std::vector<gufo::DeltaNetSeq> step(nseq);
  for (int s = 0; s < nseq; ++s) {
    const gufo_cuda_linear_seq& q = seqs[s];
    step[s] = gufo::OneTokenSeq(q.in, nullptr, q.conv_in, q.conv_out, q.ssm, q.ssm_out != nullptr ? q.ssm_out : q.ssm, q.y);
  }
  return gufo::EnqueueDeltaNetLinear(ctx, it->second, step.data(), nseq, ctx->early_state);
}

int gufo_cuda_deltanet_step_device(gufo_cuda_ctx* ctx, gufo_cuda_deltanet_layer layer, gufo_cuda_matrix ssm_alpha,
                                   gufo_cuda_matrix ssm_beta, const float* attn_norm, float rms_eps,
                                   const gufo_cuda_deltanet_step_seq* seqs, int nseq) {
  if (ctx == nullptr || attn_norm == nullptr || (seqs == nullptr && nseq > 0)) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: null pointer");
  }
  if (nseq < 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: negative sequence count");
  }
  int most = 0;
  for (int s = 0; s < nseq; ++s) {
    const gufo_cuda_deltanet_step_seq& q = seqs[s];
    if (q.n_tokens < 1 || q.n_tokens > 4) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: 1 to 4 tokens per sequence");
    }
    if (q.in == nullptr || q.h == nullptr || q.conv_in == nullptr || q.conv_out == nullptr || q.ssm == nullptr ||
        q.y == nullptr || (q.n_tokens >= 2 && (q.conv_saved == nullptr || q.ssm_spec == nullptr))) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: null pointer in a sequence");
    }
    if (q.conv_in == q.conv_out || q.conv_in == q.conv_saved || q.conv_out == q.conv_saved) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: the conv windows must be distinct buffers");
    }
    if ((reinterpret_cast<uintptr_t>(q.h) & 15) != 0 || q.h_stride % 4 != 0) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: residual rows must be 16-byte aligned");
    }
    most = q.n_tokens > most ? q.n_tokens : most;
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  auto it = ctx->deltanet_layers.find(layer);
  if (it == ctx->deltanet_layers.end()) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "deltanet_step: unknown layer handle");
  }
  const gufo::Matrix* alpha = ctx->FindMatrix(ssm_alpha);
  const gufo::Matrix* beta = ctx->FindMatrix(ssm_beta);
  if (alpha == nullptr || beta == nullptr || alpha->type != GUFO_CUDA_F32 || beta->type != GUFO_CUDA_F32 ||
      alpha->rows != it->second.value_heads || beta->rows != alpha->rows || beta->cols != alpha->cols ||
      alpha->cols % 4 != 0) {
    return Fail(GUFO_CUDA_SHAPE, "deltanet_step: ssm_alpha / ssm_beta must be F32 [hidden, value heads]");
  }
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  gufo::DeltaNetGateRows gates{};
  gates.alpha_w = reinterpret_cast<const float*>(alpha->data);
  gates.beta_w = reinterpret_cast<const float*>(beta->data);
  gates.cols = static_cast<int>(alpha->cols);
  gates.norm_w = attn_norm;
  gates.eps = rms_eps;
  // Sequences of the most tokens first: their blocks run longest.
  std::vector<gufo::DeltaNetSeq> step;
  step.reserve(nseq);
  for (int n = most; n >= 1; --n) {
    for (int s = 0; s < nseq; ++s) {
      const gufo_cuda_deltanet_step_seq& q = seqs[s];
      if (q.n_tokens == n) {
        step.push_back({q.in, q.h, q.conv_in, q.conv_saved, q.conv_out, q.ssm, q.ssm, n >= 2 ? q.ssm_spec : q.ssm, q.y,
                        q.in_stride, q.h_stride, q.y_stride, n});
      }
    }
  }
  // States may be written by the launch before this one: no early state loads.
  return gufo::EnqueueDeltaNetLinear(ctx, it->second, step.data(), nseq, false, &gates);
}

}  // extern "C"

namespace gufo {

namespace {

template <int TOK, int WIN, int SEQS>
int LaunchLinear(gufo_cuda_ctx* ctx, const LinearShape& shape, const DeltaNetSeq* seqs, int n) {
  LinearArgs<SEQS> args;
  args.shape = shape;
  for (int s = 0; s < n; ++s) {
    args.seq[s] = seqs[s];
  }
  GUFO_CUDA_TRY(LaunchOverlapped(DeltaNetLinearKernel<TOK, WIN, SEQS>, dim3(shape.value_heads, n), dim3(2 * shape.head_dim),
                                 0, ctx->stream, 1, args));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

template <int TOK>
int LaunchTokens(gufo_cuda_ctx* ctx, const LinearShape& shape, const DeltaNetSeq* seqs, int n) {
  // One or two sequences (a decode step) in a small argument block; windows of
  // up to three columns (four taps, the models' own) in few registers.
  const bool narrow = shape.conv_kernel <= 4;
  if (n <= 2) {
    return narrow ? LaunchLinear<TOK, 3, 2>(ctx, shape, seqs, n) : LaunchLinear<TOK, 7, 2>(ctx, shape, seqs, n);
  }
  return narrow ? LaunchLinear<TOK, 3, kMaxSeqs>(ctx, shape, seqs, n) : LaunchLinear<TOK, 7, kMaxSeqs>(ctx, shape, seqs, n);
}

}  // namespace

int EnqueueDeltaNetLinear(gufo_cuda_ctx* ctx, const DeltaNetLayer& l, const DeltaNetSeq* seqs, int nseq,
                          bool early_state, const DeltaNetGateRows* gate_rows) {
  LinearShape shape{};
  shape.key_heads = l.key_heads;
  shape.value_heads = l.value_heads;
  shape.head_dim = l.head_dim;
  shape.conv_kernel = l.conv_kernel;
  shape.rms_eps = l.rms_eps;
  shape.conv = l.conv;
  shape.ssm_a = l.ssm_a;
  shape.dt_bias = l.dt_bias;
  shape.ssm_norm = l.ssm_norm;
  shape.early_state = early_state ? 1 : 0;
  if (gate_rows != nullptr) {
    shape.gate_rows = *gate_rows;
  }
  for (int s0 = 0; s0 < nseq; s0 += kMaxSeqs) {
    const int n = nseq - s0 < kMaxSeqs ? nseq - s0 : kMaxSeqs;
    int most = 1;
    for (int s = s0; s < s0 + n; ++s) {
      most = seqs[s].tokens > most ? seqs[s].tokens : most;
    }
    const int rc = most == 1   ? LaunchTokens<1>(ctx, shape, seqs + s0, n)
                   : most == 2 ? LaunchTokens<2>(ctx, shape, seqs + s0, n)
                               : LaunchTokens<kMaxRunTokens>(ctx, shape, seqs + s0, n);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  return GUFO_CUDA_OK;
}

}  // namespace gufo
