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
// (sequence, value head) and each of its eight warps one tile of 16 columns.
//
// Warp layout: lane = 4 * ig + jq; jq owns four adjacent columns (one float4), ig
// owns rows ig, ig + 8, ..., so one load instruction of a warp covers eight 64-byte
// row segments. A lane keeps its dk / 8 float4 of S (64 registers at dk = 128) from
// the loads to the stores: all of a tile's state is requested from HBM at once, the
// column sums need three shuffle steps, and the block meets just once more, for the
// gated RMSNorm over the head's dk outputs.
#include "common.cuh"

#include <vector>

namespace gufo {

constexpr int kMaxHeadDim = 128;
constexpr int kDeltaThreads = kMaxHeadDim;            // one thread per column
constexpr int kMaxSeqs = 64;                          // descriptors per launch
constexpr int kMaxRunTokens = 4;                      // tokens of a sequence per launch

template <int SEQS>
struct DeltaRuleArgs {
  gufo_cuda_delta_seq seq[SEQS];
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
  // Given gates (DeltaNetSeq::gates): floats between a token's heads, and from a head's
  // alpha dot to its beta dot.
  int gate_apart;
  int gate_beta;
};

// A launch of up to SEQS sequences (a decode step's one travels light).
template <int SEQS>
struct LinearArgs {
  LinearShape shape;
  DeltaNetSeq seq[SEQS];
};

namespace {

// Two fp32 values in a register pair and the packed instructions on them: half
// the issue slots of the delta rule's arithmetic.
using Pair = unsigned long long;
__device__ __forceinline__ Pair MakePair(float a, float b) {
  Pair p;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a), "f"(b));
  return p;
}
__device__ __forceinline__ float2 Unpack(Pair p) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ Pair Fma2(Pair a, Pair b, Pair c) {
  Pair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ Pair Mul2(Pair a, Pair b) {
  Pair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// A warp's tile of COLS (8 or 16) adjacent columns of a head's state: a lane
// holds rows ig, ig + 32 / G, ... (ig = lane / G, G = COLS / 4) of four adjacent
// columns (4 * (lane % G)), as two pairs. Narrow tiles mean many warps per head.
template <int COLS>
struct NarrowTile {
  static constexpr int kGroups = COLS / 4;                 // lanes across the columns
  static constexpr int kRowGroups = 32 / kGroups;
  static constexpr int kRowsPerLane = kMaxHeadDim / kRowGroups;
  ulonglong2 s[kRowsPerLane];
};

template <int DK, int COLS>
__device__ __forceinline__ void LoadNarrowTile(NarrowTile<COLS>& tile, const float* __restrict__ src, int dk,
                                               int tile_index) {
  using T = NarrowTile<COLS>;
  const int lane = threadIdx.x & 31;
  const int col = tile_index * COLS + 4 * (lane % T::kGroups);
  const int ig = lane / T::kGroups;
  const int rows = (DK > 0 ? DK : dk) / T::kRowGroups;
  if (DK > 0) {
    dk = DK;
  }
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      tile.s[r] = *reinterpret_cast<const ulonglong2*>(src + static_cast<size_t>(r * T::kRowGroups + ig) * dk + col);
    }
  }
}

// Scalars of one token's update, for raw k and q whose norms are factors.
struct DeltaCoef {
  float decay;
  float beta;
  float k;       // |k|^-1
  float q;       // |q|^-1 dk^-1/2
  float kq;      // k . q of the raw vectors
};

// The delta rule on this warp's column tile, which becomes S'. Per column j:
//   u = decay (S^T k)_j,  delta = beta (v_j - u),  S' = decay S + k delta^T,
//   y = (S'^T q)_j = decay (S^T q)_j + (k . q) delta:
// both sums over the rows are taken in one pass over S (TileSums, which needs none
// of the token's scalars), and the update (TileUpdate) needs no second reduction.
// k2, q2: the head's raw vectors in shared memory, every value twice. DK: the head
// dim where it is known at compile time (the models' 128), else 0.
template <int DK, int COLS>
__device__ __forceinline__ void TileSums(const NarrowTile<COLS>& tile, int dk, const Pair* q2, const Pair* k2,
                                         float (&sum)[8]) {
  using T = NarrowTile<COLS>;
  const int ig = (threadIdx.x & 31) / T::kGroups;
  const int rows = (DK > 0 ? DK : dk) / T::kRowGroups;
  Pair u01 = 0, u23 = 0, w01 = 0, w23 = 0;
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      const Pair k = k2[r * T::kRowGroups + ig], q = q2[r * T::kRowGroups + ig];
      u01 = Fma2(tile.s[r].x, k, u01);
      u23 = Fma2(tile.s[r].y, k, u23);
      w01 = Fma2(tile.s[r].x, q, w01);
      w23 = Fma2(tile.s[r].y, q, w23);
    }
  }
  const float2 a = Unpack(u01), b = Unpack(u23), d = Unpack(w01), e = Unpack(w23);
  sum[0] = a.x, sum[1] = a.y, sum[2] = b.x, sum[3] = b.y, sum[4] = d.x, sum[5] = d.y, sum[6] = e.x, sum[7] = e.y;
  // Over the warp's row groups; every lane gets its columns' totals.
#pragma unroll
  for (int o = T::kGroups; o <= 16; o <<= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      sum[i] += __shfl_xor_sync(0xFFFFFFFFu, sum[i], o);
    }
  }
}

// Writes S' to dst (may be null) and the tile's outputs to out (no barrier); with
// `squares`, lane 0 also leaves the sum of their squares there.
template <int DK, int COLS>
__device__ __forceinline__ void TileUpdate(NarrowTile<COLS>& tile, const float (&sum)[8], float* __restrict__ dst, int dk,
                                           int tile_index, const Pair* k2, const float* v_in, const DeltaCoef& c,
                                           float* out, float* squares = nullptr) {
  using T = NarrowTile<COLS>;
  const int lane = threadIdx.x & 31;
  const int col = tile_index * COLS + 4 * (lane % T::kGroups);
  const int ig = lane / T::kGroups;
  if (DK > 0) {
    dk = DK;
  }
  const int rows = dk / T::kRowGroups;
  const float4 v4 = *reinterpret_cast<const float4*>(&v_in[col]);
  const float v[4] = {v4.x, v4.y, v4.z, v4.w};
  float delta[4], y[4];
  const float u_factor = c.decay * c.k, y_factor = c.decay * c.q, kq = c.kq * c.k * c.q;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    delta[i] = c.beta * (v[i] - u_factor * sum[i]);
    y[i] = fmaf(kq, delta[i], y_factor * sum[4 + i]);
    delta[i] *= c.k;
  }
  const Pair decay = MakePair(c.decay, c.decay);
  const Pair d01 = MakePair(delta[0], delta[1]), d23 = MakePair(delta[2], delta[3]);
  float* to = dst + static_cast<size_t>(ig) * dk + col;
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      const Pair k = k2[r * T::kRowGroups + ig];
      tile.s[r].x = Fma2(tile.s[r].x, decay, Mul2(k, d01));
      tile.s[r].y = Fma2(tile.s[r].y, decay, Mul2(k, d23));
      if (dst != nullptr) {
        *reinterpret_cast<ulonglong2*>(to + r * T::kRowGroups * dk) = tile.s[r];
      }
    }
  }
  if (ig == 0) {
    *reinterpret_cast<float4*>(&out[col]) = make_float4(y[0], y[1], y[2], y[3]);
  }
  if (squares != nullptr) {
    // Lanes 0 .. kGroups - 1 hold the tile's COLS outputs.
    float sq = ig == 0 ? y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3] : 0.f;
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
constexpr int kRuleCols = 16;   // columns per warp in the stand-alone delta rule

// Gates given: one warp per thread block, grid = (dk / 16, value_heads,
// sequences). The tiles of a head need nothing from one another here, and
// many small blocks per SM let one tile's stores overlap another's loads
// (16-column tiles: 1024 warps for eight sequences of sixteen heads).
//
// What bounds it: HBM from some hundred heads on, below that the chain from a launch's
// arguments over the loads to the last store. So the arguments hold as many sequences
// as the launch needs (64 always: their kilobytes come through the constant cache ahead
// of a block's first load), the update follows the retrieval in a second pass over the
// registers instead of taking both sums in one (TileSums: eight values through the
// shuffles ahead of the first store, and k . q before them), and the head dim is a
// run-time value (built in, one sequence takes 1.2 us longer: the compiler then orders
// the loads otherwise). Sixteen warps an SM may have 128 registers each; with 96, for
// twenty warps, the loads spill. Us, states from HBM, heads x dk: 16 x 128 4.1 -> 3.2,
// 128 x 128 6.8 -> 5.7, 256 x 128 8.1 -> 6.9, 1536 x 128 36.8 -> 34.5.
template <int SEQS>
__global__ void __launch_bounds__(32, 16)
DeltaRuleKernel(const __grid_constant__ DeltaRuleArgs<SEQS> args) {
  using T = NarrowTile<kRuleCols>;
  __shared__ float q[kMaxHeadDim], k[kMaxHeadDim];
  const gufo_cuda_delta_seq& seq = args.seq[blockIdx.z];
  const int head = blockIdx.y;
  const int dk = args.head_dim;
  const int kh = head % args.key_heads;
  const int lane = threadIdx.x;
  const int col = blockIdx.x * kRuleCols + 4 * (lane % T::kGroups);
  const int ig = lane / T::kGroups;
  const int rows = dk / T::kRowGroups;
  const size_t at = static_cast<size_t>(head) * dk * dk + static_cast<size_t>(ig) * dk + col;
  float4 s[T::kRowsPerLane];
  auto load = [&]() {
    const float* src = seq.state + at;
#pragma unroll
    for (int r = 0; r < T::kRowsPerLane; ++r) {
      if (r < rows) {
        s[r] = *reinterpret_cast<const float4*>(src + r * T::kRowGroups * dk);
      }
    }
  };
  GridLaunchDependents();
  if (args.early_state) {
    load();
  }
  GridDependencyWait();
  if (!args.early_state) {
    load();
  }
  for (int i = lane; i < dk; i += 32) {
    q[i] = seq.q[kh * dk + i];
    k[i] = seq.k[kh * dk + i];
  }
  const float* v = seq.v + head * dk + col;
  const float v0 = v[0], v1 = v[1], v2 = v[2], v3 = v[3];
  const float decay = seq.decay[head], beta = seq.beta[head];
  __syncwarp();
  auto over_rows = [](float4& x) {
#pragma unroll
    for (int o = T::kGroups; o <= 16; o <<= 1) {
      x.x += __shfl_xor_sync(0xFFFFFFFFu, x.x, o);
      x.y += __shfl_xor_sync(0xFFFFFFFFu, x.y, o);
      x.z += __shfl_xor_sync(0xFFFFFFFFu, x.z, o);
      x.w += __shfl_xor_sync(0xFFFFFFFFu, x.w, o);
    }
  };
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
  over_rows(u);
  const float d0 = beta * (v0 - u.x), d1 = beta * (v1 - u.y), d2 = beta * (v2 - u.z), d3 = beta * (v3 - u.w);
  float* dst = (seq.state_out != nullptr ? seq.state_out : seq.state) + at;
  float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int r = 0; r < T::kRowsPerLane; ++r) {
    if (r < rows) {
      const float ki = k[r * T::kRowGroups + ig], qi = q[r * T::kRowGroups + ig];
      const float4 n = make_float4(fmaf(s[r].x, decay, ki * d0), fmaf(s[r].y, decay, ki * d1),
                                   fmaf(s[r].z, decay, ki * d2), fmaf(s[r].w, decay, ki * d3));
      *reinterpret_cast<float4*>(dst + r * T::kRowGroups * dk) = n;
      y.x = fmaf(n.x, qi, y.x);
      y.y = fmaf(n.y, qi, y.y);
      y.z = fmaf(n.z, qi, y.z);
      y.w = fmaf(n.w, qi, y.w);
    }
  }
  over_rows(y);
  if (ig == 0) {
    float* out = seq.y + head * dk + col;
    out[0] = y.x, out[1] = y.y, out[2] = y.z, out[3] = y.w;
  }
}

__device__ __forceinline__ float Sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
// The gates' arithmetic, spelled out: one sequence (in the mixer kernel) and several
// (DeltaNetGatesKernel) get the same bits.
__device__ __forceinline__ float Dot4(const float4& a, const float4& b, float sum) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, sum))));
}
__device__ __forceinline__ float4 Times4(const float4& a, const float4& b) {
  return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
__device__ __forceinline__ float GateInverse(float squares, int cols, float eps) {
  return 1.0f / sqrtf(squares / static_cast<float>(cols) + eps);
}
__device__ __forceinline__ float Silu(float x) { return x * Sigmoid(x); }
__device__ __forceinline__ float Softplus(float x) {
  return x > 20.0f ? x : log1pf(expf(x));
}

// Mixer::Linear for one (sequence, value head), one to four tokens. grid =
// (value_heads, sequences), 2 * dk threads: thread t < dk owns channel t of the
// head's q and k and output t of the epilogue, thread dk + t channel t of v; warp w
// owns columns 16 w .. 16 w + 15 of the state. (With dk threads and 32 columns per
// warp the decode step's kernel spent 6.5 us per layer on four warps' worth of
// dependent instructions; 8 columns and 4 * dk threads gained it nothing and cost
// 32 sequences of 32 heads 55 us instead of 48.)
//
// All that does not need the state - convolutions, gate dots - is done first, token
// after token under the state's load; then a warp each works out the tokens'
// scalars, and the tokens follow one another on the state in registers with no
// block barrier between them (a warp's columns need nothing from the others'); the
// gated norms of all tokens close the block. The state is read once and written
// once (a draft's once more) whatever the tokens. The token loops are not unrolled:
// as straight code for four tokens the kernel ran out of the instruction cache.
struct LinearShared {
  Pair q2[kMaxRunTokens][kMaxHeadDim];                 // every value twice
  Pair k2[kMaxRunTokens][kMaxHeadDim];
  float v[kMaxRunTokens][kMaxHeadDim];
  float y[kMaxRunTokens][kMaxHeadDim];
  float z[kMaxRunTokens][kMaxHeadDim];
  DeltaCoef coef[kMaxRunTokens];
  float gates[kMaxRunTokens][3][8];                   // a warp's part of the input's squares and the gate dots
  float squares[kMaxRunTokens][8];                    // a warp's part of the outputs' squares
};

template <int DK, int WIN, int SEQS>
__global__ void __launch_bounds__(2 * kDeltaThreads, SEQS > 2 ? 2 : 1)
DeltaNetLinearKernel(const __grid_constant__ LinearArgs<SEQS> args) {
  __shared__ __align__(16) LinearShared sh;
  const LinearShape& a = args.shape;
  const DeltaNetSeq& seq = args.seq[blockIdx.y];
  const int n = seq.tokens;
  const int head = blockIdx.x;
  const int hk = a.key_heads;
  const int hv = a.value_heads;
  const int dk = DK > 0 ? DK : a.head_dim;
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
  // (Launches of several sequences find the dots done, DeltaNetGatesKernel.)
  constexpr int kGateAhead = 2;
  const DeltaNetGateRows& g = a.gate_rows;
  const bool gate_rows = SEQS <= 2 && g.alpha_w != nullptr;
  const float4* wa = reinterpret_cast<const float4*>(g.alpha_w + static_cast<size_t>(head) * g.cols);
  const float4* wb = reinterpret_cast<const float4*>(g.beta_w + static_cast<size_t>(head) * g.cols);
  const float4* norm = reinterpret_cast<const float4*>(g.norm_w);
  float4 wa_ahead[kGateAhead], wb_ahead[kGateAhead];   // times the norm's weights, where it has them
  auto scaled = [&](const float4& w, int i) { return norm != nullptr ? Times4(w, norm[i]) : w; };
  GridLaunchDependents();
  if (a.early_state) {
    LoadNarrowTile<DK>(state_tile, seq.ssm_in + state_at, dk, warp);
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
        wa_ahead[j] = scaled(wa[i], i);
        wb_ahead[j] = scaled(wb[i], i);
      }
    }
  }
  const float norm_w = lower ? a.ssm_norm[ch] : 0.f;
  const float ssm_a = a.ssm_a[head], dt_bias = a.dt_bias[head];
  GridDependencyWait();
  if (!a.early_state) {
    fetch_window(ch_a, ta);
    if (lower) {
      fetch_window(ch_b, tb);
    }
  }
  // What a token brings, requested a token ahead.
  struct Row {
    float a, b, z;
    float4 x[kGateAhead];
  };
  auto fetch_row = [&](int t, Row& row) {
    const float* in = seq.in + t * seq.in_stride;
    row.a = in[ch_a];
    row.b = lower ? in[ch_b] : 0.f;
    row.z = lower ? in[channels + head * dk + ch] : 0.f;
    if (gate_rows) {
      const float4* x = reinterpret_cast<const float4*>(seq.x + t * seq.x_stride);
#pragma unroll
      for (int j = 0; j < kGateAhead; ++j) {
        const int i = tid + j * threads;
        row.x[j] = i < g.cols / 4 ? x[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
  };
  Row next;
  fetch_row(0, next);
  // The state behind what is needed first: its 64 KB take their time.
  if (!a.early_state) {
    LoadNarrowTile<DK>(state_tile, seq.ssm_in + state_at, dk, warp);
  }
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    const Row row = next;
    if (t + 1 < n) {
      fetch_row(t + 1, next);
    }
    if (gate_rows) {
      // The head's alpha and beta rows against the normed input, one float4 per
      // thread and pass (GgufProjections serves these F32 rows through its own
      // dot, src/models/qwen35/gguf_projections.cpp:162-170). With norm weights
      // the input is the residual stream and the RMS norm is applied on the way
      // (DeltaNetStep::Run, src/models/qwen35_2b/deltanet.cpp:358-392): the rows
      // carry its weights and the dots are scaled by its 1 / rms afterwards.
      float sums[3] = {};
      auto pass = [&](const float4& x, const float4& av, const float4& bv) {
        sums[0] = Dot4(x, x, sums[0]);
        sums[1] = Dot4(av, x, sums[1]);
        sums[2] = Dot4(bv, x, sums[2]);
      };
#pragma unroll
      for (int j = 0; j < kGateAhead; ++j) {
        if (tid + j * threads < g.cols / 4) {
          pass(row.x[j], wa_ahead[j], wb_ahead[j]);
        }
      }
      const float4* x = reinterpret_cast<const float4*>(seq.x + t * seq.x_stride);
      for (int i = tid + kGateAhead * threads; i < g.cols / 4; i += threads) {
        pass(x[i], scaled(wa[i], i), scaled(wb[i], i));
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        sums[i] = WarpSum(sums[i]);
      }
      if (lane < 3) {
        sh.gates[t][lane][warp] = lane == 0 ? sums[0] : (lane == 1 ? sums[1] : sums[2]);
      }
    }
    const float value = conv(ta, row.a);
    if (lower) {
      const float k = conv(tb, row.b);
      sh.q2[t][ch] = MakePair(value, value);
      sh.k2[t][ch] = MakePair(k, k);
      sh.z[t][ch] = row.z;
    } else {
      sh.v[t][ch] = value;
    }
    if (owner && t >= n - 2) {
      float* to = t == n - 1 ? seq.conv_out : seq.conv_saved;
      store_window(to, ch_a, ta);
      if (lower) {
        store_window(to, ch_b, tb);
      }
    }
  }
  __syncthreads();
  // The tokens' scalars, a warp each: decay, beta, the norms of q and k.
  for (int item = warp; item < 3 * n; item += warps) {
    const int t = item / 3, which = item - 3 * t;
    if (which < 2) {
      float dot;
      if (gate_rows) {
        auto total = [&](int i) {
          float part = lane < warps ? sh.gates[t][i][lane] : 0.f;
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
          }
          return part;   // lanes 0 .. 7
        };
        const float inv = norm != nullptr ? GateInverse(total(0), g.cols, g.eps) : 1.0f;
        dot = total(1 + which) * inv;
      } else {
        dot = seq.gates[t * seq.gates_stride + head * a.gate_apart + which * a.gate_beta];
      }
      if (lane == 0 && which == 0) {
        sh.coef[t].decay = expf(ssm_a * Softplus(dot + dt_bias));
      } else if (lane == 0) {
        sh.coef[t].beta = Sigmoid(dot);
      }
    } else {
      float qq = 0.f, kk = 0.f, kq = 0.f;
      for (int i = lane; i < dk; i += 32) {
        const float q = Unpack(sh.q2[t][i]).x, k = Unpack(sh.k2[t][i]).x;
        qq = fmaf(q, q, qq);
        kk = fmaf(k, k, kk);
        kq = fmaf(k, q, kq);
      }
      qq = WarpSum(qq);
      kk = WarpSum(kk);
      kq = WarpSum(kq);
      // L2 norms (+1e-6 under the root); q also takes 1/sqrt(dk).
      if (lane < 2) {
        const float inv = 1.0f / sqrtf((lane == 0 ? qq : kk) + 1e-6f);
        (lane == 0 ? sh.coef[t].q : sh.coef[t].k) = lane == 0 ? inv * (1.0f / sqrtf(static_cast<float>(dk))) : inv;
      }
      if (lane == 0) {
        sh.coef[t].kq = kq;
      }
    }
  }
  // (The first token's sums over the state, while others work the scalars out.)
  float sums_of[8];
  TileSums<DK>(state_tile, dk, sh.q2[0], sh.k2[0], sums_of);
  __syncthreads();
#pragma unroll 1
  for (int t = 0; t < n; ++t) {
    float* dst = t == n - 1 ? seq.ssm_last + state_at : (t == n - 2 ? seq.ssm + state_at : nullptr);
    const DeltaCoef coef = sh.coef[t];
    TileUpdate<DK>(state_tile, sums_of, dst, dk, warp, sh.k2[t], sh.v[t], coef, sh.y[t], &sh.squares[t][warp]);
    if (t + 1 < n) {
      TileSums<DK>(state_tile, dk, sh.q2[t + 1], sh.k2[t + 1], sums_of);
    }
  }
  // Gated RMSNorm over the head's dk outputs: RMS(o) * w * silu(z); the warps'
  // tiles left their outputs' squares, so one barrier serves both.
  __syncthreads();
  if (lower) {
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
      float total = 0.f;
      for (int w = 0; w < warps; ++w) {
        total += sh.squares[t][w];
      }
      const float inv = 1.0f / sqrtf(total / static_cast<float>(dk) + a.rms_eps);
      seq.y[t * seq.y_stride + head * dk + ch] = sh.y[t][ch] * inv * norm_w * Silu(sh.z[t][ch]);
    }
  }
}

// The gate dots of a step of several sequences: alpha = alpha_w[head] . x and beta
// likewise, x = RMS(row) * norm_w where norm weights are given (DeltaNetStep::Run).
// A block takes eight of the 2 * value_heads rows and eight tokens, its warps the
// 128-value chunks of K round-robin, a lane four values of each. Inside the mixer
// kernel every (sequence, head) block walked its two rows and the input once per
// token, a chain of L2 round trips with nothing to hide it: 65 us for 32 sequences
// of 32 heads, against 4 us here.
//
// The dots wait for the mixer kernel in scratch that belongs to the stream, or, where
// there is none (a capture: its graph may run on any stream), in the tokens' output
// rows, whose part for a head the mixer kernel's block for that head reads before it
// overwrites it. (Always there: 45.7 instead of 44.2 us for 32 sequences of 32 heads,
// as a token's dots are then 512 bytes apart.)
constexpr int kGateTile = 8;
constexpr int kGateRowsMax = kMaxSeqs * kMaxRunTokens;
struct GatesArgs {
  DeltaNetGateRows rows;
  int value_heads;
  int tokens;
  int head_dim;
  float* out;                       // [tokens][2 * value_heads], or null: into y
  const float* x[kGateRowsMax];
  float* y[kGateRowsMax];
};

__global__ void __launch_bounds__(2 * kDeltaThreads)
DeltaNetGatesKernel(const __grid_constant__ GatesArgs a) {
  __shared__ float partial[8][kGateTile * kGateTile + kGateTile];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = blockIdx.x * kGateTile, t0 = blockIdx.y * kGateTile;
  const int count = 2 * a.value_heads;
  const float4* w[kGateTile];
#pragma unroll
  for (int r = 0; r < kGateTile; ++r) {
    const int row = min(r0 + r, count - 1);
    w[r] = reinterpret_cast<const float4*>(row < a.value_heads ? a.rows.alpha_w + static_cast<size_t>(row) * a.rows.cols
                                                               : a.rows.beta_w + static_cast<size_t>(row - a.value_heads) * a.rows.cols);
  }
  GridLaunchDependents();
  GridDependencyWait();
  float acc[kGateTile * kGateTile] = {}, sq[kGateTile] = {};
  const float4* norm = reinterpret_cast<const float4*>(a.rows.norm_w);
  for (int i = threadIdx.x; i < a.rows.cols / 4; i += blockDim.x) {
    float4 x[kGateTile];
#pragma unroll
    for (int t = 0; t < kGateTile; ++t) {
      x[t] = *(reinterpret_cast<const float4*>(a.x[min(t0 + t, a.tokens - 1)]) + i);
      sq[t] = Dot4(x[t], x[t], sq[t]);
    }
    const float4 nw = norm != nullptr ? norm[i] : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
    for (int r = 0; r < kGateTile; ++r) {
      const float4 v = Times4(w[r][i], nw);
#pragma unroll
      for (int t = 0; t < kGateTile; ++t) {
        acc[r * kGateTile + t] = Dot4(v, x[t], acc[r * kGateTile + t]);
      }
    }
  }
  int first;
  Fold<kGateTile * kGateTile>(acc, lane, &first);
#pragma unroll
  for (int j = 0; j < kFoldLeft<kGateTile * kGateTile>; ++j) {
    partial[warp][first + j] = acc[j];
  }
  Fold<kGateTile>(sq, lane, &first);
  static_assert(kFoldLeft<kGateTile> == 1, "one sum a lane");
  partial[warp][kGateTile * kGateTile + first] = sq[0];   // several lanes the same
  __syncthreads();
  const int r = threadIdx.x / kGateTile, t = threadIdx.x % kGateTile;
  if (r >= kGateTile || r0 + r >= count || t0 + t >= a.tokens) {
    return;
  }
  // Over the warps in the order of the mixer kernel's shuffles.
  auto total_of = [&](int i) {
    float p[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      p[k] = 32 * k < static_cast<int>(blockDim.x) ? partial[k][i] : 0.f;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < o; ++k) {
        p[k] += p[k + o];
      }
    }
    return p[0];
  };
  const float inv = norm != nullptr ? GateInverse(total_of(kGateTile * kGateTile + t), a.rows.cols, a.rows.eps) : 1.0f;
  const float dot = total_of(r * kGateTile + t) * inv;
  if (a.out != nullptr) {
    a.out[static_cast<size_t>(t0 + t) * count + r0 + r] = dot;
  } else {
    const int which = r0 + r < a.value_heads ? 0 : 1;
    a.y[t0 + t][(r0 + r - which * a.value_heads) * a.head_dim + which] = dot;
  }
}

template <int SEQS>
cudaError_t LaunchRule(gufo_cuda_ctx* ctx, const gufo_cuda_delta_seq* seqs, int n, int key_heads, int value_heads,
                       int head_dim) {
  DeltaRuleArgs<SEQS> args;
  for (int s = 0; s < n; ++s) {
    args.seq[s] = seqs[s];
  }
  args.key_heads = key_heads;
  args.value_heads = value_heads;
  args.head_dim = head_dim;
  args.early_state = ctx->early_state ? 1 : 0;
  return LaunchOverlapped(DeltaRuleKernel<SEQS>, dim3(head_dim / kRuleCols, value_heads, n), dim3(32), 0, ctx->stream, 1, args);
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
    GUFO_CUDA_TRY(n <= 2    ? gufo::LaunchRule<2>(ctx, seqs + s0, n, key_heads, value_heads, head_dim)
                  : n <= 16 ? gufo::LaunchRule<16>(ctx, seqs + s0, n, key_heads, value_heads, head_dim)
                            : gufo::LaunchRule<gufo::kMaxSeqs>(ctx, seqs + s0, n, key_heads, value_heads, head_dim));
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
                        q.in_stride, q.h_stride, q.y_stride, n, nullptr, 0});
      }
    }
  }
  // States may be written by the launch before this one: no early state loads.
  return gufo::EnqueueDeltaNetLinear(ctx, it->second, step.data(), nseq, false, &gates);
}

}  // extern "C"

namespace gufo {

namespace {

template <int DK, int WIN, int SEQS>
int LaunchLinear(gufo_cuda_ctx* ctx, const LinearShape& shape, const DeltaNetSeq* seqs, int n) {
  LinearArgs<SEQS> args;
  args.shape = shape;
  for (int s = 0; s < n; ++s) {
    args.seq[s] = seqs[s];
  }
  GUFO_CUDA_TRY(LaunchOverlapped(DeltaNetLinearKernel<DK, WIN, SEQS>, dim3(shape.value_heads, n), dim3(2 * shape.head_dim), 0,
                                 ctx->stream, 1, args));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

// Whether a sequence's output rows are apart from the input rows that are read after
// the gates have been left in them (a caller may put y over z).
bool OutputsApart(const DeltaNetSeq& s, size_t in_width, size_t x_width, size_t y_width) {
  auto apart = [](const float* a, size_t na, const float* b, size_t nb) {
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(a), b0 = reinterpret_cast<uintptr_t>(b);
    return a0 + 4 * na <= b0 || b0 + 4 * nb <= a0;
  };
  for (int t = 0; t < s.tokens; ++t) {
    for (int u = 0; u < s.tokens; ++u) {
      const float* y = s.y + t * s.y_stride;
      if (!apart(y, y_width, s.in + u * s.in_stride, in_width) || !apart(y, y_width, s.x + u * s.x_stride, x_width)) {
        return false;
      }
    }
  }
  return true;
}

// Fills in where the sequences find them.
int EnqueueGates(gufo_cuda_ctx* ctx, const DeltaNetGateRows& rows, int value_heads, int head_dim, float* scratch,
                 DeltaNetSeq* seqs, int n) {
  GatesArgs args;
  args.rows = rows;
  args.value_heads = value_heads;
  args.head_dim = head_dim;
  args.out = scratch;
  args.tokens = 0;
  for (int s = 0; s < n; ++s) {
    seqs[s].gates = scratch != nullptr ? scratch + static_cast<size_t>(args.tokens) * 2 * value_heads : seqs[s].y;
    seqs[s].gates_stride = scratch != nullptr ? 2 * value_heads : seqs[s].y_stride;
    for (int t = 0; t < seqs[s].tokens; ++t) {
      args.x[args.tokens] = seqs[s].x + t * seqs[s].x_stride;
      args.y[args.tokens++] = seqs[s].y + t * seqs[s].y_stride;
    }
  }
  GUFO_CUDA_TRY(LaunchOverlapped(DeltaNetGatesKernel,
                                 dim3((2 * value_heads + kGateTile - 1) / kGateTile, (args.tokens + kGateTile - 1) / kGateTile),
                                 dim3(2 * head_dim), 0, ctx->stream, 1, args));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

}  // namespace

int EnqueueDeltaNetLinear(gufo_cuda_ctx* ctx, const DeltaNetLayer& l, DeltaNetSeq* seqs, int nseq,
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
  const size_t value_dim = static_cast<size_t>(l.value_heads) * l.head_dim;
  const size_t in_width = 2 * static_cast<size_t>(l.key_heads) * l.head_dim + 2 * value_dim;
  int most = kMaxSeqs;   // sequences a launch
  uint8_t* scratch = nullptr;
  if (gate_rows != nullptr && nseq > 2) {
    const size_t want = static_cast<size_t>(kGateRowsMax) * 2 * l.value_heads * 4;
    const int rc = ctx->StreamScratch(gufo_cuda_ctx::kGatesScratch, want, 64u << 10, &scratch, nullptr);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
    for (int s = 0; scratch == nullptr && s < nseq; ++s) {
      if (!OutputsApart(seqs[s], in_width, gate_rows->cols, value_dim)) {
        most = 2;   // the gates have nowhere to wait: worked out in the mixer's blocks
      }
    }
  }
  for (int s0 = 0; s0 < nseq; s0 += most) {
    const int n = nseq - s0 < most ? nseq - s0 : most;
    DeltaNetSeq* now = seqs + s0;
    shape.gate_apart = 1;
    shape.gate_beta = l.value_heads;
    if (gate_rows == nullptr) {
      for (int s = 0; s < n; ++s) {   // behind z in the input row
        now[s].gates = now[s].in + in_width;
        now[s].gates_stride = now[s].in_stride;
      }
    } else if (n > 2) {
      if (scratch == nullptr) {
        shape.gate_apart = l.head_dim;
        shape.gate_beta = 1;
      }
      const int rc = EnqueueGates(ctx, *gate_rows, l.value_heads, l.head_dim, reinterpret_cast<float*>(scratch), now, n);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
    }
    // One or two sequences (a decode step) in a small argument block; the models' own
    // shape (heads of 128, windows of up to three columns) with its loops unrolled.
    const bool common = l.head_dim == 128 && shape.conv_kernel <= 4;
    const int rc = n <= 2 ? (common ? LaunchLinear<128, 3, 2>(ctx, shape, now, n) : LaunchLinear<0, 7, 2>(ctx, shape, now, n))
                          : (common ? LaunchLinear<128, 3, kMaxSeqs>(ctx, shape, now, n)
                                    : LaunchLinear<0, 7, kMaxSeqs>(ctx, shape, now, n));
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  return GUFO_CUDA_OK;
}

}  // namespace gufo
