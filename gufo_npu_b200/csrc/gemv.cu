// Dequant-fused GEMV / small-M GEMM over GGUF rows: the product behind
// Projections::Apply (GgufProjections::MatMul,
// src/models/qwen35/gguf_projections.cpp:239-286 in the reference).
//
// This file holds the kernels for F32 (GemvRowsF32), Q5_K and Q8_0 (GemvSplit) rows
// and the general kernel: any row count, any mix of types in one launch, 1..8
// tokens per weight read. There one warp owns one
// output row; lanes split the row's blocks so that a warp reads whole 128-byte
// lines, codes are turned into fp32 once and reused for every token, and the
// sub-block scale and min are applied per 32 (Q4_K) or 16 (Q6_K) values:
//   Q4_K:  sum_j d*sc_j * (q . x)_j  -  dmin*m_j * (sum x)_j
//   Q6_K:  d * sum_g sc_g * ((q - 32) . x)_g
// fp32 accumulation throughout; lanes are combined with warp shuffles.
// HBM-bound: algorithmic bytes are the GGUF row bytes plus x and y.
#include <cstring>

#include "gemv.cuh"
#include "gemm_tc.cuh"

namespace gufo {

namespace {

template <int M>
__device__ __forceinline__ void RowQ4K(const uint8_t* __restrict__ row, int cols,
                                       const float* x, int lane,
                                       float (&acc)[M]) {
  const int p = lane >> 3;        // sub-block pair of this lane's word
  const int c = (lane & 7) * 4;   // first value inside the sub-blocks
  const int blocks = cols / kSuperBlock;
  for (int b = 0; b < blocks; ++b) {
    const uint32_t* block = reinterpret_cast<const uint32_t*>(row + b * kQ4KBytes);
    const uint32_t dd = __ldg(block);
    const uint32_t s0 = __ldg(block + 1), s1 = __ldg(block + 2), s2 = __ldg(block + 3);
    const uint32_t q = __ldg(block + 4 + lane);
    const float d = HalfBitsToFloat(static_cast<uint16_t>(dd & 0xFFFF));
    const float dmin = HalfBitsToFloat(static_cast<uint16_t>(dd >> 16));
    int sc_lo, m_lo, sc_hi, m_hi;
    ScaleMinK4(2 * p, s0, s1, s2, &sc_lo, &m_lo);
    ScaleMinK4(2 * p + 1, s0, s1, s2, &sc_hi, &m_hi);
    const float d_lo = d * static_cast<float>(sc_lo), o_lo = dmin * static_cast<float>(m_lo);
    const float d_hi = d * static_cast<float>(sc_hi), o_hi = dmin * static_cast<float>(m_hi);
    const float l0 = static_cast<float>(q & 0xF), l1 = static_cast<float>((q >> 8) & 0xF);
    const float l2 = static_cast<float>((q >> 16) & 0xF), l3 = static_cast<float>((q >> 24) & 0xF);
    const float h0 = static_cast<float>((q >> 4) & 0xF), h1 = static_cast<float>((q >> 12) & 0xF);
    const float h2 = static_cast<float>((q >> 20) & 0xF), h3 = static_cast<float>(q >> 28);
    const int at = b * kSuperBlock + 64 * p + c;
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const float4 xl = *reinterpret_cast<const float4*>(x + static_cast<size_t>(t) * cols + at);
      const float4 xh = *reinterpret_cast<const float4*>(x + static_cast<size_t>(t) * cols + at + 32);
      const float dot_lo = l0 * xl.x + l1 * xl.y + l2 * xl.z + l3 * xl.w;
      const float dot_hi = h0 * xh.x + h1 * xh.y + h2 * xh.z + h3 * xh.w;
      const float sum_lo = (xl.x + xl.y) + (xl.z + xl.w);
      const float sum_hi = (xh.x + xh.y) + (xh.z + xh.w);
      acc[t] += d_lo * dot_lo - o_lo * sum_lo;
      acc[t] += d_hi * dot_hi - o_hi * sum_hi;
    }
  }
}

template <int M>
__device__ __forceinline__ void RowQ6K(const uint8_t* __restrict__ row, int cols,
                                       const float* x, int lane,
                                       float (&acc)[M]) {
  const int blocks = cols / kSuperBlock;
  for (int b = 0; b < blocks; ++b) {
    const Q6KBlock block = Q6KBlockAt(row, blocks, b);
    const float d = HalfBitsToFloat(__ldg(reinterpret_cast<const uint16_t*>(block.d)));
    float part[M];
#pragma unroll
    for (int t = 0; t < M; ++t) {
      part[t] = 0.f;
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const uint8_t* ql = block.ql + 64 * half;
      const uint8_t* qh = block.qh + 32 * half;
      const int8_t* sc = block.sc + 8 * half + (lane >> 4);
      const int a = __ldg(ql + lane), c = __ldg(ql + lane + 32), h = __ldg(qh + lane);
      const float w0 = static_cast<float>(static_cast<int>(__ldg(sc))) *
                       static_cast<float>(((a & 0xF) | ((h & 3) << 4)) - 32);
      const float w1 = static_cast<float>(static_cast<int>(__ldg(sc + 2))) *
                       static_cast<float>(((c & 0xF) | (((h >> 2) & 3) << 4)) - 32);
      const float w2 = static_cast<float>(static_cast<int>(__ldg(sc + 4))) *
                       static_cast<float>(((a >> 4) | (((h >> 4) & 3) << 4)) - 32);
      const float w3 = static_cast<float>(static_cast<int>(__ldg(sc + 6))) *
                       static_cast<float>(((c >> 4) | (((h >> 6) & 3) << 4)) - 32);
      const int at = b * kSuperBlock + 128 * half + lane;
#pragma unroll
      for (int t = 0; t < M; ++t) {
        const float* xt = x + static_cast<size_t>(t) * cols + at;
        part[t] += w0 * xt[0] + w1 * xt[32] + w2 * xt[64] + w3 * xt[96];
      }
    }
#pragma unroll
    for (int t = 0; t < M; ++t) {
      acc[t] += d * part[t];
    }
  }
}

// Q5_K: Q4_K's layout with a fifth code bit per value in 32 bytes of qh
// (gguf_dot::DotK4<true>, src/models/qwen35/gguf_dot.hpp:115-193).
template <int M>
__device__ __forceinline__ void RowQ5K(const uint8_t* __restrict__ row, int cols,
                                       const float* x, int lane,
                                       float (&acc)[M]) {
  const int p = lane >> 3;        // sub-block pair of this lane's word
  const int c = (lane & 7) * 4;   // first value inside the sub-blocks
  const int blocks = cols / kSuperBlock;
  for (int b = 0; b < blocks; ++b) {
    const uint32_t* block = reinterpret_cast<const uint32_t*>(row + b * kQ5KBytes);
    const uint32_t dd = __ldg(block);
    const uint32_t s0 = __ldg(block + 1), s1 = __ldg(block + 2), s2 = __ldg(block + 3);
    const uint32_t h = __ldg(block + 4 + (lane & 7)) >> (2 * p);   // qh bytes c .. c + 3, this pair's bits low
    const uint32_t q = __ldg(block + 12 + lane);
    const float d = HalfBitsToFloat(static_cast<uint16_t>(dd & 0xFFFF));
    const float dmin = HalfBitsToFloat(static_cast<uint16_t>(dd >> 16));
    int sc_lo, m_lo, sc_hi, m_hi;
    ScaleMinK4(2 * p, s0, s1, s2, &sc_lo, &m_lo);
    ScaleMinK4(2 * p + 1, s0, s1, s2, &sc_hi, &m_hi);
    const float d_lo = d * static_cast<float>(sc_lo), o_lo = dmin * static_cast<float>(m_lo);
    const float d_hi = d * static_cast<float>(sc_hi), o_hi = dmin * static_cast<float>(m_hi);
    const float l0 = static_cast<float>((q & 0xF) + ((h & 1) << 4));
    const float l1 = static_cast<float>(((q >> 8) & 0xF) + (((h >> 8) & 1) << 4));
    const float l2 = static_cast<float>(((q >> 16) & 0xF) + (((h >> 16) & 1) << 4));
    const float l3 = static_cast<float>(((q >> 24) & 0xF) + (((h >> 24) & 1) << 4));
    const float h0 = static_cast<float>(((q >> 4) & 0xF) + (((h >> 1) & 1) << 4));
    const float h1 = static_cast<float>(((q >> 12) & 0xF) + (((h >> 9) & 1) << 4));
    const float h2 = static_cast<float>(((q >> 20) & 0xF) + (((h >> 17) & 1) << 4));
    const float h3 = static_cast<float>((q >> 28) + (((h >> 25) & 1) << 4));
    const int at = b * kSuperBlock + 64 * p + c;
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const float4 xl = *reinterpret_cast<const float4*>(x + static_cast<size_t>(t) * cols + at);
      const float4 xh = *reinterpret_cast<const float4*>(x + static_cast<size_t>(t) * cols + at + 32);
      const float dot_lo = l0 * xl.x + l1 * xl.y + l2 * xl.z + l3 * xl.w;
      const float dot_hi = h0 * xh.x + h1 * xh.y + h2 * xh.z + h3 * xh.w;
      const float sum_lo = (xl.x + xl.y) + (xl.z + xl.w);
      const float sum_hi = (xh.x + xh.y) + (xh.z + xh.w);
      acc[t] += d_lo * dot_lo - o_lo * sum_lo;
      acc[t] += d_hi * dot_hi - o_hi * sum_hi;
    }
  }
}

// Q8_0: 32 int8 codes and one fp16 scale per 34-byte block; lane l takes value l
// of every block (gguf_dot::DotQ8_0, gguf_dot.hpp:31-69).
template <int M>
__device__ __forceinline__ void RowQ8_0(const uint8_t* __restrict__ row, int cols,
                                        const float* x, int lane,
                                        float (&acc)[M]) {
  const int blocks = cols / kQ8Block;
  for (int b = 0; b < blocks; ++b) {
    const uint8_t* block = row + b * kQ8Bytes;
    const float d = HalfBitsToFloat(__ldg(reinterpret_cast<const uint16_t*>(block)));
    const float w = d * static_cast<float>(static_cast<int>(static_cast<int8_t>(__ldg(block + 2 + lane))));
#pragma unroll
    for (int t = 0; t < M; ++t) {
      acc[t] = fmaf(w, x[static_cast<size_t>(t) * cols + b * kQ8Block + lane], acc[t]);
    }
  }
}

template <int M>
__device__ __forceinline__ void RowF32(const uint8_t* __restrict__ row, int cols,
                                       const float* x, int lane,
                                       float (&acc)[M]) {
  const float4* w = reinterpret_cast<const float4*>(row);
  for (int i = lane; i < cols / 4; i += 32) {
    const float4 v = __ldg(w + i);
#pragma unroll
    for (int t = 0; t < M; ++t) {
      const float4 xv = *(reinterpret_cast<const float4*>(x + static_cast<size_t>(t) * cols) + i);
      acc[t] += v.x * xv.x + v.y * xv.y + v.z * xv.z + v.w * xv.w;
    }
  }
}

template <int M>
__global__ void __launch_bounds__(256)
GemvRows(const __grid_constant__ GemvArgs args) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= args.total_rows) {
    return;
  }
  int p = 0;
  int local = row;
  while (p + 1 < args.nparts && local >= args.parts[p].rows) {
    local -= args.parts[p].rows;
    ++p;
  }
  const GemvPart& part = args.parts[p];
  const uint8_t* data = part.data + static_cast<size_t>(local) * part.row_bytes;
  const float* x = args.x;   // read with coherent loads: written while this kernel may already be resident
  float* y = args.y;
  GridLaunchDependents();
  GridDependencyWait();
  if (args.group_ids != nullptr) {
    const int id = args.group_ids[blockIdx.y];
    if (id < 0) {
      return;
    }
    data += static_cast<size_t>(id) * part.rows * part.row_bytes;
    x += static_cast<size_t>(blockIdx.y / (args.x_group_div > 1 ? args.x_group_div : 1)) * args.x_group_stride;
    y += static_cast<size_t>(blockIdx.y) * args.y_group_stride;
  }
  float acc[M];
#pragma unroll
  for (int t = 0; t < M; ++t) {
    acc[t] = 0.f;
  }
  if (part.type == GUFO_CUDA_Q4_K) {
    RowQ4K<M>(data, args.cols, x, lane, acc);
  } else if (part.type == GUFO_CUDA_Q6_K) {
    RowQ6K<M>(data, args.cols, x, lane, acc);
  } else if (part.type == GUFO_CUDA_Q5_K) {
    RowQ5K<M>(data, args.cols, x, lane, acc);
  } else if (part.type == GUFO_CUDA_Q8_0) {
    RowQ8_0<M>(data, args.cols, x, lane, acc);
  } else {
    RowF32<M>(data, args.cols, x, lane, acc);
  }
#pragma unroll
  for (int t = 0; t < M; ++t) {
    const float total = WarpSum(acc[t]);
    if (lane == 0) {
      y[static_cast<size_t>(t) * args.y_stride + part.out_offset + local] = total;
    }
  }
}

// F32 rows (alpha / beta, the router) against any number of tokens in one launch: a
// block takes eight rows and TOK tokens, its warps the 128-value chunks of K
// round-robin, a lane four values of each. All of a warp's loads of a chunk are in
// flight together and a row of 2560 values is three chunks deep, where one warp
// per row walks twenty; the inputs are read once per eight rows. 64 rows x 2560
// values: 512 tokens were 64 launches of the kernel above (1.2 ms with the gaps).
// Where eight rows a block would leave SMs without one (a router: 257 rows, 33
// blocks) a block takes two.
//
// What bounds it with many tokens: the sums over the lanes and too few warps. A block's 64
// sums a warp are folded (Fold), 62 shuffles instead of 320, and two blocks share an SM:
// 64 rows x 2560 values, 8 / 79 / 512 tokens 2.9 / 5.0 / 16.6 -> 2.4 / 4.3 / 12.0 us, 257 rows x
// 2048 (a router), 4 / 128 tokens 2.6 / 15.2 -> 2.1 / 9.6.
//
// PER_SM, the blocks an SM that registers are kept to: few, for loads in flight and the folded
// sums of several tokens. But one token's blocks that would need another round, with rows of one
// chunk a warp or in tiles of two, are better all there (us: 65536 x 1024 44 with two an SM, 38
// with five, but 12288 x 2048 12.8 and 15.1; 1024 x 2048 in tiles of two 2.8 with three, 2.3
// with six, but 600 x 4096 2.3 and 2.7); and where the matrix does not stay in the L2, tiles of
// 64 sums have an SM to themselves (8 tokens: 12288 x 2560 69 with two, 45 with one, but 4096 x
// 2048 9.5 and 10.2).
template <int kF32Rows, int TOK, int PER_SM>
__global__ void __launch_bounds__(256, PER_SM)
GemvRowsF32(const __grid_constant__ GemvArgs args, int tokens) {
  __shared__ float partial[8][kF32Rows * TOK];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int t0 = blockIdx.y * TOK;
  // Rows past the end repeat the last one, tokens past the end the last token.
  const float4* w[kF32Rows];
#pragma unroll
  for (int r = 0; r < kF32Rows; ++r) {
    int local = min(static_cast<int>(blockIdx.x) * kF32Rows + r, args.total_rows - 1);
    int p = 0;
    while (p + 1 < args.nparts && local >= args.parts[p].rows) {
      local -= args.parts[p].rows;
      ++p;
    }
    w[r] = reinterpret_cast<const float4*>(args.parts[p].data + static_cast<size_t>(local) * args.parts[p].row_bytes);
  }
  GridLaunchDependents();
  GridDependencyWait();
  constexpr int kSums = kF32Rows * TOK;
  float acc[kSums];
#pragma unroll
  for (int j = 0; j < kSums; ++j) {
    acc[j] = 0.f;
  }
  for (int i = warp * 32 + lane; i < args.cols / 4; i += 256) {
    float4 v[kF32Rows], xv[TOK];
#pragma unroll
    for (int r = 0; r < kF32Rows; ++r) {
      v[r] = __ldg(w[r] + i);
    }
#pragma unroll
    for (int t = 0; t < TOK; ++t) {
      xv[t] = *(reinterpret_cast<const float4*>(args.x + static_cast<size_t>(min(t0 + t, tokens - 1)) * args.cols) + i);
    }
#pragma unroll
    for (int r = 0; r < kF32Rows; ++r) {
#pragma unroll
      for (int t = 0; t < TOK; ++t) {
        acc[r * TOK + t] += v[r].x * xv[t].x + v[r].y * xv[t].y + v[r].z * xv[t].z + v[r].w * xv[t].w;
      }
    }
  }
  int first;
  Fold<kSums>(acc, lane, &first);
#pragma unroll
  for (int j = 0; j < kFoldLeft<kSums>; ++j) {
    partial[warp][first + j] = acc[j];   // below 32 sums several lanes store the same
  }
  __syncthreads();
  const int r = threadIdx.x / TOK, t = threadIdx.x % TOK;
  int local = static_cast<int>(blockIdx.x) * kF32Rows + r;
  if (threadIdx.x >= kF32Rows * TOK || local >= args.total_rows || t0 + t >= tokens) {
    return;
  }
  float total = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    total += partial[k][threadIdx.x];
  }
  int p = 0;
  while (p + 1 < args.nparts && local >= args.parts[p].rows) {
    local -= args.parts[p].rows;
    ++p;
  }
  args.y[static_cast<size_t>(t0 + t) * args.y_stride + args.parts[p].out_offset + local] = total;
}

template <int ROWS>
int LaunchRowsF32(gufo_cuda_ctx* ctx, const GemvArgs& args, int tokens) {
  const unsigned rows = (args.total_rows + ROWS - 1) / ROWS;
  constexpr int kMost = 65535 * 8;   // what a grid's second dimension holds of the tiles below
  if (tokens > kMost) {
    const int rc = LaunchRowsF32<ROWS>(ctx, args, kMost);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
    GemvArgs rest = args;
    rest.x += static_cast<size_t>(kMost) * args.cols;
    rest.y += static_cast<size_t>(kMost) * args.y_stride;
    return LaunchRowsF32<ROWS>(ctx, rest, tokens - kMost);
  }
  auto launch = [&](auto kernel, int tok) {
    return LaunchOverlapped(kernel, dim3(rows, (tokens + tok - 1) / tok), dim3(256), 0, ctx->stream, 1, args, tokens);
  };
  const bool beyond_l2 = static_cast<int64_t>(args.total_rows) * args.cols * 4 > (64ll << 20);
  if constexpr (ROWS == 2) {
    const bool rounds = static_cast<int>(rows) > 3 * ctx->sm_count;
    GUFO_CUDA_TRY(tokens > 4   ? launch(GemvRowsF32<2, 8, 2>, 8)
                  : tokens > 2 ? launch(GemvRowsF32<2, 4, 4>, 4)
                  : tokens > 1 ? launch(GemvRowsF32<2, 2, 4>, 2)
                  : rounds     ? launch(GemvRowsF32<2, 1, 6>, 1)
                               : launch(GemvRowsF32<2, 1, 3>, 1));
  } else {
    const bool rounds = static_cast<int>(rows) > 2 * ctx->sm_count;
    GUFO_CUDA_TRY(tokens > 4                     ? (beyond_l2 ? launch(GemvRowsF32<8, 8, 1>, 8) : launch(GemvRowsF32<8, 8, 2>, 8))
                  : tokens > 2                   ? launch(GemvRowsF32<8, 4, 2>, 4)
                  : tokens > 1                   ? launch(GemvRowsF32<8, 2, 2>, 2)
                  : rounds && args.cols <= 1024 ? launch(GemvRowsF32<8, 1, 5>, 1)
                                                 : launch(GemvRowsF32<8, 1, 2>, 1));
  }
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

// Rows of a group of GemvSplit.
constexpr int kSplitRows = 4;

// Eight weights of a Q5_K block: values 64 p + c .. + 3 and the same 32 further on
// (p = lane / 8, c = 4 (lane % 8)).
__device__ __forceinline__ void SplitWeights5(const uint4& head, uint32_t h, uint32_t q, int p, float (&w)[8]) {
  const float d = HalfBitsToFloat(static_cast<uint16_t>(head.x & 0xFFFF));
  const float dmin = HalfBitsToFloat(static_cast<uint16_t>(head.x >> 16));
  int sc_lo, m_lo, sc_hi, m_hi;
  ScaleMinK4(2 * p, head.y, head.z, head.w, &sc_lo, &m_lo);
  ScaleMinK4(2 * p + 1, head.y, head.z, head.w, &sc_hi, &m_hi);
  const float d_lo = d * static_cast<float>(sc_lo), o_lo = dmin * static_cast<float>(m_lo);
  const float d_hi = d * static_cast<float>(sc_hi), o_hi = dmin * static_cast<float>(m_hi);
  h >>= 2 * p;   // the fifth bits of this pair of sub-blocks
  const uint32_t lo = (q & 0x0F0F0F0Fu) | ((h << 4) & 0x10101010u);
  const uint32_t hi = ((q >> 4) & 0x0F0F0F0Fu) | ((h << 3) & 0x10101010u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // A byte under the exponent of 2^23, the bias taken off: no conversion.
    const float l = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7440u | i)) - 8388608.0f;
    const float g = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7440u | i)) - 8388608.0f;
    w[i] = fmaf(d_lo, l, -o_lo);
    w[4 + i] = fmaf(d_hi, g, -o_hi);
  }
}

// Q5_K and Q8_0 rows of whole 256-value blocks against up to M tokens. A thread block takes a
// group of four rows (LOOP: every gridDim.x-th), its warps the 256-value blocks of K
// round-robin, a lane eight values of each: the rows' loads of a block are in flight together
// and a row of 2048 values is one round trip deep, where one warp per row walks eight (Q8_0:
// sixty-four, a byte a lane); a token's inputs are read once for the rows. AHEAD: a warp's
// first unit is asked for ahead of the dependency wait (`early`: no bytes are borrowed) and the
// next one while it multiplies, across the groups. The sums over the lanes are folded (Fold).
//
// What bounds it: issue slots for long matrices (a value's conversion and its FMAs), a block's
// start and one load for short ones. With loads behind the wait, a block for every group and a
// butterfly per sum, and now, us at 1 / 2 / 4 / 8 tokens, held by the library: Q5_K 2048 x 2048
// 4.2 / 4.6 / 5.9 / 9.3 and 4.0 / 4.2 / 5.0 / 6.6, 24576 x 2560 46 / 50 / 78 / 101 and 45 / 48 /
// 62 / 83; Q8_0 3.3 / 4.5 / 5.8 / 8.6 and 2.6 / 4.1 / 4.7 / 6.1, 31 / 40 / 64 / 90 and 27 / 33 /
// 43 / 64. Registers are kept to what lets two blocks share an SM, three with one or two tokens
// (four for Q8_0 and one token: 2048 rows are one round then).
template <int TYPE, int M, bool AHEAD, bool LOOP = AHEAD>
__global__ void __launch_bounds__(256, M == 1 && TYPE == GUFO_CUDA_Q8_0 ? 4 : (M <= 2 ? 3 : 2))
GemvSplit(const __grid_constant__ GemvArgs args, int tokens, bool early) {
  constexpr bool kQ5 = TYPE == GUFO_CUDA_Q5_K;
  constexpr int kBlockBytes = kQ5 ? kQ5KBytes : kSuperBlock / kQ8Block * kQ8Bytes;
  constexpr int kSums = kSplitRows * M;
  __shared__ float partial[2][8][kSums];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int groups = (args.total_rows + kSplitRows - 1) / kSplitRows;
  const int blocks = args.cols / kSuperBlock;
  // The rows of a group; rows past the end repeat the last one.
  auto row_of = [&](int group, int r) {
    int local = min(group * kSplitRows + r, args.total_rows - 1);
    int p = 0;
    while (p + 1 < args.nparts && local >= args.parts[p].rows) {
      local -= args.parts[p].rows;
      ++p;
    }
    return args.parts[p].data + static_cast<size_t>(local) * args.parts[p].row_bytes;
  };
  const uint8_t* row[kSplitRows];
  auto enter = [&](int group) {
#pragma unroll
    for (int r = 0; r < kSplitRows; ++r) {
      row[r] = row_of(group, r);
    }
  };
  // Where this lane's eight inputs sit: two groups of four.
  const int at = kQ5 ? 64 * (lane >> 3) + 4 * (lane & 7) : 8 * lane;
  constexpr int kApart = kQ5 ? 32 : 4;
  // Q8_0: eight codes at a 2-byte boundary, out of aligned words.
  const int code = 34 * (lane >> 2) + 2 + 8 * (lane & 3);
  const bool odd = (code & 2) != 0;
  struct Raw {
    uint4 head[kQ5 ? kSplitRows : 1];
    uint32_t h[kQ5 ? kSplitRows : 1];
    uint32_t q[kSplitRows][kQ5 ? 1 : 3];
    uint16_t d[kQ5 ? 1 : kSplitRows];
  } raw;
  auto load = [&](int b) {
#pragma unroll
    for (int r = 0; r < kSplitRows; ++r) {
      const uint8_t* block = row[r] + static_cast<size_t>(b) * kBlockBytes;
      if constexpr (kQ5) {
        raw.head[r] = __ldg(reinterpret_cast<const uint4*>(block));
        raw.h[r] = __ldg(reinterpret_cast<const uint32_t*>(block + 16) + (lane & 7));
        raw.q[r][0] = __ldg(reinterpret_cast<const uint32_t*>(block + 48) + lane);
      } else {
        const uint32_t* words = reinterpret_cast<const uint32_t*>(block + (code & ~3));
        raw.q[r][0] = __ldg(words);
        raw.q[r][1] = __ldg(words + 1);
        raw.q[r][2] = odd ? __ldg(words + 2) : 0u;
        raw.d[r] = __ldg(reinterpret_cast<const uint16_t*>(block + 34 * (lane >> 2)));
      }
    }
  };
  enter(static_cast<int>(blockIdx.x));
  if (!early) {
    // Borrowed bytes may be what a kernel is writing that let this one start already: ahead of
    // the wait nothing but the L2, where its stores arrive too, may hold them. (Q8_0, one token:
    // 2048 x 2048 3.3 us instead of 3.5, 2048 x 6144 6.4 instead of 7.0; rows of one or two
    // blocks and Q5_K only pay for it. Read ahead they take 2.6 and 5.9.)
    GridLaunchDependents();
    if (!kQ5 && blocks >= 4 && threadIdx.x < kSplitRows) {
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row_of(static_cast<int>(blockIdx.x), threadIdx.x)),
                   "r"(blocks * kBlockBytes) : "memory");
    }
    GridDependencyWait();
  }
  if (AHEAD && warp < blocks) {
    load(warp);
  }
  GridLaunchDependents();
  GridDependencyWait();
  int buffer = 0;
#pragma unroll 1
  for (int group = static_cast<int>(blockIdx.x); group < groups;
       group = LOOP ? group + static_cast<int>(gridDim.x) : groups, buffer ^= 1) {
    if (LOOP && !AHEAD) {
      enter(group);
    }
    float acc[kSums];
#pragma unroll
    for (int j = 0; j < kSums; ++j) {
      acc[j] = 0.f;
    }
    for (int b = warp; b < blocks; b += 8) {
      // The next unit: of this group, or the first of the block's next one.
      if constexpr (!AHEAD) {
        load(b);
      }
      auto ahead = [&]() {
        if (!AHEAD) {
          return;
        }
        if (b + 8 < blocks) {
          load(b + 8);
        } else if (group + static_cast<int>(gridDim.x) < groups) {
          enter(group + static_cast<int>(gridDim.x));
          load(warp);
        }
      };
      auto weights = [&](int r, float (&w)[8]) {
        if constexpr (kQ5) {
          SplitWeights5(raw.head[r], raw.h[r], raw.q[r][0], lane >> 3, w);
        } else {
          const uint32_t pick = odd ? 0x5432u : 0x3210u;
          // Codes + 128 as bytes under the exponent of 2^23.
          const uint32_t lo = __byte_perm(raw.q[r][0], raw.q[r][1], pick) ^ 0x80808080u;
          const uint32_t hi = __byte_perm(raw.q[r][1], raw.q[r][2], pick) ^ 0x80808080u;
          const float scale = HalfBitsToFloat(raw.d[r]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            w[i] = scale * (__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7440u | i)) - 8388736.0f);
            w[4 + i] = scale * (__uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7440u | i)) - 8388736.0f);
          }
        }
      };
      auto inputs = [&](int t, float4& x0, float4& x1) {
        const float* x = args.x + static_cast<size_t>(min(t, tokens - 1)) * args.cols + b * kSuperBlock + at;
        x0 = *reinterpret_cast<const float4*>(x);
        x1 = *reinterpret_cast<const float4*>(x + kApart);
      };
      auto add = [&](float& to, const float (&w)[8], const float4& x0, const float4& x1) {
        float sum = fmaf(w[0], x0.x, fmaf(w[1], x0.y, fmaf(w[2], x0.z, w[3] * x0.w)));
        sum = fmaf(w[4], x1.x, fmaf(w[5], x1.y, fmaf(w[6], x1.z, fmaf(w[7], x1.w, sum))));
        to += sum;
      };
      if constexpr (M <= 2 && (AHEAD || (kQ5 && M == 2))) {
        // The inputs in registers, a row's weights at a time: three blocks an SM.
        float4 x0[M], x1[M];
#pragma unroll
        for (int t = 0; t < M; ++t) {
          inputs(t, x0[t], x1[t]);
        }
#pragma unroll
        for (int r = 0; r < kSplitRows; ++r) {
          float w[8];
          weights(r, w);
#pragma unroll
          for (int t = 0; t < M; ++t) {
            add(acc[r * M + t], w, x0[t], x1[t]);
          }
        }
        ahead();
      } else {
        float w[kSplitRows][8];
#pragma unroll
        for (int r = 0; r < kSplitRows; ++r) {
          weights(r, w[r]);
        }
        ahead();
#pragma unroll
        for (int t = 0; t < M; ++t) {
          float4 x0, x1;
          inputs(t, x0, x1);
#pragma unroll
          for (int r = 0; r < kSplitRows; ++r) {
            add(acc[r * M + t], w[r], x0, x1);
          }
        }
      }
    }
    int first;
    Fold<kSums>(acc, lane, &first);
    static_assert(kFoldLeft<kSums> == 1, "one sum a lane");
    partial[buffer][warp][first] = acc[0];   // several lanes the same, below 32 sums
    __syncthreads();
    const int r = threadIdx.x / M, t = threadIdx.x % M;
    int local = group * kSplitRows + r;
    if (threadIdx.x < kSums && local < args.total_rows && t < tokens) {
      float total = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        total += partial[buffer][k][threadIdx.x];
      }
      int p = 0;
      while (p + 1 < args.nparts && local >= args.parts[p].rows) {
        local -= args.parts[p].rows;
        ++p;
      }
      args.y[static_cast<size_t>(t) * args.y_stride + args.parts[p].out_offset + local] = total;
    }
  }
}

// Whether GemvSplit runs a part: whole 256-value blocks at the alignment of its loads.
bool SplitRuns(const GemvPart& part, int cols) {
  const uintptr_t align = part.type == GUFO_CUDA_Q5_K ? 16 : 4;
  return (part.type == GUFO_CUDA_Q5_K || part.type == GUFO_CUDA_Q8_0) && cols % kSuperBlock == 0 &&
         reinterpret_cast<uintptr_t>(part.data) % align == 0 && part.row_bytes % align == 0;
}

// Which form of GemvSplit. Three tokens and more read ahead, and where there are more groups
// than three rounds of blocks (fewer are dealt out by the hardware as they finish) a block
// takes several. One or two tokens:
//   - many groups of short rows (2048 values of Q5_K, 1280 with two tokens, 5120 of Q8_0): the
//     same, a block's start and its first load are much of it. A block for every group / several,
//     us: Q5_K 24576 x 1024 25.4 / 20.9, x 3072 48.9 / 49.2, x 9728 121 / 130; two tokens x 1280
//     (20000 rows) 24.6 / 23.3, x 1536 25.7 / 28.1; Q8_0 24576 x 1024 17.8 / 13.3, x 5120 43.7 /
//     44.6, x 9728 71 / 79.
//   - fewer, or longer rows: a block a group. Read ahead is what the library holds: Q8_0, but
//     not for two tokens and long rows in more than one round (4096 x 9728 19.4 us, 18.8
//     without); short Q5_K rows of one token in more than one and a half (4096 x 2048 6.9,
//     7.3 without; 2048 x 1536 3.7, 3.5 without). One token's Q8_0 rows in more than one round
//     take that form for its prefetch even where they are borrowed (5000 x 1280 5.7 us, 6.2
//     without). Many long ones keep the loop over one group, with which the compiler's code
//     is faster (24576 x 9728 80 us without it, 71 with it).
template <int TYPE>
int LaunchSplit(gufo_cuda_ctx* ctx, const GemvArgs& args, int tokens) {
  const int groups = static_cast<int>((args.total_rows + kSplitRows - 1) / kSplitRows);
  bool early = true;
  for (int p = 0; p < args.nparts; ++p) {
    early = early && !args.parts[p].borrowed;
  }
  auto resident = [&](auto kernel) { return std::max(1, ResidentBlocks(kernel, ctx->device, 256, 0, 1)); };
  auto launch = [&](auto kernel, int grid) {
    return LaunchOverlapped(kernel, dim3(grid), dim3(256), 0, ctx->stream, 1, args, tokens, early);
  };
  auto ahead = [&](auto kernel) {
    const int round = resident(kernel);
    return launch(kernel, groups <= 3 * round ? groups : round);
  };
  constexpr bool kQ5 = TYPE == GUFO_CUDA_Q5_K;
  if (tokens == 1) {
    const int round = resident(GemvSplit<TYPE, 1, true>);
    const bool many = groups > 3 * round;
    const bool shorter = args.cols <= (kQ5 ? 2048 : 5120);
    const bool read_ahead = many ? shorter : kQ5 ? shorter && early && 2 * groups > 3 * round : early || groups > round;
    GUFO_CUDA_TRY(read_ahead     ? ahead(GemvSplit<TYPE, 1, true>)
                  : kQ5 || !many ? launch(GemvSplit<TYPE, 1, false>, groups)
                                 : launch(GemvSplit<TYPE, 1, false, !kQ5>, groups));
  } else if (tokens == 2) {
    const int round = resident(GemvSplit<TYPE, 2, true>);
    const bool shorter = args.cols <= (kQ5 ? 1280 : 5120);
    const bool read_ahead = groups > 3 * round ? shorter : !kQ5 && early && (shorter || groups <= round);
    GUFO_CUDA_TRY(read_ahead ? ahead(GemvSplit<TYPE, 2, true>) : launch(GemvSplit<TYPE, 2, false>, groups));
  } else {
    GUFO_CUDA_TRY(tokens <= 4 ? ahead(GemvSplit<TYPE, 4, true>) : ahead(GemvSplit<TYPE, 8, true>));
  }
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

template <int M>
int LaunchRows(gufo_cuda_ctx* ctx, const GemvArgs& args) {
  const int warps = 8;
  const dim3 grid((args.total_rows + warps - 1) / warps, args.group_ids != nullptr ? args.groups : 1);
  GUFO_CUDA_TRY(LaunchOverlapped(GemvRows<M>, grid, dim3(warps * 32), 0, ctx->stream, 1, args));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

// Host rows into device memory, read straight from mapped pinned memory: a launch
// and a PCIe round trip, where a copy costs the copy engine's start and its
// hand-over to the next kernel (8 KB: 3 us against 10).
__global__ void __launch_bounds__(256)
FetchKernel(const float* __restrict__ src, float* __restrict__ dst, int64_t n) {
  GridLaunchDependents();
  GridDependencyWait();   // dst may still be read by the product before
  for (int64_t i = 4 * (blockIdx.x * static_cast<int64_t>(256) + threadIdx.x); i < n; i += 4 * 256 * static_cast<int64_t>(gridDim.x)) {
    if (i + 4 <= n) {
      *reinterpret_cast<float4*>(dst + i) = __ldcv(reinterpret_cast<const float4*>(src + i));
    } else {
      for (int64_t j = i; j < n; ++j) {
        dst[j] = __ldcv(src + j);
      }
    }
  }
}

}  // namespace

// Enqueues y = [W_0 x | W_1 x | ...]: many rows of Q4_K and Q6_K parts on the tcgen05
// GEMM, F32 parts in one launch for all tokens; then, at most kMaxTokens tokens a
// pass, Q4_K and Q6_K parts on the tensor-core GEMV kernels (up to kFastMaxParts of a
// format a launch; x converted in them, or once ahead of them), Q5_K and Q8_0 rows of
// whole blocks on GemvSplit and whatever is left together on the general kernel.
int LaunchGemv(gufo_cuda_ctx* ctx, const GemvArgs& base, int tokens) {
  if (tokens >= 16 && (reinterpret_cast<uintptr_t>(base.x) & 15) == 0) {
    // Many token rows: the parts the tcgen05 GEMM runs read their weights once
    // for all rows; the other parts take the 8-token passes below.
    GemvArgs tc = base, other = base;
    tc.nparts = other.nparts = 0;
    tc.total_rows = other.total_rows = 0;
    for (int p = 0; p < base.nparts; ++p) {
      GemvArgs& to = TcGemmRuns(ctx, base.parts[p].type, base.cols, tokens) ? tc : other;
      to.parts[to.nparts++] = base.parts[p];
      to.total_rows += base.parts[p].rows;
    }
    if (tc.nparts > 0) {
      const int rc = LaunchGemmTc(ctx, tc, tokens);
      if (rc != GUFO_CUDA_OK || other.nparts == 0) {
        return rc;
      }
      return LaunchGemv(ctx, other, tokens);
    }
  }
  if (!ctx->force_general) {
    GemvArgs f32 = base, other = base;
    f32.nparts = other.nparts = 0;
    f32.total_rows = other.total_rows = 0;
    for (int p = 0; p < base.nparts; ++p) {
      GemvArgs& to = base.parts[p].type == GUFO_CUDA_F32 ? f32 : other;
      to.parts[to.nparts++] = base.parts[p];
      to.total_rows += base.parts[p].rows;
    }
    if (f32.nparts > 0) {
      const int blocks = (f32.total_rows + 7) / 8 * ((tokens + 7) / 8);
      const int rc = blocks < ctx->sm_count ? LaunchRowsF32<2>(ctx, f32, tokens) : LaunchRowsF32<8>(ctx, f32, tokens);
      if (rc != GUFO_CUDA_OK || other.nparts == 0) {
        return rc;
      }
      return LaunchGemv(ctx, other, tokens);
    }
  }
  // Tokens per pass: as many as the images of the tensor-core kernels hold (eight rows
  // of 9728 values do not fit, four do: two passes, 33 us at 2560 rows of Q6_K, instead
  // of the general kernel's one, 87 us).
  int most = kMaxTokens;
  for (int p = 0; p < base.nparts && !ctx->force_general; ++p) {
    const int type = base.parts[p].type;
    if (type == GUFO_CUDA_Q4_K || type == GUFO_CUDA_Q6_K) {
      auto* fits = type == GUFO_CUDA_Q4_K ? Q4KFastFits : Q6KFastFits;
      while (fits(base.cols, 1) && !fits(base.cols, most)) {
        --most;
      }
    }
  }
  if (most < tokens) {
    const int passes = (tokens + most - 1) / most;
    most = (tokens + passes - 1) / passes;   // of one size
  }
  for (int t0 = 0; t0 < tokens; t0 += most) {
    const int m = tokens - t0 < most ? tokens - t0 : most;
    const float* x = base.x + static_cast<size_t>(t0) * base.cols;
    float* y = base.y + static_cast<size_t>(t0) * base.y_stride;
    GemvArgs rest = base;
    rest.nparts = 0;
    rest.total_rows = 0;
    rest.x = x;
    rest.y = y;
    const bool fast4 = !ctx->force_general && Q4KFastFits(base.cols, m);
    const bool fast6 = !ctx->force_general && Q6KFastFits(base.cols, m);
    // Parts of one block format share one staged image and one launch.
    for (int type : {GUFO_CUDA_Q4_K, GUFO_CUDA_Q6_K}) {
      if (!(type == GUFO_CUDA_Q4_K ? fast4 : fast6)) {
        continue;
      }
      FastGemvArgs args{};
      args.cols = base.cols;
      args.y = y;
      args.y_stride = base.y_stride;
      args.tokens = m;
      // Every thread block can stage x itself, or one staging kernel does it for all
      // and the blocks copy the image. One token: always in the block (it reads x with
      // 16-byte loads). More tokens, where the conversion is short beside a launch
      // (2.8 us of host time, and one more step of the chain): two units per warp (a
      // unit: 256 values of a row), or five where no block multiplies a second tile.
      // Two rows through a layer of 2048 x 6144: 25.0 -> 20.5 us, eight of
      // 1024 x 2048: 24.8 -> 17.3; beyond the line the conversions, repeated in every
      // block, take longer than the launch (four rows of 2560 x 9728: 40.4 -> 45.8).
      const bool aligned = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
      const int units = m * (base.cols / kSuperBlock);
      const bool small = units <= 2 * kFastWarps || (units <= 5 * kFastWarps && base.total_rows <= 16 * 2 * ctx->sm_count);
      args.prologue = (m == 1 || small) && aligned && !ctx->reuse_image ? kProloguePlain : kPrologueImage;
      args.x = x;
      bool staged = false;
      auto flush = [&]() -> int {
        if (args.nparts == 0) {
          return GUFO_CUDA_OK;
        }
        const int rc = type == GUFO_CUDA_Q4_K ? LaunchGemvQ4KFast(ctx, args) : LaunchGemvQ6KFast(ctx, args);
        args.nparts = 0;
        return rc;
      };
      for (int p = 0; p < base.nparts; ++p) {
        const GemvPart& part = base.parts[p];
        if (part.type != type) {
          continue;
        }
        if (args.prologue == kPrologueImage && !staged) {
          staged = true;
          // High nibbles of Q4_K reach the MMA as 16 q, Q6_K codes as 4 (q - 32): the
          // factors carry 1/16 and 1/4.
          const int rc = StageActivations(ctx, x, m, base.cols, type == GUFO_CUDA_Q4_K ? 32 : 16,
                                          type == GUFO_CUDA_Q4_K ? 1.0f / 16.0f : 0.25f, &args.image);
          if (rc != GUFO_CUDA_OK) {
            return rc;
          }
        }
        args.row_bytes = part.row_bytes;
        args.parts[args.nparts++] = {part.data, part.rows, part.out_offset};
        if (args.nparts == kFastMaxParts) {
          const int rc = flush();
          if (rc != GUFO_CUDA_OK) {
            return rc;
          }
        }
      }
      const int rc = flush();
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
    }
    GemvArgs split5 = rest, split8 = rest;
    for (int p = 0; p < base.nparts; ++p) {
      const GemvPart& part = base.parts[p];
      if ((fast4 && part.type == GUFO_CUDA_Q4_K) || (fast6 && part.type == GUFO_CUDA_Q6_K)) {
        continue;
      }
      GemvArgs& to = ctx->force_general || !SplitRuns(part, base.cols) ? rest
                     : part.type == GUFO_CUDA_Q5_K                     ? split5
                                                                       : split8;
      to.parts[to.nparts++] = part;
      to.total_rows += part.rows;
    }
    if (split5.nparts > 0) {
      const int rc = LaunchSplit<GUFO_CUDA_Q5_K>(ctx, split5, m);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
    }
    if (split8.nparts > 0) {
      const int rc = LaunchSplit<GUFO_CUDA_Q8_0>(ctx, split8, m);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
    }
    if (rest.nparts == 0) {
      continue;
    }
    int rc = GUFO_CUDA_OK;
    switch (m) {
      case 1: rc = LaunchRows<1>(ctx, rest); break;
      case 2: rc = LaunchRows<2>(ctx, rest); break;
      case 3: rc = LaunchRows<3>(ctx, rest); break;
      case 4: rc = LaunchRows<4>(ctx, rest); break;
      case 5: rc = LaunchRows<5>(ctx, rest); break;
      case 6: rc = LaunchRows<6>(ctx, rest); break;
      case 7: rc = LaunchRows<7>(ctx, rest); break;
      default: rc = LaunchRows<8>(ctx, rest); break;
    }
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  return GUFO_CUDA_OK;
}

namespace {

// act[g][i] = silu(x[g][i]) * x[g][n + i] for the groups that run.
__global__ void __launch_bounds__(256)
SwiGluGroups(const float* __restrict__ x, int n, int x_stride, int x_div, const int* __restrict__ ids,
             float* __restrict__ act) {
  const int g = blockIdx.y;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (ids[g] < 0 || i >= n) {
    return;
  }
  const float* in = x + static_cast<size_t>(g / x_div) * x_stride;
  const float v = in[i];
  act[static_cast<size_t>(g) * n + i] = v * (1.0f / (1.0f + expf(-v))) * in[n + i];
}

}  // namespace

// Whether a grouped gate / up product can leave silu(gate) * up by itself (two
// Q4_K parts of equal whole tiles on the tensor-core kernel).
bool GroupedSwiGluInProduct(const gufo_cuda_ctx* ctx, const GemvArgs& base) {
  const bool aligned = (reinterpret_cast<uintptr_t>(base.x) & 15) == 0 && base.x_group_stride % 4 == 0;
  return !ctx->force_general && aligned && Q4KFastFits(base.cols, 1) && base.nparts == 2 &&
         base.parts[0].type == GUFO_CUDA_Q4_K && base.parts[1].type == GUFO_CUDA_Q4_K &&
         base.parts[0].rows == base.parts[1].rows && base.parts[0].rows % 16 == 0;
}

int LaunchGemvGrouped(gufo_cuda_ctx* ctx, const GemvArgs& base, int prologue, float* scratch, bool activate) {
  if (base.group_ids == nullptr || base.groups <= 0 ||
      (prologue != kProloguePlain && prologue != kPrologueSwiGlu)) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "grouped product: ids, groups and a plain or SwiGLU input");
  }
  const bool aligned = (reinterpret_cast<uintptr_t>(base.x) & 15) == 0 && base.x_group_stride % 4 == 0;
  const bool fast4 = !ctx->force_general && aligned && Q4KFastFits(base.cols, 1);
  GemvArgs rest = base;
  rest.nparts = 0;
  rest.total_rows = 0;
  FastGemvArgs args{};
  args.cols = base.cols;
  args.y = base.y;
  args.y_stride = base.y_stride;
  args.tokens = 1;
  args.prologue = prologue;
  args.x = base.x;
  args.group_ids = base.group_ids;
  args.groups = base.groups;
  args.x_group_stride = base.x_group_stride;
  args.x_group_div = base.x_group_div;
  args.early_input = base.early_input;
  args.y_group_stride = base.y_group_stride;
  if (activate) {
    if (!GroupedSwiGluInProduct(ctx, base)) {
      return Fail(GUFO_CUDA_UNSUPPORTED_TYPE, "grouped product: these parts cannot activate their own rows");
    }
    args.epilogue = kEpilogueSwiGlu;
  }
  for (int p = 0; p < base.nparts; ++p) {
    const GemvPart& part = base.parts[p];
    if (fast4 && part.type == GUFO_CUDA_Q4_K) {
      args.row_bytes = part.row_bytes;
      args.parts[args.nparts++] = {part.data, part.rows, part.out_offset};
      if (args.nparts == kFastMaxParts) {
        const int rc = LaunchGemvQ4KFast(ctx, args);
        if (rc != GUFO_CUDA_OK) {
          return rc;
        }
        args.nparts = 0;
      }
    } else {
      rest.parts[rest.nparts++] = part;
      rest.total_rows += part.rows;
    }
  }
  if (args.nparts > 0) {
    const int rc = LaunchGemvQ4KFast(ctx, args);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  if (rest.nparts > 0) {
    if (prologue == kPrologueSwiGlu) {
      if (scratch == nullptr) {
        return Fail(GUFO_CUDA_BAD_ARGUMENT, "grouped product: no scratch for the activated input");
      }
      SwiGluGroups<<<dim3((base.cols + 255) / 256, base.groups), 256, 0, ctx->stream>>>(
          base.x, base.cols, base.x_group_stride, base.x_group_div > 1 ? base.x_group_div : 1, base.group_ids, scratch);
      ctx->launches.fetch_add(1);
      rest.x = scratch;
      rest.x_group_stride = base.cols;
      rest.x_group_div = 1;
    }
    return LaunchRows<1>(ctx, rest);
  }
  return GUFO_CUDA_OK;
}

}  // namespace gufo

using gufo::Fail;

namespace gufo {

// Validates `parts` and fills the launch arguments; ctx->mu is held.
int BuildGemvArgs(gufo_cuda_ctx* ctx, const gufo_cuda_rows* parts, int nparts,
                  GemvArgs* args) {
  if (nparts < 1 || nparts > gufo::kMaxParts) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: 1 to 8 parts per product");
  }
  int64_t total = 0;
  int64_t cols = 0;
  for (int p = 0; p < nparts; ++p) {
    const gufo::Matrix* m = ctx->FindMatrix(parts[p].w);
    if (m == nullptr) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: unknown matrix handle");
    }
    if (parts[p].first < 0 || parts[p].rows <= 0 ||
        parts[p].first + parts[p].rows > m->rows) {
      return Fail(GUFO_CUDA_SHAPE, "matmul: row range outside the matrix");
    }
    if (m->type == GUFO_CUDA_F16 || m->type == GUFO_CUDA_BF16) {
      return Fail(GUFO_CUDA_UNSUPPORTED_TYPE, "matmul: F16 / BF16 rows are dequantized only, not multiplied");
    }
    if (p == 0) {
      cols = m->cols;
    } else if (m->cols != cols) {
      return Fail(GUFO_CUDA_SHAPE, "matmul: parts differ in input width");
    }
    gufo::GemvPart& out = args->parts[p];
    out.data = m->data + static_cast<size_t>(parts[p].first) * m->row_bytes;
    out.rows = static_cast<int>(parts[p].rows);
    out.out_offset = static_cast<int>(total);
    out.type = m->type;
    out.row_bytes = static_cast<int>(m->row_bytes);
    out.borrowed = !m->owned;
    total += parts[p].rows;
  }
  if (total > INT32_MAX || cols > INT32_MAX) {
    return Fail(GUFO_CUDA_SHAPE, "matmul: product too large");
  }
  args->nparts = nparts;
  args->total_rows = static_cast<int>(total);
  args->y_stride = static_cast<int>(total);
  args->cols = static_cast<int>(cols);
  return GUFO_CUDA_OK;
}

}  // namespace gufo

extern "C" {

int gufo_cuda_matmul_device(gufo_cuda_ctx* ctx, const gufo_cuda_rows* parts,
                            int nparts, const float* device_x, int tokens,
                            float* device_y) {
  if (ctx == nullptr || parts == nullptr || device_x == nullptr || device_y == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: null pointer");
  }
  if (tokens < 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: negative token count");
  }
  if (reinterpret_cast<uintptr_t>(device_x) % 16 != 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: x must be 16-byte aligned");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  gufo::GemvArgs args{};
  int rc = gufo::BuildGemvArgs(ctx, parts, nparts, &args);
  if (rc != GUFO_CUDA_OK || tokens == 0) {
    return rc;
  }
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  args.x = device_x;
  args.y = device_y;
  return gufo::LaunchGemv(ctx, args, tokens);
}

int gufo_cuda_matmul(gufo_cuda_ctx* ctx, const gufo_cuda_rows* parts, int nparts,
                     const float* host_x, int tokens, float* host_y) {
  if (ctx == nullptr || parts == nullptr || host_x == nullptr || host_y == nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: null pointer");
  }
  if (tokens < 0) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "matmul: negative token count");
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  gufo::GemvArgs args{};
  int rc = gufo::BuildGemvArgs(ctx, parts, nparts, &args);
  if (rc != GUFO_CUDA_OK || tokens == 0) {
    return rc;
  }
  GUFO_CUDA_TRY(cudaSetDevice(ctx->device));
  const size_t x_values = static_cast<size_t>(tokens) * args.cols, x_bytes = 4 * x_values;
  const size_t y_values = static_cast<size_t>(tokens) * args.total_rows, y_bytes = 4 * y_values;
  rc = ctx->Reserve(&ctx->stage_x, &ctx->stage_x_bytes, x_bytes);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  // x: from pinned memory (the caller's, or the context's after a copy by this
  // thread) a kernel fetches it; more than kStagedBytes of pageable memory are left
  // to the driver's copy, whose fixed cost no longer counts there.
  constexpr size_t kStagedBytes = 1u << 20;
  const float* from = static_cast<const float*>(gufo::DeviceAddress(host_x, x_bytes));
  if (from == nullptr && x_bytes <= kStagedBytes &&
      ctx->ReserveHost(&ctx->host_x, &ctx->host_x_bytes, x_bytes) == GUFO_CUDA_OK) {
    std::memcpy(ctx->host_x, host_x, x_bytes);
    from = static_cast<const float*>(gufo::DeviceAddress(ctx->host_x, x_bytes));
  }
  // y: the GEMV kernels store up to kDirectValues straight into pinned memory
  // (posted writes, hidden behind the weights); more go through device memory and a
  // copy, as single rows are a poor fit for PCIe.
  constexpr size_t kDirectValues = 16384;
  float* to = static_cast<float*>(gufo::DeviceAddress(host_y, y_bytes));
  float* stage = nullptr;   // pinned memory that stands for a pageable y
  if (to == nullptr && y_bytes <= kStagedBytes &&
      ctx->ReserveHost(&ctx->host_y, &ctx->host_y_bytes, y_bytes) == GUFO_CUDA_OK) {
    stage = ctx->host_y;
    to = static_cast<float*>(gufo::DeviceAddress(stage, y_bytes));
  }
  const bool direct = to != nullptr && tokens <= gufo::kMaxTokens && y_values <= kDirectValues;
  auto enqueue = [&]() -> int {
    if (from != nullptr && reinterpret_cast<uintptr_t>(from) % 16 == 0 && x_bytes <= kStagedBytes) {
      const int blocks = static_cast<int>((x_values + 1023) / 1024);
      GUFO_CUDA_TRY(gufo::LaunchOverlapped(gufo::FetchKernel, dim3(blocks), dim3(256), 0, ctx->stream, 1, from,
                                           ctx->stage_x, static_cast<int64_t>(x_values)));
      ctx->launches.fetch_add(1);
    } else {
      GUFO_CUDA_TRY(cudaMemcpyAsync(ctx->stage_x, host_x, x_bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    args.x = ctx->stage_x;
    if (direct) {
      args.y = to;
      return gufo::LaunchGemv(ctx, args, tokens);
    }
    int status = ctx->Reserve(&ctx->stage_y, &ctx->stage_y_bytes, y_bytes);
    if (status != GUFO_CUDA_OK) {
      return status;
    }
    args.y = ctx->stage_y;
    status = gufo::LaunchGemv(ctx, args, tokens);
    if (status != GUFO_CUDA_OK) {
      return status;
    }
    GUFO_CUDA_TRY(cudaMemcpyAsync(stage != nullptr ? stage : host_y, ctx->stage_y, y_bytes, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    return GUFO_CUDA_OK;
  };
  rc = enqueue();
  // Also where it failed half way: the caller's buffers are its own again.
  const cudaError_t waited = cudaStreamSynchronize(ctx->stream);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  GUFO_CUDA_TRY(waited);
  if (stage != nullptr) {
    std::memcpy(host_y, stage, y_bytes);
  }
  return GUFO_CUDA_OK;
}

}  // extern "C"
