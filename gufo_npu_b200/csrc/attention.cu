// Decode attention of one token in one launch: Mixer::Attention
// (src/models/qwen35/decoder.cpp:267-412 in the reference) for head dimensions 64,
// 128 and 256. q/k RMSNorm and RoPE, the cache append, softmax over the cached
// positions and the output gate.
//
// What bounds it. Up to a few thousand positions, latency: the kernel boundary, one
// L2 round trip for the input row, one for the cache rows (a context's last rows sit
// in L2, older ones in HBM), the norm. The three launches this replaces (norm and
// RoPE; slices; merge) had two more boundaries, and their slices summed every dot
// product over a warp with shuffles: 40 instructions per position and query head.
//
// The split. A grid of `splits` blocks per KV head; of those only as many work as
// the context is long enough for: loading costs 10 ns per position and block, and
// merging 10 ns per query head and block (512 bytes against 1 KB at an SM's 100
// GB/s), so the sum is least at sqrt(length / group) blocks; up to kAlone positions
// one block does all, and then nothing has to be merged. A block takes its positions
// in chunks of 64, two in flight (cp.async). The last block of a KV head to arrive
// at a counter merges the partial results: as fast here as a launch of its own, and
// not paid at all by short contexts.
//
// The arithmetic. Per chunk, scores and weighted sums are mma.sync products with
// the group's (at most eight) query heads as the rows and the fp16 cache rows as they
// are. The fp32 operands (queries; probabilities) are split into two halves, rows
// 0-7 and 8-15 of the same instruction, so that 22 bits of them count, scaled by a
// power of two ahead of the split so that small ones keep their bits as well; each
// instruction's sixteen products are added up in fp32 (MmaF16). Warps take the chunk's
// positions for the scores, the query heads for the softmax, the head's dimensions for
// the sums.
//
// 8 query heads on 2 KV heads of 256: 4096 positions 12.3 -> 4.8 us, 16384 positions
// 51 -> 10.5 us; a few positions of one KV head of 128: 7.2 -> 3.1 us.
#include <cfloat>

#include "decode_device.cuh"

namespace gufo {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kChunk = 64;          // positions per stage
constexpr int kStages = 2;
constexpr int kAlone = 128;         // positions one block takes by itself
constexpr int kPadHalves = 8;       // row padding: ldmatrix rows fall in distinct banks
constexpr float kProbScale = 16384.0f;
constexpr size_t kCounterBytes = 1024;   // of the stream's scratch: counters of up to 256 KV heads

struct FastAttnArgs {
  AttnArgs a;
  int splits;
  float* sums;        // [kv_heads][splits][group][hd]
  float* stats;       // [kv_heads][splits][group][2]: maximum, sum
  unsigned* arrived;  // [kv_heads], zero between launches
};

template <int HD>
struct Smem {
  static constexpr int kPitch = HD + kPadHalves;
  alignas(16) __half k[kStages][kChunk][kPitch];
  alignas(16) __half v[kStages][kChunk][kPitch];
  alignas(16) __half q[16][kPitch];                    // rows g, g + 8: the two halves of query head g
  alignas(16) __half p[16][kChunk + kPadHalves];       // the same of its probabilities
  alignas(16) __half new_k[HD], new_v[HD];             // this token's row
  float score[8][kChunk];
  float q_scale[8];                                    // score factor of a head
  float keep[8];                                       // rescaling of the sums so far
  float top[8], total[8];
  float weight[8][kAttnMaxSplits];                       // merge: a split's factor
  int last;
};

__device__ __forceinline__ uint32_t Address(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void Ldmatrix4(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(Address(p)));
}
__device__ __forceinline__ void Ldmatrix4Trans(uint32_t (&r)[4], const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(Address(p)));
}
__device__ __forceinline__ void Ldmatrix2Trans(uint32_t& r0, uint32_t& r1, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1) : "r"(Address(p)));
}
// d = a b of sixteen values. The tensor core cuts off what does not fit its adder, so
// sums over more than that are taken with fp32 adds, which round: accumulated by the
// instruction, the outputs were up to three times as far from a float64 result as with
// fp32 arithmetic throughout (16384 positions: 7.7e-7 against 2.6e-7; now 2.4e-7). It
// costs 3 % of the time at 16000 positions and nothing up to 4096 (loops rolled to make
// up for the longer code: no faster in a step, 3 % slower at 16000).
__device__ __forceinline__ void MmaF16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void Add4(float (&d)[4], const float (&x)[4]) {
  d[0] += x[0], d[1] += x[1], d[2] += x[2], d[3] += x[3];
}

// RMSNorm and RoPE of one head by a warp: lane l ends with elements l, l + 32, ...
// (decoder.cpp:280-323). The angles are double as in the reference.
template <int HD>
__device__ __forceinline__ void NormRope(const AttnArgs& a, const float* x, const float* w, int pos, int lane,
                                         float* row, float (&out)[HD / 32]) {
  constexpr int kPer = HD / 32;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    out[i] = __ldcg(x + lane + 32 * i);
    sq = fmaf(out[i], out[i], sq);
  }
  sq = WarpSum(sq);
  const float inv = 1.0f / sqrtf(sq / static_cast<float>(HD) + a.rms_eps);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    row[lane + 32 * i] = out[i] * inv * w[lane + 32 * i];
  }
  __syncwarp();
  const int half = a.rope_dim / 2;
  for (int i = lane; i < half; i += 32) {
    const double angle = static_cast<double>(pos) * static_cast<double>(a.inv_freq[i]);
    double sd, cd;
    sincos(angle, &sd, &cd);
    const float cs = static_cast<float>(cd), sn = static_cast<float>(sd);
    const float lo = row[i], hi = row[i + half];
    row[i] = lo * cs - hi * sn;
    row[i + half] = lo * sn + hi * cs;
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    out[i] = row[lane + 32 * i];
  }
}

// A block's slice once more, for one warp's dimensions, in plain fp32: where something
// is not finite. A product of two halves turns an infinite cache value into NaN (one half
// may be zero, or of the other sign) where the fp32 product is infinite, and a score of
// minus infinity weighs nothing. out: [group][HD / 8 sums | maximum, sum of weights].
template <int HD>
__device__ __noinline__ void SliceInFp32(const AttnArgs& a, const float* in_q, int kh, int group, int pos, int begin,
                                         int end, float* row, float* out) {
  constexpr int kPer = HD / 32, kDims = HD / kWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t stride = static_cast<size_t>(a.kv_heads) * HD;
  const float scale = 1.0f / sqrtf(static_cast<float>(HD));
  for (int head = 0; head < group; ++head) {
    float q[kPer];
    NormRope<HD>(a, in_q + static_cast<size_t>(head) * 2 * HD, a.q_norm, pos, lane, row, q);
    auto score = [&](int j) {
      const __half* k = a.keys + static_cast<size_t>(j) * stride + static_cast<size_t>(kh) * HD;
      float dot = 0.f;
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        dot = fmaf(q[i], __half2float(k[lane + 32 * i]), dot);
      }
      return WarpSum(dot) * scale;
    };
    float top = -INFINITY, total = 0.f, value = 0.f;
    for (int j = begin; j < end; ++j) {
      const float s = score(j);
      top = fmaxf(top, s);
      total = s != s ? s : total;   // a NaN is the result
    }
    for (int j = begin; j < end && (top > -INFINITY || total != total); ++j) {
      const float p = expf(score(j) - top);
      total += p;
      if (lane < kDims) {
        value = fmaf(p, __half2float(a.values[static_cast<size_t>(j) * stride + static_cast<size_t>(kh) * HD + warp * kDims + lane]),
                     value);
      }
    }
    if (lane < kDims) {
      out[head * (kDims + 2) + lane] = value * kProbScale;
    }
    if (lane == 0) {
      out[head * (kDims + 2) + kDims] = top;
      out[head * (kDims + 2) + kDims + 1] = total;
    }
    __syncwarp();
  }
}

template <int HD>
__global__ void __launch_bounds__(kThreads)
AttnKernel(const __grid_constant__ FastAttnArgs f) {
  extern __shared__ __align__(16) uint8_t raw[];
  Smem<HD>& s = *reinterpret_cast<Smem<HD>*>(raw);
  const AttnArgs& a = f.a;
  constexpr int kPer = HD / 32;
  constexpr int kPieces = HD / 8;              // 16-byte pieces of a row
  const int split = blockIdx.x, kh = blockIdx.y;
  const int group = a.heads / a.kv_heads;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  GridLaunchDependents();
  GridDependencyWait();
  const int pos = *a.position + a.offset;
  const int length = pos + 1;
  int active = 1;
  if (length > kAlone) {
    active = static_cast<int>(ceilf(sqrtf(static_cast<float>(length) / static_cast<float>(group))));
    active = min(active, f.splits);
  }
  const int slice = (length + active - 1) / active;
  active = (length + slice - 1) / slice;       // no empty slice at the end
  if (split >= active) {
    return;
  }
  const int begin = split * slice;
  const int end = min(length, begin + slice);
  const int chunks = (end - begin + kChunk - 1) / kChunk;
  const bool owner = end == length;            // this block appends the token's row
  const size_t stride = static_cast<size_t>(a.kv_heads) * HD;

  // The rows of chunk c; rows past the end and this token's own are zeros for now.
  auto load = [&](int c) {
    if (c < chunks) {
      const int first = begin + c * kChunk;
      for (int i = threadIdx.x; i < kChunk * kPieces; i += kThreads) {
        const int r = i / kPieces, piece = i % kPieces;
        const int j = first + r;
        const bool there = j < end && j < pos;
        const size_t at = static_cast<size_t>(there ? j : begin) * stride + static_cast<size_t>(kh) * HD + piece * 8;
        const int bytes = there ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(Address(&s.k[c % kStages][r][piece * 8])),
                     "l"(a.keys + at), "r"(bytes) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(Address(&s.v[c % kStages][r][piece * 8])),
                     "l"(a.values + at), "r"(bytes) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < kStages; ++c) {
    load(c);
  }

  // While they are on their way: the queries (warp w: head w), and in the owner
  // this token's key and value (the last warp, after its head if it has one).
  const float scale = 1.0f / sqrtf(static_cast<float>(HD));
  const float* in_q = a.in + static_cast<size_t>(kh) * group * 2 * HD;
  const float* in_k = a.in + static_cast<size_t>(a.heads) * 2 * HD + static_cast<size_t>(kh) * HD;
  __shared__ float rows[kWarps][HD];
  if (warp < group) {
    float q[kPer];
    NormRope<HD>(a, in_q + static_cast<size_t>(warp) * 2 * HD, a.q_norm, pos, lane, rows[warp], q);
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      top = max(top, __float_as_uint(q[i]) & 0x7FFFFFFFu);
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    // The largest element to 2^12 .. 2^13: small ones stay above fp16's subnormals.
    int e = static_cast<int>(top >> 23);
    e = min(max(e, 16), 250);
    const float up = __uint_as_float(static_cast<uint32_t>(266 - e) << 23);          // 2^(139 - e)
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const float x = q[i] * up;
      const __half hi = __float2half_rn(x);
      s.q[warp][lane + 32 * i] = hi;
      s.q[8 + warp][lane + 32 * i] = __float2half_rn(x - __half2float(hi));
    }
    if (lane == 0) {
      s.q_scale[warp] = scale * __uint_as_float(static_cast<uint32_t>(e - 12) << 23);  // 2^(e - 139)
    }
  } else {
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      s.q[warp][lane + 32 * i] = __float2half_rn(0.f);
      s.q[8 + warp][lane + 32 * i] = __float2half_rn(0.f);
    }
    if (lane == 0) {
      s.q_scale[warp] = 0.f;
    }
  }
  for (int i = threadIdx.x; i < 16 * (kChunk + kPadHalves); i += kThreads) {
    (&s.p[0][0])[i] = __float2half_rn(0.f);   // the rows without a head stay zero
  }
  if (lane == 0) {
    s.top[warp] = -INFINITY;
    s.total[warp] = 0.f;
  }
  if (owner && warp == kWarps - 1) {
    float k[kPer];
    NormRope<HD>(a, in_k, a.k_norm, pos, lane, rows[warp], k);
    const float* in_v = in_k + stride;
    const size_t at = static_cast<size_t>(pos) * stride + static_cast<size_t>(kh) * HD;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      const __half hk = __float2half_rn(k[i]);
      const __half hv = __float2half_rn(__ldcg(in_v + lane + 32 * i));
      s.new_k[lane + 32 * i] = hk;
      s.new_v[lane + 32 * i] = hv;
      a.keys[at + lane + 32 * i] = hk;
      a.values[at + lane + 32 * i] = hv;
    }
  }

  constexpr int kTiles = HD / 64;              // eight-dimension tiles of a warp
  const int dim0 = warp * (HD / kWarps);
  float acc[kTiles][4];
#pragma unroll
  for (int n = 0; n < kTiles; ++n) {
    acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  }
  for (int c = 0; c < chunks; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
    const int st = c % kStages;
    const int count = min(kChunk, end - begin - c * kChunk);
    __syncthreads();
    if (owner && c == chunks - 1) {
      for (int i = threadIdx.x; i < 2 * kPieces; i += kThreads) {
        const int piece = i % kPieces;
        __half* to = i < kPieces ? s.k[st][count - 1] : s.v[st][count - 1];
        const __half* from = i < kPieces ? s.new_k : s.new_v;
        *reinterpret_cast<uint4*>(to + piece * 8) = *reinterpret_cast<const uint4*>(from + piece * 8);
      }
      __syncthreads();
    }
    // Scores: warp w takes positions 8w .. 8w + 7.
    if (8 * warp < count) {
      float d[4][4] = {};
#pragma unroll
      for (int k0 = 0; k0 < HD; k0 += 32) {
        uint32_t b[4], q0[4], q1[4];
        Ldmatrix4(b, &s.k[st][8 * warp + (lane & 7)][k0 + 8 * (lane >> 3)]);
        Ldmatrix4(q0, &s.q[lane & 15][k0 + 8 * (lane >> 4)]);
        Ldmatrix4(q1, &s.q[lane & 15][k0 + 16 + 8 * (lane >> 4)]);
        float p0[4], p1[4];
        MmaF16(p0, q0, b[0], b[1]);
        MmaF16(p1, q1, b[2], b[3]);
        Add4(p0, p1);
        Add4(d[(k0 / 32) % 4], p0);
      }
      Add4(d[0], d[1]);
      Add4(d[2], d[3]);
      Add4(d[0], d[2]);
      const float factor = s.q_scale[g];
      s.score[g][8 * warp + 2 * t] = (d[0][0] + d[0][2]) * factor;
      s.score[g][8 * warp + 2 * t + 1] = (d[0][1] + d[0][3]) * factor;
    }
    __syncthreads();
    if (warp < group) {
      const float s0 = lane < count ? s.score[warp][lane] : -INFINITY;
      const float s1 = lane + 32 < count ? s.score[warp][lane + 32] : -INFINITY;
      float top = fmaxf(s0, s1);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
      }
      const float before = s.top[warp];
      top = fmaxf(top, before);
      const float p0 = expf(s0 - top), p1 = expf(s1 - top);
      const float sum = WarpSum(p0 + p1);
      const float x0 = p0 * kProbScale, x1 = p1 * kProbScale;
      const __half h0 = __float2half_rn(x0), h1 = __float2half_rn(x1);
      s.p[warp][lane] = h0;
      s.p[warp][lane + 32] = h1;
      s.p[8 + warp][lane] = __float2half_rn(x0 - __half2float(h0));
      s.p[8 + warp][lane + 32] = __float2half_rn(x1 - __half2float(h1));
      __syncwarp();
      if (lane == 0) {
        const float keep = expf(before - top);   // 0 at the first chunk
        s.keep[warp] = keep;
        s.top[warp] = top;
        s.total[warp] = s.total[warp] * keep + sum;
      }
    }
    __syncthreads();
    // Weighted sums: warp w takes HD / 8 dimensions.
    {
      const float keep = g < group ? s.keep[g] : 0.f;
      float part[kTiles][4] = {};
      auto add = [&](int n, const uint32_t (&p)[4], uint32_t b0, uint32_t b1) {
        float x[4];
        MmaF16(x, p, b0, b1);
        Add4(part[n], x);
      };
#pragma unroll
      for (int k0 = 0; k0 < kChunk; k0 += 16) {
        if (k0 < count) {
          uint32_t p[4];
          Ldmatrix4(p, &s.p[lane & 15][k0 + 8 * (lane >> 4)]);
          if constexpr (kTiles == 1) {
            uint32_t b0, b1;
            Ldmatrix2Trans(b0, b1, &s.v[st][k0 + (lane & 15)][dim0]);
            add(0, p, b0, b1);
          } else {
#pragma unroll
            for (int n = 0; n < kTiles; n += 2) {
              uint32_t b[4];
              Ldmatrix4Trans(b, &s.v[st][k0 + (lane & 15)][dim0 + 8 * n + 8 * (lane >> 4)]);
              add(n, p, b[0], b[1]);
              add(n + 1, p, b[2], b[3]);
            }
          }
        }
      }
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[n][i] = fmaf(acc[n][i], keep, part[n][i]);
        }
      }
    }
    __syncthreads();
    load(c + kStages);
  }

  float top = g < group ? s.top[g] : 0.f, total = g < group ? s.total[g] : 0.f;
  float sum = total;
#pragma unroll
  for (int n = 0; n < kTiles; ++n) {
    sum += (acc[n][0] + acc[n][1]) + (acc[n][2] + acc[n][3]);
  }
  if (__any_sync(0xFFFFFFFFu, !(fabsf(sum) <= FLT_MAX))) {
    constexpr int kDims = HD / kWarps;
    // (The chunks' buffers are free behind the loop's last barrier.)
    float* exact = reinterpret_cast<float*>(s.k) + warp * 8 * (kDims + 2);
    SliceInFp32<HD>(a, in_q, kh, group, pos, begin, end, rows[warp], exact);
    if (g < group) {
      exact += g * (kDims + 2);
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
        acc[n][0] = exact[8 * n + 2 * t];
        acc[n][1] = exact[8 * n + 2 * t + 1];
        acc[n][2] = acc[n][3] = 0.f;
      }
      top = exact[kDims];
      total = exact[kDims + 1];
    }
  }
  // Head g's sums: the two halves' rows added; dimensions dim0 + 8n + 2t, + 1.
  auto finish = [&](int head, int e, float value, float inv_total) {
    const float gate = __ldcg(in_q + static_cast<size_t>(head) * 2 * HD + HD + e);
    a.ctx[(static_cast<size_t>(kh) * group + head) * HD + e] = value * (inv_total * SigmoidDev(gate));
  };
  if (active == 1) {
    if (g < group) {
      const float inv_total = 1.0f / (total * kProbScale);
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
        finish(g, dim0 + 8 * n + 2 * t, acc[n][0] + acc[n][2], inv_total);
        finish(g, dim0 + 8 * n + 2 * t + 1, acc[n][1] + acc[n][3], inv_total);
      }
    }
    return;
  }
  const size_t part = static_cast<size_t>(kh) * f.splits + split;
  if (g < group) {
#pragma unroll
    for (int n = 0; n < kTiles; ++n) {
      float2* to = reinterpret_cast<float2*>(f.sums + (part * group + g) * HD + dim0 + 8 * n + 2 * t);
      *to = make_float2(acc[n][0] + acc[n][2], acc[n][1] + acc[n][3]);
    }
  }
  if (warp == 0 && t == 0 && g < group) {
    f.stats[(part * group + g) * 2] = top;
    f.stats[(part * group + g) * 2 + 1] = total;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s.last = atomicAdd(f.arrived + kh, 1u) == static_cast<unsigned>(active - 1);
  }
  __syncthreads();
  if (!s.last) {
    return;
  }
  __threadfence();
  if (threadIdx.x == 0) {
    f.arrived[kh] = 0;
  }
  const size_t first = static_cast<size_t>(kh) * f.splits;
  if (warp < group) {
    // The slices' factors (at most two a lane), summed in a fixed order.
    float m[2], l[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int at = lane + 32 * i;
      const float2 ml = at < active ? __ldcg(reinterpret_cast<const float2*>(f.stats + ((first + at) * group + warp) * 2))
                                    : make_float2(-INFINITY, 0.f);
      m[i] = ml.x;
      l[i] = ml.y;
    }
    float top = fmaxf(m[0], m[1]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    }
    const float w0 = expf(m[0] - top), w1 = expf(m[1] - top);
    s.weight[warp][lane] = w0;
    s.weight[warp][lane + 32] = w1;
    const float total = WarpSum(w0 * l[0] + w1 * l[1]);
    if (lane == 0) {
      s.total[warp] = total;
    }
  }
  __syncthreads();
  const int values = group * HD;
  for (int e = 4 * threadIdx.x; e < values; e += 4 * kThreads) {
    const int head = e / HD;
    const float* from = f.sums + first * values + e;
    float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int p0 = 0; p0 < active; p0 += 16) {
      float4 v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = __ldcg(reinterpret_cast<const float4*>(from + static_cast<size_t>(min(p0 + i, active - 1)) * values));
      }
      // (Past the end a zero, not a zero weight: the last slice may hold an infinity.)
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = p0 + i < active ? v[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float w = p0 + i < active ? s.weight[head][p0 + i] : 0.f;
        sum.x = fmaf(w, v[i].x, sum.x);
        sum.y = fmaf(w, v[i].y, sum.y);
        sum.z = fmaf(w, v[i].z, sum.z);
        sum.w = fmaf(w, v[i].w, sum.w);
      }
    }
    const float inv_total = 1.0f / (s.total[head] * kProbScale);
    finish(head, e % HD, sum.x, inv_total);
    finish(head, e % HD + 1, sum.y, inv_total);
    finish(head, e % HD + 2, sum.z, inv_total);
    finish(head, e % HD + 3, sum.w, inv_total);
  }
}

template <int HD>
int Launch(gufo_cuda_ctx* ctx, const FastAttnArgs& f) {
  static bool configured[16] = {};
  if (!configured[ctx->device & 15]) {
    GUFO_CUDA_TRY(cudaFuncSetAttribute(AttnKernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(sizeof(Smem<HD>))));
    configured[ctx->device & 15] = true;
  }
  GUFO_CUDA_TRY(LaunchOverlapped(AttnKernel<HD>, dim3(f.splits, f.a.kv_heads), dim3(kThreads), sizeof(Smem<HD>),
                                 ctx->stream, 1, f));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

}  // namespace

bool AttentionFits(const AttnArgs& a) {
  return (a.head_dim == 64 || a.head_dim == 128 || a.head_dim == 256) && a.heads / a.kv_heads <= 8 &&
         ((reinterpret_cast<uintptr_t>(a.keys) | reinterpret_cast<uintptr_t>(a.values)) & 15) == 0;
}

int LaunchAttention(gufo_cuda_ctx* ctx, const AttnArgs& a) {
  FastAttnArgs f{a};
  // One resident block per SM, and no more than a warp's lanes hold twice.
  f.splits = ctx->sm_count / a.kv_heads;
  f.splits = f.splits < 1 || a.kv_heads * sizeof(unsigned) > kCounterBytes ? 1 : f.splits > kAttnMaxSplits ? kAttnMaxSplits : f.splits;
  // Counters and partial sums: a decoder's own, else the stream's, so that calls on
  // several streams share none. A captured call has to do with what the caller gave it,
  // as its graph may run beside any other: kAttnSplits slices of partials less one (for
  // the alignment), and counters in the queries' place, cleared ahead of every launch
  // (a second node of the graph).
  if (a.arrived != nullptr) {
    f.arrived = a.arrived;
    f.sums = a.partials;
  } else if (f.splits > 1) {
    const size_t want = kCounterBytes + static_cast<size_t>(f.splits) * a.heads * (a.head_dim + 2) * 4;
    uint8_t* scratch = nullptr;
    bool fresh = false;
    const int rc = ctx->StreamScratch(gufo_cuda_ctx::kAttnScratch, want, 256u << 10, &scratch, &fresh);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
    if (scratch == nullptr) {
      f.splits = f.splits < kAttnSplits ? f.splits : kAttnSplits - 1;
      f.arrived = reinterpret_cast<unsigned*>(a.queries);
      f.sums = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(a.partials) + 15) & ~static_cast<uintptr_t>(15));
    } else {
      f.arrived = reinterpret_cast<unsigned*>(scratch);
      f.sums = reinterpret_cast<float*>(scratch + kCounterBytes);
    }
    if (scratch == nullptr || fresh) {
      // All counters of a block that stays: the next call may have more KV heads.
      const size_t bytes = scratch == nullptr ? static_cast<size_t>(a.kv_heads) * 4 : kCounterBytes;
      GUFO_CUDA_TRY(cudaMemsetAsync(f.arrived, 0, bytes, ctx->stream));
    }
  }
  f.stats = f.sums + static_cast<size_t>(f.splits) * a.heads * a.head_dim;
  switch (a.head_dim) {
    case 64: return Launch<64>(ctx, f);
    case 128: return Launch<128>(ctx, f);
    default: return Launch<256>(ctx, f);
  }
}

}  // namespace gufo
