// Pieces shared by the tensor-core GEMV kernels: the fixed-point image of the
// activations, its staging kernel's interface and the int8 MMA wrappers.
//
// Why integers. A decode GEMV must stay HBM-bound, which leaves about three
// issue slots per weight; turning 4- and 6-bit codes into fp32 one by one costs
// more than that. The codes are small integers, so the kernels keep them as
// bytes and let `mma.sync.m16n8k32.s32.u8.s8` (16 rows x 32 codes per issue) do
// the multiply-adds exactly, in int32. For that the fp32 activations are held
// as 24-bit fixed point per 256-value block: x = xi * 2^-shift with |xi| < 2^22,
// xi split into three signed bytes (xi = l2 * 65536 + l1 * 256 + l0), one MMA
// column per byte plane. The result is exact up to the 2^-23 (of the block's
// largest |x|) rounding of xi, the same order as fp32 accumulation; the
// per-sub-block scales are applied to the int32 sums, then one int-to-float
// conversion per 256-value block joins the fp32 accumulator of the row.
//
// The image is built once per product by StageKernel (stage.cu) in a
// context-owned device buffer and copied into shared memory by every thread
// block of the GEMV kernel that follows: a producer kernel may also write it
// directly, since it is plain memory.
#pragma once

#include "common.cuh"

namespace gufo {

constexpr int kLimbs = 3;            // byte planes per token
constexpr int kMixLimbs = 4;         // of a mixture's input (one token): the fourth holds what rounding xi took off
constexpr int kPlanePad = 32;        // bytes: plane stride = cols + 32 keeps the
                                     // 64-bit fragment reads free of bank conflicts
constexpr int kFastWarps = 8;
constexpr int kFastThreads = kFastWarps * 32;
constexpr int kMaxTokensFast = 8;    // tokens per launch (three MMA column groups)
// Of dynamic shared memory; the kernels' own arrays (up to 4.5 KB) come on top. The line
// decides how many rows one pass over the weights takes: at 200 KB eight rows of 5120
// values went in two passes (Q6_K, 2560 rows: 20.8 us, in one 14.0).
constexpr int kFastMaxShared = 220 * 1024;

// Byte layout of the staged activations of `tokens` rows of `cols` values,
// identical in global and shared memory. Every offset is a multiple of 16.
struct ImageLayout {
  int tokens;
  int cols;
  int group;         // values per entry of `sums`: 32 (Q4_K) or 16 (Q6_K)
  int kcols;         // MMA columns, a multiple of 8 covering 3 * tokens
  int plane_stride;  // bytes between byte planes
  int scale_at;      // float [cols / 256][kcols]: 2^(8 limb - shift) * extra
  int sums_at;       // float [tokens][cols / group]: fp32 sums of x per group
  int bytes;
};

__host__ __device__ inline ImageLayout MakeImageLayout(int tokens, int cols, int group, int limbs = kLimbs) {
  ImageLayout l;
  l.tokens = tokens;
  l.cols = cols;
  l.group = group;
  l.kcols = (tokens * limbs + 7) / 8 * 8;
  l.plane_stride = cols + kPlanePad;
  l.scale_at = tokens * limbs * l.plane_stride;
  l.sums_at = l.scale_at + (cols / kSuperBlock) * l.kcols * 4;
  l.bytes = l.sums_at + tokens * (cols / group) * 4;
  return l;
}

// Enqueues the staging of x[tokens][cols] into the context's image buffer and
// returns its device address. `extra` scales the column factors.
int StageActivations(gufo_cuda_ctx* ctx, const float* x, int tokens, int cols,
                     int group, float extra, const uint8_t** image);

__device__ __forceinline__ void MmaU8S8(int (&d)[4], const uint32_t (&a)[4],
                                        uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// The same with signed rows (A) as well.
__device__ __forceinline__ void MmaS8S8(int (&d)[4], const uint32_t (&a)[4],
                                        uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 "
      "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}

// ---- bulk copies completing on a shared-memory barrier ------------------------

__device__ __forceinline__ uint32_t SharedAddress(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void MbarInit(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void MbarArrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// True, for every word: none is both 0 and ~0. But only the votes of the whole warp tell, and
// they need the word of every lane, so what depends on the answer comes behind the loads that
// went into the words. A ring slot that asynchronous copies refill is handed back behind it:
// behind a mere __syncwarp the arrival passed loads of the slot that were still under way, and
// now and then a row's weights were those of the block that came next.
__device__ __forceinline__ bool LoadsDone(uint32_t word) {
  return __any_sync(0xFFFFFFFFu, word != 0u) != 0 || __any_sync(0xFFFFFFFFu, word != ~0u) != 0;
}
__device__ __forceinline__ void MbarArriveExpectTx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool MbarTryWait(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// `bytes` (a multiple of 16; both addresses 16-byte aligned) from global to this
// block's shared memory; the barrier's pending byte count drops as they land.
__device__ __forceinline__ void BulkCopy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// SM clock cycles a block waits for bytes it requested itself before giving the
// slab up (about a second; a copy that has not landed by then never will).
constexpr long long kLandLimit = 2000000000ll;

// Converts one 256-value block of one token into the image at `image` (shared
// or global memory): the calling warp's lane holds values 8 * lane .. + 7 of the
// block in v. Writes the three byte planes, the group sums and the column
// factors of block `b`.
template <int LIMBS = kLimbs>
__device__ __forceinline__ void StageBlock(const float (&v)[8], int lane, int tok, int b,
                                           const ImageLayout& l, uint8_t* image, float extra) {
  // Largest magnitude by integer compare of the bit patterns, so that a NaN
  // (above every finite pattern) is not lost.
  uint32_t top = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    top = max(top, __float_as_uint(v[i]) & 0x7FFFFFFFu);
  }
  top = __reduce_max_sync(0xFFFFFFFFu, top);
  int e = static_cast<int>(top >> 23);  // biased exponent of the maximum
  const bool finite = e != 255;
  e = e < 22 ? 22 : e;
  // |x| < 2^(e - 126), so x * 2^(148 - e) stays below 2^22 in magnitude.
  const float up = __uint_as_float(static_cast<uint32_t>(275 - e) << 23);
  const float down = finite ? __uint_as_float(static_cast<uint32_t>(e - 21) << 23)
                            : __uint_as_float(0x7FC00000u);
  // Added to 1.5 * 2^23, x * up is rounded to its nearest integer xi in the low
  // bits of the sum (one fused multiply-add where a conversion runs at a quarter
  // of its rate). xi + 0x808080 has the balanced digits of xi, each offset by
  // 128, in its three low bytes; flipping the offset bits leaves the signed
  // bytes. (A block with an infinity or NaN: any digits, `down` is NaN.)
  uint32_t z[8];
  uint32_t rest[LIMBS == kMixLimbs ? 8 : 1];   // low bytes: the fourth limbs
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t bits = __float_as_uint(fmaf(v[i], up, 12582912.0f));
    if constexpr (LIMBS == kMixLimbs) {
      // What the rounding took off (exact, at most a half), in 254ths: -127 .. 127.
      const float off = fmaf(v[i], up, 12582912.0f - __uint_as_float(bits));
      rest[i] = __float_as_uint(fmaf(off, 254.0f, 12582912.0f));
    }
    z[i] = (bits + (0x808080u - 0x4B400000u)) ^ 0x808080u;
    sum += v[i];
  }
#pragma unroll
  for (int limb = 0; limb < kLimbs; ++limb) {
    const uint32_t pick = 0x0040u + 0x11u * limb;  // byte `limb` of both operands
    const uint32_t w0 = __byte_perm(__byte_perm(z[0], z[1], pick), __byte_perm(z[2], z[3], pick), 0x5410u);
    const uint32_t w1 = __byte_perm(__byte_perm(z[4], z[5], pick), __byte_perm(z[6], z[7], pick), 0x5410u);
    uint8_t* plane = image + static_cast<size_t>(tok * LIMBS + limb) * l.plane_stride;
    *reinterpret_cast<uint2*>(plane + b * kSuperBlock + lane * 8) = make_uint2(w0, w1);
  }
  if constexpr (LIMBS == kMixLimbs) {
    uint8_t* plane = image + static_cast<size_t>(tok * LIMBS + kLimbs) * l.plane_stride;
    *reinterpret_cast<uint2*>(plane + b * kSuperBlock + lane * 8) =
        make_uint2(__byte_perm(__byte_perm(rest[0], rest[1], 0x0040u), __byte_perm(rest[2], rest[3], 0x0040u), 0x5410u),
                   __byte_perm(__byte_perm(rest[4], rest[5], 0x0040u), __byte_perm(rest[6], rest[7], 0x0040u), 0x5410u));
  }
  // Group sums of the fp32 values: the lanes of one group are adjacent.
  const int lanes_per_group = l.group / 8;  // 4 (groups of 32) or 2 (of 16)
  for (int o = 1; o < lanes_per_group; o <<= 1) {
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  }
  if ((lane & (lanes_per_group - 1)) == 0) {
    float* sums = reinterpret_cast<float*>(image + l.sums_at);
    sums[static_cast<size_t>(tok) * (l.cols / l.group) + b * (kSuperBlock / l.group) +
         lane / lanes_per_group] = sum;
  }
  if (lane < LIMBS) {
    // (The fourth case behind its own test: as one more choice here it cost every
    // conversion of the decode step, 4 layers of 256: 683 -> 693 us for eight tokens.)
    float limb = lane == 0 ? 1.f : (lane == 1 ? 256.f : 65536.f);
    if constexpr (LIMBS == kMixLimbs) {
      limb = lane == kLimbs ? 1.f / 254.f : limb;
    }
    float* scale = reinterpret_cast<float*>(image + l.scale_at);
    scale[b * l.kcols + tok * LIMBS + lane] = down * limb * extra;
  }
}

__device__ __forceinline__ float SiluFast(float x) { return x * (1.0f / (1.0f + expf(-x))); }

// The image of a launch whose input is fused in (prologue != kPrologueImage) is
// built by every thread block in its own shared memory, in units of one
// 256-value block of one token: warp w converts units w, w + 8, ...; a lane holds
// eight adjacent values. Rows of several tokens follow one another: the residual,
// its pending add, the normed vector and a plain x `cols` floats apart, a SwiGLU
// input [gate | up] 2 * cols apart.
//
// What bounds it: one L2 round trip for what the kernel before has just written
// (0.8 us), then the issue slots of an SM whose resident blocks all convert at
// once, and block-wide reductions that nothing hides. So a norm's 1 / rms is not
// in the image: the planes are those of (h + delta) * w, and the kernel multiplies
// its row sums by 1 / rms (RowScale) when it stores them. The sum of squares then
// costs no barrier of its own, and units are independent of one another. Eight
// tokens of the 24-layer, 2048-wide decoder: 6.35 -> 6.15 ms.
//
// And the size of the code: in a step whose kernels alternate, what runs once is
// fetched through the instruction caches at every start. With two tokens the loads of
// two units are in flight together, at the price of two copies of the conversion; with
// one token, where a row of 2048 values is one unit a warp, the copies (two, and three
// for a plain row) made the kernel 100 KB instead of 72: the decoder's eight tokens
// took 5.85 instead of 5.6 ms, the 4-layer one's 760 instead of 700 us. (One loop for
// both kinds of input, a single conversion: slower again, 5.98 ms, as the norm's path
// then jumps over the activation's code.)

// The norm weights of the calling warp's first unit, for FillImage: they never
// depend on an earlier kernel, so a kernel asks for them before it waits for its
// predecessor (a layer's norm vector is read once per step: the load goes all the
// way to HBM, about as long as the whole conversion takes).
template <int TOKENS>
__device__ __forceinline__ void LoadNormAhead(const FastGemvArgs& a, float (&w)[8]) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blocks = a.cols / kSuperBlock;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    w[i] = 0.f;
  }
  if (a.prologue == kPrologueResNorm && warp < TOKENS * blocks) {
    int b = warp;
    while (TOKENS > 1 && b >= blocks) {
      b -= blocks;
    }
    const float4 v0 = *reinterpret_cast<const float4*>(a.norm_w + b * kSuperBlock + lane * 8);
    const float4 v1 = *reinterpret_cast<const float4*>(a.norm_w + b * kSuperBlock + lane * 8 + 4);
    w[0] = v0.x, w[1] = v0.y, w[2] = v0.z, w[3] = v0.w;
    w[4] = v1.x, w[5] = v1.y, w[6] = v1.z, w[7] = v1.w;
  }
}

// 1 / rms of token k after FillImage (1 without a norm): the warps' sums of
// squares added in warp order. `inv_n` = 1 / cols.
template <int TOKENS>
__device__ __forceinline__ float RowScale(const FastGemvArgs& a, const float* squares, int k, float inv_n) {
  if (a.prologue != kPrologueResNorm) {
    return 1.f;
  }
  float total = 0.f;
#pragma unroll
  for (int w = 0; w < kFastWarps; ++w) {
    total += squares[w * TOKENS + k];
  }
  return 1.0f / sqrtf(fmaf(total, inv_n, a.eps));
}

// Columns without a token keep a zero factor; independent of the input.
template <int TOKENS, int LIMBS = kLimbs>
__device__ __forceinline__ void ZeroIdleColumns(const ImageLayout& l, int blocks, uint8_t* image) {
  float* scale = reinterpret_cast<float*>(image + l.scale_at);
#pragma unroll 1
  for (int i = threadIdx.x; i < blocks * l.kcols; i += kFastThreads) {
    if (i % l.kcols >= LIMBS * TOKENS) {
      scale[i] = 0.f;
    }
  }
}

// `x` is the plain / SwiGLU input (a.x, or a group's part of it). A block that
// shares its tiles with a cluster (rank `rank` of `ks`, slabs of eight blocks
// dealt round-robin) converts only the blocks of its own slabs; the others are
// never read. keep_w: LoadNormAhead's. squares: [kFastWarps][TOKENS] in shared
// memory, for RowScale. Ends with a __syncthreads. kFastThreads threads.
template <int TOKENS, int LIMBS = kLimbs>
__device__ __forceinline__ void FillImage(const FastGemvArgs& a, const ImageLayout& l,
                                          uint8_t* image, float extra, const float* x,
                                          int rank, int ks, const float (&keep_w)[8],
                                          float* squares, float inv_n) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n = a.cols;
  const int blocks = n / kSuperBlock;
  const bool first = blockIdx.x == 0;
  auto mine = [&](int b) {
    int s = ks == 1 ? rank : b >> 3;
    while (s >= ks) {
      s -= ks;
    }
    return s == rank;
  };
  auto load8 = [&](const float* p, float (&v)[8]) {
    const float4 v0 = *reinterpret_cast<const float4*>(p);
    const float4 v1 = *reinterpret_cast<const float4*>(p + 4);
    v[0] = v0.x, v[1] = v0.y, v[2] = v0.z, v[3] = v0.w;
    v[4] = v1.x, v[5] = v1.y, v[6] = v1.z, v[7] = v1.w;
  };
  auto store8 = [&](float* p, const float (&v)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
  };
  // Unit (tok, b) of the calling warp and the next one, kFastWarps units on.
  int tok = 0, b = warp;
  auto settle = [&]() {
    while (TOKENS > 1 && b >= blocks) {
      b -= blocks;
      ++tok;
    }
  };
  auto live = [&]() { return TOKENS > 1 ? tok < TOKENS : b < blocks; };
  settle();
  if (a.prologue == kPrologueResNorm) {
    // vec::RmsNorm (src/core/vec.hpp:57-63) of the residual stream after its
    // pending add (src/models/qwen35/decoder.cpp:493,504-508).
    constexpr int kBatch = TOKENS == 2 ? 2 : 1;
    if (lane < TOKENS) {
      squares[warp * TOKENS + lane] = 0.f;
    }
    __syncwarp();
    float sq = 0.f;
    bool first_unit = true;
#pragma unroll 1
    while (live()) {
      float v[kBatch][8], d[kBatch][8], w[kBatch][8];
      int at_tok[kBatch], at_b[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        at_tok[j] = live() ? tok : -1;
        at_b[j] = b;
        if (live()) {
          const int at = b * kSuperBlock + lane * 8;
          const size_t row = static_cast<size_t>(tok) * n + at;
          load8(a.h_in + row, v[j]);
          if (a.delta != nullptr) {
            load8(a.delta + row, d[j]);
          }
          if (j > 0 || !first_unit) {
            load8(a.norm_w + at, w[j]);
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              w[j][i] = keep_w[i];
            }
          }
        }
        b += kFastWarps;
        settle();
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (at_tok[j] < 0) {
          continue;
        }
        const int at = at_b[j] * kSuperBlock + lane * 8;
        const size_t row = static_cast<size_t>(at_tok[j]) * n + at;
        if (a.delta != nullptr) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[j][i] += d[j][i];
          }
          // Partial sums of several ranks are added in rank order.
#pragma unroll 1
          for (int p = 1; p < a.delta_parts; ++p) {
            load8(a.delta + static_cast<size_t>(p) * a.delta_stride + row, d[j]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[j][i] += d[j][i];
            }
          }
        }
        if (TOKENS > 1) {
          sq = 0.f;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sq = fmaf(v[j][i], v[j][i], sq);
          w[j][i] *= v[j][i];
        }
        if (first) {
          // Block 0 writes the whole residual stream (and normed vector, below).
          store8(a.h_out + row, v[j]);
        }
        if (TOKENS > 1) {
          const float sum = WarpSum(sq);
          if (lane == 0) {
            squares[warp * TOKENS + at_tok[j]] += sum;
          }
        }
        if (mine(at_b[j])) {
          StageBlock<LIMBS>(w[j], lane, at_tok[j], at_b[j], l, image, extra);
        }
      }
      first_unit = false;
    }
    if (TOKENS == 1) {
      sq = WarpSum(sq);
      if (lane == 0) {
        squares[warp] = sq;
      }
    }
    __syncthreads();
    if (first && a.normed_out != nullptr) {
      tok = 0, b = warp;
      settle();
#pragma unroll 1
      for (; live(); b += kFastWarps, settle()) {
        const float inv = RowScale<TOKENS>(a, squares, tok, inv_n);
        const int at = b * kSuperBlock + lane * 8;
        const size_t row = static_cast<size_t>(tok) * n + at;
        float v[8], w[8];
        load8(a.h_out + row, v);   // this lane's own stores
        load8(a.norm_w + at, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[i] *= w[i] * inv;
        }
        store8(a.normed_out + row, v);
      }
    }
    if (first && threadIdx.x == 0 && a.advance != nullptr) {
      *a.advance += TOKENS;
    }
    return;
  }
  const bool act = a.prologue == kPrologueSwiGlu;
  const size_t stride = act ? 2 * static_cast<size_t>(n) : static_cast<size_t>(n);
  constexpr int kBatch = TOKENS == 2 ? 2 : 1;
#pragma unroll 1
  while (live()) {
    float v[kBatch][8], up[kBatch][8];
    int at_tok[kBatch], at_b[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const bool take = live() && mine(b);
      at_tok[j] = take ? tok : -1;
      at_b[j] = b;
      if (take) {
        const float* xt = x + tok * stride + b * kSuperBlock + lane * 8;
        load8(xt, v[j]);
        if (act) {
          load8(xt + n, up[j]);
        }
      }
      b += kFastWarps;
      settle();
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (at_tok[j] >= 0) {
        if (act) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[j][i] = SiluFast(v[j][i]) * up[j][i];
          }
        }
        StageBlock<LIMBS>(v[j], lane, at_tok[j], at_b[j], l, image, extra);
      }
    }
  }
  __syncthreads();
}

// Tiles of 16 rows are numbered across the parts of a launch, each part
// rounded up to whole tiles.
__device__ __forceinline__ int TotalTiles(const FastGemvArgs& a) {
  int tiles = 0;
#pragma unroll
  for (int p = 0; p < kFastMaxParts; ++p) {
    if (p < a.nparts) {
      tiles += (a.parts[p].rows + 15) >> 4;
    }
  }
  return tiles;
}

// Part and tile-within-part of global tile `tile`.
__device__ __forceinline__ void LocateTile(const FastGemvArgs& a, int tile, int* part, int* local) {
  int p = 0;
#pragma unroll
  for (int i = 0; i < kFastMaxParts - 1; ++i) {
    const int tiles = (a.parts[i].rows + 15) >> 4;
    if (p == i && i + 1 < a.nparts && tile >= tiles) {
      tile -= tiles;
      p = i + 1;
    }
  }
  *part = p;
  *local = tile;
}

// Byte `i` (compile-time) of a word, zero extended.
template <int I>
__device__ __forceinline__ int ByteAt(uint32_t w) {
  return static_cast<int>(__byte_perm(w, 0u, 0x4440u | I));
}

// Byte `I` of a word, a value below 2^23, as a float without the conversion
// pipe: the byte is placed under the exponent of 2^23 and the bias subtracted.
template <int I>
__device__ __forceinline__ float SmallByteToFloat(uint32_t w) {
  return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | I)) - 8388608.0f;
}

}  // namespace gufo
