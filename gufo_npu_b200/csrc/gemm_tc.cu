// Dequant-fused small-M GEMM on the fifth-generation tensor cores: the product
// behind Projections::Apply (GgufProjections::MatMul,
// src/models/qwen35/gguf_projections.cpp:239-286 in the reference) when many
// token rows share one weight read - the ragged verify batch, where every
// sequence brings a few draft tokens, and the rows of a prompt.
//
//   D[128 weight rows][N token columns] (fp32, tensor memory)
//       += W[128][64] (fp16, tensor memory) * X[N][64]^T (fp16, shared memory)
//
// per 64 columns of K; N is the tokens of a group rounded up to 16. The weights
// sit on the MMA's M and reach it through TENSOR MEMORY: a dequant thread owns
// one weight row, i.e. one lane of tensor memory, and leaves its 64 fp16 weights
// there with two tcgen05.st - no address arithmetic, no swizzle, no proxy fence,
// and none of the shared-memory bandwidth that bound the form this replaces
// (weights written to and read back from swizzled shared-memory tiles: 7 bytes
// of shared-memory traffic per weight, 16 weights per cycle and SM). An
// instruction of this shape spends N / 2 cycles, so the tensor core's time falls
// with the tokens instead of being that of 128 of them.
//
// Roles of the 23 warps of a thread block (one per SM):
//   - sixteen dequant warps in four groups of four; group p turns pair p of a
//     block (64 of its 256 values) of 128 rows into tensor memory slot p:
//     w = d*sc*q - dmin*m (DequantQ4_K, src/core/quant.cpp:33-59) in packed fp16
//     arithmetic, as d*sc*(q - 8) + (8*d*sc - dmin*m), or w = d*sc*(q - 32)
//     (DequantQ6_K, :98-125). While the tensor core reads a slot, its group is at
//     the arithmetic of the next block;
//   - one warp brings the raw blocks of 128 rows with tiled TMA (Q4_K: one box
//     of 144 bytes a row, whose row pitch is free of bank conflicts as it is;
//     Q6_K: boxes of its four planes, the wide ones swizzled);
//   - one brings the activation tiles, converted once per product into
//     fp16 tile images that already carry the swizzle (StageHalfKernel);
//   - one issues tcgen05.mma and hands the slots back with
//     tcgen05.commit;
//   - four epilogue warps read the accumulators with tcgen05.ld (lane = weight
//     row, column = token: a store instruction of a warp covers 32 adjacent
//     rows of one token) while the others are on the next tile: tensor memory
//     holds two accumulators beside the four weight slots.
//
// The loaders and the MMA warp walk their loops as whole warps, and the warp's number and
// the tensor memory's address pass through a shuffle: what such a warp computes is then the
// same in all lanes for the compiler too and stays in uniform registers, where the
// asynchronous instructions take their operands from. With the whole role behind one
// thread's predicate an MMA or commit took 47 cycles to issue (1040 of a step's 1880 at 32
// tokens), now 13.
//
// Work split. A unit is a tile of 128 weight rows against one group of tokens; it
// takes `blocks` steps of one 256-value block. Few units are shared by clusters of two to
// eight thread blocks each, whose accumulators meet in distributed shared memory
// (ReduceCluster). Otherwise the launch's units times steps are
// cut into equal contiguous ranges, one per thread block, so the SMs finish
// together whatever the number of tiles (2 x 9728 rows are 152 tiles for 148 SMs)
// where that saves more than the cuts cost (PlanTc). A tile that a cut goes through
// is finished by whichever of its thread blocks comes last, which adds the others'
// partial sums (left in scratch) to its own in block order, so the result does not
// depend on who that is. Nobody waits for another block but for those of its cluster.
//
// What bounds it: small products the chain of staging kernel (2-3 us), hand-over (1), first
// tiles (1) and the sum over a cluster (3); large ones a step, which takes the 1000 cycles of
// dequantization and hand-overs and the tensor core's time (an MMA with A in tensor memory:
// 9.5 + n / 2 cycles) nearly one after the other (StepCycles), and, in a loop of more than
// about 100 tokens, the board's power limit (1.3-1.4 GHz then). Measured, staging included, us
// at 32 / 79 / 128 / 512 tokens, with the roles behind one thread each and shares summed by the
// last block alone, and now: 19456 x 2560 Q4_K 15.9 / 18.8 / 23.3 / 57.3 and 13.9 / 16.2 / 18.8 /
// 48.9; 2560 x 9728 Q6_K 18.0 / 24.8 / 32.5 / 45.2 and 13.9 / 16.3 / 18.3 / 32.3.
//
// Each activation row is scaled by a power of two into fp16 range first and the
// outputs scaled back, so range never costs precision. Rounding w and x to
// fp16 (11 significant bits) bounds the relative L2 error of y near 4e-4.
//
// Every wait on an mbarrier is bounded: a wait that runs out records an error
// code, raises a block-wide abort flag that ends all other waits, and the
// kernel still frees its tensor memory and returns.
#include "gemm_tc.cuh"

#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <iterator>
#include <mutex>
#include <vector>

namespace gufo {

namespace {

constexpr int kTileRows = 128;      // weight rows of one MMA (its M)
constexpr int kTileK = 64;          // values per activation tile (one swizzle row of fp16)
constexpr int kGroups = 4;          // dequant groups = tensor memory slots = pairs of a block
constexpr int kSlotColumns = kTileK / 2;               // 32-bit columns of a slot: two fp16 each
constexpr int kAccColumn = kGroups * kSlotColumns;     // the accumulators' first column
constexpr int kTmemColumns = 512;
constexpr int kAccColumns = kTmemColumns - kAccColumn;
constexpr int kMaxN = kAccColumns / 2;                 // 192 token columns
constexpr int kDequantWarps = 4 * kGroups;
constexpr int kEpilogueWarp = kDequantWarps;           // four, one per lane quarter
constexpr int kRawWarp = kEpilogueWarp + 4;
constexpr int kXWarp = kRawWarp + 1;
constexpr int kMmaWarp = kXWarp + 1;
constexpr int kTcThreads = (kMmaWarp + 1) * 32;
constexpr int kMaxStages = 10;
constexpr long long kWaitCycles = 1ll << 31;           // about a second of SM clocks
constexpr long long kDrainCycles = 1ll << 27;          // the same for what a block that gave up has under way
constexpr int kHeaderBytes = 4096;                     // of the scratch: error word, counters of cut tiles
// Token rows a pass: eight of the widest groups. Their fp16 tiles and the partial sums
// are scratch that stays allocated, so it is bounded (90 MB for rows of 9728 values),
// whatever the prompt; a pass dequantizes the weights once per group anyway.
constexpr int kPassTokens = 8 * 192;
constexpr int kSharedLimit = 227 * 1024;

// The raw bytes of one block of 128 rows in shared memory.
template <int TYPE>
struct Quant;
template <>
struct Quant<GUFO_CUDA_Q4_K> {
  static constexpr int kRawBytes = kTileRows * kQ4KBytes;
  static constexpr int kRawStride = kRawBytes;
};
template <>
struct Quant<GUFO_CUDA_Q6_K> {
  // Boxes 128, 64 and 16 bytes wide.
  static constexpr int kQl = 0, kQh = kTileRows * 128, kSc = kQh + kTileRows * 64, kD = kSc + kTileRows * 16;
  static constexpr int kRawBytes = kD + kTileRows * 16;
  static constexpr int kRawStride = kRawBytes;   // 28 KiB: a multiple of 1024
};

constexpr int kTcMaxParts = 4;

struct TcPart {
  int rows;
  int tiles;               // tiles of 128 rows
  float* out;              // y + the part's first column
};

struct TcGemmArgs {
  CUtensorMap maps[kTcMaxParts * 3];   // [part][map]
  TcPart parts[kTcMaxParts];
  int nparts;
  int blocks;              // 256-value blocks per row: the steps of a unit
  int groups;              // token groups
  int n;                   // token columns of a group, a multiple of 16
  int units;               // tiles * groups
  int cluster;             // thread blocks that share every unit as a cluster (1: none do)
  int per, extra;          // steps of a thread block otherwise: per, one more for the first `extra`
  int raw_stages, x_stages;
  const uint8_t* xh;       // activation tile images [group][blocks * 4][n][64] fp16, swizzled
  const float* unscale;    // [groups * n]: factor that undoes a row's power-of-two scale
  float* partial;          // [thread block][2][n * 128]: sums of tiles that a cut goes through (PartialChunk)
  unsigned* counters;      // [thread block]: arrivals at the tile that starts there
  int tokens;
  int out_stride;          // floats between token rows of y
  int* error;              // device int: 0, or the code of the first wait that ran out
};

// MbarTryWait's test, suspended by the hardware for up to kSuspendNs first: most warps
// of the kernel wait most of the time, and polling took as many issue slots as the
// dequantization.
constexpr uint32_t kSuspendNs = 20000;
__device__ __forceinline__ bool MbarTrySuspended(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity), "r"(kSuspendNs) : "memory");
  return done != 0;
}

// Waits for the phase with `parity` to complete, for at most kWaitCycles and
// only while no thread of the block has given up. Returns false when it did
// not see the phase complete. PATIENT: suspended in between (loaders and
// epilogue, whose waits are long; waking up takes longer). Called by whole warps,
// which leave it converged: what follows are instructions of the warp as one
// (tcgen05.st, tcgen05.ld, elect.sync), and lanes that had seen the phase complete
// at different polls reached them apart.
template <bool PATIENT = false>
__device__ __forceinline__ bool BoundedWait(uint32_t bar, uint32_t parity, volatile int* abort_flag,
                                            int* error, int code) {
  bool done = MbarTryWait(bar, parity);
  if (!done) {
    const long long start = clock64();
    do {
#pragma unroll 1
      for (int i = 0; i < 32 && !done; ++i) {
        done = PATIENT ? MbarTrySuspended(bar, parity) : MbarTryWait(bar, parity);
      }
      if (!done && *abort_flag != 0) {
        break;
      }
      if (!done && clock64() - start >= kWaitCycles) {
        *abort_flag = 1;
        atomicCAS(error, 0, code);
      }
    } while (!done);
  }
  __syncwarp();
  return done;
}

// After a wait that ran out: waits, with a limit, for the phase of an asynchronous operation
// that this warp has started. A block must not end before these: copies would land in the
// shared memory of the next one, and MMAs use tensor memory that is given back.
__device__ __forceinline__ void Drain(uint32_t bar, uint32_t parity) {
  const long long start = clock64();
#pragma unroll 1
  while (!MbarTryWait(bar, parity) && clock64() - start < kDrainCycles) {
  }
  __syncwarp();
}

// The same for the fills of a ring of `stages` stages, `issued` so far, the next one to go to
// `stage` at `phase`; `full` is the barrier of stage 0.
__device__ __forceinline__ void DrainRing(uint32_t full, int stages, int stage, uint32_t phase, int issued) {
#pragma unroll 1
  for (int left = min(issued, stages); left > 0; --left) {
    if (stage == 0) {
      stage = stages;
      phase ^= 1u;
    }
    --stage;
    Drain(full + 8u * stage, phase);
  }
}

// One thread of a converged warp, for the instructions of the asynchronous units alone: the
// loops around them stay the whole warp's (see the head of this file).
__device__ __forceinline__ bool ElectOne() {
  uint32_t elected;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
  return elected != 0;
}

// A box of 128 rows at byte column x, row y of a matrix (x is a multiple of 16).
__device__ __forceinline__ void TileCopy(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// Shared-memory matrix descriptor of a K-major tile with 128-byte rows and the
// 128-byte swizzle: start address and offsets in 16-byte units, 1024 bytes
// between 8-row groups, descriptor version 1.
__device__ __forceinline__ uint64_t TileDescriptor(uint32_t shared_address) {
  uint64_t desc = 0;
  desc |= static_cast<uint64_t>((shared_address & 0x3FFFFu) >> 4);
  desc |= static_cast<uint64_t>(1) << 16;           // leading byte offset (unused with swizzle)
  desc |= static_cast<uint64_t>(1024 >> 4) << 32;   // stride byte offset
  desc |= static_cast<uint64_t>(1) << 46;           // version
  desc |= static_cast<uint64_t>(2) << 61;           // 128-byte swizzle
  return desc;
}

// D (tensor memory) += A (tensor memory) * B (shared memory).
__device__ __forceinline__ void MmaF16(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void MmaCommit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void TmemStore16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void TmemLoad16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = __uint_as_float(r[i]);
  }
}

// Within every four consecutive values of K the tiles hold them in the order
// (0, 2, 1, 3): a word yields the codes of its bytes 0 and 2 together (and 1 and
// 3), so this order lets a pair leave the arithmetic as it arrives. The
// activation tiles (StageHalfKernel) follow the same order; a contraction does
// not care how K is numbered.
//
// Four codes under the bits of kMask in the bytes of w, in packed fp16
// arithmetic: a code is masked in place under an fp16 exponent whose mantissa bit
// there is worth 1 (1024 + code for bits 0-5, 64 + code for bits 4-7: one logic
// instruction for two codes), and subtracting that power of two plus the centre
// leaves code - centre exactly.
__device__ __forceinline__ __half2 Centred(uint32_t w, uint32_t mask, uint32_t one, uint32_t bias) {
  const uint32_t biased = (w & mask) | one;
  return __hsub2(*reinterpret_cast<const __half2*>(&biased), *reinterpret_cast<const __half2*>(&bias));
}
__device__ __forceinline__ uint32_t HalfBits(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// Q4_K: scale * (code - 8) + (8 * scale - offset) of 32 nibbles (HIGH: the high
// ones) of eight words. Centring the code keeps both terms of the size of w
// itself, so rounding the scale and the constant to fp16 costs about what
// rounding w does; scale * code - offset loses three more bits to cancellation
// (measured relative L2 of a product: 7e-4 that way, 3.8e-4 centred, 2e-4 with
// fp32 arithmetic rounded once).
template <bool HIGH>
__device__ __forceinline__ void Nibbles(const uint32_t (&w)[8], __half2 scale, __half2 constant, uint32_t (&out)[16]) {
  constexpr uint32_t kMask = HIGH ? 0x00F000F0u : 0x000F000Fu;
  constexpr uint32_t kOne = HIGH ? 0x54005400u : 0x64006400u;    // 64 or 1024 as fp16 pairs
  constexpr uint32_t kBias = HIGH ? 0x54805480u : 0x64086408u;   // 72 or 1032
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    out[2 * c] = HalfBits(__hfma2(Centred(w[c], kMask, kOne, kBias), scale, constant));
    out[2 * c + 1] = HalfBits(__hfma2(Centred(w[c] >> 8, kMask, kOne, kBias), scale, constant));
  }
}

// Q6_K: scale * (code - 32) of the 32 values whose low nibbles are bits 0-3 of
// the bytes of lo and whose high bits are bits 4-5 of the bytes of hi (bits 6-7
// zero); the first sixteen take scale a, the others b. The code byte is complete
// and clean, so one byte permute puts two of them under the exponent of 1024.
__device__ __forceinline__ void SixBits(const uint32_t (&lo)[8], const uint32_t (&hi)[8], __half2 a, __half2 b,
                                        uint32_t (&out)[16]) {
  constexpr uint32_t kBias = 0x64206420u;   // 1024 + 32
  const __half2 bias = *reinterpret_cast<const __half2*>(&kBias);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t code = (lo[c] & 0x0F0F0F0Fu) | (hi[c] & ~0x0F0F0F0Fu);
    const uint32_t even = __byte_perm(code, 0x64646464u, 0x4240u), odd = __byte_perm(code, 0x64646464u, 0x4341u);
    const __half2 scale = c < 4 ? a : b;
    out[2 * c] = HalfBits(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&even), bias), scale));
    out[2 * c + 1] = HalfBits(__hmul2(__hsub2(*reinterpret_cast<const __half2*>(&odd), bias), scale));
  }
}

// The raw bytes that one dequant thread needs of a block of its row, the 64
// values of pair p, and their fp16 weights. p stays a run-time value: sixteen
// warps in one piece of code (a copy of the loop per group ran 15 % slower, out of
// the instruction cache).
template <int TYPE>
struct Pair;

template <>
struct Pair<GUFO_CUDA_Q4_K> {
  uint4 head, q0, q1;
  // A word that takes all of them.
  __device__ __forceinline__ uint32_t Any() const {
    return (head.x ^ head.y ^ head.z) ^ (head.w ^ q0.x ^ q0.y) ^ (q0.z ^ q0.w ^ q1.x) ^ (q1.y ^ q1.z ^ q1.w);
  }
  __device__ __forceinline__ void Load(const uint8_t* raw, int row, int p, int b) {
    (void)b;
    const uint8_t* block = raw + row * kQ4KBytes;
    head = *reinterpret_cast<const uint4*>(block);
    q0 = *reinterpret_cast<const uint4*>(block + 16 + 32 * p);
    q1 = *reinterpret_cast<const uint4*>(block + 32 + 32 * p);
  }
  __device__ __forceinline__ void Weights(int p, uint32_t (&lo)[16], uint32_t (&hi)[16]) const {
    const uint32_t words[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const float d = HalfBitsToFloat(static_cast<uint16_t>(head.x & 0xFFFF));
    const float dmin = HalfBitsToFloat(static_cast<uint16_t>(head.x >> 16));
    // Scales and mins of sub-blocks 2p and 2p + 1 (ScaleMinK4) in bytes 0 and 1.
    uint32_t sc = head.y & 0x3F3F3F3Fu, mn = head.z & 0x3F3F3F3Fu;
    if (p >= 2) {
      sc = (head.w & 0x0F0F0F0Fu) | ((head.y >> 2) & 0x30303030u);
      mn = ((head.w >> 4) & 0x0F0F0F0Fu) | ((head.z >> 2) & 0x30303030u);
    }
    sc >>= 16 * (p & 1);
    mn >>= 16 * (p & 1);
    auto prepare = [&](uint32_t scale_byte, uint32_t min_byte, __half2& scale2, __half2& constant2) {
      const float scale = d * static_cast<float>(scale_byte);
      scale2 = __float2half2_rn(scale);
      constant2 = __float2half2_rn(fmaf(8.0f, scale, -dmin * static_cast<float>(min_byte)));
    };
    __half2 s, c;
    prepare(sc & 0xFFu, mn & 0xFFu, s, c);
    Nibbles<false>(words, s, c, lo);
    prepare((sc >> 8) & 0xFFu, (mn >> 8) & 0xFFu, s, c);
    Nibbles<true>(words, s, c, hi);
  }
};

// Pair p: runs k = j and k = j + 2 (j = p & 1) of half h = p / 2, which share their
// 32 ql bytes: values 128 h + 32 k .. + 31, low nibbles for the first run and high
// ones for the second, two bits of the half's qh bytes at 2 k.
template <>
struct Pair<GUFO_CUDA_Q6_K> {
  using Q = Quant<GUFO_CUDA_Q6_K>;
  uint4 l0, l1, h0, h1;
  uint2 sc8;
  uint32_t d;
  __device__ __forceinline__ uint32_t Any() const {
    return (l0.x ^ l0.y ^ l0.z) ^ (l0.w ^ l1.x ^ l1.y) ^ (l1.z ^ l1.w ^ h0.x) ^ (h0.y ^ h0.z ^ h0.w) ^
           (h1.x ^ h1.y ^ h1.z) ^ (h1.w ^ sc8.x ^ sc8.y) ^ d;
  }
  __device__ __forceinline__ void Load(const uint8_t* raw, int row, int p, int b) {
    const int h = p >> 1;
    const uint8_t* ql = raw + Q::kQl + row * 128;
    const uint8_t* qh = raw + Q::kQh + row * 64;
    const int c0 = 4 * h + 2 * (p & 1);
    const int swz = row & 7, swz_h = (row >> 1) & 3;   // of the boxes' 128- and 64-byte swizzles
    l0 = *reinterpret_cast<const uint4*>(ql + ((c0 ^ swz) << 4));
    l1 = *reinterpret_cast<const uint4*>(ql + (((c0 + 1) ^ swz) << 4));
    h0 = *reinterpret_cast<const uint4*>(qh + (((2 * h) ^ swz_h) << 4));
    h1 = *reinterpret_cast<const uint4*>(qh + (((2 * h + 1) ^ swz_h) << 4));
    sc8 = *reinterpret_cast<const uint2*>(raw + Q::kSc + row * 16 + 8 * h);
    d = *reinterpret_cast<const uint16_t*>(raw + Q::kD + row * 16 + 2 * (b & (kQ6KSlabBlocks - 1)));
  }
  __device__ __forceinline__ void Weights(int p, uint32_t (&lo)[16], uint32_t (&hi)[16]) const {
    const float scale = HalfBitsToFloat(static_cast<uint16_t>(d));
    const int j = p & 1;
    // int8 scales of 16-value groups 2j, 2j + 1 (first run) and 2j + 4, 2j + 5 of this half.
    const uint32_t first = sc8.x >> (16 * j), second = sc8.y >> (16 * j);
    auto of = [&](uint32_t byte) { return __float2half2_rn(scale * static_cast<float>(static_cast<int8_t>(byte))); };
    const uint32_t low[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
    const uint32_t high[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    uint32_t nib[8], up[8], bits[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      bits[c] = (high[c] >> (2 * j)) & 0x33333333u;   // both runs' bits, at 0-1 and 4-5
      up[c] = bits[c] << 4;
      nib[c] = low[c] >> 4;
    }
    SixBits(low, up, of(first), of(first >> 8), lo);
    SixBits(nib, bits, of(second), of(second >> 8), hi);
  }
};

// First step of thread block c's range: the first `extra` ranges are a step longer, or a
// cluster's blocks take a unit's steps in even shares.
__device__ __forceinline__ int RangeStart(const TcGemmArgs& a, int c) {
  if (a.cluster > 1) {
    const int u = c / a.cluster;
    return u * a.blocks + (c - u * a.cluster) * a.blocks / a.cluster;
  }
  return c * a.per + min(c, a.extra);
}

// Where a unit works: its part, first weight row and token group.
struct Unit {
  int part;
  int row0;
  int group;
};

__device__ __forceinline__ Unit LocateUnit(const TcGemmArgs& a, int u) {
  Unit unit;
  int tile = u / a.groups;   // groups of one tile follow one another: its weights are in L2 by then
  unit.group = u - tile * a.groups;
  unit.part = 0;
#pragma unroll
  for (int p = 0; p < kTcMaxParts - 1; ++p) {
    if (unit.part == p && p + 1 < a.nparts && tile >= a.parts[p].tiles) {
      tile -= a.parts[p].tiles;
      unit.part = p + 1;
    }
  }
  unit.row0 = tile * kTileRows;
  return unit;
}

// Brings the raw blocks of the steps [step, until) into the ring, up to the first wait that
// runs out; the calling warp's lanes agree on everything, one of them issues the copies.
template <int TYPE>
struct RawLoader {
  const TcGemmArgs& a;
  uint32_t full, empty;   // barriers of stage 0
  uint32_t to;            // stage 0
  volatile int* abort_flag;
  int step, last;
  int stage = 0;
  uint32_t phase = 0;

  __device__ __forceinline__ void Run(int until) {
    using Q = Quant<TYPE>;
    while (step < until) {
      const int u = step / a.blocks;
      const Unit unit = LocateUnit(a, u);
      const CUtensorMap* map = &a.maps[unit.part * 3];
      const int row = unit.row0;
      const int end = min((u + 1) * a.blocks, until);
      for (int b = step - u * a.blocks; step < end; ++b, ++step) {
        if (!__all_sync(0xFFFFFFFFu, BoundedWait<true>(empty + 8u * stage, phase ^ 1u, abort_flag, a.error, 1))) {
          return;
        }
        const uint32_t at_shared = to + stage * Q::kRawStride;
        const uint32_t bar = full + 8u * stage;
        if (ElectOne()) {
          MbarArriveExpectTx(bar, Q::kRawBytes);
          // Rows past the end of the part arrive as zeros.
          if constexpr (TYPE == GUFO_CUDA_Q4_K) {
            TileCopy(at_shared, map, b * kQ4KBytes, row, bar);
          } else {
            // The planar device arrangement (Q6KBlockAt): a slab of n blocks stores
            // ql n x 128 | qh n x 64 | scales n x 16 | d n x 2.
            const int slab = b / kQ6KSlabBlocks;
            const int j = b - slab * kQ6KSlabBlocks;
            const int n = min(a.blocks - slab * kQ6KSlabBlocks, kQ6KSlabBlocks);
            const int at = slab * kQ6KSlabBlocks * kQ6KBytes;
            TileCopy(at_shared + Q::kQl, map, at + 128 * j, row, bar);
            TileCopy(at_shared + Q::kQh, map + 1, at + 128 * n + 64 * j, row, bar);
            TileCopy(at_shared + Q::kSc, map + 2, at + 192 * n + 16 * j, row, bar);
            TileCopy(at_shared + Q::kD, map + 2, at + 208 * n, row, bar);   // the slab's d values
          }
        }
        __syncwarp();
        if (++stage == a.raw_stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
};

// The thread blocks that share a cut tile (the unit of `blocks` steps from step
// `begin` on), from one of them.
struct CutTile {
  int from, to;
};
__device__ __forceinline__ CutTile LocateCut(const TcGemmArgs& a, int self, int begin) {
  CutTile cut{self, self};
  while (RangeStart(a, cut.from) > begin) {
    --cut.from;
  }
  while (RangeStart(a, cut.to + 1) < begin + a.blocks) {
    ++cut.to;
  }
  return cut;
}
// Which of block c's partial slots holds its share: only the first of the tile's
// blocks can have begun elsewhere.
__device__ __forceinline__ int CutSlot(const TcGemmArgs& a, const CutTile& cut, int c, int begin) {
  return c == cut.from && RangeStart(a, c) < begin ? 1 : 0;
}

// A thread block's share of a cut tile in scratch: chunks of sixteen columns, in which a
// row's four quads of columns lie 128 rows apart, so that a warp writes and reads 512
// adjacent bytes an instruction.
constexpr int kChunk = 16;
__device__ __forceinline__ float4* PartialChunk(const TcGemmArgs& a, int block, int slot, int chunk, int row) {
  return reinterpret_cast<float4*>(a.partial + ((static_cast<size_t>(block) * 2 + slot) * a.n + chunk * kChunk) * kTileRows) +
         row;
}

__device__ __forceinline__ void LeaveChunk(float4* to, const float (&v)[kChunk]) {
#pragma unroll
  for (int q = 0; q < kChunk / 4; ++q) {
    __stcg(to + q * kTileRows, make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]));
  }
}

// The outputs of a row in sixteen columns from `col0` of the unit on; `to` is the unit's
// first token row (the same for all lanes, which keeps the addresses in uniform registers).
__device__ __forceinline__ void StoreChunk(const TcGemmArgs& a, float* to, uint32_t row, int col0, int columns,
                                           const float* factor, const float (&v)[kChunk]) {
  to += static_cast<size_t>(col0) * a.out_stride;
  if (col0 + kChunk <= columns) {
#pragma unroll
    for (int q = 0; q < kChunk / 4; ++q) {
      const float4 f = *reinterpret_cast<const float4*>(&factor[col0 + 4 * q]);
      to[row] = v[4 * q] * f.x;
      to += a.out_stride;
      to[row] = v[4 * q + 1] * f.y;
      to += a.out_stride;
      to[row] = v[4 * q + 2] * f.z;
      to += a.out_stride;
      to[row] = v[4 * q + 3] * f.w;
      to += a.out_stride;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      if (col0 + j < columns) {
        to[static_cast<size_t>(j) * a.out_stride + row] = v[j] * factor[col0 + j];
      }
    }
  }
}

// Four outputs of a row, of four tokens from `to` on (the same for all lanes, which keeps
// the addresses in uniform registers).
__device__ __forceinline__ void StoreQuad(const TcGemmArgs& a, float* to, uint32_t row, int col, int columns,
                                          const float* factor, const float4& v) {
  if (col + 4 <= columns) {
    const float4 f = *reinterpret_cast<const float4*>(&factor[col]);
    to[row] = v.x * f.x;
    to += a.out_stride;
    to[row] = v.y * f.y;
    to += a.out_stride;
    to[row] = v.z * f.z;
    to += a.out_stride;
    to[row] = v.w * f.w;
  } else {
    const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (col + j < columns) {
        to[static_cast<size_t>(j) * a.out_stride + row] = w[j] * factor[col + j];
      }
    }
  }
}

// Adds up a cut tile whose shares are all at hand and stores its rows: by the first
// twenty warps, four (of 32 rows each) a chunk. The shares are added in block order, two
// on their way at a time; block `self`'s is read from tensor memory at `tmem` (self < 0:
// every share is in scratch). `factor` holds the unit's factors.
__device__ __noinline__ void AddShares(const TcGemmArgs& a, int u, int from, int to, int self, uint32_t tmem,
                                       const float* factor) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int begin = u * a.blocks;
  const CutTile cut{from, to};
  const Unit unit = LocateUnit(a, u);
  const TcPart& part = a.parts[unit.part];
  const int token0 = unit.group * a.n;
  const int columns = min(a.n, a.tokens - token0);
  const int local = (warp & 3) * 32 + lane;
  const bool live = unit.row0 + local < part.rows;
  float* out = part.out + static_cast<size_t>(token0) * a.out_stride;
#pragma unroll 1
  for (int chunk = warp >> 2; chunk * kChunk < columns; chunk += kGroups + 1) {
    auto share = [&](int c, float (&v)[kChunk]) {
      if (c == self) {
        TmemLoad16(tmem + chunk * kChunk, v);
        return;
      }
      const float4* at = PartialChunk(a, c, CutSlot(a, cut, c, begin), chunk, local);
#pragma unroll
      for (int q = 0; q < kChunk / 4; ++q) {
        const float4 w = __ldcg(at + q * kTileRows);
        v[4 * q] = w.x, v[4 * q + 1] = w.y, v[4 * q + 2] = w.z, v[4 * q + 3] = w.w;
      }
    };
    float sum[kChunk];
    share(from, sum);
    int c = from + 1;
#pragma unroll 1
    for (; c + 1 <= to; c += 2) {
      float v[kChunk], w[kChunk];
      share(c, v);
      share(c + 1, w);
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        sum[j] = (sum[j] + v[j]) + w[j];
      }
    }
    if (c <= to) {
      float v[kChunk];
      share(c, v);
#pragma unroll
      for (int j = 0; j < kChunk; ++j) {
        sum[j] += v[j];
      }
    }
    if (live) {
      StoreChunk(a, out, static_cast<uint32_t>(unit.row0 + local), chunk * kChunk, columns, factor, sum);
    }
  }
  if (threadIdx.x == 0) {
    a.counters[from] = 0;   // for the next launch
  }
}

__device__ __forceinline__ void ClusterBarrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The end of a unit that a cluster has shared, by all threads: every block's accumulator
// goes to the blocks that own its columns (four columns, a quad, in turn to each), through
// distributed shared memory into what was the pipeline's, and each owner adds the shares
// of its columns in rank order and stores them. All blocks are at it together, where one
// block used to read the others' shares from scratch at the end: 2560 x 9728 Q6_K in seven
// shares, 32 / 128 tokens 7 / 14 us of its 18 / 31.
__device__ __forceinline__ void ReduceCluster(const TcGemmArgs& a, uint32_t tmem_acc, uint32_t buffer, const uint8_t* local_buffer,
                                              const float* factor, const volatile int* abort_flag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(blockIdx.x) % a.cluster;
  const Unit unit = LocateUnit(a, static_cast<int>(blockIdx.x) / a.cluster);
  const TcPart& part = a.parts[unit.part];
  const int token0 = unit.group * a.n;
  const int columns = min(a.n, a.tokens - token0);
  const int quads = (columns + 3) / 4;
  const int each = (a.n / 4 + a.cluster - 1) / a.cluster;   // quads of an owner, at most
  ClusterBarrier();   // nobody's pipeline needs its shared memory any more
  if (warp < kDequantWarps + 4) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int row = (warp & 3) * 32 + lane;
    for (int col0 = 16 * (warp >> 2); col0 < columns; col0 += 16 * (kGroups + 1)) {
      float v[16];
      TmemLoad16(tmem_acc + (static_cast<uint32_t>((warp & 3) * 32) << 16) + col0, v);
      int owner = col0 / 4 % a.cluster, slot = col0 / 4 / a.cluster;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t to;
        asm("mapa.shared::cluster.u32 %0, %1, %2;"
            : "=r"(to) : "r"(buffer + static_cast<uint32_t>(((rank * each + slot) * kTileRows + row) * 16)), "r"(owner));
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};"
                     ::"r"(to), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3]) : "memory");
        if (++owner == a.cluster) {
          owner = 0;
          ++slot;
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  ClusterBarrier();
  if (warp < kDequantWarps + 4 && *abort_flag == 0) {
    const int row = static_cast<int>(threadIdx.x & 127);
    if (unit.row0 + row < part.rows) {
      float* out = part.out + static_cast<size_t>(token0) * a.out_stride;
      for (int slot = threadIdx.x >> 7; slot * a.cluster + rank < quads; slot += kGroups + 1) {
        const float4* from = reinterpret_cast<const float4*>(local_buffer) + slot * kTileRows + row;
        float4 sum = *from;
        for (int r = 1; r < a.cluster; ++r) {
          const float4 v = from[r * each * kTileRows];
          sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        const int col = 4 * (slot * a.cluster + rank);
        StoreQuad(a, out + static_cast<size_t>(col) * a.out_stride, static_cast<uint32_t>(unit.row0 + row), col, columns,
                  factor, sum);
      }
    }
  }
}

// What a dequant warp of group p works with.
struct DequantPlace {
  uint32_t raw_full, raw_empty;   // stage 0; eight bytes apart
  uint32_t w_full, w_empty;       // the group's slot
  const uint8_t* raw;             // stage 0
  uint32_t slot;                  // the warp's lanes of the slot
  int row;                        // this thread's row of the tile
  int p;
};

// The steps [first, last) of one dequant warp.
template <int TYPE>
__device__ __forceinline__ void DequantSteps(const TcGemmArgs& a, const DequantPlace& at, int first, int last,
                                             volatile int* abort_flag) {
  const bool leader = (threadIdx.x & 31) == 0;
  int stage = 0;
  uint32_t phase = 0, w_phase = 1;
  int b = first % a.blocks;
  const uint8_t* raw = at.raw;
  for (int step = first; step < last; ++step) {
    BoundedWait(at.raw_full + 8 * stage, phase, abort_flag, a.error, 4);
    Pair<TYPE> pair;
    pair.Load(raw, at.row, at.p, b);
    // The stage may be overwritten once every lane has its bytes, whatever they are.
    const bool loaded = LoadsDone(pair.Any());
    if (leader && loaded) {
      MbarArrive(at.raw_empty + 8 * stage);
    }
    uint32_t lo[16], hi[16];
    pair.Weights(at.p, lo, hi);
    // The tensor core has read the slot's weights of the block before.
    BoundedWait(at.w_empty, w_phase, abort_flag, a.error, 5);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    TmemStore16(at.slot, lo);
    TmemStore16(at.slot + 16, hi);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if (leader) {
      MbarArrive(at.w_full);
    }
    w_phase ^= 1u;
    raw += Quant<TYPE>::kRawStride;
    if (++stage == a.raw_stages) {
      stage = 0;
      phase ^= 1u;
      raw = at.raw;
    }
    if (++b == a.blocks) {
      b = 0;
    }
  }
}

// (The bound is that of 72 registers a thread, which leave room for a block of
// StageHalfKernel on the SM; kTcThreads threads are launched.)
template <int TYPE>
__global__ void __launch_bounds__(896, 1)
GemmTc(const __grid_constant__ TcGemmArgs a) {
  using Q = Quant<TYPE>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bar_mem[4 * kMaxStages + 2 * kGroups + 5];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(16) float factor[kMaxN];    // what undoes the scales of the unit's token rows
  __shared__ int finish;   // a cut tile whose shares are all in scratch and that is left to this block (unit + 1)
  __shared__ int others_done;
  // The swizzled tiles need a 1024-byte aligned base: activation tiles, then raw blocks.
  const uint32_t base = (SharedAddress(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - SharedAddress(smem_raw));
  const int x_bytes = 2 * a.n * kTileK * 2;   // a stage of two activation tiles
  const uint32_t raw_at = static_cast<uint32_t>(a.x_stages * x_bytes);
  const uint32_t bars = SharedAddress(bar_mem);
  auto raw_full = [&](int s) { return bars + 8u * s; };
  auto raw_empty = [&](int s) { return bars + 8u * (kMaxStages + s); };
  auto x_full = [&](int s) { return bars + 8u * (2 * kMaxStages + s); };
  auto x_empty = [&](int s) { return bars + 8u * (3 * kMaxStages + s); };
  auto w_full = [&](int g) { return bars + 8u * (4 * kMaxStages + g); };
  auto w_empty = [&](int g) { return bars + 8u * (4 * kMaxStages + kGroups + g); };
  auto acc_full = [&](int s) { return bars + 8u * (4 * kMaxStages + 2 * kGroups + s); };
  auto acc_empty = [&](int s) { return bars + 8u * (4 * kMaxStages + 2 * kGroups + 2 + s); };
  const uint32_t mma_done = bars + 8u * (4 * kMaxStages + 2 * kGroups + 4);   // after a wait that ran out
  volatile int* abort_flag = &abort_word;

  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  const int first = RangeStart(a, blockIdx.x);
  const int last = RangeStart(a, blockIdx.x + 1);

  // The first raw blocks are asked for before anything else: the weights never depend on
  // earlier kernels, and they are the longest way off.
  RawLoader<TYPE> raw_loader{a, raw_full(0), raw_empty(0), base + raw_at, abort_flag, first, last};
  if (warp == kRawWarp) {
    if (ElectOne()) {
      for (int s = 0; s < a.raw_stages; ++s) {
        MbarInit(raw_full(s), 1);
        MbarInit(raw_empty(s), kDequantWarps);
      }
      abort_word = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    raw_loader.Run(min(first + 2, last));   // (more would hold up the others: an issue takes 100 cycles and more)
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < a.x_stages; ++s) {
      MbarInit(x_full(s), 1);
      MbarInit(x_empty(s), 1);
    }
    for (int g = 0; g < kGroups; ++g) {
      MbarInit(w_full(g), 4);
      MbarInit(w_empty(g), 1);
    }
    for (int s = 0; s < 2; ++s) {
      MbarInit(acc_full(s), 1);
      MbarInit(acc_empty(s), 4);
    }
    MbarInit(mma_done, 1);
    finish = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(SharedAddress(&tmem_slot)), "r"(kTmemColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, *reinterpret_cast<volatile uint32_t*>(&tmem_slot), 0);
  // The weights never depend on earlier kernels; the activation tiles and the
  // outputs do.
  GridLaunchDependents();

  // Every role walks the steps [first, last); the stage counters run on across
  // units, so the pipeline never drains between them.
  if (warp == kRawWarp) {
    raw_loader.Run(last);
    if (__any_sync(0xFFFFFFFFu, *abort_flag != 0)) {
      DrainRing(raw_full(0), a.raw_stages, raw_loader.stage, raw_loader.phase, raw_loader.step - first);
    }
  } else if (warp == kXWarp) {
    // ---- activation tiles, two (half a step's) per stage ------------------------
    GridDependencyWait();
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    for (int step = first; step < last;) {
      const int u = step / a.blocks;
      const int group = u % a.groups;
      const int end = min((u + 1) * a.blocks, last);
      const uint8_t* from = a.xh + (static_cast<size_t>(group) * a.blocks + (step - u * a.blocks)) * 2 * x_bytes;
      int half = 2 * (end - step);
      for (step = end; half > 0; --half) {
        if (!__all_sync(0xFFFFFFFFu, BoundedWait<true>(x_empty(stage), phase ^ 1u, abort_flag, a.error, 2))) {
          step = last;
          break;
        }
        if (ElectOne()) {
          MbarArriveExpectTx(x_full(stage), x_bytes);
          BulkCopy(base + stage * x_bytes, from, x_bytes, x_full(stage));
        }
        __syncwarp();
        from += x_bytes;
        ++issued;
        if (++stage == a.x_stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    if (__any_sync(0xFFFFFFFFu, *abort_flag != 0)) {
      DrainRing(x_full(0), a.x_stages, stage, phase, issued);
    }
  } else if (warp == kMmaWarp) {
    // ---- MMA issue ---------------------------------------------------------
    // kind::f16, fp32 accumulate, fp16 A and B, both K-major, M = 128.
    {
      const uint32_t idesc = (1u << 4) | (static_cast<uint32_t>(a.n >> 3) << 17) |
                             (static_cast<uint32_t>(kTileRows >> 4) << 24);
      int xs = 0;              // stage of the step's first two activation tiles
      uint32_t x_phase = 0;
      uint32_t w_phase = 0;    // slots are filled once per block: they flip together
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int step = first; step < last;) {
        const int end = min((step / a.blocks + 1) * a.blocks, last);
        // The epilogue has read what this accumulator held before.
        BoundedWait(acc_empty(acc), acc_phase ^ 1u, abort_flag, a.error, 8);
        const uint32_t accumulator = tmem + kAccColumn + static_cast<uint32_t>(acc * a.n);
        for (uint32_t more = 0; step < end; ++step, more = 1) {
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            BoundedWait(x_full(xs), x_phase, abort_flag, a.error, 7);
            const uint64_t desc_x = TileDescriptor(base + xs * x_bytes);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int g = 2 * half + t;
              BoundedWait(w_full(g), w_phase, abort_flag, a.error, 3);
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint32_t slot = tmem + static_cast<uint32_t>(g * kSlotColumns);
              const uint64_t desc = desc_x + static_cast<uint64_t>(t * (x_bytes >> 5));   // 16-byte units
              if (ElectOne()) {
#pragma unroll
                for (int k = 0; k < kTileK / 16; ++k) {
                  // 16 values: eight columns of the slot, 32 bytes of the swizzled rows.
                  MmaF16(accumulator, slot + 8u * k, desc + 2u * k, idesc, k > 0 || g > 0 ? 1u : more);
                }
                // A commit arrives once everything issued so far has retired.
                MmaCommit(w_empty(g));
                if (t == 1) {
                  MmaCommit(x_empty(xs));
                }
              }
              __syncwarp();
            }
            if (++xs == a.x_stages) {
              xs = 0;
              x_phase ^= 1u;
            }
          }
          w_phase ^= 1u;
        }
        if (ElectOne()) {
          MmaCommit(acc_full(acc));
        }
        __syncwarp();
        acc ^= 1;
        acc_phase ^= acc == 0 ? 1u : 0u;
      }
      if (__any_sync(0xFFFFFFFFu, *abort_flag != 0)) {
        if (ElectOne()) {
          MmaCommit(mma_done);
        }
        __syncwarp();
        Drain(mma_done, 0);
      }
    }
  } else if (warp >= kEpilogueWarp && warp < kEpilogueWarp + 4) {
    // ---- epilogue: warp q reads lanes 32 q .. 32 q + 31, i.e. weight rows ------
    GridDependencyWait();
    const int quarter = warp - kEpilogueWarp;
    const int local = quarter * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int step = first; step < last;) {
      const int u = step / a.blocks;
      const Unit unit = LocateUnit(a, u);
      const TcPart& part = a.parts[unit.part];
      const int begin = u * a.blocks;
      const int end = min(begin + a.blocks, last);
      const bool whole = step == begin && end == begin + a.blocks;
      const int token0 = unit.group * a.n;
      const int columns = min(a.n, a.tokens - token0);
      asm volatile("bar.sync 1, 128;" ::: "memory");   // the factors of the unit before have been read
      for (int i = local; i < columns; i += 128) {
        factor[i] = __ldcg(a.unscale + token0 + i);
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      const bool ready = BoundedWait<true>(acc_full(acc), acc_phase, abort_flag, a.error, 6);
      if (!whole && end == last) {
        break;   // the share of a cut tile that ends the range: by all warps, below
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t from = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + kAccColumn +
                            static_cast<uint32_t>(acc * a.n);
      const uint32_t row = static_cast<uint32_t>(unit.row0 + local);
      const bool live = ready && unit.row0 + local < part.rows;
      float* to = part.out + static_cast<size_t>(token0) * a.out_stride;
      for (int col0 = 0; col0 < columns; col0 += kChunk) {
        float v[kChunk];
        TmemLoad16(from + col0, v);
        if (!whole) {
          LeaveChunk(PartialChunk(a, blockIdx.x, 0, col0 / kChunk, local), v);
        } else if (live) {
          StoreChunk(a, to, row, col0, columns, factor, v);
        }
      }
      // This accumulator may be overwritten now.
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        MbarArrive(acc_empty(acc));
      }
      acc ^= 1;
      acc_phase ^= acc == 0 ? 1u : 0u;
      if (!whole) {
        // The share of a cut tile that opens the range: left in scratch.
        __threadfence();
        asm volatile("bar.sync 1, 128;" ::: "memory");
        if (local == 0) {
          const CutTile cut = LocateCut(a, blockIdx.x, begin);
          if (atomicAdd(a.counters + cut.from, 1u) == static_cast<unsigned>(cut.to - cut.from)) {
            finish = u + 1;
          }
        }
      }
      step = end;
    }
  } else if (warp < kDequantWarps) {
    // ---- dequant: group p takes pair p of every block; a thread owns one row ------
    const DequantPlace at{raw_full(0), raw_empty(0), w_full(warp >> 2), w_empty(warp >> 2), smem + raw_at,
                          tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) +
                              static_cast<uint32_t>((warp >> 2) * kSlotColumns),
                          (warp & 3) * 32 + lane, warp >> 2};
    DequantSteps<TYPE>(a, at, first, last, abort_flag);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  // Cut tiles. Most are cut in two: the second share opens its block's range and
  // is long in scratch when the first, which ends its block's range, is complete in
  // tensor memory; all warps then add the one to the other.
  const int tail_unit = (last - 1) / a.blocks;
  const int tail_begin = tail_unit * a.blocks;
  const bool tail_opens = first >= tail_begin;   // the block's only share
  if (a.cluster > 1) {
    ReduceCluster(a, tmem + kAccColumn, base, smem, factor, abort_flag);
  } else if ((first > tail_begin || last < tail_begin + a.blocks) && warp < kDequantWarps + 4) {
    const CutTile cut = LocateCut(a, blockIdx.x, tail_begin);
    const unsigned others = static_cast<unsigned>(cut.to - cut.from);
    if (threadIdx.x == 0) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.counters + cut.from) : "memory");
      others_done = seen == others;
    }
    asm volatile("bar.sync 2, %0;" ::"n"((kDequantWarps + 4) * 32) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int acc = (tail_unit - first / a.blocks) & 1;
    const uint32_t from = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + kAccColumn +
                          static_cast<uint32_t>(acc * a.n);
    const int self = static_cast<int>(blockIdx.x);
    bool finishes = *const_cast<volatile int*>(&others_done) != 0;
    if (!finishes) {
      const int columns = min(a.n, a.tokens - (tail_unit - tail_unit / a.groups * a.groups) * a.n);
      for (int chunk = warp >> 2; chunk * kChunk < columns; chunk += kGroups + 1) {
        float v[kChunk];
        TmemLoad16(from + chunk * kChunk, v);
        LeaveChunk(PartialChunk(a, blockIdx.x, tail_opens ? 0 : 1, chunk, (warp & 3) * 32 + lane), v);
      }
      __threadfence();
      asm volatile("bar.sync 2, %0;" ::"n"((kDequantWarps + 4) * 32) : "memory");
      if (threadIdx.x == 0) {
        others_done = atomicAdd(a.counters + cut.from, 1u) == others ? 2 : 0;
      }
      asm volatile("bar.sync 2, %0;" ::"n"((kDequantWarps + 4) * 32) : "memory");
      finishes = *const_cast<volatile int*>(&others_done) == 2;
      __threadfence();
    }
    if (finishes && *abort_flag == 0) {
      AddShares(a, tail_unit, cut.from, cut.to, self, from, factor);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (finish != 0) {   // the share that opened this block's range came last
    const int u = finish - 1;
    const int token0 = (u - u / a.groups * a.groups) * a.n;
    if (threadIdx.x < min(a.n, a.tokens - token0)) {
      factor[threadIdx.x] = __ldcg(a.unscale + token0 + threadIdx.x);
    }
    __syncthreads();
    if (warp < kDequantWarps + 4) {
      const CutTile cut = LocateCut(a, blockIdx.x, u * a.blocks);
      __threadfence();
      AddShares(a, u, cut.from, cut.to, -1, 0u, factor);
    }
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns) : "memory");
  }
}

// gridDim.y blocks per token row: the row is scaled by a power of two so that its
// largest magnitude lands in [2^13, 2^14), rounded to fp16 and written into every tile
// image of its group at its swizzled place. Rows past `tokens` are zero. `six`: tile
// 2 h + j of a block holds Q6_K's runs j and j + 2 of half h (the pair a dequant group
// turns out together), else values 64 t .. 64 t + 63.
//
// Every block of a row looks for the largest magnitude itself and converts its part. The
// blocks are small enough to share an SM with a block of the GEMM (256 threads of at most
// 48 registers beside 736 of 72), whose weights are under way meanwhile; beside blocks of
// 1024 threads the GEMM's came 3 us late.
constexpr int kStageThreads = 256;
__global__ void __launch_bounds__(kStageThreads, 5)
StageHalfKernel(const float* __restrict__ x, int tokens, int cols, int group_rows, int six, uint8_t* __restrict__ xh,
                float* __restrict__ unscale) {
  __shared__ uint32_t warp_top[kStageThreads / 32];
  GridLaunchDependents();
  GridDependencyWait();
  const int token = blockIdx.x;
  const int group = token / group_rows;
  const int image_row = token - group * group_rows;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const float4* row = reinterpret_cast<const float4*>(x + static_cast<size_t>(token) * cols);
  // A thread's first chunks of eight values stay in registers between the two passes: a
  // round trip less (2560 x 4096, 32 / 79 / 512 tokens 8.6 / 10.6 / 18.6 -> 8.3 / 9.4 / 17.5 us;
  // 12288 x 2560 11.5 / 12.9 / 29.3 -> 10.8 / 12.0 / 28.8). Rows past the end are zeros.
  constexpr int kKeep = 2;
  const int chunks = cols / 8;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 keep[kKeep][2];
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    keep[i][0] = keep[i][1] = zero;
  }
  float up = 1.0f;
  if (token < tokens) {
    uint32_t top = 0;
    auto see = [&](const float4& v) {
      top = max(max(top, __float_as_uint(v.x) & 0x7FFFFFFFu), __float_as_uint(v.y) & 0x7FFFFFFFu);
      top = max(max(top, __float_as_uint(v.z) & 0x7FFFFFFFu), __float_as_uint(v.w) & 0x7FFFFFFFu);
    };
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      const int chunk = threadIdx.x + kStageThreads * i;
      if (chunk < chunks) {
        keep[i][0] = row[2 * chunk];
        keep[i][1] = row[2 * chunk + 1];
      }
    }
    if (chunks > kKeep * kStageThreads) {
#pragma unroll 4
      for (int i = threadIdx.x + 2 * kStageThreads * kKeep; i < cols / 4; i += kStageThreads) {
        see(row[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      if (i * kStageThreads < chunks) {
        see(keep[i][0]);
        see(keep[i][1]);
      }
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    if (lane == 0) {
      warp_top[warp] = top;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kStageThreads / 32; ++w) {
      top = max(top, warp_top[w]);
    }
    // Biased exponent e of the maximum: |x| < 2^(e - 126). Scale by 2^(140 - e)
    // (clamped to normal factors) so the maximum is below 2^14; inf and NaN
    // rows keep factor 1 and stay inf / NaN in fp16.
    int e = static_cast<int>(top >> 23);
    int shift = e == 255 ? 0 : 140 - e;
    shift = max(-126, min(126, shift));
    up = __uint_as_float(static_cast<uint32_t>(127 + shift) << 23);
    if (threadIdx.x == 0 && blockIdx.y == 0) {
      unscale[token] = __uint_as_float(static_cast<uint32_t>(127 - shift) << 23);
    }
  } else if (threadIdx.x == 0 && blockIdx.y == 0) {
    unscale[token] = 0.f;
  }
  const size_t tile_bytes = static_cast<size_t>(group_rows) * (kTileK * 2);
  uint8_t* image = xh + static_cast<size_t>(group) * (cols / kTileK) * tile_bytes + static_cast<size_t>(image_row) * 128;
  auto put = [&](int chunk, const float4& v0, const float4& v1) {
    // Values (0, 2, 1, 3) of every four: the order of K the weights use.
    const __half2 h0 = __floats2half2_rn(v0.x * up, v0.z * up), h1 = __floats2half2_rn(v0.y * up, v0.w * up);
    const __half2 h2 = __floats2half2_rn(v1.x * up, v1.z * up), h3 = __floats2half2_rn(v1.y * up, v1.w * up);
    const uint4 packed = make_uint4(HalfBits(h0), HalfBits(h1), HalfBits(h2), HalfBits(h3));
    int tile = chunk >> 3;   // of eight chunks
    int c = chunk & 7;
    if (six != 0) {
      const int in_block = chunk & 31;               // 32 chunks a block
      const int h = in_block >> 4, k = (in_block >> 2) & 3;
      tile = (chunk >> 5) * 4 + 2 * h + (k & 1);
      c = 4 * (k >> 1) + (in_block & 3);
    }
    *reinterpret_cast<uint4*>(image + tile * tile_bytes + ((c ^ (image_row & 7)) << 4)) = packed;
  };
  // The row's blocks take every gridDim.y-th run of kStageThreads chunks.
  const int each = static_cast<int>(gridDim.y);
  int run = static_cast<int>(blockIdx.y);
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    const int chunk = threadIdx.x + kStageThreads * i;
    if (run == i) {
      if (chunk < chunks) {
        put(chunk, keep[i][0], keep[i][1]);
      }
      run += each;
    }
  }
  if (chunks <= kKeep * kStageThreads) {
    return;
  }
#pragma unroll 4
  for (int chunk = run * kStageThreads + threadIdx.x; chunk < chunks; chunk += each * kStageThreads) {
    put(chunk, token < tokens ? row[2 * chunk] : zero, token < tokens ? row[2 * chunk + 1] : zero);
  }
}

int ReserveTc(gufo_cuda_ctx* ctx, size_t bytes) {
  if (ctx->tc_scratch_bytes >= bytes) {
    return GUFO_CUDA_OK;
  }
  // An outgrown block is kept (a captured graph may hold it); its error word
  // is not carried over: a failure is read from the current block. In few steps, so
  // that little is outgrown: one allocation serves most shapes of a model.
  constexpr size_t kSteps[] = {1u << 20, 8u << 20, 48u << 20};
  size_t floor = (bytes + kSteps[2] - 1) / kSteps[2] * kSteps[2];
  for (size_t step : kSteps) {
    if (bytes <= step) {
      floor = step;
      break;
    }
  }
  const int rc = ctx->GrowScratch(&ctx->tc_scratch, &ctx->tc_scratch_bytes, bytes, floor, "tcgen05 gemm");
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  GUFO_CUDA_TRY(cudaMemsetAsync(ctx->tc_scratch, 0, kHeaderBytes, ctx->stream));
  return GUFO_CUDA_OK;
}

// cuTensorMapEncodeTiled, a host function of the driver (looked up once).
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled TensorMapEncoder() {
  static const EncodeTiled encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) !=
            cudaSuccess || found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<EncodeTiled>(fn);
  }();
  return encode;
}

// A map of `rows` rows of `row_bytes` bytes whose boxes are 128 rows of `width` bytes.
int EncodeRows(CUtensorMap* map, const uint8_t* data, int rows, int row_bytes, int width, CUtensorMapSwizzle swizzle) {
  const EncodeTiled encode = TensorMapEncoder();
  if (encode == nullptr) {
    return Fail(GUFO_CUDA_RUNTIME, "tcgen05 gemm: the driver has no cuTensorMapEncodeTiled");
  }
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(width), kTileRows};
  const cuuint32_t ones[2] = {1, 1};
  const CUresult e = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(data), dims, strides, box, ones,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return e == CUDA_SUCCESS ? GUFO_CUDA_OK
                           : Fail(GUFO_CUDA_RUNTIME, "tcgen05 gemm: tensor map of " + std::to_string(rows) + " x " +
                                                         std::to_string(row_bytes) + " bytes: error " +
                                                         std::to_string(static_cast<int>(e)));
}

constexpr int kMaxCluster = 8;   // what every device takes

// How a product of `tokens` rows is cut: token groups of n columns, thread blocks.
struct Plan {
  int groups, n, grid, units, cluster;
};

// Cycles of a step (256 values of 128 rows), as measured: what the dequantization and its
// hand-overs take, and the tensor core's and the activation tiles' part, which grows with n.
double StepCycles(int type, int n) { return (type == GUFO_CUDA_Q4_K ? 1070 : 1300) + 8.7 * n; }

Plan PlanTc(const GemvArgs& base, const std::vector<int>& parts, int type, int tokens, int sm_count, const int* clusters) {
  const int blocks = base.cols / kSuperBlock;
  int tiles = 0;
  for (int p : parts) {
    tiles += (base.parts[p].rows + kTileRows - 1) / kTileRows;
  }
  Plan best{};
  double best_cost = 1e30;
  const int least = (tokens + kMaxN - 1) / kMaxN;
  for (int groups = least; groups <= least + 3; ++groups) {
    const int n = ((tokens + groups - 1) / groups + 15) / 16 * 16;
    if ((groups - 1) * n >= tokens) {
      continue;   // a group without tokens
    }
    const int units = tiles * groups;
    const int64_t total = static_cast<int64_t>(units) * blocks;
    auto consider = [&](int grid) {
      if (grid < 1 || grid > sm_count || grid > total) {
        return;
      }
      // Thread blocks that share a tile: one more than the even share where the cuts
      // do not fall on tile ends. Shares of which one is complete early cost the sums
      // behind the last step all the same (12288 x 2560, 128 tokens: 96 whole tiles 14.6
      // us, two groups cut over 148 blocks 18.7; 384 tokens 24.8 and 27.5); others end
      // together, and their sums go through scratch.
      const int sharing = units % grid == 0 ? 1 : (grid % units == 0 ? grid / units : (grid + units - 1) / units + 1);
      const double fix = sharing <= 1 ? 0 : (units > grid ? 5000 + 15.0 * n : 9000 + 60.0 * n + 500.0 * sharing);
      const double cost = static_cast<double>((total + grid - 1) / grid) * StepCycles(type, n) + fix + 30.0 * n;
      if (cost < best_cost) {
        best_cost = cost;
        best = Plan{groups, n, grid, units, 1};
      }
    };
    // A unit shared by a cluster: the exchange and two cluster barriers on top (2560 x
    // 9728, 79 tokens: 22.1 / 21.9 / 17.6 / 15.9 / 15.4 / 16.5 us in clusters of one to six).
    for (int k = 2; k <= kMaxCluster && k <= blocks; ++k) {
      const double cost = static_cast<double>((blocks + k - 1) / k) * StepCycles(type, n) + 3500 + 20.0 * n;
      if (clusters[k] >= units && cost < best_cost) {
        best_cost = cost;
        best = Plan{groups, n, k * units, units, k};
      }
    }
    consider(sm_count);
    for (int share = 1; share * units <= sm_count; ++share) {
      consider(share * units);
    }
    for (int rounds = 2; rounds <= 4; ++rounds) {
      if (units % rounds == 0) {
        consider(units / rounds);
      }
    }
  }
  return best;
}

// Prepares the kernel on the context's device and says how many clusters of k blocks run at
// once, each block with all of its SM's shared memory (0: not known). What the driver refuses
// is asked for again at the next product.
template <int TYPE>
int ConfigureTc(const gufo_cuda_ctx* ctx, int (&clusters)[kMaxCluster + 1]) {
  struct Device {
    bool done = false;
    int clusters[kMaxCluster + 1] = {};
  };
  static std::mutex mu;
  static Device devices[16];
  std::lock_guard<std::mutex> lock(mu);
  Device& device = devices[ctx->device & 15];
  if (!device.done) {
    GUFO_CUDA_TRY(cudaFuncSetAttribute(GemmTc<TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedLimit - 3072));
    device.done = true;
    for (int k = 2; k <= kMaxCluster; ++k) {
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeClusterDimension;
      attr.val.clusterDim = {static_cast<unsigned>(k), 1, 1};
      cudaLaunchConfig_t config = {};
      config.gridDim = dim3(static_cast<unsigned>(k));
      config.blockDim = dim3(kTcThreads);
      config.dynamicSmemBytes = kSharedLimit - 3072;
      config.attrs = &attr;
      config.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&device.clusters[k], GemmTc<TYPE>, &config) != cudaSuccess) {
        cudaGetLastError();
        device.clusters[k] = 0;
        device.done = false;
      }
    }
  }
  std::copy(std::begin(device.clusters), std::end(device.clusters), clusters);
  return GUFO_CUDA_OK;
}

template <int TYPE>
int LaunchPlan(gufo_cuda_ctx* ctx, const GemvArgs& base, const std::vector<int>& group, int tokens) {
  using Q = Quant<TYPE>;
  int clusters[kMaxCluster + 1];
  int rc = ConfigureTc<TYPE>(ctx, clusters);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  const int cols = base.cols;
  const int blocks = cols / kSuperBlock;
  const Plan plan = PlanTc(base, group, TYPE, tokens, ctx->sm_count, clusters);
  // Scratch: header (error word, counters), tile images, unscale factors, partial sums.
  const size_t rows = static_cast<size_t>(plan.groups) * plan.n;
  const size_t unscale_at = kHeaderBytes + rows * cols * 2;
  const size_t partial_at = (unscale_at + rows * 4 + 255) / 256 * 256;
  const bool cuts = plan.cluster == 1 && plan.units % plan.grid != 0;
  const size_t partial_bytes = cuts ? static_cast<size_t>(plan.grid) * 2 * kTileRows * plan.n * 4 : 0;
  rc = ReserveTc(ctx, partial_at + partial_bytes);
  if (rc != GUFO_CUDA_OK) {
    return rc;
  }
  TcGemmArgs args{};
  args.blocks = blocks;
  args.groups = plan.groups;
  args.n = plan.n;
  args.units = plan.units;
  args.cluster = plan.cluster;
  args.per = plan.units * blocks / plan.grid;
  args.extra = plan.units * blocks % plan.grid;
  args.xh = ctx->tc_scratch + kHeaderBytes;
  args.unscale = reinterpret_cast<float*>(ctx->tc_scratch + unscale_at);
  args.partial = reinterpret_cast<float*>(ctx->tc_scratch + partial_at);
  args.counters = reinterpret_cast<unsigned*>(ctx->tc_scratch + 256);
  args.tokens = tokens;
  args.out_stride = base.y_stride;
  args.error = reinterpret_cast<int*>(ctx->tc_scratch);
  for (int p : group) {
    const GemvPart& part = base.parts[p];
    const int at = args.nparts++;
    args.parts[at] = {part.rows, (part.rows + kTileRows - 1) / kTileRows, base.y + part.out_offset};
    CUtensorMap* maps = &args.maps[at * 3];
    if (TYPE == GUFO_CUDA_Q4_K) {
      rc = EncodeRows(maps, part.data, part.rows, part.row_bytes, kQ4KBytes, CU_TENSOR_MAP_SWIZZLE_NONE);
    } else {
      rc = EncodeRows(maps, part.data, part.rows, part.row_bytes, 128, CU_TENSOR_MAP_SWIZZLE_128B);
      rc = rc != GUFO_CUDA_OK ? rc : EncodeRows(maps + 1, part.data, part.rows, part.row_bytes, 64, CU_TENSOR_MAP_SWIZZLE_64B);
      rc = rc != GUFO_CUDA_OK ? rc : EncodeRows(maps + 2, part.data, part.rows, part.row_bytes, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
    }
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  // Raw blocks (one a step) and activation stages (two a step), as deep in time.
  const int x_bytes = 2 * plan.n * kTileK * 2;
  const int room = kSharedLimit - 4096;
  args.raw_stages = kMaxStages;
  do {
    --args.raw_stages;
    args.x_stages = (room - args.raw_stages * Q::kRawStride) / x_bytes;
    args.x_stages = args.x_stages < kMaxStages ? args.x_stages : kMaxStages;
  } while (args.raw_stages > 2 && args.x_stages < 2 * args.raw_stages);
  const size_t smem = 1024 + static_cast<size_t>(args.x_stages) * x_bytes + static_cast<size_t>(args.raw_stages) * Q::kRawStride;
  // As many blocks a row as leave a block an SM, up to one for every 256 chunks of eight values.
  const int chunks = cols / 8;
  int row_blocks = ctx->sm_count / static_cast<int>(rows);
  row_blocks = std::max(1, std::min(row_blocks, (chunks + kStageThreads - 1) / kStageThreads));
  GUFO_CUDA_TRY(LaunchOverlapped(StageHalfKernel, dim3(static_cast<unsigned>(rows), static_cast<unsigned>(row_blocks)),
                                 dim3(kStageThreads), 0, ctx->stream, 1, base.x,
                                 tokens, cols, plan.n, TYPE == GUFO_CUDA_Q6_K ? 1 : 0, const_cast<uint8_t*>(args.xh),
                                 const_cast<float*>(args.unscale)));
  GUFO_CUDA_TRY(LaunchOverlapped(GemmTc<TYPE>, dim3(plan.grid), dim3(kTcThreads), smem, ctx->stream, plan.cluster, args));
  ctx->launches.fetch_add(2);
  return GUFO_CUDA_OK;
}

}  // namespace

bool TcGemmRuns(const gufo_cuda_ctx* ctx, int type, int cols, int tokens) {
  if (ctx->force_general || !ctx->tc_gemm || cols % kSuperBlock != 0) {
    return false;
  }
  // "tc_gemm" = 2 sends every product of 16 or more rows here (tests).
  const int least = ctx->tc_gemm_all ? 16 : kTcMinTokens;
  return (type == GUFO_CUDA_Q4_K || type == GUFO_CUDA_Q6_K) && tokens >= least;
}

int LaunchGemmTc(gufo_cuda_ctx* ctx, const GemvArgs& base, int tokens) {
  for (int p = 0; p < base.nparts; ++p) {
    if ((reinterpret_cast<uintptr_t>(base.parts[p].data) & 15) != 0 || base.parts[p].row_bytes % 16 != 0) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "tcgen05 gemm: weight rows must be 16-byte aligned");
    }
  }
  if (tokens > kPassTokens) {
    const int passes = (tokens + kPassTokens - 1) / kPassTokens;
    const int each = ((tokens + passes - 1) / passes + 15) / 16 * 16;
    for (int t0 = 0; t0 < tokens; t0 += each) {
      GemvArgs pass = base;
      pass.x = base.x + static_cast<size_t>(t0) * base.cols;
      pass.y = base.y + static_cast<size_t>(t0) * base.y_stride;
      const int rc = LaunchGemmTc(ctx, pass, tokens - t0 < each ? tokens - t0 : each);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
    }
    return GUFO_CUDA_OK;
  }
  // Parts of one block format share a launch, up to kTcMaxParts each.
  for (int type : {GUFO_CUDA_Q4_K, GUFO_CUDA_Q6_K}) {
    std::vector<int> group;
    for (int p = 0; p <= base.nparts; ++p) {
      if (p < base.nparts && base.parts[p].type == type) {
        group.push_back(p);
      }
      if (!group.empty() && (p == base.nparts || static_cast<int>(group.size()) == kTcMaxParts)) {
        const int rc = type == GUFO_CUDA_Q4_K ? LaunchPlan<GUFO_CUDA_Q4_K>(ctx, base, group, tokens)
                                              : LaunchPlan<GUFO_CUDA_Q6_K>(ctx, base, group, tokens);
        if (rc != GUFO_CUDA_OK) {
          return rc;
        }
        group.clear();
      }
    }
  }
  return GUFO_CUDA_OK;
}

int TcGemmError(gufo_cuda_ctx* ctx, int* code) {
  *code = 0;
  if (ctx->tc_scratch == nullptr) {
    return GUFO_CUDA_OK;
  }
  GUFO_CUDA_TRY(cudaMemcpyAsync(code, ctx->tc_scratch, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GUFO_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  if (*code != 0) {
    // A kernel that gave up may have left counters behind.
    GUFO_CUDA_TRY(cudaMemsetAsync(ctx->tc_scratch, 0, kHeaderBytes, ctx->stream));
  }
  return GUFO_CUDA_OK;
}

}  // namespace gufo
