// Q4_K and Q6_K GEMV / small-M GEMM (1..8 tokens) on the int8 tensor-core path for two
// tokens and more, and for one where rows are several slabs with a ragged last one;
// the arithmetic is gemv_mma.cu's, which runs the others (LaunchVariant and
// LaunchTokens there draw the line).
//
// Work split. A persistent grid (two or three thread blocks per SM) takes the 16-row
// tiles blockIdx.x, blockIdx.x + gridDim.x, ... The unit of work is a tile's 256-value
// block: 16 rows x 144 or 210 bytes (Q6_K rows in the planar device arrangement of
// common.cuh). The units of a block's tiles are numbered through and warp w takes
// every eighth, so that K = 2560 (ten blocks) keeps eight warps as busy as K = 2048
// does. A warp copies its own units, two (Q6_K) or three (Q4_K) ahead, with cp.async
// into a ring of its own and reads them back behind nothing but a warp barrier. The
// weights never depend on an earlier kernel, so the first units are requested
// before the grid-dependency wait.
//
// At the end of a tile every warp reduces its row sums over its quads, leaves them in
// one of four exchange buffers and arrives at the buffer's mbarrier; one warp (the
// duty rotates) adds the eight up a tile later, in a fixed order, and writes y.
// Launches with few tiles share each over a thread-block cluster: the sums cross to
// the cluster's first block through distributed shared memory.
//
// What bounds it: issue slots and the latency of a block's start. In gemv_mma.cu a
// slab of eight blocks is brought in by sixteen bulk copies, one per row, and the eight
// warps meet at a barrier for every slab: at K = 2560 every second slab has work for
// two warps only, and its short copies cost as much as long ones. Here the many small
// copies go through the load / store pipe, ahead of the input vector's loads, which
// is what slabs do better where rows are whole slabs and little else is done (one
// token). Microseconds, slabs -> units:
//   Q4_K 19456 x 2560: 1 token 10.9 -> 10.0, 2: 15.0 -> 10.9, 4: 17.3 -> 13.0, 8: 26.8 -> 19.5
//   Q6_K 124160 x 2560: 1 token 64 -> 57, 2: 90 -> 72, 8: 167 -> 117
//   Q6_K 2560 x 9728: 1 token 11.3 -> 11.9, 2: 16.3 -> 13.9, 4: 19.3 -> 16.8
//   Q4_K 8192 x 2048: 1 token 4.4 -> 4.9, 2: 4.6 -> 5.3, 4: 7.6 -> 7.3, 8: 10.3 -> 10.0
// (Two tokens against whole slabs lose a little by themselves but not in a step, whose
// launches then alternate between fewer kernels: every further one costs
// instruction-cache misses at each start.)
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "peer.cuh"
#include "q4k_unit.cuh"
#include "q6k_unit.cuh"

namespace gufo {
namespace {

template <int TYPE>
struct Unit;
template <>
struct Unit<GUFO_CUDA_Q4_K> {
  static constexpr int kPieces = 9;                   // 16-byte pieces of a row's block
  static constexpr int kRow = 160;                    // bytes between rows in shared memory: 32 mod 128
  static constexpr int kAcross = 3;                   // rows one copy instruction of a warp covers
  static constexpr int kDepth = 3;
  static constexpr int kGroup = 32;                   // values per entry of the image's sums
  static constexpr bool kZeros = false;
  static constexpr float kExtra = 1.0f / 16.0f;       // high nibbles reach the MMA as 16 q
};
template <>
struct Unit<GUFO_CUDA_Q6_K> {
  static constexpr int kPieces = 14;                  // ql 8, qh 4, scales 1, the slab's eight d 1
  static constexpr int kRow = 224;                    // 96 mod 128
  static constexpr int kAcross = 2;
  static constexpr int kDepth = 2;
  static constexpr int kGroup = 16;
  static constexpr bool kZeros = true;                // a plane of zeros behind the image
  static constexpr float kExtra = 0.25f;              // codes reach the MMA as 4 (q - 32)
};

constexpr int kExchange = 4;
constexpr int kTileRows = 16;

template <int TYPE, int TOKENS>
size_t SharedBytes(int cols, int depth, int limbs = kLimbs) {
  const ImageLayout l = MakeImageLayout(TOKENS, cols, Unit<TYPE>::kGroup, limbs);
  return static_cast<size_t>(l.bytes) + (Unit<TYPE>::kZeros ? l.plane_stride : 0) +
         static_cast<size_t>(kExchange) * kFastWarps * kTileRows * TOKENS * 4 +
         static_cast<size_t>(depth) * kFastWarps * kTileRows * Unit<TYPE>::kRow;
}

// MIX: the down product of a token's chosen experts with their weighted sum (Q4_K, one
// token a thread block). The experts' inputs lie side by side, so their narrow rows (two
// blocks of 256 values) are one row that keeps eight warps busy; every unit's row sums
// go to the exchange buffer by themselves, and whoever gathers a tile adds an expert's
// blocks and then the experts in slot order, as separate launches would. (The form
// before, a warp per row and expert in fp32, spent its time in conversions and in
// staging the activated inputs once per eight rows. Together with several tile pairs a
// block in the gate / up product, a layer of 256 experts of 512 x 2048, eight of them
// for each of four tokens: 34.4 -> 21.7 us. The inputs have a fourth byte plane, which
// costs the products no instruction: with 24 bits, as elsewhere, the rows were up to
// three times as far from a float64 result as the fp32 ones.)
template <int TYPE, int TOKENS, int PER_SM, bool MIX = false>
__global__ void __launch_bounds__(kFastThreads, PER_SM)
GemvUnits(const __grid_constant__ FastGemvArgs a) {
  using U = Unit<TYPE>;
  constexpr bool kQ4 = TYPE == GUFO_CUDA_Q4_K;
  constexpr int kLimbsHere = MIX ? kMixLimbs : kLimbs;
  constexpr int kNCols = TOKENS * kLimbsHere;
  constexpr int kNB = (kNCols + 7) / 8;
  constexpr int kTileFloats = kTileRows * TOKENS;   // per warp in an exchange buffer: row sums per token
  constexpr int kUnitBytes = kTileRows * U::kRow;
  extern __shared__ __align__(16) uint8_t smem[];
  // Where the blocks of a cluster leave their sums for block 0: [8][16][TOKENS].
  __shared__ float peers[8 * kTileFloats];
  __shared__ float squares[kFastWarps * TOKENS];         // a fused norm's (FillImage)
  __shared__ float* mirror;                              // the second copy of y, if any
  __shared__ __align__(8) uint64_t full[kExchange];      // a tile's row sums are all there
  __shared__ __align__(8) uint64_t empty[kExchange];     // ... and have been added up
  __shared__ __align__(8) uint64_t staged;               // the image's copy has landed
  // The barriers need no kernel argument: set up first, while the arguments' first
  // reads (constant-cache misses) are under way.
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < kExchange; ++s) {
      MbarInit(SharedAddress(&full[s]), kFastWarps);
      MbarInit(SharedAddress(&empty[s]), 1);
    }
    MbarInit(SharedAddress(&staged), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  const ImageLayout l = MakeImageLayout(TOKENS, a.cols, U::kGroup, kLimbsHere);
  const int blocks = a.cols / kSuperBlock;
  const float* col_scale = reinterpret_cast<const float*>(smem + l.scale_at);
  const float* sums = reinterpret_cast<const float*>(smem + l.sums_at);
  // After the image: (Q6_K) a plane of zeros, the exchange buffers
  // [kExchange][warps][16 rows][TOKENS], then every warp's ring of units.
  uint8_t* zeros = smem + l.bytes;
  float* exchange = reinterpret_cast<float*>(zeros + (U::kZeros ? l.plane_stride : 0));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;
  const int t = lane & 3;
  // (MIX: [kExchange][blocks][16 rows].)
  const int exchange_floats = MIX ? blocks * kTileRows : kFastWarps * kTileFloats;
  uint8_t* ring = reinterpret_cast<uint8_t*>(exchange + kExchange * exchange_floats) + warp * (a.depth * kUnitBytes);
  // Lane planes of the two unit kinds (q4k_unit.cuh, q6k_unit.cuh): column g of
  // the first MMA column group; lanes past the last token's planes wrap onto
  // live ones, whose sums meet a zero column factor.
  const uint8_t* lane_plane = smem + (g % kNCols) * l.plane_stride + 8 * t;
  const uint8_t* none = zeros + 8 * t;
  const bool one_live = (g & 3) < kNCols && ((g < 4) == (t < 2));
  const uint8_t* lane_first = TOKENS == 1 ? (one_live ? smem + (g & 3) * l.plane_stride + 8 * t : none)
                                          : (t < 2 ? lane_plane : none);
  const uint8_t* lane_second = t < 2 ? none : lane_plane;
  // Tiles of this block: n = 0 .. my_tiles - 1 (SwiGLU epilogue: a gate tile, then
  // the up tile of the same rows). With ksplit > 1 a cluster of ksplit blocks shares
  // one tile. (No division here: a block's first units cannot be requested before
  // these are known, and nothing hides a chain of integer divisions at a kernel's
  // start; the launcher divides.)
  const bool pairs = a.epilogue == kEpilogueSwiGlu;
  const int half_tiles = pairs ? TotalTiles(a) / 2 : 0;
  const int ks = a.ksplit > 1 ? a.ksplit : 1;
  int rank = 0;
  int slot = static_cast<int>(blockIdx.x);
  int my_tiles = a.tiles_each + (slot < a.tiles_more ? (pairs ? 2 : 1) : 0);
  if (ks > 1) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(slot));
    my_tiles = 1;
  }
  int group = 0, stride = static_cast<int>(gridDim.x);
  if constexpr (MIX) {
    group = slot / a.group_blocks;
    slot -= group * a.group_blocks;
    stride = a.group_blocks;
    my_tiles = a.tiles_each + (slot < a.tiles_more ? 1 : 0);
  }
  const int* mix_ids = MIX ? a.mix_ids + group * a.mix_experts : nullptr;
  auto locate = [&](int n, int* part, int* local) {
    const int tile = pairs ? slot + (n >> 1) * stride + (n & 1) * half_tiles : slot + n * stride;
    LocateTile(a, tile, part, local);
  };
  // This warp's units: of the tiles' blocks, numbered through, every eighth (of a
  // cluster's one tile, every eighth of each rank). (want_n, want_b): the next unit
  // to request.
  const int wide = ks > 1 ? kFastWarps * ks : kFastWarps;
  int want_n = 0, want_b = rank * kFastWarps + warp;
  auto settle = [&](int& n, int& b) {
    while (b >= blocks && n < my_tiles) {
      b -= blocks;
      ++n;
    }
  };
  settle(want_n, want_b);
  // Lane l copies piece l % kPieces of rows l / kPieces, + kAcross, ... of a unit.
  const int copy_row = lane / U::kPieces;
  const int piece = lane - copy_row * U::kPieces;
  auto request = [&](int at) {
    if (want_n < my_tiles) {
      int part, local;
      locate(want_n, &part, &local);
      // Rows past the end repeat the last row; their sums are never stored.
      const int last = a.parts[part].rows - 1 - local * kTileRows;
      const uint8_t* src = a.parts[part].w + static_cast<size_t>(local) * kTileRows * a.row_bytes;
      if constexpr (MIX) {
        const int e = want_b / a.mix_blocks;
        src += static_cast<size_t>(max(mix_ids[e], 0)) * a.parts[0].rows * a.row_bytes +
               (want_b - e * a.mix_blocks) * kQ4KBytes + 16 * piece;
      } else if constexpr (kQ4) {
        src += want_b * kQ4KBytes + 16 * piece;
      } else {
        // The planar arrangement of Q6_K rows (common.cuh).
        const int slab = want_b / kQ6KSlabBlocks, j = want_b % kQ6KSlabBlocks;
        const int count = min(kQ6KSlabBlocks, blocks - slab * kQ6KSlabBlocks);
        src += slab * (kQ6KSlabBlocks * kQ6KBytes) +
               (piece < 8 ? 128 * j + 16 * piece
                          : piece < 12 ? 128 * count + 64 * j + 16 * (piece - 8)
                                       : piece == 12 ? 192 * count + 16 * j : 208 * count);
      }
      const uint32_t dst = SharedAddress(ring + at * kUnitBytes + copy_row * U::kRow + 16 * piece);
#pragma unroll
      for (int r = 0; r < kTileRows; r += U::kAcross) {
        if (copy_row < U::kAcross && r + copy_row < kTileRows) {
          const int row = min(r + copy_row, last);
          asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;" ::"r"(dst + r * U::kRow),
                       "l"(src + static_cast<size_t>(row) * a.row_bytes) : "memory");
        }
      }
      want_b += wide;
      settle(want_n, want_b);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  __syncthreads();
#pragma unroll 1
  for (int i = 0; i < U::kDepth; ++i) {
    request(i);   // a ring shorter than kDepth holds all of a warp's units
  }
  // Waits for this block's own warps and copies (bounded all the same: one that runs
  // out leaves wrong rows instead of a hung grid).
  auto wait = [&](uint64_t* bar, unsigned parity) {
    const uint32_t at = SharedAddress(bar);
    if (!MbarTryWait(at, parity)) {
      const long long start = clock64();
      while (!MbarTryWait(at, parity) && clock64() - start < kLandLimit) {
      }
    }
  };
  if constexpr (U::kZeros) {
    // Read only after the image's barrier below.
    for (int i = threadIdx.x * 16; i < l.plane_stride; i += kFastThreads * 16) {
      *reinterpret_cast<uint4*>(zeros + i) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (a.prologue != kPrologueImage) {
    ZeroIdleColumns<TOKENS, kLimbsHere>(l, blocks, smem);
  }
  float norm_ahead[8];
  LoadNormAhead<TOKENS>(a, norm_ahead);
  const float inv_n = 1.0f / static_cast<float>(a.cols);
  GridLaunchDependents();
  // The weights above never depend on earlier kernels; the image and y do.
  GridDependencyWait();
  // Row-split ranks: the input vector may still be on its way from the peers.
  PeerWaitBlock(a.peer_wait);
  if (threadIdx.x == 0) {   // read behind the image's barrier
    mirror = a.mirror != nullptr ? *a.mirror : nullptr;
  }
  if (a.prologue == kPrologueImage) {
    if (threadIdx.x == 0) {
      MbarArriveExpectTx(SharedAddress(&staged), static_cast<uint32_t>(l.bytes));
      BulkCopy(SharedAddress(smem), a.image, static_cast<uint32_t>(l.bytes), SharedAddress(&staged));
    }
    wait(&staged, 0);
    __syncthreads();   // the plane of zeros, the mirror's address
  } else {
    FillImage<TOKENS, kLimbsHere>(a, l, smem, U::kExtra, MIX ? a.x + static_cast<size_t>(group) * a.cols : a.x, rank, ks,
                      norm_ahead, squares, inv_n);
  }
  // The norm's 1 / rms of token k in lane k.
  const float lane_scale = lane < TOKENS ? RowScale<TOKENS>(a, squares, lane, inv_n) : 1.f;

  float out[kNB][4];
  float off[TOKENS];
  auto clear = [&]() {
#pragma unroll
    for (int nb = 0; nb < kNB; ++nb) {
      out[nb][0] = out[nb][1] = out[nb][2] = out[nb][3] = 0.f;
    }
#pragma unroll
    for (int k = 0; k < TOKENS; ++k) {
      off[k] = 0.f;
    }
  };
  // Output o (row o / TOKENS, token o % TOKENS) of a tile from the eight warps' row
  // sums, added in a fixed order.
  auto total_of = [&](int n, int o) {
    const float* from = exchange + (n % kExchange) * (kFastWarps * kTileFloats) + o;
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < kFastWarps; ++w) {
      total += from[w * kTileFloats];
    }
    return total;
  };
  auto store = [&](int part, int local, int o, float total) {
    const int k = o % TOKENS;
    const int row = local * kTileRows + o / TOKENS;
    if (row < a.parts[part].rows) {
      const size_t at = static_cast<size_t>(k) * a.y_stride + (pairs ? 0 : a.parts[part].y_offset) + row;
      if (a.peer_out.world > 0) {
        // Row-split ranks: this rank's rows go straight into every rank's copy
        // of the full vector (plain stores over NVLink for the peers).
        for (int p = 0; p < a.peer_out.world; ++p) {
          a.peer_out.y[p][at] = total;
        }
      } else {
        a.y[at] = total;
        if (mirror != nullptr) {
          mirror[at] = total;
        }
      }
    }
  };
  // One warp adds a finished tile up and stores it (SwiGLU: a gate tile and the up
  // tile n behind it).
  auto gather = [&](int n) {
    if (pairs) {
      wait(&full[(n - 1) % kExchange], ((n - 1) / kExchange) & 1u);
    }
    wait(&full[n % kExchange], (n / kExchange) & 1u);
    int part, local;
    locate(n, &part, &local);
    if constexpr (MIX) {
      const int row = local * kTileRows + lane;
      if (lane < kTileRows && row < a.parts[0].rows) {
        const size_t y_at = static_cast<size_t>(group) * a.y_stride + row;
        const float* from = exchange + (n % kExchange) * exchange_floats + lane;
        float v = a.mix_base != nullptr ? a.mix_base[y_at] * a.mix_scale[group] : 0.f;
#pragma unroll 1
        for (int e = 0; e < a.mix_experts; ++e) {
          float y = 0.f;
#pragma unroll 1
          for (int j = 0; j < a.mix_blocks; ++j) {
            y += from[(e * a.mix_blocks + j) * kTileRows];
          }
          if (mix_ids[e] >= 0) {
            v = a.mix_base != nullptr ? fmaf(a.mix_weights[group * a.mix_experts + e], y, v) : y;
          }
        }
        if (a.mix_base != nullptr || mix_ids[0] >= 0) {
          a.y[y_at] = v;
        }
      }
      __syncwarp();
      if (lane == 0) {
        MbarArrive(SharedAddress(&empty[n % kExchange]));
      }
      return;
    }
#pragma unroll
    for (int first = 0; first < kTileFloats; first += 32) {
      const int o = first + lane;
      const float scale = __shfl_sync(0xFFFFFFFFu, lane_scale, o % TOKENS);
      if (o < kTileFloats) {
        const float total = scale * total_of(n, o);
        if (pairs) {
          store(part, local, o, SiluFast(scale * total_of(n - 1, o)) * total);
        } else {
          store(part, local, o, total);
        }
      }
    }
    __syncwarp();
    if (lane == 0) {
      if (pairs) {
        MbarArrive(SharedAddress(&empty[(n - 1) % kExchange]));
      }
      MbarArrive(SharedAddress(&empty[n % kExchange]));
    }
  };
  // Whether this warp gathers at tile n (the last of a pair): the duty rotates.
  auto duty = [&](int n) {
    return n >= 0 && (pairs ? (n & 1) != 0 && ((n >> 1) & 7) == warp : (n & 7) == warp);
  };
  // This warp's row sums so far: the columns of token k are 3k .. 3k + 2 (one token:
  // every column; dead ones carry a zero factor), the Q4_K offsets sit in lanes t < 2
  // for row g and t >= 2 for row g + 8; summed over the quad.
  auto flush = [&](float* tile) {
#pragma unroll
    for (int k = 0; k < TOKENS; ++k) {
      float lo = 0.f, hi = 0.f;
#pragma unroll
      for (int nb = 0; nb < kNB; ++nb) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int col = nb * 8 + 2 * t + j;
          const bool of_k = TOKENS == 1 || (col < kNCols && col / kLimbs == k);
          lo += of_k ? out[nb][j] : 0.f;
          hi += of_k ? out[nb][2 + j] : 0.f;
        }
      }
      lo -= t < 2 ? off[k] : 0.f;
      hi -= t < 2 ? 0.f : off[k];
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        lo += __shfl_xor_sync(0xFFFFFFFFu, lo, o);
        hi += __shfl_xor_sync(0xFFFFFFFFu, hi, o);
      }
      if (t == 0) {
        tile[g * TOKENS + k] = lo;
        tile[(g + 8) * TOKENS + k] = hi;
      }
    }
    clear();
  };
  clear();
  int b = rank * kFastWarps + warp;
  int at = 0;   // ring position of the next unit
#pragma unroll 1
  for (int n = 0; n < my_tiles; ++n) {
    if (MIX && n >= kExchange) {
      wait(&empty[n % kExchange], (n / kExchange - 1) & 1u);
    }
#pragma unroll 1
    for (; b < blocks; b += wide) {
      // This warp's own copies, so nothing but the warp meets here.
      asm volatile("cp.async.wait_group %0;" ::"n"(U::kDepth - 1) : "memory");
      __syncwarp();
      typename std::conditional<kQ4, q4k::Q4KUnit, q6k::Q6KUnit>::type unit;
      const uint8_t* data = ring + at * kUnitBytes;
      if constexpr (kQ4) {
        q4k::LoadFragments(unit, data + g * U::kRow, data + (g + 8) * U::kRow, t);
      } else {
        q6k::LoadFragments(unit, data + g * U::kRow, data + (g + 8) * U::kRow, b % kQ6KSlabBlocks, t);
      }
      __syncwarp();
      request(at);
      at = at + 1 == a.depth ? 0 : at + 1;
      if (a.variant == 1) {
        continue;
      }
      if constexpr (kQ4) {
        q4k::Accum<TOKENS> acc;
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc.out[nb][j] = out[nb][j];
          }
        }
#pragma unroll
        for (int k = 0; k < TOKENS; ++k) {
          acc.off[k] = off[k];
        }
        q4k::MultiplyUnit<TOKENS>(unit, b, g, t, lane_plane, l, col_scale, sums, acc);
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            out[nb][j] = acc.out[nb][j];
          }
        }
#pragma unroll
        for (int k = 0; k < TOKENS; ++k) {
          off[k] = acc.off[k];
        }
      } else {
        q6k::Accum<TOKENS> acc;
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            acc.out[nb][j] = out[nb][j];
          }
        }
        q6k::MultiplyUnit<TOKENS>(unit, b, g, t, lane_first, lane_second, l, col_scale, sums, acc);
#pragma unroll
        for (int nb = 0; nb < kNB; ++nb) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            out[nb][j] = acc.out[nb][j];
          }
        }
      }
      if constexpr (MIX) {
        flush(exchange + (n % kExchange) * exchange_floats + b * kTileRows);
      }
    }
    b -= blocks;
    if constexpr (!MIX) {
      // Zeros where this warp had no block of the tile.
      if (n >= kExchange) {
        wait(&empty[n % kExchange], (n / kExchange - 1) & 1u);
      }
      flush(exchange + ((n % kExchange) * kFastWarps + warp) * kTileFloats);
    }
    __syncwarp();
    if (lane == 0) {
      MbarArrive(SharedAddress(&full[n % kExchange]));
    }
    // The tile before: by now the other warps are done with it as a rule.
    if (ks == 1 && duty(n - 1)) {
      gather(n - 1);
    }
  }
  if (ks == 1) {
    if (duty(my_tiles - 1)) {
      gather(my_tiles - 1);
    }
  } else {
    // The blocks of a cluster: their sums meet in block 0, added in rank order.
    __syncthreads();
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int o = threadIdx.x;
    float* in_leader = cluster.map_shared_rank(peers, 0) + rank * kTileFloats;
    if (o < kTileFloats) {
      in_leader[o] = total_of(0, o);
    }
    cluster.sync();
    if (rank == 0 && o < kTileFloats) {
      float total = 0.f;
      for (int p = 0; p < ks; ++p) {
        total += peers[p * kTileFloats + o];
      }
      int part, local;
      locate(0, &part, &local);
      store(part, local, o, RowScale<TOKENS>(a, squares, o % TOKENS, inv_n) * total);
    }
  }
  if (a.peer_out.world > 0) {
    PeerSignal(a.peer_out);
  }
}

template <int TYPE, int TOKENS>
int Launch(gufo_cuda_ctx* ctx, const FastGemvArgs& args) {
  constexpr int kDepth = Unit<TYPE>::kDepth;
  // One token needs few enough registers for three resident blocks per SM.
  auto* kernel = GemvUnits<TYPE, TOKENS, TOKENS == 1 ? 3 : 2>;
  size_t smem = SharedBytes<TYPE, TOKENS>(args.cols, kDepth);
  if (smem > static_cast<size_t>(kFastMaxShared)) {
    return GUFO_CUDA_TOO_LARGE;
  }
  static bool configured[16] = {};   // all the shared memory a block may have, once per device
  if (!configured[ctx->device & 15]) {
    GUFO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFastMaxShared));
    configured[ctx->device & 15] = true;
  }
  int row_tiles = 0;
  for (int p = 0; p < args.nparts; ++p) {
    row_tiles += (args.parts[p].rows + kTileRows - 1) / kTileRows;
  }
  FastGemvArgs launch = args;
  launch.variant = ctx->gemv_variant;
  launch.ksplit = 1;
  launch.depth = kDepth;
  const bool pairs = args.epilogue == kEpilogueSwiGlu;
  if (pairs && (args.nparts != 2 || args.parts[0].rows != args.parts[1].rows ||
                args.parts[0].rows % kTileRows != 0 || args.peer_out.world > 0)) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: the SwiGLU epilogue takes two parts of equal whole tiles");
  }
  if (args.group_ids != nullptr) {
    return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: a grouped launch takes one token that fits the slab kernel");
  }
  const int items = pairs ? row_tiles / 2 : row_tiles;   // tiles or tile pairs
  int grid = 0;
  if (!pairs) {
    // Few tiles and several rounds of blocks: a cluster of up to four thread blocks
    // shares each tile, where all of them can run at once. A block then has few
    // units a warp, and a shorter ring lets more of them be resident (2048 x 6144:
    // three blocks with one unit a warp each).
    const int rounds = (args.cols / kSuperBlock + kFastWarps - 1) / kFastWarps;
    for (int ks = rounds < 4 ? rounds : 4; ks >= 2 && grid == 0; --ks) {
      const int depth = std::min(kDepth, (rounds + ks - 1) / ks);
      const size_t bytes = SharedBytes<TYPE, TOKENS>(args.cols, depth);
      if (row_tiles * ks <= ResidentBlocks(kernel, ctx->device, kFastThreads, bytes, ks)) {
        launch.ksplit = ks;
        launch.depth = depth;
        smem = bytes;
        grid = row_tiles * ks;
        launch.tiles_each = 1;
        launch.tiles_more = 0;
      }
    }
  }
  if (grid == 0) {
    grid = std::max(1, std::min(items, ResidentBlocks(kernel, ctx->device, kFastThreads, smem, 1)));
    // Items per block: block b takes items b, b + grid, ...
    launch.tiles_each = items / grid * (pairs ? 2 : 1);
    launch.tiles_more = items % grid;
  }
  GUFO_CUDA_TRY(LaunchOverlapped(kernel, dim3(grid), dim3(kFastThreads), smem, ctx->stream, launch.ksplit, launch));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

constexpr int kMixPerSm = 3;

template <int TYPE, int TOKENS>
bool FitsTokens(int cols) {
  return SharedBytes<TYPE, TOKENS>(cols, Unit<TYPE>::kDepth) <= static_cast<size_t>(kFastMaxShared);
}

template <int TYPE>
bool Fits(int cols, int tokens) {
  switch (tokens) {
    case 1: return FitsTokens<TYPE, 1>(cols);
    case 2: return FitsTokens<TYPE, 2>(cols);
    case 3: return FitsTokens<TYPE, 3>(cols);
    case 4: return FitsTokens<TYPE, 4>(cols);
    case 5: return FitsTokens<TYPE, 5>(cols);
    case 6: return FitsTokens<TYPE, 6>(cols);
    case 7: return FitsTokens<TYPE, 7>(cols);
    case 8: return FitsTokens<TYPE, 8>(cols);
    default: return false;
  }
}

template <int TYPE>
int LaunchTokens(gufo_cuda_ctx* ctx, const FastGemvArgs& args) {
  switch (args.tokens) {
    case 1: return Launch<TYPE, 1>(ctx, args);
    case 2: return Launch<TYPE, 2>(ctx, args);
    case 3: return Launch<TYPE, 3>(ctx, args);
    case 4: return Launch<TYPE, 4>(ctx, args);
    case 5: return Launch<TYPE, 5>(ctx, args);
    case 6: return Launch<TYPE, 6>(ctx, args);
    case 7: return Launch<TYPE, 7>(ctx, args);
    case 8: return Launch<TYPE, 8>(ctx, args);
    default: return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: 1 to 8 tokens per launch");
  }
}

}  // namespace

namespace {
size_t MixtureShared(int cols) {
  return SharedBytes<GUFO_CUDA_Q4_K, 1>(cols, Unit<GUFO_CUDA_Q4_K>::kDepth, kMixLimbs) +
         static_cast<size_t>(kExchange) * (cols / kSuperBlock) * kTileRows * 4;
}
}  // namespace

bool MixtureFits(int cols) { return MixtureShared(cols) <= static_cast<size_t>(kFastMaxShared); }

int LaunchGemvMixture(gufo_cuda_ctx* ctx, const FastGemvArgs& args) {
  auto* kernel = GemvUnits<GUFO_CUDA_Q4_K, 1, kMixPerSm, true>;
  const size_t smem = MixtureShared(args.cols);
  static bool configured[16] = {};
  if (!configured[ctx->device & 15]) {
    GUFO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFastMaxShared));
    configured[ctx->device & 15] = true;
  }
  FastGemvArgs launch = args;
  launch.nparts = 1;
  launch.prologue = kProloguePlain;
  launch.ksplit = 1;
  launch.depth = Unit<GUFO_CUDA_Q4_K>::kDepth;
  // As many blocks an input as let the whole launch be resident in the fewest rounds of
  // tiles; a block converts its input once for all of its tiles.
  const int tiles = (args.parts[0].rows + kTileRows - 1) / kTileRows;
  const int resident = std::max(1, ResidentBlocks(kernel, ctx->device, kFastThreads, smem, 1));
  const int64_t all = static_cast<int64_t>(tiles) * args.groups;
  const int rounds = static_cast<int>((all + resident - 1) / resident);
  launch.group_blocks = (tiles + rounds - 1) / rounds;
  launch.tiles_each = tiles / launch.group_blocks;
  launch.tiles_more = tiles % launch.group_blocks;
  GUFO_CUDA_TRY(LaunchOverlapped(kernel, dim3(launch.group_blocks * args.groups), dim3(kFastThreads), smem, ctx->stream,
                                 1, launch));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

bool UnitsFit(int type, int cols, int tokens) {
  return type == GUFO_CUDA_Q4_K ? Fits<GUFO_CUDA_Q4_K>(cols, tokens) : Fits<GUFO_CUDA_Q6_K>(cols, tokens);
}

int LaunchGemvUnits(gufo_cuda_ctx* ctx, int type, const FastGemvArgs& args) {
  return type == GUFO_CUDA_Q4_K ? LaunchTokens<GUFO_CUDA_Q4_K>(ctx, args) : LaunchTokens<GUFO_CUDA_Q6_K>(ctx, args);
}

}  // namespace gufo
