// Q4_K and Q6_K GEMV (one token; more in gemv_units.cu) on the int8 tensor-core
// path: the reference's fused row dots (gguf_dot::DotK4 and DotQ6_K,
// src/models/qwen35/gguf_dot.hpp:115-188,203-290) with the code dots taken
// exactly by mma.sync (arithmetic in mma_common.cuh, the per-unit math and the
// MMA operand layouts in q4k_unit.cuh and q6k_unit.cuh).
//   Q4_K: y_r = sum_blocks [ d * sum_j sc_j (q_j . x_j)  -  dmin * sum_j m_j (sum x_j) ]
//   Q6_K: y_r = sum_blocks d * sum_g sc_g * ((q - 32) . x)_g        g = 16-value groups
//
// Work split. A persistent grid (a few thread blocks per SM) takes the 16-row
// tiles blockIdx.x, blockIdx.x + gridDim.x, ... A tile is cut into slabs of up
// to eight 256-value blocks. A slab (16 rows x <= 1152 or 1680 bytes; Q6_K rows
// in the planar device arrangement of common.cuh) is brought into a ring slot in
// shared memory by sixteen bulk copies (cp.async.bulk, one per row, rows padded
// so that the fragment reads of a quarter-warp fall in distinct banks) that
// complete on the slot's mbarrier; warp w multiplies block w of the slab. The
// weights never depend on an earlier kernel, so the first slabs are requested
// before the grid-dependency wait.
//
// Per slab the eight warps meet once: each waits for the slot's barrier, reads
// its fragments into registers, and after the block's barrier the slot is free
// again, so warp q % 8 requests the slab kStages further on into it (the duty
// rotates) while everyone multiplies. At the end of a tile a warp reduces its
// row sums over its quads and leaves them in one of two exchange buffers;
// after the next slab's barrier sixteen threads per token add the eight warps'
// sums in a fixed order and write y. Launches with few row tiles share a tile's
// slabs over a thread-block cluster: the partial sums cross to the cluster's
// first block through distributed shared memory. (Tried and dropped: no block
// barrier at all, the last warp to release a slot refilling it and the last
// warp to finish a tile adding it up, both through shared-memory counters; it
// ran 20 % slower on the 262144 x 2048 product.)
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "peer.cuh"
#include "q4k_unit.cuh"
#include "q6k_unit.cuh"

namespace gufo {
namespace {

template <int TYPE>
struct Slab;
template <>
struct Slab<GUFO_CUDA_Q4_K> {
  static constexpr int kRowBytes = q4k::kSlabRowBytes;
  static constexpr int kBytes = q4k::kSlabBytes;
  static constexpr int kDataBytes = 8 * kQ4KBytes;   // of a full slab of one row
  static constexpr int kStages = 3;
  static constexpr int kGroup = 32;                   // values per entry of the image's sums
  static constexpr bool kZeros = false;
  static constexpr float kExtra = 1.0f / 16.0f;       // high nibbles reach the MMA as 16 q
};
template <>
struct Slab<GUFO_CUDA_Q6_K> {
  static constexpr int kRowBytes = q6k::kSlabRowBytes;
  static constexpr int kBytes = q6k::kSlabBytes;
  static constexpr int kDataBytes = q6k::kSlabDataBytes;
  static constexpr int kStages = 2;
  static constexpr int kGroup = 16;
  static constexpr bool kZeros = true;                // a plane of zeros behind the image
  static constexpr float kExtra = 0.25f;              // codes reach the MMA as 4 (q - 32)
};

constexpr int kMaxStages = 3;
constexpr int kExchange = 2;
constexpr int kTileFloats = 16;   // a warp's row sums in an exchange buffer
constexpr int kPerSm = 3;         // resident blocks the registers are for

// ONE: every block of the launch multiplies a single slab, so the ring is one
// slot (a third or half of the shared memory: more blocks fit an SM, which lets a
// cluster of three split a three-slab row where two-slot blocks allowed two).
template <int TYPE, bool ONE = false>
size_t SharedBytes(int cols) {
  const ImageLayout l = MakeImageLayout(1, cols, Slab<TYPE>::kGroup);
  return static_cast<size_t>(l.bytes) + (Slab<TYPE>::kZeros ? l.plane_stride : 0) +
         static_cast<size_t>(kExchange) * kFastWarps * kTileFloats * 4 +
         static_cast<size_t>(ONE ? 1 : Slab<TYPE>::kStages) * Slab<TYPE>::kBytes;
}

// GROUPED: the routed experts' products, a group's own input each (FastGemvArgs).
// PAIRS: a block may take several (gate tile, up tile) pairs; else one, tiles blockIdx.x
// and blockIdx.x + gridDim.x (the decode step's kernel stays 1 % faster without).
template <int TYPE, bool ONE = false, bool GROUPED = false, bool PAIRS = GROUPED>
__global__ void __launch_bounds__(kFastThreads, kPerSm)
GemvMma(const __grid_constant__ FastGemvArgs a) {
  using S = Slab<TYPE>;
  constexpr bool kQ4 = TYPE == GUFO_CUDA_Q4_K;
  constexpr int kStages = ONE ? 1 : S::kStages;
  extern __shared__ __align__(16) uint8_t smem[];
  // Where the blocks of a cluster leave their sums for block 0: [2][8][16].
  __shared__ float peers[2 * 8 * kTileFloats];
  __shared__ float squares[kFastWarps];                  // a fused norm's (FillImage)
  __shared__ float* mirror;                              // the second copy of y, if any
  __shared__ __align__(8) uint64_t landed[kMaxStages];   // a slab's bytes have arrived
  // The barriers need no kernel argument: set up first, while the arguments' first
  // reads (constant-cache misses) are under way. A barrier takes eight arrivals.
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < kStages; ++s) {
      MbarInit(SharedAddress(&landed[s]), kFastWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  const ImageLayout l = MakeImageLayout(1, a.cols, S::kGroup);
  const int blocks = a.cols / kSuperBlock;
  const int slabs_per_tile = (blocks + 7) / 8;
  const float* col_scale = reinterpret_cast<const float*>(smem + l.scale_at);
  const float* sums = reinterpret_cast<const float*>(smem + l.sums_at);
  // After the image: (Q6_K) a plane of zeros, the exchange buffers
  // [kExchange][warps][16 rows], then the slab ring.
  uint8_t* zeros = smem + l.bytes;
  float* exchange = reinterpret_cast<float*>(zeros + (S::kZeros ? l.plane_stride : 0));
  uint8_t* ring = reinterpret_cast<uint8_t*>(exchange + kExchange * kFastWarps * kTileFloats);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;
  const int t = lane & 3;
  // Lane planes of the two unit kinds (q4k_unit.cuh, q6k_unit.cuh): column g of
  // the MMA's; lanes past the planes wrap onto live ones (Q4_K: their sums meet a
  // zero column factor) or read zeros (Q6_K).
  const uint8_t* lane_plane = smem + (g % kLimbs) * l.plane_stride + 8 * t;
  const bool one_live = (g & 3) < kLimbs && ((g < 4) == (t < 2));
  const uint8_t* lane_first = (one_live ? smem + (g & 3) * l.plane_stride : zeros) + 8 * t;
  const int row_tiles = TotalTiles(a);
  // With ksplit > 1 a cluster of ksplit blocks shares each tile.
  // (No division here: a block's first slabs cannot be requested before these
  // are known, and nothing hides a chain of integer divisions at a kernel's start.
  // A cluster launch has one cluster per tile; the launcher divides the rest.)
  const int ks = a.ksplit > 1 ? a.ksplit : 1;
  int rank = 0;
  int slot = static_cast<int>(blockIdx.x);
  int stride = static_cast<int>(gridDim.x);
  int group = 0;   // GROUPED: picks the matrix of each part, the input and the output
  if constexpr (GROUPED) {
    group = slot / a.group_blocks;
    slot -= group * a.group_blocks;
    stride = a.group_blocks;
  }
  const bool pairs = PAIRS && a.epilogue == kEpilogueSwiGlu;
  int my_tiles = (a.tiles_each + (slot < a.tiles_more ? 1 : 0)) * (pairs ? 2 : 1);
  int slabs_mine = slabs_per_tile;
  if (ks > 1) {
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%clusterid.x;" : "=r"(slot));
    stride = row_tiles;
    my_tiles = 1;
    slabs_mine = 0;
    for (int s = rank; s < slabs_per_tile; s += ks) {
      ++slabs_mine;
    }
  }
  const int my_slabs = my_tiles * slabs_mine;
  // A block takes tiles slot, slot + stride, ... (of its group), or (SwiGLU epilogue)
  // those gate tiles, each followed by the up tile of the same rows.
  size_t matrix = 0;
  // The ids come from an earlier kernel. Where that one lets this grid start only
  // after it has itself waited for everything before it (early_input: the router's
  // top-k, enqueued in the same call), the inputs are complete already, and the image is built while the ids
  // are still being found. The dependents (the down product) start behind this
  // wait: they may read the ids and the weights ahead of their own.
  auto choose = [&]() {
    GridDependencyWait();
    GridLaunchDependents();
    const int id = a.group_ids[group];
    matrix = static_cast<size_t>(id);
    return id >= 0;
  };
  if constexpr (GROUPED) {
    if (!a.early_input && !choose()) {
      return;
    }
  }
  auto locate = [&](int n, int* part, int* local) {
    LocateTile(a, pairs ? slot + (n >> 1) * stride + (n & 1) * (row_tiles / 2) : slot + n * stride, part, local);
  };
  __syncthreads();

  // Brings slabs of this block into their ring slots (slab q into q % kStages);
  // (n, s) = tile and own-slab index of slab q. A barrier takes eight arrivals.
  // Ahead of the first multiplication every warp requests rows 2 * warp and
  // 2 * warp + 1 of each of the `count` first slabs, a bulk copy per row and lane
  // (one warp issuing a slab's sixteen copies spends about a thousand cycles in
  // that instruction, which here nothing hides); later one warp requests a whole
  // slab while the others multiply.
  const uint32_t ring_base = SharedAddress(ring);
  auto request = [&](int q, int n, int s, int r, bool announce, int rows_announced) {
    const int slab = rank + s * ks;
    int bytes;
    if constexpr (kQ4) {
      bytes = min(8, blocks - slab * 8) * kQ4KBytes;
    } else {
      // The row's last slab runs to the (16-byte padded) end of the row.
      bytes = min(S::kDataBytes, a.row_bytes - slab * S::kDataBytes);
    }
    const int at = q % kStages;
    const uint32_t bar = SharedAddress(&landed[at]);
    if (announce) {
      MbarArriveExpectTx(bar, static_cast<uint32_t>(rows_announced * bytes));
    }
    __syncwarp(__activemask());
    int part, local;
    locate(n, &part, &local);
    // Rows past the end repeat the last row; their sums are never stored.
    const int row = min(local * 16 + r, a.parts[part].rows - 1);
    const uint8_t* src = a.parts[part].w +
                         (matrix * a.parts[part].rows + static_cast<size_t>(row)) * a.row_bytes +
                         static_cast<size_t>(slab) * S::kDataBytes;
    BulkCopy(ring_base + at * S::kBytes + r * S::kRowBytes, src, static_cast<uint32_t>(bytes), bar);
  };
  auto issue_first = [&](int count) {
    const int mine = lane >> 1;   // which of the slabs this lane requests from
    if (mine < count) {
      int n = 0, s = mine;
      while (s >= slabs_mine) {
        s -= slabs_mine;
        ++n;
      }
      request(mine, n, s, 2 * warp + (lane & 1), (lane & 1) == 0, 2);
    }
  };
  auto issue = [&](int q, int n, int s) {
    if (lane < 16) {
      request(q, n, s, lane, lane < kFastWarps, 2);
    }
  };
  // (tile, own-slab index) of the next slab to request; every thread keeps it.
  int req_n = 0, req_s = 0;
  auto advance = [&]() {
    if (++req_s == slabs_mine) {
      req_s = 0;
      ++req_n;
    }
  };
  // A warp reads its fragments ahead of the block's barrier, so the slot is free for
  // the slab kStages on as soon as the barrier has passed.
  const int requested = min(kStages, my_slabs);
  for (int q = 0; q < requested; ++q) {
    advance();
  }
  if (!GROUPED || !a.early_input) {
    issue_first(requested);
  }
  if constexpr (S::kZeros) {
    // Read only after the image's barrier below.
#pragma unroll 1
    for (int i = threadIdx.x * 16; i < l.plane_stride; i += kFastThreads * 16) {
      *reinterpret_cast<uint4*>(zeros + i) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  if (a.prologue != kPrologueImage) {
    ZeroIdleColumns<1>(l, blocks, smem);
  }
  float norm_ahead[8];
  LoadNormAhead<1>(a, norm_ahead);
  const float inv_n = 1.0f / static_cast<float>(a.cols);
  if constexpr (!GROUPED) {
    GridLaunchDependents();
    // The weights above never depend on earlier kernels; the image and y do.
    GridDependencyWait();
  }
  // Row-split ranks: the input vector may still be on its way from the peers.
  PeerWaitBlock(a.peer_wait);
  if (threadIdx.x == 0) {   // read behind the image's barrier
    mirror = a.mirror != nullptr ? *a.mirror : nullptr;
  }
  if (a.prologue == kPrologueImage) {
    const uint32_t base = SharedAddress(smem);
    for (int at = threadIdx.x * 16; at < l.bytes; at += kFastThreads * 16) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + at), "l"(a.image + at)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  } else {
    FillImage<1>(a, l, smem, S::kExtra,
                 a.x + static_cast<size_t>(group / (a.x_group_div > 1 ? a.x_group_div : 1)) * a.x_group_stride,
                 rank, ks, norm_ahead, squares, inv_n);
  }
  if (GROUPED && a.early_input) {
    if (!choose()) {
      return;
    }
    issue_first(requested);
  }
  // The norm's 1 / rms, for the threads that store row sums.
  const float row_scale = threadIdx.x < kTileFloats ? RowScale<1>(a, squares, 0, inv_n) : 1.f;

  float out[4], off;
  auto clear = [&]() { out[0] = out[1] = out[2] = out[3] = off = 0.f; };
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  // The output rows of tile n from the eight warps' row sums in exchange buffer
  // x: thread o of the callers takes row o.
  auto total_of = [&](int x, int o) {
    const float* from = exchange + x * kFastWarps * kTileFloats + o;
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < kFastWarps; ++w) {
      total += from[w * kTileFloats];
    }
    return total;
  };
  auto store = [&](int n, int o, float total) {
    int part, local;
    locate(n, &part, &local);
    const int row = local * 16 + o;
    if (row < a.parts[part].rows) {
      const size_t at = static_cast<size_t>(group) * a.y_group_stride + (a.epilogue == kEpilogueSwiGlu ? 0 : a.parts[part].y_offset) + row;
      if (a.peer_out.world > 0) {
        // Row-split ranks: this rank's rows go straight into every rank's copy
        // of the full vector (plain stores over NVLink for the peers).
#pragma unroll 1   // not in the decode step's way: unrolled it costs 4-layer steps 2 %
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
  // Every thread of the block (of the cluster's blocks) comes here. With the
  // SwiGLU epilogue a block's tiles alternate gate, up: the gate's sum waits in
  // a register for the up tile's.
  float held_gate = 0.f;
  auto gather = [&](int n) {
    const int o = threadIdx.x;
    if (ks == 1) {
      if (o < kTileFloats) {
        const float total = row_scale * total_of(n % kExchange, o);
        if (a.epilogue != kEpilogueSwiGlu) {
          store(n, o, total);
        } else if ((n & 1) == 0) {
          held_gate = total;
        } else {
          store(n, o, SiluFast(held_gate) * total);
        }
      }
      return;
    }
    float total = o < kTileFloats ? total_of(n % kExchange, o) : 0.f;
    float* slot_in_leader = cluster.map_shared_rank(peers, 0) + ((n & 1) * 8 + rank) * kTileFloats;
    if (o < kTileFloats) {
      slot_in_leader[o] = total;
    }
    cluster.sync();
    if (rank != 0 || o >= kTileFloats) {
      return;
    }
    total = 0.f;
    for (int p = 0; p < ks; ++p) {
      total += peers[((n & 1) * 8 + p) * kTileFloats + o];
    }
    store(n, o, row_scale * total);
  };
  clear();
  int n = 0, s = 0;   // tile and own-slab index being multiplied
  for (int q = 0; q < my_slabs; ++q) {
    // Slab q has landed when its barrier's phase completes (bounded: the copies
    // were issued by this block; a wait that runs out gives the slab up).
    {
      const uint32_t bar = SharedAddress(&landed[q % kStages]);
      const uint32_t parity = (q / kStages) & 1u;
      if (!MbarTryWait(bar, parity)) {
        const long long start = clock64();
        while (!MbarTryWait(bar, parity) && clock64() - start < kLandLimit) {
        }
      }
    }
    const int slab = rank + s * ks;
    const int nblk = min(8, blocks - slab * 8);
    const int b = slab * 8 + warp;
    const bool mine = warp < nblk && a.variant != 1;
    const uint8_t* data = ring + (q % kStages) * S::kBytes;
    typename std::conditional<kQ4, q4k::Q4KUnit, q6k::Q6KUnit>::type unit;
    // The block's barrier: behind it a ring slot is free (every warp is done with
    // its slab: read into registers, or multiplied) and the row sums of the tile
    // before are in the exchange buffer. Warp q % 8 requests the next slab.
    auto meet = [&]() {
      __syncthreads();
      if (q + kStages < my_slabs) {
        if (warp == (q & 7)) {
          issue(q + kStages, req_n, req_s);
        }
        advance();
      }
      if (s == 0 && n > 0) {
        gather(n - 1);
      }
    };
    if (mine) {
      if constexpr (kQ4) {
        q4k::LoadUnit(unit, data, warp, g, t);
      } else {
        q6k::LoadUnit(unit, data, warp, nblk, g, t);
      }
    }
    meet();
    if (mine) {
      typename std::conditional<kQ4, q4k::Accum<1>, q6k::Accum<1>>::type acc;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc.out[0][j] = out[j];
      }
      if constexpr (kQ4) {
        acc.off[0] = off;
        q4k::MultiplyUnit<1>(unit, b, g, t, lane_plane, l, col_scale, sums, acc);
        off = acc.off[0];
      } else {
        q6k::MultiplyUnit<1>(unit, b, g, t, lane_first, lane_first, l, col_scale, sums, acc);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        out[j] = acc.out[0][j];
      }
    }
    if (s == slabs_mine - 1) {
      // This warp's row sums of the tile: every column (dead ones carry a zero
      // factor); the Q4_K offsets sit in lanes t < 2 for row g and t >= 2 for row
      // g + 8; summed over the quad.
      float* tile = exchange + ((n % kExchange) * kFastWarps + warp) * kTileFloats;
      float lo = out[0] + out[1] - (t < 2 ? off : 0.f);
      float hi = out[2] + out[3] - (t < 2 ? 0.f : off);
#pragma unroll
      for (int o = 1; o <= 2; o <<= 1) {
        lo += __shfl_xor_sync(0xFFFFFFFFu, lo, o);
        hi += __shfl_xor_sync(0xFFFFFFFFu, hi, o);
      }
      if (t == 0) {
        tile[g] = lo;
        tile[g + 8] = hi;
      }
      clear();
      s = 0;
      ++n;
    } else {
      ++s;
    }
  }
  if (my_tiles > 0) {
    __syncthreads();
    gather(my_tiles - 1);
  }
  if (a.peer_out.world > 0) {
    PeerSignal(a.peer_out);
  }
}

// Lets the kernel use all the shared memory a block may have (once per device).
template <int TYPE, bool ONE = false, bool GROUPED = false, bool PAIRS = GROUPED>
int Configure(const gufo_cuda_ctx* ctx) {
  static bool configured[16] = {};
  if (!configured[ctx->device & 15]) {
    GUFO_CUDA_TRY(cudaFuncSetAttribute(GemvMma<TYPE, ONE, GROUPED, PAIRS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, kFastMaxShared));
    configured[ctx->device & 15] = true;
  }
  return GUFO_CUDA_OK;
}

// Picks how many blocks share a tile's slabs (1, 2, 3 or 4: the largest that
// still lets every tile run at once) and the grid for it.
template <typename Kernel>
void PlanFastGrid(Kernel kernel, int device, int threads, size_t smem, int row_tiles, int slabs,
                  int* ksplit, int* grid) {
  for (int ks = slabs < 4 ? slabs : 4; ks >= 2; --ks) {
    const int resident = ResidentBlocks(kernel, device, threads, smem, ks);
    if (row_tiles * ks <= resident) {
      *ksplit = ks;
      *grid = row_tiles * ks;
      return;
    }
  }
  int resident = ResidentBlocks(kernel, device, threads, smem, 1);
  if (resident <= 0) {
    resident = 1;
  }
  *ksplit = 1;
  *grid = row_tiles < resident ? row_tiles : resident;
}

// LaunchVariant leaves the launch to gemv_units.cu.
constexpr int kNotTaken = -1;

template <int TYPE>
int LaunchVariant(gufo_cuda_ctx* ctx, const FastGemvArgs& args) {
  const size_t smem = SharedBytes<TYPE>(args.cols);
  if (smem > static_cast<size_t>(kFastMaxShared)) {
    return kNotTaken;
  }
  {
    const int rc = Configure<TYPE>(ctx);
    if (rc != GUFO_CUDA_OK) {
      return rc;
    }
  }
  int row_tiles = 0;
  for (int p = 0; p < args.nparts; ++p) {
    row_tiles += (args.parts[p].rows + 15) / 16;
  }
  FastGemvArgs launch = args;
  launch.variant = ctx->gemv_variant;
  const int slabs = (args.cols / kSuperBlock + 7) / 8;
  int grid = 1;
  if (args.group_ids != nullptr) {
    if (TYPE != GUFO_CUDA_Q4_K) {
      return Fail(GUFO_CUDA_UNSUPPORTED_TYPE, "fast gemv: grouped launches run Q4_K only");
    }
    if (args.groups <= 0 || args.tokens != 1 || args.prologue == kPrologueImage || args.prologue == kPrologueResNorm) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: a grouped launch takes one token and a fused input");
    }
    launch.ksplit = 1;
    if (args.epilogue == kEpilogueSwiGlu &&
        (args.nparts != 2 || args.parts[0].rows != args.parts[1].rows || args.parts[0].rows % 16 != 0)) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: the SwiGLU epilogue takes two parts of equal whole tiles");
    }
  } else if (args.epilogue == kEpilogueSwiGlu) {
    if (args.nparts != 2 || args.parts[0].rows != args.parts[1].rows || args.parts[0].rows % 16 != 0 ||
        args.peer_out.world > 0) {
      return Fail(GUFO_CUDA_BAD_ARGUMENT, "fast gemv: the SwiGLU epilogue takes two parts of equal whole tiles");
    }
    launch.ksplit = 1;
    grid = row_tiles / 2;
    if (grid > ResidentBlocks(GemvMma<TYPE>, ctx->device, kFastThreads, smem, 1)) {
      // More tile pairs than resident blocks: several a block (2 x 8192 x 2048: a step of
      // twelve layers 387 -> 349 us against the unit kernel).
      if (slabs > 1 && args.cols % (8 * kSuperBlock) != 0) {
        return kNotTaken;
      }
      const int rc = Configure<TYPE, false, false, true>(ctx);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
      auto* many = GemvMma<TYPE, false, false, true>;
      const int items = grid;
      grid = std::max(1, std::min(items, ResidentBlocks(many, ctx->device, kFastThreads, smem, 1)));
      launch.tiles_each = items / grid;
      launch.tiles_more = items % grid;
      GUFO_CUDA_TRY(LaunchOverlapped(many, dim3(grid), dim3(kFastThreads), smem, ctx->stream, 1, launch));
      ctx->launches.fetch_add(1);
      return GUFO_CUDA_OK;
    }
  } else {
    // Few rows and several slabs per tile: split the tiles' slabs over a cluster.
    PlanFastGrid(GemvMma<TYPE>, ctx->device, kFastThreads, smem, row_tiles, slabs, &launch.ksplit,
                 &grid);
    if (launch.ksplit == 1 && slabs > 1 && args.cols % (8 * kSuperBlock) != 0) {
      return kNotTaken;
    }
    {
      // Rows of two to four slabs whose (tile, slab) pairs do not all get a block
      // above: the one-slab form is smaller and may hold them (a 2048 x 6144 Q6_K
      // product: clusters of three blocks with one slab each instead of two blocks
      // with two and one). Only then: every further kernel that alternates with
      // the others in a decode step costs instruction-cache misses at each start
      // (the same launches ran 0.4 us slower when products that gain no wider
      // split went to this form too).
      if (slabs >= 2 && slabs <= 4 && launch.ksplit < slabs) {
        const size_t smem_one = SharedBytes<TYPE, true>(args.cols);
        auto* one = GemvMma<TYPE, true>;
        if (Configure<TYPE, true>(ctx) == GUFO_CUDA_OK &&
            row_tiles * slabs <= ResidentBlocks(one, ctx->device, kFastThreads, smem_one, slabs)) {
          launch.ksplit = slabs;
          launch.tiles_each = 1;
          launch.tiles_more = 0;
          GUFO_CUDA_TRY(LaunchOverlapped(one, dim3(row_tiles * slabs), dim3(kFastThreads), smem_one, ctx->stream,
                                         slabs, launch));
          ctx->launches.fetch_add(1);
          return GUFO_CUDA_OK;
        }
      }
    }
  }
  if constexpr (TYPE == GUFO_CUDA_Q4_K) {
    if (args.group_ids != nullptr) {
      const int rc = Configure<TYPE, false, true>(ctx);
      if (rc != GUFO_CUDA_OK) {
        return rc;
      }
      // As many blocks a group as let the whole launch be resident in the fewest rounds
      // of tiles (pairs): a block converts its group's input once for all of its tiles
      // and streams their weights through its ring (one block per pair: 1024 blocks
      // for 32 experts of 512 rows, each with a start and a conversion of its own).
      auto* kernel = GemvMma<TYPE, false, true>;
      const int resident = std::max(1, ResidentBlocks(kernel, ctx->device, kFastThreads, smem, 1));
      const int items = args.epilogue == kEpilogueSwiGlu ? row_tiles / 2 : row_tiles;
      const int64_t all = static_cast<int64_t>(items) * args.groups;
      const int rounds = static_cast<int>((all + resident - 1) / resident);
      launch.group_blocks = (items + rounds - 1) / rounds;
      launch.tiles_each = items / launch.group_blocks;
      launch.tiles_more = items % launch.group_blocks;
      GUFO_CUDA_TRY(LaunchOverlapped(kernel, dim3(launch.group_blocks * args.groups), dim3(kFastThreads), smem,
                                     ctx->stream, 1, launch));
      ctx->launches.fetch_add(1);
      return GUFO_CUDA_OK;
    }
  }
  {
    // Tiles per block (ksplit == 1): block b takes tiles b, b + grid, ...
    launch.tiles_each = row_tiles / grid;
    launch.tiles_more = row_tiles % grid;
  }
  GUFO_CUDA_TRY(LaunchOverlapped(GemvMma<TYPE>, dim3(grid), dim3(kFastThreads), smem, ctx->stream,
                                 launch.ksplit, launch));
  ctx->launches.fetch_add(1);
  return GUFO_CUDA_OK;
}

// One token runs here, but for launches of several slabs a row of which the last is
// ragged and which no cluster shares; the rest in gemv_units.cu (the figures that draw
// the line stand there).
template <int TYPE>
int LaunchTokens(gufo_cuda_ctx* ctx, const FastGemvArgs& args) {
  const int rc = args.tokens == 1 ? LaunchVariant<TYPE>(ctx, args) : kNotTaken;
  return rc == kNotTaken ? LaunchGemvUnits(ctx, TYPE, args) : rc;
}

}  // namespace

// Whether `tokens` rows of `cols` values fit the shared-memory image.
bool Q4KFastFits(int cols, int tokens) { return UnitsFit(GUFO_CUDA_Q4_K, cols, tokens); }
bool Q6KFastFits(int cols, int tokens) { return UnitsFit(GUFO_CUDA_Q6_K, cols, tokens); }

// Enqueues the Q4_K / Q6_K parts of one launch (a staged image or a fused input).
int LaunchGemvQ4KFast(gufo_cuda_ctx* ctx, const FastGemvArgs& args) { return LaunchTokens<GUFO_CUDA_Q4_K>(ctx, args); }
int LaunchGemvQ6KFast(gufo_cuda_ctx* ctx, const FastGemvArgs& args) { return LaunchTokens<GUFO_CUDA_Q6_K>(ctx, args); }

}  // namespace gufo
