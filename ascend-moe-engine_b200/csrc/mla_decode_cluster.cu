// Decode attention with a thread-block cluster per sequence: one launch, no partials in memory and no merge kernel.
//
// The flat kernel (mla_decode_tc.cu) cuts the tiles of all sequences into one run per SM and merges partials in a
// second kernel; it is at the HBM roof when there are many tiles, but a layer costs 16 us however little there is to
// read (two launches, the partials' way through L2, the merge's two round trips). Here a sequence (and group of up to
// 64 heads) belongs to a cluster of C CTAs (1 .. 16). They share its tiles out, and because an SM has nothing better to
// do when a sequence has fewer tiles than the cluster has CTAs, also its heads: S ranges of tokens x H groups of heads,
// S * H = C, H up to 4 with at least 16 heads each. (Heads and not output columns: what bounds a CTA with one tile is
// the 27 bytes a cycle an SM takes in, and a quarter of the heads is a quarter of Q's 72 KB.) Then the CTAs of a head
// group exchange what they accumulated through distributed shared memory (every CTA ends up with 512 / S columns of its
// heads from each of the S token ranges) and each merges and writes its columns. A cluster barrier before the exchange
// (the receivers' KV stages are the mailbox, so their MMAs must have finished; not needed when nobody has more than one
// tile, because the second stage is then free from the start), and one after it.
//
// With a tile or two per CTA everything is latency, so the code between the waits is kept short: shifts for divisions
// (S, H and C are powers of two), loads issued from all warps at once.
//
// With many tiles a stage's round trip bounds the loop, some 3,500 cycles a tile with the two stages in turn (stamps):
// 2,200 to a load's last byte, 250 to the softmax's wake-up, 1,100 of softmax, 1,900 until PV, which shares the tensor pipe
// with the next tile's QK, gives the last slab group back. (QK holding back while a PV is due was 20 % slower; waits that
// spin instead of parking 1 %.)
//
// Measured (B200, graph of layers, us a layer): one sequence of 129 tokens with the append 16.4 (flat kernel and merge)
// -> 7.6, of which 0.9 from the previous layer's end to the wait's return, 0.4 issue, 1.1 latency, 1.1 QK behind the
// 91 KB that a CTA takes in, 0.6 softmax, 0.7 PV, 0.6 + 0.9 exchange, 1.0 merge; 16 sequences of 300 .. 4,096 tokens in
// pages of 16 rows 361 (CUDA-core kernel) -> 51.3; 32 sequences of up to 2,048 tokens with 16 heads 373 -> 26.1.
//
// Roles as in the flat kernel: warps 0-3 softmax, 4 producer, 5 QK, 6 PV; all eight warps take part in the exchange and
// the merge. Every wait is bounded; a CTA
// that gives up still arrives at the cluster barriers, so no peer is left waiting. The softmax warps share barriers that
// have no bound, so they give up together (see the loop).
#include <cuda.h>
#include <cuda_fp8.h>

#include "common.cuh"
#include "mla_tc_common.cuh"
#include "sm100_ptx.cuh"

namespace b200kv {

int32_t GetRowMap(const void* base, int64_t stride, int64_t rows, int32_t width, int32_t box_rows, CUtensorMap* out);
int32_t GetQMap(const void* base, int64_t head_stride, int64_t seq_stride, int32_t batch, int32_t heads, int32_t box_heads,
                CUtensorMap* out);
int32_t CheckFusedAppend(const b200kv_decode_args& a);

namespace {

using namespace mla;

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 16;
constexpr int kDvGroup = 32;     // a warp's share of an accumulator: the unit in which columns change hands
constexpr int kLeastHeads = 16;  // heads of a CTA: a multiple of the sixteen rows a softmax warp has

enum Source { kTiles = 0, kBoxes = 1, kRowList = 2, kTableRows = 3 };

// Shared memory (offsets from a 1024-byte aligned base): Q, two KV stages, the low term of P (kSplitP), barriers.
constexpr int kOffQ = 0;
constexpr int kOffKv = kOffQ + kQBytes;
constexpr int kOffLo = kOffKv + kStages * kStageBytes;
constexpr int kLoBytes = kHeads * 128;
constexpr int kMiscBytes = 2048;
constexpr int SmemBytes(bool split_p) { return kOffLo + (split_p ? kLoBytes : 0) + kMiscBytes + 1024; }
static_assert(SmemBytes(true) <= 232448, "shared memory budget exceeded");
// The exchange: (m, l) of every token range [16][64] and the mailbox of accumulators, 131,072 / H bytes. They lie over
// Q and the KV stages once all CTAs are done with their tiles, or over the second stage alone when no CTA has more than
// one tile and H > 1 (64 KB of mailbox at most). The weights made of (m, l) are this CTA's own and lie where Q was.
constexpr int kMlBytes = kMaxCluster * kHeads * 4;
constexpr int kOffMl = kOffQ + kMlBytes;
constexpr int kOffW = kOffQ;
constexpr int kOffMlDirect = kOffKv + 2 * kStageBytes - 2 * kMlBytes;
constexpr int kDirectMailBytes = kStageBytes - 2 * kMlBytes;
static_assert(kMlBytes * 3 <= kQBytes && kDirectMailBytes >= kLatent * 32 * 4 && kStages == 2, "the exchange fits");

struct Misc {
  uint64_t kv_full[kStages][kGroups];
  uint64_t kv_empty[kStages][kGroups];
  uint64_t s_full[2];
  uint64_t s_empty[2];
  uint64_t p_full[kStages];
  uint64_t q_full[kGroups];
  uint64_t o_full;
  uint64_t drain[2];
  uint64_t new_row_full;
  uint64_t patched[kGroups];  // the fused append's row is in its tile
  uint32_t tmem_base;
  int32_t abort_flag;
  float factor[kHeads];
  alignas(16) unsigned char new_row[(kLatent + kRope) * 2];
};
static_assert(sizeof(Misc) <= kMiscBytes, "Misc does not fit its reservation");

struct ClusterParams {
  const int32_t* block_table;
  int64_t max_blocks;
  const int32_t* row_index;
  int64_t row_index_stride;
  const int32_t* kv_len;
  const int32_t* kv_begin;
  int64_t pool_rows;
  const char* new_latent;
  const char* new_rope;
  int64_t new_latent_bytes;
  int64_t new_rope_bytes;
  char* pool_latent;
  char* pool_rope;
  int64_t pool_latent_bytes;
  int64_t pool_rope_bytes;
  int32_t heads;
  int32_t group_heads;  // heads of a cluster: 16, 32 or 64
  int32_t box_rows;     // kBoxes: rows of a TMA box
  int32_t block_size;
  int32_t stable_tables;
  float scale_log2;
  float nat_hi, nat_lo;  // scale / scale_log2 in two terms: from the kernel's log2 domain back to natural logarithms
  __nv_bfloat16* out;
  uint8_t* out_q;
  uint8_t* out_scale;
  float* lse;
  float* user_o;
  float* user_m;
  float* user_l;
  int32_t* status;
};

// This CTA's part of its sequence.
struct Share {
  int ranges;        // S: token ranges, a power of two
  int ranges_log2;
  int range;         // this CTA's
  int t_lo, t_hi;    // its tiles
  int head_lo;       // its first head inside the cluster's group
  int heads;         // how many: 16, 32 or 64
  int first_peer;    // cluster rank of the first CTA of the same heads
};

// one_tile: no CTA is to have more than one tile, if there are CTAs enough.
__device__ __forceinline__ Share ShareOf(int tiles, int cluster, int rank, int group_heads, bool one_tile) {
  int log2 = 31 - __clz(cluster), heads = group_heads;
  // Halving the ranges halves what a CTA sends (64 KB at 64 heads and some 30 bytes a cycle) and the heads of Q it loads,
  // and adds tiles (72 KB at 27 bytes a cycle): worth it while it adds none, and from 64 heads also for the second tile
  // of some CTAs (one sequence of 1,024 tokens: 16.1 us in 16 ranges, 12.9 us in 8).
  while (heads > kLeastHeads && log2 > 0 && (2 * tiles <= (1 << log2) || (!one_tile && heads == kHeads && 2 * tiles <= (3 << log2)))) {
    --log2;
    heads >>= 1;
  }
  Share s;
  s.ranges = 1 << log2;
  s.ranges_log2 = log2;
  s.range = rank & (s.ranges - 1);
  const int group = rank >> log2;
  s.head_lo = group * heads;
  s.heads = heads;
  s.first_peer = group << log2;
  s.t_lo = (tiles * s.range) >> log2;  // (at most 2^25 tiles x 16 ranges)
  s.t_hi = (tiles * (s.range + 1)) >> log2;
  return s;
}

// A bounded wait by all lanes of a warp together. A phase that is complete already, the usual case for a tile's later slab
// groups, costs a probe and no call.
__device__ __forceinline__ bool WarpWait(uint32_t bar, uint32_t parity, Misc* misc, int32_t* status, int site) {
  if (__all_sync(0xffffffffu, ptx::MbarTestWait(bar, parity))) return true;
  return __all_sync(0xffffffffu, BoundedWait(bar, parity, misc, status, site));
}

template <int kSource, bool kSplitP>
__global__ void __launch_bounds__(kThreads, 1)
    MlaDecodeClusterKernel(const __grid_constant__ CUtensorMap latent_map, const __grid_constant__ CUtensorMap rope_map,
                           const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap q16_map,
                           ClusterParams p) {
  constexpr bool kCopied = kSource == kRowList || kSource == kTableRows;  // rows arrive by cp.async (generic proxy), one arrival a lane
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = ptx::SmemAddr(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* smem = smem_dyn + (base - raw);
  Misc* misc = reinterpret_cast<Misc*>(smem + kOffLo + (kSplitP ? kLoBytes : 0));
  const uint32_t q_addr = base + kOffQ;
  const uint32_t kv_addr = base + kOffKv;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cluster = gridDim.x;  // the grid is one cluster wide: a CTA's rank is its x
  const int rank = blockIdx.x;
  const int seq = blockIdx.y;
  const int head_first = blockIdx.z * p.group_heads;
  auto bar = [&](const uint64_t* b) { return ptx::SmemAddr(b); };

  if (p.stable_tables != 0) GridDependencyTrigger();
  const uint64_t drop_policy = ptx::L2PolicyEvictFirst();
  // Pool row at which tile t of the sequence starts; -1 (after recording it) for a missing or bad table entry, which
  // loads read as row 0 and stores skip.
  auto tile_row_checked = [&](int begin, int t) -> int64_t {
    const int tok = begin + t * kTile;
    const int64_t table_col = tok / p.block_size;
    const int64_t block = table_col < p.max_blocks ? p.block_table[static_cast<int64_t>(seq) * p.max_blocks + table_col] : -1;
    int64_t row = block * p.block_size + tok % p.block_size;
    if (block < 0 || row + kTile > p.pool_rows) {
      RecordError(p.status, B200KV_DEV_BAD_BLOCK, seq, tok / p.block_size, static_cast<int32_t>(block));
      row = -1;
    }
    return row;
  };
  // One slab of tile i, the announcement of its group's bytes with the group's first slab (the barrier counts one
  // arrival, so a phase cannot complete before it whichever thread's load lands first).
  auto issue_slab = [&](int64_t row, int i, int slab) {
    const int stage = i % kStages, group = min(slab >> 1, kGroups - 1);
    const uint32_t dst = kv_addr + stage * kStageBytes + slab * kSlabBytes;
    const uint32_t full = bar(&misc->kv_full[stage][group]);
    if (slab < 8 && (slab & 1) == 0) ptx::MbarArriveExpectTx(full, (group == kGroups - 1 ? 3 : 2) * kSlabBytes);
    if (slab < 8) {
      ptx::TmaLoad2DHint(dst, &latent_map, 64 * slab, static_cast<int32_t>(row), full, drop_policy);
    } else {
      ptx::TmaLoad2DHint(dst, &rope_map, 0, static_cast<int32_t>(row), full, drop_policy);
    }
  };

  // ---- setup: barriers and TMEM, which need nothing of the caller's, then the wait for the preceding kernel --------
  if (warp == 4 && lane == 0) {
    for (int s = 0; s < kStages; ++s) {
      for (int k = 0; k < kGroups; ++k) {
        ptx::MbarInit(bar(&misc->kv_full[s][k]), kCopied ? 32 : 1);
        ptx::MbarInit(bar(&misc->kv_empty[s][k]), 1);
      }
      ptx::MbarInit(bar(&misc->p_full[s]), kSoftmaxWarps);
      ptx::MbarInit(bar(&misc->s_full[s]), 1);
      ptx::MbarInit(bar(&misc->s_empty[s]), kSoftmaxWarps);
    }
    for (int k = 0; k < kGroups; ++k) {
      ptx::MbarInit(bar(&misc->q_full[k]), 1);
      ptx::MbarInit(bar(&misc->patched[k]), 1);
    }
    ptx::MbarInit(bar(&misc->o_full), 1);
    ptx::MbarInit(bar(&misc->drain[0]), 1);
    ptx::MbarInit(bar(&misc->drain[1]), 1);
    ptx::MbarInit(bar(&misc->new_row_full), 1);
    misc->abort_flag = 0;
    ptx::FenceBarrierInit();
    if constexpr (!kCopied) {
      ptx::PrefetchTensorMap(&latent_map);
      ptx::PrefetchTensorMap(&rope_map);
    }
    ptx::PrefetchTensorMap(&q_map);
    ptx::PrefetchTensorMap(&q16_map);
  }
  if (warp == 5) {
    ptx::TmemAlloc(ptx::SmemAddr(&misc->tmem_base), kTmemCols);
    ptx::TmemRelinquish();
  }
  __syncwarp();
  ptx::ClusterArrive();  // (waited for before the exchange: the peers have started)
  if (p.stable_tables == 0) {
    GridDependencyWait();
    GridDependencyTrigger();
  }
  const int len = max(p.kv_len[seq], 0);
  const int begin = p.kv_begin ? p.kv_begin[seq] : 0;
  const Share share = ShareOf(TilesOf(len), cluster, rank, p.group_heads, p.out_q != nullptr);
  const int n = share.t_hi - share.t_lo;
  const bool appends = p.new_latent != nullptr && n > 0 && share.t_hi == TilesOf(len);  // the new row is in this CTA's last tile
  int64_t first_row = 0;
  if (kSource == kTiles && warp >= 4 && n > 0) first_row = max(tile_row_checked(begin, share.t_lo), static_cast<int64_t>(0));
  ptx::TcFenceBeforeSync();
  __syncthreads();
  ptx::TcFenceAfterSync();
  if (p.stable_tables != 0) GridDependencyWait();  // Q, the new rows and the pool are the preceding kernels' to write

  // The first loads leave from all warps at once: a warp issues one cp.async.bulk.tensor in some 90 ns however many of
  // its lanes take part, so eighteen of them (Q and a tile) from one warp took 1.9 us of a 12 us launch. Warp w < 4 brings
  // Q's slab group w, warps 4-6 three slabs of the first tile each. Q: all 64 head rows of a slab in one box, or boxes of
  // sixteen when the CTA has fewer heads (the MMA's other rows then hold anything: a row of S depends on its own row of Q
  // only, and nothing reads those).
  if (n > 0 && lane == 0) {
    if (warp < 4) {
      const uint32_t qbar = bar(&misc->q_full[warp]);
      const int slabs = warp == kGroups - 1 ? 3 : 2;
      ptx::MbarArriveExpectTx(qbar, slabs * share.heads * 128);
      for (int c = 2 * warp; c < 2 * warp + slabs; ++c) {
        if (share.heads == kHeads) {
          ptx::TmaLoad3D(q_addr + c * kQSlabBytes, &q_map, 64 * c, head_first, seq, qbar);
        } else {
          for (int h = 0; h < share.heads; h += kLeastHeads) {
            ptx::TmaLoad3D(q_addr + c * kQSlabBytes + h * 128, &q16_map, 64 * c, head_first + share.head_lo + h, seq, qbar);
          }
        }
      }
    } else if constexpr (kSource == kTiles) {
      for (int c = 3 * (warp - 4); c < min(3 * (warp - 4) + 3, 9); ++c) issue_slab(first_row, 0, c);
    }
    if (warp == 4 && appends) {  // the sequence's new row, towards shared memory
      const uint32_t full = bar(&misc->new_row_full);
      ptx::MbarArriveExpectTx(full, (kLatent + kRope) * 2);
      ptx::BulkLoad(ptx::SmemAddr(misc->new_row), p.new_latent + seq * p.new_latent_bytes, kLatent * 2, full);
      ptx::BulkLoad(ptx::SmemAddr(misc->new_row) + kLatent * 2, p.new_rope + seq * p.new_rope_bytes, kRope * 2, full);
    }
  }
  __syncwarp();

  const uint32_t tmem = misc->tmem_base;
  bool ok = true;
  float m_run[2] = {kLowest, kLowest};  // reference maxima of this thread's two rows, log2 domain
  float l_run[2] = {0.0f, 0.0f};

  if (warp == 4 && n > 0) {
    // ======================= producer ===========================================================
    if constexpr (kCopied) {
      // An instruction of the warp moves four rows' 128 bytes of one slab; row numbers are found a tile ahead.
      const int g_sub = lane >> 3;
      const uint32_t g_chunk = lane & 7;
      int rid[kTile / 4];
      auto rows_of = [&](int t) {
        // A lane looks two of the tile's rows up; a row past the end is row 0, masked by the softmax and zeroed before PV.
        int mine[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int j = t * kTile + 32 * k + lane;
          mine[k] = 0;
          if (j < len) {
            if constexpr (kSource == kRowList) {
              if (j < p.row_index_stride) mine[k] = p.row_index[static_cast<int64_t>(seq) * p.row_index_stride + j];
              if (mine[k] < 0 || mine[k] >= p.pool_rows) {
                RecordError(p.status, B200KV_DEV_BAD_BLOCK, seq, j, mine[k]);
                mine[k] = 0;
              }
            } else {
              const int tok = begin + j;
              const int column = tok / p.block_size;
              const int64_t block =
                  tok >= 0 && column < p.max_blocks ? p.block_table[static_cast<int64_t>(seq) * p.max_blocks + column] : -1;
              const int64_t r = block * p.block_size + (tok - column * p.block_size);
              if (block < 0 || r >= p.pool_rows) {
                RecordError(p.status, B200KV_DEV_BAD_BLOCK, seq, column, static_cast<int32_t>(block));
              } else {
                mine[k] = static_cast<int>(r);
              }
            }
          }
        }
#pragma unroll
        for (int q = 0; q < kTile / 4; ++q) rid[q] = __shfl_sync(0xffffffffu, mine[q >> 3], (4 * q + g_sub) & 31);
      };
      const char* latent_lane = p.pool_latent + g_chunk * 16;
      rows_of(share.t_lo);
      for (int i = 0; i < n && ok; ++i) {
        const int stage = i % kStages;
        const uint32_t dst_lane = kv_addr + stage * kStageBytes + g_sub * 128;
        const char* src[kTile / 4];
#pragma unroll
        for (int q = 0; q < kTile / 4; ++q) src[q] = latent_lane + rid[q] * p.pool_latent_bytes;
#pragma unroll 1
        for (int c = 0; c < kGroups && ok; ++c) {
          if (i >= kStages) {
            ok = WarpWait(bar(&misc->kv_empty[stage][c]), ((i / kStages) & 1) ^ 1, misc, p.status, 210);
            if (!ok) break;
          }
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            const int slab = 2 * c + k;
#pragma unroll
            for (int q = 0; q < kTile / 4; ++q) {  // row r = 4 q + g_sub, so r % 8 = 4 (q % 2) + g_sub
              ptx::CpAsync16(dst_lane + slab * kSlabBytes + q * 512 + ((g_chunk ^ (4 * (q & 1) + g_sub)) << 4),
                             src[q] + slab * 128);
            }
          }
          if (c == kGroups - 1) {
#pragma unroll
            for (int q = 0; q < kTile / 4; ++q) {
              ptx::CpAsync16(dst_lane + 8 * kSlabBytes + q * 512 + ((g_chunk ^ (4 * (q & 1) + g_sub)) << 4),
                             p.pool_rope + rid[q] * p.pool_rope_bytes + g_chunk * 16);
            }
          }
          ptx::CpAsyncArriveOn(bar(&misc->kv_full[stage][c]));
        }
        if (ok && i + 1 < n) rows_of(share.t_lo + i + 1);
      }
      if (!ok) asm volatile("cp.async.wait_all;" ::: "memory");  // aborting: the copies land before the CTA goes on
    } else {
      // A lane has up to kUnits boxes of a tile (slab-major, so a lane's come in the order in which PV gives the groups
      // back). The warp polls together and a lane issues a box the moment its group is free.
      constexpr int kUnits = kSource == kTiles ? 1 : 3;
      const int boxes_log2 = kSource == kTiles ? 0 : __clz(p.box_rows) - __clz(kTile);
      const int units = 9 << boxes_log2, box_mask = (1 << boxes_log2) - 1;
      int64_t rows[kUnits];
      auto rows_of = [&](int t) {  // the pool rows of this lane's boxes of tile t
        if constexpr (kSource == kTiles) {
          rows[0] = tile_row_checked(begin, t);
          if (rows[0] < 0) rows[0] = 0;
        } else {
#pragma unroll
          for (int k = 0; k < kUnits; ++k) {
            const int u = lane + 32 * k;
            const int tok = t * kTile + (u & box_mask) * p.box_rows;
            rows[k] = 0;  // a box past the sequence's end: any rows will do
            if (u >= units || tok >= len) continue;
            const int column = tok / p.block_size;
            const int64_t block = column < p.max_blocks ? p.block_table[static_cast<int64_t>(seq) * p.max_blocks + column] : -1;
            const int64_t r = block * p.block_size + (tok - column * p.block_size);
            if (block < 0 || r + p.box_rows > p.pool_rows) {
              RecordError(p.status, B200KV_DEV_BAD_BLOCK, seq, column, static_cast<int32_t>(block));
            } else {
              rows[k] = r;
            }
          }
        }
      };
      const int my_group = lane < 6 ? (lane >> 1) : kGroups - 1;  // kTiles: lane s < 9 owns slab s
      constexpr int kFirst = kSource == kTiles ? 1 : 0;           // the first tile is on its way
      int issued = kFirst;
      if (kFirst < n) rows_of(share.t_lo + kFirst);
      for (int i = kFirst; i < n && ok; ++i) {
        const int stage = i % kStages;
        const uint32_t parity = ((i / kStages) & 1) ^ 1;
        int k = 0;
        uint64_t start = 0;
        for (uint32_t it = 0;; ++it) {
          if constexpr (kSource == kTiles) {
            if (k == 0 && (lane >= 9 || i < kStages || ptx::MbarTestWait(bar(&misc->kv_empty[stage][my_group]), parity))) {
              if (lane < 9) issue_slab(rows[0], i, lane);
              k = kUnits;
            }
          } else if (k < kUnits) {
            const int u = lane + 32 * k;
            const int slab = u >> boxes_log2, box = u & box_mask, group = min(slab >> 1, kGroups - 1);
            if (u >= units) {
              k = kUnits;
            } else if (i < kStages || ptx::MbarTestWait(bar(&misc->kv_empty[stage][group]), parity)) {
              const uint32_t full = bar(&misc->kv_full[stage][group]);
              const uint32_t dst = kv_addr + stage * kStageBytes + slab * kSlabBytes + box * p.box_rows * 128;
              const int32_t row = static_cast<int32_t>(k == 0 ? rows[0] : k == 1 ? rows[1] : rows[2]);
              if (box == 0 && slab < 8 && (slab & 1) == 0) ptx::MbarArriveExpectTx(full, (group == kGroups - 1 ? 3 : 2) * kSlabBytes);
              if (slab < 8) {
                ptx::TmaLoad2DHint(dst, &latent_map, 64 * slab, row, full, drop_policy);
              } else {
                ptx::TmaLoad2DHint(dst, &rope_map, 0, row, full, drop_policy);
              }
              ++k;
            }
          }
          if (__all_sync(0xffffffffu, k >= kUnits)) break;
          if ((it & 1023u) == 1023u) {
            const uint64_t now = ptx::GlobalTimerNs();
            if (start == 0) start = now;
            if (__any_sync(0xffffffffu, Aborting(misc) || now - start > 1000000000ull)) {
              if (!Aborting(misc) && lane == 0) RaiseTimeout(misc, p.status, 210, parity);
              ok = false;
              break;
            }
          }
        }
        if (!ok) break;
        issued = i + 1;
        if (issued < n) rows_of(share.t_lo + issued);
      }
      if (appends) {
        // The new row goes into its tile where the tile lies, in shared memory, group by group as both land, and to the
        // pool for the steps to come; the tile's own load need not wait for it. (The CTAs of all head groups put it into
        // their copies of the tile; one writes the pool.)
        const int last = n - 1, r = len - 1 - (share.t_hi - 1) * kTile;
        const int64_t row = share.head_lo == 0 ? tile_row_checked(begin, share.t_hi - 1) : -1;
        const int4* src = reinterpret_cast<const int4*>(misc->new_row);
        unsigned char* tile = smem + kOffKv + (last % kStages) * kStageBytes;
        ok = WarpWait(bar(&misc->new_row_full), 0, misc, p.status, 212);
        for (int g = 0; g < kGroups && ok; ++g) {
          ok = WarpWait(bar(&misc->kv_full[last % kStages][g]), (last / kStages) & 1, misc, p.status, 213);
          if (!ok) break;
          const int c = 16 * g + lane;  // 16-byte chunks: eight to a slab's 128-byte row
          if (lane < (g == kGroups - 1 ? 24 : 16)) {
            *reinterpret_cast<int4*>(tile + (c >> 3) * kSlabBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = src[c];
          }
          ptx::FenceProxyAsyncShared();
          __syncwarp();
          if (lane == 0) ptx::MbarArrive(bar(&misc->patched[g]));
        }
        if (ok && row >= 0) {  // nothing is written through a bad table entry
          for (int c = lane; c < (kLatent + kRope) / 8; c += 32) {
            char* dst = c < kLatent / 8 ? p.pool_latent + (row + r) * p.pool_latent_bytes + c * 16
                                        : p.pool_rope + (row + r) * p.pool_rope_bytes + (c - kLatent / 8) * 16;
            *reinterpret_cast<int4*>(dst) = src[c];
          }
        }
      }
      if (!ok && lane == 0) {  // aborting: loads that are on their way land first
        auto settle = [&](const uint64_t* b, uint32_t parity) {
          const uint64_t t0 = ptx::GlobalTimerNs();
          while (!ptx::MbarTryWait(bar(b), parity)) {
            if (ptx::GlobalTimerNs() - t0 > 200000000ull) break;
          }
        };
        if (appends) settle(&misc->new_row_full, 0);
        for (int i = max(0, issued - kStages); i < issued; ++i) {
          for (int k = 0; k < kGroups; ++k) settle(&misc->kv_full[i % kStages][k], (i / kStages) & 1);
        }
      }
    }
  } else if (warp == 5 && n > 0) {
    // ======================= QK =================================================================
    const uint64_t q_desc = ptx::SmemDescSw128(q_addr, 16, 1024);
    const uint64_t k_desc0 = ptx::SmemDescSw128(kv_addr, 16, 1024);
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const int n_u = __shfl_sync(0xffffffffu, n, 0);
    for (int i = 0; i < n_u && ok; ++i) {
      const int stage = i % kStages, buf = kSplitP ? 0 : i & 1;
      const uint32_t kv_parity = (i / kStages) & 1;
      const uint64_t kdesc = DescAt(k_desc0, stage * kStageBytes);
      const uint32_t d = tmem_u + kTmemColS + kTile * buf;
      constexpr uint32_t kNext = kSplitP ? kTile : 0;  // kSplitP: an accumulator per slab group
      auto group_ready = [&](int c) {
        ok = WarpWait(bar(&misc->kv_full[stage][c]), kv_parity, misc, p.status, 224 + c);
        if (ok && i == 0) ok = WarpWait(bar(&misc->q_full[c]), 0, misc, p.status, 222);
        if (ok && appends && i == n_u - 1) ok = WarpWait(bar(&misc->patched[c]), 0, misc, p.status, 223);
        if (!ok) return;
        ptx::TcFenceAfterSync();
        if constexpr (kCopied) ptx::FenceProxyAsyncShared();
      };
      if (i >= (kSplitP ? 1 : 2)) ok = WarpWait(bar(&misc->s_empty[buf]), ((kSplitP ? i : i >> 1) & 1) ^ 1, misc, p.status, 228);
      if (ok) group_ready(0);
      if (!ok) break;
      IssueQkGroup<0, 2, kSplitP>(q_desc, kdesc, d);
      group_ready(1);
      if (!ok) break;
      IssueQkGroup<2, 2, kSplitP>(q_desc, kdesc, d + kNext);
      group_ready(2);
      if (!ok) break;
      IssueQkGroup<4, 2, kSplitP>(q_desc, kdesc, d + 2 * kNext);
      group_ready(3);
      if (!ok) break;
      IssueQkGroup<6, 3, kSplitP>(q_desc, kdesc, d + 3 * kNext);
      if (ptx::ElectOne()) ptx::TcCommit(bar(&misc->s_full[buf]));
    }
  } else if (warp == 6 && n > 0) {
    // ======================= PV =================================================================
    const uint32_t idesc = __shfl_sync(0xffffffffu, share.heads == 16 ? ptx::InstrDescBf16(128, 16, 1, 0) : share.heads == 32 ? ptx::InstrDescBf16(128, 32, 1, 0) : ptx::InstrDescBf16(128, 64, 1, 0), 0);
    const uint64_t k_desc0 = ptx::SmemDescSw128(kv_addr, 16, 1024);
    const uint64_t v_desc0 = ptx::SmemDescSw128(kv_addr, kSlabBytes, 1024);
    const uint64_t lo_desc = ptx::SmemDescSw128(base + kOffLo, 16, 1024);
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    const int n_u = __shfl_sync(0xffffffffu, n, 0);
    for (int i = 0; i < n_u && ok; ++i) {
      const int stage = i % kStages;
      const int valid = len - (share.t_lo + i) * kTile;
      if (valid < kTile) {
        // Rows past the sequence's end hold whatever the pool held; zero them so 0 * NaN cannot reach O. This warp has
        // nothing else to do until P is there. (QK may still be reading these rows; their scores are masked.)
        for (int c = 0; c < kGroups && ok; ++c) ok = WarpWait(bar(&misc->kv_full[stage][c]), (i / kStages) & 1, misc, p.status, 220);
        if (!ok) break;
        unsigned char* stage_ptr = smem + kOffKv + stage * kStageBytes;
        for (int idx = lane; idx < (kTile - valid) * 64; idx += 32) {
          *reinterpret_cast<int4*>(stage_ptr + ((idx >> 3) & 7) * kSlabBytes + (valid + (idx >> 6)) * 128 + (idx & 7) * 16) = make_int4(0, 0, 0, 0);
        }
        ptx::FenceProxyAsyncShared();
        __syncwarp();
      }
      ok = WarpWait(bar(&misc->p_full[stage]), (i / kStages) & 1, misc, p.status, 221);
      if (!ok) break;
      ptx::TcFenceAfterSync();
      if constexpr (kCopied) ptx::FenceProxyAsyncShared();
      const uint32_t stage_off = stage * kStageBytes;
      const uint64_t pdesc = DescAt(k_desc0, stage_off + 8 * kSlabBytes);
      const uint64_t vdesc = DescAt(v_desc0, stage_off);
#pragma unroll
      for (int tm = 0; tm < 4; ++tm) {
#pragma unroll
        for (int ks = 0; ks < kTile / 16; ++ks) {
          const uint64_t a = DescAt(vdesc, 2 * tm * kSlabBytes + ks * 2048);
          const uint32_t acc = (i == 0 && ks == 0) ? 0u : 1u;
          if (ptx::ElectOne()) ptx::MmaF16SS(tmem_u + 64 * tm, a, DescAt(pdesc, ks * 32), idesc, acc);
          if constexpr (kSplitP) {
            if (ptx::ElectOne()) ptx::MmaF16SS(tmem_u + 64 * tm, a, DescAt(lo_desc, ks * 32), idesc, 1u);
          }
        }
        if (ptx::ElectOne()) ptx::TcCommit(bar(&misc->kv_empty[stage][tm]));
      }
    }
    if (ok && ptx::ElectOne()) ptx::TcCommit(bar(&misc->o_full));
  } else if (warp < 4 && n > 0) {
    // ======================= softmax ============================================================
    const int quad_row = lane >> 2;
    const int quad_col = (lane & 3) * 2;
    const int head0 = warp * 16 + quad_row;  // and head0 + 8: this thread's two rows
    const uint32_t lane_base = static_cast<uint32_t>(warp * 32) << 16;
    const bool has_rows = warp * 16 < share.heads;  // otherwise the warp only keeps step with the others
    // The four warps leave the loop together: a wait can run out for one of them and not for another, and whoever stayed
    // would stand at the named barriers for good. So a warp whose wait ran out goes through the barriers that the others
    // will come to: it asks for the rescaling path, where all four leave on one vote. The usual path carries no vote.
    auto leave_with_the_others = [&](bool at_the_vote) {
      if (!at_the_vote) ptx::NamedBarrierOr(1, kSoftmaxThreads, true);
      ptx::NamedBarrierOr(2, kSoftmaxThreads, true);
    };
    for (int i = 0; i < n; ++i) {
      const int buf = kSplitP ? 0 : i & 1, stage = i % kStages;
      const int valid = min(kTile, len - (share.t_lo + i) * kTile);
      ok = WarpWait(bar(&misc->s_full[buf]), (kSplitP ? i : i >> 1) & 1, misc, p.status, 230);
      if (!ok) {
        leave_with_the_others(false);
        break;
      }
      ptx::TcFenceAfterSync();
      uint32_t sr[32];
      if (has_rows) {
        ptx::TmemLd16x256bX8(tmem + lane_base + kTmemColS + kTile * buf, sr);
        ptx::TmemWaitLd();
        if constexpr (kSplitP) {
#pragma unroll 1
          for (int c = 1; c < kGroups; ++c) {
            uint32_t more[32];
            ptx::TmemLd16x256bX8(tmem + lane_base + kTmemColS + kTile * c, more);
            ptx::TmemWaitLd();
#pragma unroll
            for (int j = 0; j < 32; ++j) sr[j] = __float_as_uint(__uint_as_float(sr[j]) + __uint_as_float(more[j]));
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) sr[j] = 0u;
      }
      ptx::TcFenceBeforeSync();
      __syncwarp();
      if (lane == 0) ptx::MbarArrive(bar(&misc->s_empty[buf]));
      float x[2][16];  // x[r][2k + e] = score of row head0 + 8r, token 8k + quad_col + e
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        x[0][2 * k] = __uint_as_float(sr[4 * k]);
        x[0][2 * k + 1] = __uint_as_float(sr[4 * k + 1]);
        x[1][2 * k] = __uint_as_float(sr[4 * k + 2]);
        x[1][2 * k + 1] = __uint_as_float(sr[4 * k + 3]);
      }
      if (valid < kTile) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (8 * (j >> 1) + quad_col + (j & 1) >= valid) {
            x[0][j] = -INFINITY;
            x[1][j] = -INFINITY;
          }
        }
      }
      bool rescale = false;
      float neg_m[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float t[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) t[j] = fmaxf(x[r][2 * j], x[r][2 * j + 1]);
        float raw_max = fmaxf(fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])), fmaxf(fmaxf(t[4], t[5]), fmaxf(t[6], t[7])));
        raw_max = fmaxf(raw_max, __shfl_xor_sync(0xffffffffu, raw_max, 1));
        raw_max = fmaxf(raw_max, __shfl_xor_sync(0xffffffffu, raw_max, 2));
        const float tile_max = raw_max * p.scale_log2;
        const bool moves = tile_max > m_run[r] + kRescaleThreshold;
        const float m_new = moves ? tile_max : m_run[r];
        const float factor = i == 0 ? 1.0f : ptx::Ex2Approx(m_run[r] - m_new);
        m_run[r] = m_new;
        rescale |= moves && i > 0;
        if ((lane & 3) == 0) misc->factor[head0 + 8 * r] = factor;
        l_run[r] *= factor;
        neg_m[r] = -m_run[r];
      }
      uint32_t packed[2][8], packed_lo[2][kSplitP ? 8 : 1];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        float part[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float p0 = ptx::Ex2Approx(fmaf(x[r][2 * k], p.scale_log2, neg_m[r]));
          const float p1 = ptx::Ex2Approx(fmaf(x[r][2 * k + 1], p.scale_log2, neg_m[r]));
          const __nv_bfloat162 hi = __floats2bfloat162_rn(p0, p1);
          packed[r][k] = *reinterpret_cast<const uint32_t*>(&hi);
          if constexpr (kSplitP) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(p0 - __low2float(hi), p1 - __high2float(hi));
            packed_lo[r][k] = *reinterpret_cast<const uint32_t*>(&lo);
          }
          part[k] = p0 + p1;
        }
        float sum = ((part[0] + part[1]) + (part[2] + part[3])) + ((part[4] + part[5]) + (part[6] + part[7]));
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        l_run[r] += sum;
      }
      const bool any_rescale = ptx::NamedBarrierOr(1, kSoftmaxThreads, rescale);
      if (i > 0 && (any_rescale || kSplitP)) {
        // PV of the previous tile must have drained: before its accumulators are rescaled (rare), and before the one
        // buffer of P's low term is written again. (It ran under this tile's exponentials.)
        ok = WarpWait(bar(&misc->kv_empty[(i - 1) % kStages][kGroups - 1]), ((i - 1) / kStages) & 1, misc, p.status, 231);
        if (!ok) {
          if (any_rescale || i + 1 < n) leave_with_the_others(any_rescale);  // (after the last tile nobody comes to them)
          break;
        }
        ptx::TcFenceAfterSync();
      }
      if (any_rescale) {
        if (ptx::NamedBarrierOr(2, kSoftmaxThreads, false)) {
          ok = false;
          break;
        }
#pragma unroll 1
        for (int tm = 0; tm < 4; ++tm) {
#pragma unroll 1
          for (int half = 0; half < 2; ++half) {
            uint32_t o[32];
            const uint32_t addr = tmem + lane_base + 64 * tm + 32 * half;
            ptx::TmemLd32(addr, o);
            ptx::TmemWaitLd();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * misc->factor[32 * half + j]);
            ptx::TmemSt32(addr, o);
          }
        }
        ptx::TmemWaitSt();
        ptx::TcFenceBeforeSync();
      }
      unsigned char* stage_ptr = smem + kOffKv + stage * kStageBytes;
#pragma unroll
      for (int r = 0; r < 2; ++r) {  // P over the stage's rope slab: row = head, chunks of 16 bytes swizzled by the row
        const uint32_t in_slab = (head0 + 8 * r) * 128 + quad_col * 2;
        const uint32_t swizzle = static_cast<uint32_t>(quad_row << 4);
        const uint32_t prow = ptx::SmemAddr(stage_ptr + 8 * kSlabBytes + in_slab) ^ swizzle;
#pragma unroll
        for (int k = 0; k < 8; ++k) ptx::StShared32(prow ^ static_cast<uint32_t>(k << 4), packed[r][k]);
        if constexpr (kSplitP) {
          const uint32_t lrow = (base + kOffLo + in_slab) ^ swizzle;
#pragma unroll
          for (int k = 0; k < 8; ++k) ptx::StShared32(lrow ^ static_cast<uint32_t>(k << 4), packed_lo[r][k]);
        }
      }
      ptx::FenceProxyAsyncShared();
      if (any_rescale) ptx::NamedBarrier(2, kSoftmaxThreads);  // factors are read before the next tile rewrites them
      __syncwarp();
      if (lane == 0) ptx::MbarArrive(bar(&misc->p_full[stage]));
    }
    if (ok) ok = WarpWait(bar(&misc->o_full), 0, misc, p.status, 232);
    ptx::TcFenceAfterSync();
  }
  if (warp == 5 || warp == 6) {
    // Nothing of this warp's tensor work may be in flight when shared memory changes hands and TMEM is freed.
    __syncwarp();
    if (ptx::ElectOne()) {
      const uint32_t drain = bar(&misc->drain[warp - 5]);
      ptx::TcCommit(drain);
      const uint64_t t0 = ptx::GlobalTimerNs();
      while (!ptx::MbarTryWait(drain, 0)) {
        if (ptx::GlobalTimerNs() - t0 > 200000000ull) break;
      }
    }
  }
  __syncwarp();

  // ======================= exchange and merge =====================================================
  const bool direct = TilesOf(len) <= share.ranges && share.heads <= 32;  // the same in all CTAs of the cluster
  const int columns_log2 = 9 - share.ranges_log2;  // this CTA merges 512 / S output columns: range * columns ..
  const int columns = 1 << columns_log2;
  const int quads = share.heads >> 2;
  const int first = head_first + share.head_lo;
  const bool want_partial = p.user_o != nullptr;
  // What every call of an engine is: bf16 rows of whole heads, nothing else. The code for it is kept to the instructions
  // that do the work (a warp alone on its scheduler takes some six cycles for each); the rest goes through `emit`.
  const bool plain = !want_partial && p.out_q == nullptr && first + share.heads <= p.heads;
  // Four heads of one output column: lane = column, so an output store of the warp is 64 contiguous bytes of a row.
  auto emit = [&](int quad, int dv, const float (&acc)[4]) {  // every lane of the warp calls
    const int64_t row0 = static_cast<int64_t>(seq) * p.heads + first + 4 * quad;
    const int valid = p.heads - first - 4 * quad;  // heads of the quad that exist: four or more but for an odd count's last
    if (want_partial) {
      float* dst = p.user_o + row0 * kLatent + dv;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < valid) dst[i * kLatent] = acc[i];
      }
      return;
    }
    __nv_bfloat16 y[4];
    __nv_bfloat16* dst = p.out + row0 * kLatent + dv;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = __float2bfloat16_rn(acc[i]);
      if (i < valid) dst[i * kLatent] = y[i];
    }
    if (p.out_q != nullptr) {  // (64 heads: every quad is whole)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // The 32 columns of a row that a warp holds are one MX block, as in the flat kernel's merge.
        const float x = __bfloat162float(y[i]);
        const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(x) & 0x7fffffffu);
        const bool nan = top > 0x7f800000u;
        const MxScale block = MxScaleOf(__uint_as_float(top), nan);
        const uint32_t code = nan ? (((__float_as_uint(x) >> 24) & 0x80u) | 0x7fu)
                                  : static_cast<uint32_t>(__nv_cvt_float_to_fp8(__fmul_rn(x, block.inv), __NV_SATFINITE, __NV_E4M3));
        p.out_q[(row0 + i) * kLatent + dv] = static_cast<uint8_t>(code);
        if (lane == 0) p.out_scale[(row0 + i) * (kLatent / 32) + (dv >> 5)] = static_cast<uint8_t>(block.code);
      }
    }
  };
  auto emit_ml = [&](int h, float big, float total) {  // head h of this CTA's
    if (first + h >= p.heads) return;
    const int64_t at = static_cast<int64_t>(seq) * p.heads + first + h;
    // (The weights are exp2(s * scale_log2 - big) with scale_log2 rounded once; going back by the quotient of the two scales,
    // and rounding once more at the end, the log-sum-exp is as close to the scores' as with natural exponentials.)
    if (want_partial) {
      p.user_m[at] = big == -INFINITY ? big : fmaf(big, p.nat_hi, big * p.nat_lo);
      p.user_l[at] = total;
    } else if (p.lse != nullptr) {
      p.lse[at] = total == 0.0f ? -INFINITY : fmaf(big, p.nat_hi, fmaf(big, p.nat_lo, logf(total)));
    }
  };
  // (m, l) of this CTA's token range: lane j < 16 of a softmax warp takes row j of the warp's sixteen.
  const int from = 4 * (lane & 7);
  const float m_lo = __shfl_sync(0xffffffffu, m_run[0], from), m_hi = __shfl_sync(0xffffffffu, m_run[1], from);
  const float l_lo = __shfl_sync(0xffffffffu, l_run[0], from), l_hi = __shfl_sync(0xffffffffu, l_run[1], from);
  const bool failed = __any_sync(0xffffffffu, !ok);
  const float m_row = (lane & 8) ? m_hi : m_lo;
  const float l_row = failed ? 0.0f : ((lane & 8) ? l_hi : l_lo);
  const bool has_row = warp < 4 && lane < 16 && warp * 16 < share.heads;
  const int h_row = warp * 16 + lane;
  // The accumulators: warp w reads lanes 32 (w % 4) .. of numbers w / 4 and w / 4 + 2.
  const uint32_t acc_base = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 64 * (warp >> 2);
  const int dv_warp = 128 * (warp >> 2) + 32 * (warp & 3);  // output column of lane 0 in the first of the two, + 256 in the other
  if (n > 0 && warp >= 4) WarpWait(bar(&misc->o_full), 0, misc, p.status, 233);
  ptx::ClusterWait();

  if (share.ranges == 1 && plain) {
    // Nobody to exchange with: out of the accumulators straight into the rows.
    float* s_norm = reinterpret_cast<float*>(smem + kOffW);
    if (has_row) {
      s_norm[h_row] = l_row == 0.0f ? 0.0f : 1.0f / l_row;
      emit_ml(h_row, m_row, l_row);
    }
    __syncthreads();
    ptx::TcFenceAfterSync();
#pragma unroll 1
    for (int part = 0; part < 4; ++part) {  // 32 heads of one of the two accumulators
      const int half = part & 1, dv = dv_warp + 256 * (part >> 1) + lane;
      if (32 * half >= share.heads) continue;
      uint32_t o[32];
      ptx::TmemLd32(acc_base + 128 * (part >> 1) + 32 * half, o);
      ptx::TmemWaitLd();
      if (n == 0) {
#pragma unroll
        for (int q = 0; q < 32; ++q) o[q] = 0u;  // an empty sequence: nothing was accumulated
      }
      __nv_bfloat16* dst = p.out + (static_cast<int64_t>(seq) * p.heads + first + 32 * half) * kLatent + dv;
      const float4* norm = reinterpret_cast<const float4*>(s_norm + 32 * half);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (q == 4 && share.heads == kLeastHeads) break;
        const float4 w = norm[q];
        dst[(4 * q) * kLatent] = __float2bfloat16_rn(__uint_as_float(o[4 * q]) * w.x);
        dst[(4 * q + 1) * kLatent] = __float2bfloat16_rn(__uint_as_float(o[4 * q + 1]) * w.y);
        dst[(4 * q + 2) * kLatent] = __float2bfloat16_rn(__uint_as_float(o[4 * q + 2]) * w.z);
        dst[(4 * q + 3) * kLatent] = __float2bfloat16_rn(__uint_as_float(o[4 * q + 3]) * w.w);
      }
    }
    ptx::TcFenceBeforeSync();
    __syncthreads();
    if (warp == 5) {
      ptx::TcFenceAfterSync();
      ptx::TmemDealloc(tmem, kTmemCols);
    }
    return;
  }

  if (!direct) {
    ptx::ClusterArrive();
    ptx::ClusterWait();  // every CTA is done with its tiles: the KV stages and Q's place of all of them are free
  }
  ptx::TcFenceAfterSync();
  const uint32_t ml_off = direct ? kOffMlDirect : kOffMl;  // m, then l
  const uint32_t mail_off = direct ? kOffKv + kStageBytes : kOffKv;
  const uint32_t mail_mine = base + mail_off + share.range * (columns * share.heads * 4);
  if (has_row) {
    const uint32_t at = static_cast<uint32_t>(share.range * kHeads + h_row) * 4;
#pragma unroll 4
    for (int s = 0; s < share.ranges; ++s) {
      const uint32_t dst = ptx::MapToRank(base + ml_off + at, share.first_peer + s);
      ptx::StClusterF32(dst, m_row);
      ptx::StClusterF32(dst + kMlBytes, l_row);
    }
  }
  // O^T: a warp's 32 columns of an accumulator lie inside one CTA's share. The mailbox is [range][head quad][columns]
  // [4 heads] fp32, so a store of the warp is 512 contiguous bytes. (A CTA that failed sends l = 0, which makes what it
  // sends here count for nothing.)
  if (n > 0) {
    uint32_t dst[2];
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const int dv = dv_warp + 256 * a;
      dst[a] = ptx::MapToRank(mail_mine + ((dv & (columns - 1)) + lane) * 16, static_cast<uint32_t>(share.first_peer + (dv >> columns_log2)));
    }
    if (share.heads == kLeastHeads) {
      uint32_t o[2][16];
      ptx::TmemLd16(acc_base, o[0]);
      ptx::TmemLd16(acc_base + 128, o[1]);
      ptx::TmemWaitLd();
#pragma unroll
      for (int a = 0; a < 2; ++a) {
#pragma unroll
        for (int j = 0; j < 4; ++j) ptx::StClusterV4(dst[a] + j * columns * 16, o[a][4 * j], o[a][4 * j + 1], o[a][4 * j + 2], o[a][4 * j + 3]);
      }
    } else {
#pragma unroll 1
      for (int half = 0; half < share.heads >> 5; ++half) {
        uint32_t o[2][32];
        ptx::TmemLd32(acc_base + 32 * half, o[0]);
        ptx::TmemLd32(acc_base + 128 + 32 * half, o[1]);
        ptx::TmemWaitLd();
#pragma unroll
        for (int a = 0; a < 2; ++a) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            ptx::StClusterV4(dst[a] + (8 * half + j) * columns * 16, o[a][4 * j], o[a][4 * j + 1], o[a][4 * j + 2], o[a][4 * j + 3]);
          }
        }
      }
    }
    ptx::TcFenceBeforeSync();
  }
  __syncwarp();
  ptx::ClusterArrive();
  ptx::ClusterWait();
  if (warp == 5) {
    ptx::TcFenceAfterSync();
    ptx::TmemDealloc(tmem, kTmemCols);
  }

  // A unit is 32 columns x 4 heads. A warp takes consecutive units, quad after quad, and works a quad's weights out for
  // itself (lane = range x head, the maxima and sums are shuffles).
  const float* s_m = reinterpret_cast<const float*>(smem + ml_off);
  const float* s_l = reinterpret_cast<const float*>(smem + ml_off + kMlBytes);
  float4* s_w = reinterpret_cast<float4*>(smem + kOffW) + warp * kMaxCluster;  // [range] of the warp's present quad
  const int groups_log2 = columns_log2 - 5;  // columns / 32
  const int units = quads << groups_log2;
  const int unit_hi = units * (warp + 1) / kWarps;
  const float4* mail = reinterpret_cast<const float4*>(smem + mail_off);
  int have_quad = -1;
  bool whole = false;  // every range has a weight for each of the quad's heads
  for (int unit = units * warp / kWarps; unit < unit_hi; ++unit) {
    const int quad = unit >> groups_log2, group = unit & ((1 << groups_log2) - 1);
    if (first + 4 * quad >= p.heads) break;  // (units walk the quads upwards)
    if (quad != have_quad) {
      have_quad = quad;
      const int h = 4 * quad + (lane & 3);
      float m[2], l[2];
      float big = -INFINITY, total = 0.0f;
      bool zero = false;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int s = (lane >> 2) + 8 * k;
        l[k] = s < share.ranges ? s_l[s * kHeads + h] : 0.0f;
        m[k] = l[k] > 0.0f ? s_m[s * kHeads + h] : -INFINITY;
        big = fmaxf(big, m[k]);
      }
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, off));
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        m[k] = l[k] > 0.0f ? exp2f(m[k] - big) : l[k];  // the range's weight: zero without a sum, NaN if that is NaN
        zero |= (lane >> 2) + 8 * k < share.ranges && !(m[k] > 0.0f);
        total = fmaf(l[k], m[k], total);
      }
#pragma unroll
      for (int off = 4; off < 32; off <<= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
      whole = !__any_sync(0xffffffffu, zero);  // (and: the previous quad's weights have been read)
      const float norm = want_partial ? 1.0f : (total == 0.0f ? 0.0f : 1.0f / total);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int s = (lane >> 2) + 8 * k;
        if (s < share.ranges) reinterpret_cast<float*>(s_w)[4 * s + (lane & 3)] = m[k] * norm;
      }
      if (share.range == 0 && lane < 4 && group == 0) emit_ml(h, big, total);
      __syncwarp();
    }
    const int local = group * kDvGroup + lane;
    const float4* row = &mail[(quad << columns_log2) + local];
    const int step = quads << columns_log2;  // from one range to the next
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (whole) {
#pragma unroll 4
      for (int s = 0; s < share.ranges; ++s) {
        const float4 w = s_w[s], v = row[s * step];
        acc[0] = fmaf(v.x, w.x, acc[0]);
        acc[1] = fmaf(v.y, w.y, acc[1]);
        acc[2] = fmaf(v.z, w.z, acc[2]);
        acc[3] = fmaf(v.w, w.w, acc[3]);
      }
    } else {
#pragma unroll 1
      for (int s = 0; s < share.ranges; ++s) {
        const float4 w = s_w[s], v = row[s * step];
        // A range without tiles sent nothing: its weight is zero and its place holds anything.
        acc[0] = fmaf(w.x != 0.0f ? v.x : 0.0f, w.x, acc[0]);
        acc[1] = fmaf(w.y != 0.0f ? v.y : 0.0f, w.y, acc[1]);
        acc[2] = fmaf(w.z != 0.0f ? v.z : 0.0f, w.z, acc[2]);
        acc[3] = fmaf(w.w != 0.0f ? v.w : 0.0f, w.w, acc[3]);
      }
    }
    const int dv = (share.range << columns_log2) + local;
    if (plain) {
      __nv_bfloat16* dst = p.out + (static_cast<int64_t>(seq) * p.heads + first + 4 * quad) * kLatent + dv;
#pragma unroll
      for (int i = 0; i < 4; ++i) dst[i * kLatent] = __float2bfloat16_rn(acc[i]);
    } else {
      emit(quad, dv, acc);
    }
  }
}

using ClusterKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, ClusterParams);

template <int kSource, bool kSplitP>
ClusterKernel KernelOf() {
  return reinterpret_cast<ClusterKernel>(&MlaDecodeClusterKernel<kSource, kSplitP>);
}

cudaLaunchConfig_t ConfigOf(int32_t cluster, int32_t seqs, int32_t head_groups, int32_t smem, cudaStream_t stream,
                            cudaLaunchAttribute (&attrs)[2]) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(cluster), static_cast<unsigned>(seqs), static_cast<unsigned>(head_groups));
  config.blockDim = dim3(kThreads);
  config.dynamicSmemBytes = static_cast<size_t>(smem);
  config.stream = stream;
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attrs;
  config.numAttrs = 2;
  return config;
}

// How many clusters of 1, 2, 4, 8, 16 CTAs the current device holds at once (index: log2 of the size), and the
// kernels' opt-ins; looked up once per thread and device (a thread that goes from device to device keeps them all; a device
// number beyond the table is looked up whenever it comes after another).
struct ClusterLimits {
  int device = -1;
  int32_t most[5] = {};
};
constexpr int kKnownDevices = 16;

int32_t LimitsOf(const ClusterLimits** out) {
  static thread_local ClusterLimits known[kKnownDevices];
  int device = 0;
  if (int32_t rc = CheckCuda(cudaGetDevice(&device), "cudaGetDevice")) return rc;
  ClusterLimits& limits = known[device % kKnownDevices];
  if (device != limits.device) {
    const struct {
      ClusterKernel kernel;
      int smem;
    } kernels[] = {{KernelOf<kTiles, false>(), SmemBytes(false)},
                   {KernelOf<kRowList, false>(), SmemBytes(false)},
                   {KernelOf<kTiles, true>(), SmemBytes(true)},
                   {KernelOf<kBoxes, true>(), SmemBytes(true)},
                   {KernelOf<kTableRows, true>(), SmemBytes(true)}};
    for (const auto& k : kernels) {
      const void* fn = reinterpret_cast<const void*>(k.kernel);
      if (int32_t rc = CheckCuda(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem), "cluster decode smem opt-in")) return rc;
      if (int32_t rc = CheckCuda(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "cluster decode size opt-in")) return rc;
    }
    for (int k = 0; k < 5; ++k) {
      cudaLaunchAttribute attrs[2];
      cudaLaunchConfig_t config = ConfigOf(1 << k, 1, 1, SmemBytes(true), nullptr, attrs);
      config.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, reinterpret_cast<const void*>(KernelOf<kTableRows, true>()), &config) != cudaSuccess) {
        cudaGetLastError();  // a size the device does not offer
        clusters = 0;
      }
      limits.most[k] = clusters;
    }
    limits.device = device;
  }
  *out = &limits;
  return B200KV_OK;
}

// The largest box of 8, 16 or 32 rows (the swizzle's atom is eight rows) that no block boundary cuts; 0 when there is none.
int32_t BoxRowsOf(int32_t block_size) {
  return block_size % 32 == 0 ? 32 : block_size % 16 == 0 ? 16 : block_size % 8 == 0 ? 8 : 0;
}

// The heads that share a cluster and its reads of the history.
int32_t GroupHeadsOf(int32_t heads) { return heads <= 16 ? 16 : heads <= 32 ? 32 : kHeads; }

// The largest cluster with which all sequences (x head groups) are resident at once; single CTAs when none is.
int32_t ClusterSizeFor(const ClusterLimits& limits, int64_t units) {
  for (int k = 4; k > 0; --k) {
    if (units <= limits.most[k]) return 1 << k;
  }
  return 1;
}

int32_t Launch(const b200kv_decode_args& a, int source, bool split_p, int32_t cluster, int32_t group_heads, cudaStream_t stream,
               int32_t* status) {
  const int32_t box_rows = source == kBoxes ? BoxRowsOf(a.block_size) : kTile;
  CUtensorMap latent_map{}, rope_map{}, q_map, q16_map;
  if (source == kTiles || source == kBoxes) {
    if (int32_t rc = GetRowMap(a.pool.latent, a.pool.latent_row_stride, a.pool.pool_rows, kLatent, box_rows, &latent_map)) return rc;
    if (int32_t rc = GetRowMap(a.pool.rope, a.pool.rope_row_stride, a.pool.pool_rows, kRope, box_rows, &rope_map)) return rc;
  }
  if (int32_t rc = GetQMap(a.q, a.q_head_stride, a.q_seq_stride, a.batch, a.heads, kHeads, &q_map)) return rc;
  if (int32_t rc = GetQMap(a.q, a.q_head_stride, a.q_seq_stride, a.batch, a.heads, kLeastHeads, &q16_map)) return rc;
  ClusterParams p{};
  p.block_table = a.block_table;
  p.max_blocks = a.max_blocks;
  p.row_index = a.row_index;
  p.row_index_stride = a.row_index_stride;
  p.kv_len = a.kv_len;
  p.kv_begin = a.kv_begin;
  p.pool_rows = a.pool.pool_rows;
  p.new_latent = static_cast<const char*>(a.new_latent);
  p.new_rope = static_cast<const char*>(a.new_rope);
  p.new_latent_bytes = a.new_latent_stride * 2;
  p.new_rope_bytes = a.new_rope_stride * 2;
  p.pool_latent = static_cast<char*>(a.pool.latent);
  p.pool_rope = static_cast<char*>(a.pool.rope);
  p.pool_latent_bytes = a.pool.latent_row_stride * 2;
  p.pool_rope_bytes = a.pool.rope_row_stride * 2;
  p.heads = a.heads;
  p.group_heads = group_heads;
  p.box_rows = box_rows;
  p.block_size = a.block_size;
  p.stable_tables = (a.flags & B200KV_DECODE_STABLE_TABLES) != 0 ? 1 : 0;
  p.scale_log2 = a.scale * 1.4426950408889634f;
  const double nat = static_cast<double>(a.scale) / static_cast<double>(p.scale_log2);
  p.nat_hi = static_cast<float>(nat);
  p.nat_lo = static_cast<float>(nat - static_cast<double>(p.nat_hi));
  p.out = static_cast<__nv_bfloat16*>(a.out);
  p.out_q = static_cast<uint8_t*>(a.out_fp8);
  p.out_scale = static_cast<uint8_t*>(a.out_scale);
  p.lse = a.lse;
  p.user_o = a.partial_o;
  p.user_m = a.partial_m;
  p.user_l = a.partial_l;
  p.status = status;
  cudaLaunchAttribute attrs[2];
  const cudaLaunchConfig_t config =
      ConfigOf(cluster, a.batch, (a.heads + group_heads - 1) / group_heads, SmemBytes(split_p), stream, attrs);
  const ClusterKernel kernel = source == kTiles     ? (split_p ? KernelOf<kTiles, true>() : KernelOf<kTiles, false>())
                               : source == kBoxes   ? KernelOf<kBoxes, true>()
                               : source == kRowList ? KernelOf<kRowList, false>()
                                                    : KernelOf<kTableRows, true>();
  return CheckCuda(cudaLaunchKernelEx(&config, kernel, latent_map, rope_map, q_map, q16_map, p), "cluster decode launch");
}

}  // namespace

// Up to how many tiles in its longest sequence a batch is better off here than in the flat kernel, which spreads all
// tiles over all SMs but pays for two launches and the merge of every sequence's parts. Both sides measured (us a layer,
// flat -> here; all sequences of the length / lengths from a sixteenth of it):
//   16 CTAs  1 x 2,048: 15.7 -> 15.9, 1 x 4,096: 16.1 -> 19.5; 2 x 2,048: 20.5 -> 15.9, 2 x 4,096: 21.5 -> 19.8; 3 x 4,096:
//            17.5 -> 19.8; 4 x 2,048: 18.5 -> 16.4
//    8 CTAs  12 x 1,024: 17.5 -> 16.4; 8 x 2,048: 18.9 -> 19.2
//    4 CTAs  16 x 1,024: 18.5 -> 18.6, 32 x 1,024: 22.5 -> 21.1 / 20.3 -> 20.1; 32 x 4,096: 44.3 -> 43.9 / 33.1 -> 42.6
//    2 CTAs  64 x 512: 27.4 -> 21.7 / 23.9 -> 21.0, 64 x 768: / 26.7 -> 25.6
//    1 CTA   128 x 512: 41.5 -> 25.7; in more than one wave 256 x 512: 65.9 -> 56.6, 600 x 64: 68.8 -> 60.9
int64_t MostTilesFor(int32_t cluster, int32_t batch) {
  switch (cluster) {
    case 16: return batch == 2 ? 64 : 32;
    case 8: return 16;
    case 4: return 16;
    case 2: return 12;
    default: return 8;
  }
}

// Work small enough for the cluster kernel: *launched says whether the call was taken. The caller has checked that the
// flat kernel could take it.
int32_t TryDecodeCluster(const b200kv_decode_args& a, cudaStream_t stream, int32_t* status, bool* launched) {
  *launched = false;
  if (int32_t rc = CheckFusedAppend(a)) return rc;
  if (a.max_ctas > 0 || a.batch > 65535) return B200KV_OK;  // a caller's grid limit is the flat kernel's
  const ClusterLimits* limits = nullptr;
  if (int32_t rc = LimitsOf(&limits)) return rc;
  const int32_t cluster = ClusterSizeFor(*limits, a.batch);
  // The lengths are on the device; the table (or row list) says how many tiles a sequence can have at most.
  const int64_t most_tiles = a.row_index != nullptr ? (a.row_index_stride + kTile - 1) / kTile
                                                    : a.max_blocks * ((a.block_size + kTile - 1) / kTile);
  if (most_tiles > MostTilesFor(cluster, a.batch)) return B200KV_OK;
  // The weights are rounded to bf16 against the maximum of a CTA's first tile, so which tiles share a CTA moves results by
  // roundings: nothing in a bf16 row, but one in a hundred of its FP8 codes. Quantised calls keep their bytes: they come
  // here only where every tile has a CTA and a maximum of its own, as the flat kernel has it for so few tiles.
  if (a.out_fp8 != nullptr && most_tiles > cluster) return B200KV_OK;
  *launched = true;
  return Launch(a, a.row_index != nullptr ? kRowList : kTiles, false, cluster, kHeads, stream, status);
}

// Geometries that the 64-row tiles do not fit: any block size and any number of heads.
bool ClusterSupportsAny(const b200kv_decode_args& a) {
  return a.row_index == nullptr && a.new_latent == nullptr && a.partial_o == nullptr && a.q_head_stride % 8 == 0 && a.q_seq_stride % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(a.q) & 15u) == 0 && (a.batch == 1 || a.q_seq_stride > 0) &&
         a.q_seq_stride < (1ll << 38) && a.q_head_stride < (1ll << 30) &&  // (a batch that shares one query has no tensor map)
         a.pool.pool_rows <= INT32_MAX && a.batch <= 65535 && a.heads <= 65535 * kHeads;
}

int32_t LaunchDecodeClusterAny(const b200kv_decode_args& a, cudaStream_t stream, int32_t* status) {
  const ClusterLimits* limits = nullptr;
  if (int32_t rc = LimitsOf(&limits)) return rc;
  const int32_t group_heads = GroupHeadsOf(a.heads);
  const int64_t units = static_cast<int64_t>(a.batch) * ((a.heads + group_heads - 1) / group_heads);
  // TMA wants boxes that lie inside a block; a shard's first token may be anywhere, so shards go row by row.
  const int source = a.kv_begin != nullptr                ? kTableRows
                     : a.block_size % kTile == 0          ? kTiles
                     : BoxRowsOf(a.block_size) != 0       ? kBoxes
                                                          : kTableRows;
  return Launch(a, source, true, ClusterSizeFor(*limits, units), group_heads, stream, status);
}

}  // namespace b200kv
