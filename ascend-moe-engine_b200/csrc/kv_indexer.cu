// Sparse-selection indexer in front of attention: for every sequence, the k tokens of its paged history
// that score highest against the step's index query,
//   score_t = sum_h w_h * ReLU(qs_h * ks_t * (Q_h . K_t)),   Q_h, K_t FP8 E4M3 vectors of 128,
// as token positions, best first. The reference vendors this operator (aclnnQuantLightningIndexer) and
// plans it but does not apply it (include/moe/pipeline/pipeline.hpp:57-66). The positions go to
// b200kv_resolve_rows and from there to the decode attention over single-row blocks.
//
// The score kernel in this file runs on CUDA cores and is the reproducible one (the tensor-core score kernel
// is kv_indexer_tc.cu; b200kv_indexer_topk chooses). The arithmetic is fixed
// to the operation (one thread owns a token and runs the same fp32 fma chains as the CPU statement: over
// d = 0..127 for each head, then over the heads), so scores are bit-identical with the oracle and the
// selection is exact: tokens are ordered by (score descending, position ascending) as 64-bit keys; histograms find the
// k-th key's neighbourhood, and the keys up to there are sorted.
#include <cuda_fp8.h>

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace b200kv {
namespace {

constexpr int kIndexDim = 128;
constexpr int kMaxIndexHeads = 64;
constexpr int kScoreThreads = 128;
constexpr int kSortThreads = 1024;
constexpr int kMaxK = 2048;

__device__ __forceinline__ float E4m3ToFloat(uint32_t byte) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(byte), __NV_E4M3);
  return __half2float(*reinterpret_cast<const __half*>(&h));
}

struct ScoreParams {
  const uint8_t* q;        // [B][heads][128] fp8
  const float* q_scale;    // [B][heads]
  const __nv_bfloat16* w;  // [B][heads]
  int32_t heads;
  const uint8_t* key_pool;  // [rows][key_stride] fp8
  int64_t key_stride;
  const float* k_scale;  // [rows]
  int64_t pool_rows;
  const int32_t* block_table;
  int64_t max_blocks;
  const int32_t* kv_len;
  int32_t block_size;
  float* scores;  // [B][score_stride]
  int64_t score_stride;
  int32_t* status;
};

// Grid (token tiles of 128, sequence). The sequence's query (as fp32) and per-head coefficients sit in
// shared memory; a thread keeps its token's key row in registers and runs the chains.
__global__ void __launch_bounds__(kScoreThreads) IndexerScoreKernel(ScoreParams p) {
  GridDependencyTrigger();
  GridDependencyWait();
  __shared__ __align__(16) float q_s[kMaxIndexHeads * kIndexDim];
  __shared__ float qs_s[kMaxIndexHeads];
  __shared__ float w_s[kMaxIndexHeads];
  const int b = blockIdx.y;
  const int len = p.kv_len[b];
  const int t0 = blockIdx.x * kScoreThreads;
  if (t0 >= len) return;
  for (int i = threadIdx.x; i < p.heads * kIndexDim; i += kScoreThreads) {
    q_s[i] = E4m3ToFloat(p.q[static_cast<int64_t>(b) * p.heads * kIndexDim + i]);
  }
  for (int i = threadIdx.x; i < p.heads; i += kScoreThreads) {
    qs_s[i] = p.q_scale[b * p.heads + i];
    w_s[i] = __bfloat162float(p.w[b * p.heads + i]);
  }
  __syncthreads();
  const int t = t0 + threadIdx.x;
  if (t >= len) return;
  const int64_t column = t / p.block_size;
  const int64_t block = column < p.max_blocks ? p.block_table[static_cast<int64_t>(b) * p.max_blocks + column] : -1;
  const int64_t row = block * p.block_size + t % p.block_size;
  if (block < 0 || row >= p.pool_rows) {
    RecordError(p.status, B200KV_DEV_BAD_BLOCK, b, static_cast<int32_t>(column), static_cast<int32_t>(block));
    p.scores[b * p.score_stride + t] = -INFINITY;
    return;
  }
  float k[kIndexDim];
  {
    const int4* src = reinterpret_cast<const int4*>(p.key_pool + row * p.key_stride);
#pragma unroll
    for (int c = 0; c < kIndexDim / 16; ++c) {
      const int4 v = src[c];
      const uint32_t words[4] = {static_cast<uint32_t>(v.x), static_cast<uint32_t>(v.y), static_cast<uint32_t>(v.z),
                                 static_cast<uint32_t>(v.w)};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 4; ++e) k[16 * c + 4 * j + e] = E4m3ToFloat((words[j] >> (8 * e)) & 0xffu);
      }
    }
  }
  const float ks = p.k_scale[row];
  float score = 0.0f;
  for (int h = 0; h < p.heads; ++h) {
    const float4* qh = reinterpret_cast<const float4*>(q_s + h * kIndexDim);
    float dot = 0.0f;
#pragma unroll
    for (int d4 = 0; d4 < kIndexDim / 4; ++d4) {
      const float4 qv = qh[d4];
      dot = __fmaf_rn(qv.x, k[4 * d4], dot);
      dot = __fmaf_rn(qv.y, k[4 * d4 + 1], dot);
      dot = __fmaf_rn(qv.z, k[4 * d4 + 2], dot);
      dot = __fmaf_rn(qv.w, k[4 * d4 + 3], dot);
    }
    const float scaled = __fmul_rn(__fmul_rn(qs_s[h], ks), dot);
    const float s = scaled > 0.0f ? scaled : 0.0f;
    score = __fmaf_rn(w_s[h], s, score);
  }
  p.scores[b * p.score_stride + t] = score;
}

// Key that sorts ascending into (score descending, position ascending): high word = the complement of the
// score's order-preserving integer image, low word = the position. A NaN score counts as -infinity; +0 and
// -0 compare equal.
__device__ __forceinline__ uint64_t SortKey(float score, uint32_t position) {
  if (score != score) score = -INFINITY;
  score += 0.0f;
  uint32_t bits = __float_as_uint(score);
  bits = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);  // ascending with the value
  return (static_cast<uint64_t>(~bits) << 32) | position;
}

// The selection. The k best tokens are the k smallest 64-bit keys, all distinct. A cluster of C CTAs (1 .. 16, one for
// every 4,096 tokens of the longest sequence, as long as the batch fits the GPU at once) takes a sequence, a CTA a
// consecutive C-th of it, the score images of its first 8,192 tokens in registers.
//
//   bound    The k-th key is narrowed down by histograms of 512 bins over the range in which it lies, the first range
//            being that of the sequence's scores (equal steps of the image between the smallest and the largest, so the
//            bins that matter are thinly filled; bins of leading bits would put nearly all scores of a sequence into a
//            handful). Every CTA reads the others' histograms through distributed shared memory and draws the same
//            conclusion. The passes end when the keys up to the chosen bin's end are few enough to be sorted (half as
//            many again as wanted): one pass for scores without far outliers. Scores that are equal
//            are told apart by position, in histograms of positions, only when there are too many of them.
//   collect  The histograms also say where each bin's keys belong in the order and which part of a bin is which CTA's, so
//            a CTA can write its keys up to the bound straight to their bins' places in the list.
//   order    Inside a bin the list is in no order: a key's place is its bin's start plus the number of smaller keys in the
//            bin. The CTAs share the list's entries out (a key is sent to those whose entries its bin overlaps: small
//            stores to another SM go at one in three or four cycles, so sending all to all took 4 us), several threads to
//            a key. Bins hold tens of keys, so this is a few thousand comparisons a CTA in place of a sort; where scores
//            are so equal that bins get large, one CTA sorts the list.
//
// Bound by latencies: a cluster barrier costs some 0.6 us and there are three. It replaces a radix select by leading
// digits in one CTA (sequences up to 8,192 tokens; atomics on a few bins serialise), and for longer sequences in two
// levels, of which the second, one CTA among the candidates of all chunks, took the most time.
constexpr int kBins = 512;
constexpr int kBinsLog2 = 9;
constexpr int kHeldPerThread = 8;
constexpr int kListKeys = 4096;  // keys that can be collected
constexpr int kMaxCluster = 16;
constexpr int kTokensPerCta = 4096;
constexpr int kFewTokens = 128;  // up to so many keys are ordered by comparing all with all (7.2 us a call; with 500 keys 17.5 against 8.9)
// Comparisons, per CTA and key of the padded list, from which on sorting the list is the shorter way: a CTA compares some
// 20,000 pairs a us. (512 keys in groups of 64 / 128 / 256 equal scores, one CTA: 1.6 / 3.2 / 6.0 us compared.)
constexpr uint32_t kComparisonsPerKey = 100;
// What SortKeys makes of a list of so many keys: a power of two, four keys to each thread of a warp at least.
__device__ __forceinline__ uint32_t PaddedKeys(uint32_t keys) {
  return keys <= 128 ? 128u : 1u << (32 - __clz(static_cast<int>(keys - 1)));
}

struct SelectParams {
  const float* scores;
  int64_t score_stride;
  const int32_t* kv_len;
  int32_t k;
  int32_t* index;       // [batch][k]
  int32_t* n_selected;  // [batch]
  const int32_t* block_table;
  int64_t max_blocks;
  int32_t block_size;
  int64_t pool_rows;
  int32_t* rows_out;    // [batch][k] or null
  int32_t cluster_log2; // of the CTAs that take a sequence
  int32_t* status;
};

struct SelectShared {
  alignas(16) uint64_t all[kListKeys];      // the list: the keys up to the bound, bin after bin; filled where this CTA's entries' bins lie
  alignas(16) uint64_t scratch[kListKeys];  // this CTA's keys on their way to the lists; the sort's other buffer
  uint16_t place[kListKeys];    // ... and where they go
  alignas(16) uint32_t hist[2][kBins];  // by parity of the pass: the peers read one while the next is cleared
  alignas(16) uint32_t peers[kMaxCluster][kBins];
  uint32_t start[kBins + 1];  // place of a bin's first key in the list
  uint32_t next[kBins + 1];   // place of this CTA's next key of a bin; entry kBins: of the keys below the last range
  uint32_t n_mine;
  uint32_t lo[kMaxCluster], hi[kMaxCluster];  // smallest and largest image of each CTA
  uint32_t below[kMaxCluster];                // each CTA's keys below the last range
  uint32_t warp_a[32], warp_b[32];
  uint32_t chosen[3];  // bin, keys in the bins before it, keys in it
};

// Bitonic sort, ascending, of 4 * threads keys (threads a power of two, 32 .. 1024; the block's first ones): thread t has
// keys 4 t .. 4 t + 3 in registers. Partners one or two away sit in the same thread, up to 64 away in the same warp; the
// others are exchanged through the two buffers in turn, one barrier a step. A step costs its latencies and, above all, its
// branches, so it has none: 512 / 1,024 / 2,048 keys take 2.3 / 4.2 / 7.2 us (branches on the two sides of an exchange: 6 /
// 11 / 24 us).
__device__ void SortKeys(uint64_t* data, uint64_t* other, int threads) {
  const int tid = threadIdx.x;
  uint64_t key[4];
  auto read = [&](const uint64_t* from, int thread, uint64_t (&to)[4]) {
    const ulonglong2 a = reinterpret_cast<const ulonglong2*>(from)[2 * thread], b = reinterpret_cast<const ulonglong2*>(from)[2 * thread + 1];
    to[0] = a.x, to[1] = a.y, to[2] = b.x, to[3] = b.y;
  };
  auto write = [&](uint64_t* to) {
    reinterpret_cast<ulonglong2*>(to)[2 * tid] = make_ulonglong2(key[0], key[1]);
    reinterpret_cast<ulonglong2*>(to)[2 * tid + 1] = make_ulonglong2(key[2], key[3]);
  };
  auto order_pair = [&](uint64_t& a, uint64_t& b, bool up) {  // a before b, or the other way round
    const uint64_t x = a, y = b;
    const bool swap = (x > y) == up;
    a = swap ? y : x;
    b = swap ? x : y;
  };
  auto meet = [&](const uint64_t (&theirs)[4], bool smaller) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool take = (theirs[j] < key[j]) == smaller;  // (no branches: they diverge)
      key[j] = take ? theirs[j] : key[j];
    }
  };
  read(data, tid, key);
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  order_pair(key[0], key[1], true);
  order_pair(key[2], key[3], false);
  uint64_t* buffer = data;
  for (int size = 1; size <= threads; size <<= 1) {  // in threads: runs of 4 * size keys
    const bool up = (tid & size) == 0;
    int stride = size >> 1;  // in threads
    for (; stride >= 32; stride >>= 1) {
      write(buffer);
      asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
      uint64_t theirs[4];
      read(buffer, tid ^ stride, theirs);
      meet(theirs, ((tid & stride) == 0) == up);
      buffer = buffer == data ? other : data;
    }
    for (; stride > 0; stride >>= 1) {
      uint64_t theirs[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) theirs[j] = __shfl_xor_sync(0xffffffffu, key[j], stride);
      meet(theirs, ((tid & stride) == 0) == up);
    }
    order_pair(key[0], key[2], up);
    order_pair(key[1], key[3], up);
    order_pair(key[0], key[1], up);
    order_pair(key[2], key[3], up);
  }
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  write(data);
}

__global__ void __launch_bounds__(kSortThreads) IndexerSelectKernel(SelectParams p) {
  extern __shared__ __align__(16) unsigned char select_smem[];
  SelectShared& sh = *reinterpret_cast<SelectShared*>(select_smem);
  GridDependencyTrigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cluster_log2 = p.cluster_log2, cluster = 1 << cluster_log2;
  const int rank = blockIdx.x & (cluster - 1), b = blockIdx.x >> cluster_log2;
  auto cluster_sync = [&]() {
    if (cluster > 1) {
      __syncwarp();
      ptx::ClusterArrive();
      ptx::ClusterWait();
    } else {
      __syncthreads();
    }
  };
  static_assert(2 * kBins <= kSortThreads, "one thread clears one bin");
  if (tid < 2 * kBins) sh.hist[tid / kBins][tid % kBins] = 0;
  if (tid == 0) sh.n_mine = 0;
  if (cluster > 1) {
    __syncwarp();
    ptx::ClusterArrive();  // (waited for before the first exchange: the peers have started)
  }
  GridDependencyWait();
  const int len = max(p.kv_len[b], 0);
  const int k = p.k;
  const int kept = min(len, k);
  if (rank == 0) {
    if (tid == 0) p.n_selected[b] = kept;
    for (int i = kept + tid; i < k; i += kSortThreads) {
      p.index[b * k + i] = -1;
      if (p.rows_out != nullptr) p.rows_out[b * k + i] = -1;
    }
  }
  if (kept == 0) {  // all CTAs of the cluster
    if (cluster > 1) ptx::ClusterWait();
    return;
  }
  auto write = [&](uint64_t key, int place) {
    const int32_t t = static_cast<int32_t>(key & 0xffffffffu);
    p.index[b * k + place] = t;
    if (p.rows_out != nullptr) {  // the selection as pool rows, what ResolveRowsKernel would make of it
      const int64_t column = t / p.block_size;
      const int64_t block = column < p.max_blocks ? p.block_table[static_cast<int64_t>(b) * p.max_blocks + column] : -1;
      const int64_t r = block * p.block_size + t % p.block_size;
      int32_t out_row = -1;
      if (block < 0 || r >= p.pool_rows) {
        RecordError(p.status, B200KV_DEV_BAD_BLOCK, b, place, t);
      } else {
        out_row = static_cast<int32_t>(r);
      }
      p.rows_out[b * k + place] = out_row;
    }
  };
  // Entries entry_lo .. entry_hi of the list, several neighbouring threads to each: a key's place is its bin's start plus the
  // smaller keys of the bin.
  auto order = [&](int entry_lo, int entry_hi, auto&& bin_of) {
    int team_log2 = 0;
    while (team_log2 < 5 && (entry_hi - entry_lo) << (team_log2 + 1) <= kSortThreads) ++team_log2;
    const int member = tid & ((1 << team_log2) - 1);
    for (int e0 = entry_lo; e0 < entry_hi; e0 += kSortThreads >> team_log2) {  // the same trip count for all threads
      const int entry = e0 + (tid >> team_log2);
      const bool live = entry < entry_hi;
      uint64_t key = 0;
      uint2 bin = make_uint2(0u, 0u);
      if (live) {
        key = sh.all[entry];
        bin = bin_of(static_cast<uint32_t>(key >> 32), static_cast<uint32_t>(key));
      }
      int place = 0;
#pragma unroll 4
      for (uint32_t i = bin.x + member; i < bin.y; i += 1u << team_log2) place += sh.all[i] < key ? 1 : 0;
      for (int off = 1; off < 1 << team_log2; off <<= 1) place += __shfl_xor_sync(0xffffffffu, place, off);
      place += static_cast<int>(bin.x);
      if (live && member == 0 && place < kept) write(key, place);
    }
  };
  if (len <= kFewTokens) {  // one bin: what the histograms would spare is less than they cost
    if (cluster > 1) ptx::ClusterWait();
    if (rank != 0) return;
    for (int e = tid; e < len; e += kSortThreads) sh.all[e] = SortKey(p.scores[b * p.score_stride + e], static_cast<uint32_t>(e));
    __syncthreads();
    order(0, len, [&](uint32_t, uint32_t) { return make_uint2(0u, static_cast<uint32_t>(len)); });
    return;
  }
  const int per = (len + cluster - 1) >> cluster_log2;
  const int first = min(rank * per, len);
  const int n = min(per, len - first);
  const float* row = p.scores + b * p.score_stride + first;
  // The high word of the key (ascending = better) of this thread's elements tid, tid + 1024, ..., the first eight held.
  uint32_t held[kHeldPerThread];
#pragma unroll
  for (int j = 0; j < kHeldPerThread; ++j) {
    const int e = tid + j * kSortThreads;
    held[j] = e < n ? static_cast<uint32_t>(SortKey(row[e], 0u) >> 32) : 0u;
  }
  auto for_each = [&](auto&& body) {  // image and position of every element of this thread
#pragma unroll
    for (int j = 0; j < kHeldPerThread; ++j) {
      if (j * kSortThreads >= n) break;
      const int e = tid + j * kSortThreads;
      if (e < n) body(held[j], static_cast<uint32_t>(first + e));
    }
    for (int e = tid + kHeldPerThread * kSortThreads; e < n; e += kSortThreads) {
      body(static_cast<uint32_t>(SortKey(row[e], 0u) >> 32), static_cast<uint32_t>(first + e));
    }
  };

  uint32_t img_lo = ~0u, img_hi = 0u;
  for_each([&](uint32_t image, uint32_t) {
    img_lo = min(img_lo, image);
    img_hi = max(img_hi, image);
  });
  img_lo = __reduce_min_sync(0xffffffffu, img_lo);
  img_hi = __reduce_max_sync(0xffffffffu, img_hi);
  if (lane == 0) {
    sh.warp_a[warp] = img_lo;
    sh.warp_b[warp] = img_hi;
  }
  __syncthreads();
  if (cluster > 1) ptx::ClusterWait();
  if (warp == 0) {
    img_lo = __reduce_min_sync(0xffffffffu, sh.warp_a[lane]);
    img_hi = __reduce_max_sync(0xffffffffu, sh.warp_b[lane]);
    if (lane < cluster) {
      ptx::StClusterB32(ptx::MapToRank(ptx::SmemAddr(&sh.lo[rank]), lane), img_lo);
      ptx::StClusterB32(ptx::MapToRank(ptx::SmemAddr(&sh.hi[rank]), lane), img_hi);
    }
  }
  cluster_sync();
  img_lo = __reduce_min_sync(0xffffffffu, sh.lo[lane & (cluster - 1)]);
  img_hi = __reduce_max_sync(0xffffffffu, sh.hi[lane & (cluster - 1)]);
  if (img_lo == img_hi) {  // all scores equal: the first positions, in order
    for (int i = rank * kSortThreads + tid; i < kept; i += kSortThreads << cluster_log2) write(static_cast<uint64_t>(i), i);
    return;
  }

  // The wanted key is the `rank_left`-th of those with a value in [lo, hi]; all `taken` keys below are wanted, `run` of
  // them those of CTA number `warp`. The value is the image or, when there are too many keys of one image, the position
  // of those that have it.
  uint32_t lo = img_lo, hi = img_hi, tied = 0;
  bool by_position = false;
  uint32_t bound;
  auto value_of = [&](uint32_t image, uint32_t position) { return by_position ? position : image; };
  auto below = [&](uint32_t image, uint32_t position) {  // wanted whatever the last range's bins say
    return by_position ? image < tied || (image == tied && position < lo) : image < lo;
  };
  auto up_to_bound = [&](uint32_t image, uint32_t position) {
    return by_position ? image < tied || (image == tied && position <= bound) : image <= bound;
  };
  uint32_t rank_left = static_cast<uint32_t>(kept), taken = 0, run = 0, total;
  int shift;
  bool dense;  // bins so full that sorting is the shorter way
  const uint32_t enough = static_cast<uint32_t>(min(kListKeys, k + max(k >> 1, 128)));
  for (int pass = 0;; ++pass) {
    const uint32_t span = hi - lo;
    shift = max(0, 32 - kBinsLog2 - __clz(static_cast<int>(span)));
    uint32_t* hist = sh.hist[pass & 1];
    if (!by_position) {
      for_each([&](uint32_t image, uint32_t) {
        if (image - lo <= span) atomicAdd(&hist[(image - lo) >> shift], 1u);
      });
    } else {
      for_each([&](uint32_t image, uint32_t position) {
        if (image == tied && position - lo <= span) atomicAdd(&hist[(position - lo) >> shift], 1u);
      });
    }
    cluster_sync();
    if (warp < cluster) {  // the bins of CTA `warp`, four at a time
      const uint32_t src = ptx::MapToRank(ptx::SmemAddr(hist), warp) + lane * 16;
      uint32_t v[kBins / 128][4];
#pragma unroll
      for (int q = 0; q < kBins / 128; ++q) ptx::LdClusterV4(src + q * 512, v[q][0], v[q][1], v[q][2], v[q][3]);
#pragma unroll
      for (int q = 0; q < kBins / 128; ++q) reinterpret_cast<uint4*>(sh.peers[warp])[32 * q + lane] = make_uint4(v[q][0], v[q][1], v[q][2], v[q][3]);
      if (lane == 0) sh.below[warp] = run;
    }
    if (pass > 0 && tid < kBins) sh.hist[(pass + 1) & 1][tid] = 0;  // (the peers are done with it: they have passed the barrier)
    __syncthreads();
    uint32_t mine = 0, earlier = 0, incl = 0;  // of bin `tid`: all keys, those of the CTAs before this one
    if (tid < kBins) {
      for (int c = 0; c < cluster; ++c) {
        const uint32_t v = sh.peers[c][tid];
        mine += v;
        earlier += c < rank ? v : 0u;
      }
      incl = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += up;
      }
      if (lane == 31) sh.warp_a[warp] = incl;
    }
    __syncthreads();
    if (tid < kBins) {
      uint32_t before = incl - mine;
      for (int w = 0; w < warp; ++w) before += sh.warp_a[w];
      if (tid == 0) sh.start[0] = taken;
      sh.start[tid + 1] = taken + before + mine;
      sh.next[tid] = taken + before + earlier;
      if (before < rank_left && rank_left <= before + mine) {  // one thread
        sh.chosen[0] = tid;
        sh.chosen[1] = before;
        sh.chosen[2] = mine;
      }
      // The comparisons that ordering bin by bin would take: a bin's size squared. (Whatever lies beyond the chosen bin
      // counts as nothing: it starts at or after the wanted rank.)
      const uint32_t squares = __reduce_add_sync(0xffffffffu, before < rank_left ? mine * min(mine, 8192u) : 0u);
      if (lane == 0) sh.warp_b[warp] = squares;
    }
    __syncthreads();
    const uint32_t bin = sh.chosen[0], before = sh.chosen[1], in_bin = sh.chosen[2];
    const uint32_t offset = (bin << shift) | ((1u << shift) - 1);
    bound = offset >= span ? hi : lo + offset;
    total = taken + before + in_bin;
    if (total <= enough) {  // (a bin of one position holds one key: the passes end)
      uint32_t squares = taken * taken;
      for (int w = 0; w < kBins / 32; ++w) squares += sh.warp_b[w];
      dense = squares > (kComparisonsPerKey * PaddedKeys(total)) << cluster_log2;
      if (!dense || total <= kMaxK) break;  // (a pass more, 2.5 us, is shorter than sorting 4,096 keys instead of 2,048)
    }
    if (warp < cluster) {
      uint32_t sum = 0;
      for (uint32_t t = lane; t < bin; t += 32) sum += sh.peers[warp][t];
      run += __reduce_add_sync(0xffffffffu, sum);
    }
    taken += before;
    rank_left -= before;
    lo += bin << shift;
    hi = bound;
    if (shift == 0) {  // too many keys of one image
      by_position = true;
      tied = lo;
      lo = 0;
      hi = static_cast<uint32_t>(len) - 1;
    }
  }
  if (tid == 0) {
    uint32_t at = 0;
    for (int c = 0; c < rank; ++c) at += sh.below[c];
    sh.next[kBins] = at;
  }
  __syncthreads();

  auto bin_of = [&](uint32_t image, uint32_t position) {  // a key's bin in the list: its first entry and the one after its last
    if (below(image, position)) return make_uint2(0u, taken);
    const uint32_t bin = (value_of(image, position) - lo) >> shift;
    return make_uint2(sh.start[bin], sh.start[bin + 1]);
  };
  for_each([&](uint32_t image, uint32_t position) {
    if (!up_to_bound(image, position)) return;
    const uint32_t bin = below(image, position) ? static_cast<uint32_t>(kBins) : (value_of(image, position) - lo) >> shift;
    const uint32_t at = atomicAdd(&sh.next[bin], 1u);
    const uint64_t key = (static_cast<uint64_t>(image) << 32) | position;
    if (cluster == 1) {
      sh.all[at] = key;
    } else {  // written to the lists below, where the stores are shared out
      const uint32_t i = atomicAdd(&sh.n_mine, 1u);
      sh.scratch[i] = key;
      sh.place[i] = static_cast<uint16_t>(at);
    }
  });
  if (cluster > 1) {
    __syncthreads();
    // A key goes to the CTAs whose entries of the list its bin overlaps (to the one that sorts, if sorting it is).
    const int items = static_cast<int>(sh.n_mine) << cluster_log2;
    for (int item = tid; item < items; item += kSortThreads) {
      const int i = item >> cluster_log2, c = item & (cluster - 1);
      const uint64_t key = sh.scratch[i];
      const uint2 bin = bin_of(static_cast<uint32_t>(key >> 32), static_cast<uint32_t>(key));
      const bool theirs = dense ? c == 0 : (total * c) >> cluster_log2 < bin.y && (total * (c + 1)) >> cluster_log2 > bin.x;
      if (theirs) ptx::StClusterB64(ptx::MapToRank(ptx::SmemAddr(&sh.all[sh.place[i]]), c), key);
    }
  }
  cluster_sync();

  const int keys = static_cast<int>(total);
  if (!dense) {
    order((keys * rank) >> cluster_log2, (keys * (rank + 1)) >> cluster_log2, bin_of);
    return;
  }
  if (rank != 0) return;
  const int padded = static_cast<int>(PaddedKeys(total));
  for (int i = keys + tid; i < padded; i += kSortThreads) sh.all[i] = ~0ull;
  __syncthreads();
  if (tid < padded / 4) SortKeys(sh.all, sh.scratch, padded / 4);
  __syncthreads();
  for (int i = tid; i < kept; i += kSortThreads) write(sh.all[i], i);
}

int32_t LaunchSelect(SelectParams p, int32_t batch, int64_t max_kv_len, cudaStream_t stream) {
  // How many clusters of 1, 2, 4, 8, 16 CTAs a device holds at once; looked up once per thread and device (a device number
  // beyond the table whenever it comes after another).
  constexpr int kKnownDevices = 16;
  struct Limits {
    int device = -1;
    int32_t most[5] = {};
  };
  static thread_local Limits known[kKnownDevices];
  int device = 0;
  if (int32_t rc = CheckCuda(cudaGetDevice(&device), "cudaGetDevice")) return rc;
  Limits& limits = known[device % kKnownDevices];
  cudaLaunchConfig_t config = {};
  config.blockDim = dim3(kSortThreads);
  config.dynamicSmemBytes = sizeof(SelectShared);
  config.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attrs;
  if (device != limits.device) {
    if (int32_t rc = CheckCuda(cudaFuncSetAttribute(IndexerSelectKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(sizeof(SelectShared))), "indexer top-k smem opt-in")) return rc;
    if (int32_t rc = CheckCuda(cudaFuncSetAttribute(IndexerSelectKernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "indexer top-k cluster opt-in")) return rc;
    for (int i = 0; i < 5; ++i) {
      attrs[0].val.clusterDim.x = 1u << i;
      config.gridDim = dim3(1u << i);
      config.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, IndexerSelectKernel, &config) != cudaSuccess) {
        cudaGetLastError();  // a size the device does not offer
        clusters = 0;
      }
      limits.most[i] = clusters;
    }
    limits.device = device;
  }
  int size = 0;
  while (size < 4 && max_kv_len > static_cast<int64_t>(kTokensPerCta) << size) ++size;
  while (size > 0 && batch > limits.most[size]) --size;
  p.cluster_log2 = size;
  attrs[0].val.clusterDim.x = 1u << size;
  config.gridDim = dim3(static_cast<unsigned>(batch) << size);  // (in x, which has room for any batch)
  config.numAttrs = 2;
  return CheckCuda(cudaLaunchKernelEx(&config, IndexerSelectKernel, p), "indexer top-k launch");
}

}  // namespace
}  // namespace b200kv

namespace b200kv {
bool IndexerTcSupports(int32_t heads, int32_t block_size, int64_t key_stride, int64_t pool_rows);
int32_t LaunchIndexerScoreTc(const void* q, const float* q_scale, const void* weights, int32_t heads, const void* key_pool,
                             int64_t key_stride, const float* k_scale, int64_t pool_rows, const int32_t* block_table,
                             int64_t max_blocks, const int32_t* kv_len, int32_t batch, int32_t block_size, int64_t max_kv_len,
                             float* scores, int64_t score_stride, cudaStream_t stream, int32_t* status);
}  // namespace b200kv

using namespace b200kv;

namespace {
// Scores [batch][stride] fp32. Sequences of more than 8,192 tokens have always asked for room for 2,048 keys a chunk of
// that length behind the scores; the selection no longer needs it, callers' plans are sized by it.
constexpr int64_t kPlanChunk = 8192;
int64_t ScoreStrideOf(int64_t max_kv_len) { return (max_kv_len + 3) & ~3ll; }
int64_t ChunksOf(int64_t max_kv_len) { return (max_kv_len + kPlanChunk - 1) / kPlanChunk; }
size_t ScoreBytesOf(int32_t batch, int64_t max_kv_len) {
  return (static_cast<size_t>(batch) * static_cast<size_t>(ScoreStrideOf(max_kv_len)) * sizeof(float) + 15) & ~static_cast<size_t>(15);
}
}  // namespace

extern "C" size_t b200kv_indexer_workspace_bytes(int32_t batch, int64_t max_kv_len) {
  if (batch <= 0 || max_kv_len <= 0) return 0;
  const int64_t chunks = ChunksOf(max_kv_len);
  return ScoreBytesOf(batch, max_kv_len) +
         (chunks > 1 ? static_cast<size_t>(batch) * static_cast<size_t>(chunks) * kMaxK * sizeof(uint64_t) : 0);
}

extern "C" int32_t b200kv_indexer_topk(const b200kv_indexer_args* args, void* stream, b200kv_status_word* status) {
  if (int32_t rc = FaultCheck("b200kv_indexer_topk")) return rc;
  if (args == nullptr) {
    SetLastError("indexer_topk: args is null");
    return B200KV_ERR_NULLPTR;
  }
  const b200kv_indexer_args& a = *args;
  if (a.batch == 0) return B200KV_OK;
  if (a.q == nullptr || a.q_scale == nullptr || a.weights == nullptr || a.key_pool == nullptr || a.k_scale == nullptr ||
      a.block_table == nullptr || a.kv_len == nullptr || a.index_out == nullptr || a.n_selected_out == nullptr ||
      a.workspace == nullptr) {
    SetLastError("indexer_topk: q, q_scale, weights, key_pool, k_scale, block_table, kv_len, outputs and workspace must "
                 "be non-null");
    return B200KV_ERR_NULLPTR;
  }
  if (a.batch < 0 || a.heads < 1 || a.heads > kMaxIndexHeads || a.k < 1 || a.k > kMaxK || a.block_size <= 0 ||
      a.max_blocks <= 0 || a.max_kv_len <= 0 || a.pool_rows <= 0 || a.key_stride < kIndexDim || a.key_stride % 16 != 0 ||
      (reinterpret_cast<uintptr_t>(a.key_pool) & 15u) != 0 ||
      a.workspace_bytes < b200kv_indexer_workspace_bytes(a.batch, a.max_kv_len)) {
    SetLastError("indexer_topk refused: batch %d, heads %d (1..%d), k %d (1..%d), block_size %d, max_kv_len %lld, key stride "
                 "%lld (>= 128, multiple of 16, 16-byte aligned pool), workspace %zu of %zu bytes",
                 a.batch, a.heads, kMaxIndexHeads, a.k, kMaxK, a.block_size, static_cast<long long>(a.max_kv_len),
                 static_cast<long long>(a.key_stride), a.workspace_bytes,
                 b200kv_indexer_workspace_bytes(a.batch, a.max_kv_len));
    return B200KV_ERR_INVALID;
  }
  const bool tc_ok = IndexerTcSupports(a.heads, a.block_size, a.key_stride, a.pool_rows) &&
                     (reinterpret_cast<uintptr_t>(a.q) & 15u) == 0;  // its TMA loads want a 16-byte aligned query
  if ((a.variant != B200KV_INDEXER_AUTO && a.variant != B200KV_INDEXER_EXACT && a.variant != B200KV_INDEXER_TCGEN05) ||
      (a.variant == B200KV_INDEXER_TCGEN05 && !tc_ok)) {
    SetLastError("indexer_topk refused: variant %d (the tensor-core score kernel needs heads <= 64, block_size %% 64 == 0 and a "
                 "16-byte aligned q; heads %d, block_size %d)", a.variant, a.heads, a.block_size);
    return B200KV_ERR_INVALID;
  }
  const bool use_tc = tc_ok && a.variant != B200KV_INDEXER_EXACT;
  ScoreParams p{};
  p.q = static_cast<const uint8_t*>(a.q);
  p.q_scale = a.q_scale;
  p.w = static_cast<const __nv_bfloat16*>(a.weights);
  p.heads = a.heads;
  p.key_pool = static_cast<const uint8_t*>(a.key_pool);
  p.key_stride = a.key_stride;
  p.k_scale = a.k_scale;
  p.pool_rows = a.pool_rows;
  p.block_table = a.block_table;
  p.max_blocks = a.max_blocks;
  p.kv_len = a.kv_len;
  p.block_size = a.block_size;
  p.scores = static_cast<float*>(a.workspace);
  p.score_stride = ScoreStrideOf(a.max_kv_len);
  p.status = status;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (use_tc) {
    if (int32_t rc = LaunchIndexerScoreTc(a.q, a.q_scale, a.weights, a.heads, a.key_pool, a.key_stride, a.k_scale, a.pool_rows,
                                          a.block_table, a.max_blocks, a.kv_len, a.batch, a.block_size, a.max_kv_len, p.scores,
                                          p.score_stride, s, status)) {
      return rc;
    }
  } else {
    const dim3 grid(static_cast<unsigned>((a.max_kv_len + kScoreThreads - 1) / kScoreThreads), static_cast<unsigned>(a.batch));
    if (int32_t rc = CheckCuda(LaunchOverlapped(IndexerScoreKernel, grid, dim3(kScoreThreads), 0, s, p), "indexer score launch")) {
      return rc;
    }
  }
  SelectParams sp{};
  sp.scores = p.scores;
  sp.score_stride = p.score_stride;
  sp.kv_len = a.kv_len;
  sp.k = a.k;
  sp.index = a.index_out;
  sp.n_selected = a.n_selected_out;
  sp.block_table = a.block_table;
  sp.max_blocks = a.max_blocks;
  sp.block_size = a.block_size;
  sp.pool_rows = a.pool_rows;
  sp.rows_out = a.rows_out;
  sp.status = static_cast<int32_t*>(status);
  return LaunchSelect(sp, a.batch, a.max_kv_len, s);
}
