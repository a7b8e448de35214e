// The stages on either side of the KV path, as kernels of their own:
//
//   producer  RMSNorm of the appended row's 512-wide latent, rotary embedding ("half" pairing) of its
//             64-wide rope slice, and the write of both into the paged pool, in ONE kernel, so the
//             normalised row never makes a round trip through an activation buffer; the same launch
//             rotates the query's rope slices in place (the reference runs these as three operators,
//             stages 6-8 of src/pipeline/pipeline.cpp:212-234).
//   consumer  block-32 MX quantisation of the attention output to FP8 E4M3 with E8M0 scales (stage 10,
//             src/pipeline/pipeline.cpp:250-258).
//
// All three are memory-bound element-wise work: one warp per row or vector, 16-byte accesses. Their
// arithmetic is fixed to the operation (explicit round-to-nearest intrinsics, a fixed reduction order),
// so that results are bit-identical with the CPU statement of the same rules:
//   RMSNorm: lane L sums fma(x, x, a) over elements 8L..8L+7 then 256+8L..256+8L+7; butterfly over
//            xor 16, 8, 4, 2, 1; r = 1 / sqrt(a/512 + eps); y = bf16((x * r) * g).
//   RoPE:    y_i = bf16(fma(-x_(i+32), s_i, x_i * c_i)); y_(i+32) = bf16(fma(x_i, s_(i+32), x_(i+32) * c_(i+32))).
//   MX:      e = floor(log2 max|x|) - 8 clamped to [-127, 127] (all zero: -127); scale byte e + 127;
//            q = e4m3(x * 2^-e), nearest even, saturating; a NaN in the block makes scale and values NaN.
#include <cuda_fp8.h>

#include "common.cuh"

namespace b200kv {
namespace {

constexpr int kLatent = B200KV_LATENT_DIM;
constexpr int kRope = B200KV_ROPE_DIM;
static_assert(kLatent == 512 && kRope == 64, "the lane assignment below is written for 512 + 64");
constexpr int kWarpsPerCta = 8;

struct ProducerParams {
  b200kv_pool_view pool;
  const __nv_bfloat16* kv_a;
  int64_t kv_a_stride;
  const __nv_bfloat16* gamma;
  float eps;
  const __nv_bfloat16* cos;
  int64_t cos_stride;
  const __nv_bfloat16* sin;
  int64_t sin_stride;
  const int32_t* slots;
  int64_t tokens;
  __nv_bfloat16* q_rope;  // [tokens][heads][64] rotated in place, or null
  int64_t q_token_stride;
  int64_t q_head_stride;
  int32_t heads;
  __nv_bfloat16* latent_out;  // optional copies of what went into the pool (the reference's act buffers)
  int64_t latent_out_stride;
  __nv_bfloat16* rope_out;
  int64_t rope_out_stride;
  float* rstd_out;
  int32_t* status;
};

__device__ __forceinline__ float Bf16Bits(uint32_t packed, int hi) {
  return __uint_as_float(hi ? (packed & 0xffff0000u) : (packed << 16));
}

__device__ __forceinline__ uint32_t PackBf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Rotates eight pairs (i, i + 32) held as two 16-byte chunks: x1 = elements 8j..8j+7, x2 = 32+8j..32+8j+7.
__device__ __forceinline__ void RotateChunks(const int4& x1, const int4& x2, const int4& c1, const int4& c2, const int4& s1,
                                             const int4& s2, int4* y1, int4* y2) {
  const uint32_t a[4] = {static_cast<uint32_t>(x1.x), static_cast<uint32_t>(x1.y), static_cast<uint32_t>(x1.z), static_cast<uint32_t>(x1.w)};
  const uint32_t b[4] = {static_cast<uint32_t>(x2.x), static_cast<uint32_t>(x2.y), static_cast<uint32_t>(x2.z), static_cast<uint32_t>(x2.w)};
  const uint32_t ca[4] = {static_cast<uint32_t>(c1.x), static_cast<uint32_t>(c1.y), static_cast<uint32_t>(c1.z), static_cast<uint32_t>(c1.w)};
  const uint32_t cb[4] = {static_cast<uint32_t>(c2.x), static_cast<uint32_t>(c2.y), static_cast<uint32_t>(c2.z), static_cast<uint32_t>(c2.w)};
  const uint32_t sa[4] = {static_cast<uint32_t>(s1.x), static_cast<uint32_t>(s1.y), static_cast<uint32_t>(s1.z), static_cast<uint32_t>(s1.w)};
  const uint32_t sb[4] = {static_cast<uint32_t>(s2.x), static_cast<uint32_t>(s2.y), static_cast<uint32_t>(s2.z), static_cast<uint32_t>(s2.w)};
  uint32_t ya[4], yb[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    float lo[2], hi[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float x_lo = Bf16Bits(a[w], h), x_hi = Bf16Bits(b[w], h);
      lo[h] = __fmaf_rn(-x_hi, Bf16Bits(sa[w], h), __fmul_rn(x_lo, Bf16Bits(ca[w], h)));
      hi[h] = __fmaf_rn(x_lo, Bf16Bits(sb[w], h), __fmul_rn(x_hi, Bf16Bits(cb[w], h)));
    }
    ya[w] = PackBf16(lo[0], lo[1]);
    yb[w] = PackBf16(hi[0], hi[1]);
  }
  *y1 = make_int4(ya[0], ya[1], ya[2], ya[3]);
  *y2 = make_int4(yb[0], yb[1], yb[2], yb[3]);
}

// The same for two pairs, (i, i + 32) and (i + 1, i + 33), held as one word each.
__device__ __forceinline__ void RotateWord(uint32_t x1, uint32_t x2, uint32_t c1, uint32_t c2, uint32_t s1, uint32_t s2,
                                           uint32_t* y1, uint32_t* y2) {
  float lo[2], hi[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float x_lo = Bf16Bits(x1, h), x_hi = Bf16Bits(x2, h);
    lo[h] = __fmaf_rn(-x_hi, Bf16Bits(s1, h), __fmul_rn(x_lo, Bf16Bits(c1, h)));
    hi[h] = __fmaf_rn(x_lo, Bf16Bits(s2, h), __fmul_rn(x_hi, Bf16Bits(c2, h)));
  }
  *y1 = PackBf16(lo[0], lo[1]);
  *y2 = PackBf16(hi[0], hi[1]);
}

__device__ __forceinline__ uint32_t LoadWord(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }
__device__ __forceinline__ void StoreWord(__nv_bfloat16* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }
__device__ __forceinline__ int4 LoadChunk(const __nv_bfloat16* p) { return *reinterpret_cast<const int4*>(p); }
__device__ __forceinline__ void StoreChunk(__nv_bfloat16* p, const int4& v) { *reinterpret_cast<int4*>(p) = v; }

constexpr int kRowsPerPass = 2;  // rows a warp has in flight, a half-warp each where a row's work is scalar

// Two fp32 values in one 64-bit register, for the packed multiplication (each half rounded to nearest on its own).
__device__ __forceinline__ uint64_t Pair(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ uint64_t MulPair(uint64_t a, uint64_t b) {
  uint64_t v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ uint32_t PackPair(uint64_t v) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return PackBf16(lo, hi);
}

// Vectors (query rope slices, [tokens][heads][64], in place): four lanes a vector, kRounds times eight of them in flight.
template <int kRounds>
__device__ __forceinline__ void RotateVectors(const ProducerParams& p, int64_t first_vector, int64_t vectors) {
  const int lane = threadIdx.x & 31;
  const int64_t first = first_vector + (lane >> 2);
  const int j = 8 * (lane & 3);
  __nv_bfloat16* x[kRounds];
  int64_t token[kRounds];
  int4 x1[kRounds], x2[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const int64_t v = first + 8 * k;
    x[k] = nullptr;
    if (v >= vectors) continue;
    token[k] = v / p.heads;
    x[k] = p.q_rope + token[k] * p.q_token_stride + (v - token[k] * p.heads) * p.q_head_stride + j;
    x1[k] = LoadChunk(x[k]);
    x2[k] = LoadChunk(x[k] + 32);
  }
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    if (x[k] == nullptr) continue;
    const __nv_bfloat16* c = p.cos + token[k] * p.cos_stride + j;
    const __nv_bfloat16* s = p.sin + token[k] * p.sin_stride + j;
    int4 y1, y2;
    RotateChunks(x1[k], x2[k], LoadChunk(c), LoadChunk(c + 32), LoadChunk(s), LoadChunk(s + 32), &y1, &y2);
    StoreChunk(x[k], y1);
    StoreChunk(x[k] + 32, y2);
  }
}

// Vectors alone, and those of large calls: 60 registers, so 32 warps an SM, and two rounds in flight once every warp has
// that many. us for 32 / 1,024 / 16,384 tokens x 64 heads: 1.9 / 5.4 / 50.5 in the rows' kernel, 1.7 / 3.7 / 45.4 so.
template <int kRounds>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) RotateKernel(ProducerParams p) {
  GridDependencyTrigger();
  GridDependencyWait();
  const int64_t vectors = p.tokens * p.heads;
  const int64_t step = ((static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5) * (8 * kRounds);
  for (int64_t v = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * (8 * kRounds); v < vectors; v += step) {
    RotateVectors<kRounds>(p, v, vectors);
  }
}

// The rows' part is bound by instruction issue before it is bound by HBM, so the instructions are counted: a row's values
// are unpacked once and kept, the two multiplications of a pair of values are packed ones, the square root and the
// division of both rows run at once in the warp's two halves, and a rope slice is rotated by sixteen lanes, a word each
// (four lanes with 16-byte chunks left the warp's other lanes idle for 120 instructions). That takes 128 registers and so
// two CTAs an SM, whose warps therefore read a pass ahead; the grid is what is resident, each warp walking its passes.
// us for 16,384 / 49,157 / 131,072 rows: 11.3 / 28.4 / 68.2 before (4.9 TB/s), 10.9 / 26.2 / 63.1 without reading ahead,
// 12.1 / 24.4 / 57.5 with eight CTAs an SM in the grid, 8.5 / 22.9 / 55.9 (6.0 TB/s) so.
constexpr int kResidentCtas = 2;
// kVectors: the launch also rotates the query's vectors, so many times eight a pass (calls of up to some thousand tokens).
template <int kVectors>
__global__ void __launch_bounds__(kWarpsPerCta * 32, kResidentCtas) ProducerKernel(ProducerParams p) {
  GridDependencyTrigger();
  GridDependencyWait();
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t rows = p.tokens;
  const int64_t row_items = (rows + kRowsPerPass - 1) / kRowsPerPass;
  constexpr int kItemVectors = kVectors > 0 ? 8 * kVectors : 8;
  const int64_t vectors = kVectors > 0 ? p.tokens * p.heads : 0;
  const int64_t vector_items = (vectors + kItemVectors - 1) / kItemVectors;
  // gamma of this lane's columns 8 lane .. + 7 and 256 + 8 lane .. + 7
  const uint4 ga = *reinterpret_cast<const uint4*>(p.gamma + 8 * lane), gb = *reinterpret_cast<const uint4*>(p.gamma + 256 + 8 * lane);
  const uint32_t gamma[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
  // What a pass reads, read a pass ahead: the two rows' latent halves, then (lanes 0-15 for the first row, 16-31 for the
  // second) the slot and the words of the rope slice and its cos / sin.
  const int half = lane >> 4;
  const int word = 2 * (lane & 15);  // this lane's rope elements word, word + 1 and word + 32, word + 33
  struct {
    int4 xa[kRowsPerPass], xb[kRowsPerPass];
    uint32_t x1, x2, c1, c2, s1, s2;
    int slot;
  } ahead{};
  auto read = [&](int64_t item) {
    const int64_t t0 = item * kRowsPerPass, t = t0 + half;
#pragma unroll
    for (int r = 0; r < kRowsPerPass; ++r) {
      if (t0 + r < rows) {
        const __nv_bfloat16* row = p.kv_a + (t0 + r) * p.kv_a_stride;
        ahead.xa[r] = LoadStream16(row + 8 * lane);
        ahead.xb[r] = LoadStream16(row + 256 + 8 * lane);
      }
    }
    ahead.slot = t < rows && p.slots != nullptr ? p.slots[t] : -1;
    if (p.cos != nullptr && t < rows) {
      const __nv_bfloat16* x = p.kv_a + t * p.kv_a_stride + kLatent + word;
      const __nv_bfloat16* c = p.cos + t * p.cos_stride + word;
      const __nv_bfloat16* s = p.sin + t * p.sin_stride + word;
      ahead.x1 = LoadWord(x);
      ahead.x2 = LoadWord(x + 32);
      ahead.c1 = LoadWord(c);
      ahead.c2 = LoadWord(c + 32);
      ahead.s1 = LoadWord(s);
      ahead.s2 = LoadWord(s + 32);
    }
  };
  if (warp < row_items) read(warp);
  for (int64_t item = warp; item < row_items + vector_items; item += n_warps) {
    if constexpr (kVectors > 0) {
      if (item >= row_items) {
        RotateVectors<kVectors>(p, (item - row_items) * kItemVectors, vectors);
        continue;
      }
    }
    const int64_t t0 = item * kRowsPerPass;
    const int64_t t = t0 + half;  // this half-warp's row
    const bool rotates = p.cos != nullptr && t < rows;
    int4 xa[kRowsPerPass] = {ahead.xa[0], ahead.xa[1]}, xb[kRowsPerPass] = {ahead.xb[0], ahead.xb[1]};
    int slot = ahead.slot;
    const uint32_t x1 = ahead.x1, x2 = ahead.x2, c1 = ahead.c1, c2 = ahead.c2, s1 = ahead.s1, s2 = ahead.s2;
    if (item + n_warps < row_items) read(item + n_warps);
    // The rows' values, in pairs, and the sums of their squares.
    uint64_t x[kRowsPerPass][8];
    float a[kRowsPerPass];
#pragma unroll
    for (int r = 0; r < kRowsPerPass; ++r) {
      const uint32_t w[8] = {static_cast<uint32_t>(xa[r].x), static_cast<uint32_t>(xa[r].y), static_cast<uint32_t>(xa[r].z),
                             static_cast<uint32_t>(xa[r].w), static_cast<uint32_t>(xb[r].x), static_cast<uint32_t>(xb[r].y),
                             static_cast<uint32_t>(xb[r].z), static_cast<uint32_t>(xb[r].w)};
      a[r] = 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float lo = Bf16Bits(w[k], 0), hi = Bf16Bits(w[k], 1);
        a[r] = __fmaf_rn(lo, lo, a[r]);
        a[r] = __fmaf_rn(hi, hi, a[r]);
        x[r][k] = Pair(lo, hi);
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int r = 0; r < kRowsPerPass; ++r) a[r] = __fadd_rn(a[r], __shfl_xor_sync(0xffffffffu, a[r], off));
    }
    const float mine = (lane & 16) ? a[1] : a[0];
    const float rstd = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(mine, 1.0f / 512.0f), p.eps)));
    const bool bad = slot >= p.pool.pool_rows;
    if ((lane & 15) == 0 && t < rows) {
      if (p.rstd_out != nullptr) p.rstd_out[t] = rstd;
      if (bad && p.slots != nullptr) RecordError(p.status, B200KV_DEV_BAD_SLOT, static_cast<int32_t>(t), slot);
    }
    if (bad) slot = -1;
    if (rotates) {
      uint32_t y1, y2;
      RotateWord(x1, x2, c1, c2, s1, s2, &y1, &y2);
      if (slot >= 0) {
        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.pool.rope) + static_cast<int64_t>(slot) * p.pool.rope_row_stride + word;
        StoreWord(dst, y1);
        StoreWord(dst + 32, y2);
      }
      if (p.rope_out != nullptr) {
        __nv_bfloat16* dst = p.rope_out + t * p.rope_out_stride + word;
        StoreWord(dst, y1);
        StoreWord(dst + 32, y2);
      }
    }
    uint32_t y[kRowsPerPass][8];
    {
      const float scale0 = __shfl_sync(0xffffffffu, rstd, 0), scale1 = __shfl_sync(0xffffffffu, rstd, 16);
      const uint64_t scale[kRowsPerPass] = {Pair(scale0, scale0), Pair(scale1, scale1)};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint64_t g = Pair(Bf16Bits(gamma[k], 0), Bf16Bits(gamma[k], 1));
#pragma unroll
        for (int r = 0; r < kRowsPerPass; ++r) y[r][k] = PackPair(MulPair(MulPair(x[r][k], scale[r]), g));
      }
    }
#pragma unroll
    for (int r = 0; r < kRowsPerPass; ++r) {
      const int row_slot = __shfl_sync(0xffffffffu, slot, 16 * r);
      if (t0 + r >= rows) continue;  // warp-uniform
      const int4 ya = make_int4(y[r][0], y[r][1], y[r][2], y[r][3]), yb = make_int4(y[r][4], y[r][5], y[r][6], y[r][7]);
      if (p.latent_out != nullptr) {
        __nv_bfloat16* dst = p.latent_out + (t0 + r) * p.latent_out_stride;
        *reinterpret_cast<int4*>(dst + 8 * lane) = ya;
        *reinterpret_cast<int4*>(dst + 256 + 8 * lane) = yb;
      }
      if (row_slot >= 0) {
        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.pool.latent) + static_cast<int64_t>(row_slot) * p.pool.latent_row_stride;
        StoreStream16(dst + 8 * lane, ya);
        StoreStream16(dst + 256 + 8 * lane, yb);
      }
    }
  }
}

// A warp takes 32 consecutive blocks of a row (2 KB): lane l loads the 16-byte chunks l, l + 32, l + 64 and
// l + 96 of that span, so loads and stores are contiguous across the warp; a block's four chunks sit in four
// neighbouring lanes, which agree on the block's maximum with two shuffles.
__global__ void __launch_bounds__(256)
    MxQuantKernel(const __nv_bfloat16* x, int64_t x_stride, int64_t rows, int64_t blocks_per_row, uint8_t* q,
                  int64_t q_stride, uint8_t* scales, int64_t scale_stride) {
  GridDependencyTrigger();
  GridDependencyWait();
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  const int64_t spans_per_row = (blocks_per_row + 31) / 32;
  for (int64_t item = warp; item < rows * spans_per_row; item += n_warps) {
    const int64_t r = item / spans_per_row, first_block = (item % spans_per_row) * 32;
    const __nv_bfloat16* src = x + r * x_stride + 32 * first_block;
    const int64_t chunks = (blocks_per_row - first_block < 32 ? blocks_per_row - first_block : 32) * 4;
    int4 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = lane + 32 * k;
      v[k] = c < chunks ? LoadStream16(src + 8 * c) : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = lane + 32 * k;
      const uint32_t w[4] = {static_cast<uint32_t>(v[k].x), static_cast<uint32_t>(v[k].y), static_cast<uint32_t>(v[k].z),
                             static_cast<uint32_t>(v[k].w)};
      float amax = 0.0f;
      int nan = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float lo = fabsf(Bf16Bits(w[i], 0)), hi = fabsf(Bf16Bits(w[i], 1));
        nan |= (lo != lo || hi != hi) ? 1 : 0;
        amax = fmaxf(amax, fmaxf(lo, hi));
      }
#pragma unroll
      for (int off = 1; off <= 2; off <<= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        nan |= __shfl_xor_sync(0xffffffffu, nan, off);
      }
      uint32_t out[2];
      const MxScale block = MxScaleOf(amax, nan != 0);
      const uint8_t scale = static_cast<uint8_t>(block.code);
      if (nan) {
        out[0] = (((w[0] >> 8) & 0x80u) | 0x7fu) | ((((w[0] >> 24) & 0x80u) | 0x7fu) << 8) |
                 ((((w[1] >> 8) & 0x80u) | 0x7fu) << 16) | ((((w[1] >> 24) & 0x80u) | 0x7fu) << 24);
        out[1] = (((w[2] >> 8) & 0x80u) | 0x7fu) | ((((w[2] >> 24) & 0x80u) | 0x7fu) << 8) |
                 ((((w[3] >> 8) & 0x80u) | 0x7fu) << 16) | ((((w[3] >> 24) & 0x80u) | 0x7fu) << 24);
      } else {
        const float inv = block.inv;
        uint32_t b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          b[i] = __nv_cvt_float2_to_fp8x2(make_float2(__fmul_rn(Bf16Bits(w[i], 0), inv), __fmul_rn(Bf16Bits(w[i], 1), inv)),
                                          __NV_SATFINITE, __NV_E4M3);
        }
        out[0] = b[0] | (b[1] << 16);
        out[1] = b[2] | (b[3] << 16);
      }
      if (c < chunks) {
        *reinterpret_cast<uint2*>(q + r * q_stride + 32 * first_block + 8 * c) = make_uint2(out[0], out[1]);
        if ((c & 3) == 0) scales[r * scale_stride + first_block + (c >> 2)] = scale;
      }
    }
  }
}

bool Aligned(const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; }

int32_t LaunchProducer(const ProducerParams& p, void* stream, const char* what) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t sms = CurrentDeviceSmCount();
  const int64_t rows = p.kv_a != nullptr ? p.tokens : 0, vectors = p.q_rope != nullptr ? p.tokens * p.heads : 0;
  auto grid_for = [](int64_t items, int64_t cap) {
    const int64_t want = (items + kWarpsPerCta - 1) / kWarpsPerCta;
    return dim3(static_cast<unsigned>(want < cap ? want : cap));
  };
  const int64_t row_items = (rows + kRowsPerPass - 1) / kRowsPerPass, vector_items = (vectors + 7) / 8;
  // One launch up to seven and three quarters passes a warp; beyond that the vectors get a kernel of their own, with twice the
  // warps on an SM. Two rounds of vectors a pass cost one and a half times as much as one, so they pay where they make the
  // passes fewer by more. us for 1,024 / 1,536 / 2,048 / 2,300 tokens x 64 heads (3.7 .. 8.3 passes) in one launch with one
  // round 5.70 / 7.54 / 9.35 / 10.3, with two 4.96 / 6.38 / 7.87 / 9.41, in two launches 6.53 / 8.56 / 8.85 / 8.85 (one kernel
  // of 64 registers, before: 5.79 / 7.42 / 8.29 / 9.66).
  const int64_t resident = sms * kResidentCtas * kWarpsPerCta;
  if (rows > 0 && vectors > 0 && 4 * (row_items + vector_items) <= 31 * resident) {
    const int64_t one = row_items + vector_items, two = row_items + (vectors + 15) / 16;
    const bool rounds_of_two = 2 * ((one + resident - 1) / resident) > 3 * ((two + resident - 1) / resident);
    return CheckCuda(LaunchOverlapped(rounds_of_two ? ProducerKernel<2> : ProducerKernel<1>, grid_for(rounds_of_two ? two : one, sms * kResidentCtas),
                                      dim3(kWarpsPerCta * 32), 0, st, p), what);
  }
  if (rows > 0) {
    if (int32_t rc = CheckCuda(LaunchOverlapped(ProducerKernel<0>, grid_for(row_items, sms * kResidentCtas), dim3(kWarpsPerCta * 32), 0, st,
                                               p), what)) return rc;
  }
  if (vectors == 0) return B200KV_OK;
  // Two rounds for 32 tokens, which leave half the warps without work: 2.05 us, one: 1.66.
  if (vector_items <= sms * 4 * kWarpsPerCta) {
    return CheckCuda(LaunchOverlapped(RotateKernel<1>, grid_for(vector_items, sms * 4), dim3(kWarpsPerCta * 32), 0, st, p), what);
  }
  return CheckCuda(LaunchOverlapped(RotateKernel<2>, grid_for((vector_items + 1) / 2, sms * 4), dim3(kWarpsPerCta * 32), 0, st, p), what);
}

}  // namespace

int32_t ValidatePoolView(const b200kv_pool_view* pool);

}  // namespace b200kv

using namespace b200kv;

extern "C" int32_t b200kv_append_fused(const b200kv_producer_args* args, void* stream, b200kv_status_word* status) {
  if (int32_t rc = FaultCheck("b200kv_append_fused")) return rc;
  if (args == nullptr) {
    SetLastError("append_fused: args is null");
    return B200KV_ERR_NULLPTR;
  }
  const b200kv_producer_args& a = *args;
  if (int32_t rc = ValidatePoolView(&a.pool)) return rc;
  if (a.n_tokens == 0) return B200KV_OK;
  if (a.kv_a == nullptr || a.gamma == nullptr || a.cos == nullptr || a.sin == nullptr || a.slot_mapping == nullptr) {
    SetLastError("append_fused: kv_a, gamma, cos, sin and slot_mapping must be non-null");
    return B200KV_ERR_NULLPTR;
  }
  if (a.n_tokens < 0 || !(a.eps >= 0.0f) || a.kv_a_stride < B200KV_LATENT_DIM + B200KV_ROPE_DIM || a.kv_a_stride % 8 != 0 ||
      !Aligned(a.kv_a, 16) || !Aligned(a.gamma, 16) || a.cos_stride < 0 || a.sin_stride < 0 || a.cos_stride % 8 != 0 ||
      a.sin_stride % 8 != 0 || !Aligned(a.cos, 16) || !Aligned(a.sin, 16) || a.pool.rope_row_stride % 8 != 0 ||
      (a.q_rope != nullptr && (a.heads <= 0 || a.q_head_stride < B200KV_ROPE_DIM || a.q_head_stride % 8 != 0 ||
                               a.q_token_stride % 8 != 0 || !Aligned(a.q_rope, 16))) ||
      (a.latent_out != nullptr && (!Aligned(a.latent_out, 16) || a.latent_out_stride % 8 != 0 ||
                                   a.latent_out_stride < B200KV_LATENT_DIM)) ||
      (a.rope_out != nullptr && (a.rope_out_stride < B200KV_ROPE_DIM || a.rope_out_stride % 8 != 0 ||
                                 !Aligned(a.rope_out, 16)))) {
    SetLastError("append_fused refused: n_tokens %lld, eps %g, kv_a stride %lld (>= 576), heads %d; every tensor needs a "
                 "16-byte aligned base and strides that are multiples of 8 elements",
                 static_cast<long long>(a.n_tokens), static_cast<double>(a.eps), static_cast<long long>(a.kv_a_stride),
                 a.heads);
    return B200KV_ERR_INVALID;
  }
  ProducerParams p{};
  p.pool = a.pool;
  p.kv_a = static_cast<const __nv_bfloat16*>(a.kv_a);
  p.kv_a_stride = a.kv_a_stride;
  p.gamma = static_cast<const __nv_bfloat16*>(a.gamma);
  p.eps = a.eps;
  p.cos = static_cast<const __nv_bfloat16*>(a.cos);
  p.cos_stride = a.cos_stride;
  p.sin = static_cast<const __nv_bfloat16*>(a.sin);
  p.sin_stride = a.sin_stride;
  p.slots = a.slot_mapping;
  p.tokens = a.n_tokens;
  p.q_rope = static_cast<__nv_bfloat16*>(a.q_rope);
  p.q_token_stride = a.q_token_stride;
  p.q_head_stride = a.q_head_stride;
  p.heads = a.heads;
  p.latent_out = static_cast<__nv_bfloat16*>(a.latent_out);
  p.latent_out_stride = a.latent_out_stride;
  p.rope_out = static_cast<__nv_bfloat16*>(a.rope_out);
  p.rope_out_stride = a.rope_out_stride;
  p.rstd_out = a.rstd_out;
  p.status = status;
  return LaunchProducer(p, stream, "append_fused launch");
}

extern "C" int32_t b200kv_rmsnorm512(const void* x, int64_t x_stride, const void* gamma, float eps, int64_t rows, void* y,
                                     int64_t y_stride, float* rstd, void* stream) {
  if (rows == 0) return B200KV_OK;
  if (x == nullptr || gamma == nullptr || y == nullptr) {
    SetLastError("rmsnorm512: x, gamma and y must be non-null");
    return B200KV_ERR_NULLPTR;
  }
  if (rows < 0 || !(eps >= 0.0f) || x_stride < B200KV_LATENT_DIM || x_stride % 8 != 0 || y_stride < B200KV_LATENT_DIM ||
      y_stride % 8 != 0 || !Aligned(x, 16) || !Aligned(y, 16) || !Aligned(gamma, 16)) {
    SetLastError("rmsnorm512 refused: rows %lld, strides %lld/%lld (multiples of 8, >= 512), 16-byte aligned x, gamma, y",
                 static_cast<long long>(rows), static_cast<long long>(x_stride), static_cast<long long>(y_stride));
    return B200KV_ERR_INVALID;
  }
  ProducerParams p{};
  p.kv_a = static_cast<const __nv_bfloat16*>(x);
  p.kv_a_stride = x_stride;
  p.gamma = static_cast<const __nv_bfloat16*>(gamma);
  p.eps = eps;
  p.tokens = rows;
  p.latent_out = static_cast<__nv_bfloat16*>(y);
  p.latent_out_stride = y_stride;
  p.rstd_out = rstd;
  return LaunchProducer(p, stream, "rmsnorm512 launch");
}

extern "C" int32_t b200kv_rope_half64(void* x, int64_t token_stride, int64_t vector_stride, const void* cos,
                                      int64_t cos_stride, const void* sin, int64_t sin_stride, int64_t tokens,
                                      int32_t vectors, void* stream) {
  if (tokens == 0 || vectors == 0) return B200KV_OK;
  if (x == nullptr || cos == nullptr || sin == nullptr) {
    SetLastError("rope_half64: x, cos and sin must be non-null");
    return B200KV_ERR_NULLPTR;
  }
  if (tokens < 0 || vectors < 0 || vector_stride < B200KV_ROPE_DIM || cos_stride < 0 || sin_stride < 0 ||
      vector_stride % 8 != 0 || token_stride % 8 != 0 || cos_stride % 8 != 0 || sin_stride % 8 != 0 || !Aligned(x, 16) ||
      !Aligned(cos, 16) || !Aligned(sin, 16)) {
    SetLastError("rope_half64 refused: tokens %lld, vectors %d, vector stride %lld (>= 64); x, cos and sin need 16-byte "
                 "aligned bases and strides that are multiples of 8 elements",
                 static_cast<long long>(tokens), vectors, static_cast<long long>(vector_stride));
    return B200KV_ERR_INVALID;
  }
  ProducerParams p{};
  p.cos = static_cast<const __nv_bfloat16*>(cos);
  p.cos_stride = cos_stride;
  p.sin = static_cast<const __nv_bfloat16*>(sin);
  p.sin_stride = sin_stride;
  p.tokens = tokens;
  p.q_rope = static_cast<__nv_bfloat16*>(x);
  p.q_token_stride = token_stride;
  p.q_head_stride = vector_stride;
  p.heads = vectors;
  return LaunchProducer(p, stream, "rope_half64 launch");
}

extern "C" int32_t b200kv_mx_quant_e4m3(const void* x, int64_t x_stride, int64_t rows, int64_t cols, void* q,
                                        int64_t q_stride, void* scales, int64_t scale_stride, void* stream) {
  if (int32_t rc = FaultCheck("b200kv_mx_quant_e4m3")) return rc;
  if (rows == 0 || cols == 0) return B200KV_OK;
  if (x == nullptr || q == nullptr || scales == nullptr) {
    SetLastError("mx_quant_e4m3: x, q and scales must be non-null");
    return B200KV_ERR_NULLPTR;
  }
  if (rows < 0 || cols < 0 || cols % 32 != 0 || x_stride < cols || x_stride % 8 != 0 || q_stride < cols ||
      q_stride % 16 != 0 || scale_stride < cols / 32 || !Aligned(x, 16) || !Aligned(q, 16)) {
    SetLastError("mx_quant_e4m3 refused: rows %lld, cols %lld (multiple of 32), strides %lld/%lld/%lld, x and q 16-byte "
                 "aligned with strides that keep every block of 32 aligned",
                 static_cast<long long>(rows), static_cast<long long>(cols), static_cast<long long>(x_stride),
                 static_cast<long long>(q_stride), static_cast<long long>(scale_stride));
    return B200KV_ERR_INVALID;
  }
  const int64_t total = rows * ((cols / 32 + 31) / 32);  // warp items: spans of 32 blocks
  const int64_t want = (total + 7) / 8;
  const int64_t cap = static_cast<int64_t>(CurrentDeviceSmCount()) * 8;
  const int grid = static_cast<int>(want < cap ? want : cap);
  return CheckCuda(LaunchOverlapped(MxQuantKernel, dim3(grid), dim3(256), 0, static_cast<cudaStream_t>(stream),
                                    static_cast<const __nv_bfloat16*>(x), x_stride, rows, cols / 32,
                                    static_cast<uint8_t*>(q), q_stride, static_cast<uint8_t*>(scales), scale_stride),
                   "mx_quant_e4m3 launch");
}
