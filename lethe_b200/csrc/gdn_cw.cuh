// Helpers of the channel-wise kernels, in which thread (block of 16 tokens, channel) owns a 16-token column of everything
// that has a channel axis: column access to tiles, packed fp32 pairs, lane sums.
#pragma once
#include "gdn_common.cuh"

namespace lg {

__device__ __forceinline__ float half_of(uint32_t pair, int hi) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&pair));
  return hi ? f.y : f.x;
}
__device__ __forceinline__ float in16(uint16_t x, int f16) {
  if (f16) return __half2float(__ushort_as_half(x));
  return __uint_as_float(static_cast<uint32_t>(x) << 16);
}
__device__ __forceinline__ void store_f16_sat(unsigned char* dst, float x) {
  *reinterpret_cast<uint16_t*>(dst) = static_cast<uint16_t>(f16x2_sat(x, 0.f));
}
// a 16-bit token-major tile [64 tokens][D channels] as TMA leaves it: this thread's 16-token column, as fp16 pairs
__device__ __forceinline__ void read_column(const unsigned char* tile, int blk, int d, int f16, uint32_t* out) {
  const unsigned char* base = tile + (d >> 6) * 8192 + blk * 2048 + (d & 7) * 2;
  const int ch = (d >> 3) & 7;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint16_t a = *reinterpret_cast<const uint16_t*>(base + (2 * j) * 128 + ((ch ^ ((2 * j) & 7)) << 4));
    const uint16_t b = *reinterpret_cast<const uint16_t*>(base + (2 * j + 1) * 128 + ((ch ^ ((2 * j + 1) & 7)) << 4));
    out[j] = f16 ? (static_cast<uint32_t>(b) << 16 | a) : f16x2_sat(in16(a, 0), in16(b, 0));
  }
}
// 16 values of this thread's column into a [channel][token] tile (128-byte rows, SW128)
__device__ __forceinline__ void write_column(unsigned char* tile, int blk, int d, const float* x) {
  *reinterpret_cast<uint4*>(tile + sw128_chunk(d, 2 * blk, 128)) = pack8_f16(x);
  *reinterpret_cast<uint4*>(tile + sw128_chunk(d, 2 * blk + 1, 128)) = pack8_f16(x + 8);
}
// one 16-bit result of token r into a token-major tile [64 tokens][channels], the image a tensor-map store takes
__device__ __forceinline__ void stage16(unsigned char* tile, int r, int d, float x, int f16) {
  *reinterpret_cast<uint16_t*>(tile + sw128_off(r, d, 64)) =
      f16 ? static_cast<uint16_t>(f16x2_sat(x, 0.f)) : __bfloat16_as_ushort(__float2bfloat16_rn(x));
}

// two such results, of tokens r and r + 1
__device__ __forceinline__ void stage16_two(unsigned char* tile, int r, int d, f2 x, int f16) {
  float lo, hi;
  unpack2(x, lo, hi);
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  const uint32_t u = f16 ? f16x2_sat(lo, hi) : *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint16_t*>(tile + sw128_off(r, d, 64)) = static_cast<uint16_t>(u);
  *reinterpret_cast<uint16_t*>(tile + sw128_off(r + 1, d, 64)) = static_cast<uint16_t>(u >> 16);
}
__device__ __forceinline__ f2 pair_of(uint32_t halves) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&halves));
  return pack2(f.x, f.y);
}

// 16 columns of block blk of row r of a [token][token] tile (128-byte rows)
__device__ __forceinline__ void write_row16(unsigned char* tile, int r, int blk, const float* x) {
  *reinterpret_cast<uint4*>(tile + sw128_chunk(r, 2 * blk, 64)) = pack8_f16(x);
  *reinterpret_cast<uint4*>(tile + sw128_chunk(r, 2 * blk + 1, 64)) = pack8_f16(x + 8);
}

// Sums over the 32 lanes of eight values per lane: lane l ends up with the total of value (l >> 2).
__device__ __forceinline__ float warp_sum8(float* v, int lane) {
#pragma unroll
  for (int w = 4, o = 16; w >= 1; w >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float send = up ? v[j] : v[j + w];
      const float keep = up ? v[j + w] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

// The same of four values: lane l ends up with the total of value (l >> 3).
__device__ __forceinline__ float warp_sum4(float* v, int lane) {
#pragma unroll
  for (int w = 2, o = 16; w >= 1; w >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float send = up ? v[j] : v[j + w];
      const float keep = up ? v[j + w] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
#pragma unroll
  for (int o = 4; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// Decays between this thread's block of 16 tokens and the others, for its channel: cdn[J] from the end of block J to the
// first token of this one (J < blk), cup[I - 1] from the end of this block to the first token of block I (I > blk), pre /
// post the whole decay of the blocks before / after.  Bb: products of a block's alphas, Af: its first alpha, [4][128].
struct BlockDecays { float cdn[3], cup[3], pre, post; };
__device__ __forceinline__ BlockDecays block_decays(const float* Bb, const float* Af, int blk, int d) {
  BlockDecays r;
  float bm[4], am[4], own = 1.f;
  r.pre = r.post = 1.f;
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    bm[m] = Bb[m * kK + d];
    am[m] = Af[m * kK + d];
    if (m == blk) own = am[m];
    if (m < blk) r.pre *= bm[m];
    if (m > blk) r.post *= bm[m];
  }
#pragma unroll
  for (int J = 0; J < 3; ++J) {
    r.cdn[J] = own;
#pragma unroll
    for (int m = J + 1; m < 4; ++m)
      if (m < blk) r.cdn[J] *= bm[m];
    r.cup[J] = am[J + 1];
#pragma unroll
    for (int m = 1; m <= J; ++m)
      if (m > blk) r.cup[J] *= bm[m];
  }
  return r;
}

}  // namespace lg
