// T = (I + M)^-1 for a strictly lower-triangular 64 x 64 M in fp32 (CUDA cores), on threads 0-255 of a CTA (every thread of
// the CTA must call: four CTA-wide barriers inside).  The inverses of the four 16 x 16 diagonal blocks by forward
// substitution, one column per thread; then twice, for blocks of 16 and of 32,
//   [[A, 0], [C, B]]^-1 = [[A^-1, 0], [-B^-1 (C A^-1), B^-1]].
//
// Bound by latency and by the wavefronts of shared-memory loads.  In every product a thread owns two columns and two or four
// rows: the left factor is kept transposed, so that either operand of a step is one load.  Five stages of 16-long dot products
// on 16 x 16 blocks, a lane reading its own left row and four or eight columns, took 3.2 k
// cycles alone on an SM and 4.3 k beside a second CTA; this takes 2.4 k (prepare, 4096 chunks: 144 -> 132 us).
#pragma once
#include "gdn_common.cuh"

namespace lg {

constexpr int kMt = 68;                     // M transposed: element (row r, column s) at [s * kMt + r], zero for r <= s
constexpr int kT32 = 36, kT16 = 20;         // row strides of 32 x 32 and 16 x 16 blocks
constexpr int kInvMtFloats = 64 * kMt, kInvScratchFloats = 2 * 32 * kT32 + 4 * 16 * kT16;

// c[column][row pair] = sum_k left[k * SL + row] right[k * SR + column] for 2 R rows and two columns
template <int R, int KD, int SL, int SR>
__device__ __forceinline__ void tile_product(f2 (*c)[R], const float* left, const float* right) {
#pragma unroll
  for (int r = 0; r < R; ++r) c[0][r] = c[1][r] = pack2(0.f, 0.f);
#pragma unroll
  for (int k = 0; k < KD; ++k) {
    const float2 x = *reinterpret_cast<const float2*>(right + k * SR);
    const f2 x0 = pack2(x.x, x.x), x1 = pack2(x.y, x.y);
    f2 m[R];
    if (R == 2) ld_pairs(left + k * SL, m);
    else m[0].u = *reinterpret_cast<const unsigned long long*>(left + k * SL);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      c[0][r] = fma2(m[r], x0, c[0][r]);
      c[1][r] = fma2(m[r], x1, c[1][r]);
    }
  }
}
// the rows of such a tile, two columns each, at dst + row * stride
template <int R>
__device__ __forceinline__ void store_tile(const f2 (*c)[R], float* dst, int stride, float sign) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float a0, a1, b0, b1;
    unpack2(c[0][r], a0, a1);
    unpack2(c[1][r], b0, b1);
    *reinterpret_cast<float2*>(dst + 2 * r * stride) = make_float2(sign * a0, sign * b0);
    *reinterpret_cast<float2*>(dst + (2 * r + 1) * stride) = make_float2(sign * a1, sign * b1);
  }
}

// Mt: kInvMtFloats, overwritten.  scratch: kInvScratchFloats.  T leaves as fp16 in rows 0-63 of the 128-row tile TA.
// diag: the diagonal 16 x 16 blocks, transposed like Mt, SD floats between rows and DB between blocks; of what is not below the
// diagonal only the diagonal itself is read, as zero.
template <int SD = kMt, int DB = 16 * kMt + 16>
__device__ __forceinline__ void unit_lower_inverse64(float* Mt, const float* diag, float* scratch, unsigned char* TA, int tid) {
  const int warp = tid >> 5, lane = tid & 31;
  float* T11 = scratch;                     // rows 0-31 of T
  float* T22t = T11 + 32 * kT32;            // rows 32-63 of its right half, transposed
  float* D0t = T22t + 32 * kT32;            // the first two diagonal blocks transposed (the first for symmetry only)
  float* D2 = D0t + 2 * 16 * kT16;          // the last two as they are
  float* Y = Mt + 32 * kMt;                 // 32 x 32 at stride kMt, where M has zeros
  if (tid < 64) {                           // forward substitution, two rows per packed FMA
    const int b = tid >> 4, j = tid & 15;
    const float* M = diag + b * DB;
    f2 x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = pack2(2 * q == j ? 1.f : 0.f, 2 * q + 1 == j ? 1.f : 0.f);
#pragma unroll
    for (int k = 0; k < 15; ++k) {
      float lo, hi;
      unpack2(x[k >> 1], lo, hi);
      const float xk = (k & 1) ? -hi : -lo;
      const f2 xx = pack2(xk, xk);
#pragma unroll
      for (int p4 = (k + 1) >> 2; p4 < 4; ++p4) {
        f2 m[2];
        ld_pairs(M + k * SD + 4 * p4, m);
#pragma unroll
        for (int t = 0; t < 2; ++t)
          if (2 * (2 * p4 + t) + 1 > k) x[2 * p4 + t] = fma2(m[t], xx, x[2 * p4 + t]);
      }
    }
    // every thread stores its column both ways: with the two stores that nothing reads left out, branches between the
    // others took 1.0 k cycles
    float* row = b < 2 ? T11 + 16 * b * (kT32 + 1) + j : D2 + (b - 2) * 16 * kT16 + j;
    float* col = b < 2 ? D0t + (16 * b + j) * kT16 : T22t + 16 * (b - 2) * (kT32 + 1) + j * kT32;
    const int sr = b < 2 ? kT32 : kT16;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float lo, hi;
      unpack2(x[q], lo, hi);
      row[2 * q * sr] = lo;
      row[(2 * q + 1) * sr] = hi;
      *reinterpret_cast<unsigned long long*>(col + 2 * q) = x[q].u;
    }
  } else if (tid < 256) {                   // zeros above the diagonal
    const int u = tid - 64;
    if (u < 128) {
      tile_st_chunk(TA, u >> 2, 4 + (u & 3), 128, make_uint4(0u, 0u, 0u, 0u));
    } else {
      const int i = (u - 128) >> 2, e = 4 * (u & 3);
      *reinterpret_cast<float4*>(T11 + i * kT32 + 16 + e) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(T22t + (16 + i) * kT32 + e) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __syncthreads();
  // ---- blocks of 16: two warps per pair of blocks
  {
    const int pr = warp >> 1, c0 = 2 * (lane & 7), i0 = 8 * (warp & 1) + 2 * (lane >> 3);
    float* Yp = Mt + pr * (32 * kMt + 32);  // over the first diagonal block of the pair, stride kMt
    f2 c[2][1];
    if (tid < 128) {
      if (pr == 0) tile_product<1, 16, kMt, kT32>(c, Mt + 16 + i0, T11 + c0);
      else tile_product<1, 16, kMt, kT16>(c, Mt + 32 * kMt + 48 + i0, D2 + c0);
      store_tile<1>(c, Yp + i0 * kMt + c0, kMt, 1.f);
    }
    __syncthreads();
    if (tid < 128) {
      if (pr == 0) {
        tile_product<1, 16, kT16, kMt>(c, D0t + 16 * kT16 + i0, Yp + c0);
        store_tile<1>(c, T11 + (16 + i0) * kT32 + c0, kT32, -1.f);
      } else {
        tile_product<1, 16, kT32, kMt>(c, T22t + 16 * (kT32 + 1) + i0, Yp + c0);
        float lo, hi;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          unpack2(c[e][0], lo, hi);
          *reinterpret_cast<float2*>(T22t + (c0 + e) * kT32 + 16 + i0) = make_float2(-lo, -hi);
        }
      }
    }
  }
  __syncthreads();
  // ---- blocks of 32: four warps; the others turn the diagonal blocks of T to fp16
  const int c0 = 2 * (lane & 15), i0 = 8 * (warp & 3) + 4 * (lane >> 4);
  f2 c[2][2];
  if (tid < 128) {
    tile_product<2, 32, kMt, kT32>(c, Mt + 32 + i0, T11 + c0);
    store_tile<2>(c, Y + i0 * kMt + c0, kMt, 1.f);
  } else if (tid < 256) {
    const int ch = warp & 3;                // row `lane` of either block, one 16-byte piece
    float v[8];
    ld8(T11 + lane * kT32 + 8 * ch, v);
    tile_st_chunk(TA, lane, ch, 128, pack8_f16(v));
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = T22t[(8 * ch + e) * kT32 + lane];
    tile_st_chunk(TA, 32 + lane, 4 + ch, 128, pack8_f16(v));
  }
  __syncthreads();
  if (tid < 128) {
    tile_product<2, 32, kT32, kMt>(c, T22t + i0, Y + c0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float a0, a1, b0, b1;
      unpack2(c[0][r], a0, a1);
      unpack2(c[1][r], b0, b1);
      *reinterpret_cast<uint32_t*>(TA + sw128_off(32 + i0 + 2 * r, c0, 128)) = f16x2_sat(-a0, -b0);
      *reinterpret_cast<uint32_t*>(TA + sw128_off(33 + i0 + 2 * r, c0, 128)) = f16x2_sat(-a1, -b1);
    }
  }
}

}  // namespace lg
