// Channel-wise gate (one log decay per token, head and key channel): the `prepare` kernel.
//
// With a per-channel decay the ratio exp(G_i,d - G_s,d) sits inside the contraction over d, so
// M[i,s] = beta_i sum_d k[i,d] k[s,d] ratio(i,s)[d] and A[i,s] are not plain Gram products (reference:
// gdn2_chunkwise_cw.py:155-157,168-169).  The 64-token chunk is cut into four blocks of 16 rows:
//   * row block I against earlier blocks: left operand rows x[i] e[i], decayed from the first token of their block, right
//     operand rows k[s] decayed from s to the first token of block I (96 of them for I = 1, 2, 3); tcgen05 products;
//   * the four diagonal 16 x 16 blocks: exact fp32 sums on the CUDA cores, while the products run.
// Everything after M and A (inverse, WY factors, state map) is the scalar-gate kernel's, with per-channel decays in the
// operand scalings.
//
// Layout and decays are those of the backward (gdn_cw_bwd.cu): thread (block of 16 tokens, channel) builds its 16-token
// columns of every decayed operand in registers from alpha = exp(g), the only exponential, and stores them as
// [channel][token] tiles; ratios are products of alphas.  The diagonal blocks need sums over channels instead: there a
// half-warp takes the rows j and 15 - j of a block, a lane eight channels of them.  The 16 rows fall into groups of four:
// inside its own group a row goes down the source rows with ratio(i, s) = ratio(i, s + 1) alpha(s + 1); for an earlier
// group the source rows lie ready in fp32, decayed to the end of their group, and the row carries its decay from there, so
// that a pair costs two FMAs per channel and no ratio.  All in fp32, and every factor is a decay between two rows that lie
// between s and i.  (Walking every pair with a running ratio took 6.8 k cycles per chunk, this 4.8 k.)
//
// NB: blocks of 16 tokens per thread.  2: 256 threads on six tiles that change hands, two persistent CTAs per SM, so that
// one chunk's barriers, product waits and loads lie under the other's arithmetic; k, q and alpha go to registers after the diagonal
// sums and the operands take their tiles.  1: 512 threads, for a launch that gives every SM one chunk at most, where only the
// length of a chunk's own chain counts.  Measured (us, d_v = 128; one CTA of 512 threads with twice the memory before): 8192
// chunks 590 -> 559, 8000 chunks 582 -> 547, 512 chunks 54 -> 49, without the delta term 4096 chunks 209 -> 190, per-channel gates 512
// chunks 70 -> 59; 128 chunks 20.5 either way.
#include "gdn_cw.cuh"
#include "gdn_inverse.cuh"
#include "host_util.h"

namespace lg {

constexpr int kDg = 17;                               // row stride (floats) of the diagonal-block buffers

// Six tiles of 16 KB that change hands:
//   tile       0            1            2                3            4                        5
//   loaded     k            q            g, then alpha (fp32)          k to the end of its four rows (fp32), decays over four rows
//   products   k e          q e          k to the start of later blocks   k exp(G_last - G)     b gamma k
//   inverse    M and scratch             [T; A]           v, beta v    "                        "
//   then       w            u            "                "            P (without the delta term R)
struct PrepCwSmem {
  static constexpr int kTile = 16384, oF = 6 * kTile;
  // floats: diagonal blocks of A and M [64][kDg] each, betas [64], Bb and Af [4][128]
  static constexpr int kFloats = 128 * kDg + 64 + 1024;
  static constexpr int kBytes = oF + kFloats * 4 + static_cast<int>(sizeof(CtaShared)) + 1024;
};

// Sums over the 16 lanes of a half-warp of N values per lane (N = 16 or 8): lane l ends up with the total of value l
// (N = 16) or l >> 1 (N = 8).
template <int N>
__device__ __forceinline__ float half_warp_sum(float* v, int lane) {
#pragma unroll
  for (int w = N / 2, o = 8; w >= 1; w >>= 1, o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < w; ++j) {
      const float send = up ? v[j] : v[j + w];
      const float keep = up ? v[j + w] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if (N == 8) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}
// four neighbouring 16-bit values as two packed pairs
template <bool F16>
__device__ __forceinline__ void ld4_pairs(const unsigned char* src, f2* out) {
  const uint2 u = *reinterpret_cast<const uint2*>(src);
  if (F16) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    out[0] = pack2(a.x, a.y);
    out[1] = pack2(b.x, b.y);
  } else {
    out[0] = pack2(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u));
    out[1] = pack2(__uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
  }
}

// kNorm: q and k are normalised on the way in.  Four lanes have a token's 128 channels; the eight rows of a warp take the
// same 16-byte piece at a time, so the swizzle keeps them off one another's banks.  A kernel of its own reads and writes q and k
// once more: 84 us of the 1036 us of a forward over 16000 tokens and 32 heads, against 978 us with the rows normalised here.
enum CwIn { kInBf16, kInF16, kInNorm };
__device__ __forceinline__ void normalise_rows(unsigned char* t, int warp, int lane, int f16, float eps) {
  const int part = lane >> 3;
  const int r = (warp & 7) * 8 + (lane & 7);
  float x[4][8], ss = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    unpack8_in(tile_ld_chunk(t, r, part + 4 * j, 64), x[j], f16);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss = fmaf(x[j][e], x[j][e], ss);
  }
  ss += __shfl_xor_sync(0xffffffffu, ss, 8);
  ss += __shfl_xor_sync(0xffffffffu, ss, 16);
  const float s = rsqrtf(ss + eps);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[j][e] *= s;
    tile_st_chunk(t, r, part + 4 * j, 64, pack8_f16(x[j]));
  }
}

template <int V, bool DELTA, bool FULL, CwIn IN, int NB>
__global__ void __launch_bounds__(512 / NB, NB)
prepare_cw_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                  const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mg, const __grid_constant__ NormMaps mn) {
  constexpr bool F16 = IN != kInBf16, NORM = IN == kInNorm;      // the type of the tiles once they are here
  constexpr int kThreads = 512 / NB;
  using S = PrepCwSmem;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  auto tile = [&](int i) { return sm + i * S::kTile; };
  unsigned char *tK = tile(0), *tQ = tile(1), *LA = tile(0), *KR = tile(2), *KD = tile(4), *GK = tile(5);
  unsigned char *TA = tile(2), *BV = tile(3), *WU = tile(0), *SP = tile(4);
  float *G = reinterpret_cast<float*>(tile(2)), *kfd = reinterpret_cast<float*>(tile(4)), *Bg = kfd + 48 * kK;
  float* Mt = reinterpret_cast<float*>(tile(0));
  static_assert((kInvMtFloats + kInvScratchFloats) * 4 <= 2 * S::kTile, "M and the inverse's scratch");
  float* Adg = reinterpret_cast<float*>(sm + S::oF);
  float* Mdg = Adg + 64 * kDg;
  float* betas = Mdg + 64 * kDg;
  float* Bb = betas + 64;
  float* Af = Bb + 512;
  CtaShared* cs = reinterpret_cast<CtaShared*>(Af + 512);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, b0 = (warp >> 2) * NB, d = quad * 32 + lane;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *in0 = &cs->bar[0], *in1 = &cs->bar[1], *m1 = &cs->bar[2], *m2 = &cs->bar[3], *m3 = &cs->bar[4];
  const int nchunks = p.nbh * p.cn;
  struct At { int bh, c, z, b, h; };
  auto at = [&](int n) {
    At a;
    a.bh = p.bh0 + n / p.cn;
    a.c = p.c0 + n % p.cn;
    a.z = a.bh * p.NT + a.c;
    a.b = a.bh / p.H;
    a.h = a.bh % p.H;
    return a;
  };
  auto load_kqg = [&](const At& a) {      // (tid 0)
    mbar_expect_tx(in0, 65536u);
    tma_load_4d(tile(2), &mg, in0, 0, a.h, a.c * kC, a.b);
    for (int t = 0; t < 2; ++t) {
      tma_load_4d(tK + t * 8192, &mk, in0, t * 64, a.h, a.c * kC, a.b);
      tma_load_4d(tQ + t * 8192, &mq, in0, t * 64, a.h, a.c * kC, a.b);
    }
  };
  auto load_v = [&](const At& a) {
    mbar_expect_tx(in1, V * 128u);
    for (int t = 0; t < V / 64; ++t) tma_load_4d(BV + t * 8192, &mv, in1, t * 64, a.h, a.c * kC, a.b);
  };
  if (tid == 0) {
    cs->abort_flag = 0;
    for (int i = 0; i < 5; ++i) mbar_init(&cs->bar[i], 1);
    fence_mbar_init();
    fence_proxy_async();
    load_kqg(at(blockIdx.x));
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;      // M | A blocks; [w | u]; [P | R]

  uint32_t ph = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const At a = at(n);
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    const int rows = p.rows_of(a.c);
    const size_t tok0 = (static_cast<size_t>(a.b) * p.L + a.c * kC) * p.H + a.h;
    float beta_r = 1.f;
    if (DELTA && !FULL && tid < 64) beta_r = tid < rows ? p.beta[tok0 + static_cast<size_t>(tid) * p.H] : 0.f;

    // ---- alphas, in place of g; decays of the blocks
    mbar_wait_warp(in0, ph, ctl, 501);
    if (NORM) {
#pragma unroll
      for (int w = 0; w < NB; ++w) {
        const int wq = warp + w * (16 / NB);
        normalise_rows(wq < 8 ? tK : tQ, wq & 7, lane, p.qk16, p.l2_eps);
      }
      fence_proxy_async();
    }
    if (DELTA && tid < 64) betas[tid] = beta_r;
    if (tid == 0) bulk_wait_read();        // the chunk before has left tiles 4 and 5
    __syncthreads();
    if (NORM && tid == 0 && p.keep_norm) {
      for (int t = 0; t < p.Kr / 64; ++t) {
        tma_store_4d(&mn.k, tK + t * 8192, t * 64, a.h, a.c * kC, a.b);
        tma_store_4d(&mn.q, tQ + t * 8192, t * 64, a.h, a.c * kC, a.b);
      }
      bulk_commit();
    }
#pragma unroll 1
    for (int blk = b0; blk < b0 + NB; ++blk) {
      float al[16], B = 1.f;
      uint32_t kp[8];
      read_column(tK, blk, d, F16, kp);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float* gi = G + (blk * 16 + i) * kK + d;
        al[i] = exp2f(*gi * kLog2e);
        *gi = al[i];
      }
#pragma unroll
      for (int A = 0; A < 4; ++A) {        // decays over four rows, and k to the end of its four
        float f = 1.f;
#pragma unroll
        for (int i = 4 * A + 3; i >= 4 * A; --i) {
          if (A < 3) kfd[(blk * 12 + i) * kK + d] = half_of(kp[i >> 1], i & 1) * f;
          f *= al[i];
        }
        Bg[(blk * 4 + A) * kK + d] = f;
        B *= f;
      }
      Bb[blk * kK + d] = B;
      Af[blk * kK + d] = al[0];
    }
    __syncthreads();
    // ---- diagonal blocks, exact.  Half-warp (block, j): rows j and 15 - j - 17 pairs for every j, 5 of them inside the
    // rows' own groups and 3 x 4 with earlier groups; lane: channels 4 c .. 4 c + 3 of either half.
#pragma unroll 1
    for (int it = 0; it < NB; ++it) {
      const int c = lane & 15, j = warp & 7, db = (NB == 1 ? warp >> 3 : it) * 2 + (lane >> 4);
      const float* al0 = G + 4 * c;        // alpha of row r: + 128 r; the other half: + 64
      const unsigned char* kt = tK + (c & 1) * 8;
      const unsigned char* qt = tQ + (c & 1) * 8;
      auto at16 = [&](int r) { return r * 128 + (((c >> 1) ^ (r & 7)) << 4); };
      const f2 one = pack2(1.f, 1.f), zero = pack2(0.f, 0.f);
      // sums of one row against one source row: A, and M where the delta term wants it
      auto dots = [&](const f2* t, const f2* qi, const f2* ki, float& sa, float& sm_) {
        f2 aa = zero, mm = zero;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          aa = fma2(qi[e], t[e], aa);
          if (DELTA) mm = fma2(ki[e], t[e], mm);
        }
        sa = sum2(aa);
        sm_ = DELTA ? sum2(mm) : 0.f;
      };
      auto store = [&](int i, int s, bool is_m, float x) {
        const int r = db * 16 + i;
        if (is_m) Mdg[r * kDg + s] = s < i ? betas[r] * x : 0.f;
        else Adg[r * kDg + s] = p.scale * x;
      };
      const int i0 = 15 - j, i1 = j;
      f2 q0[4], k0[4], q1[4], k1[4];               // the two rows; later times their decay
      float v[16];
      auto own_group = [&](int i, f2* qi, f2* ki, float* out) {
        const int r = db * 16 + i;
        ld4_pairs<F16>(qt + at16(r), qi);
        ld4_pairs<F16>(qt + 8192 + at16(r), qi + 2);
        ld4_pairs<F16>(kt + at16(r), ki);
        ld4_pairs<F16>(kt + 8192 + at16(r), ki + 2);
        if (FULL) {
          const float* bp = p.bch + (tok0 + static_cast<size_t>(r) * p.H) * kK + 4 * c;
          f2 b[4];
          ld_pairs(bp, b);
          ld_pairs(bp + 64, b + 2);
#pragma unroll
          for (int e = 0; e < 4; ++e) ki[e] = mul2(ki[e], b[e]);
        }
        f2 ratio[4] = {one, one, one, one};
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          out[u] = out[4 + u] = 0.f;
          if (u > (i & 3)) continue;               // (the same for the whole warp)
          const int s = (i & ~3) + u, rs = db * 16 + s;
          f2 ks[4], as[4];
          ld4_pairs<F16>(kt + at16(rs), ks);
          ld4_pairs<F16>(kt + 8192 + at16(rs), ks + 2);
          ld_pairs(al0 + kK * rs, as);
          ld_pairs(al0 + kK * rs + 64, as + 2);
#pragma unroll
          for (int e = 0; e < 4; ++e) ks[e] = mul2(ratio[e], ks[e]);
          dots(ks, qi, ki, out[u], out[4 + u]);
#pragma unroll
          for (int e = 0; e < 4; ++e) ratio[e] = mul2(ratio[e], as[e]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {              // the row's decay from the end of the group before its own
          qi[e] = mul2(qi[e], ratio[e]);
          if (DELTA) ki[e] = mul2(ki[e], ratio[e]);
        }
      };
      own_group(i0, q0, k0, v);
      own_group(i1, q1, k1, v + 8);
      {
        const float t = half_warp_sum<16>(v, lane);
        const int i = (c & 8) ? i1 : i0, s = (i & ~3) + (c & 3);
        if (s <= i) store(i, s, (c & 4) != 0, t);
      }
      // earlier group B of a row; then the row's decay goes on over that group
      auto earlier = [&](int B, f2* qi, f2* ki, float* out) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          f2 t[4];
          ld_pairs(kfd + (db * 12 + 4 * B + u) * kK + 4 * c, t);
          ld_pairs(kfd + (db * 12 + 4 * B + u) * kK + 64 + 4 * c, t + 2);
          dots(t, qi, ki, out[u], out[4 + u]);
        }
        if (B > 0) {
          f2 g[4];
          ld_pairs(Bg + (db * 4 + B) * kK + 4 * c, g);
          ld_pairs(Bg + (db * 4 + B) * kK + 64 + 4 * c, g + 2);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            qi[e] = mul2(qi[e], g[e]);
            if (DELTA) ki[e] = mul2(ki[e], g[e]);
          }
        }
      };
      // row 15 - j has three earlier groups for j < 4 and two otherwise, row j none and one
      const int B0 = (i0 >> 2) - 1;
      earlier(B0, q0, k0, v);
      earlier(B0 - 1, q0, k0, v + 8);
      {
        const float t = half_warp_sum<16>(v, lane);
        store(i0, 4 * (B0 - (c >> 3)) + (c & 3), (c & 4) != 0, t);
      }
      if (j < 4) earlier(0, q0, k0, v);
      else earlier(0, q1, k1, v);
      {
        const float t = half_warp_sum<8>(v, lane);
        store(j < 4 ? i0 : i1, (c >> 1) & 3, (c & 8) != 0, t);
      }
    }
    // ---- this thread's columns: decays, k, q
    float al[NB][16];
    uint32_t kp[NB][8], qp[NB][8];
#pragma unroll
    for (int bb = 0; bb < NB; ++bb) {
      read_column(tK, b0 + bb, d, F16, kp[bb]);
      read_column(tQ, b0 + bb, d, F16, qp[bb]);
#pragma unroll
      for (int i = 0; i < 16; ++i) al[bb][i] = G[((b0 + bb) * 16 + i) * kK + d];
    }
    if (NORM && tid == 0) bulk_wait_read();      // the normalised rows have left
    __syncthreads();                             // k, q, alpha and the decayed rows are read: their tiles become operands
    // ---- operand tiles
#pragma unroll
    for (int bb = 0; bb < NB; ++bb) {
      const int blk = b0 + bb;
      const BlockDecays bd = block_decays(Bb, Af, blk, d);
      const float gam0 = bd.pre * al[bb][0];     // gamma of the block's first token
      if (blk == 3) reinterpret_cast<float*>(p.saved + p.lay.ad)[static_cast<size_t>(a.z) * kK + d] = bd.pre * Bb[3 * kK + d];
      float x[16], y[16], f = 1.f, e = 1.f;
#pragma unroll
      for (int i = 15; i >= 0; --i) {            // k to the end of its block ...
        x[i] = half_of(kp[bb][i >> 1], i & 1) * f;
        f *= al[bb][i];
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) y[i] = x[i] * bd.post;
      write_column(KD, blk, d, y);
#pragma unroll
      for (int I = 1; I < 4; ++I) {              // ... and on to the start of every later block
        if (I <= blk) continue;
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = x[i] * bd.cup[I - 1];
        // columns: block 3's 48 and block 1's 16 in the first atom, block 2's 32 in the second
        unsigned char* t = KR + (I == 2 ? 16384 : 0);
        write_column(t, I == 1 ? 3 : blk, d, y);
      }
      // scale gamma q leaves for its record, the image of a [64 tokens][128 channels] tile: a warp writes 64 bytes of a row
      unsigned char* qg = p.saved + p.lay.qg + static_cast<size_t>(a.z) * 16384;
      const float sg = p.scale * gam0;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i) e *= al[bb][i];
        y[i] = half_of(qp[bb][i >> 1], i & 1) * e;
        store_f16_sat(qg + sw128_off(blk * 16 + i, d, 64), y[i] * sg);
      }
      write_column(LA + 16384, blk, d, y);
      if (DELTA) {
        e = 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (i) e *= al[bb][i];
          x[i] = half_of(kp[bb][i >> 1], i & 1) * e;
          if (FULL) x[i] *= p.bch[(tok0 + static_cast<size_t>(blk * 16 + i) * p.H) * kK + d];
        }
        write_column(LA, blk, d, x);             // left factor of M (without the row's beta)
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] *= FULL ? gam0 : gam0 * betas[blk * 16 + i];
        write_column(GK, blk, d, x);
      }
    }
    sync_for_issue();

    // ---- off-diagonal blocks of M (rows 0-63) and A (rows 64-127) on the tensor cores
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(LA), 128, true}, Tile{smem_u32(KR), 128, true}, 64, 128, 0u);
      issue_product_led(leader, tmem + 64, Tile{smem_u32(LA), 128, true}, Tile{smem_u32(KR) + 16384, 128, true}, 32, 128, 0u);
      umma_commit_led(leader, m1);
    }
    __syncwarp();
    mbar_wait_warp(m1, ph, ctl, 502);
    tc_fence_after();
    if (tid == 0) load_v(a);
#pragma unroll 1
    for (int blk = b0; blk < b0 + NB; ++blk) {
      // thread: accumulator lane t = quad * 32 + lane (row r of M for lanes 0-63, of A for 64-127), columns of block blk
      const int t = d, r = t & 63, I = r >> 4, I0 = 2 * (quad & 1);      // a warp's lanes are rows of blocks I0 and I0 + 1
      float x[16], y[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) x[e] = 0.f;
      auto col = [](int rb, int cb) { return rb == 1 ? 48 : (rb == 2 ? 64 : 0) + 16 * cb; };
      if (blk < I0 + 1) {
        tmem_ld16(tmem + lane_base + col(I0 + 1, blk), y);
        tmem_ld_wait();
        if (I == I0 + 1)
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = y[e];
      }
      if (blk < I0) {
        tmem_ld16(tmem + lane_base + col(I0, blk), y);
        tmem_ld_wait();
        if (I == I0)
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = y[e];
      }
      if (t < 64) {
        if (DELTA) {
          const float be = betas[r];
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            x[e] *= be;
            if (I == blk) x[e] = blk * 16 + e < r ? Mdg[r * kDg + e] : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 16; ++e) Mt[(blk * 16 + e) * kMt + r] = x[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          x[e] *= p.scale;
          if (I == blk) x[e] = blk * 16 + e <= r ? Adg[r * kDg + e] : 0.f;
        }
        write_row16(TA, 64 + r, blk, x);
      }
    }
    tc_fence_before();
    __syncthreads();

    // ---- beta v (w v) on the warps that have no part in the inverse, or not in its first step
    constexpr int kFirst = NB == 1 ? 256 : 64;
    if (tid >= kFirst) {
      mbar_wait_warp(in1, ph, ctl, 505);
      for (int idx = tid - kFirst; idx < 64 * (V / 8); idx += kThreads - kFirst) {
        const int r = idx / (V / 8), ch = idx % (V / 8);
        float x[8];
        unpack8_bf16(tile_ld_chunk(BV, r, ch, 64), x);
        if (DELTA && FULL) {
          float wv[8];
          ld8(p.wch + (tok0 + static_cast<size_t>(r) * p.H) * V + ch * 8, wv);
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] *= wv[i];
        } else {
          const float be = DELTA ? betas[r] : 1.f;
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] *= be;
        }
        tile_st_chunk(BV, r, ch, 64, pack8_f16(x));
      }
    }
    // ---- T = (I + M)^-1 (fp32, CUDA cores)
    if (DELTA) {
      unit_lower_inverse64(Mt, Mt + kInvMtFloats, TA, tid);
      sync_for_issue();
      // ---- [w | u] = T [b gamma k | beta v]
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, tmem, Tile{smem_u32(TA), 128, false}, Tile{smem_u32(GK), 128, false}, 128, 64, 0u);
        issue_product_led(leader, tmem + 128, Tile{smem_u32(TA), 128, false}, Tile{smem_u32(BV), 64, true}, V, 64, 0u);
        umma_commit_led(leader, m2);
        if (tid == 0) {
          if (p.lean < 2) bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta, TA, 16384);
          else bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, TA + 8192, 8192);      // A only
          bulk_commit();
        }
      }
      __syncwarp();
      mbar_wait_warp(m2, ph, ctl, 503);
      tc_fence_after();
      if (quad < 2) {                      // rows 0-63; the warps of a quadrant split the columns
#pragma unroll 1
        for (int jb = warp >> 2; jb < (128 + V) / 32; jb += 4 / NB) {
          float x[32];
          tmem_ld32(tmem + lane_base + jb * 32, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) tile_st_chunk(WU, d, jb * 4 + i, 64, pack8_f16(x + 8 * i));
        }
      }
      sync_for_issue();
    } else {
      fence_proxy_async();
      __syncthreads();
      if (tid == 0) {                      // A only: without the delta term nothing reads T
        bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, TA + 8192, 8192);
        bulk_commit();
      }
    }

    // ---- [P | R] = kd^T [w | u]   (no delta: R = kd^T v)
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(KD), 128, false}, Tile{smem_u32(DELTA ? WU : BV), 64, true}, DELTA ? 128 + V : V, 64, 0u);
      umma_commit_led(leader, m3);
      if (tid == 0) {
        if (DELTA) {
          bulk_s2g(p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w, WU, 16384);
          bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, WU + 16384, V * 128);
        } else if (!p.lean) {            // (u is v)
          bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, BV, V * 128);
        }
        bulk_commit();
      }
    }
    __syncwarp();
    mbar_wait_warp(m3, ph, ctl, 504);
    tc_fence_after();
    if (tid == 0 && more) {                // tiles 0 to 3 are dead once their records have left
      bulk_wait_read();
      load_kqg(at(n + gridDim.x));
    }
    // P leaves as its record image through the tiles of the last operands, R (16 columns of a row are 32 bytes of its record,
    // the rows of a warp 1 KB) directly; the warps of a lane quadrant split the columns
    unsigned char* r_g = p.saved + p.lay.r + static_cast<size_t>(a.z) * p.lay.sz_r;
#pragma unroll 1
    for (int jb = warp >> 2; jb < (DELTA ? 128 + V : V) / 32; jb += 4 / NB) {
      float x[32];
      tmem_ld32(tmem + lane_base + jb * 32, x);
      tmem_ld_wait();
      if (!DELTA || jb < 4) {              // P; R without the delta term, a plain tile image
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(SP, d, jb * 4 + i, 128, pack8_f16(x + 8 * i));
      } else {
        const int c8 = (jb - 4) * 4;
#pragma unroll
        for (int i = 0; i < 4; i += 2) st_global_32(r_g + rrec_off(d, c8 + i), pack8_f16(x + 8 * i), pack8_f16(x + 8 * i + 8));
      }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      if (DELTA) bulk_s2g(p.saved + p.lay.p + static_cast<size_t>(a.z) * p.lay.sz_p, SP, 32768);
      else bulk_s2g(r_g, SP, V * 256);
      bulk_commit();
    }
  }
  if (tid == 0) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

template <int V, bool DELTA, bool FULL, CwIn IN, int NB>
static int launch_prepare_cw_n(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                               const CUtensorMap& mg, const NormMaps& mn, int sms, cudaStream_t st) {
  constexpr int smem = PrepCwSmem::kBytes;
  static_assert(2 * (smem + 1024) <= 228 * 1024, "two CTAs per SM");
  auto kern = prepare_cw_kernel<V, DELTA, FULL, IN, NB>;
  static SmemAttr attr;
  if (attr.set(kern, smem)) return kErrLaunch;
  const int n = p.nbh * p.cn, most = NB * sms;
  kern<<<n < most ? n : most, 512 / NB, smem, st>>>(p, mq, mk, mv, mg, mn);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
template <int V, bool DELTA, bool FULL, CwIn IN>
static int launch_prepare_cw_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                               const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st) {
  const int sms = sm_count();
  if (sms <= 0) return kErrDevice;
  // (the line between the two: see NB above)
  return p.nbh * p.cn <= sms ? launch_prepare_cw_n<V, DELTA, FULL, IN, 1>(p, mq, mk, mv, mg, mn, sms, st)
                             : launch_prepare_cw_n<V, DELTA, FULL, IN, 2>(p, mq, mk, mv, mg, mn, sms, st);
}
template <int V, bool DELTA, bool FULL>
static int launch_prepare_cw_f(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                               const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st) {
  if (p.l2_eps > 0.f) return launch_prepare_cw_t<V, DELTA, FULL, kInNorm>(p, mq, mk, mv, mg, mn, st);
  return p.qk16 ? launch_prepare_cw_t<V, DELTA, FULL, kInF16>(p, mq, mk, mv, mg, mn, st)
                : launch_prepare_cw_t<V, DELTA, FULL, kInBf16>(p, mq, mk, mv, mg, mn, st);
}
template <int V>
static int launch_prepare_cw_v(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                               const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st) {
  if (!p.delta) return launch_prepare_cw_f<V, false, false>(p, mq, mk, mv, mg, mn, st);
  return p.bch ? launch_prepare_cw_f<V, true, true>(p, mq, mk, mv, mg, mn, st) : launch_prepare_cw_f<V, true, false>(p, mq, mk, mv, mg, mn, st);
}

int launch_prepare_cw(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                      const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st) {
  return p.V == 64 ? launch_prepare_cw_v<64>(p, mq, mk, mv, mg, mn, st) : launch_prepare_cw_v<128>(p, mq, mk, mv, mg, mn, st);
}

}  // namespace lg
