// Channel-wise gate (one log decay per token, head and key channel): the `prepare` kernel.
//
// With a per-channel decay the ratio exp(G_i,d - G_s,d) sits inside the contraction over d, so
// M[i,s] = beta_i sum_d k[i,d] k[s,d] ratio(i,s)[d] and A[i,s] are not plain Gram products (reference:
// gdn2_chunkwise_cw.py:155-157,168-169).  The 64-token chunk is cut into four blocks of 16 rows:
//   * row block I against earlier blocks: left operand rows x[i] e[i], decayed from the first token of their block, right
//     operand rows k[s] decayed from s to the first token of block I (96 of them for I = 1, 2, 3); tcgen05 products;
//   * the four diagonal 16 x 16 blocks: exact fp32 sums on the CUDA cores.
// Everything after M and A (inverse, WY factors, state map) is the scalar-gate kernel's, with per-channel decays in the
// operand scalings.
//
// Layout and decays are those of the backward (gdn_cw_bwd.cu): thread (block of 16 tokens, channel) builds its 16-token
// columns of every decayed operand in registers from alpha = exp(g), the only exponential, and stores them as
// [channel][token] tiles; ratios are products of alphas.  The diagonal blocks need sums over channels instead: there a
// half-warp has a block, a lane eight channels of it.  The 16 rows fall into groups of four.  Inside a group the source rows
// are carried along, decayed to the row in hand.  For an earlier group they lie ready in fp32, decayed to the end of their
// group, and the four rows of the later group, decayed from there, stay in registers while the source rows go by: a pair costs
// two packed FMAs per two channels, and a source row is loaded once for four rows.  All in fp32, and every factor is a decay
// between two rows that lie between s and i.  (Two rows of a block per half-warp, each loading its source rows: 11 k warp
// instructions per chunk, now 7 k; 35 k against 29 k for the whole kernel.)
//
// NB: blocks of 16 tokens per thread.  2: 256 threads on six tiles that change hands, two persistent CTAs per SM, so that
// one chunk's barriers, product waits and loads lie under the other's arithmetic; k, q and alpha go to registers after the diagonal
// sums and the operands take their tiles.  1: 512 threads, for a launch that gives every SM one chunk at most, where only the
// length of a chunk's own chain counts.  Measured (us, d_v = 128; one CTA of 512 threads with twice the memory / two of 256 /
// these diagonal sums, loads that come early, beta a chunk ahead): 8192 chunks 590 / 559 / 486 (480 with the abort flag behind the waits); 512 chunks 54 / 49 / 44; without the
// delta term 4096 chunks 209 / 190 / 158; per-channel gates 512 chunks 70 / 59 / 52; 128 chunks 20 in each.
//
// Loads: k and q of the next chunk as soon as the inverse is done, g when w and u have left its tiles, behind a prefetch to L2 that
// was issued before the inverse; the write gates of the full op are requested under the first products.
// Bound by the chain of phases of a chunk and by shared memory (LSU data pipe 57 % busy, issue slots 46 %).  Cycles per chunk by
// clock samples of one of two CTAs (d_v = 128): waits for loads 1.9 k, alphas 1.9 k, diagonal blocks 6.3 k, columns and operands
// 4.6 k, products and epilogue of M and A 3.1 k, inverse 5.6 k, w and u 2.3 k, P and R 3.7 k.
#include "gdn_cw.cuh"
#include "gdn_inverse.cuh"
#include "host_util.h"

namespace lg {

// row strides (floats) of the diagonal blocks: A by rows, M by columns (transposed, as the inverse reads it)
constexpr int kDg = 17, kDm = 20;

// Six tiles of 16 KB that change hands:
//   tile       0            1            2                3                4                    5
//   loaded     k            q            g, then alpha (fp32)              k to the end of its four rows (fp32), decays over four rows
//   products   k e          q e          b gamma k        k to blocks 3, 1 k exp(G_last - G)    k to block 2
//   inverse    M and scratch             "                v, beta v        "                    [T; A]  (without delta: 2)
//   then       the next k   and q        w                u                P                    (without delta: R)
//   then       "            "            the next g                        "
struct PrepCwSmem {
  static constexpr int kTile = 16384, oF = 6 * kTile;
  // floats: diagonal blocks of M [64][kDm] and A [64][kDg], betas [2][64], Bb and Af [4][128]
  static constexpr int kFloats = 64 * (kDm + kDg) + 128 + 1024;
  static constexpr int kBytes = oF + kFloats * 4 + 2 * static_cast<int>(sizeof(ChunkAt)) + static_cast<int>(sizeof(CtaShared)) + 1024;
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
  unsigned char *tK = tile(0), *tQ = tile(1), *LA = tile(0), *KR = tile(3), *KR2 = tile(5), *KD = tile(4), *GK = tile(2);
  unsigned char *TA = tile(DELTA ? 5 : 2), *BV = tile(3), *WU = tile(2), *SP = tile(4);
  float *G = reinterpret_cast<float*>(tile(2)), *kfd = reinterpret_cast<float*>(tile(4)), *Bg = kfd + 48 * kK;
  float* Mt = reinterpret_cast<float*>(tile(0));
  static_assert((kInvMtFloats + kInvScratchFloats) * 4 <= 2 * S::kTile, "M and the inverse's scratch");
  float* Mdg = reinterpret_cast<float*>(sm + S::oF);
  float* Adg = Mdg + 64 * kDm;
  float* betas2 = Adg + 64 * kDg;                      // of this chunk and the next
  float* Bb = betas2 + 128;
  float* Af = Bb + 512;
  ChunkAt* where = reinterpret_cast<ChunkAt*>(Af + 512);      // this chunk and the next
  CtaShared* cs = reinterpret_cast<CtaShared*>(where + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, b0 = (warp >> 2) * NB;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *in0 = &cs->bar[0], *in1 = &cs->bar[1], *m1 = &cs->bar[2], *m2 = &cs->bar[3], *m3 = &cs->bar[4];
  const int nchunks = p.nbh * p.cn;
  auto load_k = [&](const ChunkAt& a) {      // (one thread each)
    mbar_expect_tx(in0, 65536u);
    for (int t = 0; t < 2; ++t) tma_load_4d(tK + t * 8192, &mk, in0, t * 64, a.h, a.c * kC, a.b);
  };
  auto load_q = [&](const ChunkAt& a) {
    for (int t = 0; t < 2; ++t) tma_load_4d(tQ + t * 8192, &mq, in0, t * 64, a.h, a.c * kC, a.b);
  };
  auto load_g = [&](const ChunkAt& a) { tma_load_4d(tile(2), &mg, in0, 0, a.h, a.c * kC, a.b); };
  auto load_v = [&](const ChunkAt& a) {
    mbar_expect_tx(in1, V * 128u);
    for (int t = 0; t < V / 64; ++t) tma_load_4d(BV + t * 8192, &mv, in1, t * 64, a.h, a.c * kC, a.b);
  };
  if (tid == 0) {
    where[0] = chunk_at(p, blockIdx.x);
    cs->abort_flag = 0;
    for (int i = 0; i < 5; ++i) mbar_init(&cs->bar[i], i == 2 || i == 3 ? 2 : 1);
    fence_mbar_init();
    fence_proxy_async();
    load_k(where[0]);
    load_q(where[0]);
    load_g(where[0]);
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;      // M | A blocks; [w | u]; [P | R]

  // gates of a chunk, fetched while the chunk before is worked on: beta to shared memory; per channel to L2, by lines of 128 bytes
  auto fetch_gates = [&](const ChunkAt& a, float* betas) {
    const int last = p.rows_of(a.c) - 1;
    const size_t tok0 = (static_cast<size_t>(a.b) * p.L + a.c * kC) * p.H + a.h;
    if (FULL) {
      for (int t = tid; t < 256; t += kThreads) {
        const size_t tok = tok0 + static_cast<size_t>(t >> 2) * p.H;
        prefetch_l2(p.bch + tok * kK + (t & 3) * 32);
        prefetch_l2(p.wch + tok * V + (t & (V / 32 - 1)) * 32);
      }
    } else if (tid < 64) {
      async_copy4(betas + tid, p.beta + tok0 + static_cast<size_t>(min(tid, last)) * p.H, tid <= last);
    }
  };
  if (DELTA) fetch_gates(where[0], betas2);
  uint32_t ph = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const float* betas = betas2 + 64 * ph;
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    int d = quad * 32 + lane;                  // this thread's channel; addresses made from it are made anew in every phase
    auto anew = [&]() { asm volatile("" : "+r"(d)); };
    anew();
    auto token = [&](int r) {                  // row r of the chunk in the user's tensors
      const ChunkAt a = where[ph];
      return (static_cast<size_t>(a.b) * p.L + a.c * kC + r) * p.H + a.h;
    };
    auto rec = [&](size_t off, size_t size) { return p.saved + off + static_cast<size_t>(where[ph].z) * size; };

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
    if (DELTA && !FULL) async_copy_wait();
    if (tid == 0) bulk_wait_read();        // the chunk before has left tiles 4 and 5
    __syncthreads();
    if (NORM && tid == 0 && p.keep_norm) {
      const ChunkAt a = where[ph];
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
    if (tid == kThreads - 1 && more) where[ph ^ 1u] = chunk_at(p, n + gridDim.x);
    // ---- diagonal blocks, exact.  A half-warp has one block, a lane its channels 4 c .. 4 c + 3 of either half.  Work comes in two
    // kinds: the ten pairs of a group of four rows, and the sixteen of a group's rows with an earlier group, whose rows lie ready,
    // decayed to the end of their group.  A warp takes the same of either kind for its two blocks; a block's ten pieces are dealt
    // out by their length.
    {
      constexpr int kW = 16 / NB / 2;              // warps per two blocks
      const int db = 2 * (warp / kW) + (lane >> 4);
      int c = lane & 15;
      asm volatile("" : "+r"(c));
      const int w = NB == 2 ? (warp + 2 * (warp / kW)) & 3 : warp & 7;      // (the SM's quarters get the same)
      // own group of rows, or none; rows A with the earlier groups B, B - 1, ... (nB of them)
      const int own = NB == 2 || w < 4 ? w : -1;
      const int A = NB == 2 ? (w == 0 ? 3 : w == 1 ? 2 : w == 2 ? 3 : 1) : (w == 0 || w == 7 ? 2 : w == 1 ? 1 : 3);
      int B = NB == 2 ? (w == 0 ? 2 : w == 1 ? 1 : 0) : (w == 4 ? 2 : w == 5 || w == 7 ? 1 : 0);
      int nB = NB == 2 ? (w < 2 ? 2 : 1) : (w == 2 || w == 3 ? 0 : 1);
      const unsigned char* kt = tK + (c & 1) * 8;
      const unsigned char* qt = tQ + (c & 1) * 8;
      auto at16 = [&](int r) { return r * 128 + (((c >> 1) ^ (r & 7)) << 4); };
      auto row = [&](const unsigned char* t, int r, f2* x) {
        ld4_pairs<F16>(t + at16(r), x);
        ld4_pairs<F16>(t + 8192 + at16(r), x + 2);
      };
      auto row32 = [&](const float* x, int r, f2* y) {
        ld_pairs(x + r * kK + 4 * c, y);
        ld_pairs(x + r * kK + 64 + 4 * c, y + 2);
      };
      auto times = [&](f2* x, const f2* y) {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = mul2(x[e], y[e]);
      };
      auto erase = [&](int r, f2* x) {             // per-channel erase gate of the row
        const float* bp = p.bch + token(r) * kK + 4 * c;
        f2 b[4];
        ld_pairs(bp, b);
        ld_pairs(bp + 64, b + 2);
        times(x, b);
      };
      auto dot = [&](const f2* x, const f2* y) {
        f2 s = mul2(x[0], y[0]);
#pragma unroll
        for (int e = 1; e < 4; ++e) s = fma2(x[e], y[e], s);
        return sum2(s);
      };
      auto store = [&](int i, int s, bool is_m, float x) {
        const int r = db * 16 + i;
        if (is_m) Mdg[(db * 16 + s) * kDm + i] = FULL ? x : betas[r] * x;
        else Adg[r * kDg + s] = p.scale * x;
      };
      if (own >= 0) {
        f2 t[4][4];                                // source rows, decayed to the row in hand
        float v[16];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int rr = db * 16 + 4 * own + r;
          f2 q[4], k[4], a4[4];
          row(qt, rr, q);
          row(kt, rr, k);
          if (r) {
            row32(G, rr, a4);
#pragma unroll
            for (int s = 0; s < r; ++s) times(t[s], a4);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) t[r][e] = k[e];
          if (DELTA && FULL) erase(rr, k);
#pragma unroll
          for (int s = 0; s <= r; ++s) {
            v[r * (r + 1) / 2 + s] = dot(q, t[s]);
            if (s < r) v[10 + r * (r - 1) / 2 + s] = DELTA ? dot(k, t[s]) : 0.f;
          }
        }
        const float x = half_warp_sum<16>(v, lane);
        // lane c: rows and source rows of A's ten values, then of M's six, two bits each
        constexpr uint32_t kOwnRow = 0xfe9ffa94u, kOwnSrc = 0x910e4910u;
        const int r = static_cast<int>(kOwnRow >> (2 * c)) & 3, s = static_cast<int>(kOwnSrc >> (2 * c)) & 3;
        if (DELTA || c < 10) store(4 * own + r, 4 * own + s, c >= 10, x);
        if (DELTA && c < 10 && r == s) Mdg[(db * 16 + 4 * own + s) * kDm + 4 * own + s] = 0.f;
      }
      if (nB > 0) {
        f2 q[4][4], k[4][4], e4[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {              // the rows, decayed from the end of the group before theirs
          const int rr = db * 16 + 4 * A + r;
          row(qt, rr, q[r]);
          if (DELTA) row(kt, rr, k[r]);
          if (DELTA && FULL) erase(rr, k[r]);
          if (r == 0) {
            row32(G, rr, e4);
          } else {
            f2 a4[4];
            row32(G, rr, a4);
            times(e4, a4);
          }
          times(q[r], e4);
          if (DELTA) times(k[r], e4);
        }
        auto over = [&](int m) {                   // ... and over group m
          f2 g[4];
          row32(Bg, db * 4 + m, g);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            times(q[r], g);
            if (DELTA) times(k[r], g);
          }
        };
#pragma unroll 1
        for (int m = A - 1; m > B; --m) over(m);
#pragma unroll 1
        for (;;) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float v[16];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              f2 t[4];
              row32(kfd, db * 12 + 4 * B + 2 * h + u, t);
#pragma unroll
              for (int r = 0; r < 4; ++r) {
                v[8 * u + 2 * r] = dot(q[r], t);
                v[8 * u + 2 * r + 1] = DELTA ? dot(k[r], t) : 0.f;
              }
            }
            const float x = half_warp_sum<16>(v, lane);
            if (DELTA || !(c & 1)) store(4 * A + ((c >> 1) & 3), 4 * B + 2 * h + (c >> 3), c & 1, x);
          }
          if (--nB == 0) break;
          over(B--);
        }
      }
    }
    anew();
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
      if (blk == 3) reinterpret_cast<float*>(p.saved + p.lay.ad)[static_cast<size_t>(where[ph].z) * kK + d] = bd.pre * Bb[3 * kK + d];
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
        // columns: block 3's 48 and block 1's 16 in one tile, block 2's 32 in the other
        write_column(I == 2 ? KR2 : KR, I == 1 ? 3 : blk, d, y);
      }
      // scale gamma q leaves for its record, the image of a [64 tokens][128 channels] tile: a warp writes 64 bytes of a row
      unsigned char* qg = rec(p.lay.qg, 16384);
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
        if (FULL) {
          const float* bp = p.bch + token(blk * 16) * kK + d;
#pragma unroll
          for (int i = 0; i < 16; ++i) y[i] = bp[static_cast<size_t>(i) * p.H * kK];
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (i) e *= al[bb][i];
          x[i] = half_of(kp[bb][i >> 1], i & 1) * e;
          if (FULL) x[i] *= y[i];
        }
        write_column(LA, blk, d, x);             // left factor of M (without the row's beta)
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] *= FULL ? gam0 : gam0 * betas[blk * 16 + i];
        write_column(GK, blk, d, x);
      }
    }
    sync_for_issue();

    anew();
    // ---- off-diagonal blocks of M (rows 0-63) and A (rows 64-127) on the tensor cores
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(LA), 128, true}, Tile{smem_u32(KR), 128, true}, 64, 128, 0u);
      umma_commit_led(leader, m1);
    } else if (warp == 1) {                      // (two warps share the issue, some 45 cycles per product)
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem + 64, Tile{smem_u32(LA), 128, true}, Tile{smem_u32(KR2), 128, true}, 32, 128, 0u);
      umma_commit_led(leader, m1);
    } else if (warp == 2 && lane == 0 && more) {      // the next g and v to L2: g's tiles are free late, and v is wanted soon then
      const ChunkAt a = where[ph ^ 1u];
      tma_prefetch_4d(&mg, 0, a.h, a.c * kC, a.b);
      for (int t = 0; t < V / 64; ++t) tma_prefetch_4d(&mv, t * 64, a.h, a.c * kC, a.b);
    }
    __syncwarp();
    constexpr int kWv = 64 * (V / 8) / kThreads;
    float wv[FULL ? kWv : 1][8];               // write gates of this thread's pieces of v, requested in the products' shadow
    if (FULL)
#pragma unroll
      for (int j = 0; j < kWv; ++j) {
        const int idx = tid + j * kThreads;
        ld8(p.wch + token(idx / (V / 8)) * V + (idx % (V / 8)) * 8, wv[FULL ? j : 0]);
      }
    mbar_wait_warp(m1, ph, ctl, 502);
    tc_fence_after();
    if (tid == 0) load_v(where[ph]);
    if (DELTA && more) fetch_gates(where[ph ^ 1u], betas2 + 64 * (ph ^ 1u));
    // thread: accumulator lane quad * 32 + lane (row r of M for lanes 0-63, of A for 64-127), columns of block blk.  A warp's lanes are
    // rows of blocks I0 and I0 + 1.  Of M only the blocks below the diagonal ones go to Mt, which has it transposed.
    {
      const int r = d & 63, I = r >> 4, I0 = 2 * (quad & 1);
      auto col = [](int rb, int cb) { return rb == 1 ? 48 : (rb == 2 ? 64 : 0) + 16 * cb; };
#pragma unroll 1
      for (int blk = b0; blk < b0 + NB; ++blk) {
        float x[16];
        if (blk <= I0) {
          float y[16];
          tmem_ld16(tmem + lane_base + col(I0 + 1, blk), x);
          tmem_ld16(tmem + lane_base + col(I0, blk < I0 ? blk : 0), y);      // (not used for blk = I0)
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = I == I0 ? y[e] : x[e];
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = 0.f;
        }
        if (quad < 2) {
          if (DELTA && blk < I) {
            const float be = betas[r];
#pragma unroll
            for (int e = 0; e < 16; ++e) Mt[(blk * 16 + e) * kMt + r] = FULL ? x[e] : x[e] * be;
          }
        } else {
          if (blk < I) {
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] *= p.scale;
          } else if (blk == I) {
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = e <= (r & 15) ? Adg[r * kDg + e] : 0.f;
          } else if (blk > I) {
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = 0.f;
          }
          write_row16(TA, 64 + r, blk, x);
        }
      }
    }
    tc_fence_before();
    __syncthreads();

    anew();
    // ---- beta v (w v) on the warps that have no part in the inverse, or not in its first step
    constexpr int kFirst = FULL ? 0 : NB == 1 ? 256 : 64, kStep = kThreads - kFirst;
    if (tid >= kFirst) {
      mbar_wait_warp(in1, ph, ctl, 505);
#pragma unroll
      for (int j = 0; j < (64 * (V / 8) + kStep - 1) / kStep; ++j) {
        const int idx = tid - kFirst + j * kStep, r = idx / (V / 8), ch = idx % (V / 8);
        if (idx >= 64 * (V / 8)) break;
        float x[8];
        unpack8_bf16(tile_ld_chunk(BV, r, ch, 64), x);
        if (FULL) {
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] *= wv[FULL ? j : 0][i];
        } else if (DELTA) {
          const float be = betas[r];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] *= be;
        }
        tile_st_chunk(BV, r, ch, 64, pack8_f16(x));
      }
    }
    auto next_kq = [&]() {                 // tiles 0 and 1 are dead; by warps that have no part in the next step
      if (more && lane == 0 && warp == 2) load_k(where[ph ^ 1u]);
      if (more && lane == 0 && warp == 3) load_q(where[ph ^ 1u]);
      __syncwarp();
    };
    // ---- T = (I + M)^-1 (fp32, CUDA cores)
    if (DELTA) {
      unit_lower_inverse64<kDm, 16 * kDm>(Mt, Mdg, Mt + kInvMtFloats, TA, tid);
      sync_for_issue();
      next_kq();
      // ---- [w | u] = T [b gamma k | beta v]
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, tmem, Tile{smem_u32(TA), 128, false}, Tile{smem_u32(GK), 128, false}, 128, 64, 0u);
        umma_commit_led(leader, m2);
        if (tid == 0) {
          if (p.lean < 2) bulk_s2g(rec(p.lay.ta, p.lay.sz_ta), TA, 16384);
          else bulk_s2g(rec(p.lay.ta, p.lay.sz_ta) + 8192, TA + 8192, 8192);      // A only
          bulk_commit();
        }
      } else if (warp == 1) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, tmem + 128, Tile{smem_u32(TA), 128, false}, Tile{smem_u32(BV), 64, true}, V, 64, 0u);
        umma_commit_led(leader, m2);
      }
      __syncwarp();
      anew();
      mbar_wait_warp(m2, ph, ctl, 503);
      tc_fence_after();
      if (quad < 2) {                      // rows 0-63; the warps of a quadrant split the columns
#pragma unroll 1
        for (int jb = 2 * (warp >> 2); jb < (128 + V) / 32; jb += 8 / NB) {
          float x[64];
          tmem_ld32(tmem + lane_base + jb * 32, x);
          tmem_ld32(tmem + lane_base + jb * 32 + 32, x + 32);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) tile_st_chunk(WU, d, jb * 4 + i, 64, pack8_f16(x + 8 * i));
        }
      }
      if (tid == 0) bulk_wait_read();      // [T; A] has left tile 5
      sync_for_issue();
    } else {
      fence_proxy_async();
      __syncthreads();
      next_kq();
      if (tid == 0) {                      // A only: without the delta term nothing reads T
        bulk_s2g(rec(p.lay.ta, p.lay.sz_ta) + 8192, TA + 8192, 8192);
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
          bulk_s2g(rec(p.lay.w, p.lay.sz_w), WU, 16384);
          bulk_s2g(rec(p.lay.u, p.lay.sz_u), WU + 16384, V * 128);
        } else if (!p.lean) {            // (u is v)
          bulk_s2g(rec(p.lay.u, p.lay.sz_u), BV, V * 128);
        }
        bulk_commit();
      }
    }
    __syncwarp();
    anew();
    mbar_wait_warp(m3, ph, ctl, 504);
    tc_fence_after();
    if (tid == 0 && more) {                // tiles 2 and 3 are dead once their records have left
      bulk_wait_read();
      load_g(where[ph ^ 1u]);
    }
    // P leaves as its record image through the tiles of the last operands, R (16 columns of a row are 32 bytes of its record,
    // the rows of a warp 1 KB) directly; the warps of a lane quadrant split the columns
    unsigned char* r_g = rec(p.lay.r, p.lay.sz_r);
#pragma unroll 1
    for (int jb = 2 * (warp >> 2); jb < (DELTA ? 128 + V : V) / 32; jb += 8 / NB) {
      float x[64];
      tmem_ld32(tmem + lane_base + jb * 32, x);
      tmem_ld32(tmem + lane_base + jb * 32 + 32, x + 32);
      tmem_ld_wait();
      if (!DELTA || jb < 4) {              // P; R without the delta term, a plain tile image
#pragma unroll
        for (int i = 0; i < 8; ++i) tile_st_chunk(SP, d, jb * 4 + i, 128, pack8_f16(x + 8 * i));
      } else {
        const int c8 = (jb - 4) * 4;
#pragma unroll
        for (int i = 0; i < 8; i += 2) st_global_32(r_g + rrec_off(d, c8 + i), pack8_f16(x + 8 * i), pack8_f16(x + 8 * i + 8));
      }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      if (DELTA) bulk_s2g(rec(p.lay.p, p.lay.sz_p), SP, 32768);
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

// Two value sizes, three forms of the op, three of the inputs and two of the grid are 36 kernels: the half with 128 value channels is
// compiled from gdn_cw_fwd_v128.cu, which includes this file (whole build on eight cores 53 s in one piece, 29 s like this).
int launch_prepare_cw_v128(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                           const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st)
#ifdef LETHE_CW_FWD_V128
{
  return launch_prepare_cw_v<128>(p, mq, mk, mv, mg, mn, st);
}
#else
;
int launch_prepare_cw(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                      const CUtensorMap& mg, const NormMaps& mn, cudaStream_t st) {
  return p.V == 64 ? launch_prepare_cw_v<64>(p, mq, mk, mv, mg, mn, st) : launch_prepare_cw_v128(p, mq, mk, mv, mg, mn, st);
}
#endif

}  // namespace lg
