// Channel-wise gate: the chunk-parallel backward after the adjoint state scan, one kernel for Stage B and the WY /
// triangular-inverse VJP.  With v_new, h (state entering the chunk), dh (adjoint of the state leaving it) and
// ratio(i, s)[d] the decay of channel d from token s to token i:
//
//   dv2  = kd dh + A^T do                         dA = do v_new^T,  C0 = scale tril(dA)
//   dw   = -dv2 h^T                               dbv = T^T dv2,  dbgk = T^T dw
//   C1 = dM = strict_lower(-(dbv u^T + dbgk w^T)),  u = T (w v), w = T (b gamma k)       (the forward's WY factors)
//   out1_c[i,d] = sum_{s<=i} C_c[i,s] k[s,d] ratio(i,s)[d]
//   out2[s,d]   = sum_{i>=s} (C0[i,s] q[i,d] + C1[i,s] (b k)[i,d]) ratio(i,s)[d]
//   dq = scale gamma (do h^T) + out1_0            dbk = gamma dbgk + out1_1
//   dk' = de (v_new dh^T) + out2                  dk = dk' + b dbk
//   dv = w dbv,  db = dbk k,  dw_gate = dbv v     dG = q dq + (b k) dbk - k dk'   (+ the chunk's end term)
//   dg = reverse cumulative sum of dG
//
// Reference: closed channel-wise Stage B gdn2_assemble.py:521-585, channel-wise K#2 gdn2_assemble.py:407-473, the SIMT
// kernel gdn2_sb_einsum.py:44-76 for the decay-coupled sums.
//
// Layout.  Every result that has a feature axis is computed TRANSPOSED: its accumulator has the 128 key (or value)
// channels in the tensor-memory lanes and the 64 tokens in the columns.  That uses all 128 rows of the products, and
// thread (block of 16 tokens, channel) - 512 of them - then owns a 16-token column of everything: gates, k, q, the
// accumulators, the exact diagonal sums and the final gradients meet in its registers.  Nothing is exchanged between
// threads but per-block decay products and a few row sums.  Operands the threads build are stored transposed too
// ([channel][token] tiles, two 16-byte stores per thread); a tile serves K-major or MN-major.
//
// Decays.  alpha_i = exp(g_i) is the only exponential (16 per thread); every ratio is a product of alphas between its
// two tokens, so each factor is <= 1 and >= the ratio: nothing overflows and nothing vanishes before the ratio does.
// Off-diagonal 16 x 16 blocks (I, J), I > J, of the pair sums go through the tensor cores as (k f_J) and (x e_I) -
// decayed to the end of block J and from the start of block I - into an accumulator per block pair, and the decay
// between the two, one number per channel, is applied in fp32 by the thread that reads it.  The diagonal blocks are
// exact fp32 recurrences: going down the rows, k[s] ratio(i,s) is multiplied by alpha_i per row; going up, the column
// sums are (Horner).  No exponentials, one packed multiply and two packed FMAs per two pairs and sum.
//
// dM.  The VJP of the inverse is -T^T dT T^T with dT = dv2 (w v)^T + dw (b gamma k)^T; since T^T dv2 = dbv, T^T dw = dbgk, T (w v)
// = u and T (b gamma k) = w, that is -(dbv u^T + dbgk w^T): one product behind dbv and dbgk, which are wanted anyway, instead of
// three in a row, for 32 KB more to read per chunk.  Its error, and that v_new is to be made of the same u and w: gdn_bwd_main.cu.
//
// What bounds it: the chain of four dependent product groups and the CUDA-core phases (issue slots 43 % busy); 300 KB of traffic
// per chunk are 12 k cycles of an SM's share of HBM.  The CTA is persistent and fetches the next chunk's tiles into the ones that
// are dead once its last products are issued, under the longest CUDA-core phase.  Inside a group the products that the chain waits
// for are issued first and the rest of the epilogue before lies in the next group's shadow.
// us at d_v = 128, before (dT, X = dT T^T and dM as three groups, 88 to 440 bytes a thread of spilled loads, 0 to 48 now, all copies
// issued by one thread, beta and the per-channel gates read when they were needed) and then: 8192 chunks 920 -> 789 (773 with the abort flag behind the waits); 4096 without the
// delta term 301 -> 267; 512 with per-channel gates 113 -> 79.
// Cycles per chunk by clock samples of one CTA (d_v = 128): operand columns and waits for the tiles 4.9 k, group 1 2.5 k, the rest
// up to dM 7.0 k, column sums with the decay assembly 5.0 k, row sums with the gradients 5.6 k, gate gradient and stores 2.2 k; 27.1 k
// in all.  Without the delta term 5.1, 3.1, 0.6, 3.5, 2.8, 1.7: 16.8 k; with per-channel gates 30.9 k.
#include "gdn_cw.cuh"
#include "host_util.h"

namespace lg {

constexpr int kCwThreads = 512;

struct CwBars {
  uint64_t in0, in1, inU, mA, mB, mW, mV, mX, mO;
  uint32_t tmem_slot;
  int abort_flag;
};

// What runs in a launch.  A call that is cut between Stage B and the WY VJP (kernel_mask 4, then 8) gives the bits of the
// uncut one: the first half leaves its product results, the second half forms all sums from them.
enum CwMode {
  kCwAll,        // the backward with the delta term
  kCwNoDelta,    // without it: no WY half
  kCwStageB,     // the products of Stage B; leaves dv2, dw, do h^T (in DGB), v_new dh^T (in DKB), C0 and the end terms
                 // (in RB, which nothing reads after the adjoint scan)
  kCwWy          // everything after them, from those records
};
constexpr int kRecDiag = 8192, kRecEnd = kRecDiag + 4096;     // RB: C0 as a 64-row tile, its diagonal blocks, end terms
__device__ __forceinline__ size_t rec_at(int i, int d) { return static_cast<size_t>(i) * kK + d; }    // DGB, DKB: fp32 [64][128]

template <int V, bool WY>
struct CwSmem {
  static constexpr int kVT = V * 128;                    // a [64 tokens][V] or [V][64 tokens] tile
  static constexpr int oK = 0;                           // k as loaded; then k f            [channel][token]
  static constexpr int oQ = oK + 16384;                  // q as loaded; then q e
  static constexpr int oV = oQ + 16384;                  // v (without delta: v_new)         token-major
  static constexpr int oG = oV + kVT;                    // g as loaded (32 KB); then kd, then dw | WY factor w
  static constexpr int oDO = oG + 32768;                 // do                               token-major
  static constexpr int oDV = oDO + kVT;                  // dv2  [value channel][token]; then dv on its way out
  static constexpr int oTA = oDV + kVT;                  // [T; A]
  static constexpr int oC = oTA + 16384;                 // v_new; then C0 / C1 by row block; then dq on its way out
  static constexpr int oH = oC + 16384;                  // h; then T^T dw, T^T dv2 [channel][token]; then dg on its way out
  static constexpr int oDH = oH + 32768;                 // dh; then (b k) e (16 KB), WY factor u; then dk on its way out
  static constexpr int kDH = 16384 + kVT;
  static constexpr int oCd = oDH + kDH;                  // diagonal blocks of C0, C1 in fp32: [2][64][16]
  static constexpr int oF = oCd + 8192;                  // floats: Bb [4][128], Af [4][128], Et [4][128], red [2][4][64], betas [2][64]
  static constexpr int kFloats = 3 * 512 + 512 + 128;
  static constexpr int kBytes = oF + kFloats * 4 + static_cast<int>(sizeof(CwBars)) + 2 * static_cast<int>(sizeof(ChunkAt)) + 1024;
  static constexpr int CR = WY ? 32 : 16;        // rows of the C tile per row block
};

// FULL: per-channel erase and write gates (a compile-time choice: a branch on it in every row of the pair sums kept the
// compiler from overlapping one row with the next, 8.9 k cycles per chunk instead of the 2.9 k of one sum)
template <int V, CwMode MODE, bool FULL>
__global__ void __launch_bounds__(kCwThreads, 1)
bwd_cw_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
              const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mdo,
              const __grid_constant__ CUtensorMap mg, const __grid_constant__ CwOutMaps mo) {
  constexpr bool SB = MODE != kCwWy, WY = MODE == kCwAll || MODE == kCwWy, DELTA = MODE != kCwNoDelta;
  constexpr bool CUT = MODE == kCwStageB || MODE == kCwWy;
  using S = CwSmem<V, WY>;
  constexpr int CR = S::CR;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  unsigned char *tK = sm + S::oK, *tQ = sm + S::oQ, *tV = sm + S::oV, *tKD = sm + S::oG, *tW = sm + S::oG + 16384;
  unsigned char *tDW = tKD, *tDO = sm + S::oDO, *tDV = sm + S::oDV, *tTA = sm + S::oTA, *tVN = sm + (DELTA ? S::oC : S::oV), *tC = sm + S::oC;
  unsigned char *oQt = tC, *oKt = sm + S::oDH, *oVt = tDV;
  float* oGt = reinterpret_cast<float*>(sm + S::oH);
  unsigned char *tH = sm + S::oH, *tDH = sm + S::oDH, *tBE = sm + S::oDH, *tU = sm + S::oDH + 16384;
  unsigned char *tBK = tH, *tBV = tH + 16384;
  const float* G = reinterpret_cast<const float*>(sm + S::oG);
  float* Cd0 = reinterpret_cast<float*>(sm + S::oCd);
  float* Cd1 = Cd0 + 1024;
  float* Bb = reinterpret_cast<float*>(sm + S::oF);      // products of a block's alphas
  float* Af = Bb + 512;                                  // first alpha of a block
  float* Et = Af + 512;                                  // a block's part of the end term
  float* St = reinterpret_cast<float*>(tU);              // gate-gradient totals of a block, once u is dead
  float* red = Et + 512;
  float* betas2 = red + 512;                             // of this chunk and the next
  ChunkAt* where = reinterpret_cast<ChunkAt*>(betas2 + 128);      // this chunk and the next
  CwBars* bars = reinterpret_cast<CwBars*>(where + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, blk = warp >> 2;
  CtaCtl ctl{p.status, &bars->abort_flag};
  const int nchunks = p.nbh * p.cn;
  // The loads of a chunk, in parts by when their destinations are free in the chunk before, and its stores are shared by four
  // threads, the first of every block's warps: one thread would issue for some 1 k cycles while the others wait for it.  A tile
  // that a store reads is loaded by the thread that issued the store.
  const bool lead = (warp & 3) == 0 && lane == 0;
  auto load_part1 = [&](const ChunkAt& a) {
    const int l0 = a.c * kC;
    if (blk == 0) {
      mbar_expect_tx(&bars->in0, 32768u + 16384u + 16384u);
      mbar_expect_tx(&bars->in1, (SB ? 2u * V * 128 + 2u * V * 256 : 0u) + (DELTA ? 16384u : 8192u) + (WY ? V * 128u : 0u));
      tma_load_4d(sm + S::oG, &mg, &bars->in0, 0, a.h, l0, a.b);
    } else if (blk == 1) {
      if (WY || !DELTA) for (int t = 0; t < V / 64; ++t) tma_load_4d(tV + t * 8192, &mv, &bars->in1, t * 64, a.h, l0, a.b);
    } else if (blk == 2) {
      if (DELTA) bulk_g2s(tTA, p.saved + p.lay.ta + static_cast<size_t>(a.z) * 16384, 16384, &bars->in1);
      else bulk_g2s(tTA + 8192, p.saved + p.lay.ta + static_cast<size_t>(a.z) * 16384 + 8192, 8192, &bars->in1);
    } else if (SB) {
      for (int t = 0; t < V / 64; ++t) tma_load_4d(tDO + t * 8192, &mdo, &bars->in1, t * 64, a.h, l0, a.b);
    }
  };
  auto load_part2 = [&](const ChunkAt& a) {
    for (int t = 0; t < 2; ++t) {
      if (blk == 2) tma_load_4d(tK + t * 8192, &mk, &bars->in0, t * 64, a.h, a.c * kC, a.b);
      if (blk == 3) tma_load_4d(tQ + t * 8192, &mq, &bars->in0, t * 64, a.h, a.c * kC, a.b);
    }
  };
  auto load_rec = [&](const ChunkAt& a) {      // v_new, h
    if (blk == 0 && DELTA) bulk_g2s(tVN, p.saved + p.lay.vn + static_cast<size_t>(a.z) * p.lay.sz_vn, V * 128, &bars->in1);
    if (blk == 2) bulk_g2s(tH, p.saved + p.lay.hc + static_cast<size_t>(a.z + a.b * p.H + a.h) * p.lay.sz_hc, V * 256, &bars->in1);
  };
  auto load_dh = [&](const ChunkAt& a) {
    if (blk == 1) bulk_g2s(tDH, p.scratch + p.lay.dh + static_cast<size_t>(a.z) * p.lay.sz_dh, V * 256, &bars->in1);
  };

  if (tid == 0) {
    where[0] = chunk_at(p, blockIdx.x);
    bars->abort_flag = 0;
    mbar_init(&bars->in0, 1); mbar_init(&bars->in1, 1); mbar_init(&bars->inU, 1); mbar_init(&bars->mA, 1); mbar_init(&bars->mB, 1);
    mbar_init(&bars->mW, 1); mbar_init(&bars->mV, 1); mbar_init(&bars->mX, 1); mbar_init(&bars->mO, 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (lead) {
    // Older than whatever kernel of the path comes just before this one: the caller's tensors and [T; A].  v_new (the output
    // kernel) and h (the forward scan) only where this call has put the adjoint scan in between; with kernels picked one by one
    // any of the three may be the last.  (Late everywhere: SSD forward and backward 175.1 us instead of 172.3 at 1692 chunks, 557.8
    // instead of 555.3 at 4096; with the delta term no difference.)
    if (SB) {
      const ChunkAt a = where[0];
      load_part1(a);
      load_part2(a);
      if (p.after_scan) load_rec(a);
    }
  }
  const uint32_t tmem = bars->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  // accumulators, [lane = channel][column = token] except dA and dM ([token][token], lanes 0-63); what shares
  // columns has been read before it is overwritten
  const uint32_t cDV = tmem, cDA = tmem + 64, cDQ = tmem + 128, cDWt = tmem + 192, cDK = tmem + 256, cO1 = tmem + 320;
  const uint32_t cDBV = tmem, cT = tmem + 64, cDBK = tmem + 192, cO2 = tmem;
  griddep_wait();
  griddep_launch();
  if (lead) {
    const ChunkAt a = where[0];
    if (SB) {
      if (!p.after_scan) load_rec(a);
      load_dh(a);
    } else {
      load_part1(a);
      load_part2(a);
    }
  }
  const uint32_t aK = smem_u32(tK), aQ = smem_u32(tQ), aC = smem_u32(tC), aBE = smem_u32(tBE);

  // gates of a chunk, fetched while the chunk before is worked on: beta to shared memory; per channel to L2, a line of 128 bytes a thread
  auto fetch_gates = [&](const ChunkAt& a, float* betas) {
    const int t = tid & 255, r = FULL ? t >> 2 : tid, last = p.rows_of(a.c) - 1;
    const size_t tok = (static_cast<size_t>(a.b) * p.L + a.c * kC + min(r, last)) * p.H + a.h;
    if (FULL) prefetch_l2(tid < 256 ? p.bch + tok * kK + (t & 3) * 32 : p.wch + tok * V + (t & (V / 32 - 1)) * 32);
    else if (tid < 64) async_copy4(betas + tid, p.beta + tok, r <= last);
  };
  if (WY) fetch_gates(where[0], betas2);
  uint32_t ph = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const float* betas = betas2 + 64 * ph;
    int d = quad * 32 + lane;                       // this thread's channel
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    auto token = [&](int r) {                       // row r of the chunk in the user's tensors
      const ChunkAt a = where[ph];
      return (static_cast<size_t>(a.b) * p.L + a.c * kC + r) * p.H + a.h;
    };

    // ---- this thread's column: decays, k, q
    float al[16];
    uint32_t kp[8], qp[8];
    // Between two phases: what the compiler has made from the channel (tile addresses) and from k and q (fp32 values) is made anew
    // in the next one; kept, it goes to local memory, which misses L1 beside 226 KB of shared memory (88 to 440 bytes a thread; 16 to
    // 48 are left in the instantiations with the delta term or without a WY half, none in Stage B by itself).
    auto anew = [&]() {
      asm volatile("" : "+r"(d));
#pragma unroll
      for (int j = 0; j < 8; ++j) asm volatile("" : "+r"(kp[j]), "+r"(qp[j]));
    };
    mbar_wait_warp(&bars->in0, ph, ctl, 601);
#pragma unroll
    for (int i = 0; i < 16; ++i) al[i] = exp2f(G[(blk * 16 + i) * kK + d] * kLog2e);
    read_column(tK, blk, d, p.qk16, kp);
    read_column(tQ, blk, d, p.qk16, qp);
    {
      float B = 1.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) B *= al[i];
      Bb[blk * kK + d] = B;
      Af[blk * kK + d] = al[0];
    }
    if (WY && !FULL) async_copy_wait();
    if (lead && n != static_cast<int>(blockIdx.x)) {
      bulk_wait_read();                             // the results of the chunk before have left their tiles
      if (SB) {
        load_rec(where[ph]);
        load_dh(where[ph]);
      }
    }
    __syncthreads();          // the raw tiles are read, the block products are there
    if (WY && tid == 0) {
      mbar_expect_tx(&bars->inU, 16384u + V * 128u);
      bulk_g2s(tW, p.saved + p.lay.w + static_cast<size_t>(where[ph].z) * 16384, 16384, &bars->inU);
      if (!SB) bulk_g2s(tU, p.saved + p.lay.u + static_cast<size_t>(where[ph].z) * p.lay.sz_u, V * 128, &bars->inU);
    }
    auto kv = [&](int i) { return half_of(kp[i >> 1], i & 1); };
    auto qv = [&](int i) { return half_of(qp[i >> 1], i & 1); };
    uint32_t bkp[FULL ? 8 : 1];                     // b k
    if (FULL) {
      const float* bg = p.bch + token(blk * 16) * kK + d;
      float b[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) b[i] = bg[static_cast<size_t>(i) * p.H * kK];
#pragma unroll
      for (int j = 0; j < 8; ++j) bkp[FULL ? j : 0] = f16x2_sat(kv(2 * j) * b[2 * j], kv(2 * j + 1) * b[2 * j + 1]);
    }
    auto bkv = [&](int i) { return FULL ? half_of(bkp[FULL ? i >> 1 : 0], i & 1) : kv(i) * betas[blk * 16 + i]; };
    // ---- operand tiles
    {
      float x[16], e = 1.f, f = 1.f;
#pragma unroll
      for (int i = 15; i >= 0; --i) {
        x[i] = kv(i) * f;
        f *= al[i];
      }
      write_column(tK, blk, d, x);
      if (SB) {
        const float post = block_decays(Bb, Af, blk, d).post;
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] *= post;
        write_column(tKD, blk, d, x);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i) e *= al[i];
        x[i] = qv(i) * e;
      }
      write_column(tQ, blk, d, x);
    }
    anew();
    mbar_wait_warp(&bars->in1, ph, ctl, 602);
    if (SB) {
      for (int idx = tid; idx < 64 * (V / 8); idx += kCwThreads) {
        const int r = idx / (V / 8), ch = idx % (V / 8);
        float x[8];
        unpack8_bf16(tile_ld_chunk(tDO, r, ch, 64), x);
        tile_st_chunk(tDO, r, ch, 64, pack8_f16(x));
        if (!DELTA) {
          unpack8_bf16(tile_ld_chunk(tVN, r, ch, 64), x);
          tile_st_chunk(tVN, r, ch, 64, pack8_f16(x));
        }
      }
    }
    // records of a call that is cut, or that keeps everything
    auto rec = [&](size_t off, size_t size) { return p.scratch + off + static_cast<size_t>(where[ph].z) * size; };
    auto rec32 = [&](size_t off, size_t size) { return reinterpret_cast<float*>(rec(off, size)); };
    const bool keep = CUT || !p.lean;
    if (!SB) {      // the first half of the call left dv2 and dw as token-major records
      const unsigned char *dw_g = rec(p.lay.dw, p.lay.sz_dw), *dv2_g = rec(p.lay.dv2, p.lay.sz_dv2), *rb_g = rec(p.lay.rb, p.lay.sz_rb);
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = __half2float(*reinterpret_cast<const __half*>(dw_g + sw128_off(blk * 16 + i, d, 64)));
      write_column(tDW, blk, d, x);
      if (d < V) {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = __half2float(*reinterpret_cast<const __half*>(dv2_g + sw128_off(blk * 16 + i, d, 64)));
        write_column(tDV, blk, d, x);
      }
      if (quad < 2) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          tile_st_chunk(tC, (d >> 4) * CR + (d & 15), 2 * blk + j, 64,
                        *reinterpret_cast<const uint4*>(rb_g + sw128_chunk(d, 2 * blk + j, 64)));
      }
      for (int idx = tid; idx < 1024; idx += kCwThreads) Cd0[idx] = reinterpret_cast<const float*>(rb_g + kRecDiag)[idx];
      Et[blk * kK + d] = reinterpret_cast<const float*>(rb_g + kRecEnd)[blk * kK + d];
    }
    sync_for_issue();

    if (tid == kCwThreads - 1 && more) where[ph ^ 1u] = chunk_at(p, n + gridDim.x);
    // ---- group 1: dv2^T, dA; (v_new dh^T)^T; dq_inter^T.  What the chain needs first is issued first.
    if (SB) {
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cDV, Tile{smem_u32(tDH), 128, true}, Tile{smem_u32(tKD), 128, true}, 64, 128, 0u);
        issue_product_led(leader, cDV, Tile{smem_u32(tDO), 64, true}, Tile{smem_u32(tTA) + 8192, 64, true}, 64, 64, 1u);
        umma_commit_led(leader, &bars->mA);
        issue_product_led(leader, cDA, Tile{smem_u32(tDO), 64, false}, Tile{smem_u32(tVN), 64, false}, 64, V, 0u);
        issue_product_led(leader, cDK, Tile{smem_u32(tDH), 128, false}, Tile{smem_u32(tVN), 64, false}, 64, V, 0u);
        if (MODE == kCwAll) umma_commit_led(leader, &bars->mB);
        issue_product_led(leader, cDQ, Tile{smem_u32(tH), 128, false}, Tile{smem_u32(tDO), 64, false}, 64, V, 0u);
        if (MODE != kCwAll) umma_commit_led(leader, &bars->mB);
      }
      __syncwarp();
      // in their shadow: this block's quarter of <dh, h> of channel d (both images are only read)
      float endt = 0.f;
#pragma unroll
      for (int q = 0; q < V / 32; ++q) {
        float x[8], y[8];
        unpack8_f16(tile_ld_chunk(tDH, d, blk * (V / 32) + q, 128), x);
        unpack8_f16(tile_ld_chunk(tH, d, blk * (V / 32) + q, 128), y);
#pragma unroll
        for (int e = 0; e < 8; ++e) endt = fmaf(x[e], y[e], endt);
      }
      const BlockDecays bd = block_decays(Bb, Af, blk, d);
      endt *= bd.pre * Bb[blk * kK + d] * bd.post;  // exp(G_last) <dh, h>
      anew();
      mbar_wait_warp(&bars->mA, ph, ctl, 603);
      tc_fence_after();
      if (d < V) {
        float x[16];
        tmem_ld16(cDV + lane_base + blk * 16, x);
        tmem_ld_wait();
        if (DELTA) {
          write_column(tDV, blk, d, x);
          if (keep) {
            unsigned char* dv2_g = rec(p.lay.dv2, p.lay.sz_dv2);
#pragma unroll
            for (int i = 0; i < 16; ++i) store_f16_sat(dv2_g + sw128_off(blk * 16 + i, d, 64), x[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) stage16(oVt, blk * 16 + i, d, x[i], 0);
        }
      }
      // ---- group 2: dw^T = -h dv2^T, and T^T dv2
      if (DELTA) {
        sync_for_issue();
        if (warp == 0) {
          tc_fence_after();
          const uint32_t leader = elect_leader();
          issue_product_led(leader, cDWt, Tile{smem_u32(tH), 128, false}, Tile{smem_u32(tDV), V, true}, 64, V, 0u);
          if (WY) issue_product_led(leader, cDBV, Tile{smem_u32(tDV), V, false}, Tile{smem_u32(tTA), 64, true}, 64, 64, 0u);
          umma_commit_led(leader, &bars->mW);
        }
        __syncwarp();
      }
      // in its shadow: the rest of the end term, C0, (b k) e
      mbar_wait_warp(&bars->mB, ph, ctl, 604);      // v_new and dh are dead from here on
      tc_fence_after();
      if (WY && tid == 0) bulk_g2s(tU, p.saved + p.lay.u + static_cast<size_t>(where[ph].z) * p.lay.sz_u, V * 128, &bars->inU);
      {
        float x[16], f = bd.post;
        tmem_ld16(cDK + lane_base + blk * 16, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 15; i >= 0; --i) {             // + sum_i k (v_new dh^T) exp(G_last - G_i)
          endt = fmaf(x[i] * kv(i), f, endt);
          f *= al[i];
        }
        Et[blk * kK + d] = endt;
        if (MODE == kCwStageB) {
          float *dkb_g = rec32(p.lay.dkb, p.lay.sz_dkb), *dgb_g = rec32(p.lay.dgb, p.lay.sz_dgb);
#pragma unroll
          for (int i = 0; i < 16; ++i) dkb_g[rec_at(blk * 16 + i, d)] = x[i];
          reinterpret_cast<float*>(rec(p.lay.rb, p.lay.sz_rb) + kRecEnd)[blk * kK + d] = endt;
          tmem_ld16(cDQ + lane_base + blk * 16, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) dgb_g[rec_at(blk * 16 + i, d)] = x[i];
        }
      }
      if (quad < 2) {                               // C0 = scale tril(dA): row i, columns of block blk
        const int i = d, ib = i >> 4;
        float x[16];
        tmem_ld16(cDA + lane_base + blk * 16, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = (blk * 16 + j <= i) ? p.scale * x[j] : 0.f;
        write_row16(tC, ib * CR + (i & 15), blk, x);
        if (ib == blk) {
          st8(Cd0 + i * 16, x);
          st8(Cd0 + i * 16 + 8, x + 8);
        }
        if (MODE == kCwStageB) {
          unsigned char* rb_g = rec(p.lay.rb, p.lay.sz_rb);
          write_row16(rb_g, i, blk, x);
          if (ib == blk) {
            st8(reinterpret_cast<float*>(rb_g + kRecDiag) + i * 16, x);
            st8(reinterpret_cast<float*>(rb_g + kRecDiag) + i * 16 + 8, x + 8);
          }
        }
      }
    } else if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, cDBV, Tile{smem_u32(tDV), V, false}, Tile{smem_u32(tTA), 64, true}, 64, 64, 0u);
      umma_commit_led(leader, &bars->mW);
    }
    __syncwarp();
    if (WY) {                                       // (b k) e, where dh was
      float x[16], e = 1.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        if (i) e *= al[i];
        x[i] = bkv(i) * e;
      }
      write_column(tBE, blk, d, x);
    }
    anew();
    if (DELTA) {
      mbar_wait_warp(&bars->mW, ph, ctl, 605);      // h is dead from here on
      tc_fence_after();
    }
    if (SB && DELTA) {
      float x[16];
      tmem_ld16(cDWt + lane_base + blk * 16, x);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = -x[i];
      if (WY) write_column(tDW, blk, d, x);
      if (keep) {
        unsigned char* dw_g = rec(p.lay.dw, p.lay.sz_dw);
#pragma unroll
        for (int i = 0; i < 16; ++i) store_f16_sat(dw_g + sw128_off(blk * 16 + i, d, 64), x[i]);
      }
    }
    if (WY) {
      if (d < V) {
        float x[16];
        tmem_ld16(cDBV + lane_base + blk * 16, x);
        tmem_ld_wait();
        write_column(tBV, blk, d, x);
      }
      mbar_wait_warp(&bars->inU, ph, ctl, 606);
      sync_for_issue();
      // ---- group 3: T^T dw; the first part of dM = -(dbv u^T + dbgk w^T)
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cDBK, Tile{smem_u32(tDW), 128, false}, Tile{smem_u32(tTA), 64, true}, 64, 64, 0u);
        umma_commit_led(leader, &bars->mV);
        issue_product_led(leader, cT, Tile{smem_u32(tBV), V, true}, Tile{smem_u32(tU), 64, false}, 64, V, 0u, true);
      }
      __syncwarp();
      if (more) fetch_gates(where[ph ^ 1u], betas2 + 64 * (ph ^ 1u));
      mbar_wait_warp(&bars->mV, ph, ctl, 607);
      tc_fence_after();
      {
        float x[16];
        tmem_ld16(cDBK + lane_base + blk * 16, x);
        tmem_ld_wait();
        write_column(tBK, blk, d, x);
      }
      sync_for_issue();
      // ---- group 4: the second part
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cT, Tile{smem_u32(tBK), 128, true}, Tile{smem_u32(tW), 64, false}, 64, 128, 1u, true);
        umma_commit_led(leader, &bars->mX);
      }
      __syncwarp();
      anew();
      // in its shadow: dv and the value part of the gate gradients
      if (d < V) {
        float x[16], wv[FULL ? 16 : 1];
        const size_t step = static_cast<size_t>(p.H) * V, first = FULL ? token(blk * 16) * V + d : 0;
        if (FULL)
#pragma unroll
          for (int i = 0; i < 16; ++i) wv[FULL ? i : 0] = p.wch[first + i * step];
        uint32_t vp[8];
        read_column(tV, blk, d, 0, vp);
        tmem_ld16(cDBV + lane_base + blk * 16, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          f2 g, y = pack2(x[2 * j], x[2 * j + 1]);
          if (FULL) g = pack2(wv[FULL ? 2 * j : 0], wv[FULL ? 2 * j + 1 : 0]);
          else g.u = *reinterpret_cast<const unsigned long long*>(betas + blk * 16 + 2 * j);
          stage16_two(oVt, blk * 16 + 2 * j, d, mul2(g, y), 0);
          unpack2(mul2(y, pair_of(vp[j])), x[2 * j], x[2 * j + 1]);
        }
        if (FULL) {
#pragma unroll
          for (int i = 0; i < 16; ++i) p.dwch[first + i * step] = x[i];
        } else {
          const float s0 = warp_sum8(x, lane), s1 = warp_sum8(x + 8, lane);
          if ((lane & 3) == 0) {
            red[256 + quad * 64 + blk * 16 + (lane >> 2)] = s0;
            red[256 + quad * 64 + blk * 16 + 8 + (lane >> 2)] = s1;
          }
        }
      }
      mbar_wait_warp(&bars->mX, ph, ctl, 609);
      tc_fence_after();
      if (quad < 2) {
        const int i = d, ib = i >> 4;
        float x[16];
        tmem_ld16(cT + lane_base + blk * 16, x);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) x[j] = (blk * 16 + j < i) ? x[j] : 0.f;
        write_row16(tC, ib * CR + 16 + (i & 15), blk, x);
        if (ib == blk) {
          st8(Cd1 + i * 16, x);
          st8(Cd1 + i * 16 + 8, x + 8);
        }
      }
      sync_for_issue();
    }

    if (!DELTA) sync_for_issue();
    if (MODE == kCwStageB) {
      sync_for_issue();
      if (lead && more) {
        load_part1(where[ph ^ 1u]);
        load_part2(where[ph ^ 1u]);
      }
      continue;
    }
    if (tid == 0) {                                 // dv (written before the last barrier)
      const ChunkAt a = where[ph];
      for (int t = 0; t < V / 64; ++t) tma_store_4d(&mo.dv, oVt + t * 8192, t * 64, a.h, a.c * kC, a.b);
      bulk_commit();
    }
    // ---- pair sums of the off-diagonal blocks, one accumulator per block pair.  out1: for source block J the rows of
    // all later blocks are neighbours in the C tile; out2: for row block I the columns of all earlier ones are.
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      constexpr uint32_t kAcc1[3] = {0, 3 * CR, 5 * CR};
#pragma unroll
      for (int J = 0; J < 3; ++J)
        umma_led(leader, cO1 + kAcc1[J], make_desc(aK + 32 * J, 16u, 1024u), make_desc(aC + (J + 1) * CR * 128 + 32 * J, 16u, 1024u),
                 make_idesc(128, (3 - J) * CR, false, false), 0u);
      constexpr uint32_t kAcc2[3] = {0, 16, 48};
#pragma unroll
      for (int I = 1; I < 4; ++I) {
        const uint32_t rowsI = aC + I * CR * 128, idesc = make_idesc(128, 16 * I, false, true);
        umma_led(leader, cO2 + kAcc2[I - 1], make_desc(aQ + 32 * I, 16u, 1024u), make_desc(rowsI, 8192u, 1024u), idesc, 0u);
        if (WY)
          umma_led(leader, cO2 + kAcc2[I - 1], make_desc(aBE + 32 * I, 16u, 1024u), make_desc(rowsI + 2048, 8192u, 1024u), idesc, 1u);
      }
      umma_commit_led(leader, &bars->mO);
    }
    __syncwarp();
    if (lead && more) load_part1(where[ph ^ 1u]);      // g, v, do, [T; A]: their tiles are dead

    anew();
    // ---- diagonal blocks, column sums: rows from the last to the first, sum(s) <- alpha sum(s) + C x
    const float* c0 = Cd0 + blk * 256;
    const float* c1 = Cd1 + blk * 256;
    f2 a2[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a2[j] = pack2(0.f, 0.f);
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      f2 xq, xb;
      { const float x = qv(i); xq = pack2(x, x); }
      if (WY) { const float x = bkv(i); xb = pack2(x, x); }
      const float an = i < 15 ? al[i + 1] : 1.f;
      const f2 dec = pack2(an, an), dec_lo = pack2(an, 1.f);
#pragma unroll
      for (int j4 = 0; j4 <= i / 4; ++j4) {
        f2 u0[2], u1[2];
        ld_pairs(c0 + i * 16 + 4 * j4, u0);
        if (WY) ld_pairs(c1 + i * 16 + 4 * j4, u1);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int j = 2 * j4 + t;
          if (j > i / 2) continue;
          f2 m = a2[j];
          if (i < 15) m = mul2(m, (j < i / 2 || (i & 1)) ? dec : dec_lo);   // (dec_lo: the upper column is row i + 1's own)
          m = fma2(u0[t], xq, m);
          if (WY) m = fma2(u1[t], xb, m);
          a2[j] = m;
        }
      }
    }
    mbar_wait_warp(&bars->mO, ph, ctl, 610);
    tc_fence_after();
    if (lead && more) load_part2(where[ph ^ 1u]);         // k, q: the last products that read those tiles are done
    const BlockDecays bd = block_decays(Bb, Af, blk, d);
    const float gam0 = bd.pre * al[0];              // gamma of the block's first token
    // dk' without the gate part: de (v_new dh^T) + out2
    float dkp[16];
    {
      float x[16];
#pragma unroll
      for (int j = 0; j < 8; ++j) unpack2(a2[j], dkp[2 * j], dkp[2 * j + 1]);
      float t2[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) t2[i] = 0.f;
#pragma unroll
      for (int I = 1; I < 4; ++I) {
        if (I <= blk) continue;
        tmem_ld16(cO2 + lane_base + (I == 1 ? 0 : I == 2 ? 16 : 48) + 16 * blk, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) t2[i] = fmaf(bd.cup[I - 1], x[i], t2[i]);
      }
      if (SB) {
        tmem_ld16(cDK + lane_base + blk * 16, x);
        tmem_ld_wait();
      } else {
        const float* dkb_g = rec32(p.lay.dkb, p.lay.sz_dkb);
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = dkb_g[rec_at(blk * 16 + i, d)];
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) t2[i] = fmaf(bd.post, x[i], t2[i]);
      float f = 1.f;
#pragma unroll
      for (int i = 15; i >= 0; --i) {
        dkp[i] = fmaf(f, t2[i], dkp[i]);
        f *= al[i];
      }
    }
    anew();
    // ---- diagonal blocks, row sums (kr(s) = k(s) ratio(i, s)), and the gradients of each row; dG where dg will be
    f2 kr[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) kr[j] = pack2(0.f, 0.f);
    float e = 1.f;
    f2 dsum = pack2(0.f, 0.f);
    const f2 minus = pack2(-1.f, -1.f);
#pragma unroll
    for (int qt = 0; qt < 4; ++qt) {                // four rows at a time: eight spill
      float o0[4], o1[WY ? 4 : 1], x[4], bi[FULL ? 4 : 1];
      if (FULL) {
        const float* bg = p.bch + token(blk * 16 + 4 * qt) * kK + d;
#pragma unroll
        for (int i = 0; i < 4; ++i) bi[FULL ? i : 0] = bg[static_cast<size_t>(i) * p.H * kK];
      }
      if (SB) {
        tmem_ld4(cDQ + lane_base + blk * 16 + 4 * qt, x);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = rec32(p.lay.dgb, p.lay.sz_dgb)[rec_at(blk * 16 + 4 * qt + i, d)];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) o0[i] = p.scale * gam0 * x[i];
      if (WY) {
        tmem_ld4(cDBK + lane_base + blk * 16 + 4 * qt, x);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) o1[i] = gam0 * x[i];
      }
#pragma unroll
      for (int J = 0; J < 3; ++J) {
        if (J >= blk) continue;
        const uint32_t at1 = cO1 + lane_base + (J == 0 ? 0 : J == 1 ? 3 * CR : 5 * CR) + (blk - 1 - J) * CR + 4 * qt;
        float y[WY ? 4 : 1];
        tmem_ld4(at1, x);
        if (WY) tmem_ld4(at1 + 16, y);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o0[i] = fmaf(bd.cdn[J], x[i], o0[i]);
          if (WY) o1[i] = fmaf(bd.cdn[J], y[i], o1[i]);
        }
      }
#pragma unroll
      for (int i4 = 0; i4 < 4; ++i4) {
        const int i = 4 * qt + i4;
        const float ai = i ? al[i] : 1.f, k_i = kv(i);
        e *= ai;
        const f2 dec = pack2(ai, ai);
        f2 s0[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)}, s1[2] = {s0[0], s0[0]};     // two chains each
#pragma unroll
        for (int j4 = 0; j4 <= i / 4; ++j4) {
          f2 u0[2], u1[2];
          ld_pairs(c0 + i * 16 + 4 * j4, u0);
          if (WY) ld_pairs(c1 + i * 16 + 4 * j4, u1);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int j = 2 * j4 + t;
            if (j > i / 2) continue;
            if (j < i / 2) {
              kr[j] = mul2(kr[j], dec);
            } else if (i & 1) {
              kr[j] = pack2(kv(i - 1) * ai, k_i);
            } else {
              kr[j] = pack2(k_i, 0.f);
            }
            s0[t] = fma2(u0[t], kr[j], s0[t]);
            if (WY) s1[t] = fma2(u1[t], kr[j], s1[t]);
          }
        }
        o0[i4] = fmaf(e, o0[i4], sum2(s0[0]) + sum2(s0[1]));             // dq
        if (WY) o1[i4] = fmaf(e, o1[i4], sum2(s1[0]) + sum2(s1[1]));     // d(b k)
      }
      float val[WY ? 4 : 1];
#pragma unroll
      for (int j = 0; j < 2; ++j) {                 // two rows: dG = q dq + (b k) dbk - k dk',  dk = dk' + b dbk
        const int i = 4 * qt + 2 * j;
        const f2 k2 = pair_of(kp[i >> 1]), dq2 = pack2(o0[2 * j], o0[2 * j + 1]);
        f2 dk2 = pack2(dkp[i], dkp[i + 1]), u = mul2(minus, dk2);
        if (WY) {
          const f2 dbk = pack2(o1[WY ? 2 * j : 0], o1[WY ? 2 * j + 1 : 0]), v2 = mul2(dbk, k2);
          f2 b2;
          if (FULL) b2 = pack2(bi[FULL ? 2 * j : 0], bi[FULL ? 2 * j + 1 : 0]);
          else b2.u = *reinterpret_cast<const unsigned long long*>(betas + blk * 16 + i);
          u = fma2(b2, dbk, u);
          dk2 = fma2(b2, dbk, dk2);
          unpack2(v2, val[WY ? 2 * j : 0], val[WY ? 2 * j + 1 : 0]);
        }
        const f2 dG = fma2(k2, u, mul2(pair_of(qp[i >> 1]), dq2));
        dsum = add2(dsum, dG);
        stage16_two(oQt, blk * 16 + i, d, dq2, p.qk16);
        stage16_two(oKt, blk * 16 + i, d, dk2, p.qk16);
        unpack2(dG, oGt[(blk * 16 + i) * kK + d], oGt[(blk * 16 + i + 1) * kK + d]);
      }
      if (FULL) {
        float* db = p.dbch + token(blk * 16 + 4 * qt) * kK + d;
#pragma unroll
        for (int i = 0; i < 4; ++i) db[static_cast<size_t>(i) * p.H * kK] = val[WY ? i : 0];
      }
      if (WY && !FULL) {
        const float s = warp_sum4(val, lane);
        if ((lane & 7) == 0) red[quad * 64 + blk * 16 + 4 * qt + (lane >> 3)] = s;
      }
    }
    // ---- gate gradient: reverse cumulative sum over the chunk, the end term counting for every row
    const float endt = (Et[d] + Et[kK + d]) + (Et[2 * kK + d] + Et[3 * kK + d]);
    St[blk * kK + d] = sum2(dsum);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    {
      float acc = endt;
#pragma unroll
      for (int m = 3; m > 0; --m)
        if (m > blk) acc += St[m * kK + d];
#pragma unroll
      for (int i = 15; i >= 0; --i) {
        float* g = oGt + (blk * 16 + i) * kK + d;
        acc += *g;
        *g = acc;
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (lead && blk < 3) {
      const ChunkAt a = where[ph];
      if (blk < 2)
        for (int t = 0; t < p.Kr / 64; ++t)
          tma_store_4d(blk == 0 ? &mo.dq : &mo.dk, (blk == 0 ? oQt : oKt) + t * 8192, t * 64, a.h, a.c * kC, a.b);
      else
        tma_store_4d(&mo.dg, oGt, 0, a.h, a.c * kC, a.b);
      bulk_commit();
    }
    if (WY && !FULL && tid < p.rows_of(where[ph].c)) {
      const float er = (red[tid] + red[64 + tid]) + (red[128 + tid] + red[192 + tid]);
      float wr = red[256 + tid] + red[320 + tid];
      if (V == 128) wr += red[384 + tid] + red[448 + tid];
      const size_t o = token(tid);
      if (p.dbeta_w) {
        p.dbeta_w[o] = wr;
        p.dbeta[o] = er;
      } else {
        p.dbeta[o] = er + wr;
      }
    }
  }
  if (lead) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------
template <int V, CwMode MODE, bool FULL>
static int launch_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                    const CUtensorMap& mdo, const CUtensorMap& mg, const CwOutMaps& mo, cudaStream_t st) {
  constexpr int smem = CwSmem<V, MODE == kCwAll || MODE == kCwWy>::kBytes;
  static_assert(smem <= 232448, "227 KB per CTA");
  static SmemAttr attr;
  if (attr.set(bwd_cw_kernel<V, MODE, FULL>, smem)) return kErrLaunch;
  const int sms = sm_count();
  if (sms <= 0) return kErrDevice;
  const int n = p.nbh * p.cn;
  if (launch_dependent(bwd_cw_kernel<V, MODE, FULL>, dim3(n < sms ? n : sms), dim3(kCwThreads), smem, st, p, mq, mk, mv, mdo, mg, mo) !=
      cudaSuccess) return kErrLaunch;
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
template <CwMode MODE, bool FULL = false>
static int launch_v(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                    const CUtensorMap& mdo, const CUtensorMap& mg, const CwOutMaps& mo, cudaStream_t st) {
  return p.V == 64 ? launch_t<64, MODE, FULL>(p, mq, mk, mv, mdo, mg, mo, st) : launch_t<128, MODE, FULL>(p, mq, mk, mv, mdo, mg, mo, st);
}

// mask bit 4: Stage B, bit 8: WY VJP (delta variants only); both together are one kernel
int launch_bwd_main_cw(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                       const CUtensorMap& mdo, const CUtensorMap& mg, const CwOutMaps& mo, cudaStream_t st, uint32_t mask) {
  const bool sb = mask & 4u, wy = (mask & 8u) && p.delta;
  if (!p.delta) return sb ? launch_v<kCwNoDelta>(p, mq, mk, mv, mdo, mg, mo, st) : kOk;
  if (sb && !wy) return launch_v<kCwStageB>(p, mq, mk, mv, mdo, mg, mo, st);
  if (p.bch)
    return sb ? launch_v<kCwAll, true>(p, mq, mk, mv, mdo, mg, mo, st) : launch_v<kCwWy, true>(p, mq, mk, mv, mdo, mg, mo, st);
  return sb ? launch_v<kCwAll>(p, mq, mk, mv, mdo, mg, mo, st) : launch_v<kCwWy>(p, mq, mk, mv, mdo, mg, mo, st);
}

}  // namespace lg
