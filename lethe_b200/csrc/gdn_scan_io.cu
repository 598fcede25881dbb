// State scan and the chunk-parallel kernel beside it in one, for the channel-wise gate and calls with many pairs:
//
//   forward :  x_{c+1} = a_c x_c - P_c x_c + R_c            and   [w x ; (scale gamma q) x] = [w; qg] x_c,
//                                                                 v_new = u - w x,  o = qg x + A v_new      (output_kernel)
//   adjoint :  x_{c-1} = a_c x_c - P_c^T x_c + Rb_c         with  Rb_c = qg^T do - w^T (A^T do)             (bwd_pre_kernel)
//
// Apart, the forward writes the state records and reads them again, and the adjoint writes and reads Rb: 32 KB each way and chunk
// at d_v = 128, and both kernels are bound by HBM once there are pairs enough to fill the GPU with scans of 64 columns.  Here a CTA
// walks the chunks of a pair with 64 columns of the state, and the work of the other kernel for the same chunk and columns runs
// beside the serial step: on the same tensor pipe, on warps of its own, behind the state (forward; the state operand that the
// step multiplies with P serves [w; qg] too) or ahead of it (adjoint; Rb stays in tensor memory).  An evaluation (lean 2)
// leaves no state records at all.
//
// Bits: every sum is formed as in scan_kernel, output_kernel and bwd_pre_kernel (Rb is rounded to fp16 as its record is), so the
// results do not depend on which kernels a call takes.
//
// Warps: 0-15 the state, thread (group of 16 columns, key channel) as in scan_kernel; 16 copies; 17, 18 the step's products (without
// the delta term 17 stores the records); 19 and 24 the other kernel's first and second product; 20-23 its epilogues, tensor-memory
// quadrants 0-3.  With both products on one warp the first of a chunk waited for the epilogue between those of the chunk before, and
// the step for the first (1.45 us a step of the evaluation, 1.27 with two warps, 1.10 with the epilogue's loads ahead of its stores).
//
// Bound by HBM for many pairs (64 pairs x 128 chunks, d_v = 128: forward 5.9 TB/s of its bytes), by a chain of 1.05 to 1.2 us a step for few.
// us, the two kernels / this one (forward; evaluation; adjoint), d_v = 128, pairs x chunks, with the delta term: 19 x 128
// 157 / 157; 153 / 147; 149 / 150;  32 x 250 368 / 310; 354 / 275; 346 / 292;  64 x 128 298 / 258; 284 / 184; 272 / 178;  d_v = 64: 40 x 128
// 182 / 163; 175 / 147; 171 / 156;  140 x 64 210 / 185; 198 / 152; 186 / 138;  160 x 64 279 / 250; 267 / 209; 250 / 210.  Records of few chunks
// ahead prefetched to L2 make it slower (64 x 128, forward, none / two / four / six chunks ahead: 283 / 304 / 339 / 359), but for the decays
// and R, which the state warps load to registers (without the delta term, 64 x 64, adjoint: 73 us without, 56 with).
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

constexpr int kIoW = 64, kIoVs = 16, kIoStateWarps = 16, kIoThreads = 25 * 32;
constexpr int kIoX = 128 * kIoW * 2;                       // a state operand tile

// Rings: P; ring 1: what the product behind needs, w qg (forward: stacked [w; qg]); ring 2: A with u (forward) or do (adjoint), which
// an epilogue works on.  Without the delta term ring 1 has all of a chunk.
template <bool ADJOINT, bool DELTA>
struct IoSmem {
  static constexpr int kP = DELTA ? 2 : 1, oP = 2 * kIoX;
  static constexpr int oQ = 0, oDO = DELTA ? 0 : 16384;               // adjoint (do in ring 2 with the delta term)
  static constexpr int oNA = 16384, oNU = oNA + 8192, oNR = oNU + 8192;      // forward without the delta term
  static constexpr int kOne = DELTA ? 32768 : ADJOINT ? 24576 : oNR + 16384;
  static constexpr int kNOne = DELTA ? 2 : ADJOINT ? 6 : 4, oOne = oP + (DELTA ? kP * 32768 : 0);
  static constexpr int kNTwo = DELTA ? 4 : 1, oTwo = oOne + kNOne * kOne;
  static constexpr int oBar = oTwo + (DELTA ? kNTwo * 16384 : 0), kBytes = oBar + 512 + 1024;
};
struct IoBars {
  uint64_t p_full[2], p_free[2], mma, one_full[6], one_free[6], two_full[4], two_free[4];
  uint64_t x_full[2], x_free[2];      // state operand written; read by everything (without the delta term)
  uint64_t conv[2];                   // do is fp16 (adjoint)
  uint64_t m1[2], ready[2], m2[2];    // first product; its epilogue is the second one's operand; second product
  uint64_t acc_free[2];               // the accumulator of the second product has been read
  uint32_t tmem_slot;
  int abort_flag;
};
static_assert(sizeof(IoBars) <= 512, "");

template <bool ADJOINT, bool DELTA>
__global__ void __launch_bounds__(kIoThreads, 1)
scan_io_kernel(const Problem p, const __grid_constant__ CUtensorMap mio, const __grid_constant__ CUtensorMap mv) {
  using S = IoSmem<ADJOINT, DELTA>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  IoBars* bars = reinterpret_cast<IoBars*>(sm + S::oBar);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int v0 = blockIdx.x * kIoW, bh = blockIdx.y + p.bh0, V = p.V, NT = p.NT;
  const int b = bh / p.H, h = bh % p.H;
  const bool keep = ADJOINT || p.lean < 2;           // state records (and v_new) are read by a later kernel
  CtaCtl ctl{p.status, &bars->abort_flag};
  auto xb = [&](int it) { return sm + (it & 1) * kIoX; };
  auto stage1 = [&](int it) { return sm + S::oOne + (it % S::kNOne) * S::kOne; };
  auto stage2 = [&](int it) { return sm + S::oTwo + (it % S::kNTwo) * 16384; };
  auto round_of = [](int it, int n) { return static_cast<uint32_t>((it / n) & 1); };      // phase of the it-th use of a ring of n
  auto chunk_of = [&](int it) { return ADJOINT ? NT - 1 - it : it; };
  auto rec = [&](const unsigned char* base, int it, size_t size) { return base + (static_cast<size_t>(bh) * NT + chunk_of(it)) * size; };

  if (tid == 0) {
    bars->abort_flag = 0;
    mbar_init(&bars->mma, 2);
    for (int i = 0; i < 6; ++i) {
      mbar_init(&bars->one_full[i], 1);
      mbar_init(&bars->one_free[i], ADJOINT || DELTA ? 1 : 1 + kIoStateWarps);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&bars->two_full[i], 1);
      mbar_init(&bars->two_free[i], !ADJOINT && keep ? 2 : 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->p_full[i], 1);
      mbar_init(&bars->p_free[i], 2);
      mbar_init(&bars->x_full[i], DELTA ? 1 : kIoStateWarps);
      mbar_init(&bars->x_free[i], (ADJOINT ? 0 : 1) + (keep ? 1 : 0));
      mbar_init(&bars->conv[i], 2);
      mbar_init(&bars->m1[i], 1);
      mbar_init(&bars->ready[i], 2);
      mbar_init(&bars->m2[i], 1);
      mbar_init(&bars->acc_free[i], ADJOINT ? kIoStateWarps : 2);
    }
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
  const uint32_t tmem = bars->tmem_slot, lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const uint32_t cAcc = tmem, cSide = tmem + 128, cV = tmem + 256;      // step's two halves; second product (two, alternating); A^T do
  griddep_wait();
  griddep_launch();

  if (warp == kIoStateWarps) {
    // ---- copies
    if (lane == 0) {
      auto w_of = [&](int it) { return rec(p.saved + p.lay.w, it, p.lay.sz_w); };
      auto qg_of = [&](int it) { return rec(p.saved + p.lay.qg, it, 16384); };
      auto a_of = [&](int it) { return rec(p.saved + p.lay.ta, it, p.lay.sz_ta) + 8192; };
      auto p_of = [&](int it) { return rec(p.saved + p.lay.p, it, 32768); };
      auto r_of = [&](int it) { return rec(p.saved + p.lay.r, it, p.lay.sz_r) + static_cast<size_t>(v0 >> 6) * 16384; };
      auto u_of = [&](int it) { return rec(p.saved + p.lay.u, it, p.lay.sz_u) + static_cast<size_t>(v0 >> 6) * 8192; };
      for (int it = 0; it < NT; ++it) {
        // what the state warps load to registers a step ahead, to L2 now
        bulk_prefetch(rec(p.saved + p.lay.ad, it, 512), 512);
        if (!ADJOINT && DELTA) bulk_prefetch(r_of(it), 16384);
        auto load_two = [&]() {
          const int s2 = it % S::kNTwo;
          uint64_t* f2 = &bars->two_full[s2];
          if (it >= S::kNTwo) mbar_wait(&bars->two_free[s2], round_of(it - S::kNTwo, S::kNTwo), ctl, 701);
          mbar_expect_tx(f2, 16384u);
          if (ADJOINT) {
            tma_load_4d(stage2(it), &mio, f2, v0, h, chunk_of(it) * kC, b);
            bulk_g2s(stage2(it) + 8192, a_of(it), 8192u, f2);
          } else {
            bulk_g2s(stage2(it), a_of(it), 8192u, f2);
            bulk_g2s(stage2(it) + 8192, u_of(it), 8192u, f2);
          }
        };
        // (in the order in which they are free and wanted: a wait for one must not hold up another)
        if (DELTA && ADJOINT) load_two();
        if (DELTA) {
          const int s = it % S::kP;
          if (it >= S::kP) mbar_wait(&bars->p_free[s], round_of(it - S::kP, S::kP), ctl, 702);
          mbar_expect_tx(&bars->p_full[s], 32768u);
          bulk_g2s(sm + S::oP + s * 32768, p_of(it), 32768u, &bars->p_full[s]);
        }
        const int s = it % S::kNOne;
        unsigned char* t = stage1(it);
        uint64_t* f = &bars->one_full[s];
        if (it >= S::kNOne) mbar_wait(&bars->one_free[s], round_of(it - S::kNOne, S::kNOne), ctl, 703);
        mbar_expect_tx(f, static_cast<uint32_t>(S::kOne));
        if (DELTA && !ADJOINT) {
          for (int i = 0; i < 2; ++i) {
            bulk_g2s(t + i * 16384, w_of(it) + i * 8192, 8192u, f);
            bulk_g2s(t + i * 16384 + 8192, qg_of(it) + i * 8192, 8192u, f);
          }
          load_two();
        } else {
          bulk_g2s(t + S::oQ, qg_of(it), 16384u, f);
          if (DELTA) bulk_g2s(t + 16384, w_of(it), 16384u, f);
          else if (ADJOINT) tma_load_4d(t + S::oDO, &mio, f, v0, h, chunk_of(it) * kC, b);
        }
        if (!DELTA && !ADJOINT) {
          bulk_g2s(t + S::oNA, a_of(it), 8192u, f);
          tma_load_4d(t + S::oNU, &mv, f, v0, h, chunk_of(it) * kC, b);      // v_new = v
          bulk_g2s(t + S::oNR, r_of(it), 16384u, f);
        }
      }
    }
    __syncwarp();
  } else if (warp == kIoStateWarps + 1 || warp == kIoStateWarps + 2) {
    // ---- the step's products, half of the contraction each, and the records of the state
    const int m = warp - kIoStateWarps - 1;
    auto record = [&](int it) {
      const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
      return (ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc) + (ADJOINT ? z : z + bh) * p.lay.sz_hc + static_cast<size_t>(v0 >> 6) * 16384;
    };
    if (DELTA) {
      const uint32_t leader = elect_leader();
      const uint64_t b_desc0 = make_desc(smem_u32(sm), 16384u, 1024u);
      const uint32_t idesc = make_idesc(128, kIoW, ADJOINT, true), acc = cAcc + static_cast<uint32_t>(m * kIoW);
      for (int it = 0; it < NT; ++it) {
        const int st = it % S::kP;
        mbar_wait_warp(&bars->p_full[st], round_of(it, S::kP), ctl, 704);
        if (m == 0) {          // the other operand tile is recorded, and [w; qg] x is done with it: it may be written again
          if (lane == 0 && keep) bulk_wait_read();
          if (!ADJOINT && it > 0) mbar_wait_warp(&bars->m1[(it - 1) & 1], round_of(it - 1, 2), ctl, 705);
          __syncwarp();
        }
        asm volatile("bar.sync 1, %0;" ::"n"((kIoStateWarps + 2) * 32) : "memory");
        tc_fence_after();
        const uint32_t pa = smem_u32(sm + S::oP + st * 32768);
        const uint64_t a_desc0 = ADJOINT ? make_desc(pa, 16384u, 1024u) : make_desc(pa, 16u, 1024u);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          const int j = m * 4 + jj;
          const uint32_t aoff = ADJOINT ? static_cast<uint32_t>(j * 2048) >> 4 : static_cast<uint32_t>((j >> 2) * 16384 + (j & 3) * 32) >> 4;
          const uint32_t boff = static_cast<uint32_t>(j * 2048 + (it & 1) * kIoX) >> 4;
          umma_led(leader, acc, a_desc0 + aoff, b_desc0 + boff, idesc, jj > 0 ? 1u : 0u);
        }
        umma_commit_led(leader, &bars->mma);
        umma_commit_led(leader, &bars->p_free[st]);
        if (m == 0 && lane == 0) {
          if (!ADJOINT) mbar_arrive(&bars->x_full[it & 1]);
          if (keep) {
            bulk_s2g(record(it), xb(it), kIoX);      // the operand tile is the record's image
            bulk_commit();
          }
        }
        __syncwarp();
      }
    } else if (m == 0 && lane == 0 && keep) {
      for (int it = 0; it < NT; ++it) {
        mbar_wait(&bars->x_full[it & 1], round_of(it, 2), ctl, 706);
        bulk_s2g(record(it), xb(it), kIoX);
        bulk_commit();
        bulk_wait_read();
        mbar_arrive(&bars->x_free[it & 1]);
      }
    }
    if (m == 0 && lane == 0) bulk_wait_read();
    __syncwarp();
  } else if (warp == kIoStateWarps + 3) {
    // ---- first product of the other kernel: [w; qg] x (without the delta term qg x), A^T do
    const uint32_t leader = elect_leader();
    if (!ADJOINT || DELTA) {
      for (int it = 0; it < NT; ++it) {
        const int s = it % S::kNOne;
        const uint32_t t = smem_u32(stage1(it)), t2 = smem_u32(stage2(it));
        if (ADJOINT) {
          if (it > 1) mbar_wait_warp(&bars->ready[it & 1], round_of(it - 2, 2), ctl, 707);      // the accumulator has been read
          mbar_wait_warp(&bars->two_full[it % S::kNTwo], round_of(it, S::kNTwo), ctl, 708);
          mbar_wait_warp(&bars->conv[it & 1], round_of(it, 2), ctl, 709);
          tc_fence_after();
          issue_product_led(leader, cV + static_cast<uint32_t>((it & 1) * kIoW), Tile{t2, 64, true}, Tile{t2, 64, true}, kIoW, 64, 0u);      // rows 64-127
          umma_commit_led(leader, &bars->m1[it & 1]);
        } else {
          const Tile x{smem_u32(xb(it)), 128, true};
          const uint32_t acc = cSide + static_cast<uint32_t>((it & 1) * kIoW);
          mbar_wait_warp(&bars->one_full[s], round_of(it, S::kNOne), ctl, 710);
          if (it > 1) mbar_wait_warp(&bars->acc_free[it & 1], round_of(it - 2, 2), ctl, 711);
          mbar_wait_warp(&bars->x_full[it & 1], round_of(it, 2), ctl, 712);
          tc_fence_after();
          if (DELTA) issue_product_led(leader, acc, Tile{t, 128, false}, x, kIoW, 128, 0u);
          else issue_product_led(leader, acc, Tile{t - 8192, 64, false}, x, kIoW, 128, 0u);      // (rows 64-127)
          umma_commit_led(leader, &bars->m1[it & 1]);
          umma_commit_led(leader, DELTA ? &bars->one_free[s] : &bars->x_free[it & 1]);
        }
      }
    }
  } else if (warp == kIoStateWarps + 8) {
    // ---- second product: o (rows 64-127), Rb.  A warp of its own: behind the epilogue of the first product it would hold up the next
    const uint32_t leader = elect_leader();
    for (int it = 0; it < NT; ++it) {
      const uint32_t t = smem_u32(stage1(it)), acc = cSide + static_cast<uint32_t>((it & 1) * kIoW);
      if (ADJOINT) {
        if (it > 1) mbar_wait_warp(&bars->acc_free[it & 1], round_of(it - 2, 2), ctl, 713);
        mbar_wait_warp(&bars->one_full[it % S::kNOne], round_of(it, S::kNOne), ctl, 714);
        mbar_wait_warp(DELTA ? &bars->ready[it & 1] : &bars->conv[it & 1], round_of(it, 2), ctl, 715);      // A^T do is an operand, where A was
        tc_fence_after();
        const uint32_t t2 = DELTA ? smem_u32(stage2(it)) : t + S::oDO;
        issue_product_led(leader, acc, Tile{t + S::oQ, 64, true}, Tile{t2, 64, true}, kIoW, 64, 0u);
        if (DELTA) issue_product_led(leader, acc, Tile{t + 16384, 64, true}, Tile{t2 + 8192, 64, true}, kIoW, 64, 1u, true);
        umma_commit_led(leader, &bars->m2[it & 1]);
        umma_commit_led(leader, &bars->one_free[it % S::kNOne]);
        if (DELTA) umma_commit_led(leader, &bars->two_free[it % S::kNTwo]);
      } else {
        mbar_wait_warp(DELTA ? &bars->two_full[it % S::kNTwo] : &bars->one_full[it % S::kNOne], round_of(it, DELTA ? S::kNTwo : S::kNOne), ctl, 716);
        mbar_wait_warp(&bars->m1[it & 1], round_of(it, 2), ctl, 717);
        mbar_wait_warp(&bars->ready[it & 1], round_of(it, 2), ctl, 718);      // v_new
        tc_fence_after();
        const uint32_t a = DELTA ? smem_u32(stage2(it)) : t + S::oNA, vn = a + 8192;
        issue_product_led(leader, acc, Tile{a - 8192, 64, false}, Tile{vn, 64, true}, kIoW, 64, 1u);
        umma_commit_led(leader, &bars->m2[it & 1]);
      }
    }
  } else if (warp > kIoStateWarps + 3) {
    // ---- epilogues of the other products
    const int quad = warp & 3, r = (quad & 1) * 32 + lane;
    auto pair_sync = [&]() {           // quadrants 0 and 1, or 2 and 3
      if (quad < 2) asm volatile("bar.sync 2, 64;" ::: "memory");
      else asm volatile("bar.sync 3, 64;" ::: "memory");
    };
    auto to_f16 = [&](unsigned char* t) {      // a [64][64] bf16 tile, by quadrants 0 and 1
      uint4 c[8];              // (all loads before the first store)
#pragma unroll
      for (int i = 0; i < 8; ++i) c[i] = *reinterpret_cast<const uint4*>(t + (r + 64 * i) * 16);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float x[8];
        unpack8_bf16(c[i], x);
        *reinterpret_cast<uint4*>(t + (r + 64 * i) * 16) = pack8_f16(x);
      }
    };
    auto arrive = [&](uint64_t* bar) {         // what this warp has written is for the asynchronous proxy
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    const bool first = (quad & 1) == 0 && lane == 0;
    if (ADJOINT) {
      for (int it = 0; it < NT; ++it) {
        unsigned char* t = DELTA ? stage2(it) : stage1(it) + S::oDO;
        if (quad < 2) {
          mbar_wait_warp(DELTA ? &bars->two_full[it % S::kNTwo] : &bars->one_full[it % S::kNOne], round_of(it, DELTA ? S::kNTwo : S::kNOne), ctl, 719);
          to_f16(t);
          if (it > 1) mbar_wait_warp(&bars->m2[it & 1], round_of(it - 2, 2), ctl, 720);      // (a phase later would pass for this one)
          arrive(&bars->conv[it & 1]);
        } else if (DELTA) {
          mbar_wait_warp(&bars->m1[it & 1], round_of(it, 2), ctl, 721);
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            float x[32];
            tmem_ld32(cV + (it & 1) * kIoW + lane_base + 32 * j, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) tile_st_chunk(t + 8192, r, 4 * j + i, 64, pack8_f16(x + 8 * i));
          }
          arrive(&bars->ready[it & 1]);
        }
      }
    } else if (quad < 2) {
      constexpr int kN = S::kNTwo;
      for (int it = 0; it < NT; ++it) {
        if (DELTA) {
          unsigned char* u = stage2(it) + 8192;
          mbar_wait_warp(&bars->two_full[it % kN], round_of(it, kN), ctl, 722);
          uint4 un[2] = {tile_ld_chunk(u, r, 0, 64), tile_ld_chunk(u, r, 1, 64)};      // (loads ahead of the stores before them)
          mbar_wait_warp(&bars->m1[it & 1], round_of(it, 2), ctl, 723);
          tc_fence_after();
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float x[16], u16[16];
            tmem_ld16(cSide + (it & 1) * kIoW + lane_base + 16 * j, x);
            unpack8_f16(un[0], u16);
            unpack8_f16(un[1], u16 + 8);
            if (j < 3)
#pragma unroll
              for (int i = 0; i < 2; ++i) un[i] = tile_ld_chunk(u, r, 2 * j + 2 + i, 64);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) u16[e] -= x[e];
#pragma unroll
            for (int i = 0; i < 2; ++i) tile_st_chunk(u, r, 2 * j + i, 64, pack8_f16(u16 + 8 * i));
          }
          arrive(&bars->ready[it & 1]);
          if (keep) {
            pair_sync();
            if (first) {
              bulk_wait_read();
              if (it > 0) mbar_arrive(&bars->two_free[(it - 1) % kN]);
              bulk_s2g(p.saved + p.lay.vn + (static_cast<size_t>(bh) * NT + it) * p.lay.sz_vn + static_cast<size_t>(v0 >> 6) * 8192, u, 8192);
              bulk_commit();
            }
            __syncwarp();
          }
        } else {
          mbar_wait_warp(&bars->one_full[it % S::kNOne], round_of(it, S::kNOne), ctl, 724);
          to_f16(stage1(it) + S::oNU);
          if (it > 1) mbar_wait_warp(&bars->m2[it & 1], round_of(it - 2, 2), ctl, 725);      // (as above)
          arrive(&bars->ready[it & 1]);
        }
      }
      if (first) bulk_wait_read();
    } else {
      for (int it = 0; it < NT; ++it) {
        mbar_wait_warp(&bars->m2[it & 1], round_of(it, 2), ctl, 726);
        tc_fence_after();
        unsigned char* a = DELTA ? stage2(it) : stage1(it) + S::oNA;      // A is dead: o leaves from there
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float x[32];
          tmem_ld32(cSide + (it & 1) * kIoW + lane_base + 32 * j, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) tile_st_chunk(a, r, 4 * j + i, 64, pack8_bf16(x + 8 * i));
        }
        arrive(&bars->acc_free[it & 1]);
        pair_sync();
        if (first) {
          bulk_wait_read();
          constexpr int kN = S::kNTwo;
          if (it > 0) mbar_arrive(DELTA ? &bars->two_free[(it - 1) % kN] : &bars->one_free[(it - 1) % S::kNOne]);
          tma_store_4d(&mio, a, v0, h, it * kC, b);
          bulk_commit();
        }
        __syncwarp();
      }
      if (first) bulk_wait_read();
    }
  } else {
    // ---- the state: thread d of a group holds 16 columns of row d of x in fp32 (scan_kernel)
    const int d = tid & 127, g = tid >> 7, vg = v0 + g * kIoVs;
    const __half* Rg = reinterpret_cast<const __half*>(p.saved + p.lay.r);
    const float* ADg = reinterpret_cast<const float*>(p.saved + p.lay.ad);
    const size_t rofs = (static_cast<size_t>(vg / 16) * kK + d) * 16;
    auto piece = [&](int q) { return d * 128 + (((g * 2 + q) ^ (d & 7)) << 4); };      // of this thread's row of a tile image
    float x[kIoVs];
    {
      const float* x0 = ADJOINT ? p.dhT : p.h0;
#pragma unroll
      for (int j = 0; j < kIoVs; ++j) x[j] = x0 && d < p.Kr ? x0[(static_cast<size_t>(bh) * p.Kr + d) * V + vg + j] : 0.f;
    }
    uint4 rnext[2];
    // Without the delta term a step is shorter than the decay's way here: two steps ahead.
    float a_next = 0.f, a_later = 0.f;
    auto load_next = [&](int it) {
      const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
      if (!ADJOINT && DELTA) {
        const __half* rp = Rg + z * kK * V + rofs;
        rnext[0] = *reinterpret_cast<const uint4*>(rp);
        rnext[1] = *reinterpret_cast<const uint4*>(rp + 8);
      }
      if (DELTA) a_next = ADg[z * kK + d];
      else a_later = ADg[z * kK + d];
    };
    load_next(0);
    if (!DELTA) {
      a_next = a_later;
      if (NT > 1) load_next(1);
    }
    for (int it = 0; it < NT; ++it) {
      unsigned char* X = xb(it);
      if (!DELTA && it > 1) mbar_wait_warp(&bars->x_free[it & 1], round_of(it - 2, 2), ctl, 727);
#pragma unroll
      for (int q = 0; q < 2; ++q) *reinterpret_cast<uint4*>(X + piece(q)) = pack8_f16(x + 8 * q);
      fence_proxy_async();
      tc_fence_before();
      if (DELTA) {
        asm volatile("bar.arrive 1, %0;" ::"n"((kIoStateWarps + 2) * 32) : "memory");
      } else {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->x_full[it & 1]);
      }
      // in the shadow of the products: this chunk's input and decay
      const int s = it % S::kNOne;
      const float a = a_next;
      float rr[kIoVs];
      if (ADJOINT) {
        mbar_wait_warp(&bars->m2[it & 1], round_of(it, 2), ctl, 728);
        tc_fence_after();
        float t[kIoVs];
        tmem_ld16(cSide + (it & 1) * kIoW + lane_base + g * kIoVs, t);
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int q = 0; q < 2; ++q) unpack8_f16(pack8_f16(t + 8 * q), rr + 8 * q);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->acc_free[it & 1]);
      } else if (DELTA) {
#pragma unroll
        for (int q = 0; q < 2; ++q) unpack8_f16(rnext[q], rr + 8 * q);
      } else {
        const unsigned char* R = stage1(it) + S::oNR;
        mbar_wait_warp(&bars->one_full[s], round_of(it, S::kNOne), ctl, 729);
#pragma unroll
        for (int q = 0; q < 2; ++q) unpack8_f16(*reinterpret_cast<const uint4*>(R + piece(q)), rr + 8 * q);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->one_free[s]);
      }
      if (DELTA) {
        if (it + 1 < NT) load_next(it + 1);
#pragma unroll
        for (int j = 0; j < kIoVs; ++j) rr[j] = fmaf(a, x[j], rr[j]);
        mbar_wait_warp(&bars->mma, round_of(it, 1), ctl, 730);
        tc_fence_after();
        float a0[kIoVs], a1[kIoVs];
        tmem_ld16(cAcc + lane_base + g * kIoVs, a0);
        tmem_ld16(cAcc + kIoW + lane_base + g * kIoVs, a1);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < kIoVs; ++j) x[j] = rr[j] - a0[j] - a1[j];
      } else {
        a_next = a_later;
        if (it + 2 < NT) load_next(it + 2);
#pragma unroll
        for (int j = 0; j < kIoVs; ++j) x[j] = fmaf(a, x[j], rr[j]);
      }
    }
    if (!ADJOINT && keep) {            // the final state as one more record
      unsigned char* last = p.saved + p.lay.hc + (static_cast<size_t>(bh) * (NT + 1) + NT) * p.lay.sz_hc;
#pragma unroll
      for (int q = 0; q < 2; ++q) *reinterpret_cast<uint4*>(last + sw128_chunk(d, vg / 8 + q, 128)) = pack8_f16(x + 8 * q);
    }
    float* xT = ADJOINT ? p.dh0 : p.hT;
    if (xT && d < p.Kr) {
#pragma unroll
      for (int j = 0; j < kIoVs; j += 4)
        *reinterpret_cast<float4*>(xT + (static_cast<size_t>(bh) * p.Kr + d) * V + vg + j) = make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

template <bool ADJOINT, bool DELTA>
static int launch_scan_io_t(const Problem& p, const CUtensorMap& mio, const CUtensorMap& mv, cudaStream_t st) {
  constexpr int smem = IoSmem<ADJOINT, DELTA>::kBytes;
  static_assert(smem <= 232448, "227 KB per CTA");
  static SmemAttr attr;
  if (attr.set(scan_io_kernel<ADJOINT, DELTA>, smem)) return kErrLaunch;
  const cudaError_t e = launch_dependent(scan_io_kernel<ADJOINT, DELTA>, dim3(p.V / kIoW, p.nbh), dim3(kIoThreads), smem, st, p, mio, mv);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

// Whether a call takes this kernel instead of the two: its records are not for the caller (lean), the whole sequence in one call, and
// pairs enough.  With the delta term that is where the scan has 64 columns per CTA anyway (launch_scan).  Without it the scan is
// spread over four times as many CTAs, and the others over all SMs.  The adjoint is the faster from a third of the SMs on, the
// forward where it fills three fifths of them in its last round too (64 chunks, us, the two / this one: forward, evaluation, adjoint, by
// CTAs here: 48 51 / 50, 51 / 50, 37 / 41; 64 63 / 72, 63 / 61, 50 / 48; 96 92 / 79, 92 / 65, 76 / 48; 128 119 / 88, 119 / 70, 100 / 52;
// 160 145 / 151, 145 / 128, 122 / 96; 250 chunks, 64 CTAs 229 / 254, 229 / 220, 196 / 166).  By the whole problem, since calls on
// ranges of its pairs run beside one another.
//
// Short sequences: a CTA has the whole SM, and its start (barriers, tensor memory, the first loads) is as long for one chunk as for many,
// so a row of rounds of them loses to kernels that share the SMs.  us, the two / this one, pairs x chunks, without the delta term, d_v =
// 128: forward 256 x 1 34 / 43, x 2 50 / 58, x 4 81 / 85, x 6 118 / 117, x 8 155 / 149; evaluation 256 x 2 50 / 54, x 3 69 / 69, x 4 81 / 79;
// adjoint 1024 x 1 118 / 142, x 2 202 / 216, x 3 286 / 288, x 4 409 / 397; d_v = 64, forward 512 x 4 110 / 120, x 6 155 / 160, x 8 200 / 200,
// evaluation x 4 110 / 116, x 6 155 / 155.  With it only the forward over one chunk: d_v = 128, 256 pairs 50 / 54, 512 90 / 93; two chunks 79 / 79.
static bool scan_io_rule(int gate, int delta, int V, int pairs, int NT, uint32_t lean, bool adjoint, int sms) {
  if (gate != LETHE_GATE_CHANNEL || sms <= 0) return false;
  const int ctas = V / kIoW * pairs, rounds = (ctas + sms - 1) / sms;
  if (delta) return 4 * ctas > sms && (adjoint || NT > 1 || rounds <= 2);
  if (adjoint) return 3 * ctas > sms && (NT > 2 || rounds <= 2);
  const int least = lean == 2u ? (V == 64 ? 6 : 3) : (V == 64 ? 8 : 6);
  return 5 * ctas > 3 * rounds * sms && (NT >= least || rounds == 1);
}
bool scan_io_serves(const Problem& p, bool adjoint) {
  return p.lean && p.cn == p.NT && scan_io_rule(p.gate, p.delta, p.V, p.B * p.H, p.NT, p.lean, adjoint, sm_count());
}
// ... for lethe_gdn_joint_scans, which a captured step is planned with
int scan_io_joint(const LetheGdnDims& d, uint32_t lean, int sms) {
  auto serves = [&](bool adjoint) { return scan_io_rule(d.gate, d.delta, d.V, d.B * d.H, d.L / kC, lean, adjoint, sms); };
  return (serves(false) ? LETHE_JOINT_FORWARD : 0) | (serves(true) ? LETHE_JOINT_ADJOINT : 0);
}
// mio: o (forward) or do (adjoint)
int launch_scan_io(const Problem& p, bool adjoint, const CUtensorMap& mio, const CUtensorMap& mv, cudaStream_t st) {
  if (adjoint) return p.delta ? launch_scan_io_t<true, true>(p, mio, mv, st) : launch_scan_io_t<true, false>(p, mio, mv, st);
  return p.delta ? launch_scan_io_t<false, true>(p, mio, mv, st) : launch_scan_io_t<false, false>(p, mio, mv, st);
}

}  // namespace lg
