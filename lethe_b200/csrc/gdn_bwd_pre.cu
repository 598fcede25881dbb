// Input of the adjoint state scan, chunk-parallel:
//   Rb = (scale gamma q)^T do - w^T (A^T do)
// (reference: the terms of the reverse scan K#1, gdn2_assemble.py:71-99).
//
// Bound by HBM (88 KB per chunk at d_v = 128) and, per chunk, by a chain of load, conversion, two dependent products and
// store.  Persistent CTAs of 256 threads, three or four per SM, fill each other's gaps; a CTA fetches the next do
// and A once its last products are done, q and w once the result, staged where they were, has left.  8192 chunks,
// channel-wise, d_v = 128: 150 -> 128 us; 4096 chunks, scalar, d_v = 64: 56 -> 51.  With gates and (scalar gate) tiles
// requested a chunk ahead: scalar, d_v = 128, 512 chunks 19.4 -> 17.3; without the delta term d_v = 64, 1692 chunks 22.6 -> 19.5.
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

constexpr int kPreThreads = 256;

// KW: 64 only without the delta term and with one decay or none, as in prepare_nodelta_kernel
template <int V, bool DELTA, int KW = kK>
struct PreSmem {
  static constexpr int oW = 16384, oDO = DELTA ? oW + 16384 : V * KW * 2;     // (Rb is staged over q and w)
  static constexpr int oA = oDO + V * 128;                                    // A (its 128-row view starts 64 rows early)
  static constexpr int oDV = oA;                                              // then A^T do (64 x V) in its place
  static constexpr int kUsed = DELTA ? oDV + V * 128 : oA, kCtas = DELTA && V == 128 ? 3 : 4;
  static constexpr int kBytes = kUsed + 2 * 256 + static_cast<int>(sizeof(CtaShared)) + 1024;
};

// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA, bool CW, int KW>
__global__ void __launch_bounds__(kPreThreads, PreSmem<V, DELTA, KW>::kCtas)
bwd_pre_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mdo) {
  using S = PreSmem<V, DELTA, KW>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  unsigned char *QG = sm, *Wt = sm + S::oW, *DO = sm + S::oDO, *At_ = sm + S::oA, *DVL = sm + S::oDV;
  float* sgs = reinterpret_cast<float*>(sm + S::kUsed);       // [2][64] scale gamma (scalar gate)
  CtaShared* cs = reinterpret_cast<CtaShared*>(sgs + 128);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *full = &cs->bar[0], *mma = &cs->bar[1];
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
  auto load_do = [&](const At& a) {
    mbar_expect_tx(full, KW * 128u + V * 128u + (DELTA ? 16384u + 8192u : 0u));
    for (int i = 0; i < V / 64; ++i) tma_load_4d(DO + i * 8192, &mdo, full, i * 64, a.h, a.c * kC, a.b);
    if (DELTA) bulk_g2s(At_, p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, 8192, full);
  };
  auto load_q = [&](const At& a) {
    // scale * gamma * q: built below from q, or - channel-wise gate - read as the record the forward's prepare kernel left
    if (CW) bulk_g2s(QG, p.saved + p.lay.qg + static_cast<size_t>(a.z) * 16384, 16384, full);
    else for (int i = 0; i < KW / 64; ++i) tma_load_4d(QG + i * 8192, &mq, full, i * 64, a.h, a.c * kC, a.b);
    if (DELTA) bulk_g2s(Wt, p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w, 16384, full);
  };
  auto fetch_gates = [&](const At& a, float* o) {
    if (p.gate == LETHE_GATE_SCALAR) warp_copy_gates(p, p.g, a.b, a.c, a.h, lane, o);
  };
  // what the loads will want, to L2; not channel-wise, where nothing is converted and HBM is the bound (8192 chunks: 127 us without, 134
  // with; scalar gate without the delta term, d_v = 64, 1692 chunks 22.5 without, 20 with)
  auto prefetch = [&](const At& a) {
    for (int i = 0; i < V / 64; ++i) tma_prefetch_4d(&mdo, i * 64, a.h, a.c * kC, a.b);
    for (int i = 0; i < KW / 64; ++i) tma_prefetch_4d(&mq, i * 64, a.h, a.c * kC, a.b);
    if (DELTA) {
      bulk_prefetch(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, 8192);
      bulk_prefetch(p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w, 16384);
    }
  };

  if (tid == 0) {
    cs->abort_flag = 0;
    mbar_init(full, 1);
    mbar_init(mma, 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, V);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  griddep_launch();
  if (tid == 0) {
    const At a = at(blockIdx.x);
    load_do(a);
    load_q(a);
  }
  if (!CW && warp == 1) {
    fetch_gates(at(blockIdx.x), sgs);
    warp_scaled_gammas(p, lane, sgs);
  }
  if (!CW) __syncthreads();

  uint32_t ph = 0, pm = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const At a = at(n);
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    if (!CW && warp == 1 && more) fetch_gates(at(n + gridDim.x), sgs + (ph ^ 1u) * 64);
    mbar_wait_warp(full, ph, ctl, 401);
    if (!CW) {
      const float* sg = sgs + ph * 64;
      constexpr int kN = KW * 8 / kPreThreads;
      uint4 c[kN];
      float f[kN];
#pragma unroll
      for (int u = 0; u < kN; ++u) {                 // (all loads ahead of the first store: see output_kernel)
        const int idx = tid + u * kPreThreads, r = idx / (KW / 8);
        c[u] = tile_ld_chunk(QG, r, idx % (KW / 8), 64);
        f[u] = sg[r];
      }
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        const int idx = tid + u * kPreThreads, r = idx / (KW / 8);
        float x[8];
        unpack8_in(c[u], x, p.qk16);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= f[u];
        tile_st_chunk(QG, r, idx % (KW / 8), 64, pack8_f16(x));
      }
    }
    for (int idx = tid; idx < 64 * (V / 8); idx += kPreThreads) {
      uint4* c = reinterpret_cast<uint4*>(DO + idx * 16);
      float x[8];
      unpack8_bf16(*c, x);
      *c = pack8_f16(x);
    }
    sync_for_issue();
    if (DELTA) {
      if (warp == 0) {      // rows 64-127: A^T do
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, tmem, Tile{smem_u32(At_) - 8192, 64, true}, Tile{smem_u32(DO), 64, true}, V, 64, 0u);
        umma_commit_led(leader, mma);
      }
      __syncwarp();
      if (!CW && warp == 1 && more) warp_scaled_gammas(p, lane, sgs + (ph ^ 1u) * 64);
      wait_products(mma, pm, ctl, 402);
      if (quad >= 2) {
#pragma unroll
        for (int jj = 0; jj < V / 64; ++jj) {
          const int cb = half * (V / 2) + jj * 32;
          float d[32];
          tmem_ld32(tmem + lane_base + cb, d);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) tile_st_chunk(DVL, row - 64, cb / 8 + i, 64, pack8_f16(d + 8 * i));
        }
      }
      sync_for_issue();
    }
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(QG), 64, true}, Tile{smem_u32(DO), 64, true}, V, 64, 0u);
      if (DELTA) issue_product_led(leader, tmem, Tile{smem_u32(Wt), 64, true}, Tile{smem_u32(DVL), 64, true}, V, 64, 1u, true);
      umma_commit_led(leader, mma);
    } else if (!CW && warp == 2 && lane == 0 && more) {
      prefetch(at(n + gridDim.x));
    }
    __syncwarp();
    if (!DELTA && !CW && warp == 1 && more) warp_scaled_gammas(p, lane, sgs + (ph ^ 1u) * 64);
    wait_products(mma, pm, ctl, 403);
    if (tid == 0 && more) load_do(at(n + gridDim.x));
    unsigned char* SR = QG;   // q and w are dead: Rb is staged there as its record image
#pragma unroll
    for (int jj = 0; jj < V / 64; ++jj) {
      const int cb = half * (V / 2) + jj * 32;
      float d[32];
      tmem_ld32(tmem + lane_base + cb, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (DELTA) *reinterpret_cast<uint4*>(SR + rrec_off(row, cb / 8 + i)) = pack8_f16(d + 8 * i);
        else if (row < KW) tile_st_chunk(SR, row, cb / 8 + i, KW, pack8_f16(d + 8 * i));     // no delta term: plain tile image
      }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (tid == 0) {
      store_image<V, KW>(p.scratch + p.lay.rb + static_cast<size_t>(a.z) * p.lay.sz_rb, SR);
      bulk_commit();
      bulk_wait_read();
      if (more) load_q(at(n + gridDim.x));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, V);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA, bool CW, int KW = kK>
static int launch_pre_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mdo, cudaStream_t st) {
  using S = PreSmem<V, DELTA, KW>;
  static SmemAttr attr;
  if (attr.set(bwd_pre_kernel<V, DELTA, CW, KW>, S::kBytes)) return kErrLaunch;
  const int sms = sm_count(), n = p.nbh * p.cn;
  if (sms <= 0) return kErrDevice;
  // Not launched early: its CTAs would hold room that the kernel before, or one of another stream, could use.  Captured step,
  // us, plain / early, scalar gate, d_v = 64: 512 chunks 107 / 116, 2048 335 / 341, 4096 572 / 597; channel-wise, d_v = 128: 512
  // 190 / 199, 8192 2074 / 2046 (early is the better one at the largest, scalar d_v = 128 at 4096 842 / 815 too); one chain: no
  // more than 1 % either way up to 2048 chunks, 4096 596 / 614.
  bwd_pre_kernel<V, DELTA, CW, KW><<<n < S::kCtas * sms ? n : S::kCtas * sms, kPreThreads, S::kBytes, st>>>(p, mq, mdo);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
int launch_bwd_pre(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mdo, cudaStream_t st) {
  if (p.gate == LETHE_GATE_CHANNEL) {
    if (p.V == 64) return p.delta ? launch_pre_t<64, true, true>(p, mq, mdo, st) : launch_pre_t<64, false, true>(p, mq, mdo, st);
    return p.delta ? launch_pre_t<128, true, true>(p, mq, mdo, st) : launch_pre_t<128, false, true>(p, mq, mdo, st);
  }
  if (p.Kw == 64) return p.V == 64 ? launch_pre_t<64, false, false, 64>(p, mq, mdo, st) : launch_pre_t<128, false, false, 64>(p, mq, mdo, st);
  if (p.V == 64) return p.delta ? launch_pre_t<64, true, false>(p, mq, mdo, st) : launch_pre_t<64, false, false>(p, mq, mdo, st);
  return p.delta ? launch_pre_t<128, true, false>(p, mq, mdo, st) : launch_pre_t<128, false, false>(p, mq, mdo, st);
}

}  // namespace lg
