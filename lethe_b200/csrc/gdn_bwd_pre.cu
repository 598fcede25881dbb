// Input of the adjoint state scan, chunk-parallel: one CTA of 128 threads per chunk,
//   Rb = (scale gamma q)^T do - w^T (A^T do)
// (reference: the terms of the reverse scan K#1, gdn2_assemble.py:71-99).
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA, bool CW>
__global__ void __launch_bounds__(128)
bwd_pre_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mdo) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = CW ? align1024(smem_raw) : align1024_generic(smem_raw);   // measured per variant
  unsigned char* QG = sm;                    // 16 KB: scale gamma q (64 x 128)
  unsigned char* Wt = QG + 16384;            // 16 KB: w
  unsigned char* DO = Wt + 16384;            // do (64 x V)
  unsigned char* TAt = DO + V * 128;         // 16 KB: [T | A]
  unsigned char* DVL = TAt + 16384;          // A^T do (64 x V)
  float* fs = reinterpret_cast<float*>(DVL + V * 128);
  float* Gs = fs;
  float* tmp = fs + 64;
  CtaShared* cs = reinterpret_cast<CtaShared*>(fs + 72);

  const int tid = threadIdx.x, warp = tid >> 5;
  const int bh = p.bh0 + blockIdx.x / p.cn, c = p.c0 + blockIdx.x % p.cn, z = bh * p.NT + c, b = bh / p.H, h = bh % p.H;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t* bar_load = &cs->bar[0];
  uint64_t* bar_mma = &cs->bar[1];
  if (tid == 0) {
    cs->abort_flag = 0;
    mbar_init(bar_load, 1);
    mbar_init(bar_mma, 1);
    fence_mbar_init();
    fence_proxy_async();
    mbar_expect_tx(bar_load, 16384u + V * 128u + (DELTA ? 32768u : 0u));
    // scale * gamma * q: built below from q, or - channel-wise gate - read as the record the forward's prepare kernel left
    if (CW) bulk_g2s(QG, p.saved + p.lay.qg + static_cast<size_t>(z) * 16384, 16384, bar_load);
    else for (int a = 0; a < 2; ++a) tma_load_4d(QG + a * 8192, &mq, bar_load, a * 64, h, c * kC, b);
    for (int a = 0; a < V / 64; ++a) tma_load_4d(DO + a * 8192, &mdo, bar_load, a * 64, h, c * kC, b);
    if (DELTA) {
      bulk_g2s(Wt, p.saved + p.lay.w + static_cast<size_t>(z) * p.lay.sz_w, 16384, bar_load);
      bulk_g2s(TAt, p.saved + p.lay.ta + static_cast<size_t>(z) * p.lay.sz_ta, 16384, bar_load);
    }
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, 2 * V);     // two accumulators of V columns: three CTAs fit an SM at d_v = 64
    tmem_relinquish();
  }
  float gval = 0.f;
  if (tid < p.rows_of(c) && p.gate == LETHE_GATE_SCALAR) gval = p.g[(static_cast<size_t>(b) * p.L + c * kC + tid) * p.H + h];
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot;
  const float G = chunk_cumsum(gval, tid, tmp);
  if (tid < 64) Gs[tid] = G;
  __syncthreads();
  mbar_wait_warp(bar_load, 0, ctl, 401);
  if (!CW) {
    for (int idx = tid; idx < 64 * 16; idx += 128) {
      const int r = idx >> 4, ch = idx & 15;
      float x[8];
      unpack8_in(tile_ld_chunk(QG, r, ch, 64), x, p.qk16);
      const float sg = p.scale * __expf(Gs[r]);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] *= sg;
      tile_st_chunk(QG, r, ch, 64, pack8_f16(x));
    }
  }
  for (int idx = tid; idx < 64 * (V / 8); idx += 128) {
    const int r = idx / (V / 8), ch = idx % (V / 8);
    float x[8];
    unpack8_bf16(tile_ld_chunk(DO, r, ch, 64), x);
    tile_st_chunk(DO, r, ch, 64, pack8_f16(x));
  }
  sync_for_issue();
  uint32_t ph = 0;
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  if (DELTA) {
    // rows 64-127: A^T do
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(TAt), 64, true}, Tile{smem_u32(DO), 64, true}, V, 64, 0u);
      issue_product_led(leader, tmem + V, Tile{smem_u32(QG), 64, true}, Tile{smem_u32(DO), 64, true}, V, 64, 0u);
      umma_commit_led(leader, bar_mma);
    }
    wait_products(bar_mma, ph, ctl, 402);
    if (tid >= 64) {
#pragma unroll
      for (int jb = 0; jb < V / 32; ++jb) {
        float d[32];
        tmem_ld32(tmem + lane_base + jb * 32, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(DVL, tid - 64, jb * 4 + i, 64, pack8_f16(d + 8 * i));
      }
    }
    sync_for_issue();
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem + V, Tile{smem_u32(Wt), 64, true}, Tile{smem_u32(DVL), 64, true}, V, 64, 1u, true);
      umma_commit_led(leader, bar_mma);
    }
  } else if (warp == 0) {
    tc_fence_after();
    const uint32_t leader = elect_leader();
    issue_product_led(leader, tmem + V, Tile{smem_u32(QG), 64, true}, Tile{smem_u32(DO), 64, true}, V, 64, 0u);
    umma_commit_led(leader, bar_mma);
  }
  wait_products(bar_mma, ph, ctl, 403);
  {
    unsigned char* SR = QG;   // q and w are dead: Rb is staged there as its record image
#pragma unroll
    for (int jb = 0; jb < V / 32; ++jb) {
      float d[32];
      tmem_ld32(tmem + V + lane_base + jb * 32, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (DELTA) *reinterpret_cast<uint4*>(SR + rrec_off(tid, jb * 4 + i)) = pack8_f16(d + 8 * i);
        else tile_st_chunk(SR, tid, jb * 4 + i, 128, pack8_f16(d + 8 * i));     // no delta term: plain tile image
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(p.scratch + p.lay.rb + static_cast<size_t>(z) * p.lay.sz_rb, SR, V * 256);
      bulk_commit();
      bulk_wait_read();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 2 * V);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA, bool CW>
static int launch_pre_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mdo, cudaStream_t st) {
  const int smem = 16384 * 3 + V * 256 + 128 * 4 + 1024;
  static SmemAttr attr;
  if (attr.set(bwd_pre_kernel<V, DELTA, CW>, smem)) return kErrLaunch;
  bwd_pre_kernel<V, DELTA, CW><<<p.nbh * p.cn, 128, smem, st>>>(p, mq, mdo);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
int launch_bwd_pre(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mdo, cudaStream_t st) {
  if (p.gate == LETHE_GATE_CHANNEL) {
    if (p.V == 64) return p.delta ? launch_pre_t<64, true, true>(p, mq, mdo, st) : launch_pre_t<64, false, true>(p, mq, mdo, st);
    return p.delta ? launch_pre_t<128, true, true>(p, mq, mdo, st) : launch_pre_t<128, false, true>(p, mq, mdo, st);
  }
  if (p.V == 64) return p.delta ? launch_pre_t<64, true, false>(p, mq, mdo, st) : launch_pre_t<64, false, false>(p, mq, mdo, st);
  return p.delta ? launch_pre_t<128, true, false>(p, mq, mdo, st) : launch_pre_t<128, false, false>(p, mq, mdo, st);
}

}  // namespace lg
