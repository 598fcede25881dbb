// Chunk-parallel forward kernels: `prepare` (UT / WY transform and the per-chunk state map) and
// `output` (v_new and o from the chunk-entry states).  One CTA per chunk: 256 threads in `prepare`,
// 128 in `output`.
//
// All tensor-core products are tcgen05 with M = 128, fp16 operands in SW128 shared-memory tiles and
// fp32 accumulators in TMEM; two 64-row operands that share the other operand are stacked into one
// 128-row tile so that a single product serves both (rows 0-63 of the accumulator belong to the
// first, rows 64-127 to the second).
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

constexpr int kMs = 68;  // row stride (floats) of the fp32 copy of M used by the inverse

// ---------------------------------------------------------------------------------------------
// prepare: per chunk
//   G = cumsum(g), ratio[i,s] = exp(G_i - G_s) (s <= i)
//   [KK; QK] = [k; q] k^T                                    (product 1)
//   M = strict_lower(beta_i ratio KK), A = tril(scale ratio QK), T = (I + M)^-1  (fp32, CUDA cores)
//   [w | u] = T [beta gamma k | beta v]                      (product 2)
//   [P | R] = kd^T [w | u],  kd = k exp(G_last - G_i)        (product 3)
// Reference: gdn2_chunkwise.py:130-158 of the reference project; P and R fold its state update
// h' = exp(G_last) h + kd^T (u - w h) into h' = exp(G_last) h - P h + R.
// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA>
__global__ void __launch_bounds__(256)
prepare_kernel(const Problem p, const __grid_constant__ CUtensorMap mq,
               const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mv) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = DELTA ? align1024(smem_raw) : align1024_generic(smem_raw);   // measured per variant
  unsigned char* KQ = sm;                      // 32 KB: rows 0-63 k, rows 64-127 q; later M (fp32), then [w | u]
  unsigned char* BGK = sm + 32768;             // 16 KB: beta gamma k   (64 x 128)
  unsigned char* BV = BGK + 16384;             // beta v (64 x V), directly behind BGK: one N = 128 + V operand
  unsigned char* KD = BV + V * 128;            // 16 KB: kd            (64 x 128)
  unsigned char* TA = KD + 16384;              // 16 KB: [T; A]        (128 x 64)
  float* fs = reinterpret_cast<float*>(TA + 16384);
  float* Gs = fs;            // [64] cumulative log decay
  float* betas = fs + 64;    // [64]
  float* decs = fs + 128;    // [64] exp(G_last - G_i)
  float* bgs = fs + 192;     // [64] beta_i exp(G_i)
  float* tmp = fs + 256;     // [2]
  CtaShared* cs = reinterpret_cast<CtaShared*>(fs + 264);
  float* Msm = reinterpret_cast<float*>(KQ);           // [64][kMs]
  float* Tsm = Msm + 64 * kMs;                          // scratch of the inverse (kInvScratchFloats)
  unsigned char* WU = KQ;

  // Threads 0-127 and 128-255 reach the same TMEM lanes (lane quadrant = warp & 3): the two halves take
  // the same rows and split the columns of every epilogue.
  const int tid = threadIdx.x, warp = tid >> 5, tq = tid & 127, half = tid >> 7;
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
    mbar_expect_tx(bar_load, 32768u + V * 128u);
    for (int a = 0; a < 2; ++a) {
      tma_load_4d(KQ + a * 16384, &mk, bar_load, a * 64, h, c * kC, b);
      tma_load_4d(KQ + a * 16384 + 8192, &mq, bar_load, a * 64, h, c * kC, b);
    }
    for (int a = 0; a < V / 64; ++a) tma_load_4d(BV + a * 8192, &mv, bar_load, a * 64, h, c * kC, b);
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, 256);
    tmem_relinquish();
  }
  float gval = 0.f, bval = 1.f;
  if (tid < p.rows_of(c)) {
    const size_t tok = (static_cast<size_t>(b) * p.L + c * kC + tid) * p.H + h;
    if (p.gate == LETHE_GATE_SCALAR) gval = p.g[tok];
    if (DELTA) bval = p.beta[tok];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot;


  // ---- gate: cumulative log decay of the chunk
  const float G = chunk_cumsum(gval, tid, tmp);
  if (tid < 64) {
    Gs[tid] = G;
    betas[tid] = bval;
  }
  __syncthreads();
  const float Glast = Gs[63];
  if (tid < 64) {
    decs[tid] = __expf(Glast - G);
    bgs[tid] = bval * __expf(G);
  }
  if (tid < kK) reinterpret_cast<float*>(p.saved + p.lay.ad)[static_cast<size_t>(z) * kK + tid] = __expf(Glast);
  __syncthreads();

  // ---- operands: k, q -> fp16 in place; kd, beta gamma k, beta v
  mbar_wait_warp(bar_load, 0, ctl, 201);
  for (int idx = tid; idx < 64 * 16; idx += 256) {
    const int r = idx >> 4, ch = idx & 15;
    float x[8], y[8];
    unpack8_in(tile_ld_chunk(KQ, r, ch, 128), x, p.qk16);
    tile_st_chunk(KQ, r, ch, 128, pack8_f16(x));
    const float de = decs[r];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = x[i] * de;
    tile_st_chunk(KD, r, ch, 64, pack8_f16(y));
    if (DELTA) {
      const float bg = bgs[r];
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] = x[i] * bg;
      tile_st_chunk(BGK, r, ch, 64, pack8_f16(y));
    }
    unpack8_in(tile_ld_chunk(KQ, 64 + r, ch, 128), x, p.qk16);
    tile_st_chunk(KQ, 64 + r, ch, 128, pack8_f16(x));
  }
  for (int idx = tid; idx < 64 * (V / 8); idx += 256) {
    const int r = idx / (V / 8), ch = idx % (V / 8);
    float x[8];
    unpack8_bf16(tile_ld_chunk(BV, r, ch, 64), x);
    const float be = DELTA ? betas[r] : 1.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= be;
    tile_st_chunk(BV, r, ch, 64, pack8_f16(x));
  }
  fence_proxy_async();
  __syncthreads();

  // ---- product 1: [KK; QK] = [k; q] k^T
  if (warp == 0) {
    tc_fence_after();
    const uint32_t leader = elect_leader();
    issue_product_led(leader, tmem, Tile{smem_u32(KQ), 128, false}, Tile{smem_u32(KQ), 128, false}, 64, 128, 0u);
    umma_commit_led(leader, bar_mma);
  }
  __syncwarp();
  mbar_wait_warp(bar_mma, 0, ctl, 202);
  tc_fence_after();
  const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
  {
    // each half takes 32 of the 64 columns; rows 0-31 (lane quadrant 0 of either operand half) have
    // nothing right of column 31, so the triangle is cut per warp
    const bool live = (half == 0) || ((warp & 1) != 0);
    float d[32];
    if (live) {
      tmem_ld32(tmem + lane_base + half * 32, d);
      tmem_ld_wait();
    }
    if (tq < 64) {
      if (DELTA) {
        const int r = tq;
        const float Gr = Gs[r], be = betas[r];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int s = half * 32 + j;
          float m = 0.f;
          if (live) m = (s < r) ? be * __expf(Gr - Gs[s]) * d[j] : 0.f;
          Msm[r * kMs + s] = m;
        }
      }
    } else {
      const int r = tq - 64;
      const float Gr = Gs[r];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int s8 = half * 4 + q;
        float a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = 0.f;
        if (live) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int s = s8 * 8 + i;
            a[i] = (s <= r) ? p.scale * __expf(Gr - Gs[s]) * d[q * 8 + i] : 0.f;
          }
        }
        tile_st_chunk(TA, 64 + r, s8, 128, pack8_f16(a));
      }
    }
  }
  tc_fence_before();
  __syncthreads();

  // ---- T = (I + M)^-1 (fp32, CUDA cores)
  if (DELTA) {
    unit_lower_inverse64_blocked<kMs>(Msm, Tsm, TA, tid);
  } else if (tid < 64) {
    {
#pragma unroll
      for (int i = 0; i < 64; ++i)
        *reinterpret_cast<__half*>(TA + sw128_off(i, tid, 128)) = __float2half_rn((i == tid) ? 1.f : 0.f);
    }
  }
  fence_proxy_async();
  __syncthreads();

  uint32_t ph = 1;
  if (DELTA) {
    // ---- product 2: [w | u] = T [beta gamma k | beta v]
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(TA), 128, false}, Tile{smem_u32(BGK), 64, true}, 128 + V, 64, 0u);
      umma_commit_led(leader, bar_mma);
      if (tid == 0) bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(z) * p.lay.sz_ta, TA, 16384);
      if (tid == 0) bulk_commit();
    }
    __syncwarp();
    mbar_wait_warp(bar_mma, ph, ctl, 203);
    ph ^= 1;
    tc_fence_after();
    if (tq < 64) {
      constexpr int kHalf2 = (128 + V) / 64;
#pragma unroll
      for (int jb = half * kHalf2; jb < (half + 1) * kHalf2; ++jb) {
        float d[32];
        tmem_ld32(tmem + lane_base + jb * 32, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(WU, tq, jb * 4 + i, 64, pack8_f16(d + 8 * i));
      }
    }
    tc_fence_before();
    fence_proxy_async();
    __syncthreads();
  } else if (tid == 0) {
    bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(z) * p.lay.sz_ta, TA, 16384);
    bulk_commit();
  }

  // ---- product 3: [P | R] = kd^T [w | u]   (no delta: R = kd^T v)
  constexpr int N3 = DELTA ? 128 + V : V;
  if (warp == 0) {
    tc_fence_after();
    const uint32_t leader = elect_leader();
    issue_product_led(leader, tmem, Tile{smem_u32(KD), 64, true}, Tile{smem_u32(DELTA ? WU : BV), 64, true}, N3, 64, 0u);
    umma_commit_led(leader, bar_mma);
    if (DELTA) {
      if (tid == 0) bulk_s2g(p.saved + p.lay.w + static_cast<size_t>(z) * p.lay.sz_w, WU, 16384);
      if (tid == 0) bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(z) * p.lay.sz_u, WU + 16384, V * 128);
    } else {
      if (tid == 0 && !p.lean) bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(z) * p.lay.sz_u, BV, V * 128);      // (u is v)
    }
    if (tid == 0) bulk_commit();
  }
  __syncwarp();
  mbar_wait_warp(bar_mma, ph, ctl, 204);
  tc_fence_after();
  // P and R are staged as their record images in tiles nothing reads any more and leave by bulk
  // stores: P behind BGK (beta gamma k, beta v, kd are dead), R where k and q were once the stores
  // of [w | u] have finished reading it.
  if (tid == 0) bulk_wait_read();
  __syncthreads();
  {
    unsigned char* SP = BGK;
    unsigned char* SR = KQ;
    constexpr int kHalf3 = N3 / 64;
#pragma unroll 1
    for (int jb = half * kHalf3; jb < (half + 1) * kHalf3; ++jb) {
      float d[32];
      tmem_ld32(tmem + lane_base + jb * 32, d);
      tmem_ld_wait();
      if (DELTA && jb < 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(SP, tq, jb * 4 + i, 128, pack8_f16(d + 8 * i));
      } else {
        const int c8 = (jb - (DELTA ? 4 : 0)) * 4;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (DELTA) *reinterpret_cast<uint4*>(SR + rrec_off(tq, c8 + i)) = pack8_f16(d + 8 * i);
          else tile_st_chunk(SR, tq, c8 + i, 128, pack8_f16(d + 8 * i));     // no delta term: plain tile image
        }
      }
    }
    fence_proxy_async();
    __syncthreads();
    if (tid == 0) {
      if (DELTA) bulk_s2g(p.saved + p.lay.p + static_cast<size_t>(z) * p.lay.sz_p, SP, 32768);
      bulk_s2g(p.saved + p.lay.r + static_cast<size_t>(z) * p.lay.sz_r, SR, V * 256);
      bulk_commit();
    }
  }
  if (tid == 0) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------------
// output: per chunk, given the state h entering it
//   [w h ; (scale gamma q) h] = [w; qg] h                    (product 1)
//   v_new = u - w h
//   o = qg h + A v_new                                       (product 2 accumulates onto rows 64-127)
// Reference: gdn2_chunkwise.py:146-153.
//
// Bound by HBM (120 KB per chunk at d_v = 128, channel-wise gate).  Persistent CTAs; results leave as tensor-map / bulk
// stores from dead tiles (o where w was, v_new where u was).  Channel-wise, d_v = 128: one CTA per SM with two stages, a
// chunk's tiles arrive while the chunk before is computed (8192 chunks: 193 -> 152 us, 0.99 of the copy bandwidth on its
// bytes).  Shorter chunks and those whose q and v are converted here are bound by the chain of latencies, which two or
// three CTAs of one stage each hide better (scalar gate, d_v = 64, 4096 chunks: 59 us against 71 us with two stages;
// d_v = 128 without the delta term: 78 against 86).
// ---------------------------------------------------------------------------------------------
constexpr int kOutThreads = 256;

template <int V, bool CW>
struct OutSmem {
  static constexpr int oA = 32768;                   // behind [w; qg]: A (its 128-row view starts 64 rows early)
  static constexpr int oH = oA + 8192;               // state image
  static constexpr int oU = oH + V * 256;            // u, then v_new
  static constexpr int kStage = oU + V * 128, kStages = V == 64 || !CW ? 1 : 2, kCtas = V == 64 ? 3 : CW ? 1 : 2;
  static constexpr int kBytes = kStages * kStage + 2 * 256 + static_cast<int>(sizeof(CtaShared)) + 1024;
};

template <int V, bool DELTA, bool CW>
__global__ void __launch_bounds__(kOutThreads, OutSmem<V, CW>::kCtas)
output_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mv,
              const __grid_constant__ CUtensorMap mo) {
  using S = OutSmem<V, CW>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  float* sgs = reinterpret_cast<float*>(sm + S::kStages * S::kStage);      // [2][64] scale gamma (scalar gate)
  CtaShared* cs = reinterpret_cast<CtaShared*>(sgs + 128);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, half = warp >> 2;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *full = &cs->bar[0], *m1 = &cs->bar[2], *m2 = &cs->bar[3];
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
  auto load = [&](const At& a, int s) {              // everything but h (tid 0)
    unsigned char* t = sm + s * S::kStage;
    mbar_expect_tx(&full[s], 16384u + (DELTA ? 16384u : 0u) + V * 128u + 8192u + V * 256u);
    for (int i = 0; i < 2; ++i) {
      // the query operand: q from the user tensor (scaled below), or - channel-wise gate - the record of
      // scale * gamma * q that the prepare kernel left (two 64-row atoms of 8 KB)
      if (CW) bulk_g2s(t + i * 16384 + 8192, p.saved + p.lay.qg + static_cast<size_t>(a.z) * 16384 + i * 8192, 8192, &full[s]);
      else tma_load_4d(t + i * 16384 + 8192, &mq, &full[s], i * 64, a.h, a.c * kC, a.b);
      if (DELTA) bulk_g2s(t + i * 16384, p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w + i * 8192, 8192, &full[s]);
    }
    bulk_g2s(t + S::oA, p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, 8192, &full[s]);
    if (DELTA) bulk_g2s(t + S::oU, p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, V * 128, &full[s]);
    else for (int i = 0; i < V / 64; ++i) tma_load_4d(t + S::oU + i * 8192, &mv, &full[s], i * 64, a.h, a.c * kC, a.b);    // v_new = v
  };
  auto load_h = [&](const At& a, int s) {
    bulk_g2s(sm + s * S::kStage + S::oH, p.saved + p.lay.hc + static_cast<size_t>(a.z + a.bh) * p.lay.sz_hc, V * 256, &full[s]);
  };
  auto gates = [&](const At& a, float* o) { warp_scaled_gammas(p, a.b, a.c, a.h, lane, o); };

  const int n0 = blockIdx.x, n1 = n0 + gridDim.x;
  if (tid == 0) {
    cs->abort_flag = 0;
    for (int i = 0; i < 4; ++i) mbar_init(&cs->bar[i], 1);
    fence_mbar_init();
    fence_proxy_async();
    load(at(n0), 0);                                 // inputs and records older than the scan
    if (S::kStages == 2 && n1 < nchunks) load(at(n1), 1);
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, V);
    tmem_relinquish();
  }
  if (!CW && warp == 1) gates(at(n0), sgs);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  griddep_wait();
  griddep_launch();
  if (tid == 0) {                                    // the state images, written by the scan just before this kernel
    load_h(at(n0), 0);
    if (S::kStages == 2 && n1 < nchunks) load_h(at(n1), 1);
  }

  int it = 0;
  for (int n = n0; n < nchunks; n += gridDim.x, ++it) {
    const At a = at(n);
    const int s = it % S::kStages, g2 = it & 1;
    const uint32_t ph = static_cast<uint32_t>(it & 1);
    unsigned char *WQ = sm + s * S::kStage, *At_ = WQ + S::oA, *HT = WQ + S::oH, *VN = WQ + S::oU;
    mbar_wait_warp(&full[s], static_cast<uint32_t>((it / S::kStages) & 1), ctl, 211);
    if (!CW) {
      const float* sg = sgs + g2 * 64;
      for (int idx = tid; idx < 64 * 16; idx += kOutThreads) {
        const int r = idx >> 4, ch = idx & 15;
        float x[8];
        unpack8_in(tile_ld_chunk(WQ, 64 + r, ch, 128), x, p.qk16);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= sg[r];
        tile_st_chunk(WQ, 64 + r, ch, 128, pack8_f16(x));
      }
    }
    if (!DELTA) {
      for (int idx = tid; idx < 64 * (V / 8); idx += kOutThreads) {
        uint4* c = reinterpret_cast<uint4*>(VN + idx * 16);
        float x[8];
        unpack8_bf16(*c, x);
        *c = pack8_f16(x);
      }
    }
    if (!CW || !DELTA) sync_for_issue();             // (otherwise nothing was written, and the chunk before ended in a barrier)
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(WQ), 128, false}, Tile{smem_u32(HT), 128, true}, V, 128, 0u);
      if (!DELTA) issue_product_led(leader, tmem, Tile{smem_u32(At_) - 8192, 64, false}, Tile{smem_u32(VN), 64, true}, V, 64, 1u);
      umma_commit_led(leader, DELTA ? m1 : m2);
      if (S::kStages == 2 && tid == 0 && it > 0 && n + static_cast<int>(gridDim.x) < nchunks) {      // the other stage's results have left it
        bulk_wait_read();
        const At nx = at(n + gridDim.x);
        load(nx, s ^ 1);
        load_h(nx, s ^ 1);
      }
    }
    __syncwarp();
    if (!CW && warp == 1 && n + static_cast<int>(gridDim.x) < nchunks) gates(at(n + gridDim.x), sgs + (g2 ^ 1) * 64);
    if (DELTA) {
      mbar_wait_warp(m1, ph, ctl, 212);
      tc_fence_after();
      if (quad < 2) {                                // v_new, where u was
        const int r = quad * 32 + lane;
#pragma unroll
        for (int jj = 0; jj < V / 64; ++jj) {
          const int cb = half * (V / 2) + jj * 32;
          float d[32];
          tmem_ld32(tmem + lane_base + cb, d);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float u8[8];
            unpack8_f16(tile_ld_chunk(VN, r, cb / 8 + i, 64), u8);
#pragma unroll
            for (int e = 0; e < 8; ++e) u8[e] -= d[8 * i + e];
            tile_st_chunk(VN, r, cb / 8 + i, 64, pack8_f16(u8));
          }
        }
      }
      sync_for_issue();
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, tmem, Tile{smem_u32(At_) - 8192, 64, false}, Tile{smem_u32(VN), 64, true}, V, 64, 1u);
        umma_commit_led(leader, m2);
      }
      __syncwarp();
    }
    mbar_wait_warp(m2, ph, ctl, 213);
    tc_fence_after();
    if (quad >= 2) {                                 // o as a token-major tile where w (without delta: nothing) was
      const int r = (quad - 2) * 32 + lane;
#pragma unroll
      for (int jj = 0; jj < V / 64; ++jj) {
        const int cb = half * (V / 2) + jj * 32;
        float d[32];
        tmem_ld32(tmem + lane_base + cb, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(WQ + (cb >> 6) * 16384 + r * 128 + ((((cb >> 3) + i) & 7) ^ (r & 7)) * 16) = pack8_bf16(d + 8 * i);
      }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      for (int i = 0; i < V / 64; ++i) tma_store_4d(&mo, WQ + i * 16384, i * 64, a.h, a.c * kC, a.b);
      if (DELTA || !p.lean) bulk_s2g(p.saved + p.lay.vn + static_cast<size_t>(a.z) * p.lay.sz_vn, VN, V * 128);
      bulk_commit();
      if (S::kStages == 1 && n + static_cast<int>(gridDim.x) < nchunks) {
        bulk_wait_read();
        const At nx = at(n + gridDim.x);
        load(nx, 0);
        load_h(nx, 0);
      }
    }
  }
  if (tid == 0) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, V);
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
template <int V, bool DELTA>
static int launch_prepare_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk,
                            const CUtensorMap& mv, cudaStream_t st) {
  const int smem = 32768 + 16384 + V * 128 + 16384 + 16384 + 264 * 4 + static_cast<int>(sizeof(CtaShared)) + 1024;
  auto kern = prepare_kernel<V, DELTA>;
  static SmemAttr attr;
  if (attr.set(kern, smem)) return kErrLaunch;
  kern<<<p.nbh * p.cn, 256, smem, st>>>(p, mq, mk, mv);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
template <int V, bool DELTA, bool CW>
static int launch_output_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  constexpr int smem = OutSmem<V, CW>::kBytes;
  auto kern = output_kernel<V, DELTA, CW>;
  static SmemAttr attr;
  if (attr.set(kern, smem)) return kErrLaunch;
  const int sms = sm_count(), n = p.nbh * p.cn;
  if (sms <= 0) return kErrDevice;
  if (launch_dependent(kern, dim3(n < OutSmem<V, CW>::kCtas * sms ? n : OutSmem<V, CW>::kCtas * sms), dim3(kOutThreads), smem, st, p, mq, mv, mo) != cudaSuccess) return kErrLaunch;
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

int launch_prepare(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                   cudaStream_t st) {
  if (p.V == 64) return p.delta ? launch_prepare_t<64, true>(p, mq, mk, mv, st) : launch_prepare_t<64, false>(p, mq, mk, mv, st);
  return p.delta ? launch_prepare_t<128, true>(p, mq, mk, mv, st) : launch_prepare_t<128, false>(p, mq, mk, mv, st);
}
template <bool CW>
static int launch_output_cw(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  if (p.V == 64) return p.delta ? launch_output_t<64, true, CW>(p, mq, mv, mo, st) : launch_output_t<64, false, CW>(p, mq, mv, mo, st);
  return p.delta ? launch_output_t<128, true, CW>(p, mq, mv, mo, st) : launch_output_t<128, false, CW>(p, mq, mv, mo, st);
}
int launch_output(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  return p.gate == LETHE_GATE_CHANNEL ? launch_output_cw<true>(p, mq, mv, mo, st) : launch_output_cw<false>(p, mq, mv, mo, st);
}

}  // namespace lg
