// Chunk-parallel forward kernels: `prepare` (UT / WY transform and the per-chunk state map) and
// `output` (v_new and o from the chunk-entry states).  Persistent CTAs of 256 threads, one chunk at a time.
//
// All tensor-core products are tcgen05 with M = 128, fp16 operands in SW128 shared-memory tiles and
// fp32 accumulators in TMEM; two 64-row operands that share the other operand are stacked into one
// 128-row tile so that a single product serves both (rows 0-63 of the accumulator belong to the
// first, rows 64-127 to the second).
#include "gdn_inverse.cuh"
#include "host_util.h"

namespace lg {

// ---------------------------------------------------------------------------------------------
// prepare, scalar gate (or none): per chunk
//   G = cumsum(g), ratio[i,s] = exp(G_i - G_s) (s <= i)
//   [KK; QK] = [k; q] k^T                                              (product 1)
//   M = strict_lower(beta_i ratio KK), A = tril(scale ratio QK), T = (I + M)^-1  (fp32, CUDA cores)
//   w = (T diag(beta gamma)) k,  u = (T diag(beta)) v                  (product 2, both T's stacked)
//   [P | R] = kd^T [w | u],  kd = k exp(G_last - G_i)                  (product 3)
// Reference: gdn2_chunkwise.py:130-158 of the reference project; P and R fold its state update
// h' = exp(G_last) h + kd^T (u - w h) into h' = exp(G_last) h - P h + R.
//
// Bound by HBM (128 KB per chunk at d_v = 64) and by the chain of phases of a chunk, about 9 k cycles.  Two persistent CTAs
// per SM; the next k, q and v are fetched as soon as their tiles are dead (k and q under product 3 and the last epilogue),
// and the gates are summed a chunk ahead by one warp.  With one CTA per chunk instead, the wait for the first loads and the
// start of the CTA were 40 % of its time.  The gates are applied to the columns of T, not to k and v: half the elements.
// 4096 chunks: d_v = 64 167 -> 132 us, d_v = 128 183 -> 143; without the delta term (below) d_v = 128 121 -> 85.  With loads ahead of the
// stores to swizzled tiles, the abort flag behind the waits and the first gates summed under the first product 132 -> 127, 512 chunks 21.6
// -> 20.3, 128 chunks 9.1 -> 8.5.
// The gates of the next chunk come by asynchronous copies to shared memory, its place from one thread, and (not at d_v = 128) its
// tiles are prefetched to L2 under product 1: without the delta term d_v = 128 79 -> 70, with it within 2 %.
// ---------------------------------------------------------------------------------------------
constexpr int kPrepThreads = 256;

struct PrepGates {
  float G[64], beta[64], dec[64], bg[64];     // cumulative log decay; beta; exp(G_last - G); beta exp(G)
};

// Gates of a chunk by one warp, two neighbouring tokens per lane: fetched a chunk ahead, then summed; also the record of the
// chunk's whole decay.
__device__ __forceinline__ void prep_fetch_gates(const Problem& p, int b, int c, int h, int lane, PrepGates* o) {
  if (p.gate == LETHE_GATE_SCALAR) warp_copy_gates(p, p.g, b, c, h, lane, o->G);
  if (p.delta) warp_copy_gates(p, p.beta, b, c, h, lane, o->beta);
}
__device__ __forceinline__ void prep_gates(const Problem& p, int z, int lane, PrepGates* o) {
  async_copy_wait();
  float g[2] = {0.f, 0.f}, be[2] = {1.f, 1.f};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    if (p.gate == LETHE_GATE_SCALAR) g[e] = o->G[2 * lane + e];
    if (p.delta) be[e] = o->beta[2 * lane + e];
  }
  float sum = g[0] + g[1];
#pragma unroll
  for (int w = 1; w < 32; w <<= 1) {
    const float y = __shfl_up_sync(0xffffffffu, sum, w);
    if (lane >= w) sum += y;
  }
  const float G1 = sum, G0 = sum - g[1], last = __shfl_sync(0xffffffffu, sum, 31);
  *reinterpret_cast<float2*>(o->G + 2 * lane) = make_float2(G0, G1);
  *reinterpret_cast<float2*>(o->beta + 2 * lane) = make_float2(be[0], be[1]);
  *reinterpret_cast<float2*>(o->dec + 2 * lane) = make_float2(__expf(last - G0), __expf(last - G1));
  *reinterpret_cast<float2*>(o->bg + 2 * lane) = make_float2(be[0] * __expf(G0), be[1] * __expf(G1));
  const float a = __expf(last);
  *reinterpret_cast<float4*>(p.saved + p.lay.ad + static_cast<size_t>(z) * kK * 4 + lane * 16) = make_float4(a, a, a, a);
}

// k and q into the 128-row tile [k; q] (tid 0)
template <int KW = kK>
__device__ __forceinline__ void prep_load_kq(unsigned char* KQ, const CUtensorMap* mk, const CUtensorMap* mq, uint64_t* bar, const ChunkAt& a) {
  mbar_expect_tx(bar, KW * 256u);
  for (int t = 0; t < KW / 64; ++t) {
    tma_load_4d(KQ + t * 16384, mk, bar, t * 64, a.h, a.c * kC, a.b);
    tma_load_4d(KQ + t * 16384 + 8192, mq, bar, t * 64, a.h, a.c * kC, a.b);
  }
}
// ... and what a chunk will load to L2, under the products of the chunk before: its tiles are free late
template <int V, int KW = kK>
__device__ __forceinline__ void prep_prefetch(const CUtensorMap* mk, const CUtensorMap* mq, const CUtensorMap* mv, const ChunkAt& a) {
  for (int t = 0; t < KW / 64; ++t) {
    tma_prefetch_4d(mk, t * 64, a.h, a.c * kC, a.b);
    tma_prefetch_4d(mq, t * 64, a.h, a.c * kC, a.b);
  }
  for (int t = 0; t < V / 64; ++t) tma_prefetch_4d(mv, t * 64, a.h, a.c * kC, a.b);
}
template <int V>
__device__ __forceinline__ void prep_load_v(unsigned char* Vt, const CUtensorMap* mv, uint64_t* bar, const ChunkAt& a) {
  mbar_expect_tx(bar, V * 128u);
  for (int t = 0; t < V / 64; ++t) tma_load_4d(Vt + t * 8192, mv, bar, t * 64, a.h, a.c * kC, a.b);
}
// The rows of the tile [k; q] normalised, as lethe_gdn_l2norm_qk does (x rsqrt(sum x^2 + eps) in fp32, one rounding to fp16) and to its
// bits: every sum is formed in its order.  Four lanes have a row; the eight rows of a pass take the same 16-byte piece at a time, so the
// swizzle keeps them off one another's banks.  A kernel of its own took a launch and another pass over q and k (prefill of 1000 tokens,
// 8 heads: 26.6 us, now 21.5).
// kPass: passes whose loads come together, ahead of the first store
template <int KW = kK, int kPass = 2>
__device__ __forceinline__ void prep_normalise_rows(unsigned char* KQ, int r0, int part, int f16, float eps) {
  constexpr int kN = KW / 32;
  uint4 c[kPass][kN];
#pragma unroll
  for (int u = 0; u < kPass; ++u)
#pragma unroll
    for (int j = 0; j < kN; ++j) c[u][j] = tile_ld_chunk(KQ, r0 + 8 * u, part + 4 * j, 128);
#pragma unroll
  for (int u = 0; u < kPass; ++u) {
    float x[kN][8], sp[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      unpack8_in(c[u][j], x[j], f16);
      sp[j] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) sp[j] = fmaf(x[j][e], x[j][e], sp[j]);
    }
    // the order of row_sum: pieces 8 apart, then 4, 2 and 1
    float ss = kN == 4 ? (sp[0] + sp[kN - 2]) + (sp[1] + sp[kN - 1]) : sp[0] + sp[1];
    ss += __shfl_xor_sync(0xffffffffu, ss, 16);
    ss += __shfl_xor_sync(0xffffffffu, ss, 8);
    const float s = rsqrtf(ss + eps);
#pragma unroll
    for (int j = 0; j < kN; ++j) {
#pragma unroll
      for (int e = 0; e < 8; ++e) x[j][e] *= s;
      tile_st_chunk(KQ, r0 + 8 * u, part + 4 * j, 128, pack8_f16(x[j]));
    }
  }
}
template <int KW = kK, int kPass = 2>
__device__ __forceinline__ void prep_normalise(unsigned char* KQ, int warp, int lane, int f16, float eps) {
  const int r0 = warp * 16 + (lane & 7), part = lane >> 3;
#pragma unroll 1
  for (int r = 0; r < 16; r += 8 * kPass) prep_normalise_rows<KW, kPass>(KQ, r0 + r, part, f16, eps);
}
// ... on their way out: q for the output kernel, both for a backward (tid 0, behind a barrier)
__device__ __forceinline__ void prep_store_norm(const Problem& p, const NormMaps& mn, const unsigned char* KQ, const ChunkAt& a) {
  for (int t = 0; t < p.Kr / 64; ++t) {
    tma_store_4d(&mn.q, KQ + t * 16384 + 8192, t * 64, a.h, a.c * kC, a.b);
    if (p.keep_norm) tma_store_4d(&mn.k, KQ + t * 16384, t * 64, a.h, a.c * kC, a.b);
  }
  bulk_commit();
}
// a tile of bf16 to fp16 in place, whatever its shape
template <int N = kPrepThreads>
__device__ __forceinline__ void prep_to_f16(unsigned char* t, int bytes, int tid) {      // on N threads
  for (int i = tid * 16; i < bytes; i += N * 16) {
    float x[8];
    unpack8_bf16(*reinterpret_cast<const uint4*>(t + i), x);
    *reinterpret_cast<uint4*>(t + i) = pack8_f16(x);
  }
}
// kd = k exp(G_last - G), a 64-row tile
__device__ __forceinline__ void prep_kd(unsigned char* KD, const unsigned char* KQ, const float* dec, int tid) {
  constexpr int kN = 64 * 16 / kPrepThreads;
  uint4 c[kN];
  float f[kN];
#pragma unroll
  for (int u = 0; u < kN; ++u) {                  // (all loads ahead of the first store: see output_kernel)
    const int idx = tid + u * kPrepThreads;
    c[u] = tile_ld_chunk(KQ, idx >> 4, idx & 15, 128);
    f[u] = dec[idx >> 4];
  }
#pragma unroll
  for (int u = 0; u < kN; ++u) {
    const int idx = tid + u * kPrepThreads;
    float x[8];
    unpack8_f16(c[u], x);
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] *= f[u];
    tile_st_chunk(KD, idx >> 4, idx & 15, 64, pack8_f16(x));
  }
}
// 32 columns (from 32 half) of row r of a product, times the decay between the tokens and `f`; zero from column `end` on.
// Everything in registers first: with a store or a branch between them the exponentials run one at a time (2.7 k cycles).
// The exponent is not clamped: what it gives right of `end` is dropped, and left of it a clamp would hide a log decay above
// zero, and make "no decay" of the NaN between two tokens behind a decay of minus infinity.
__device__ __forceinline__ void prep_decay_row(float* d, const float* Gs, int r, int half, int end, float f) {
  const float Gr = Gs[r];
  float g[32];
#pragma unroll
  for (int q = 0; q < 4; ++q) ld8(Gs + half * 32 + 8 * q, g + 8 * q);
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float x = f * __expf(Gr - g[j]) * d[j];
    d[j] = half * 32 + j < end ? x : 0.f;
  }
}
// the 32 columns of row r of A: lane quadrants 0 of either half have nothing right of column 31 (live)
__device__ __forceinline__ void prep_row_a(unsigned char* A, const float* Gs, float* d, int r, int half, bool live, float scale) {
  if (live) prep_decay_row(d, Gs, r, half, r + 1, scale);
#pragma unroll
  for (int q = 0; q < 4; ++q) tile_st_chunk(A, r, half * 4 + q, 64, live ? pack8_f16(d + 8 * q) : make_uint4(0u, 0u, 0u, 0u));
}

template <int V>
struct PrepSmem {
  static constexpr int oTA = 32768;              // behind [k; q]: [T; A]; then, with kd, P on its way out
  static constexpr int oKD = oTA + 16384;        // M in fp32 and the scratch of its inverse (29 KB); then kd
  static constexpr int oW = oKD + 16384;         // [T diag(beta gamma); T diag(beta)]; then w; then R (d_v = 128: with u) on its way out
  static constexpr int oV = oW + 16384;          // v; then u
  static constexpr int kUsed = oV + V * 128, kBytes = kUsed + 2 * static_cast<int>(sizeof(PrepGates) + sizeof(ChunkAt)) + static_cast<int>(sizeof(CtaShared)) + 1024;
  static_assert((kInvMtFloats + kInvScratchFloats) * 4 <= 32768, "scratch of the inverse");
};

// NORM: q and k are normalised on the way in (as a branch it cost 1 to 3 % where they are not)
template <int V, bool NORM>
__global__ void __launch_bounds__(kPrepThreads, 2)
prepare_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
               const __grid_constant__ CUtensorMap mv, const __grid_constant__ NormMaps mn) {
  using S = PrepSmem<V>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  unsigned char *KQ = sm, *TA = sm + S::oTA, *KD = sm + S::oKD, *W = sm + S::oW, *Vt = sm + S::oV;
  float* Mt = reinterpret_cast<float*>(KD);
  PrepGates* gates = reinterpret_cast<PrepGates*>(sm + S::kUsed);
  ChunkAt* where = reinterpret_cast<ChunkAt*>(gates + 2);      // this chunk and the next
  CtaShared* cs = reinterpret_cast<CtaShared*>(where + 2);
  // Threads 0-127 and 128-255 reach the same TMEM lanes (lane quadrant = warp & 3): the two halves take
  // the same rows and split the columns of every epilogue.
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, half = warp >> 2, tq = tid & 127;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *full_kq = &cs->bar[0], *full_v = &cs->bar[1], *mma = &cs->bar[2];
  const int nchunks = p.nbh * p.cn;

  if (tid == 0) {
    cs->abort_flag = 0;
    for (int i = 0; i < 3; ++i) mbar_init(&cs->bar[i], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  {
    const ChunkAt a = chunk_at(p, blockIdx.x);       // (divisions and the maps' way here lie under the kernel before)
    if (tid == 0) {
      where[0] = a;
      prefetch_map(&mk);
      prefetch_map(&mq);
      prefetch_map(&mv);
    }
    griddep_wait();
    griddep_launch();
    if (tid == 0) {
      prep_load_kq(KQ, &mk, &mq, full_kq, a);
      prep_load_v<V>(Vt, &mv, full_v, a);
    }
    if (warp == 1) prep_fetch_gates(p, a.b, a.c, a.h, lane, gates);      // (summed under product 1: waited for here, they held it up)
  }
  __syncthreads();

  uint32_t ph = 0, pm = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const ChunkAt a = where[ph];
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    const PrepGates& gt = gates[ph];
    if (tid == kPrepThreads - 1 && more) where[ph ^ 1u] = chunk_at(p, n + gridDim.x);

    const bool first = n == static_cast<int>(blockIdx.x);
    mbar_wait_warp(full_kq, ph, ctl, 201);
    if (NORM) prep_normalise(KQ, warp, lane, p.qk16, p.l2_eps);
    else if (!p.qk16) prep_to_f16(KQ, 32768, tid);
    if (tid == 0 && !first) {
      bulk_wait_read();                              // P and R of the chunk before have left their tiles
      if (V == 128) prep_load_v<V>(Vt, &mv, full_v, a);
    }
    sync_for_issue();

    // ---- product 1: [KK; QK] = [k; q] k^T
    if (NORM) {
      if (tid == kPrepThreads - 1) prep_store_norm(p, mn, KQ, a);
      __syncwarp();
    }
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(KQ), 128, false}, Tile{smem_u32(KQ), 128, false}, 64, 128, 0u);
      umma_commit_led(leader, mma);
    } else if (warp == 1) {
      if (first) prep_gates(p, a.z, lane, gates);
      if (more) {
        const ChunkAt nx = where[ph ^ 1u];
        prep_fetch_gates(p, nx.b, nx.c, nx.h, lane, gates + (ph ^ 1u));
      }
    } else if (V == 64 && warp == 2 && lane == 0 && more) {      // (4096 chunks, us, without / with: d_v = 64 135 / 131, 128 143 / 148)
      prep_prefetch<V>(&mk, &mq, &mv, where[ph ^ 1u]);
    }
    if (first) __syncthreads();                      // the gates
    wait_products(mma, pm, ctl, 202);
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
        if (live) prep_decay_row(d, gt.G, tq, half, tq, gt.beta[tq]);
#pragma unroll
        for (int j = 0; j < 32; ++j) Mt[(half * 32 + j) * kMt + tq] = live ? d[j] : 0.f;
      } else {
        prep_row_a(TA + 8192, gt.G, d, tq - 64, half, live, p.scale);
      }
    }
    tc_fence_before();
    __syncthreads();

    // ---- T = (I + M)^-1 (fp32, CUDA cores); v to fp16 on the warps that have no part in its first step (d_v = 128: behind it, v
    // was requested late)
    if (V == 64 && tid >= 64) {
      mbar_wait_warp(full_v, ph, ctl, 203);
      prep_to_f16<kPrepThreads - 64>(Vt, V * 128, tid - 64);
    }
    unit_lower_inverse64(Mt, Mt, Mt + kInvMtFloats, TA, tid);
    if (V == 128) {
      mbar_wait_warp(full_v, ph, ctl, 203);
      prep_to_f16(Vt, V * 128, tid);
    }
    __syncthreads();
    {
      const int ch = tid & 7, r0 = tid >> 3;
      float bg[8], be[8];
      ld8(gt.bg + ch * 8, bg);
      ld8(gt.beta + ch * 8, be);
      const uint4 c[2] = {tile_ld_chunk(TA, r0, ch, 128), tile_ld_chunk(TA, r0 + kPrepThreads / 8, ch, 128)};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = r0 + u * (kPrepThreads / 8);
        float t[8], x[8];
        unpack8_f16(c[u], t);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = t[i] * bg[i];
        tile_st_chunk(W, r, ch, 128, pack8_f16(x));
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = t[i] * be[i];
        tile_st_chunk(W, 64 + r, ch, 128, pack8_f16(x));
      }
    }
    sync_for_issue();

    // ---- product 2: w in rows 0-63, u in rows 64-127
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(W), 128, false}, Tile{smem_u32(KQ), 128, true}, 128, 64, 0u);
      issue_product_led(leader, tmem + 128, Tile{smem_u32(W), 128, false}, Tile{smem_u32(Vt), 64, true}, V, 64, 0u);
      umma_commit_led(leader, mma);
      if (tid == 0) {
        if (p.lean < 2) bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta, TA, 16384);
        else bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, TA + 8192, 8192);      // A only
        bulk_commit();
      }
      __syncwarp();
    }
    prep_kd(KD, KQ, gt.dec, tid);                    // in its shadow
    wait_products(mma, pm, ctl, 204);
    if (quad < 2) {
#pragma unroll
      for (int jj = 0; jj < 2; ++jj) {
        const int cb = half * 64 + jj * 32;
        float d[32];
        tmem_ld32(tmem + lane_base + cb, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(W, tq, cb / 8 + i, 64, pack8_f16(d + 8 * i));
      }
    } else {
#pragma unroll
      for (int jj = 0; jj < V / 64; ++jj) {
        const int cb = half * (V / 2) + jj * 32;
        float d[32];
        tmem_ld32(tmem + 128 + lane_base + cb, d);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(Vt, tq - 64, cb / 8 + i, 64, pack8_f16(d + 8 * i));
      }
    }
    if (tid == 0) bulk_wait_read();                  // [T; A] have left their tile
    if (NORM && tid == kPrepThreads - 1) bulk_wait_read();      // ... and the normalised rows
    sync_for_issue();

    // ---- product 3: [P | R] = kd^T [w | u]
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(KD), 64, true}, Tile{smem_u32(W), 64, true}, 128, 64, 0u);
      issue_product_led(leader, tmem + 128, Tile{smem_u32(KD), 64, true}, Tile{smem_u32(Vt), 64, true}, V, 64, 0u);
      umma_commit_led(leader, mma);
      if (tid == 0) {
        if (more) prep_load_kq(KQ, &mk, &mq, full_kq, where[ph ^ 1u]);        // nothing reads k and q any more
        bulk_s2g(p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w, W, 16384);
        bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, Vt, V * 128);
        bulk_commit();
      }
    }
    __syncwarp();
    if (warp == 1 && more) prep_gates(p, where[ph ^ 1u].z, lane, gates + (ph ^ 1u));
    wait_products(mma, pm, ctl, 205);
    // P leaves from where [T; A] and kd were, R from where w (and u) were once their stores have read them
#pragma unroll
    for (int jj = 0; jj < 2; ++jj) {
      const int cb = half * 64 + jj * 32;
      float d[32];
      tmem_ld32(tmem + lane_base + cb, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) tile_st_chunk(TA, tq, cb / 8 + i, 128, pack8_f16(d + 8 * i));
    }
    fence_proxy_async();
    if (tid == 0) {
      bulk_wait_read();
      if (V == 64 && more) prep_load_v<V>(Vt, &mv, full_v, where[ph ^ 1u]);
    }
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(p.saved + p.lay.p + static_cast<size_t>(a.z) * p.lay.sz_p, TA, 32768);
      bulk_commit();
    }
#pragma unroll
    for (int jj = 0; jj < V / 64; ++jj) {
      const int cb = half * (V / 2) + jj * 32;
      float d[32];
      tmem_ld32(tmem + 128 + lane_base + cb, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(W + rrec_off(tq, cb / 8 + i)) = pack8_f16(d + 8 * i);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      bulk_s2g(p.saved + p.lay.r + static_cast<size_t>(a.z) * p.lay.sz_r, W, V * 256);
      bulk_commit();
    }
  }
  if (tid == 0) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 256);
}

// Without the delta term u = v, and only A and R = kd^T v are left: two independent products, one wait.
// KW: key channels of the tensors.  With 64 the other half of every tile, product and record is left out, here and in the kernels
// behind (what a product of 128 rows leaves in the lanes of the other 64 is not read): SSD, 36 pairs x 47 chunks, d_v = 64, us,
// 128 / 64: prepare 32 / 18, output 17 / 12, scan input 16 / 13, main 53 / 45, the training step 156 / 135.
template <int V, int KW>
struct PrepNdSmem {
  // R leaves from where kd (and as far as it is longer, v) was
  static constexpr int oA = KW * 256, oKD = oA + 8192, oV = oKD + KW * 128;
  static constexpr int kUsed = oV + V * 128, kBytes = kUsed + 2 * static_cast<int>(sizeof(PrepGates) + sizeof(ChunkAt)) + static_cast<int>(sizeof(CtaShared)) + 1024;
  static constexpr int kCols = V == 64 ? 128 : 256, kCtas = V == 64 ? 3 : 2;      // q k^T and R side by side in tensor memory
};

template <int V, int KW, bool NORM>
__global__ void __launch_bounds__(kPrepThreads, PrepNdSmem<V, KW>::kCtas)
prepare_nodelta_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                       const __grid_constant__ CUtensorMap mv, const __grid_constant__ NormMaps mn) {
  using S = PrepNdSmem<V, KW>;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  unsigned char *KQ = sm, *A = sm + S::oA, *KD = sm + S::oKD, *Vt = sm + S::oV;
  PrepGates* gates = reinterpret_cast<PrepGates*>(sm + S::kUsed);
  ChunkAt* where = reinterpret_cast<ChunkAt*>(gates + 2);      // this chunk and the next
  CtaShared* cs = reinterpret_cast<CtaShared*>(where + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, half = warp >> 2, tq = tid & 127;
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t *full_kq = &cs->bar[0], *full_v = &cs->bar[1], *mma = &cs->bar[2];
  const int nchunks = p.nbh * p.cn;

  if (tid == 0) {
    cs->abort_flag = 0;
    for (int i = 0; i < 3; ++i) mbar_init(&cs->bar[i], 1);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, S::kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  griddep_wait();
  griddep_launch();
  {
    const ChunkAt a = chunk_at(p, blockIdx.x);
    if (tid == 0) {
      where[0] = a;
      prep_load_kq<KW>(KQ, &mk, &mq, full_kq, a);
      prep_load_v<V>(Vt, &mv, full_v, a);
    }
    if (warp == 1) {
      prep_fetch_gates(p, a.b, a.c, a.h, lane, gates);
      prep_gates(p, a.z, lane, gates);
    }
  }
  __syncthreads();

  uint32_t ph = 0, pm = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const ChunkAt a = where[ph];
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    const PrepGates& gt = gates[ph];
    if (tid == kPrepThreads - 1 && more) where[ph ^ 1u] = chunk_at(p, n + gridDim.x);

    mbar_wait_warp(full_kq, ph, ctl, 206);
    const int f16 = NORM ? 1 : p.qk16;               // the type of the tile from here on
    if (NORM) {
      prep_normalise<KW, V == 64 && KW == kK ? 1 : 2>(KQ, warp, lane, p.qk16, p.l2_eps);
      fence_proxy_async();
      __syncthreads();
      if (tid == kPrepThreads - 1) prep_store_norm(p, mn, KQ, a);
    }
    for (int idx = tid; idx < KW * 8; idx += kPrepThreads) {
      const int r = idx / (KW / 8), ch = idx % (KW / 8);
      float x[8];
      unpack8_in(tile_ld_chunk(KQ, r, ch, 128), x, f16);
      if (!f16) tile_st_chunk(KQ, r, ch, 128, pack8_f16(x));
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] *= gt.dec[r];
      tile_st_chunk(KD, r, ch, 64, pack8_f16(x));
      if (!f16) {
        unpack8_bf16(tile_ld_chunk(KQ, 64 + r, ch, 128), x);
        tile_st_chunk(KQ, 64 + r, ch, 128, pack8_f16(x));
      }
    }
    mbar_wait_warp(full_v, ph, ctl, 207);
    prep_to_f16(Vt, V * 128, tid);
    sync_for_issue();
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, tmem, Tile{smem_u32(KQ), 128, false}, Tile{smem_u32(KQ), 128, false}, 64, KW, 0u);
      issue_product_led(leader, tmem + 64, Tile{smem_u32(KD), 64, true}, Tile{smem_u32(Vt), 64, true}, V, 64, 0u);
      umma_commit_led(leader, mma);
      if (tid == 0 && !p.lean) {
        bulk_s2g(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, Vt, V * 128);      // (u is v)
        bulk_commit();
      }
    } else if (warp == 1 && more) {
      const ChunkAt nx = where[ph ^ 1u];
      prep_fetch_gates(p, nx.b, nx.c, nx.h, lane, gates + (ph ^ 1u));
    } else if (warp == 2 && lane == 0 && more) {
      prep_prefetch<V, KW>(&mk, &mq, &mv, where[ph ^ 1u]);
    }
    __syncwarp();
    wait_products(mma, pm, ctl, 208);
    if (NORM) {                                      // the normalised rows have left
      if (tid == kPrepThreads - 1) bulk_wait_read();
      __syncthreads();
    }
    if (tid == 0 && more) prep_load_kq<KW>(KQ, &mk, &mq, full_kq, where[ph ^ 1u]);
    if (!p.lean) {
      if (tid == 0) bulk_wait_read();
      __syncthreads();
    }
    if (quad >= 2) {
      const bool live = (half == 0) || ((warp & 1) != 0);
      float d[32];
      if (live) {
        tmem_ld32(tmem + lane_base + half * 32, d);
        tmem_ld_wait();
      }
      prep_row_a(A, gt.G, d, tq - 64, half, live, p.scale);
    }
#pragma unroll
    for (int jj = 0; jj < V / 64; ++jj) {
      const int cb = half * (V / 2) + jj * 32;
      float d[32];
      tmem_ld32(tmem + 64 + lane_base + cb, d);
      tmem_ld_wait();
      if (tq < KW)
#pragma unroll
        for (int i = 0; i < 4; ++i) tile_st_chunk(KD, tq, cb / 8 + i, KW, pack8_f16(d + 8 * i));
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      store_image<V, KW>(p.saved + p.lay.r + static_cast<size_t>(a.z) * p.lay.sz_r, KD);
      bulk_s2g(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, A, 8192);
      bulk_commit();
      bulk_wait_read();
      if (more) prep_load_v<V>(Vt, &mv, full_v, where[ph ^ 1u]);
    }
    if (warp == 1 && more) prep_gates(p, where[ph ^ 1u].z, lane, gates + (ph ^ 1u));
    __syncthreads();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, S::kCols);
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
// d_v = 128 without the delta term: 78 against 86).  With one stage a chunk's loads start when the chunk before has left;
// they are prefetched to L2 and its gates fetched ahead (d_v = 128 without the delta term, 4096 chunks: 76 -> 71.6).
// ---------------------------------------------------------------------------------------------
constexpr int kOutThreads = 256;

template <int V, bool CW, int KW = kK>
struct OutSmem {
  static constexpr int oA = KW > V ? KW * 256 : V * 256;      // behind [w; qg], and o: A (its 128-row view starts 64 rows early)
  static constexpr int oH = oA + 8192;               // state image
  static constexpr int oU = oH + V * KW * 2;         // u, then v_new
  static constexpr int kStage = oU + V * 128, kStages = V == 64 || !CW ? 1 : 2, kCtas = V == 64 ? (KW == 64 ? 4 : 3) : CW ? 1 : 2;
  static constexpr int kBytes = kStages * kStage + 2 * 256 + static_cast<int>(sizeof(CtaShared)) + 1024;
};

// KW: 64 only without the delta term and with one decay or none, as in prepare_nodelta_kernel.  64 registers at d_v = 64, where the
// memory holds three CTAs per SM: with more of them the next call's first kernel overlaps less (8 pairs x 16 chunks, forward 24.3
// us, now 21.3).
template <int V, bool DELTA, bool CW, int KW>
__global__ void __launch_bounds__(kOutThreads, V == 64 ? 4 : OutSmem<V, CW, KW>::kCtas)
output_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mv,
              const __grid_constant__ CUtensorMap mo) {
  using S = OutSmem<V, CW, KW>;
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
    mbar_expect_tx(&full[s], KW * 128u + (DELTA ? 16384u : 0u) + V * 128u + 8192u + V * KW * 2u);
    for (int i = 0; i < KW / 64; ++i) {
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
    load_image<V, KW>(sm + s * S::kStage + S::oH, p.saved + p.lay.hc + static_cast<size_t>(a.z + a.bh) * p.lay.sz_hc, &full[s]);
  };
  auto fetch_gates = [&](const At& a, float* o) {
    if (p.gate == LETHE_GATE_SCALAR) warp_copy_gates(p, p.g, a.b, a.c, a.h, lane, o);
  };
  auto prefetch = [&](const At& a) {                 // what load and load_h will want, to L2
    for (int i = 0; i < KW / 64; ++i)
      if (!CW) tma_prefetch_4d(&mq, i * 64, a.h, a.c * kC, a.b);
    if (CW) bulk_prefetch(p.saved + p.lay.qg + static_cast<size_t>(a.z) * 16384, 16384);
    if (DELTA) bulk_prefetch(p.saved + p.lay.w + static_cast<size_t>(a.z) * p.lay.sz_w, 16384);
    bulk_prefetch(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta + 8192, 8192);
    if (DELTA) bulk_prefetch(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, V * 128);
    else for (int i = 0; i < V / 64; ++i) tma_prefetch_4d(&mv, i * 64, a.h, a.c * kC, a.b);
    prefetch_image<V, KW>(p.saved + p.lay.hc + static_cast<size_t>(a.z + a.bh) * p.lay.sz_hc);
  };

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
  if (!CW && warp == 1) {
    fetch_gates(at(n0), sgs);
    warp_scaled_gammas(p, lane, sgs);
  }
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
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    if (!CW && warp == 1 && more) fetch_gates(at(n + gridDim.x), sgs + (g2 ^ 1) * 64);
    mbar_wait_warp(&full[s], static_cast<uint32_t>((it / S::kStages) & 1), ctl, 211);
    if (!CW) {
      const float* sg = sgs + g2 * 64;
      constexpr int kN = KW * 8 / kOutThreads;
      uint4 c[kN];
      float f[kN];
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        const int idx = tid + u * kOutThreads, r = idx / (KW / 8);
        c[u] = tile_ld_chunk(WQ, 64 + r, idx % (KW / 8), 128);
        f[u] = sg[r];
      }
#pragma unroll
      for (int u = 0; u < kN; ++u) {
        const int idx = tid + u * kOutThreads, r = idx / (KW / 8);
        float x[8];
        unpack8_in(c[u], x, p.qk16);
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] *= f[u];
        tile_st_chunk(WQ, 64 + r, idx % (KW / 8), 128, pack8_f16(x));
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
      issue_product_led(leader, tmem, Tile{smem_u32(WQ), 128, false}, Tile{smem_u32(HT), KW, true}, V, KW, 0u);
      if (!DELTA) issue_product_led(leader, tmem, Tile{smem_u32(At_) - 8192, 64, false}, Tile{smem_u32(VN), 64, true}, V, 64, 1u);
      umma_commit_led(leader, DELTA ? m1 : m2);
      if (S::kStages == 2 && tid == 0 && it > 0 && n + static_cast<int>(gridDim.x) < nchunks) {      // the other stage's results have left it
        bulk_wait_read();
        const At nx = at(n + gridDim.x);
        load(nx, s ^ 1);
        load_h(nx, s ^ 1);
      }
    } else if (S::kStages == 1 && warp == 2 && lane == 0 && more) {
      prefetch(at(n + gridDim.x));
    }
    __syncwarp();
    if (!CW && warp == 1 && more) warp_scaled_gammas(p, lane, sgs + (g2 ^ 1) * 64);
    if (DELTA) {
      // A store to a swizzled tile keeps every later shared-memory load behind it, whatever the two addresses: loads come first, here
      // while the products run.
      uint4 un[V / 16];                              // this thread's pieces of u
      if (quad < 2)
#pragma unroll
        for (int i = 0; i < V / 16; ++i) un[i] = tile_ld_chunk(VN, quad * 32 + lane, half * (V / 16) + i, 64);
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
            unpack8_f16(un[4 * jj + i], u8);
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
      if (DELTA ? p.lean < 2 : !p.lean) bulk_s2g(p.saved + p.lay.vn + static_cast<size_t>(a.z) * p.lay.sz_vn, VN, V * 128);
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
template <typename Kern, typename... Maps>
static int launch_persistent(Kern kern, SmemAttr& attr, int smem, int ctas, cudaStream_t st, bool early, const Problem& p, const Maps&... maps) {
  if (attr.set(kern, smem)) return kErrLaunch;
  const int sms = sm_count(), n = p.nbh * p.cn;
  if (sms <= 0) return kErrDevice;
  const int grid = n < ctas * sms ? n : ctas * sms;
  if (!early) kern<<<grid, 256, smem, st>>>(p, maps...);
  else if (launch_dependent(kern, dim3(grid), dim3(256), smem, st, p, maps...) != cudaSuccess) return kErrLaunch;
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
template <int V>
static int launch_prepare_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const NormMaps& mn, cudaStream_t st) {
  static SmemAttr attr[6];
  // Not early for a later part of the sequences of at most two rounds: its CTAs would take the SMs that the scan of the first
  // part starts on.  Captured step, us, plain / early, by chunks of the later part: 224 (d_v = 64) 107.0 / 108.2, 224 (d_v = 128)
  // 143 / 140, 828 281 / 284, 896 328 / 336, 2048 584 / 573.  So the line could lie between 900 and 2000 as well; below it the
  // two differ by less than two captures of the same step do (2 %).
  const int sms = sm_count();
  const bool early = p.c0 == 0 || p.nbh * p.cn > 4 * sms;
  const bool norm = p.l2_eps > 0.f;
  auto delta = [&](auto kern, SmemAttr& at) { return launch_persistent(kern, at, PrepSmem<V>::kBytes, 2, st, early, p, mq, mk, mv, mn); };
  auto nodelta = [&](auto kern, SmemAttr& at, int smem, int ctas) { return launch_persistent(kern, at, smem, ctas, st, early, p, mq, mk, mv, mn); };
  if (p.delta) return norm ? delta(prepare_kernel<V, true>, attr[0]) : delta(prepare_kernel<V, false>, attr[1]);
  using S64 = PrepNdSmem<V, 64>;
  using S128 = PrepNdSmem<V, kK>;
  if (p.Kw == 64)
    return norm ? nodelta(prepare_nodelta_kernel<V, 64, true>, attr[2], S64::kBytes, S64::kCtas)
                : nodelta(prepare_nodelta_kernel<V, 64, false>, attr[3], S64::kBytes, S64::kCtas);
  return norm ? nodelta(prepare_nodelta_kernel<V, kK, true>, attr[4], S128::kBytes, S128::kCtas)
              : nodelta(prepare_nodelta_kernel<V, kK, false>, attr[5], S128::kBytes, S128::kCtas);
}
template <int V, bool DELTA, bool CW, int KW = kK>
static int launch_output_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  static SmemAttr attr;
  // A part of the sequences (a captured step that overlaps parts): early CTAs would wait in room that a scan or a chunk kernel
  // of another part needs.  Captured step, us, plain / early, scalar gate, d_v = 64: 256 chunks 83 / 89, 512 107 / 111, 2048
  // 335 / 341, 4096 572 / 586; channel-wise: 512 150 / 157 (d_v = 64) and 190 / 191 (128), 8192 2074 / 2057 (early is the better
  // one there).  Without the delta term the kernels are short and the gaps count: 512 59 / 57, 4096 553 / 541 and 727 / 695.
  const bool early = !DELTA || p.cn == p.NT;
  return launch_persistent(output_kernel<V, DELTA, CW, KW>, attr, OutSmem<V, CW, KW>::kBytes, OutSmem<V, CW, KW>::kCtas, st, early, p, mq, mv, mo);
}

int launch_prepare(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const NormMaps& mn,
                   cudaStream_t st) {
  return p.V == 64 ? launch_prepare_t<64>(p, mq, mk, mv, mn, st) : launch_prepare_t<128>(p, mq, mk, mv, mn, st);
}
template <bool CW>
static int launch_output_cw(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  if (p.V == 64) return p.delta ? launch_output_t<64, true, CW>(p, mq, mv, mo, st) : launch_output_t<64, false, CW>(p, mq, mv, mo, st);
  return p.delta ? launch_output_t<128, true, CW>(p, mq, mv, mo, st) : launch_output_t<128, false, CW>(p, mq, mv, mo, st);
}
int launch_output(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mv, const CUtensorMap& mo, cudaStream_t st) {
  if (p.Kw == 64) return p.V == 64 ? launch_output_t<64, false, false, 64>(p, mq, mv, mo, st) : launch_output_t<128, false, false, 64>(p, mq, mv, mo, st);
  return p.gate == LETHE_GATE_CHANNEL ? launch_output_cw<true>(p, mq, mv, mo, st) : launch_output_cw<false>(p, mq, mv, mo, st);
}

}  // namespace lg
