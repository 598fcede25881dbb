// Scalar gate (and none): the chunk-parallel backward after the adjoint state scan, Stage B and the WY / triangular-inverse
// VJP in one kernel.  With T = (I + strict_lower(M))^-1, A the masked attention, ratio(i, s) = exp(G_i - G_s), de_i =
// exp(G_last - G_i), gamma_i = exp(G_i):
//
//   dv2 = de (k dh) + A^T do              dA = tril(do v_new^T),  DS = scale ratio dA
//   dq  = scale gamma (do h^T) + DS k     dw = -dv2 h^T
//   dbv = T^T dv2,  dv = beta dbv         dbgk = T^T dw,  p_i = <dbgk_i, k_i>
//   dM  = strict_lower(-(dbv u^T + dbgk w^T)),   dkk = beta_i ratio dM       (u, w: the forward's WY factors)
//   dk  = de (v_new dh^T) + DS^T q + (dkk + dkk^T) k + beta gamma dbgk
//   dbeta = <dbv, v> + gamma p + sum_s dM ratio KK
//   dg = reverse cumulative sum of dG, dG_i = <scale gamma (do h^T), q> + rowsum(dA A) - colsum(dA A) - de_i <v_new, k dh>
//        + rowsum(dkk KK) - colsum(dkk KK) + beta p gamma,   and at the chunk's last row  exp(G_last) <dh, h> + sum_i dde_i
//
// The gate gradient is a reverse cumulative sum in which large terms cancel (row sums against column sums, every -dde_i
// against the + sum dde of the last row); each such pair is formed from the same fp32 numbers: colsum(dA A)_s =
// <v_new_s, (A^T do)_s>, sum_d dde = <v_new, de (k dh)>, and both sums of dkk KK come from the same products.
// Reference: closed Stage B gdn2_assemble.py:521-585 (scalar form), K#2 gdn2_assemble.py:102-147.
//
// Layout.  What has a key-channel axis on one side and tokens on the other is computed transposed, [128 channels in the
// lanes][64 tokens in the columns], so that all rows of the M = 128 products count; what is [token][value channel] or
// [token][token] keeps tokens in the lanes (64 of 128; for dv2 in lanes 64-127, through views that start 64 rows early).
// Decays and gates are applied in fp32 in the epilogues; no scaled copy of k, q or v is ever an operand.
//
// dM.  The VJP of the inverse is -T^T dT T^T with dT = dv2 (beta v)^T + dw (beta gamma k)^T; since T^T dv2 = dbv, T^T dw = dbgk,
// T (beta v) = u and T (beta gamma k) = w, that is -(dbv u^T + dbgk w^T): one product behind two that are wanted anyway, instead of
// dT, X = dT T^T and -T^T X in a row.
// The fp16 records u and w are also what the forward makes v_new = u - w h of.  The rounding e_u, e_w of a row of theirs is one
// vector for a whole column of dM and adds up in dg, more so the more the keys resemble one another.  But what it leaves in
// rowsum(dkk KK) - colsum(dkk KK) is <dv2, e_u> + <dw, e_w> (less <dbv, (I + M) e_u> and the same of w), and in Stage B's -<v_new, dv2>
// the negative of that: with the same records in both places it cancels.  2-norm error of dg in 1e-4, with dM from dT (from
// dbv v^T and dbgk k^T: the same) / as here, for independent keys 4.3 / 4.25, behind a SiLU 5.8 / 5.3, behind a ReLU 12.6 / 10.0, around a
// common direction 8.3 / 7.0; channel-wise gate 5.4 / 5.35, 5.6 / 5.5, 6.65 / 6.3, 8.2 / 8.2.  dbeta: 3.19 / 3.20, 3.8 / 3.8, 5.9 / 5.7, 7.1 /
// 6.65, and at decays near zero around a common direction 9.2 / 9.5.  By itself, without v_new beside it, this form has up to
// twice the error of the other in dg.
//
// Two CTAs share an SM at d_v = 64 (256 tensor-memory columns, 112 KB): five dependent product groups per chunk are a chain
// of latencies that one CTA cannot fill.  CTAs are persistent and fetch the next chunk's tiles as theirs fall free, which is late
// for most of them: all are prefetched to L2 under the first products, and copies are issued by threads that issue no products.
// us, with six groups and without the prefetch, and now: d_v = 64, 512 chunks 44 -> 40, 4096 230 -> 226; d_v = 128, 512 chunks 62
// -> 54; without the delta term d_v = 128, 4096 chunks 265 -> 191, d_v = 64, 1692 chunks 75 -> 64, later 57 -> 55.5 (loads
// ahead of the stores to swizzled tiles), with 64 key channels 45.
#include "gdn_cw.cuh"
#include "host_util.h"

namespace lg {


// What runs in a launch; a call cut into its two halves (kernel_mask 4, then 8) gives the bits of the uncut one.
enum ScMode {
  kScAll,        // the backward with the delta term
  kScNoDelta,    // without it: no WY half
  kScStageB,     // up to dq and dw; leaves dv2, dw, v_new dh^T (in DKB), the gate gradient so far (in DGB), DS (in RB, which
                 // nothing reads after the adjoint scan)
  kScWy          // the rest, from those records
};

struct ScBars {
  uint64_t in0, in1, inU, m1, m2, m3, m4, m5;
  uint32_t tmem_slot;
  int abort_flag;
};

struct ScGates { float G[64], beta[64], de[64], gam[64]; };      // cumulative log decay, beta, de, gamma

// KW: 64 only in kScNoDelta, as in prepare_nodelta_kernel
template <int V, int KW = kK>
struct ScSmem {
  static constexpr int kVT = V * 128, kHT = V * KW * 2;
  static constexpr int oQ = 0;                      // q; then (d_v = 64) dk on its way out
  static constexpr int oK = oQ + KW * 128;             // k (directly behind q: early view)
  static constexpr int oDO = oK + KW * 128;            // do; with v_new behind it, then dq on its way out, then (d_v = 64) w
  static constexpr int oVN = oDO + kVT;             // v_new
  static constexpr int oV = oVN + kVT;              // v; then dv on its way out
  static constexpr int oT = oV + kVT;               // T; then dkk
  static constexpr int oA = oT + 8192;              // A (directly behind T: early view); then DS
  static constexpr int oH = oA + 8192;              // h; then dw, then dbgk [channel][token]
  static constexpr int oDH = oH + kHT;          // dh; then dv2, then dbv [token][V], and (d_v = 64) u behind it
  static constexpr int oOwn = oDH + kHT;        // d_v = 128 has room for tiles of their own: dk, w, u
  static constexpr bool kOwn = V == 128;
  static constexpr int oDK = kOwn ? oOwn : oQ, oW = kOwn ? oOwn + 16384 : oDO, oU = kOwn ? oOwn + 32768 : oDH + kVT;
  static constexpr int oF = kOwn ? oOwn + (KW == kK ? 49152 : 8192) : oOwn;
  // warps that reach one lane quadrant: they split the columns of every epilogue
  static constexpr int kCg = V == 64 ? 2 : 4, kThreads = 128 * kCg;
  // floats: gates of this chunk and the next; t1q [4][64], pq [4][64]; t2p, t3p, ddep, rsp, dbm, rvp [kCg][64] each;
  // csp [2][64]; red [32]
  static constexpr int kFloats = 2 * 256 + 2 * 256 + 6 * 64 * kCg + 128 + 32;
  // An A operand of 64 rows is read as 128: 16 KB from the start of its tile, dbv the last of them.
  static constexpr int kUsed = oF + kFloats * 4 + static_cast<int>(sizeof(ScBars) + 2 * sizeof(ChunkAt)), kRead = oDH + kVT + 8192;
  static constexpr int kBytes = (kUsed > kRead ? kUsed : kRead) + 1024;
  static constexpr uint32_t kCols = V == 64 ? 256u : 512u;
};

// N values per lane: their sums over the warp's lanes, value i to out[i]
template <int N>
__device__ __forceinline__ void warp_sums(float* v, int lane, float* out) {
#pragma unroll
  for (int u = 0; u < N / 8; ++u) {
    const float s = warp_sum8(v + 8 * u, lane);
    if ((lane & 3) == 0) out[8 * u + (lane >> 2)] = s;
  }
}

template <int V, ScMode MODE, int KW>
__global__ void __launch_bounds__(ScSmem<V, KW>::kThreads, V == 64 ? 2 : 1)
bwd_sc_kernel(const Problem p, const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
              const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mdo, const __grid_constant__ OutMaps mo) {
  using S = ScSmem<V, KW>;
  static_assert(KW == kK || MODE == kScNoDelta, "");
  constexpr bool SB = MODE != kScWy, WY = MODE == kScAll || MODE == kScWy, DELTA = MODE != kScNoDelta;
  constexpr int kCg = S::kCg, kU = 4 / kCg, kThreads = S::kThreads;
  constexpr bool CUT = MODE == kScStageB || MODE == kScWy;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  unsigned char *tQ = sm + S::oQ, *tK = sm + S::oK, *tDO = sm + S::oDO, *tVN = sm + S::oVN, *tV = sm + S::oV, *tT = sm + S::oT;
  unsigned char *tA = sm + S::oA, *tDS = tA, *tH = sm + S::oH, *tDW = tH, *tDH = sm + S::oDH, *tDV = tDH;
  unsigned char *tBV = tDH, *tBK = tH, *tW = sm + S::oW, *tU = sm + S::oU, *tKKd = tT, *oQt = tDO, *oKt = sm + S::oDK, *oVt = tV;
  ScGates* gates = reinterpret_cast<ScGates*>(sm + S::oF);
  float *t1q = reinterpret_cast<float*>(gates + 2), *pq = t1q + 256;
  float *t2p = pq + 256, *t3p = t2p + 64 * kCg, *ddep = t3p + 64 * kCg, *rsp = ddep + 64 * kCg, *dbm = rsp + 64 * kCg;
  float *rvp = dbm + 64 * kCg, *csp = rvp + 64 * kCg;
  float* red = csp + 128;
  ChunkAt* where = reinterpret_cast<ChunkAt*>(red + 32);      // this chunk and the next
  ScBars* bars = reinterpret_cast<ScBars*>(where + 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, cg = warp >> 2, d = quad * 32 + lane;
  const int c0 = cg * 16 * kU;                    // this thread's tokens / columns of every 64-column accumulator
  CtaCtl ctl{p.status, &bars->abort_flag};
  const int nchunks = p.nbh * p.cn;
  // loads of a chunk (tid 0), by when their destinations fall free in the chunk before
  constexpr uint32_t kIn0 = KW * 256u + (WY ? V * 128u : 0u) + (DELTA ? 16384u : 8192u) + (SB ? 2u * V * 128 + S::kHT : V * 128u);
  auto load_do = [&](const ChunkAt& a) {               // do, and without the delta term v as v_new
    mbar_expect_tx(&bars->in0, kIn0);
    for (int t = 0; t < V / 64; ++t) {
      if (SB) tma_load_4d(tDO + t * 8192, &mdo, &bars->in0, t * 64, a.h, a.c * kC, a.b);
      if (!DELTA) tma_load_4d(tVN + t * 8192, &mv, &bars->in0, t * 64, a.h, a.c * kC, a.b);
    }
  };
  auto load_v = [&](const ChunkAt& a) {
    if (WY) for (int t = 0; t < V / 64; ++t) tma_load_4d(tV + t * 8192, &mv, &bars->in0, t * 64, a.h, a.c * kC, a.b);
  };
  auto load_rec = [&](const ChunkAt& a) {              // v_new, h (dv2 where the first half of the call left it)
    if (SB && DELTA) bulk_g2s(tVN, p.saved + p.lay.vn + static_cast<size_t>(a.z) * p.lay.sz_vn, V * 128, &bars->in0);
    if (SB) load_image<V, KW>(tH, p.saved + p.lay.hc + static_cast<size_t>(a.z + a.b * p.H + a.h) * p.lay.sz_hc, &bars->in0);
    else bulk_g2s(tDV, p.scratch + p.lay.dv2 + static_cast<size_t>(a.z) * p.lay.sz_dv2, V * 128, &bars->in0);
  };
  auto load_dh = [&](const ChunkAt& a) {
    mbar_expect_tx(&bars->in1, static_cast<uint32_t>(S::kHT));
    load_image<V, KW>(tDH, p.scratch + p.lay.dh + static_cast<size_t>(a.z) * p.lay.sz_dh, &bars->in1);
  };
  auto load_b = [&](const ChunkAt& a) {                // [T; A], k
    const unsigned char* ta = p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta;
    if (DELTA) bulk_g2s(tT, ta, 16384, &bars->in0);
    else bulk_g2s(tA, ta + 8192, 8192, &bars->in0);
    for (int t = 0; t < KW / 64; ++t) tma_load_4d(tK + t * 8192, &mk, &bars->in0, t * 64, a.h, a.c * kC, a.b);
  };
  auto load_w = [&](const ChunkAt& a) {                // the forward's WY factors
    mbar_expect_tx(&bars->inU, 16384u);
    bulk_g2s(tW, p.saved + p.lay.w + static_cast<size_t>(a.z) * 16384, 16384, &bars->inU);
  };
  auto load_u = [&](const ChunkAt& a) {
    mbar_expect_tx(&bars->inU, V * 128u);
    bulk_g2s(tU, p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, V * 128, &bars->inU);
  };
  // what a chunk will load, to L2: its tiles are free late (before this its loads were waited for, 2 to 5 k cycles per chunk)
  auto prefetch = [&](const ChunkAt& a) {
    for (int t = 0; t < KW / 64; ++t) {
      tma_prefetch_4d(&mq, t * 64, a.h, a.c * kC, a.b);
      tma_prefetch_4d(&mk, t * 64, a.h, a.c * kC, a.b);
    }
    for (int t = 0; t < V / 64; ++t) {
      tma_prefetch_4d(&mdo, t * 64, a.h, a.c * kC, a.b);
      tma_prefetch_4d(&mv, t * 64, a.h, a.c * kC, a.b);
    }
    if (DELTA) bulk_prefetch(p.saved + p.lay.vn + static_cast<size_t>(a.z) * p.lay.sz_vn, V * 128);
    prefetch_image<V, KW>(p.saved + p.lay.hc + static_cast<size_t>(a.z + a.b * p.H + a.h) * p.lay.sz_hc);
    prefetch_image<V, KW>(p.scratch + p.lay.dh + static_cast<size_t>(a.z) * p.lay.sz_dh);
    if (WY) {
      bulk_prefetch(p.saved + p.lay.w + static_cast<size_t>(a.z) * 16384, 16384);
      bulk_prefetch(p.saved + p.lay.u + static_cast<size_t>(a.z) * p.lay.sz_u, V * 128);
    }
    bulk_prefetch(p.saved + p.lay.ta + static_cast<size_t>(a.z) * p.lay.sz_ta, 16384);
  };
  auto load_q = [&](const ChunkAt& a) {
    for (int t = 0; t < KW / 64; ++t) tma_load_4d(tQ + t * 8192, &mq, &bars->in0, t * 64, a.h, a.c * kC, a.b);
  };

  if (tid == 0) {
    bars->abort_flag = 0;
    mbar_init(&bars->in0, 1); mbar_init(&bars->in1, 1); mbar_init(&bars->m1, 2); mbar_init(&bars->m2, 2);
    mbar_init(&bars->m3, 1); mbar_init(&bars->m4, 1); mbar_init(&bars->m5, 1); mbar_init(&bars->inU, 2);
    fence_mbar_init();
    fence_proxy_async();
    // Older than whatever kernel of the path comes just before this one: the caller's tensors and [T; A].  v_new (the output
    // kernel) and h (the forward scan) only where this call has put the adjoint scan in between; with kernels picked one by one
    // any of the three may be the last.  (Late everywhere: SSD forward and backward 175.1 us instead of 172.3 at 1692 chunks, 557.8
    // instead of 555.3 at 4096; with the delta term no difference.)
    if (SB) {
      const ChunkAt a = chunk_at(p, blockIdx.x);
      load_do(a);
      load_v(a);
      load_b(a);
      load_q(a);
      if (p.after_scan) load_rec(a);
    }
  }
  if (warp == 0) {
    tmem_alloc(&bars->tmem_slot, S::kCols);
    tmem_relinquish();
  }
  // gates of a chunk, by one warp, two neighbouring tokens per lane: fetched a chunk ahead, then summed
  auto fetch_gates = [&](const ChunkAt& a, ScGates* o) {
    if (p.gate == LETHE_GATE_SCALAR) warp_copy_gates(p, p.g, a.b, a.c, a.h, lane, o->G);
    if (WY) warp_copy_gates(p, p.beta, a.b, a.c, a.h, lane, o->beta);
  };
  auto sum_gates = [&](ScGates* o) {
    async_copy_wait();
    float g[2] = {0.f, 0.f}, be[2] = {1.f, 1.f};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (p.gate == LETHE_GATE_SCALAR) g[e] = o->G[2 * lane + e];
      if (WY) be[e] = o->beta[2 * lane + e];
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
    *reinterpret_cast<float2*>(o->de + 2 * lane) = make_float2(__expf(last - G0), __expf(last - G1));
    *reinterpret_cast<float2*>(o->gam + 2 * lane) = make_float2(__expf(G0), __expf(G1));
  };

  ChunkAt a = chunk_at(p, blockIdx.x);
  if (warp == 2) {
    fetch_gates(a, gates);
    sum_gates(gates);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_slot, lane_base = static_cast<uint32_t>(quad * 32) << 16;
  // columns; an accumulator that shares columns with an earlier one is issued after that one has been read
  const uint32_t cD = tmem, cAo = tmem + V, cDA = tmem + 2 * V, cDK = tmem + 2 * V + 64;      // k dh, A^T do, dA, (v_new dh^T)^T
  const uint32_t cDQ = tmem, cDWt = tmem + 64, cQI = tmem + 128;                               // (do h^T)^T, (dv2 h^T)^T, (DS k)^T
  const uint32_t cKK = tmem, cBK = tmem + 64, cBV = V == 64 ? tmem + 128 : tmem + 320 + 64;    // k k^T, (T^T dw)^T, T^T dv2
  const uint32_t cX = tmem + 128, cAcc = tmem;                                                 // dM, dk sums
  griddep_wait();
  griddep_launch();
  if (tid == 0) {
    if (!SB) {
      load_do(a);
      load_v(a);
      load_b(a);
      load_q(a);
    }
    if (!SB || !p.after_scan) load_rec(a);
    if (SB) load_dh(a);
  }

  uint32_t ph = 0;
  for (int n = blockIdx.x; n < nchunks; n += gridDim.x, ph ^= 1u) {
    const bool more = n + static_cast<int>(gridDim.x) < nchunks;
    if (tid == kThreads - 1 && more) where[ph ^ 1u] = chunk_at(p, n + gridDim.x);      // (read behind the next barrier)
    const int rows = p.rows_of(a.c);
    const size_t tok0 = (static_cast<size_t>(a.b) * p.L + a.c * kC) * p.H + a.h;
    unsigned char* dv2_g = p.scratch + p.lay.dv2 + static_cast<size_t>(a.z) * p.lay.sz_dv2;
    unsigned char* dw_g = p.scratch + p.lay.dw + static_cast<size_t>(a.z) * p.lay.sz_dw;
    unsigned char* rb_g = p.scratch + p.lay.rb + static_cast<size_t>(a.z) * p.lay.sz_rb;
    float* dkb_g = reinterpret_cast<float*>(p.scratch + p.lay.dkb + static_cast<size_t>(a.z) * p.lay.sz_dkb);
    float* dgb_g = reinterpret_cast<float*>(p.scratch + p.lay.dgb + static_cast<size_t>(a.z) * p.lay.sz_dgb);
    const bool keep = CUT || !p.lean;

    const ScGates& gt = gates[ph];
    if (tid == 0 && n != static_cast<int>(blockIdx.x)) {
      bulk_wait_read();                             // dk of the chunk before has left its tile
      if (!S::kOwn) load_q(a);
    }
    if (WY && tid == 0 && (S::kOwn || !SB)) {       // w and u where their tiles are free already
      load_w(a);
      load_u(a);
    }

    // ---- operands to fp16 in place
    mbar_wait_warp(&bars->in0, ph, ctl, 411);
    if (!p.qk16) {
      for (int idx = tid; idx < 2 * KW * 8; idx += kThreads) {       // q and k lie behind each other
        uint4* c = reinterpret_cast<uint4*>(tQ + idx * 16);
        float x[8];
        unpack8_bf16(*c, x);
        *c = pack8_f16(x);
      }
    }
    if (SB) {
      for (int idx = tid; idx < (DELTA ? 1 : 2) * 64 * (V / 8); idx += kThreads) {      // do (and, without delta, v behind it)
        uint4* c = reinterpret_cast<uint4*>(tDO + idx * 16);
        float x[8];
        unpack8_bf16(*c, x);
        *c = pack8_f16(x);
      }
    }
    if (!SB) {                                      // the first half of the call left DS and dw
      for (int idx = tid; idx < 512; idx += kThreads) reinterpret_cast<uint4*>(tDS)[idx] = reinterpret_cast<const uint4*>(rb_g)[idx];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
          x[i] = __half2float(*reinterpret_cast<const __half*>(dw_g + sw128_off(c0 + 16 * u + i, d, 64)));
        write_column(tDW, kU * cg + u, d, x);
      }
    }
    sync_for_issue();
    const ChunkAt& nx = where[ph ^ 1u];
    if (warp == 2 && more) fetch_gates(nx, gates + (ph ^ 1u));

    if (SB) {
      mbar_wait_warp(&bars->in1, ph, ctl, 415);
      // ---- group 1 (two warps issue): k dh (lanes 64-127), (v_new dh^T)^T | A^T do (lanes 64-127), dA
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cD, Tile{smem_u32(tK) - 8192, 64, false}, Tile{smem_u32(tDH), KW, true}, V, KW, 0u);
        issue_product_led(leader, cDK, Tile{smem_u32(tDH), KW, false}, Tile{smem_u32(tVN), 64, false}, 64, V, 0u);
        umma_commit_led(leader, &bars->m1);
      } else if (warp == 4) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cAo, Tile{smem_u32(tA) - 8192, 64, true}, Tile{smem_u32(tDO), 64, true}, V, 64, 0u);
        issue_product_led(leader, cDA, Tile{smem_u32(tDO), 64, false}, Tile{smem_u32(tVN), 64, false}, 64, V, 0u);
        umma_commit_led(leader, &bars->m1);
      } else if (warp == 1 && lane == 0 && more) {
        prefetch(nx);
      }
      __syncwarp();
      // in their shadow: <dh, h>, element by element on two images of one layout
      float dhh = 0.f;
      for (int idx = tid; idx < KW * V / 8; idx += kThreads) {
        float x[8], y[8];
        unpack8_f16(*reinterpret_cast<const uint4*>(tDH + idx * 16), x);
        unpack8_f16(*reinterpret_cast<const uint4*>(tH + idx * 16), y);
#pragma unroll
        for (int i = 0; i < 8; ++i) dhh += x[i] * y[i];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) dhh += __shfl_xor_sync(0xffffffffu, dhh, o);
      if (lane == 0) red[16 + warp] = dhh;
      __syncthreads();                              // every thread has read dh
      mbar_wait_warp(&bars->m1, ph, ctl, 412);
      tc_fence_after();
      if (quad >= 2) {                              // dv2
        const int r = d - 64;
        const float de = gt.de[r];
        float t3 = 0.f, dde = 0.f;
        constexpr int kNv = V / (8 * kCg);          // (all loads ahead of the first store: see output_kernel)
        uint4 vc[kNv];
#pragma unroll
        for (int i = 0; i < kNv; ++i) vc[i] = tile_ld_chunk(tVN, r, cg * kNv + i, 64);
#pragma unroll
        for (int jj = 0; jj < V / (16 * kCg); ++jj) {
          const int cb = cg * (V / kCg) + jj * 16;
          float x[16], y[16];
          tmem_ld16(cAo + lane_base + cb, x);
          tmem_ld16(cD + lane_base + cb, y);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            float vn[8];
            unpack8_f16(vc[2 * jj + q], vn);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float kd_dh = de * y[8 * q + e];
              t3 += vn[e] * x[8 * q + e];
              dde += vn[e] * kd_dh;
              x[8 * q + e] += kd_dh;
            }
            if (DELTA) tile_st_chunk(tDV, r, cb / 8 + q, 64, pack8_f16(x + 8 * q));
            else tile_st_chunk(oVt, r, cb / 8 + q, 64, pack8_bf16(x + 8 * q));
          }
        }
        t3p[cg * 64 + r] = t3 + dde;
        ddep[cg * 64 + r] = dde;
      } else {                                      // dA -> DS, where A was
        const int r = d;
        const float Gr = gt.G[r];
        float t2 = 0.f;
        uint4 ac[2 * kU];                           // A[r, s] (holds scale * ratio already)
#pragma unroll
        for (int i = 0; i < 2 * kU; ++i) ac[i] = tile_ld_chunk(tA, r, c0 / 8 + i, 64);
        float e[16 * kU];
#pragma unroll
        for (int i = 0; i < 16 * kU; i += 8) ld8(gt.G + c0 + i, e + i);
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          float x[16];
          tmem_ld16(cDA + lane_base + c0 + 16 * u, x);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int s8 = c0 / 8 + 2 * u + q;
            float av[8], y[8];
            unpack8_f16(ac[2 * u + q], av);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int s = s8 * 8 + i;
              const float da = (s <= r) ? x[8 * q + i] : 0.f;
              t2 += da * av[i];
              y[i] = (s <= r) ? p.scale * __expf(Gr - e[16 * u + 8 * q + i]) * da : 0.f;
            }
            tile_st_chunk(tDS, r, s8, 64, pack8_f16(y));
          }
        }
        t2p[cg * 64 + r] = t2;
      }
      sync_for_issue();
      if (WY && !S::kOwn && tid == 32) load_u(a);   // dh is dead

      // ---- group 2: (do h^T)^T, (DS k)^T | (dv2 h^T)^T
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cDQ, Tile{smem_u32(tH), KW, false}, Tile{smem_u32(tDO), 64, false}, 64, V, 0u);
        umma_commit_led(leader, &bars->m2);
        if (tid == 0) {
          if (!DELTA) for (int t = 0; t < V / 64; ++t) tma_store_4d(&mo.dv, oVt + t * 8192, t * 64, a.h, a.c * kC, a.b);
          else if (keep) bulk_s2g(dv2_g, tDV, V * 128);
          if (CUT) bulk_s2g(rb_g, tDS, 8192);
          bulk_commit();
        }
      } else if (warp == 4) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cQI, Tile{smem_u32(tK), 64, true}, Tile{smem_u32(tDS), 64, false}, 64, 64, 0u);
        if (DELTA) issue_product_led(leader, cDWt, Tile{smem_u32(tH), 128, false}, Tile{smem_u32(tDV), 64, false}, 64, V, 0u);
        umma_commit_led(leader, &bars->m2);
      }
      __syncwarp();
      mbar_wait_warp(&bars->m2, ph, ctl, 413);
      tc_fence_after();
      float t1[16 * kU];
      const f2 scale2 = pack2(p.scale, p.scale);
      if (KW == kK || quad < 2) {                   // (with 64 channels the other lanes hold none)
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          uint32_t qp[8];
          float x[16], y[16];
          read_column(tQ, kU * cg + u, d, 1, qp);
          tmem_ld16(cDQ + lane_base + c0 + 16 * u, x);
          tmem_ld16(cQI + lane_base + c0 + 16 * u, y);
          f2 g[8];
#pragma unroll
          for (int j = 0; j < 8; j += 2) ld_pairs(gt.gam + c0 + 16 * u + 2 * j, g + j);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {               // two tokens
            const int r = c0 + 16 * u + 2 * j;
            const f2 dq = mul2(mul2(scale2, g[j]), pack2(x[2 * j], x[2 * j + 1]));
            unpack2(mul2(dq, pair_of(qp[j])), t1[16 * u + 2 * j], t1[16 * u + 2 * j + 1]);
            stage16_two(oQt, r, d, add2(dq, pack2(y[2 * j], y[2 * j + 1])), p.qk16);
          }
          if (DELTA) {
            tmem_ld16(cDWt + lane_base + c0 + 16 * u, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = -x[i];
            if (WY) write_column(tDW, kU * cg + u, d, x);
            if (keep)
#pragma unroll
              for (int i = 0; i < 16; ++i) store_f16_sat(dw_g + sw128_off(c0 + 16 * u + i, d, 64), x[i]);
          }
          if (MODE == kScStageB) {
            tmem_ld16(cDK + lane_base + c0 + 16 * u, x);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) dkb_g[static_cast<size_t>(c0 + 16 * u + i) * kK + d] = x[i];
          }
        }
        warp_sums<16 * kU>(t1, lane, t1q + quad * 64 + c0);
      }
      if (tid == 0 && keep) bulk_wait_read();       // dv2 has left its tile, which becomes dbv
      sync_for_issue();
      if (tid == 96) {                              // (a thread that issues no products: it waits)
        for (int t = 0; t < p.Kr / 64; ++t) tma_store_4d(&mo.dq, oQt + t * 8192, t * 64, a.h, a.c * kC, a.b);
        bulk_commit();
        bulk_wait_read();
        if (WY && !S::kOwn) load_w(a);
      }
      __syncwarp();
    }
    // gate gradient of Stage B (token tid), before the cumulative sum
    float dG = 0.f;
    auto over_cg = [&](const float* x) {
      float s = x[tid] + x[64 + tid];
      if (kCg == 4) s += x[128 + tid] + x[192 + tid];
      return s;
    };
    auto end_term = [&]() {                         // exp(G_last) <dh, h> + sum dde, for the chunk's last row (after a barrier)
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 4 * kCg; ++w) s += red[16 + w];
      return s * gt.gam[63] + (red[12] + red[13]);
    };
    if (SB) {
      if (tid < 64) {
        float sdde = over_cg(ddep);    // sum over the chunk's rows, fixed tree
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sdde += __shfl_xor_sync(0xffffffffu, sdde, o);
        if (lane == 0) red[12 + warp] = sdde;
        dG = ((t1q[tid] + t1q[64 + tid]) + (KW == kK ? t1q[128 + tid] + t1q[192 + tid] : 0.f)) + over_cg(t2p) - over_cg(t3p);
      }
    } else if (tid < 64) {
      dG = dgb_g[tid];
    }
    if (MODE == kScStageB) {
      __syncthreads();
      if (tid < 64) dgb_g[tid] = dG + (tid == 63 ? end_term() : 0.f);
      if (warp == 2 && more) sum_gates(gates + (ph ^ 1u));
      if (tid == 0 && more) {
        bulk_wait_read();
        load_do(nx);
        load_v(nx);
        load_rec(nx);
        load_dh(nx);
        load_b(nx);
        if (S::kOwn) load_q(nx);
      }
      tc_fence_before();
      __syncthreads();
      if (more) a = nx;
      continue;
    }
    if (WY) {
      // ---- group 3: T^T dv2, (T^T dw)^T; k k^T
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cBV, Tile{smem_u32(tT), 64, true}, Tile{smem_u32(tDV), 64, true}, V, 64, 0u);
        issue_product_led(leader, cBK, Tile{smem_u32(tDW), 128, false}, Tile{smem_u32(tT), 64, true}, 64, 64, 0u);
        umma_commit_led(leader, &bars->m3);
        issue_product_led(leader, cKK, Tile{smem_u32(tK), 64, false}, Tile{smem_u32(tK), 64, false}, 64, 128, 0u);
      }
      __syncwarp();
      mbar_wait_warp(&bars->m3, ph, ctl, 421);
      tc_fence_after();
#pragma unroll
      for (int u = 0; u < kU; ++u) {                // dbgk, where dw was
        float x[16];
        tmem_ld16(cBK + lane_base + c0 + 16 * u, x);
        tmem_ld_wait();
        write_column(tBK, kU * cg + u, d, x);
      }
      // dbv (lanes 0-63) as an operand, where dv2 was; dv = beta dbv where v was, and the value part of dbeta
      float rv = 0.f;
      auto dbv_columns = [&](bool operand, bool result) {
        const int r = d;
        const float be = gt.beta[r];
        constexpr int kNv = V / (8 * kCg);
        uint4 vc[kNv];
        if (result)
#pragma unroll
          for (int i = 0; i < kNv; ++i) vc[i] = tile_ld_chunk(tV, r, cg * kNv + i, 64);
#pragma unroll
        for (int jj = 0; jj < V / (16 * kCg); ++jj) {
          const int cb = cg * (V / kCg) + jj * 16;
          float x[16];
          tmem_ld16(cBV + lane_base + cb, x);
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            if (operand) tile_st_chunk(tBV, r, cb / 8 + q, 64, pack8_f16(x + 8 * q));
            if (!result) continue;
            float vv[8];
            unpack8_bf16(vc[2 * jj + q], vv);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              rv += x[8 * q + e] * vv[e];
              x[8 * q + e] *= be;
            }
            tile_st_chunk(oVt, r, cb / 8 + q, 64, pack8_bf16(x + 8 * q));
          }
        }
        if (result) rvp[cg * 64 + r] = rv;
      };
      if (quad < 2) dbv_columns(true, V == 64);     // (d_v = 64: dM takes the columns)
      mbar_wait_warp(&bars->inU, ph, ctl, 422);
      sync_for_issue();
      // ---- group 4: dM = -(dbv u^T + dbgk w^T)
      if (warp == 0) {
        tc_fence_after();
        const uint32_t leader = elect_leader();
        issue_product_led(leader, cX, Tile{smem_u32(tBV), 64, false}, Tile{smem_u32(tU), 64, false}, 64, V, 0u, true);
        issue_product_led(leader, cX, Tile{smem_u32(tBK), 128, true}, Tile{smem_u32(tW), 64, false}, 64, 128, 1u, true);
        umma_commit_led(leader, &bars->m4);
      }
      __syncwarp();
      // in its shadow: p_i = <(T^T dw)_i, k_i>, and dv at d_v = 128
      {
        float v[16 * kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          uint32_t kp[8];
          float x[16];
          read_column(tK, kU * cg + u, d, 1, kp);
          tmem_ld16(cBK + lane_base + c0 + 16 * u, x);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) v[16 * u + i] = x[i] * half_of(kp[i >> 1], i & 1);
        }
        warp_sums<16 * kU>(v, lane, pq + quad * 64 + c0);
      }
      if (V == 128 && quad < 2) dbv_columns(false, true);
      mbar_wait_warp(&bars->m4, ph, ctl, 424);
      tc_fence_after();
      if (quad < 2) {                               // dkk = beta ratio dM, where T was; row and column sums of e = dkk KK
        const int r = d;
        const float Gr = gt.G[r], be = gt.beta[r];
        float rse = 0.f, dbe = 0.f, ev[16 * kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          float x[16], y[16];
          tmem_ld16(cX + lane_base + c0 + 16 * u, x);
          tmem_ld16(cKK + lane_base + c0 + 16 * u, y);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int sidx = c0 + 16 * u + j;
            const float m = (sidx < r) ? x[j] * __expf(Gr - gt.G[sidx]) : 0.f;      // dM * ratio, strictly lower
            dbe += m * y[j];
            x[j] = m * be;
            const float e = x[j] * y[j];
            rse += e;
            ev[16 * u + j] = e;
          }
          write_row16(tKKd, r, kU * cg + u, x);
        }
        rsp[cg * 64 + r] = rse;
        dbm[cg * 64 + r] = dbe;
        warp_sums<16 * kU>(ev, lane, csp + quad * 64 + c0);      // over this warp's 32 rows
      }
      sync_for_issue();
    }
    // ---- last group: DS^T q (+ (dkk + dkk^T) k)
    if (tid == 96) {
      if (WY) {                                     // dv, staged before the last barrier
        for (int t = 0; t < V / 64; ++t) tma_store_4d(&mo.dv, oVt + t * 8192, t * 64, a.h, a.c * kC, a.b);
        bulk_commit();
      }
      if (more) {
        load_do(nx);                                // dq has left (this thread has waited for it), w is read
        if (WY) {
          bulk_wait_read();
          load_v(nx);
        }
      }
    }
    __syncwarp();
    if (warp == 0) {
      tc_fence_after();
      const uint32_t leader = elect_leader();
      issue_product_led(leader, cAcc, Tile{smem_u32(tQ), 64, true}, Tile{smem_u32(tDS), 64, true}, 64, 64, 0u);
      if (WY) {
        issue_product_led(leader, cAcc, Tile{smem_u32(tK), 64, true}, Tile{smem_u32(tKKd), 64, false}, 64, 64, 1u);
        issue_product_led(leader, cAcc, Tile{smem_u32(tK), 64, true}, Tile{smem_u32(tKKd), 64, true}, 64, 64, 1u);
      }
      umma_commit_led(leader, &bars->m5);
      if (tid == 0 && more) {          // h / dw / dbgk, dv2 / dbv and u are read
        load_rec(nx);
        if (SB) load_dh(nx);
      }
    }
    __syncwarp();
    if (warp == 2 && more) sum_gates(gates + (ph ^ 1u));
    mbar_wait_warp(&bars->m5, ph, ctl, 425);
    tc_fence_after();
    if (tid == 0 && more) {                         // [T; A], k and q are read
      load_b(nx);
      if (S::kOwn) load_q(nx);
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (KW < kK && quad >= 2) break;
      float x[16], y[16];
      if (SB) {
        tmem_ld16(cDK + lane_base + c0 + 16 * u, y);
      } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[i] = dkb_g[static_cast<size_t>(c0 + 16 * u + i) * kK + d];
      }
      tmem_ld16(cAcc + lane_base + c0 + 16 * u, x);
      tmem_ld_wait();
      auto pair_at = [](const float* t) {
        f2 r;
        r.u = *reinterpret_cast<const unsigned long long*>(t);
        return r;
      };
      f2 acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        acc[j] = fma2(pair_at(gt.de + c0 + 16 * u + 2 * j), pack2(y[2 * j], y[2 * j + 1]), pack2(x[2 * j], x[2 * j + 1]));
      if (WY) {
        tmem_ld16(cBK + lane_base + c0 + 16 * u, y);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int r = c0 + 16 * u + 2 * j;
          acc[j] = fma2(mul2(pair_at(gt.beta + r), pair_at(gt.gam + r)), pack2(y[2 * j], y[2 * j + 1]), acc[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) stage16_two(oKt, c0 + 16 * u + 2 * j, d, acc[j], p.qk16);
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      for (int t = 0; t < p.Kr / 64; ++t) tma_store_4d(&mo.dk, oKt + t * 8192, t * 64, a.h, a.c * kC, a.b);
      bulk_commit();
    }
    if (tid < 64) {
      if (SB && tid == 63) dG += end_term();
      if (WY) {
        const float gam = gt.gam[tid];
        const float pks = (pq[tid] + pq[64 + tid]) + (pq[128 + tid] + pq[192 + tid]);
        const float db = over_cg(dbm), rvs = over_cg(rvp), rse = over_cg(rsp), cse = csp[tid] + csp[64 + tid];
        if (tid < rows) {
          const size_t o = tok0 + static_cast<size_t>(tid) * p.H;
          if (p.dbeta_w) {
            p.dbeta_w[o] = rvs;
            p.dbeta[o] = gam * pks + db;
          } else {
            p.dbeta[o] = rvs + gam * pks + db;
          }
        }
        dG = dG + rse - cse + gt.beta[tid] * pks * gam;
      }
    }
    const float acc = chunk_rev_cumsum(dG, tid, red);
    if (tid < rows && p.gate == LETHE_GATE_SCALAR) p.dg[tok0 + static_cast<size_t>(tid) * p.H] = acc;
    if (more) a = nx;
  }
  if (tid == 0 || tid == 96) bulk_wait_read();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, S::kCols);
}

// ---------------------------------------------------------------------------------------------
template <int V, ScMode MODE, int KW = kK>
static int launch_t(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                    const CUtensorMap& mdo, const OutMaps& mo, cudaStream_t st) {
  constexpr int smem = ScSmem<V, KW>::kBytes, per_sm = V == 64 ? 2 : 1;
  static_assert(per_sm * (smem + 1024) <= 228 * 1024, "CTAs per SM");
  static SmemAttr attr;
  if (attr.set(bwd_sc_kernel<V, MODE, KW>, smem)) return kErrLaunch;
  const int sms = sm_count();
  if (sms <= 0) return kErrDevice;
  const int n = p.nbh * p.cn, most = per_sm * sms;
  if (launch_dependent(bwd_sc_kernel<V, MODE, KW>, dim3(n < most ? n : most), dim3(ScSmem<V, KW>::kThreads), smem, st, p, mq, mk, mv, mdo, mo) !=
      cudaSuccess) return kErrLaunch;
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
template <ScMode MODE>
static int launch_v(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                    const CUtensorMap& mdo, const OutMaps& mo, cudaStream_t st) {
  return p.V == 64 ? launch_t<64, MODE>(p, mq, mk, mv, mdo, mo, st) : launch_t<128, MODE>(p, mq, mk, mv, mdo, mo, st);
}

// mask bit 4: Stage B, bit 8: WY VJP (delta variants only); both together are one kernel
int launch_bwd_main(const Problem& p, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                    const CUtensorMap& mdo, const OutMaps& mo, cudaStream_t st, uint32_t mask) {
  const bool sb = mask & 4u, wy = (mask & 8u) && p.delta;
  if (!p.delta && !sb) return kOk;
  if (p.Kw == 64)
    return p.V == 64 ? launch_t<64, kScNoDelta, 64>(p, mq, mk, mv, mdo, mo, st) : launch_t<128, kScNoDelta, 64>(p, mq, mk, mv, mdo, mo, st);
  if (!p.delta) return launch_v<kScNoDelta>(p, mq, mk, mv, mdo, mo, st);
  if (sb && wy) return launch_v<kScAll>(p, mq, mk, mv, mdo, mo, st);
  return sb ? launch_v<kScStageB>(p, mq, mk, mv, mdo, mo, st) : launch_v<kScWy>(p, mq, mk, mv, mdo, mo, st);
}

}  // namespace lg
