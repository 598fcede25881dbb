// The serial part of the path: the chunk-to-chunk state recurrence, forward and adjoint.
//
//   forward :  x_{c+1} = a_c * x_c - P_c   x_c + R_c      c = 0 .. NT-1     (x_0 = h0)
//   adjoint :  x_{c-1} = a_c * x_c - P_c^T x_c + Rb_c     c = NT-1 .. 0     (x_NT = dhT)
//
// a_c is the chunk's decay per key channel, P_c = kd^T w (128 x 128) and R_c / Rb_c (128 x V) come
// from the chunk-parallel kernels.  The recurrence is independent per column of x, so the grid is
// (V / columns) x (B*H): every CTA owns some columns, keeps them as fp32 in registers and does ONE product per chunk, with
// P streamed through a ring of shared-memory stages by bulk copies that run ahead of the recurrence.  The state seen by
// chunk c is written out as a shared-memory tile image for the chunk-parallel kernels.  Three kernels: 64 columns per CTA on
// tcgen05 (few CTAs, P read once or twice per pair), 8 to 32 on warp-level matrix instructions (the shorter step), and one without
// a product where there is no delta term; the rules stand at launch_scan.
// Reference: the forward recurrence gdn2_chunkwise.py:155-158 and the reverse scan K#1
// gdn2_assemble.py:71-99 of the reference project, after substituting v_new / dv2.
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

constexpr int kStages = 3;
constexpr int kMmaWarps = 2;   // warps that issue the step's products (each its own accumulator)
// 64 columns of the state per CTA on sixteen state-holding warps, 16 columns of a row per thread (four groups of four warps, thread
// d = key channel d), then one warp that streams P and two that issue products
constexpr int kVs = 16, kGr = 4, kW = kVs * kGr;

// Step barrier of the delta path: the state-holding warps arrive once the operand is written (and go
// on to work that does not depend on the product), the issuing warps wait for them.
template <int kN>
__device__ __forceinline__ void step_arrive() { asm volatile("bar.arrive 1, %0;" ::"n"(kN) : "memory"); }
template <int kN>
__device__ __forceinline__ void step_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kN) : "memory"); }

constexpr int kScanThreads = (4 * kGr + 1 + kMmaWarps) * 32;

template <bool ADJOINT>
__global__ void __launch_bounds__(kScanThreads, 1)
scan_kernel(const Problem p) {
  constexpr int kTmemCols = kMmaWarps * kW;
  constexpr int kXB = 128 * kW * 2;                  // bytes of the state operand tile
  constexpr int kStateWarps = 4 * kGr, kStepBarrier = (kStateWarps + kMmaWarps) * 32;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024_generic(smem_raw);
  unsigned char* Pst = sm;                          // kStages x 32 KB
  // x as the B operand, contracted along its rows (row k = key channel k, 64 columns): thread k stores pieces of row k
  unsigned char* XB0 = sm + kStages * 32768;        // two of them, alternating: the step before's is still being recorded
  CtaShared* cs = reinterpret_cast<CtaShared*>(XB0 + 2 * kXB);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int v0 = blockIdx.x * kW, bh = blockIdx.y + p.bh0;
  // This launch walks the chunks [c0, c0 + cn) of every pair (all NT of them in an ordinary call), forward in
  // chunk order, the adjoint in reverse.  A launch that does not start at the sequence's first (adjoint: last)
  // chunk takes its fp32 state from the carry buffer the launch before it left, and one that does not end at
  // the other end leaves its state there: a scan cut into chunk ranges is bit-identical to one launch.
  const int V = p.V, NT = p.NT, n = p.cn;
  const bool seg_first = ADJOINT ? (p.c0 + p.cn == NT) : (p.c0 == 0);
  const bool seg_last = ADJOINT ? (p.c0 == 0) : (p.c0 + p.cn == NT);
  CtaCtl ctl{p.status, &cs->abort_flag};
  uint64_t* bar_full = &cs->bar[0];                 // [kStages] P stage loaded
  uint64_t* bar_free = &cs->bar[kStages];           // [kStages] the products reading the stage are done
  uint64_t* bar_mma = &cs->bar[2 * kStages];        // the step's products are done

  if (tid == 0) {
    cs->abort_flag = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_free[s], kMmaWarps);
    }
    mbar_init(bar_mma, kMmaWarps);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(&cs->tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = cs->tmem_slot;
  auto chunk_of = [&](int it) { return ADJOINT ? p.c0 + n - 1 - it : p.c0 + it; };
  // Record of the state a chunk sees: this CTA's columns in the image of [128][V].  The operand tile is that image and
  // leaves as one bulk copy; stores by the state warps, a row of pieces per thread, held up the step that followed them (1.08 us
  // a step with them, 0.7 like this).
  auto record = [&](int it) {
    const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
    return (ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc) + (ADJOINT ? z : z + bh) * p.lay.sz_hc + static_cast<size_t>(v0 >> 6) * 16384;
  };
  // The kernel before this one wrote R (forward) or Rb (adjoint); P comes from the same kernel in the
  // forward and from the forward call in the adjoint, whose producer may start at once.
  if (!(ADJOINT && warp == kStateWarps)) {
    griddep_wait();
    griddep_launch();
  }

  if (warp == kStateWarps) {
    // ---- producer: keeps the ring of P stages full
    if (lane == 0) {
      const unsigned char* Pg = p.saved + p.lay.p;
      for (int it = 0; it < n; ++it) {
        const int st = it % kStages;
        if (it >= kStages) mbar_wait(&bar_free[st], static_cast<uint32_t>(((it / kStages) - 1) & 1), ctl, 303);
        mbar_expect_tx(&bar_full[st], 32768u);
        const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
        bulk_g2s(Pst + st * 32768, Pg + z * 32768, 32768u, &bar_full[st]);
        // What the state warps load to registers a step ahead goes to L2 now, three steps ahead: a step is shorter than its way from
        // HBM (us, without / with, forward and adjoint alike: 40 pairs x 128 chunks, d_v = 64, 109 / 94; 64 x 64 63 / 52; d_v = 128 19 x 128
        // 105 / 93, 64 x 64 74 / 63; the decays alone 2 %).  In the adjoint not before the kernel that makes Rb has ended.
        if (ADJOINT && it < kStages) continue;
        if (ADJOINT && it == kStages) griddep_wait();
        bulk_prefetch(p.saved + p.lay.ad + z * 512, 512);
        bulk_prefetch((ADJOINT ? p.scratch + p.lay.rb : p.saved + p.lay.r) + z * p.lay.sz_r + static_cast<size_t>(v0 >> 6) * 16384, 16384);
      }
    }
  } else if (warp > kStateWarps) {
    // ---- product issue: warp m takes contraction steps [m * 8 / kMmaWarps, ...) into accumulator m.
    // All lanes stay on the path (uniform descriptors); the elected lane issues.
    const int m = warp - kStateWarps - 1;
    constexpr int kPer = 8 / kMmaWarps;
    const uint32_t leader = elect_leader();
    // A = the P stage (contracted along its columns forward, along its rows for the adjoint),
    // B = the state operand; one 16-element contraction step moves each by a fixed amount
    const uint64_t b_desc0 = make_desc(smem_u32(XB0), 16384u, 1024u);
    const uint32_t idesc = make_idesc(128, kW, ADJOINT, true);
    const uint32_t acc = tmem + static_cast<uint32_t>(m * kW);
    for (int it = 0; it < n; ++it) {
      const int st = it % kStages;
      mbar_wait_warp(&bar_full[st], static_cast<uint32_t>((it / kStages) & 1), ctl, 301);
      if (m == 0 && lane == 0) bulk_wait_read();     // the other operand tile is recorded: it may be written again
      step_sync<kStepBarrier>();
      tc_fence_after();
      const uint32_t pa = smem_u32(Pst + st * 32768);
      const uint64_t a_desc0 = ADJOINT ? make_desc(pa, 16384u, 1024u) : make_desc(pa, 16u, 1024u);
#pragma unroll
      for (int jj = 0; jj < kPer; ++jj) {
        const int j = m * kPer + jj;
        // byte offsets of contraction step j, in the descriptors' 16-byte units
        const uint32_t aoff = ADJOINT ? static_cast<uint32_t>(j * 2048) >> 4
                                      : static_cast<uint32_t>((j >> 2) * 16384 + (j & 3) * 32) >> 4;
        const uint32_t boff = static_cast<uint32_t>(j * 32 * kW + (it & 1) * kXB) >> 4;      // 16 rows of 2 kW bytes per step
        umma_led(leader, acc, a_desc0 + aoff, b_desc0 + boff, idesc, jj > 0 ? 1u : 0u);
      }
      umma_commit_led(leader, bar_mma);
      umma_commit_led(leader, &bar_free[st]);
      if (m == 0 && lane == 0) {       // the operand tile is the record's image
        bulk_s2g(record(it), XB0 + (it & 1) * kXB, kXB);
        bulk_commit();
      }
    }
    if (m == 0 && lane == 0) bulk_wait_read();
  } else {
    // ---- the state: thread d of a group holds kVs columns of row d of x in fp32
    const int d = tid & 127, g = tid >> 7, vg = v0 + g * kVs;      // group g: columns [vg, vg + kVs)
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const __half* Rg = reinterpret_cast<const __half*>(ADJOINT ? p.scratch + p.lay.rb : p.saved + p.lay.r);
    const float* ADg = reinterpret_cast<const float*>(p.saved + p.lay.ad);
    unsigned char* Xg = ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc;
    const size_t szx = p.lay.sz_hc;
    // R / Rb records are [V / 16 column blocks][128 rows][16 columns]: this CTA's block, this thread's row
    const size_t rofs = (static_cast<size_t>(vg / 16) * kK + d) * 16;

    float* carry = reinterpret_cast<float*>(ADJOINT ? p.scratch + p.lay.carry_b : p.saved + p.lay.carry_f);
    float x[kVs];
    {
      const float* x0 = seg_first ? (ADJOINT ? p.dhT : p.h0) : carry;
      const int nrow = seg_first ? p.Kr : kK;      // user states have the real channel count
#pragma unroll
      for (int j = 0; j < kVs; ++j) x[j] = x0 && d < nrow ? x0[(static_cast<size_t>(bh) * nrow + d) * V + vg + j] : 0.f;
    }
    constexpr int kPieces = kVs / 8;             // 16-byte pieces of this thread's row
    uint4 rnext[kPieces];
    auto load_r = [&](int chunk) {
      // the record is cut into blocks of 16 columns: piece q lies in block q / 2 of this CTA's blocks
      const __half* r = Rg + (static_cast<size_t>(bh) * NT + chunk) * kK * V + rofs;
#pragma unroll
      for (int q = 0; q < kPieces; ++q)
        rnext[q] = *reinterpret_cast<const uint4*>(r + (q >> 1) * (kK * 16) + (q & 1) * 8);
    };
    load_r(chunk_of(0));
    float a_next = ADg[(static_cast<size_t>(bh) * NT + chunk_of(0)) * kK + d];

    for (int it = 0; it < n; ++it) {
      unsigned char* XB = XB0 + (it & 1) * kXB;
      // critical path: the state as a tensor-core operand
      {
#pragma unroll
        for (int q = 0; q < kPieces; ++q)
          *reinterpret_cast<uint4*>(XB + d * (2 * kW) + (((g * kPieces + q) ^ (d & 7)) << 4)) = pack8_f16(x + 8 * q);
      }
      fence_proxy_async();
      tc_fence_before();
      step_arrive<kStepBarrier>();
      // in the shadow of the product: this chunk's input and decay, the next chunk's loads
      const float a = a_next;
      float rr[kVs];
#pragma unroll
      for (int q = 0; q < kPieces; ++q) unpack8_f16(rnext[q], rr + 8 * q);
#pragma unroll
      for (int j = 0; j < kVs; ++j) rr[j] = fmaf(a, x[j], rr[j]);
      if (it + 1 < n) {
        const int cn = chunk_of(it + 1);
        load_r(cn);
        a_next = ADg[(static_cast<size_t>(bh) * NT + cn) * kK + d];
      }
      mbar_wait_warp(bar_mma, static_cast<uint32_t>(it & 1), ctl, 302);
      tc_fence_after();
      static_assert(kMmaWarps == 2, "two accumulators of kW columns, one per half of the contraction");
      float a0[kVs], a1[kVs];
      tmem_ld16(tmem + lane_base + g * kVs, a0);
      tmem_ld16(tmem + lane_base + kW + g * kVs, a1);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < kVs; ++j) x[j] = rr[j] - a0[j] - a1[j];      // (in the order of scan_mma_kernel)
    }
    if (!ADJOINT && seg_last) {   // the final state as one more record
      unsigned char* rec = Xg + (static_cast<size_t>(bh) * (NT + 1) + NT) * szx;
#pragma unroll
      for (int q = 0; q < kPieces; ++q)
        *reinterpret_cast<uint4*>(rec + sw128_chunk(d, vg / 8 + q, 128)) = pack8_f16(x + 8 * q);
    }
    float* xT = seg_last ? (ADJOINT ? p.dh0 : p.hT) : carry;
    const int nrow = seg_last ? p.Kr : kK;
    if (xT && d < nrow) {
#pragma unroll
      for (int j = 0; j < kVs; j += 4)
        *reinterpret_cast<float4*>(xT + (static_cast<size_t>(bh) * nrow + d) * V + vg + j) =
            make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------------------------------------
// The same recurrence for few columns per CTA, on warp-level matrix instructions (mma.sync): a step is a chain of latencies, not a
// matter of throughput, and there the accumulator that lies in the registers which also hold the state, and the operand that
// is loaded to registers ahead, beat tcgen05 with its commit, mbarrier and tensor-memory read.  Warps own 16 kM rows of the
// state in the accumulator layout of m16n8k16; per step they leave them as fp16 in shared memory, and after one barrier of the
// state warps each reads all rows as the other operand.  Its rows of P (forward; columns, adjoint), R and the decays of the next
// step are fetched to registers between the products; a producer warp keeps a ring of stages.
// With y = -x the step is y <- (a y - R) + P fp16(x).
//
// The sums are those of scan_kernel, bit for bit (a chain of 16-long products rounds alike in either kind of matrix instruction; the
// tests compare them): each half of the contraction from zero, then bracket + first half + second half.  So a pair's results do
// not depend on how many others are in the call, and heads cut over several GPUs give the bits of the whole.  Starting the
// accumulator with the bracket instead saved the two additions and gave bits that tcgen05 cannot (us a step, so / as here: 8 columns
// 0.39 / 0.39, 16 0.53 / 0.51, 32 0.79 / 0.79; fetching R and storing the record between the products pays for the additions).
//
// Bound by the matrix pipe (17 cycles for a product of 16 x 8 x 16 per SM quarter, so 0.14 us per 8 columns) behind 0.25 us of
// barrier, operand loads and P's way to registers: 0.38 us a step with 8 columns, 0.48 with 16, 0.79 with 32; tcgen05 took 0.69
// with 16 (same measure: slope over the number of chunks, L2 cold) and takes 0.68 with 64.  With the fetch behind the products
// instead of between them 16 columns took 0.62, with four warps of kM = 2 at 32 columns the step is 0.92.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma_f16(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_first(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {      // the same from zero
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

template <int kW, int kSt>
struct ScanMmaSmem {
  static constexpr int kR = kW < 16 ? 4096 : kW * 256;                            // whole blocks of 16 columns
  static constexpr int oR = 32768, oA = oR + kR, kStage = oA + 512;               // P, R, decays of a chunk
  static constexpr int oX = kSt * kStage, kX = 128 * kW * 2;                      // two operand tiles, alternating
  static constexpr int oBar = oX + 2 * kX, kBytes = oBar + 2 * kSt * 8 + 16 + 1024;
};

template <bool ADJOINT, int kW, int kSt, int kM>
__global__ void __launch_bounds__(32 * (8 / kM + 1), 1)
scan_mma_kernel(const Problem p) {
  using S = ScanMmaSmem<kW, kSt>;
  constexpr int kN = kW / 8, kWarps = 8 / kM, kThreads = 32 * kWarps;      // n-tiles; warps of kM m-tiles each
  constexpr int kRec = (128 * kN + kThreads - 1) / kThreads;      // 16-byte pieces of a record per thread
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024(smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + S::oBar);
  uint64_t* empty = full + kSt;
  int* abort_flag = reinterpret_cast<int*>(empty + kSt);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int v0 = blockIdx.x * kW, bh = blockIdx.y + p.bh0, V = p.V, NT = p.NT, n = p.cn;
  const bool seg_first = ADJOINT ? (p.c0 + p.cn == NT) : (p.c0 == 0);        // chunk ranges as in scan_kernel
  const bool seg_last = ADJOINT ? (p.c0 == 0) : (p.c0 + p.cn == NT);
  CtaCtl ctl{p.status, abort_flag};
  if (tid == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kSt; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    fence_mbar_init();
  }
  __syncthreads();
  auto chunk_of = [&](int it) { return ADJOINT ? p.c0 + n - 1 - it : p.c0 + it; };
  const unsigned char* Rg = ADJOINT ? p.scratch + p.lay.rb : p.saved + p.lay.r;

  if (warp == kWarps) {
    // ---- producer.  P and the decays are older than the kernel before in the adjoint scan, whose R is not.
    if (lane == 0) {
      auto load_p = [&](int it) {
        unsigned char* st = sm + (it % kSt) * S::kStage;
        const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
        mbar_expect_tx(&full[it % kSt], S::kStage);
        bulk_g2s(st, p.saved + p.lay.p + z * 32768, 32768u, &full[it % kSt]);
        bulk_g2s(st + S::oA, p.saved + p.lay.ad + z * 512, 512u, &full[it % kSt]);
      };
      auto load_r = [&](int it) {
        const size_t z = static_cast<size_t>(bh) * NT + chunk_of(it);
        bulk_g2s(sm + (it % kSt) * S::kStage + S::oR, Rg + z * p.lay.sz_r + static_cast<size_t>(v0 / 16) * 4096, S::kR, &full[it % kSt]);
      };
      const int first = n < kSt ? n : kSt;
      if (!ADJOINT) griddep_wait();
      for (int it = 0; it < first; ++it) load_p(it);
      if (ADJOINT) griddep_wait();
      for (int it = 0; it < first; ++it) load_r(it);
      for (int it = kSt; it < n; ++it) {
        mbar_wait(&empty[it % kSt], static_cast<uint32_t>(((it / kSt) - 1) & 1), ctl, 303);
        load_p(it);
        load_r(it);
      }
    }
    return;
  }

  // ---- the state
  griddep_wait();
  griddep_launch();
  const int g = lane >> 2, t = lane & 3, m0 = 16 * kM * warp;
  float* carry = reinterpret_cast<float*>(ADJOINT ? p.scratch + p.lay.carry_b : p.saved + p.lay.carry_f);
  unsigned char* Xg = ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc;
  float y[kM][kN][4];
  {
    const float* x0 = seg_first ? (ADJOINT ? p.dhT : p.h0) : carry;
    const int nrow = seg_first ? p.Kr : kK;          // user states have the real channel count
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int j = 0; j < kN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int d = m0 + 16 * m + 8 * e + g;
          float2 v = make_float2(0.f, 0.f);
          if (x0 && d < nrow) v = *reinterpret_cast<const float2*>(x0 + (static_cast<size_t>(bh) * nrow + d) * V + v0 + 8 * j + 2 * t);
          y[m][j][2 * e] = -v.x;
          y[m][j][2 * e + 1] = -v.y;
        }
  }
  // operand tile: rows of kW columns, 16-byte pieces swizzled so that eight rows of one piece lie on different banks
  auto piece = [](int r, int q) { return r * (2 * kW) + ((q ^ (kW == 8 ? 0 : kW == 16 ? (r >> 2) & 1 : (r >> 1) & 3)) << 4); };
  constexpr int kB = (kN + 1) / 2;                   // blocks of 16 columns
  // rows (adjoint: columns) m0 .. m0 + 31 of P, contraction step j
  auto fetch_a = [&](uint32_t P, int j, uint32_t (*A)[8][4]) {
#pragma unroll
    for (int m = 0; m < kM; ++m) {
      if (ADJOINT) {
        const int r = 16 * j + (lane & 7) + ((lane >> 4) << 3), ch = (m0 + 16 * m) / 8 + ((lane >> 3) & 1);
        ldsm4t(P + sw128_chunk(r, ch, 128), A[m][j]);
      } else {
        ldsm4(P + sw128_chunk(m0 + 16 * m + (lane & 15), 2 * j + (lane >> 4), 128), A[m][j]);
      }
    }
  };
  auto fetch_r = [&](int s, uint32_t (*R)[kB][4], float (*a)[2]) {      // ... and R and the decays
    const uint32_t P = smem_u32(sm + s * S::kStage);
#pragma unroll
    for (int m = 0; m < kM; ++m) {
#pragma unroll
      for (int b = 0; b < kB; ++b)
        ldsm4(P + S::oR + b * 4096 + (m0 + 16 * m + (lane & 15)) * 32 + (kW == 8 ? (v0 >> 3) & 1 : lane >> 4) * 16, R[m][b]);
      const float* ad = reinterpret_cast<const float*>(sm + s * S::kStage + S::oA) + m0 + 16 * m + g;
      a[m][0] = ad[0];
      a[m][1] = ad[8];
    }
  };
  auto free_stage = [&](int s) {
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
  };
  auto wait_stage = [&](int it) { mbar_wait_warp(&full[it % kSt], static_cast<uint32_t>((it / kSt) & 1), ctl, 301); };
  uint4 rec[kRec];
  auto record_at = [&](int i, const unsigned char* X) {      // this thread's i-th piece of the operand tile
    const int idx = (tid + kThreads * i) % (128 * kN);
    return X + piece(idx / (kW / 8), idx % (kW / 8));
  };
  auto record = [&](int record, int i) {             // ... into the image of [128][V]
    unsigned char* dst = Xg + static_cast<size_t>(record) * p.lay.sz_hc + static_cast<size_t>(v0 >> 6) * 16384;
    const int idx = tid + kThreads * i, r = idx / (kW / 8), q = idx % (kW / 8);
    if (idx < 128 * kN) *reinterpret_cast<uint4*>(dst + r * 128 + (((((v0 & 63) >> 3) + q) ^ (r & 7)) << 4)) = rec[i];
  };
  auto store_x = [&](unsigned char* X) {
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int j = 0; j < kN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<uint32_t*>(X + piece(m0 + 16 * m + 8 * e + g, j) + 4 * t) = f16x2_sat(-y[m][j][2 * e], -y[m][j][2 * e + 1]);
  };
  auto sync4 = [] { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); };
  uint32_t A0[kM][8][4], A1[kM][8][4], R[kM][kB][4];
  float a[kM][2], acc[kM][kN][4];
  auto add_half = [&]() {
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int j = 0; j < kN; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) y[m][j][e] += acc[m][j][e];
  };
  auto step = [&](int it, uint32_t (*A)[8][4], uint32_t (*An)[8][4]) {
    unsigned char* X = sm + S::oX + (it & 1) * S::kX;
    store_x(X);
    // (a y - R) while the other warps arrive
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int j = 0; j < kN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&R[m][j >> 1][2 * (j & 1) + e]));
          y[m][j][2 * e] = fmaf(a[m][e], y[m][j][2 * e], -r.x);
          y[m][j][2 * e + 1] = fmaf(a[m][e], y[m][j][2 * e + 1], -r.y);
        }
    const bool more = it + 1 < n;
    if (more) wait_stage(it + 1);
    const uint32_t Pn = smem_u32(sm + ((it + 1) % kSt) * S::kStage), xa = smem_u32(X);
    sync4();
    // products, and between them what the next step needs: the matrix pipe takes some 16 cycles for each
    constexpr int kJ = kW == 32 ? 4 : 8;             // contraction steps whose operand is in registers at a time
    // Contraction step behind which R is fetched and the record stored (8: behind the last).  us for 128 chunks, forward / adjoint,
    // both behind the last and like this: 8 columns 57 / 59 and 57 / 57 (other places up to 67 / 63), 16 columns 85 / 85 and 75 / 77,
    // 32 columns 115 / 115 and 111 / 107.
    constexpr int kFetch = kW == 8 ? (ADJOINT ? 1 : 8) : kW == 16 ? 3 : ADJOINT ? 5 : 2, kStore = kW == 16 ? 5 : 8;
    auto store_record = [&]() {
#pragma unroll
      for (int i = 0; i < kRec; ++i) record(bh * (ADJOINT ? NT : NT + 1) + chunk_of(it), i);
    };
#pragma unroll
    for (int h = 0; h < 8 / kJ; ++h) {
      uint32_t B[kJ][kN][2];
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
        if (kW == 8) {
          if (j % 2 == 0) {
            uint32_t r[4];
            ldsm4t(xa + piece(16 * (h * kJ + j) + lane, 0), r);
            B[j][0][0] = r[0]; B[j][0][1] = r[1];
            B[(j + 1) % kJ][0][0] = r[2]; B[(j + 1) % kJ][0][1] = r[3];
          }
        } else {
#pragma unroll
          for (int b = 0; b < kB; ++b) {
            uint32_t r[4];
            ldsm4t(xa + piece(16 * (h * kJ + j) + (lane & 15), 2 * b + (lane >> 4)), r);
            B[j][(2 * b) % kN][0] = r[0]; B[j][(2 * b) % kN][1] = r[1];
            B[j][(2 * b + 1) % kN][0] = r[2]; B[j][(2 * b + 1) % kN][1] = r[3];
          }
        }
      }
      if (h == 0)
#pragma unroll
        for (int i = 0; i < kRec; ++i) rec[i] = *reinterpret_cast<const uint4*>(record_at(i, X));
#pragma unroll
      for (int j = 0; j < kJ; ++j) {
#pragma unroll
        for (int b = 0; b < kN; ++b)
#pragma unroll
          for (int m = 0; m < kM; ++m) {
            if (j % 4) mma_f16(acc[m][b], A[m][h * kJ + j], B[j][b][0], B[j][b][1]);
            else mma_f16_first(acc[m][b], A[m][h * kJ + j], B[j][b][0], B[j][b][1]);
          }
        if (more) fetch_a(Pn, h * kJ + j, An);
        if (h * kJ + j == 3) add_half();
        if (h * kJ + j == kFetch && more) fetch_r((it + 1) % kSt, R, a);
        if (h * kJ + j == kStore) store_record();
      }
    }
    if (kFetch == 8 && more) fetch_r((it + 1) % kSt, R, a);
    add_half();
    if (more) free_stage((it + 1) % kSt);
    if (kStore == 8) store_record();
  };
  wait_stage(0);
#pragma unroll
  for (int j = 0; j < 8; ++j) fetch_a(smem_u32(sm), j, A0);
  fetch_r(0, R, a);
  free_stage(0);
  for (int it = 0; it < n; it += 2) {
    step(it, A0, A1);
    if (it + 1 < n) step(it + 1, A1, A0);
  }
  if (!ADJOINT && seg_last) {                        // the final state as one more record
    unsigned char* X = sm + S::oX + (n & 1) * S::kX;
    store_x(X);
    sync4();
#pragma unroll
    for (int i = 0; i < kRec; ++i) {
      rec[i] = *reinterpret_cast<const uint4*>(record_at(i, X));
      record(bh * (NT + 1) + NT, i);
    }
  }
  float* xT = seg_last ? (ADJOINT ? p.dh0 : p.hT) : carry;
  const int nrow = seg_last ? p.Kr : kK;
  if (xT) {
#pragma unroll
    for (int m = 0; m < kM; ++m)
#pragma unroll
      for (int j = 0; j < kN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int d = m0 + 16 * m + 8 * e + g;
          if (d < nrow)
            *reinterpret_cast<float2*>(xT + (static_cast<size_t>(bh) * nrow + d) * V + v0 + 8 * j + 2 * t) =
                make_float2(-y[m][j][2 * e], -y[m][j][2 * e + 1]);
        }
  }
}

// ---------------------------------------------------------------------------------------------
// Without the delta term the recurrence is x <- a x + R per element: no product, nothing serial but the
// chunk order, and the kernel is bound by reading R and writing the state records once.  Every thread
// owns one 16-byte piece (8 columns) of one row of the state; a warp covers four whole 128-byte rows
// of a record atom, so every access is a full line.  What is on the way from HBM decides the speed: a thread copies the R of
// the next kDepth chunks to shared memory behind its own back.  (As loads to registers, 16 or 8 of them, a wait for one was a wait for
// all that shared its scoreboard, six for a warp, and a step took 0.6 us: 36 pairs x 94 and 188 chunks, d_v = 64, 55 and 114 us, now
// 18 and 40; 64 pairs x 64, d_v = 128, 59, now 46.)
// Slots, whole sequences: 32, one CTA per SM, where that holds the whole grid (in pairs on the first free SMs they share their intake:
// captured step, 16 pairs x 8, d_v = 64, us, 16 / 32 30.6 / 28.8) and for more than 16 chunks (40, 48 and 80 pairs x 64, d_v = 128, 8 / 16 /
// 32: 36 / 39 / 33, 46 / 39 / 36, 63 / 62 / 57).  Shorter ones do not fill that ring, and with many pairs one CTA per SM is a long row of nearly
// empty rounds: 16 slots, and for 8 chunks at most and more CTAs than two per SM 8, four CTAs per SM (three in the forward over 5 to 8
// chunks with d_v = 64: 1024 pairs x 8, three / four 224 / 254; with 64 key channels 169 / 151, and no difference at d_v = 128).  SSD, d_v =
// 128, forward and backward, registers as above / always 32 slots / now: 256 pairs x 1 28 and 38 / 38 and 50 / 26 and 36; 1024 x 1 81 and
// 103 / 120 and 151 / 77 and 95; 256 x 4 58 and 83 / 70 and 95 / 58 and 82; d_v = 64, 1024 x 8 234 and 348 / 239 and 359 / 224 and 348.
// A range of chunks (captured step) has chunk kernels beside it, which need the room: 16 while two CTAs per SM hold the whole grid, 8 beyond
// (captured step, SSD, 16 pairs x 32, d_v = 128, 8 / 16 / 32 88 / 78 / 84; GLA, 64 pairs x 64, 603 / 613 / 625).
// R / Rb and the state records are 128-row tile images, of which rows from Kw on are neither read nor written.
// Grid: (V / 64 atoms x Kw / 32 row blocks, pairs) x 256 threads.
// ---------------------------------------------------------------------------------------------
// A ring of kDepth slots of 16 bytes of R and the row's decay per thread, filled by the thread itself.
template <int kDepth>
struct ScanNdSmem {
  static constexpr int kAd = kDepth * 256 * 16, kBytes = kAd + kDepth * 256 * 4;
};
template <bool ADJOINT, int kDepth>
__global__ void __launch_bounds__(256)
scan_nodelta_kernel(const Problem p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint4* ring = reinterpret_cast<uint4*>(smem_raw) + threadIdx.x;
  float* ring_ad = reinterpret_cast<float*>(smem_raw + ScanNdSmem<kDepth>::kAd) + threadIdx.x;
  const int tid = threadIdx.x, blocks = p.Kw / 32;
  const int atom = blockIdx.x / blocks, d = (blockIdx.x - atom * blocks) * 32 + (tid >> 3), c8 = tid & 7;
  const int bh = blockIdx.y + p.bh0, V = p.V, NT = p.NT, n = p.cn;
  const bool seg_first = ADJOINT ? (p.c0 + p.cn == NT) : (p.c0 == 0);        // chunk ranges as in scan_kernel
  const bool seg_last = ADJOINT ? (p.c0 == 0) : (p.c0 + p.cn == NT);
  const int col0 = atom * 64 + c8 * 8;
  griddep_wait();
  griddep_launch();
  float* carry = reinterpret_cast<float*>(ADJOINT ? p.scratch + p.lay.carry_b : p.saved + p.lay.carry_f);
  const size_t szx = p.lay.sz_hc;
  const uint32_t off = sw128_chunk(d, atom * 8 + c8, 128);     // this thread's piece inside any 128-row image
  // records of the chunk that the walk starts with, and the way to the next
  const size_t z0 = static_cast<size_t>(bh) * NT + (ADJOINT ? p.c0 + n - 1 : p.c0);
  const long long dir = ADJOINT ? -1 : 1;
  const unsigned char* Rg = (ADJOINT ? p.scratch + p.lay.rb : p.saved + p.lay.r) + z0 * p.lay.sz_r + off;
  const float* ADg = reinterpret_cast<const float*>(p.saved + p.lay.ad) + z0 * kK + d;
  unsigned char* X = (ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc) + (ADJOINT ? z0 : z0 + bh) * szx + off;

  float x[8];
  {
    const float* x0 = seg_first ? (ADJOINT ? p.dhT : p.h0) : carry;
    const int nrow = seg_first ? p.Kr : kK;        // user states have the real channel count
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = x0 && d < nrow ? x0[(static_cast<size_t>(bh) * nrow + d) * V + col0 + j] : 0.f;
  }
  auto fetch = [&](int it) {                       // (a group for every step, empty behind the last)
    if (it < n) {
      const int s = it % kDepth;
      async_copy16(ring + s * 256, Rg + it * dir * static_cast<long long>(p.lay.sz_r));
      async_copy4(ring_ad + s * 256, ADg + it * dir * kK, true);
    }
    async_copy_commit();
  };
#pragma unroll 1
  for (int it = 0; it < kDepth - 1; ++it) fetch(it);
#pragma unroll 1
  for (int it = 0; it < n; ++it, X += dir * static_cast<long long>(szx)) {
    *reinterpret_cast<uint4*>(X) = pack8_f16(x);
    async_copy_wait_but<kDepth - 2>();
    fetch(it + kDepth - 1);                        // into the slot that the step before has read
    const int s = it % kDepth;
    const float a = ring_ad[s * 256];
    float rr[8];
    unpack8_f16(ring[s * 256], rr);
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = fmaf(a, x[e], rr[e]);
  }
  if (!ADJOINT && seg_last) *reinterpret_cast<uint4*>(X) = pack8_f16(x);      // the final state as one more record
  float* xT = seg_last ? (ADJOINT ? p.dh0 : p.hT) : carry;
  const int nrow = seg_last ? p.Kr : kK;
  if (xT && d < nrow) {
    float* dst = xT + (static_cast<size_t>(bh) * nrow + d) * V + col0;
    *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(x[4], x[5], x[6], x[7]);
  }
}

static int launch_scan_wide(const Problem& p, bool adjoint, cudaStream_t st) {
  constexpr int smem = kStages * 32768 + 2 * 128 * kW * 2 + static_cast<int>(sizeof(CtaShared)) + 1024;
  const dim3 grid(p.V / kW, p.nbh);
  static SmemAttr attr[2];
  if (attr[0].set(scan_kernel<false>, smem) || attr[1].set(scan_kernel<true>, smem)) return kErrLaunch;
  const cudaError_t e = adjoint ? launch_dependent(scan_kernel<true>, grid, dim3(kScanThreads), smem, st, p)
                                : launch_dependent(scan_kernel<false>, grid, dim3(kScanThreads), smem, st, p);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

template <int kCols>
static int launch_scan_few(const Problem& p, bool adjoint, cudaStream_t st) {
  // Four stages (three to five are within 3 %, two are 20 to 40 % slower).  More than half of an SM's memory on purpose: launched
  // early, CTAs settle in pairs on the first SMs that the kernel before leaves, and share their intake.
  constexpr int kM = kCols == 32 ? 1 : 2, kSt = 4, smem = ScanMmaSmem<kCols, kSt>::kBytes;
  static_assert(smem > 118000 && smem <= 232448, "one CTA per SM");
  const dim3 grid(p.V / kCols, p.nbh), block(32 * (8 / kM + 1));
  static SmemAttr attr[2];
  if (attr[0].set(scan_mma_kernel<false, kCols, kSt, kM>, smem) || attr[1].set(scan_mma_kernel<true, kCols, kSt, kM>, smem)) return kErrLaunch;
  const cudaError_t e = adjoint ? launch_dependent(scan_mma_kernel<true, kCols, kSt, kM>, grid, block, smem, st, p)
                                : launch_dependent(scan_mma_kernel<false, kCols, kSt, kM>, grid, block, smem, st, p);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

// Shared memory with which `most` CTAs fit an SM's 228 KB (each takes 1 KB more) and another does not.
constexpr int scan_share(int most) { return 233472 / (most + 1) - 512; }
// kMost: CTAs per SM at most, 3 or more (0: as many as the ring leaves room for)
template <int kDepth, int kMost = 0>
static int launch_scan_nodelta(const Problem& p, bool adjoint, cudaStream_t st) {
  const dim3 g((p.V / 64) * (p.Kw / 32), p.nbh);
  constexpr int ring = ScanNdSmem<kDepth>::kBytes, smem = kMost && scan_share(kMost) > ring ? scan_share(kMost) : ring;
  constexpr int limit = ring > scan_share(3) ? ring : scan_share(3);      // (one limit per kernel, whatever kMost)
  static_assert(kMost == 0 || (kMost >= 3 && smem <= limit), "");
  static SmemAttr attr[2];
  if (attr[0].set(scan_nodelta_kernel<false, kDepth>, limit) || attr[1].set(scan_nodelta_kernel<true, kDepth>, limit)) return kErrLaunch;
  const cudaError_t e = adjoint ? launch_dependent(scan_nodelta_kernel<true, kDepth>, g, dim3(256), smem, st, p)
                                : launch_dependent(scan_nodelta_kernel<false, kDepth>, g, dim3(256), smem, st, p);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

int launch_scan_io(const Problem&, bool adjoint, const CUtensorMap& mio, const CUtensorMap& mv, cudaStream_t);
int launch_scan(const Problem& p, bool adjoint, cudaStream_t st, const CUtensorMap* mv) {
  if (p.io) return launch_scan_io(p, adjoint, *p.io, mv ? *mv : *p.io, st);
  const int sms = sm_count();
  if (sms <= 0) return kErrDevice;
  if (!p.delta) {
    const int ctas = (p.V / 64) * (p.Kw / 32) * p.nbh, n = p.cn;
    if (n < p.NT) return ctas <= 2 * sms ? launch_scan_nodelta<16>(p, adjoint, st) : launch_scan_nodelta<8>(p, adjoint, st);
    if (n > 16 || ctas <= sms) return launch_scan_nodelta<32>(p, adjoint, st);
    if (n > 8 || ctas <= 2 * sms) return launch_scan_nodelta<16>(p, adjoint, st);
    const bool three = !adjoint && n > 4 && p.V == 64 && p.Kw == kK;
    return three ? launch_scan_nodelta<8, 3>(p, adjoint, st) : launch_scan_nodelta<8, 4>(p, adjoint, st);
  }
  // Warp-level products or tcgen05 (the same bits): by the whole problem, since calls on ranges of its pairs run beside one another.
  // The line is where 16 columns no longer give every CTA an SM of its own: up to it they are the shorter scan (alone, us, 16 / 32 / 64
  // columns, 64 chunks, d_v = 64, 37 pairs 43 / 61 / 59; d_v = 128, 18 pairs 41 / 60 / 58), beyond it not (38 pairs 74 / 60 / 59; 20 pairs
  // 72 / 60 / 58).  There 32 and 64 are alike while 32 have an SM each and a little beyond (forward and backward, 32 / 64: d_v = 64, 38 x 64 172 and
  // 222 / 170 and 225, 64 x 64 244 and 324 / 246 and 329; d_v = 128, 32 x 64 177 and 246 / 179 and 246), and 64 the better the more there is
  // to read, since P is read half as often (32 x 250 639 and 981 / 619 and 919; 64 x 64 334 and 475 / 297 and 439).
  if ((p.V / 16) * p.B * p.H > sms) return launch_scan_wide(p, adjoint, st);
  const int c8 = (p.V / 8) * p.nbh;            // CTAs with 8 columns each
  if (p.cn < p.NT) {
    // A range of the sequences (captured step): chunk kernels of another range run beside the scan, and an SM that a scan CTA sits
    // on is lost to them.  Few CTAs then count for more than a short step.  Captured step, us, 8 / 16 / 32 / 64 columns, pairs x chunks, d_v = 64:
    // 4 x 32 62 / 68 / 86 / 96, 8 x 32 71 / 76 / 89 / 98, 12 x 32 101 / 94 / 98 / 112, 16 x 32 129 / 116 / 107 / 121, 24 x 64 278 / 250 / 254 /
    // 267, 32 x 64 347 / 321 / 316 / 327, 64 x 64 639 / 573 / 567 / 542; d_v = 128: 6 x 32 83 / 78 / 90 / 102, 10 x 32 121 / 105 / 106 / 117, 16 x 32
    // 173 / 152 / 135 / 141, 8 x 128 274 / 249 / 302 / 311, 64 x 64 964 / 838 / 814 / 758; channel-wise, d_v = 128: 3 x 128 184 / 206 / 258 / 251, 16 x
    // 32 210 / 189 / 179 / 167.  So 16 and 64 columns each have a range of sizes where they would be the better ones; the rule knows 8 and
    // 32 only.
    return 3 * c8 <= 2 * sms ? launch_scan_few<8>(p, adjoint, st) : launch_scan_few<32>(p, adjoint, st);
  }
  // A whole sequence: the fewest columns with which every CTA has an SM of its own.  Chain of a step, us, 8 / 16 / 32 columns, d_v = 64:
  // 16 x 32 118 / 121 / 138; 18 x 64 210 / 226 / 261; 32 x 32 208 / 188 / 207; d_v = 128: 9 x 64 170 / 180 / 219; 18 x 32 170 / 152 / 167.
  return c8 <= sms ? launch_scan_few<8>(p, adjoint, st) : launch_scan_few<16>(p, adjoint, st);
}

}  // namespace lg
