// The serial part of the path: the chunk-to-chunk state recurrence, forward and adjoint.
//
//   forward :  x_{c+1} = a_c * x_c - P_c   x_c + R_c      c = 0 .. NT-1     (x_0 = h0)
//   adjoint :  x_{c-1} = a_c * x_c - P_c^T x_c + Rb_c     c = NT-1 .. 0     (x_NT = dhT)
//
// a_c is the chunk's decay per key channel, P_c = kd^T w (128 x 128) and R_c / Rb_c (128 x V) come
// from the chunk-parallel kernels.  The recurrence is independent per column of x, so the grid is
// (V / 16) x (B*H): every CTA owns 16 columns, keeps them as fp32 in registers (thread d = key
// channel d) and does ONE tcgen05 product per chunk, with P streamed through a ring of shared-memory
// stages by bulk copies that run ahead of the recurrence.  The state seen by chunk c is written out
// as a shared-memory tile image for the chunk-parallel kernels.
// Reference: the forward recurrence gdn2_chunkwise.py:155-158 and the reverse scan K#1
// gdn2_assemble.py:71-99 of the reference project, after substituting v_new / dv2.
#include "gdn_common.cuh"
#include "host_util.h"

namespace lg {

constexpr int kStages = 3;
constexpr int kMmaWarps = 2;   // warps that issue the step's products (each its own accumulator)
// Columns of the state per CTA: 16 on four state-holding warps or 64 on sixteen (kGr groups of four warps, 16 columns
// per thread either way).  The narrow CTA has the shorter step, 0.5 us against 0.7 us; but every CTA of a (batch, head)
// pair streams all of P, so the wide form moves a quarter of its bytes from L2 - see the rule in launch_scan.
// warps 0 .. 4 kGr - 1 hold the state (thread d = key channel d), then one warp streams P, two issue products
constexpr int kVs = 16;

// Step barrier of the delta path: the state-holding warps arrive once the operand is written (and go
// on to work that does not depend on the product), the issuing warps wait for them.
template <int kN>
__device__ __forceinline__ void step_arrive() { asm volatile("bar.arrive 1, %0;" ::"n"(kN) : "memory"); }
template <int kN>
__device__ __forceinline__ void step_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kN) : "memory"); }

template <int kGr>
constexpr int kScanThreads = (4 * kGr + 1 + kMmaWarps) * 32;

template <bool ADJOINT, int kGr>
__global__ void __launch_bounds__(kScanThreads<kGr>, kGr == 1 ? 2 : 1)
scan_kernel(const Problem p) {
  constexpr int kW = kVs * kGr;                      // columns of this CTA: 16 or 64
  constexpr int kTmemCols = kMmaWarps * kW;         // 32 or 128
  constexpr int kXB = 128 * kW * 2;                  // bytes of the state operand tile
  constexpr int kStateWarps = 4 * kGr, kStepBarrier = (kStateWarps + kMmaWarps) * 32;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align1024_generic(smem_raw);
  unsigned char* Pst = sm;                          // kStages x 32 KB
  // x as the B operand, contracted along its rows (row k = key channel k, kW columns = 32 or 128 bytes):
  // atoms of 8 rows with the swizzle of that width, so that thread k stores its row as 16-byte pieces
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
  // Record of the state a chunk sees: this CTA's columns in the image of [128][V].  At 64 columns the operand tile is that
  // image and leaves as one bulk copy; stores by the state warps, a row of pieces per thread, held up the step that
  // followed them (1.08 us a step with them, 0.7 like this).  At 16 columns they cost next to nothing.
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
        bulk_g2s(Pst + st * 32768, Pg + (static_cast<size_t>(bh) * NT + chunk_of(it)) * 32768, 32768u, &bar_full[st]);
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
    const uint64_t b_desc0 = kW == 16 ? make_desc_sw32(smem_u32(XB0), 16u, 256u) : make_desc(smem_u32(XB0), 16384u, 1024u);
    const uint32_t idesc = make_idesc(128, kW, ADJOINT, true);
    const uint32_t acc = tmem + static_cast<uint32_t>(m * kW);
    for (int it = 0; it < n; ++it) {
      const int st = it % kStages;
      mbar_wait_warp(&bar_full[st], static_cast<uint32_t>((it / kStages) & 1), ctl, 301);
      if (kW == 64 && m == 0 && lane == 0) bulk_wait_read();     // the other operand tile is recorded: it may be written again
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
      if (kW == 64 && m == 0 && lane == 0) {       // the operand tile is the record's image
        bulk_s2g(record(it), XB0 + (it & 1) * kXB, kXB);
        bulk_commit();
      }
    }
    if (kW == 64 && m == 0 && lane == 0) bulk_wait_read();
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
        // 32-byte swizzle: the two pieces of rows 4-7 of an atom swap; 128-byte swizzle: piece q of row r sits at q ^ (r & 7)
        const int sw = kW == 16 ? (d >> 2) & 1 : d & 7;
#pragma unroll
        for (int q = 0; q < kPieces; ++q)
          *reinterpret_cast<uint4*>(XB + d * (2 * kW) + (((g * kPieces + q) ^ sw) << 4)) = pack8_f16(x + 8 * q);
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
      if (kW < 64) {
        unsigned char* rec = record(it);
#pragma unroll
        for (int q = 0; q < kPieces; ++q)
          *reinterpret_cast<uint4*>(rec + d * 128 + (((((vg & 63) >> 3) + q) ^ (d & 7)) << 4)) = pack8_f16(x + 8 * q);
      }
      mbar_wait_warp(bar_mma, static_cast<uint32_t>(it & 1), ctl, 302);
      tc_fence_after();
      static_assert(kMmaWarps == 2, "two accumulators of kW columns, one per half of the contraction");
      float a0[kVs], a1[kVs];
      tmem_ld16(tmem + lane_base + g * kVs, a0);
      tmem_ld16(tmem + lane_base + kW + g * kVs, a1);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < kVs; ++j) x[j] = rr[j] - (a0[j] + a1[j]);
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
// Without the delta term the recurrence is x <- a x + R per element: no product, nothing serial but the
// chunk order, and the kernel is bound by reading R and writing the state records once.  Every thread
// owns one 16-byte piece (8 columns) of one row of the state; a warp covers four whole 128-byte rows
// of a record atom, so every access is a full line.  A thread keeps the R of the next
// kDepth chunks on the way: 16 while two CTAs per SM hold the whole grid, 8 beyond that, where four do (B H = 36, d_v = 64, 47
// chunks: forward and backward 184 us with 8, 176 with 16; B H = 64, d_v = 128, 64 chunks: 554 us with 8, 603 with 16).
// R / Rb and the state records are 128-row tile images.
// Grid: (V / 64 atoms x 4 row blocks, pairs) x 256 threads.
// ---------------------------------------------------------------------------------------------
template <bool ADJOINT, int kDepth>
__global__ void __launch_bounds__(256, kDepth == 16 ? 2 : 4)
scan_nodelta_kernel(const Problem p) {
  const int tid = threadIdx.x;
  const int atom = blockIdx.x >> 2, d = (blockIdx.x & 3) * 32 + (tid >> 3), c8 = tid & 7;
  const int bh = blockIdx.y + p.bh0, V = p.V, NT = p.NT, n = p.cn;
  const bool seg_first = ADJOINT ? (p.c0 + p.cn == NT) : (p.c0 == 0);        // chunk ranges as in scan_kernel
  const bool seg_last = ADJOINT ? (p.c0 == 0) : (p.c0 + p.cn == NT);
  const int col0 = atom * 64 + c8 * 8;
  griddep_wait();
  griddep_launch();
  float* carry = reinterpret_cast<float*>(ADJOINT ? p.scratch + p.lay.carry_b : p.saved + p.lay.carry_f);
  const unsigned char* Rg = ADJOINT ? p.scratch + p.lay.rb : p.saved + p.lay.r;
  const float* ADg = reinterpret_cast<const float*>(p.saved + p.lay.ad);
  unsigned char* Xg = ADJOINT ? p.scratch + p.lay.dh : p.saved + p.lay.hc;
  const size_t szx = p.lay.sz_hc;
  const uint32_t off = sw128_chunk(d, atom * 8 + c8, 128);     // this thread's piece inside any 128-row image
  auto chunk_of = [&](int it) { return ADJOINT ? p.c0 + n - 1 - it : p.c0 + it; };

  float x[8];
  {
    const float* x0 = seg_first ? (ADJOINT ? p.dhT : p.h0) : carry;
    const int nrow = seg_first ? p.Kr : kK;        // user states have the real channel count
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = x0 && d < nrow ? x0[(static_cast<size_t>(bh) * nrow + d) * V + col0 + j] : 0.f;
  }
  uint4 rb[kDepth];
  float ab[kDepth];
  auto load = [&](int j, int it) {
    if (it < n) {
      const size_t zj = static_cast<size_t>(bh) * NT + chunk_of(it);
      rb[j] = *reinterpret_cast<const uint4*>(Rg + zj * p.lay.sz_r + off);
      ab[j] = ADg[zj * kK + d];
    }
  };
#pragma unroll
  for (int j = 0; j < kDepth; ++j) load(j, j);
  for (int it0 = 0; it0 < n; it0 += kDepth) {
#pragma unroll
    for (int j = 0; j < kDepth; ++j) {
      if (it0 + j < n) {
        const size_t zj = static_cast<size_t>(bh) * NT + chunk_of(it0 + j);
        *reinterpret_cast<uint4*>(Xg + (ADJOINT ? zj : zj + bh) * szx + off) = pack8_f16(x);
        float rr[8];
        unpack8_f16(rb[j], rr);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = fmaf(ab[j], x[e], rr[e]);
        load(j, it0 + j + kDepth);
      }
    }
  }
  if (!ADJOINT && seg_last)   // the final state as one more record
    *reinterpret_cast<uint4*>(Xg + (static_cast<size_t>(bh) * (NT + 1) + NT) * szx + off) = pack8_f16(x);
  float* xT = seg_last ? (ADJOINT ? p.dh0 : p.hT) : carry;
  const int nrow = seg_last ? p.Kr : kK;
  if (xT && d < nrow) {
    float* dst = xT + (static_cast<size_t>(bh) * nrow + d) * V + col0;
    *reinterpret_cast<float4*>(dst) = make_float4(x[0], x[1], x[2], x[3]);
    *reinterpret_cast<float4*>(dst + 4) = make_float4(x[4], x[5], x[6], x[7]);
  }
}

constexpr int kScanAloneBytes = 118000;
template <int kGr>
static int launch_scan_t(const Problem& p, bool adjoint, cudaStream_t st) {
  constexpr int kW = kVs * kGr;
  int smem = kStages * 32768 + 2 * 128 * kW * 2 + static_cast<int>(sizeof(CtaShared)) + 1024;
  // Launched early, CTAs of 16 columns settle in pairs on the first SMs that the kernel before leaves, and share their intake;
  // asking for more than half of an SM's memory keeps them apart (one chain, us: 16 pairs x 32 chunks 131 -> 122, d_v = 128 166
  // -> 152, 32 x 64 373 -> 357).  Not when the sequences are cut: the next range's scan then waits on the SMs of this one, not
  // on others (captured step, alone / in pairs: 16 x 32 116 / 107, channel-wise 199 / 190; 8 x 32, with room for all, 75 / 83).
  if (kGr == 1 && p.cn == p.NT) smem = kScanAloneBytes;
  dim3 grid(p.V / kW, p.nbh);
  if (adjoint) {
    static SmemAttr attr;
    if (attr.set(scan_kernel<true, kGr>, kGr == 1 ? kScanAloneBytes : smem)) return kErrLaunch;
    if (launch_dependent(scan_kernel<true, kGr>, grid, dim3(kScanThreads<kGr>), smem, st, p) != cudaSuccess) return kErrLaunch;
  } else {
    static SmemAttr attr;
    if (attr.set(scan_kernel<false, kGr>, kGr == 1 ? kScanAloneBytes : smem)) return kErrLaunch;
    if (launch_dependent(scan_kernel<false, kGr>, grid, dim3(kScanThreads<kGr>), smem, st, p) != cudaSuccess) return kErrLaunch;
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

template <int kDepth>
static int launch_scan_nodelta(const Problem& p, bool adjoint, bool alone, cudaStream_t st) {
  const dim3 g((p.V / 64) * 4, p.nbh);
  const int smem = alone && p.cn == p.NT ? kScanAloneBytes : 0;      // as above: one CTA per SM
  static SmemAttr attr[2];
  if (attr[0].set(scan_nodelta_kernel<false, kDepth>, kScanAloneBytes) || attr[1].set(scan_nodelta_kernel<true, kDepth>, kScanAloneBytes)) return kErrLaunch;
  const cudaError_t e = adjoint ? launch_dependent(scan_nodelta_kernel<true, kDepth>, g, dim3(256), smem, st, p)
                                : launch_dependent(scan_nodelta_kernel<false, kDepth>, g, dim3(256), smem, st, p);
  return e == cudaSuccess ? kOk : kErrLaunch;
}

int launch_scan(const Problem& p, bool adjoint, cudaStream_t st) {
  const int sms = sm_count();
  if (sms <= 0) return kErrDevice;
  if (!p.delta) {
    const int ctas = (p.V / 64) * 4 * p.nbh;
    return ctas <= 2 * sms ? launch_scan_nodelta<16>(p, adjoint, ctas <= sms, st) : launch_scan_nodelta<8>(p, adjoint, false, st);
  }
  // 16 columns per CTA while every CTA has an SM of its own (B H = 16: 19.7 us for 32 chunks against 25.8); beyond that
  // the CTAs share the SMs' intake from L2 and P's repeats count (d_v = 128, us for 64 chunks, 16 / 64 columns: B H = 24
  // 61.8 / 57, 32 63 / 60, 48 119 / 67, 64 122 / 76, 128 252 / 156)
  return (p.V / 16) * p.nbh <= sms ? launch_scan_t<1>(p, adjoint, st) : launch_scan_t<4>(p, adjoint, st);
}

}  // namespace lg
