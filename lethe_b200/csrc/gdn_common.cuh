// Shared definitions of the GDN kernels: problem description, workspace layout, small device helpers.
//
// Work decomposition.  A "chunk" is 64 consecutive tokens of one (batch, head) pair; chunks are
// numbered z = (b*H + h)*NT + c.  Chunk-parallel kernels run persistent CTAs, one chunk at a time;
// the scan kernels run one CTA per (b, h, slice of 8 to 64 columns of V) and walk the chunks in order.
//
// Per-chunk records in the workspaces ("image" = the SW128 shared-memory tile image, so that a
// record moves between global and shared memory with one contiguous bulk copy):
//   saved (forward -> backward)
//     TA    16 KB   image, 128 rows x 64: rows 0-63 T = (I + strict_lower(M))^-1, rows 64-127 A
//     W     16 KB   image, 64 x 128: WY factor w = T (beta gamma k)
//     U     64 x V  image: u = T (beta v)             (no delta term: v itself, left out of a lean call, as is VN)
//     P     32 KB   image, 128 x 128: kd^T w           (state transition, without the decay)
//     R     128 x V fp16 row-major: kd^T u            (state input)
//     Hc    128 x V image: state entering the chunk; NT + 1 records per (b, h), the last one being
//           the final state, so record index is (b*H + h)*(NT + 1) + c
//     VN    64 x V  image: v_new = u - w h
//     AD    128 fp32: exp(G_last) per key channel     (the decay of the chunk)
//     QG    channel-wise gate only: 16 KB image, 64 x 128: scale * gamma * q, the query operand of the output
//           kernel and of the adjoint scan's input kernel (written by prepare, which has q and the gate in
//           registers anyway, so that those two kernels need neither the gate nor a conversion)
//   scratch (backward only)
//     RB    128 x V fp16 row-major: (q gamma)^T do - w^T (A^T do)
//     DH    128 x V image: adjoint of the state leaving the chunk
//     DV2   64 x V  image: adjoint of v_new
//     DW    64 x 128 image: adjoint of w
//     DKB   64 x 128 fp32, DGB 64 x 128 (channel-wise) or 64 fp32 (scalar): what Stage B leaves for the WY VJP beside DV2
//           and DW when a call is cut between them (the uncut backward keeps all of it on chip)
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "../../include/lethe_gdn.h"
#include "tiles.cuh"

namespace lg {

constexpr int kC = 64;    // chunk length
constexpr int kK = 128;   // key dimension

struct Layout {
  // byte offsets of the record arrays inside `saved` / `scratch`, and record sizes
  size_t ta, w, u, p, r, hc, vn, ad, qg, carry_f, saved_total;
  size_t rb, dh, dv2, dw, dkb, dgb, carry_b, scratch_total;
  size_t sz_ta, sz_w, sz_u, sz_p, sz_r, sz_hc, sz_vn, sz_ad;
  size_t sz_rb, sz_dh, sz_dv2, sz_dw, sz_dkb, sz_dgb;
};

__host__ inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

__host__ inline Layout make_layout(const LetheGdnDims& d) {
  Layout l{};
  const size_t Z = static_cast<size_t>(d.B) * d.H * (d.L / kC);
  const size_t V = d.V;
  l.sz_ta = 16384; l.sz_w = 16384; l.sz_u = kC * V * 2; l.sz_p = 32768; l.sz_r = kK * V * 2;
  l.sz_hc = kK * V * 2; l.sz_vn = kC * V * 2; l.sz_ad = kK * 4;
  size_t o = 0;
  l.ta = o; o = align_up(o + Z * l.sz_ta, 1024);
  l.w = o;  o = align_up(o + Z * l.sz_w, 1024);
  l.u = o;  o = align_up(o + Z * l.sz_u, 1024);
  l.p = o;  o = align_up(o + Z * l.sz_p, 1024);
  l.r = o;  o = align_up(o + Z * l.sz_r, 1024);
  l.hc = o; o = align_up(o + (Z + static_cast<size_t>(d.B) * d.H) * l.sz_hc, 1024);
  l.vn = o; o = align_up(o + Z * l.sz_vn, 1024);
  l.ad = o; o = align_up(o + Z * l.sz_ad, 1024);
  if (d.gate == LETHE_GATE_CHANNEL) {
    l.qg = o; o = align_up(o + Z * static_cast<size_t>(16384), 1024);
  }
  // fp32 master state handed from one chunk-range call of the forward scan to the next ([B, H, K, V])
  l.carry_f = o; o = align_up(o + static_cast<size_t>(d.B) * d.H * kK * V * 4, 1024);
  l.saved_total = o;
  l.sz_rb = kK * V * 2; l.sz_dh = kK * V * 2; l.sz_dv2 = kC * V * 2; l.sz_dw = 16384;
  l.sz_dkb = kC * kK * 4; l.sz_dgb = (d.gate == LETHE_GATE_CHANNEL ? kC * kK : kC) * 4;
  o = 0;
  l.rb = o;  o = align_up(o + Z * l.sz_rb, 1024);
  l.dh = o;  o = align_up(o + Z * l.sz_dh, 1024);
  l.dv2 = o; o = align_up(o + Z * l.sz_dv2, 1024);
  l.dw = o;  o = align_up(o + Z * l.sz_dw, 1024);
  l.dkb = o; o = align_up(o + Z * l.sz_dkb, 1024);
  l.dgb = o; o = align_up(o + Z * l.sz_dgb, 1024);
  l.carry_b = o; o = align_up(o + static_cast<size_t>(d.B) * d.H * kK * V * 4, 1024);   // the same for the adjoint scan
  l.scratch_total = o;
  return l;
}

// Everything a kernel needs besides its tensor maps.
struct Problem {
  int B, H, L, NT, V, gate, delta;   // L: tokens of the user tensors (the last chunk may be partly filled)
  int Kr;            // key channels of the user tensors (64 or 128); the kernels work on 128, missing ones are zero
  int Kw;            // key channels that these calls work on: Kr for one decay or none without the delta term, 128 elsewhere
  int bh0, nbh;      // the (batch, head) pairs this call works on: [bh0, bh0 + nbh) of the B * H pairs
  int c0, cn;        // the chunks of every pair this call works on: [c0, c0 + cn) of the NT chunks
  uint32_t lean;     // 1: intermediates that no later kernel of the call reads are not written; 2: nor what only a backward reads
  int qk16;          // non-zero: q, k, dq, dk hold fp16 instead of bf16
  float scale;
  const CUtensorMap* io;      // host only: the scan takes the kernel beside it along (launch_scan), whose tensor this is
  int after_scan;    // the same call launched the adjoint scan just before the main kernel
  float l2_eps;      // > 0: the prepare kernel normalises q and k (q for the output kernel too, where that reads it)
  int keep_norm;     // ... and stores the normalised rows
  const __nv_bfloat16 *q, *k, *v, *d_o;
  const float *g, *beta, *h0, *dhT;
  __nv_bfloat16 *o, *dq, *dk, *dv;
  float *hT, *dg, *dbeta, *dh0, *dbeta_w;
  // full op only (null otherwise): per-channel erase gate [B,L,H,K], write gate [B,L,H,V] and their gradients
  const float *bch, *wch;
  float *dbch, *dwch;
  unsigned char* saved;
  unsigned char* scratch;
  Layout lay;
  int* status;

  // rows of chunk c that hold tokens (all kC but for the last chunk of a ragged sequence).  The tensor maps end at
  // the real token and channel counts, so the missing rows and channels of every tile read as zero and are not stored;
  // a kernel that goes to memory by itself tests the row.  A row with k = v = q = 0, g = 0, beta = 0 leaves the state alone.
  __device__ __forceinline__ int rows_of(int c) const { return min(kC, L - c * kC); }
};

// ---------------------------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------------------------
// Inclusive suffix sum of one value per thread over threads 0..63 (x_t + x_{t+1} + ... + x_63; two warps); every thread of
// the CTA must call it (it contains __syncthreads).  `tmp` is a shared float[2].
__device__ __forceinline__ float chunk_rev_cumsum(float x, int tid, float* tmp) {
  const int lane = tid & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float y = __shfl_down_sync(0xffffffffu, x, o);
    if (lane + o < 32) x += y;
  }
  if (tid == 32) tmp[0] = x;
  __syncthreads();
  if (tid < 32) x += tmp[0];
  return x;
}

constexpr float kLog2e = 1.4426950408889634f;

// Control block at the start of every kernel: barriers, TMEM slot, abort flag.
struct CtaShared {
  uint64_t bar[8];
  uint32_t tmem_slot;
  int abort_flag;
};


// Next 1024-byte boundary of the dynamic shared memory window, two ways.  `align1024` is plain
// pointer arithmetic on the shared symbol, so the compiler keeps the shared address space and emits
// shared-memory loads and stores; `align1024_generic` goes through an integer, after which every
// access is a generic one.  Same addresses, different instruction selection and scheduling.  The chunk
// kernels want the first (us, generic against shared: prepare 148 / 135 at 4096 chunks, channel-wise 667 /
// 590 at 8192; main 270 / 224 and 1051 / 915; output and scan input within 3 %, once 78 / 70).  The scan of
// 64 columns per CTA is 1-3 % faster with the second (64.7 / 63.4 for 32 pairs x 64 chunks).
__device__ __forceinline__ unsigned char* align1024(unsigned char* p) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
  return p + ((1024u - (a & 1023u)) & 1023u);
}
__device__ __forceinline__ unsigned char* align1024_generic(unsigned char* p) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 1023) & ~static_cast<uintptr_t>(1023));
}

// Called by all threads before one thread issues products that read tiles written by this CTA's
// threads and / or overwrite accumulators that this CTA's threads have been reading.
__device__ __forceinline__ void sync_for_issue() {
  tc_fence_before();
  fence_proxy_async();
  __syncthreads();
}

// Called by all threads after the issuing thread committed to `bar`: waits for the products.
__device__ __forceinline__ void wait_products(uint64_t* bar, uint32_t& phase, const CtaCtl& ctl, int code) {
  __syncwarp();
  mbar_wait_warp(bar, phase, ctl, code);
  phase ^= 1u;
  tc_fence_after();
}

// ---- packed pairs of fp32 ----------------------------------------------------------------------------------------
struct f2 { unsigned long long u; };
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.u) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.u)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.u) : "l"(a.u), "l"(b.u));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.u) : "l"(a.u), "l"(b.u), "l"(c.u));
  return r;
}
// two neighbouring pairs from shared memory (16-byte aligned)
__device__ __forceinline__ void ld_pairs(const float* src, f2* out) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(src);
  out[0].u = v.x;
  out[1].u = v.y;
}
__device__ __forceinline__ float sum2(f2 a) {
  float lo, hi;
  unpack2(a, lo, hi);
  return lo + hi;
}

// eight consecutive floats (16-byte aligned)
__device__ __forceinline__ void ld8(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8(float* p, const float* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}

// 32 bytes at a 32-byte boundary of global memory, one sector per lane
__device__ __forceinline__ void st_global_32(unsigned char* dst, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
               "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

// Four bytes of global memory to shared memory behind this thread's back, or zero.
__device__ __forceinline__ void async_copy4(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}
__device__ __forceinline__ void async_copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void async_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_copy_wait_but() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }      // all but the N latest groups
__device__ __forceinline__ void async_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// With the delta term the scan's input records R / Rb (128 rows x V columns, fp16) are stored as V / 16 column blocks of
// [128 rows][16 columns]: a scan CTA takes whole blocks, contiguous pieces of 4 KB.  Byte offset of
// the 8-column piece `col8` of `row` (without the delta term they are plain 128-row tile images, read by
// scan_nodelta_kernel with full-line accesses):
__device__ __forceinline__ uint32_t rrec_off(int row, int col8) {
  return static_cast<uint32_t>((col8 >> 1) * 4096 + row * 32 + (col8 & 1) * 16);
}

// A record of [128 rows][V] as a tile of its first KW rows in shared memory (atoms of KW rows), and back.
template <int V, int KW>
__device__ __forceinline__ void load_image(unsigned char* dst, const unsigned char* rec, uint64_t* bar) {
  if (KW == kK) bulk_g2s(dst, rec, V * 256, bar);
  else for (int i = 0; i < V / 64; ++i) bulk_g2s(dst + i * KW * 128, rec + i * 16384, KW * 128, bar);
}
template <int V, int KW>
__device__ __forceinline__ void prefetch_image(const unsigned char* rec) {
  if (KW == kK) bulk_prefetch(rec, V * 256);
  else for (int i = 0; i < V / 64; ++i) bulk_prefetch(rec + i * 16384, KW * 128);
}
template <int V, int KW>
__device__ __forceinline__ void store_image(unsigned char* rec, const unsigned char* src) {
  if (KW == kK) bulk_s2g(rec, src, V * 256);
  else for (int i = 0; i < V / 64; ++i) bulk_s2g(rec + i * 16384, src + i * KW * 128, KW * 128);
}

// Where the n-th chunk of a call is: record index, and batch, head and chunk in the user's tensors.  One thread works it out
// (divisions) and leaves it in shared memory for the others.
struct __align__(16) ChunkAt { int z, b, h, c; };
__device__ __forceinline__ ChunkAt chunk_at(const Problem& p, int n) {
  const int q = n / p.cn, bh = p.bh0 + q;
  ChunkAt a;
  a.c = p.c0 + n - q * p.cn;
  a.z = bh * p.NT + a.c;
  a.b = bh / p.H;
  a.h = bh - a.b * p.H;
  return a;
}

// One value per token of chunk c to shared memory by one warp, two neighbouring tokens per lane, zero behind the last token; each
// lane waits for its own (async_copy_wait) and reads them.  A chunk's gates are fetched like this a chunk ahead: a load to registers
// is waited for by the warp that issues it, and by all others at the next barrier.
__device__ __forceinline__ void warp_copy_gates(const Problem& p, const float* src, int b, int c, int h, int lane, float* dst) {
  const int last = p.rows_of(c) - 1;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int t = 2 * lane + e;
    async_copy4(dst + t, src + (static_cast<size_t>(b) * p.L + c * kC + min(t, last)) * p.H + h, t <= last);
  }
}
// scale * gamma_t of the 64 tokens of a chunk by one warp (scalar gate or none): from the decays that warp_copy_gates brought
__device__ __forceinline__ void warp_scaled_gammas(const Problem& p, int lane, float* io) {
  float g[2] = {0.f, 0.f};
  if (p.gate == LETHE_GATE_SCALAR) {
    async_copy_wait();
    g[0] = io[2 * lane];
    g[1] = io[2 * lane + 1];
  }
  float sum = g[0] + g[1];
#pragma unroll
  for (int w = 1; w < 32; w <<= 1) {
    const float y = __shfl_up_sync(0xffffffffu, sum, w);
    if (lane >= w) sum += y;
  }
  *reinterpret_cast<float2*>(io + 2 * lane) = make_float2(p.scale * __expf(sum - g[1]), p.scale * __expf(sum));
}

}  // namespace lg
