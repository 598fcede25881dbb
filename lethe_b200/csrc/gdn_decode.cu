// Token-serial form of the path for generation: one recurrence step per (batch, head) pair with the
// state kept in HBM between calls,
//
//   S <- S * exp(g);   v_new = beta (v - k^T S);   S <- S + k v_new^T;   o = (scale q)^T S
//
// (reference gdn_backward.py:45-53, one iteration of its token loop; beta == null drops the delta term).
// The step is bound by reading and writing the fp32 state once: K x V x 4 bytes each way per pair.
// One CTA of 4 V threads per pair: four threads share column c of S (32 rows each) and keep their
// entries in registers between the two passes over the column (first k^T S, then the update and q^T S), so the state crosses HBM
// exactly once in each direction and every load of a warp is one contiguous row segment.  No tensor
// cores: 4 flops per state byte.
#include <cuda_bf16.h>

#include "../../include/lethe_gdn.h"
#include "host_util.h"

namespace lg {

constexpr int kDK = 128;

struct DecodeProblem {
  int BH, H, V, gate, delta;
  float scale;
  const void *q, *k, *v;      // bf16, or fp32 (rounded to bf16 as read)
  const float *g, *beta;
  float* state;
  __nv_bfloat16* o;
};

// kSplit threads share a column of S (kDK / kSplit rows each).
constexpr int kSplit = 4;

template <bool F32>
__device__ __forceinline__ float token_in(const void* x, size_t i) {
  if (F32) return __bfloat162float(__float2bfloat16_rn(static_cast<const float*>(x)[i]));
  return __bfloat162float(static_cast<const __nv_bfloat16*>(x)[i]);
}

template <int V, bool F32>
__global__ void __launch_bounds__(kSplit * V, 1024 / (kSplit * V))
decode_step_kernel(const DecodeProblem p) {
  __shared__ float ks[kDK], qs[kDK], as[kDK], part[kSplit][V];
  const int bh = blockIdx.x, c = threadIdx.x % V, part_id = threadIdx.x / V;   // rows [kRows part_id, + kRows)
  for (int d = threadIdx.x; d < kDK; d += kSplit * V) {
    ks[d] = token_in<F32>(p.k, static_cast<size_t>(bh) * kDK + d);
    qs[d] = p.scale * token_in<F32>(p.q, static_cast<size_t>(bh) * kDK + d);
    float a = 1.f;
    if (p.gate == LETHE_GATE_SCALAR) a = __expf(p.g[bh]);
    else if (p.gate == LETHE_GATE_CHANNEL) a = __expf(p.g[static_cast<size_t>(bh) * kDK + d]);
    as[d] = a;
  }
  constexpr int kRows = kDK / kSplit;
  float* S = p.state + (static_cast<size_t>(bh) * kDK + part_id * kRows) * V + c;
  float col[kRows];
#pragma unroll
  for (int d = 0; d < kRows; ++d) col[d] = S[static_cast<size_t>(d) * V];   // all loads in flight at once
  __syncthreads();
  const float* kh = ks + part_id * kRows;
  const float* qh = qs + part_id * kRows;
  const float* ah = as + part_id * kRows;
  float ksum = 0.f;
#pragma unroll
  for (int d = 0; d < kRows; ++d) {
    col[d] *= ah[d];
    ksum += kh[d] * col[d];
  }
  part[part_id][c] = ksum;
  __syncthreads();
  ksum = 0.f;
#pragma unroll
  for (int s = 0; s < kSplit; ++s) ksum += part[s][c];
  float vn = token_in<F32>(p.v, static_cast<size_t>(bh) * V + c);
  if (p.delta) vn = p.beta[bh] * (vn - ksum);
  float o = 0.f;
#pragma unroll
  for (int d = 0; d < kRows; ++d) {
    col[d] += kh[d] * vn;
    o += qh[d] * col[d];
    S[static_cast<size_t>(d) * V] = col[d];
  }
  __syncthreads();
  part[part_id][c] = o;
  __syncthreads();
  if (part_id == 0) {
    float os = 0.f;
#pragma unroll
    for (int s = 0; s < kSplit; ++s) os += part[s][c];
    p.o[static_cast<size_t>(bh) * V + c] = __float2bfloat16_rn(os);
  }
}

// The same step for more pairs than the kernel above holds at a time, d_v = 128.  There a CTA's loads, sums and stores
// follow one another and only the neighbouring CTA fills the gaps.  Here two persistent CTAs per SM keep the next state of
// each in flight (cp.async into slots that only the copying thread reads) while the present one is in registers: 2048 pairs
// 53.3 -> 49.1 us (5.5 TB/s; about 4 us of it start and drain), 1024 pairs 28.7 -> 27.0, 592 pairs 16.9 -> 16.5
// (two full rounds, where the rule's line is); 445 pairs 14.6 -> 16.2.  Three CTAs per SM spill; two or three slots for one CTA leave the SM idle at its barriers (57 us).
constexpr int kRingThreads = 256, kRingCtas = 2, kRingWarps = kRingThreads / 32, kRingRows = kDK / kRingWarps;
constexpr int kRingBytes = kDK * 128 * 4;

__device__ __forceinline__ void copy_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <bool F32>
__global__ void __launch_bounds__(kRingThreads, kRingCtas)
decode_ring_kernel(const DecodeProblem p) {
  constexpr int V = 128;
  extern __shared__ __align__(16) float4 slots[];                    // [row of the warp][thread]
  __shared__ float ks[2][kDK], as[kDK], qs[kDK], bs;
  __shared__ __align__(16) float vs[V];
  __shared__ __align__(16) float kpart[kRingWarps][V], opart[kRingWarps][V];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;         // rows [kRingRows warp, +), columns [4 lane, +4)
  const size_t own = static_cast<size_t>(warp * kRingRows) * 32 + lane;
  auto fetch = [&](int bh) {
    if (bh < p.BH) {
      const float4* src = reinterpret_cast<const float4*>(p.state + static_cast<size_t>(bh) * kDK * V) + own;
      const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(slots + tid));
#pragma unroll
      for (int r = 0; r < kRingRows; ++r) copy_async16(dst + r * kRingThreads * 16, src + r * 32);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the token's vectors: k, q, decay by threads 0-127, v and beta by the others
  float t0 = 0.f, t1 = 0.f, t2 = 1.f;
  auto token = [&](int bh) {
    if (bh >= p.BH) return;
    if (tid < kDK) {
      t0 = token_in<F32>(p.k, static_cast<size_t>(bh) * kDK + tid);
      t1 = p.scale * token_in<F32>(p.q, static_cast<size_t>(bh) * kDK + tid);
      if (p.gate == LETHE_GATE_SCALAR) t2 = __expf(p.g[bh]);
      else if (p.gate == LETHE_GATE_CHANNEL) t2 = __expf(p.g[static_cast<size_t>(bh) * kDK + tid]);
    } else if (tid < kDK + V) {
      t0 = token_in<F32>(p.v, static_cast<size_t>(bh) * V + tid - kDK);
      if (tid == kDK && p.delta) t1 = p.beta[bh];
    }
  };
  auto put_k = [&](int buf) {                  // read before the first barrier of a step (k: up to the second)
    if (tid < kDK) {
      ks[buf][tid] = t0;
      as[tid] = t2;
    }
  };
  auto put_qv = [&]() {                        // read between the barriers
    if (tid < kDK) qs[tid] = t1;
    else if (tid < kDK + V) vs[tid - kDK] = t0;
    if (tid == kDK) bs = t1;
  };
  const int step = gridDim.x;
  fetch(blockIdx.x);
  token(blockIdx.x);
  put_k(0);
  __syncthreads();
  int it = 0;
  for (int bh = blockIdx.x; bh < p.BH; bh += step, ++it) {
    const int buf = it & 1;
    put_qv();
    token(bh + step);
    float4 col[kRingRows];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int r = 0; r < kRingRows; ++r) col[r] = slots[r * kRingThreads + tid];
    fetch(bh + step);                                  // a slot is its thread's own: free once read
    const float *kh = ks[buf] + warp * kRingRows, *qh = qs + warp * kRingRows, *ah = as + warp * kRingRows;
    float4 ksum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kRingRows; ++r) {
      const float a = ah[r], k = kh[r];
      col[r].x *= a; col[r].y *= a; col[r].z *= a; col[r].w *= a;
      ksum.x += k * col[r].x; ksum.y += k * col[r].y; ksum.z += k * col[r].z; ksum.w += k * col[r].w;
    }
    auto total = [&](const float (*part)[V]) {
      float4 t = *reinterpret_cast<const float4*>(&part[0][4 * lane]);
#pragma unroll
      for (int w = 1; w < kRingWarps; ++w) {
        const float4 y = *reinterpret_cast<const float4*>(&part[w][4 * lane]);
        t.x += y.x; t.y += y.y; t.z += y.z; t.w += y.w;
      }
      return t;
    };
    *reinterpret_cast<float4*>(&kpart[warp][4 * lane]) = ksum;
    __syncthreads();
    put_k(buf ^ 1);
    float4 vn = *reinterpret_cast<const float4*>(&vs[4 * lane]);
    if (p.delta) {
      const float4 t = total(kpart);
      const float be = bs;
      vn.x = be * (vn.x - t.x); vn.y = be * (vn.y - t.y); vn.z = be * (vn.z - t.z); vn.w = be * (vn.w - t.w);
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float4* dst = reinterpret_cast<float4*>(p.state + static_cast<size_t>(bh) * kDK * V) + own;
#pragma unroll
    for (int r = 0; r < kRingRows; ++r) {
      const float k = kh[r], q = qh[r];
      col[r].x += k * vn.x; col[r].y += k * vn.y; col[r].z += k * vn.z; col[r].w += k * vn.w;
      o.x += q * col[r].x; o.y += q * col[r].y; o.z += q * col[r].z; o.w += q * col[r].w;
      dst[r * 32] = col[r];
    }
    *reinterpret_cast<float4*>(&opart[warp][4 * lane]) = o;
    __syncthreads();
    if (warp == 0) {
      const float4 t = total(opart);
      __nv_bfloat162 lo = __floats2bfloat162_rn(t.x, t.y), hi = __floats2bfloat162_rn(t.z, t.w);
      __nv_bfloat162* od = reinterpret_cast<__nv_bfloat162*>(p.o + static_cast<size_t>(bh) * V + 4 * lane);
      od[0] = lo;
      od[1] = hi;
    }
  }
}

// d_v = 64 stays with one CTA per pair: eight of half the size per SM overlap as well (2048 pairs: 26.8 us, ring 27.5).
template <bool F32>
static int launch_decode(const DecodeProblem& p, cudaStream_t st) {
  if (p.V == 64) {
    decode_step_kernel<64, F32><<<p.BH, kSplit * 64, 0, st>>>(p);
  } else {
    const int sms = sm_count();
    if (sms <= 0) return kErrDevice;
    const bool aligned = reinterpret_cast<uintptr_t>(p.state) % 16 == 0 && reinterpret_cast<uintptr_t>(p.o) % 4 == 0;
    if (p.BH >= 4 * sms && aligned) {
      static SmemAttr attr;
      if (attr.set(decode_ring_kernel<F32>, kRingBytes)) return kErrLaunch;
      decode_ring_kernel<F32><<<kRingCtas * sms, kRingThreads, kRingBytes, st>>>(p);
    } else {
      decode_step_kernel<128, F32><<<p.BH, kSplit * 128, 0, st>>>(p);
    }
  }
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

}  // namespace lg

extern "C" int lethe_gdn_decode_step(const LetheGdnDecodeArgs* a, void* stream) {
  using namespace lg;
  if (!a || !a->q || !a->k || !a->v || !a->state || !a->o) return kErrNull;
  if (a->B <= 0 || a->H <= 0 || a->K != kDK || (a->V != 64 && a->V != 128)) return kErrDims;
  if (a->gate != LETHE_GATE_NONE && a->gate != LETHE_GATE_SCALAR && a->gate != LETHE_GATE_CHANNEL) return kErrFlags;
  if (a->gate != LETHE_GATE_NONE && !a->g) return kErrNull;
  if (a->delta && !a->beta) return kErrNull;
  DeviceGuard guard(a->state);
  if (!guard.ok) return kErrDevice;
  DecodeProblem p;
  p.BH = a->B * a->H;
  p.H = a->H;
  p.V = a->V;
  p.gate = a->gate;
  p.delta = a->delta;
  p.scale = a->scale;
  p.q = a->q;
  p.k = a->k;
  p.v = a->v;
  p.g = a->g;
  p.beta = a->beta;
  p.state = a->state;
  p.o = static_cast<__nv_bfloat16*>(a->o);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return a->in_f32 ? launch_decode<true>(p, st) : launch_decode<false>(p, st);
}
