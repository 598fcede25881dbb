// Gates of the six-input surface (reference gdn_layer.py:99-111), where g, b and w come per channel even when a model
// has one decay and one beta per token-head: the test that finds this out and compacts them, and the way back.  Both
// are element-wise and bound by HBM: one pass over the gates each.
#include <cuda_bf16.h>

#include <algorithm>

#include "../../include/lethe_gdn.h"
#include "host_util.h"

namespace lg {

constexpr int kGateThreads = 256;
constexpr int kGateRowsPerWarp = 4;     // rows a warp requests before it looks at the first: 5 KB in flight per warp

struct RegimeProblem {
  const float *g, *b, *w;
  float *g0, *b0;
  long long rows;
  uint32_t *flags, *work;      // work[0]: tests that have failed somewhere; work[1]: CTAs that are done
};

// A warp takes kGateRowsPerWarp rows at a time (K = 128: one float4 per lane and row), grid-stride.  Three tests can
// fail; once all three have, nothing more has to be read, which is what a call with independent gates sees at its
// first rows.  The last CTA publishes the verdict: `flags` may be a mapped host word that the caller polls, which
// costs the call no copy and no synchronisation with whatever else the stream holds.
template <int V>
__global__ void __launch_bounds__(kGateThreads)
gate_regime_kernel(const RegimeProblem p) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (kGateThreads / 32);
  const long long first = static_cast<long long>(blockIdx.x) * (kGateThreads / 32) + (threadIdx.x >> 5);
  constexpr int R = kGateRowsPerWarp;
  constexpr int WV = V / 32;
  uint32_t bad = 0;
  // what a row's values rule out
  auto rules_out = [&](const float4& g, const float4& b, const float* w, float gf, float bf) {
    const bool g_one = g.x == gf && g.y == gf && g.z == gf && g.w == gf;
    bool one = b.x == bf && b.y == bf && b.z == bf && b.w == bf;
    bool none = b.x == 0.f && b.y == 0.f && b.z == 0.f && b.w == 0.f;
#pragma unroll
    for (int e = 0; e < WV; ++e) {
      one = one && w[e] == bf;
      none = none && w[e] == 1.f;
    }
    return (g_one ? 0u : LETHE_REGIME_SCALAR_GATE) | (one ? 0u : LETHE_REGIME_ONE_BETA) | (none ? 0u : LETHE_REGIME_NO_DELTA);
  };
  auto load_w = [&](long long r, float* w) {
    if (WV == 4) *reinterpret_cast<float4*>(w) = reinterpret_cast<const float4*>(p.w + r * V)[lane];
    else *reinterpret_cast<float2*>(w) = reinterpret_cast<const float2*>(p.w + r * V)[lane];
  };
  // Many rows: one of each warp first.  Independent gates show there, and the first batch of all warps, 29 MB, is not read (32768 rows, the call
  // that waits for it: 20.2 / 16.1 us; gates of one value per row take as long as before).
  if (p.rows >= R * warps) {
    const long long r = first * R;
    const float4 g = reinterpret_cast<const float4*>(p.g + r * 128)[lane], b = reinterpret_cast<const float4*>(p.b + r * 128)[lane];
    float w[WV];
    load_w(r, w);
    bad = __reduce_or_sync(0xffffffffu, rules_out(g, b, w, __shfl_sync(0xffffffffu, g.x, 0), __shfl_sync(0xffffffffu, b.x, 0)));
  }
  for (long long r0 = first * R; r0 < p.rows && bad != 7u; r0 += warps * R) {
    float4 g[R], b[R];
    float w[R][WV];
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const long long r = min(r0 + u, p.rows - 1);
      g[u] = reinterpret_cast<const float4*>(p.g + r * 128)[lane];
      b[u] = reinterpret_cast<const float4*>(p.b + r * 128)[lane];
      load_w(r, w[u]);
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const float gf = __shfl_sync(0xffffffffu, g[u].x, 0), bf = __shfl_sync(0xffffffffu, b[u].x, 0);
      bad |= rules_out(g[u], b[u], w[u], gf, bf);
      if (lane == 0 && r0 + u < p.rows) {
        p.g0[r0 + u] = gf;
        p.b0[r0 + u] = bf;
      }
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (*reinterpret_cast<volatile uint32_t*>(p.work) == 7u) break;
  }
  __shared__ uint32_t cta_bad;
  if (threadIdx.x == 0) cta_bad = 0;
  __syncthreads();
  if (lane == 0 && bad) atomicOr(&cta_bad, bad);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (cta_bad) atomicOr(p.work, cta_bad);
    __threadfence();
    if (atomicAdd(p.work + 1, 1u) == gridDim.x - 1) {
      const uint32_t failed = atomicExch(p.work, 0u);
      p.work[1] = 0u;
      // Whoever sees the word may hand `work` to a kernel on another stream at once, which nothing but this fence orders
      // behind the two stores that clear it.
      __threadfence_system();
      *reinterpret_cast<volatile uint32_t*>(p.flags) = LETHE_REGIME_DONE | (~failed & 7u);
    }
  }
}

struct SpreadProblem {
  const float *dg0, *db0, *dw0;
  float *dg, *db, *dw;
  long long rows;
};

// One warp per row and pass: three coalesced row stores.
template <int V>
__global__ void __launch_bounds__(kGateThreads)
gate_spread_kernel(const SpreadProblem p) {
  const int lane = threadIdx.x & 31;
  const long long warps = static_cast<long long>(gridDim.x) * (kGateThreads / 32);
  for (long long r = static_cast<long long>(blockIdx.x) * (kGateThreads / 32) + (threadIdx.x >> 5); r < p.rows; r += warps) {
    if (p.dg) {
      const float x = p.dg0 ? p.dg0[r] * (1.f / 128) : 0.f;
      reinterpret_cast<float4*>(p.dg + r * 128)[lane] = make_float4(x, x, x, x);
    }
    if (p.db) {
      const float x = p.db0 ? p.db0[r] * (1.f / 128) : 0.f;
      reinterpret_cast<float4*>(p.db + r * 128)[lane] = make_float4(x, x, x, x);
    }
    if (p.dw) {
      const float x = p.dw0 ? p.dw0[r] * (1.f / V) : 0.f;
      if (V == 128) reinterpret_cast<float4*>(p.dw + r * V)[lane] = make_float4(x, x, x, x);
      else reinterpret_cast<float2*>(p.dw + r * V)[lane] = make_float2(x, x);
    }
  }
}

// bf16 to fp32 or back, 8 values a thread
template <bool TO_F32>
__global__ void __launch_bounds__(kGateThreads)
convert_kernel(const void* __restrict__ src, void* __restrict__ dst, long long n) {
  const long long i = (static_cast<long long>(blockIdx.x) * kGateThreads + threadIdx.x) * 8;
  if (i >= n) return;
  const __nv_bfloat16* s16 = static_cast<const __nv_bfloat16*>(src);
  const float* s32 = static_cast<const float*>(src);
  __nv_bfloat16* d16 = static_cast<__nv_bfloat16*>(dst);
  float* d32 = static_cast<float*>(dst);
  if (i + 8 > n) {
    for (long long j = i; j < n; ++j) {
      if (TO_F32) d32[j] = __bfloat162float(s16[j]);
      else d16[j] = __float2bfloat16_rn(s32[j]);
    }
    return;
  }
  if (TO_F32) {
    const uint4 u = *reinterpret_cast<const uint4*>(s16 + i);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
    float4 o[2];
    float* f = reinterpret_cast<float*>(o);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      f[2 * j] = __uint_as_float(w[j] << 16);
      f[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
    reinterpret_cast<float4*>(d32 + i)[0] = o[0];
    reinterpret_cast<float4*>(d32 + i)[1] = o[1];
  } else {
    const float4 a = reinterpret_cast<const float4*>(s32 + i)[0], b = reinterpret_cast<const float4*>(s32 + i)[1];
    const __nv_bfloat162 h[4] = {__floats2bfloat162_rn(a.x, a.y), __floats2bfloat162_rn(a.z, a.w), __floats2bfloat162_rn(b.x, b.y),
                                 __floats2bfloat162_rn(b.z, b.w)};
    *reinterpret_cast<uint4*>(d16 + i) = *reinterpret_cast<const uint4*>(h);
  }
}

static bool gates_aligned(const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }

}  // namespace lg

extern "C" int lethe_gdn_gate_regime(const float* g, const float* b, const float* w, int64_t rows, int32_t K, int32_t V,
                                     float* g0, float* b0, uint32_t* flags, uint32_t* work, void* stream) {
  using namespace lg;
  if (!g || !b || !w || !g0 || !b0 || !flags || !work) return kErrNull;
  if (rows <= 0 || K != 128 || (V != 64 && V != 128)) return kErrDims;
  if (!gates_aligned(g) || !gates_aligned(b) || !gates_aligned(w)) return kErrAlign;
  DeviceGuard guard(g);
  const int sms = sm_count();
  if (!guard.ok || sms <= 0) return kErrDevice;
  const RegimeProblem p{g, b, w, g0, b0, rows, flags, work};
  const int64_t per_cta = (kGateThreads / 32) * kGateRowsPerWarp;
  // four CTAs per SM: enough bytes in flight for HBM, few enough CTAs to finish in one wave
  const unsigned grid = static_cast<unsigned>(std::min(static_cast<int64_t>(4 * sms), (rows + per_cta - 1) / per_cta));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (V == 64) gate_regime_kernel<64><<<grid, kGateThreads, 0, st>>>(p);
  else gate_regime_kernel<128><<<grid, kGateThreads, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

extern "C" int lethe_gdn_gate_spread(const float* dg0, const float* db0, const float* dw0, int64_t rows, int32_t K, int32_t V,
                                     float* dg, float* db, float* dw, void* stream) {
  using namespace lg;
  if (!dg && !db && !dw) return kErrNull;
  if (rows <= 0 || K != 128 || (V != 64 && V != 128)) return kErrDims;
  if (!gates_aligned(dg) || !gates_aligned(db) || !gates_aligned(dw)) return kErrAlign;
  DeviceGuard guard(dg ? dg : db ? db : dw);
  const int sms = sm_count();
  if (!guard.ok || sms <= 0) return kErrDevice;
  const SpreadProblem p{dg0, db0, dw0, dg, db, dw, rows};
  const unsigned grid = static_cast<unsigned>(std::min(static_cast<int64_t>(8 * sms), (rows + kGateThreads / 32 - 1) / (kGateThreads / 32)));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (V == 64) gate_spread_kernel<64><<<grid, kGateThreads, 0, st>>>(p);
  else gate_spread_kernel<128><<<grid, kGateThreads, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}

extern "C" int lethe_gdn_convert(const void* src, void* dst, int64_t n, int32_t to_f32, void* stream) {
  using namespace lg;
  if (!src || !dst) return kErrNull;
  if (n <= 0) return kErrDims;
  if (!gates_aligned(src) || !gates_aligned(dst)) return kErrAlign;
  DeviceGuard guard(src);
  if (!guard.ok) return kErrDevice;
  const int64_t per_cta = kGateThreads * 8, grid = (n + per_cta - 1) / per_cta;
  if (grid > 0x7fffffff) return kErrDims;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (to_f32) convert_kernel<true><<<static_cast<unsigned>(grid), kGateThreads, 0, st>>>(src, dst, n);
  else convert_kernel<false><<<static_cast<unsigned>(grid), kGateThreads, 0, st>>>(src, dst, n);
  return cudaGetLastError() == cudaSuccess ? kOk : kErrLaunch;
}
