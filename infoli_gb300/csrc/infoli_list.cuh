// Coupling over entry lists: 16-bit entries (the senders' places in shared
// memory) streamed from L2 or HBM, one receiver's piece per lane.  Shared by
// the stream kernel (infoli_stream.cu) and the batched kernel (infoli_batch.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "infoli_ptx.cuh"

namespace infoli {

// Where V_dend x kVScale is held instead of V_dend (kVScale^2 = log2(e) / 100),
// a coupling term's exponent is -(dV')^2 with dV' = kVScale dV, one multiply less
// per edge; the sums are scaled back once per receiver.
constexpr float kVScale = 0.12011224087864497f;
constexpr float kInvVScale = 8.325546111576978f;

// The entries are read once per step: past L1, and in L2 with a policy that
// keeps the share of the lines that fits (`keep`; the rest is
// evicted first, so it does not push out the others).  L1::no_allocate alone
// is treated as streaming by L2 too: 40 MB of entries then hit L2 at 17 %.
__device__ __forceinline__ uint64_t l2_policy(float keep) {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.L2::evict_first.b64 %0, %1;" : "=l"(p) : "f"(keep));
  return p;
}
__device__ __forceinline__ uint4 ld_stream4(const uint4* p, uint64_t pol) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ uint2 ld_stream2(const uint2* p, uint64_t pol) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
               : "=r"(v.x), "=r"(v.y)
               : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float4 ld_streamg(const float4* p, uint64_t pol) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "l"(pol));
  return v;
}

// N entries of a lane (two per word of o): -(their terms) into nt (two
// accumulators: even and odd entries), in V_dend x kVScale (the exponent is
// -(dV')^2), or with PLAIN in V_dend itself (the difference is scaled for the
// exponent alone: an operation more per pair of entries, but no rounding of the
// voltages before their difference is taken).  All gathers first, then the arithmetic in stages: a warp then
// waits once per block and not once per pair of entries (2.03 against 2.7
// cycles of an SM per warp and entry in a loop over shared memory without bank
// conflicts; the SFU and the FMA pipe take about one each).
template <int N, bool BYTE>
__device__ __forceinline__ void stream_gather(const float* sm, const uint4* o, float2* x) {
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const unsigned w = k % 4 == 0 ? o[k / 4].x : k % 4 == 1 ? o[k / 4].y : k % 4 == 2 ? o[k / 4].z : o[k / 4].w;
    if (BYTE) {
      const unsigned char* b = reinterpret_cast<const unsigned char*>(sm);
      x[k] = make_float2(*reinterpret_cast<const float*>(b + (w & 0xffffu)), *reinterpret_cast<const float*>(b + (w >> 16)));
    } else {
      x[k] = make_float2(sm[w & 0xffffu], sm[w >> 16]);
    }
  }
}

template <int N, bool EDGE_G, bool PLAIN = false>
__device__ __forceinline__ void stream_terms(float2* x, const float4* g, float2 nvc2, float2& nt) {
  const float2 c08 = make_float2(0.8f, 0.8f), c02 = make_float2(0.2f, 0.2f);
#pragma unroll
  for (int k = 0; k < N / 2; ++k) x[k] = __fadd2_rn(x[k], nvc2);  // -V
  float2 e[N / 2];
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const float2 d = PLAIN ? __fmul2_rn(x[k], make_float2(kVScale, kVScale)) : x[k];
    const float2 sq = __fmul2_rn(d, d);
    e[k] = make_float2(ex2_approx(-sq.x), ex2_approx(-sq.y));
  }
#pragma unroll
  for (int k = 0; k < N / 2; ++k) {
    const float2 f = __ffma2_rn(c08, e[k], c02);
    if (EDGE_G) x[k] = __fmul2_rn(k % 2 ? make_float2(g[k / 2].z, g[k / 2].w) : make_float2(g[k / 2].x, g[k / 2].y), x[k]);
    nt = __ffma2_rn(f, x[k], nt);
  }
}

// Running sum of a lane-chunk, negated.  With KAHAN every block of up to
// sixteen entries (summed per accumulator first) is added compensated.  Finer
// blocks change little: the gap-junction current of 20,000 cells x 100 senders
// is 6.2e-8 of its size from 64 bits this way, 6.1e-8 with every term
// compensated (5.9e-8 where one thread adds a whole row so; 7.1e-8 without),
// and the state after 1,000 steps of 100,000 x 100 the same 9.56e-8, at 3 % more
// time.
template <bool KAHAN>
struct StreamSum {
  float2 acc = make_float2(-0.0f, -0.0f), cmp = make_float2(0.0f, 0.0f);
  __device__ __forceinline__ float2 start() const { return KAHAN ? make_float2(-0.0f, -0.0f) : acc; }
  __device__ __forceinline__ void add(float2 nt) {
    if (!KAHAN) {
      acc = nt;
      return;
    }
    const float2 m1 = make_float2(-1.0f, -1.0f);
    const float2 ny = __fadd2_rn(nt, cmp);
    const float2 ns = __fadd2_rn(acc, ny);
    const float2 dt = __ffma2_rn(acc, m1, ns);
    cmp = __ffma2_rn(dt, m1, ny);
    acc = ns;
  }
  // The sum: with KAHAN the rounding of the last addition and the
  // compensations are applied once.
  __device__ __forceinline__ float total() const {
    const float a0 = -acc.x, a1 = -acc.y;
    float sum = a0 + a1;
    if (KAHAN) {
      const float bb = sum - a0;
      sum += ((a0 - (sum - bb)) + (a1 - bb)) - (cmp.x + cmp.y);
    }
    return sum;
  }
};

}  // namespace infoli
