// Pieces shared by the persistent step kernels: the coupling's constants, the
// gate state in shared memory, the trace countdown.
#pragma once
#include "infoli_kernels.cuh"

namespace infoli {

constexpr float kNegLog2eOver100 = -0.014426950408889634f;  // -log2(e)/100
// Stamped plans keep V_dend x kVScale in the window copy and the scaled-V cell
// array (kVScale^2 = log2(e) / 100): a coupling term's exponent is then
// -(dV')^2 with dV' = kVScale dV, one multiply less per edge; the partial sums
// are scaled back once per receiver.
constexpr float kVScale = 0.12011224087864497f;
constexpr float kInvVScale = 8.325546111576978f;

// Gate state of local cell r from / to shared memory (field f at
// sG[f * cap + r]), only the fields the units in `mask` use.
__device__ __forceinline__ Gates load_gates(const float* sG, const double* sCa, int cap, int r, unsigned mask) {
  Gates g;
  if (mask & 0x01u) g.q = sG[F_Q * cap + r];
  if (mask & 0x02u) {
    g.r = sG[F_R * cap + r];
    g.s = sG[F_S * cap + r];
    g.Ca = sCa[r];
    g.ICaH = sG[F_ICAH * cap + r];
  }
  if (mask & 0x04u) {
    g.k = sG[F_K * cap + r];
    g.l = sG[F_L * cap + r];
    g.gCaL = sG[F_GCAL * cap + r];
  }
  if (mask & 0x08u) g.h = sG[F_H * cap + r];
  if (mask & 0x10u) {
    g.n = sG[F_N * cap + r];
    g.p = sG[F_P * cap + r];
  }
  if (mask & 0x20u) g.xs = sG[F_XS * cap + r];
  if (mask & 0x40u) g.ha = sG[F_HA * cap + r];
  if (mask & 0x80u) g.xa = sG[F_XA * cap + r];
  return g;
}

__device__ __forceinline__ void store_gates(float* sG, double* sCa, int cap, int r, unsigned mask, const Gates& g) {
  if (mask & 0x01u) sG[F_Q * cap + r] = g.q;
  if (mask & 0x02u) {
    sG[F_R * cap + r] = g.r;
    sG[F_S * cap + r] = g.s;
    sCa[r] = g.Ca;
    sG[F_ICAH * cap + r] = g.ICaH;
  }
  if (mask & 0x04u) {
    sG[F_K * cap + r] = g.k;
    sG[F_L * cap + r] = g.l;
  }
  if (mask & 0x08u) {
    sG[F_M * cap + r] = g.m;
    sG[F_H * cap + r] = g.h;
  }
  if (mask & 0x10u) {
    sG[F_N * cap + r] = g.n;
    sG[F_P * cap + r] = g.p;
  }
  if (mask & 0x20u) sG[F_XS * cap + r] = g.xs;
  if (mask & 0x40u) {
    sG[F_MA * cap + r] = g.ma;
    sG[F_HA * cap + r] = g.ha;
  }
  if (mask & 0x80u) sG[F_XA * cap + r] = g.xa;
}

// Unit currents of local cell r in shared memory (current k at sI[k * cap + r]).
__device__ __forceinline__ void store_currents(float* sI, int cap, int r, unsigned mask, const Currents& c) {
  if (mask & 0x01u) sI[0 * cap + r] = c.I_h;
  if (mask & 0x02u) {
    sI[1 * cap + r] = c.I_CaH;
    sI[2 * cap + r] = c.I_K_Ca;
  }
  if (mask & 0x04u) sI[3 * cap + r] = c.I_CaL;
  if (mask & 0x08u) sI[4 * cap + r] = c.I_Na_s;
  if (mask & 0x10u) sI[5 * cap + r] = c.I_Kdr_s;
  if (mask & 0x20u) sI[6 * cap + r] = c.I_K_s;
  if (mask & 0x40u) sI[7 * cap + r] = c.I_Na_a;
  if (mask & 0x80u) sI[8 * cap + r] = c.I_K_a;
}

__device__ __forceinline__ Currents load_currents(const float* sI, int cap, int r) {
  Currents c;
  c.I_h = sI[0 * cap + r];
  c.I_CaH = sI[1 * cap + r];
  c.I_K_Ca = sI[2 * cap + r];
  c.I_CaL = sI[3 * cap + r];
  c.I_Na_s = sI[4 * cap + r];
  c.I_Kdr_s = sI[5 * cap + r];
  c.I_K_s = sI[6 * cap + r];
  c.I_Na_a = sI[7 * cap + r];
  c.I_K_a = sI[8 * cap + r];
  return c;
}

// Trace rows fall on the steps that are multiples of trace_every.  A
// countdown per thread replaces a per-step integer division (it sat on the
// voltage threads' path every step).
struct TraceClock {
  int every, left;
  __device__ TraceClock(int every_, int step0)
      : every(every_), left(every_ > 0 ? (every_ - step0 % every_) % every_ : -1) {}
  // true on a trace step; advances to the next step
  __device__ bool take() {
    const bool now = left == 0;
    if (every > 0) left = now ? every - 1 : left - 1;
    return now;
  }
};

}  // namespace infoli
