// Pieces shared by the persistent step kernels: the coupling's constants, the
// gate state in shared memory, the trace countdown.
#pragma once
#include "infoli_kernels.cuh"
#include "infoli_list.cuh"

namespace infoli {

constexpr float kNegLog2eOver100 = -0.014426950408889634f;  // -log2(e)/100

// One gate unit of local cell r on shared-memory state: its gates (field f at
// sG[f * cap + r], Ca2+ in sCa), the compartment's voltage (sV: V_dend, V_soma,
// V_axon, cap apart) in, its currents (current k at sI[k * cap + r]) out.  One
// block of code per unit behind one switch: with loads, arithmetic and stores
// each behind eight tests of a unit mask, a warp went through 32 branches for
// one unit.
__device__ __forceinline__ void unit_step(const ModelParams& P, int u, const float* sV, float* sG, double* sCa,
                                          float* sI, int cap, int r) {
  Volts v{};
  Gates g{};
  Currents c{};
  switch (u) {
    case 0:
      v.Vd = sV[r];
      g.q = sG[F_Q * cap + r];
      unit_q(P, v, g, c);
      sG[F_Q * cap + r] = g.q;
      sI[0 * cap + r] = c.I_h;
      break;
    case 1:
      v.Vd = sV[r];
      g.r = sG[F_R * cap + r];
      g.s = sG[F_S * cap + r];
      g.Ca = sCa[r];
      g.ICaH = sG[F_ICAH * cap + r];
      unit_rs(P, v, g, c);
      sG[F_R * cap + r] = g.r;
      sG[F_S * cap + r] = g.s;
      sCa[r] = g.Ca;
      sG[F_ICAH * cap + r] = g.ICaH;
      sI[1 * cap + r] = c.I_CaH;
      sI[2 * cap + r] = c.I_K_Ca;
      break;
    case 2:
      v.Vs = sV[cap + r];
      g.k = sG[F_K * cap + r];
      g.l = sG[F_L * cap + r];
      g.gCaL = sG[F_GCAL * cap + r];
      unit_kl(P, v, g, c);
      sG[F_K * cap + r] = g.k;
      sG[F_L * cap + r] = g.l;
      sI[3 * cap + r] = c.I_CaL;
      break;
    case 3:
      v.Vs = sV[cap + r];
      g.h = sG[F_H * cap + r];
      unit_mh(P, v, g, c);
      sG[F_M * cap + r] = g.m;
      sG[F_H * cap + r] = g.h;
      sI[4 * cap + r] = c.I_Na_s;
      break;
    case 4:
      v.Vs = sV[cap + r];
      g.n = sG[F_N * cap + r];
      g.p = sG[F_P * cap + r];
      unit_np(P, v, g, c);
      sG[F_N * cap + r] = g.n;
      sG[F_P * cap + r] = g.p;
      sI[5 * cap + r] = c.I_Kdr_s;
      break;
    case 5:
      v.Vs = sV[cap + r];
      g.xs = sG[F_XS * cap + r];
      unit_xs(P, v, g, c);
      sG[F_XS * cap + r] = g.xs;
      sI[6 * cap + r] = c.I_K_s;
      break;
    case 6:
      v.Va = sV[2 * cap + r];
      g.ha = sG[F_HA * cap + r];
      unit_mha(P, v, g, c);
      sG[F_MA * cap + r] = g.ma;
      sG[F_HA * cap + r] = g.ha;
      sI[7 * cap + r] = c.I_Na_a;
      break;
    default:
      v.Va = sV[2 * cap + r];
      g.xa = sG[F_XA * cap + r];
      unit_xa(P, v, g, c);
      sG[F_XA * cap + r] = g.xa;
      sI[8 * cap + r] = c.I_K_a;
      break;
  }
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
