// Stream plans: networks whose edges do not stay on chip.
//
// A cluster of 1, 2 or 4 CTAs owns a run of receivers; each CTA of it holds
// one share of the senders' V_dend whole in shared memory and, every step,
// streams the entries (16-bit index, with per-edge conductances a float more)
// of all the cluster's receivers in that share from L2 or HBM.  An entry
// costs one shared-memory read and about five issued instructions; each lane
// reduces lane-chunks of its own (no shuffles), 32 chunks of like length to a
// group, groups dealt to warps by length when the plan is made.  The owner of
// a receiver adds its partial sums over the cluster (distributed shared
// memory) and runs the cell update.
//
// Per step and CTA: publish V_dend, arrive at the grid barrier; the gate
// units (own voltages only) run while the barrier completes and while the
// last warp's first lane, which waits for it, has the share copied in by bulk
// copies; then coupling, exchange of the partial sums, second half of the
// voltage step.
#include <cstdio>

#include "infoli_kernels.cuh"
#include "infoli_ptx.cuh"
#include "infoli_step.cuh"

namespace infoli {

namespace {

constexpr int kCopyBytes = 32768;  // one bulk copy of a share moves at most this much

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned cluster_ctas() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r));
  return r;
}

// Address in shared::cluster space of `local` (a shared-memory address of this
// CTA) in CTA `peer` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, unsigned peer) {
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(local), "r"(peer));
  return ra;
}
__device__ __forceinline__ float ld_peer(uint32_t a) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_peer2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}

// The entries are read once per step: past L1, and in L2 with a policy that
// keeps the share of the lines that fits (StepArgs::l2_keep; the rest is
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

// Four entries of a lane: -(their terms) into nt (two accumulators: entries
// 0, 2 and 1, 3), in V_dend x kVScale (the exponent is -(dV')^2).
template <bool EDGE_G>
__device__ __forceinline__ void stream_quad(const float* sm, uint2 o, float4 g4, float2 nvc2, float2& nt) {
  const float2 c08 = make_float2(0.8f, 0.8f), c02 = make_float2(0.2f, 0.2f);
  const unsigned i[4] = {o.x & 0xffffu, o.x >> 16, o.y & 0xffffu, o.y >> 16};
  const float2 gg[2] = {make_float2(g4.x, g4.y), make_float2(g4.z, g4.w)};
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 nv = __fadd2_rn(make_float2(sm[i[2 * h]], sm[i[2 * h + 1]]), nvc2);  // -V
    const float2 sq = __fmul2_rn(nv, nv);
    const float2 e = make_float2(ex2_approx(-sq.x), ex2_approx(-sq.y));
    float2 f = __ffma2_rn(c08, e, c02);
    if (EDGE_G) f = __fmul2_rn(gg[h], f);
    nt = __ffma2_rn(f, nv, nt);
  }
}

// Running sum of a lane-chunk, negated.  With KAHAN every block of up to
// eight entries (summed per accumulator first) is added compensated.
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
};

// A warp's groups of lane-chunks, partial sums into `part` (pairs of sum and
// compensation with KAHAN).
template <bool KAHAN, bool EDGE_G>
__device__ __forceinline__ void couple_stream(const StepArgs& a, const CtaWork& w, int warp, int lane, const float* sm,
                                              const float* rows, float* part, uint64_t pol) {
  const int* wt = a.probes + w.pad0 + warp;
  const int g0 = w.group_begin + __ldg(wt), g1 = w.group_begin + __ldg(wt + 1);
  for (int g = g0; g < g1; ++g) {
    const int2 gd = __ldg(a.gdesc + g);  // {first quad row, quads per lane}
    const unsigned ld = (unsigned)__ldg(a.gcol + (size_t)g * 32 + lane);
    const uint4* pe = reinterpret_cast<const uint4*>(a.edges) + (size_t)gd.x * 16 + lane;
    const float4* pg = EDGE_G ? reinterpret_cast<const float4*>(a.edge_g) + (size_t)gd.x * 32 + lane : nullptr;
    const int np = gd.y >> 1;
    const bool odd = gd.y & 1;
    const float4 one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    uint4 c0 = make_uint4(0, 0, 0, 0), c1 = c0;
    float4 ga = one, gb = one;
    uint2 tail = make_uint2(0, 0);
    float4 gt = one;
    if (np > 0) {
      c0 = ld_stream4(pe, pol);
      if (EDGE_G) {
        ga = ld_streamg(pg, pol);
        gb = ld_streamg(pg + 32, pol);
      }
    }
    if (!EDGE_G && np > 1) c1 = ld_stream4(pe + 32, pol);
    if (odd) {
      tail = ld_stream2(reinterpret_cast<const uint2*>(pe - lane + np * 32) + lane, pol);
      if (EDGE_G) gt = ld_streamg(pg + np * 64, pol);
    }
    const float nvc = -rows[ld & 0xffffu];
    const float2 nvc2 = make_float2(nvc, nvc);
    StreamSum<KAHAN> s;
    for (int p = 0; p < np; ++p) {
      const uint4 c = c0;
      const float4 g_a = ga, g_b = gb;
      // the next pair's loads are in flight while this one is computed (two
      // pairs ahead without conductances)
      if (EDGE_G) {
        if (p + 1 < np) {
          c0 = ld_stream4(pe + (p + 1) * 32, pol);
          ga = ld_streamg(pg + (p + 1) * 64, pol);
          gb = ld_streamg(pg + (p + 1) * 64 + 32, pol);
        }
      } else {
        c0 = c1;
        if (p + 2 < np) c1 = ld_stream4(pe + (p + 2) * 32, pol);
      }
      float2 nt = s.start();
      stream_quad<EDGE_G>(sm, make_uint2(c.x, c.y), g_a, nvc2, nt);
      stream_quad<EDGE_G>(sm, make_uint2(c.z, c.w), g_b, nvc2, nt);
      s.add(nt);
    }
    if (odd) {
      float2 nt = s.start();
      stream_quad<EDGE_G>(sm, tail, gt, nvc2, nt);
      s.add(nt);
    }
    const unsigned slot = ld >> 16;
    if (KAHAN) {
      // error-free sum of the two accumulators; its error joins the compensation
      const float a0 = -s.acc.x, a1 = -s.acc.y;
      const float sum = a0 + a1;
      const float bb = sum - a0;
      const float err = (a0 - (sum - bb)) + (a1 - bb);
      reinterpret_cast<float2*>(part)[slot] = make_float2(sum, (s.cmp.x + s.cmp.y) - err);
    } else {
      part[slot] = -(s.acc.x + s.acc.y);
    }
  }
}

// Sum of an owned receiver's partial sums over the cluster's CTAs, in sender
// order (TwoSum per addition with KAHAN, the errors and compensations applied
// once).
template <bool KAHAN>
__device__ __forceinline__ float combine_stream(const int2* slots, int cs, const float* part) {
  const uint32_t base = smem_u32(part);
  float s = 0.0f, e = 0.0f, c = 0.0f;
  for (int k = 0; k < cs; ++k) {
    const int2 sl = __ldg(slots + k);
    const uint32_t pa = cs > 1 ? peer_addr(base, (unsigned)k) : base;
#pragma unroll 4
    for (int q = 0; q < sl.y; ++q) {
      if (KAHAN) {
        const float2 p = cs > 1 ? ld_peer2(pa + 8u * (uint32_t)(sl.x + q)) : reinterpret_cast<const float2*>(part)[sl.x + q];
        const float t = s + p.x;
        const float bp = t - s;
        e += (s - (t - bp)) + (p.x - bp);
        c += p.y;
        s = t;
      } else {
        s += cs > 1 ? ld_peer(pa + 4u * (uint32_t)(sl.x + q)) : part[sl.x + q];
      }
    }
  }
  return KAHAN ? s + (e - c) : s;
}

__device__ __forceinline__ bool stream_wait(const StepArgs& a, uint64_t* bar, unsigned parity, volatile int* s_abort) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*s_abort) return false;
    if (globaltimer_ns() - t0 > a.timeout_ns) {
      atomicCAS(a.err, 0, DEV_ERR_COPY_TIMEOUT);
      return false;
    }
  }
  return true;
}

template <bool KAHAN, bool EDGE_G, bool SPLIT>
__global__ void __launch_bounds__(kStreamThreads, 1) stream_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_abort;
  __shared__ unsigned long long s_prof[4];  // cycles: gate units, wait for the share, coupling, rest
  const StreamLayout L = stream_layout(a.shape);
  const float* sm = reinterpret_cast<const float*>(smem_raw);
  float* part = reinterpret_cast<float*>(smem_raw + L.part);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + L.mbar);
  const int cs = a.shape.cluster, share = a.shape.tile_cap, cap = a.shape.cells_cap;
  float* sV = reinterpret_cast<float*>(smem_raw + L.cells);  // SPLIT: V_dend, V_soma, V_axon, nine currents
  float* sI = sV + 3 * cap;
  double* sCa = reinterpret_cast<double*>(smem_raw + L.gca);
  float* sG = reinterpret_cast<float*>(smem_raw + L.gates);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // A launch whose clusters are not the plan's (a tool that relaunches the
  // kernel without its attributes) would read shared memory of CTAs that are
  // not there: every CTA returns instead.
  if (cluster_ctas() != (unsigned)cs) {
    if (tid == 0) atomicCAS(a.err, 0, DEV_ERR_CONFIG);
    return;
  }
  const CtaWork w = a.cta[blockIdx.x];
  const bool owner = tid < w.n_cells;
  const int cell = w.cell_begin + tid;
  const long long np = a.n_pad;
  // this CTA's share of V_dend: cells [lo, lo + nshare), and with cluster > 1
  // the cluster's rows (copies of whole 16-byte units)
  const int lo = w.pad1 * share;
  const int nshare = lo < a.n_cells ? min(share, (a.n_cells - lo + 3) & ~3) : 0;
  const int row_lo = w.tile_begin & ~3;
  const int nrow = cs > 1 ? ((w.tile_begin + w.n_tiles + 3) & ~3) - row_lo : 0;
  const float* rows = cs > 1 ? sm + share + (w.tile_begin & 3) : sm + w.tile_begin;
  const bool producer = tid == kStreamThreads - 32;
  if (tid == 0) {
    mbar_init(mbar, 1);
    fence_mbar_init();
    s_abort = 0;
  }
  Volts v{};
  Gates g{};
  float my_amp = 0.0f;
  int my_onset = 0, my_off = 0;
  if (owner) {
    const float* st = a.st;
    v.Vd = a.vd[a.step0 & 1][cell];
    v.Vs = st[F_VS * np + cell];
    v.Va = st[F_VA * np + cell];
    if (SPLIT) {
      for (int f = F_Q; f < F_COUNT; ++f) sG[f * cap + tid] = st[f * np + cell];
      sCa[tid] = a.ca[cell];
      sV[tid] = v.Vd;
      sV[cap + tid] = v.Vs;
      sV[2 * cap + tid] = v.Va;
    } else {
      g.q = st[F_Q * np + cell];
      g.r = st[F_R * np + cell];
      g.s = st[F_S * np + cell];
      g.Ca = a.ca[cell];
      g.ICaH = st[F_ICAH * np + cell];
      g.gCaL = st[F_GCAL * np + cell];
      g.k = st[F_K * np + cell];
      g.l = st[F_L * np + cell];
      g.m = st[F_M * np + cell];
      g.h = st[F_H * np + cell];
      g.n = st[F_N * np + cell];
      g.p = st[F_P * np + cell];
      g.xs = st[F_XS * np + cell];
      g.ma = st[F_MA * np + cell];
      g.ha = st[F_HA * np + cell];
      g.xa = st[F_XA * np + cell];
    }
    if (a.stim_kind == STIM_CELL) {
      my_amp = a.cell_amp[cell];
      my_onset = a.cell_onset[cell];
    }
    if (a.cell_step_off) my_off = a.cell_step_off[cell];
    a.vds[a.step0 & 1][cell] = v.Vd * kVScale;
  }
  const VoltCoef vk = volt_coef(a.P);
  const uint64_t pol = l2_policy(a.l2_keep);
  unsigned bar_target = 0;
  int row = 0;
  TraceClock tclock(a.trace_every, a.step0);
  const bool prof = a.prof != nullptr && tid == 0;
  if (prof) s_prof[0] = s_prof[1] = s_prof[2] = s_prof[3] = 0;
  __syncthreads();
  const uint64_t ns_begin = prof ? globaltimer_ns() : 0;
  const uint64_t cy_begin = prof ? clock64() : 0;
  uint64_t t_prev = cy_begin;
  auto mark = [&](int k) {
    if (!prof) return;
    const uint64_t t = clock64();
    s_prof[k] += t - t_prev;
    t_prev = t;
  };
  for (int st = 0; st < a.n_steps; ++st) {
    const int step = a.step0 + st;
    const bool trace_now = tclock.take();
    // V^step is written (and every thread past a CTA barrier): arrive
    if (tid == 0) {
      __threadfence();
      if ((int)blockIdx.x != a.stall_cta) red_release_gpu_add(a.bar, 1u);
    }
    bar_target += gridDim.x;

    // ---------------- gate units (own voltages only), first half of the voltage step
    VoltHalf vh{};
    if (SPLIT) {
      const int items = ((w.n_cells + 31) >> 5) * kUnits;
      for (int it = warp; it < items; it += kStreamWarps) {
        const int c = (it / kUnits) * 32 + lane;
        const unsigned m = 1u << (it % kUnits);
        if (c < w.n_cells) {
          const Volts u = {sV[c], sV[cap + c], sV[2 * cap + c]};
          Currents cur;
          Gates gs = load_gates(sG, sCa, cap, c, m);
          run_units(a.P, m, u, gs, cur);
          store_gates(sG, sCa, cap, c, m, gs);
          if (m & 0x01u) sI[0 * cap + c] = cur.I_h;
          if (m & 0x02u) {
            sI[1 * cap + c] = cur.I_CaH;
            sI[2 * cap + c] = cur.I_K_Ca;
          }
          if (m & 0x04u) sI[3 * cap + c] = cur.I_CaL;
          if (m & 0x08u) sI[4 * cap + c] = cur.I_Na_s;
          if (m & 0x10u) sI[5 * cap + c] = cur.I_Kdr_s;
          if (m & 0x20u) sI[6 * cap + c] = cur.I_K_s;
          if (m & 0x40u) sI[7 * cap + c] = cur.I_Na_a;
          if (m & 0x80u) sI[8 * cap + c] = cur.I_K_a;
        }
      }
    } else if (owner) {
      Currents cur;
      run_units(a.P, 0xffu, v, g, cur);
      vh = voltage_first(a.P, vk, v, cur);
    }

    mark(0);
    // ---------------- the share of V^step into shared memory
    if (producer) {
      bool ok = true;
      if (ld_acquire_gpu(a.bar) < bar_target) {
        const uint64_t t0 = globaltimer_ns();
        while (ld_acquire_gpu(a.bar) < bar_target) {
          if (ld_relaxed_gpu(a.err) != 0 || globaltimer_ns() - t0 > a.timeout_ns) {
            atomicCAS(a.err, 0, DEV_ERR_BARRIER_TIMEOUT);
            *(volatile int*)&s_abort = 1;
            ok = false;
            break;
          }
        }
      }
      if (ok) {
        fence_proxy_async_global();
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(mbar, (unsigned)(nshare + nrow) * 4u);
        const float* src = a.vds[step & 1];
        for (int o = 0; o < nshare * 4; o += kCopyBytes)
          bulk_g2s(smem_raw + o, reinterpret_cast<const unsigned char*>(src + lo) + o,
                   (unsigned)min(kCopyBytes, nshare * 4 - o), mbar);
        if (nrow) bulk_g2s(smem_raw + L.rows, src + row_lo, (unsigned)nrow * 4u, mbar);
      }
    }
    __syncwarp();

    // ---------------- coupling
    if (!stream_wait(a, mbar, (unsigned)st & 1u, &s_abort)) s_abort = 1;
    mark(1);
    couple_stream<KAHAN, EDGE_G>(a, w, warp, lane, sm, rows, part, pol);
    if (cs > 1)
      cluster_sync_all();  // every CTA's partial sums (and abort flags) are there
    else
      __syncthreads();
    mark(2);

    // ---------------- owners: the receiver's sum, second half of the voltage step
    if (owner) {
      float ic = combine_stream<KAHAN>(a.cell_slots + (size_t)cell * cs, cs, part) * kInvVScale;
      if (!EDGE_G) ic *= a.g_uniform;
      const int ls = step + my_off;
      float iapp;
      if (a.stim_kind == STIM_PULSE)
        iapp = (ls >= a.stim_start && ls < a.stim_end) ? a.stim_amp : 0.0f;
      else if (a.stim_kind == STIM_CELL)
        iapp = (ls >= my_onset && ls < my_onset + a.stim_dur) ? my_amp : 0.0f;
      else
        iapp = a.stim_table[(size_t)st * np + cell];
      if (SPLIT) {
        Currents cur;
        cur.I_h = sI[0 * cap + tid];
        cur.I_CaH = sI[1 * cap + tid];
        cur.I_K_Ca = sI[2 * cap + tid];
        cur.I_CaL = sI[3 * cap + tid];
        cur.I_Na_s = sI[4 * cap + tid];
        cur.I_Kdr_s = sI[5 * cap + tid];
        cur.I_K_s = sI[6 * cap + tid];
        cur.I_Na_a = sI[7 * cap + tid];
        cur.I_K_a = sI[8 * cap + tid];
        vh = voltage_first(a.P, vk, v, cur);
      }
      v.Vd = voltage_second(a.P, vk, v.Vd, vh, ic, iapp);
      v.Vs = vh.Vs;
      v.Va = vh.Va;
      a.vds[(step + 1) & 1][cell] = v.Vd * kVScale;
      if (SPLIT) {
        sV[tid] = v.Vd;
        sV[cap + tid] = v.Vs;
        sV[2 * cap + tid] = v.Va;
      }
      if (trace_now) {
        float* tr = a.trace + (size_t)row * a.trace_nq * np + cell;
        int qi = 0;
        if (a.trace_mask & TRACE_AXON) tr[(qi++) * np] = v.Va;
        if (a.trace_mask & TRACE_SOMA) tr[(qi++) * np] = v.Vs;
        if (a.trace_mask & TRACE_DEND) tr[(qi++) * np] = v.Vd;
      }
    }
    if (trace_now) ++row;
    if (cs > 1 && tid == kStreamThreads - 1) {
      // a CTA that gave up takes its cluster with it (no CTA may leave while
      // another reads its shared memory)
      int ab = 0;
      for (int k = 0; k < cs; ++k) ab |= __float_as_int(ld_peer(peer_addr(smem_u32(&s_abort), (unsigned)k)));
      if (ab) s_abort = 1;
    }
    __syncthreads();
    mark(3);
    if (s_abort) break;
  }
  if (prof) {
    unsigned long long* pr = a.prof + (size_t)blockIdx.x * kProfSlots;
    atomicAdd(pr + PROF_UNITS, s_prof[0]);
    atomicAdd(pr + PROF_STAGE, s_prof[1]);
    atomicAdd(pr + PROF_COUPLE, s_prof[2]);
    atomicAdd(pr + PROF_UPDATE, s_prof[3]);
    atomicAdd(pr + PROF_STEPS, (unsigned long long)a.n_steps);
    atomicAdd(pr + PROF_SPAN_NS, (unsigned long long)(globaltimer_ns() - ns_begin));
    atomicAdd(pr + PROF_SPAN_CYCLES, (unsigned long long)(clock64() - cy_begin));
  }
  if (cs > 1) cluster_sync_all();

  if (owner) {
    float* st = a.st;
    a.vd[(a.step0 + a.n_steps) & 1][cell] = v.Vd;
    st[F_VS * np + cell] = v.Vs;
    st[F_VA * np + cell] = v.Va;
    if (SPLIT) {
      for (int f = F_Q; f < F_COUNT; ++f) st[f * np + cell] = sG[f * cap + tid];
      a.ca[cell] = sCa[tid];
    } else {
      st[F_Q * np + cell] = g.q;
      st[F_R * np + cell] = g.r;
      st[F_S * np + cell] = g.s;
      a.ca[cell] = g.Ca;
      st[F_ICAH * np + cell] = g.ICaH;
      st[F_GCAL * np + cell] = g.gCaL;
      st[F_K * np + cell] = g.k;
      st[F_L * np + cell] = g.l;
      st[F_M * np + cell] = g.m;
      st[F_H * np + cell] = g.h;
      st[F_N * np + cell] = g.n;
      st[F_P * np + cell] = g.p;
      st[F_XS * np + cell] = g.xs;
      st[F_MA * np + cell] = g.ma;
      st[F_HA * np + cell] = g.ha;
      st[F_XA * np + cell] = g.xa;
    }
  }
}

const void* stream_fn(bool kahan, bool edge_g, bool split) {
#define INFOLI_STREAM_FN(K, G) \
  (split ? (const void*)stream_kernel<K, G, true> : (const void*)stream_kernel<K, G, false>)
  if (kahan) return edge_g ? INFOLI_STREAM_FN(true, true) : INFOLI_STREAM_FN(true, false);
  return edge_g ? INFOLI_STREAM_FN(false, true) : INFOLI_STREAM_FN(false, false);
#undef INFOLI_STREAM_FN
}

void stream_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int grid, int cluster, size_t smem,
                   cudaStream_t stream) {
  cfg = cudaLaunchConfig_t{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kStreamThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
}

}  // namespace

cudaError_t launch_stream_kernel(const StepArgs& a, int grid, cudaStream_t stream) {
  const size_t smem = stream_layout(a.shape).total;
  const void* fn = stream_fn(a.shape.kahan != 0, a.edge_g != nullptr, a.shape.split_units != 0);
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  stream_config(cfg, at, grid, a.shape.cluster, smem, stream);
  void* args[] = {const_cast<StepArgs*>(&a)};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

int max_stream_ctas(int cluster, size_t smem) {
  const void* fn = stream_fn(true, true, false);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  stream_config(cfg, at, cluster, cluster, smem, nullptr);
  cudaLaunchAttribute only = at[1];
  cfg.attrs = &only;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n * cluster;
}

}  // namespace infoli
