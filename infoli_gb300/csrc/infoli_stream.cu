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
#include "infoli_list.cuh"
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
__device__ __forceinline__ void st_peer(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// A warp's groups of lane-chunks, partial sums into `part`, in blocks of N
// entries per lane, then what is left of a group: with N = 16 up to a pair of
// quads, and a quad.  The next block's entries are loaded before this one's
// arithmetic, across groups too, and the first group's before `wait` (the wait
// for V_dend): no load latency stands between blocks.
template <bool KAHAN, bool EDGE_G, bool PLAIN, bool BYTE, int N, class Wait>
__device__ __forceinline__ void couple_stream(const StepArgs& a, const CtaWork& w, int warp, int lane, const float* sm,
                                              const float* rows, float* part, uint64_t pol, Wait wait) {
  const int* wt = a.probes + w.pad0 + warp;
  const int g0 = w.group_begin + __ldg(wt), g1 = w.group_begin + __ldg(wt + 1);
  const uint4* ent = reinterpret_cast<const uint4*>(a.edges) + lane;
  const float4* eg = EDGE_G ? reinterpret_cast<const float4*>(a.edge_g) + lane : nullptr;
  uint4 c[N / 8];
  float4 gc[EDGE_G ? N / 4 : 1];
  auto load_c = [&](int quad_row) {
#pragma unroll
    for (int i = 0; i < N / 8; ++i) c[i] = ld_stream4(ent + (size_t)quad_row * 16 + i * 32, pol);
  };
  auto load_g = [&](int quad_row, float4* d) {
#pragma unroll
    for (int i = 0; i < N / 4; ++i) d[i] = ld_streamg(eg + (size_t)(quad_row + i) * 32, pol);
  };
  int2 gd = make_int2(0, 0);  // {first quad row, quads per lane}
  unsigned ld = 0;
  if (g0 < g1) {
    gd = __ldg(a.gdesc + g0);
    ld = (unsigned)__ldg(a.gcol + (size_t)g0 * 32 + lane);
    if (gd.y >= N / 4) {
      load_c(gd.x);
      if (EDGE_G) load_g(gd.x, gc);
    }
  }
  wait();
  for (int g = g0; g < g1; ++g) {
    int2 gn = make_int2(0, 0);
    unsigned ln = 0;
    if (g + 1 < g1) {
      gn = __ldg(a.gdesc + g + 1);
      ln = (unsigned)__ldg(a.gcol + (size_t)(g + 1) * 32 + lane);
    }
    const int end = gd.x + gd.y / (N / 4) * (N / 4);
    const bool pair = N == 16 && (gd.y & 2), odd = gd.y & 1;
    uint4 left_pair = make_uint4(0, 0, 0, 0);
    uint2 left_quad = make_uint2(0, 0);
    float4 gt = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    const float nvc = -rows[ld & 0xffffu];
    const float2 nvc2 = make_float2(nvc, nvc);
    StreamSum<KAHAN> s;
    auto next_group = [&]() {  // what follows this group's whole blocks
      if (pair) left_pair = ld_stream4(ent + (size_t)end * 16, pol);
      if (odd) {
        const int q = end + (pair ? 2 : 0);
        left_quad = ld_stream2(reinterpret_cast<const uint2*>(ent - lane + (size_t)q * 16) + lane, pol);
        if (EDGE_G) gt = ld_streamg(eg + (size_t)q * 32, pol);
      }
      if (gn.y >= N / 4) load_c(gn.x);
    };
    if (end == gd.x) {
      next_group();
      if (EDGE_G && gn.y >= N / 4) load_g(gn.x, gc);
    }
    for (int q = gd.x; q < end; q += N / 4) {
      float2 x[N / 2];
      stream_gather<N, BYTE>(sm, c, x);
      const bool more = q + N / 4 < end;
      const int nq = more ? q + N / 4 : gn.y >= N / 4 ? gn.x : -1;
      if (more)
        load_c(q + N / 4);
      else
        next_group();
      float2 nt = s.start();
      if (EDGE_G) {
        float4 now[N / 4];
#pragma unroll
        for (int i = 0; i < N / 4; ++i) now[i] = gc[i];
        if (nq >= 0) load_g(nq, gc);
        stream_terms<N, EDGE_G, PLAIN>(x, now, nvc2, nt);
      } else {
        stream_terms<N, EDGE_G, PLAIN>(x, gc, nvc2, nt);
      }
      s.add(nt);
    }
    if (pair) {
      float2 x[4], nt = s.start();
      stream_gather<8, BYTE>(sm, &left_pair, x);
      stream_terms<8, false, PLAIN>(x, &gt, nvc2, nt);
      s.add(nt);
    }
    if (odd) {
      float2 x[2], nt = s.start();
      const uint4 o = make_uint4(left_quad.x, left_quad.y, 0u, 0u);
      stream_gather<4, BYTE>(sm, &o, x);
      stream_terms<4, EDGE_G, PLAIN>(x, &gt, nvc2, nt);
      s.add(nt);
    }
    part[ld >> 16] = s.total();
    gd = gn;
    ld = ln;
  }
}

// Sum of a receiver's partial sums by `width` lanes (`sub`: this lane's place;
// with width > 1 all lanes of the warp call it), in a fixed order, with KAHAN
// an error-free sum per addition whose errors are applied once.  Valid in the
// lanes with sub == 0.
template <bool KAHAN>
__device__ __forceinline__ float sum_slots(uint32_t slots, const float* part, int sub, int width) {
  const int first = slots & 0xffffu, count = slots >> 16;
  float s = 0.0f, e = 0.0f;
  auto add = [&](float x) {
    const float t = s + x;
    if (KAHAN) {
      const float bp = t - s;
      e += (s - (t - bp)) + (x - bp);
    }
    s = t;
  };
#pragma unroll 4
  for (int q = sub; q < count; q += width) add(part[first + q]);
  for (int o = 1; o < width; o <<= 1) {
    const float s2 = __shfl_down_sync(0xffffffffu, s, o);
    const float e2 = KAHAN ? __shfl_down_sync(0xffffffffu, e, o) : 0.0f;
    add(s2);
    e += e2;
  }
  return KAHAN ? s + e : s;
}

__device__ __forceinline__ bool stream_wait(const StepArgs& a, uint64_t* bar, unsigned parity, volatile int* s_abort) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (*s_abort) return false;
    if (globaltimer_ns() - t0 > a.timeout_ns) {
      device_error(a, DEV_ERR_COPY_TIMEOUT);
      return false;
    }
  }
  return true;
}

template <bool KAHAN, bool EDGE_G, bool PLAIN, bool BYTE, int N>
__global__ void __launch_bounds__(kStreamThreads, 1) stream_kernel(const __grid_constant__ StepArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr float kScale = PLAIN ? 1.0f : kVScale, kBack = PLAIN ? 1.0f : kInvVScale;
  // A wait of the step gave up, for even and odd steps: past a step's last
  // barrier its flag stays as it is until every warp has read it, while the
  // producer may already set the next step's (a warp that read that one would
  // leave a step before the others, which wait for it without a limit).
  __shared__ int s_abort[2];
  __shared__ int s_copied;  // steps of the launch whose copies have been issued
  __shared__ float s_peer[kStreamMaxCluster];  // set by a CTA of the cluster that gave up
  __shared__ unsigned long long s_prof[4];  // cycles: gate units, wait for the share, coupling, rest
  const StreamLayout L = stream_layout(a.shape);
  const float* sm = reinterpret_cast<const float*>(smem_raw);
  float* part = reinterpret_cast<float*>(smem_raw + L.part);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(smem_raw + L.mbar);
  float* sums = reinterpret_cast<float*>(smem_raw + L.sums);
  uint32_t* s_slots = reinterpret_cast<uint32_t*>(smem_raw + L.slots);
  float* s_app = reinterpret_cast<float*>(smem_raw + L.app);
  const int cs = a.shape.cluster, share = a.shape.tile_cap, cap = a.shape.cells_cap;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // A launch whose clusters are not the plan's (a tool that relaunches the
  // kernel without its attributes) would read shared memory of CTAs that are
  // not there: every CTA returns instead.
  if (cluster_ctas() != (unsigned)cs) {
    if (tid == 0) device_error(a, DEV_ERR_CONFIG);
    return;
  }
  const CtaWork w = a.cta[blockIdx.x];
  const bool owner = tid < w.n_cells;  // one thread per owned cell
  const int cell = w.cell_begin + tid;
  // Lanes that add a receiver's partial sums: one, or with few cells of many
  // slots each (dense rows) as many as the CTA has for each of its cells, up
  // to 8; the sums then go through shared memory to the owners.
  int wlog = 0;
  if (cs == 1 && w.n_slots > 4 * w.n_cells)
    while (wlog < 3 && (2 * w.n_cells << wlog) <= kStreamThreads) ++wlog;
  const int width = 1 << wlog;
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
    s_abort[0] = s_abort[1] = s_copied = 0;
    for (int k = 0; k < kStreamMaxCluster; ++k) s_peer[k] = 0.0f;
  }
  const int row0 = cs == 1 ? w.cell_begin : w.tile_begin, nrows = cs == 1 ? w.n_cells : w.n_tiles;
  for (int q = tid; q < nrows; q += kStreamThreads) {
    const int2 s = __ldg(a.cell_slots + (size_t)(row0 + q) * cs + w.pad1);
    s_slots[q] = (uint32_t)s.x | (uint32_t)s.y << 16;
  }
  Volts v{};
  if (owner) {
    const float* st = a.st;
    v.Vd = a.vd[a.step0 & 1][cell];
    v.Vs = st[F_VS * np + cell];
    v.Va = st[F_VA * np + cell];
    a.vds[a.step0 & 1][cell] = v.Vd * kScale;
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
  for (int st_i = 0; st_i < a.n_steps; ++st_i) {
    const int step = a.step0 + st_i;
    int* const gave_up = s_abort + (st_i & 1);
    const bool trace_now = tclock.take();
    // V^step is written and every thread past a CTA barrier: arrive (the
    // release covers the CTA's writes)
    if (producer && (int)blockIdx.x != a.stall_cta) red_release_gpu_add(a.bar, 1u);
    bar_target += gridDim.x;

    // ---------------- gate units (own voltages only), first half of the voltage step
    VoltHalf vh{};
    if (owner) {
      // The gate state stays in global memory (L2) between steps, so that the
      // coupling has the registers; its loads and stores, like the units, run
      // while the barrier and the copy complete.  (In registers: 15.9 against
      // 12.9 us per step at 100,000 cells, with spills and no room for loads
      // in flight; in shared memory with the units spread over all warps: 4.7
      // against 3.5 us at 10,000 cells x 40 senders, through two more waits
      // inside the CTA.)
      float* st = a.st + cell;
      Gates g;
      g.q = st[F_Q * np];
      g.r = st[F_R * np];
      g.s = st[F_S * np];
      g.Ca = a.ca[cell];
      g.ICaH = st[F_ICAH * np];
      g.gCaL = st[F_GCAL * np];
      g.k = st[F_K * np];
      g.l = st[F_L * np];
      g.h = st[F_H * np];
      g.n = st[F_N * np];
      g.p = st[F_P * np];
      g.xs = st[F_XS * np];
      g.ha = st[F_HA * np];
      g.xa = st[F_XA * np];
      float iapp;
      if (a.stim_kind == STIM_PULSE) {
        iapp = (step >= a.stim_start && step < a.stim_end) ? a.stim_amp : 0.0f;
      } else if (a.stim_kind == STIM_CELL) {
        const int onset = __ldg(a.cell_onset + cell);
        iapp = (step >= onset && step < onset + a.stim_dur) ? __ldg(a.cell_amp + cell) : 0.0f;
      } else {
        iapp = a.stim_table[(size_t)st_i * np + cell];
      }
      s_app[tid] = iapp;
      Currents cur;
      run_units(a.P, v, g, cur);
      st[F_Q * np] = g.q;
      st[F_R * np] = g.r;
      st[F_S * np] = g.s;
      a.ca[cell] = g.Ca;
      st[F_ICAH * np] = g.ICaH;
      st[F_K * np] = g.k;
      st[F_L * np] = g.l;
      st[F_H * np] = g.h;
      st[F_N * np] = g.n;
      st[F_P * np] = g.p;
      st[F_XS * np] = g.xs;
      st[F_HA * np] = g.ha;
      st[F_XA * np] = g.xa;
      if (st_i + 1 == a.n_steps) {  // m and m_a follow from the voltages alone
        st[F_M * np] = g.m;
        st[F_MA * np] = g.ma;
      }
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
            device_error(a, DEV_ERR_BARRIER_TIMEOUT);
            *(volatile int*)gave_up = 1;
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
        s_copied = st_i + 1;
      }
    }
    __syncwarp();

    // ---------------- coupling
    couple_stream<KAHAN, EDGE_G, PLAIN, BYTE, N>(a, w, warp, lane, sm, rows, part, pol, [&]() {
      if (!stream_wait(a, mbar, (unsigned)st_i & 1u, gave_up)) *gave_up = 1;
      mark(1);
    });
    const int per = cs > 1 ? (w.n_tiles + cs - 1) / cs : 0;  // rows of a CTA of the cluster
    const int sr = tid >> wlog;  // the receiver that this thread adds slots of
    const uint32_t slots = sr < nrows ? s_slots[sr] : 0u;
    __syncthreads();
    if (cs > 1) {
      // every row's sum over this share goes to its owner's CTA (a store: a
      // remote load would stand in the update's way)
      for (int q = tid; q < w.n_tiles; q += kStreamThreads) {
        const float s = sum_slots<KAHAN>(s_slots[q], part, 0, 1);
        const int k = (q >= per) + (q >= 2 * per) + (q >= 3 * per);
        st_peer(peer_addr(smem_u32(sums + w.pad1 * cap + (q - k * per)), (unsigned)k), s);
      }
      if (*gave_up && tid < cs) st_peer(peer_addr(smem_u32(s_peer + w.pad1), (unsigned)tid), 1.0f);
      cluster_sync_all();
    }
    mark(2);

    // ---------------- owners: the receiver's sum, second half of the voltage step
    float ic = 0.0f;
    if (width > 1) {
      const float s = sum_slots<KAHAN>(slots, part, (tid & (width - 1)), width);
      if (sr < w.n_cells && (tid & (width - 1)) == 0) sums[sr] = s;
      __syncthreads();
      if (owner) ic = sums[tid];
    } else if (cs == 1) {
      if (owner) ic = sum_slots<KAHAN>(slots, part, 0, 1);
    } else if (owner) {
      for (int k = 0; k < cs; ++k) ic += sums[k * cap + tid];
    }
    if (owner) {
      ic *= kBack;
      if (!EDGE_G) ic *= a.g_uniform;
      v.Vd = voltage_second(a.P, vk, v.Vd, vh, ic, s_app[tid]);
      v.Vs = vh.Vs;
      v.Va = vh.Va;
      a.vds[(step + 1) & 1][cell] = v.Vd * kScale;
      if (trace_now) {
        float* tr = a.trace + (size_t)row * a.trace_nq * np + cell;
        int qi = 0;
        if (a.trace_mask & TRACE_AXON) tr[(qi++) * np] = v.Va;
        if (a.trace_mask & TRACE_SOMA) tr[(qi++) * np] = v.Vs;
        if (a.trace_mask & TRACE_DEND) tr[(qi++) * np] = v.Vd;
      }
    }
    if (trace_now) ++row;
    // a CTA that gave up takes its cluster with it (no CTA may leave while
    // another writes to its shared memory)
    if (cs > 1 && tid < cs && s_peer[tid] != 0.0f) *gave_up = 1;
    __syncthreads();
    mark(3);
    if (*gave_up) break;
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
  // The other warps' waits may run out just as the grid barrier completes: the
  // copies issued then still land in this CTA's shared memory before it leaves.
  if (producer && s_copied > 0) {
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(mbar, (unsigned)(s_copied - 1) & 1u) && globaltimer_ns() - t0 <= a.timeout_ns) {
    }
  }
  __syncwarp();
  if (cs > 1) cluster_sync_all();

  if (owner) {
    float* st = a.st;
    a.vd[(a.step0 + a.n_steps) & 1][cell] = v.Vd;
    st[F_VS * np + cell] = v.Vs;
    st[F_VA * np + cell] = v.Va;
  }
}

template <bool G, bool P, int N>
const void* stream_fn2(bool kahan, bool byte_off) {
  if (kahan) return byte_off ? (const void*)stream_kernel<true, G, P, true, N> : (const void*)stream_kernel<true, G, P, false, N>;
  return byte_off ? (const void*)stream_kernel<false, G, P, true, N> : (const void*)stream_kernel<false, G, P, false, N>;
}

const void* stream_fn(const SmemShape& s, bool edge_g) {
  const bool k = s.kahan != 0, b = s.byte_off != 0;
  if (edge_g) return stream_fn2<true, true, 8>(k, b);
  if (s.block == 8) return s.plain ? stream_fn2<false, true, 8>(k, b) : stream_fn2<false, false, 8>(k, b);
  return s.plain ? stream_fn2<false, true, 16>(k, b) : stream_fn2<false, false, 16>(k, b);
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
  const void* fn = stream_fn(a.shape, a.edge_g != nullptr);
  cudaError_t e = allow_shared_memory((const void*)fn);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  stream_config(cfg, at, grid, a.shape.cluster, smem, stream);
  void* args[] = {const_cast<StepArgs*>(&a)};
  return cudaLaunchKernelExC(&cfg, fn, args);
}

int max_stream_ctas(int cluster, size_t smem) {
  const void* fn = stream_fn2<true, true, 8>(true, false);
  if (allow_shared_memory((const void*)fn) != cudaSuccess) return 0;
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
