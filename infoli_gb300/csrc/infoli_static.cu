// Allocation-free entry point: infoli_run_noalloc.
//
// Some callers cannot allocate device memory while they drive the
// simulation: hosts that reserved a fixed device-memory arena at start-up and
// hand the library pieces of it (an allocation outside the arena can fail or
// break the budget), foreign-language bindings whose runtime's allocator owns
// every device buffer (memory taken behind its back escapes its accounting),
// and loops running beside other GPU work that cannot take the device-wide
// synchronisation cudaFree (and often cudaMalloc) implies.  For them this file
// offers one entry point that allocates nothing: the caller passes the
// network, the state and the trace buffer in device memory, and the only
// scratch the kernel needs -- the V_dend double buffer shared between CTAs,
// the grid-barrier counter and the error word -- lives in one file-scope
// static __device__ array of fixed size (kNoAllocMaxCells cells, about 0.5
// MiB), which every GPU that loads the library keeps until the process exits.
//
// The kernel walks the CSR lists as they are (nothing is planned, nothing is
// kept between calls), a group of 4 to 32 lanes per receiver, with V_dend read
// from the shared scratch buffer through L2; the cells are spread over up to
// one CTA per SM, their state in shared memory, the gate units over all warps
// and run while the step's grid barrier completes.  The barrier
// counter is 64-bit, so one call may run any number of steps without it
// wrapping.  Malformed topology (a sender id outside [0, n), a NULL column
// array with edges, a decreasing or negative row_ptr) is recorded in the
// error word and the bad read is skipped, so it never reads outside the
// caller's buffers through a bad index; row_ptr[n] itself cannot be checked
// against the length of the caller's arrays and is the caller's contract.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "../../include/infoli_gpu.h"
#include "infoli_cell.cuh"
#include "infoli_internal.h"
#include "infoli_ptx.cuh"
#include "infoli_step.cuh"

namespace infoli {
namespace {

constexpr int kNoAllocMaxCells = 65536;  // largest network the static scratch holds
constexpr int kNoAllocBlock = 512;
constexpr int kNoAllocWarps = kNoAllocBlock / 32;
// A CTA takes at least a warp's worth of cells (a small network stays on few
// SMs, with a cheaper grid barrier) and at most its threads.
constexpr int kNoAllocMinCells = 32;
constexpr int kNoAllocLoads = 8;  // V_dend loads in flight per lane
constexpr int kMaxDevices = 64;

// Scratch layout: [0, 256) 64-bit barrier counter at 0 + error word at 64
// (zeroed before every launch); [256, ...) V_dend double buffer,
// 2 x kNoAllocMaxCells floats.
constexpr int kErrBarrier = 1, kErrSender = 2, kErrRowPtr = 3;
constexpr size_t kCtlBytes = 256;
constexpr size_t kScratchBytes = kCtlBytes + 2 * sizeof(float) * (size_t)kNoAllocMaxCells;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

struct NoAllocArgs {
  ModelParams P;
  int n, step0, n_steps;
  const int64_t* row_ptr;
  const int32_t* col;
  const float* g;
  float g_uniform;
  int pulse_start, pulse_end;
  float pulse_amp;
  float* state;        // INFOLI_NSTATE x n, reference order (V_dend first)
  float* trace_axon;   // n_steps x n, or null
  unsigned char* scratch;  // device address of g_noalloc_scratch
  unsigned long long timeout_ns;
};

// Shared memory of a CTA of `cap` cells: V_dend, V_soma, V_axon, nine unit
// currents, the gap-junction current, the gate state, Ca2+, the edge ranges.
enum { kNoAllocCellFloats = 13 };
__host__ __device__ inline size_t noalloc_smem(int cap) {
  return (size_t)cap * ((kNoAllocCellFloats + kGateFloats) * sizeof(float) + sizeof(double) + 2 * sizeof(int64_t));
}

// Sum over the edges of one receiver of g f(V) V by `width` lanes (a power of
// two; `sub` is this lane's place among them), in all of them.
__device__ __forceinline__ float noalloc_row(const NoAllocArgs& a, const float* vcur, int64_t e0, int64_t e1, float vc,
                                             int sub, int width, int* err) {
  float acc = 0.0f;
  for (int64_t e = e0 + sub; e < e1; e += (int64_t)kNoAllocLoads * width) {
    int s[kNoAllocLoads];
    float vs[kNoAllocLoads], gg[kNoAllocLoads];
#pragma unroll
    for (int u = 0; u < kNoAllocLoads; ++u) {
      const int64_t k = e + (int64_t)u * width;
      s[u] = k < e1 ? __ldg(a.col + k) : -1;
      gg[u] = a.g && k < e1 ? __ldg(a.g + k) : 1.0f;
      if (k < e1 && (unsigned)s[u] >= (unsigned)a.n) {  // malformed topology: recorded, never read outside the buffer
        atomicCAS(err, 0, kErrSender);
        s[u] = -1;
      }
    }
#pragma unroll
    for (int u = 0; u < kNoAllocLoads; ++u)
      vs[u] = s[u] >= 0 ? __ldcg(vcur + s[u]) : vc;  // L2: written by other CTAs this launch
#pragma unroll
    for (int u = 0; u < kNoAllocLoads; ++u) {
      const float V = vc - vs[u];
      const float f = fmaf(0.8f, ex2_approx((V * V) * kNegLog2eOver100), 0.2f);
      if (s[u] >= 0) acc += (gg[u] * f) * V;
    }
  }
  for (int o = width >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// What bounds a step: the grid barrier and the L2 round trips to the senders'
// V_dend, so a CTA has few cells and every lane eight loads in flight.
// 5,003 cells x 60 senders, per-edge g, 200 steps: 1,030 us per call
// against 5,180 with one thread per cell on 10 CTAs (the edges of a row one
// after another, the gate units after them).
__global__ void __launch_bounds__(kNoAllocBlock, 2) noalloc_step_kernel(const __grid_constant__ NoAllocArgs a,
                                                                         int cells_per_cta, int cap) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int s_abort;
  double* sCa = reinterpret_cast<double*>(smem_raw);
  int64_t* sE0 = reinterpret_cast<int64_t*>(sCa + cap);
  int64_t* sE1 = sE0 + cap;
  float* sV = reinterpret_cast<float*>(sE1 + cap);
  float* sI = sV + 3 * cap;   // nine unit currents
  float* sIc = sI + 9 * cap;  // gap-junction current
  float* sG = sIc + cap;      // gate state, field f of cell c at sG[f * cap + c]
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(a.scratch);
  int* err = reinterpret_cast<int*>(a.scratch + 64);
  float* vd[2] = {reinterpret_cast<float*>(a.scratch + kCtlBytes),
                  reinterpret_cast<float*>(a.scratch + kCtlBytes) + kNoAllocMaxCells};
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = blockIdx.x * cells_per_cta;
  const int nc = min(cells_per_cta, a.n - c0);
  const bool own = tid < nc;
  const size_t N = (size_t)a.n, c = (size_t)c0 + tid;

  // state order of the ABI's arrays, by device field
  const int field[] = {-1, F_R, F_S, F_Q, -2, F_ICAH, F_GCAL, -3, F_M, F_H, F_N, F_P, F_XS, F_K, F_L, -4, F_MA, F_HA, F_XA};
  if (own) {
    const float* s = a.state;
    sV[tid] = s[0 * N + c];
    sV[cap + tid] = s[7 * N + c];
    sV[2 * cap + tid] = s[15 * N + c];
    sCa[tid] = (double)s[4 * N + c];
#pragma unroll
    for (int k = 0; k < INFOLI_NSTATE; ++k)
      if (field[k] >= 0) sG[field[k] * cap + tid] = s[k * N + c];
    vd[a.step0 & 1][c] = sV[tid];
    // this cell's edge range, checked once (a bad row is recorded and skipped)
    int64_t e0 = a.row_ptr[c], e1 = a.row_ptr[c + 1];
    if (e0 < 0 || e1 < e0) {
      atomicCAS(err, 0, kErrRowPtr);
      e1 = e0 = 0;
    } else if (e1 > e0 && a.col == nullptr) {
      atomicCAS(err, 0, kErrSender);
      e1 = e0;
    }
    sE0[tid] = e0;
    sE1[tid] = e1;
  }
  if (tid == 0) s_abort = 0;
  // lanes per receiver: as many as the CTA has for each of its cells, at
  // least 4 (rows then read in 16-byte pieces)
  int width = 4;
  while (width < 32 && width * 2 * nc <= kNoAllocBlock) width *= 2;
  const int groups = kNoAllocBlock / width, sub = tid % width;
  const VoltCoef vk = volt_coef(a.P);
  unsigned long long target = 0;
  __syncthreads();
  for (int t = 0; t < a.n_steps; ++t) {
    const int step = a.step0 + t;
    // V^step is written: arrive, run the gate units (own voltages only), wait
    if (tid == 0) {
      __threadfence();
      red_release_gpu_add_u64(bar, 1ull);
    }
    target += gridDim.x;
    const int items = ((nc + 31) >> 5) * kUnits;
    for (int it = warp; it < items; it += kNoAllocWarps) {
      const int k = (it / kUnits) * 32 + lane;
      if (k < nc) unit_step(a.P, it % kUnits, sV, sG, sCa, sI, cap, k);
    }
    if (tid == kNoAllocBlock - 32) {
      const uint64_t t0 = globaltimer_ns();
      while (ld_acquire_gpu_u64(bar) < target) {
        if (ld_relaxed_gpu(err) != 0 || globaltimer_ns() - t0 > a.timeout_ns) {
          atomicCAS(err, 0, kErrBarrier);
          s_abort = 1;
          break;
        }
      }
    }
    __syncthreads();
    if (s_abort) break;
    const float* vcur = vd[step & 1];
    for (int k0 = 0; k0 < nc; k0 += groups) {  // whole warps, with or without a receiver
      const int k = k0 + tid / width;
      const bool row = k < nc;
      const float sum = noalloc_row(a, vcur, row ? sE0[k] : 0, row ? sE1[k] : 0, row ? sV[k] : 0.0f, sub, width, err);
      if (row && sub == 0) sIc[k] = sum;
    }
    __syncthreads();
    if (own) {
      const float ic = a.g ? sIc[tid] : sIc[tid] * a.g_uniform;
      const float iapp = (step >= a.pulse_start && step < a.pulse_end) ? a.pulse_amp : 0.0f;
      Volts v = {sV[tid], sV[cap + tid], sV[2 * cap + tid]};
      voltage_step(a.P, vk, v, load_currents(sI, cap, tid), ic, iapp);
      vd[(step + 1) & 1][c] = v.Vd;
      sV[tid] = v.Vd;
      sV[cap + tid] = v.Vs;
      sV[2 * cap + tid] = v.Va;
      if (a.trace_axon) a.trace_axon[(size_t)t * N + c] = v.Va;
    }
    __syncthreads();
  }
  if (own) {
    float* s = a.state;
    s[0 * N + c] = sV[tid];
    s[7 * N + c] = sV[cap + tid];
    s[15 * N + c] = sV[2 * cap + tid];
    s[4 * N + c] = (float)sCa[tid];
#pragma unroll
    for (int k = 0; k < INFOLI_NSTATE; ++k)
      if (field[k] >= 0 && field[k] != F_GCAL) s[k * N + c] = sG[field[k] * cap + tid];
  }
}

std::mutex g_scratch_mu;
unsigned char* g_scratch_addr[kMaxDevices];

}  // namespace
}  // namespace infoli

using namespace infoli;

extern "C" int infoli_run_noalloc(const float* params, int n_cells, const int64_t* d_row_ptr, const int32_t* d_col,
                                  const float* d_g, float g_uniform, int pulse_start, int pulse_end, float pulse_amp,
                                  float* d_state, int step0, int n_steps, float* d_trace_axon, void* stream) {
  infoli__clear_error();
  if (!params || !d_row_ptr || !d_state || n_cells <= 0 || n_steps < 0 || step0 < 0)
    return infoli__fail(INFOLI_ERR_ARG, "run_noalloc: bad argument");
  if ((long long)step0 + (long long)n_steps > (long long)INT_MAX)
    return infoli__fail(INFOLI_ERR_ARG, "run_noalloc: step0 + n_steps exceeds INT_MAX");
  if (n_cells > kNoAllocMaxCells)
    return infoli__fail(INFOLI_ERR_CAPACITY,
                        "run_noalloc: %d cells exceed the static scratch limit of %d cells; use infoli_sim_create",
                        n_cells, kNoAllocMaxCells);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return infoli__fail(INFOLI_ERR_ARG, "run_noalloc: device %d out of range", dev);
  unsigned char* scratch = nullptr;
  {
    // once per device, with that device current: the symbol's device address
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess)
        return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      g_scratch_addr[dev] = static_cast<unsigned char*>(p);
    }
    scratch = g_scratch_addr[dev];
  }
  int nsm = 0;
  e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess)
    return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: cudaDeviceGetAttribute: %s", cudaGetErrorString(e));
  // as many CTAs as SMs, or as the caller's environment allows it beside other
  // work (two of them fit on an SM)
  int most = nsm;
  if (const char* s = getenv("INFOLI_NOALLOC_CTAS")) most = std::max(1, std::min(nsm, atoi(s)));
  most = std::max(most, (n_cells + kNoAllocBlock - 1) / kNoAllocBlock);
  const int per_cta = std::max(kNoAllocMinCells, (n_cells + most - 1) / most);
  const int grid = (n_cells + per_cta - 1) / per_cta, cap = (per_cta + 31) & ~31;
  const size_t smem = noalloc_smem(cap);
  if (per_cta > kNoAllocBlock)
    return infoli__fail(INFOLI_ERR_CAPACITY, "run_noalloc: %d cells need more than one thread per cell on %d SMs",
                        n_cells, nsm);
  int per_sm = 0;
  e = cudaFuncSetAttribute(noalloc_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)noalloc_smem(kNoAllocBlock));
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, noalloc_step_kernel, kNoAllocBlock, smem);
  if (e != cudaSuccess)
    return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: occupancy query: %s", cudaGetErrorString(e));
  if (grid > per_sm * nsm)
    return infoli__fail(INFOLI_ERR_CAPACITY, "run_noalloc: %d CTAs cannot be co-resident (%d allowed)", grid,
                        per_sm * nsm);
  NoAllocArgs a{};
  static_assert(sizeof(ModelParams) == INFOLI_NPARAM * sizeof(float), "param layout");
  memcpy(&a.P, params, sizeof(ModelParams));
  a.n = n_cells;
  a.step0 = step0;
  a.n_steps = n_steps;
  a.row_ptr = d_row_ptr;
  a.col = d_col;
  a.g = d_g;
  a.g_uniform = g_uniform;
  a.pulse_start = pulse_start;
  a.pulse_end = pulse_end;
  a.pulse_amp = pulse_amp;
  a.state = d_state;
  a.trace_axon = d_trace_axon;
  a.scratch = scratch;
  a.timeout_ns = infoli__wait_timeout_ns();
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the barrier counter and the error word must start at zero
  e = cudaMemsetAsync(scratch, 0, kCtlBytes, s);
  if (e != cudaSuccess) return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: cudaMemsetAsync: %s", cudaGetErrorString(e));
  int cells = per_cta, cap_arg = cap;
  void* args[] = {&a, &cells, &cap_arg};
  e = cudaLaunchCooperativeKernel((const void*)noalloc_step_kernel, dim3(grid), dim3(kNoAllocBlock), args, smem, s);
  if (e != cudaSuccess) return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: launch: %s", cudaGetErrorString(e));
  // the error word comes back on the caller's stream: a plain cudaMemcpy would
  // go to the legacy default stream and wait for every blocking stream
  int err = 0;
  e = cudaMemcpyAsync(&err, scratch + 64, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: %s", cudaGetErrorString(e));
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return infoli__fail(INFOLI_ERR_CUDA, "run_noalloc: %s", cudaGetErrorString(e));
  if (err == kErrSender)
    return infoli__fail(INFOLI_ERR_ARG, "run_noalloc: a sender id is outside [0, n_cells) (or d_col is NULL)");
  if (err == kErrRowPtr) return infoli__fail(INFOLI_ERR_ARG, "run_noalloc: d_row_ptr is negative or decreasing");
  if (err) return infoli__fail(INFOLI_ERR_TIMEOUT, "run_noalloc: grid barrier wait gave up");
  return INFOLI_OK;
}
