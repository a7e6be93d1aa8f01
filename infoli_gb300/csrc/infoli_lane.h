// The batched cluster kernel's per-CTA record and the "lane": the serving
// loop's way of running small networks through that kernel, each on device
// buffers of its own, joining and leaving between launches of a few thousand
// steps.  Internal to libinfoli_gpu.so (infoli_batch.cu, infoli_serve.cu).
#pragma once
#include <cstdint>
#include <vector_types.h>

namespace infoli {

// One CTA slot of a cluster of the batched kernel.  Every CTA of a cluster
// belongs to the same network, so n_steps, step0 and the pulse are the same
// in all of them.
struct alignas(16) BatchCta {
  int net;           // network, -1: idle slot
  int rank;          // rank of this CTA inside its network (0 .. ncta-1)
  int ncta;          // CTAs of the network
  int rank0;         // cluster rank of the network's first CTA (ranks are contiguous)
  int cbeg, ncell;   // owned cells [cbeg, cbeg + ncell), network-local
  int n;             // cells in the network
  int wpr;           // bitmask words per receiver row, ceil(n / 32)
  float* st;         // state: field f of the network's cell c at st[f * T + cell_base + c]
  double* ca;        // Ca2+ of the network's cell c at ca[cell_base + c] (FP64 between launches)
  // entry lists (batches): group g of the CTA (receivers 32 g ..) is grp[g] =
  // {first pair row, pairs}, a pair row being 32 lanes x 8 entries of ent (16-bit
  // byte offsets into the V_dend buffer); null: bitmask rows
  const uint4* ent;
  const int2* grp;
  const uint32_t* bits;  // word w of receiver r at bits[w * n + r] (two zero words after each row)
  long long T;       // SoA stride of st
  long long cell_base;
  float g;           // conductance of every edge of the network
  int resident;      // rows of the owned receivers kept in shared memory
  int cl_sync;       // the cluster holds a network of several CTAs: cluster barrier per step
  int n_steps;       // steps of this launch; < 0: the launch's count
  int step0;         // index of the first step; < 0: the batch's device step counter
  int pulse_start, pulse_end;
  float pulse_amp;
  int pad0;
};

// ---- rules for entry lists (batches)
enum { kListMaxCtas = 16 };  // CTAs per network

// CTAs of `block` threads of a network whose receivers take `lanes` lanes each.
inline int list_ctas(int n, int lanes, int block) { return (n * lanes + block - 1) / block; }

// Lanes per receiver: two where they cost no further CTA, and for networks
// whose CTAs would still run when all others are done (more than 3/4 of an
// SM's share of the whole batch each), as long as the device runs clusters of
// that many CTAs (runs[cs]; beyond 8 that depends on the device).
inline int list_lanes(int n, double edges, double all_edges, int block, int sms, const bool runs[kListMaxCtas + 1]) {
  const int one = list_ctas(n, 1, block), two = list_ctas(n, 2, block);
  if (two > kListMaxCtas || !runs[two]) return 1;
  return two == one || edges / one > 0.75 * all_edges / sms ? 2 : 1;
}

// Entry lists (16 bits per edge, 512 bytes per pair row) rather than bitmask
// rows: where they take no more than half of the free memory, and with the
// bitmasks that they are packed from no more than nine tenths.
inline bool lists_fit(long long pair_rows, long long bit_words, double mem_free) {
  const double entries = (double)pair_rows * 512.0;
  return pair_rows <= INT32_MAX && entries <= 0.5 * mem_free && entries + (double)bit_words * 4.0 <= 0.9 * mem_free;
}

// One network of a lane launch.
struct LaneNet {
  float* st;             // [INFOLI_NSTATE * n] device SoA (reference order; the Ca2+ row is not used)
  double* ca;            // [n] device Ca2+
  const uint32_t* bits;  // [n * (ceil(n/32) + 2)] device rows, infoli__lane_pack_bits layout
  int n;
  float g;
  int step0, n_steps;
  int pulse_start, pulse_end;
  float pulse_amp;
};

}  // namespace infoli

struct infoli_lane;

// Networks of at most this many cells run in the lane (clusters of up to 8
// CTAs of 1,024 threads).
enum { kLaneMaxCells = 8192 };

// Host: a CSR network (receiver rows) as the batched kernel's bitmask rows,
// word-major (word w of receiver r at out[w * n + r]), most-significant bit
// first, self bits cleared, two zero words after every row:
// n * (ceil(n/32) + 2) words.  Returns 0, or -1 for a sender outside [0, n).
int infoli__lane_pack_bits(int n, const int64_t* row_ptr, const int32_t* col, uint32_t* out);
// CTAs (= SMs, one 1,024-thread CTA per SM) a network of n cells takes.
int infoli__lane_ctas(int n);
int infoli__lane_create(int device, const float* params, int kahan, infoli_lane** out);
// Launches n_steps of every network (each its own n_steps, step0 and pulse)
// asynchronously on the lane's streams; nets must stay valid until the
// launch has finished (infoli__lane_query != 0).  The networks' clusters are
// grouped by size, one kernel per group, the groups running concurrently.
int infoli__lane_launch(infoli_lane* L, const infoli::LaneNet* nets, int count);
// 1 when the last launch has finished, 0 while it runs, < 0 on an error.
int infoli__lane_query(infoli_lane* L);
// The lane's own stream (launches are ordered after work queued on it).
void* infoli__lane_stream(infoli_lane* L);
void infoli__lane_destroy(infoli_lane* L);
