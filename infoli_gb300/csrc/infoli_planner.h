// Host planner: cuts a CSR network into the CTA / tile / chunk work items of
// the persistent step kernel (see infoli_plan.h for the device-side view).
#pragma once
#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

#include "infoli_plan.h"

namespace infoli {

// Length of every per-cell device array for n cells: a multiple of 32 with
// 32 spare entries, so tile ends rounded up to 16 bytes stay in bounds.
inline int pad_cells(int n) { return ((n + 31) / 32) * 32 + 32; }

struct alignas(8) int2_t {
  int x, y;
};

struct alignas(8) CellSlots {
  int begin;  // first partial slot, relative to the CTA
  int count;  // number of slots (chunks) of this receiver
};

struct PlanInput {
  int n = 0;                       // receivers 0..n-1 (also the sender id space)
  const int64_t* row_ptr = nullptr;
  const int32_t* col = nullptr;
  const float* g = nullptr;        // per-edge conductance or null
  int grid = 0;                    // CTAs to use (0: heuristic, capped by grid_max)
  int grid_max = 0;                // co-resident CTA limit
  int threads = 1024;              // threads per CTA
  size_t smem_budget = 0;          // dynamic shared memory per CTA (bytes)
  int kahan = 0;
  int no_resident = 0;             // force per-step reads of the static work from global memory
  int sync_mode = 0;               // kSyncAuto / kSyncBarrier / kSyncStamped
  int reorder = 1;                 // stamped plans: try a locality-preserving cell order
  const int* cta_starts = nullptr; // optional CTA cell ranges (grid + 1 entries; internal)
  int no_stream = 0;               // auto mode: no stream plans
  // stream plans over sender shares: most co-resident CTAs in clusters of 2
  // and of 4 (0: none, -1: grid_max, rounded down to whole clusters)
  int cluster_ctas[2] = {-1, -1};
};

// Locality reordering is tried for stamped plans whose largest window is at
// least kReorderMinWindowRatio x the cells per CTA and at most half the
// network, on networks of at most kReorderMaxEdges edges; it is kept when it
// shrinks the largest window by at least a fifth.
enum { kReorderMinWindowRatio = 4, kReorderIters = 160 };
constexpr int64_t kReorderMaxEdges = 32ll << 20;

enum { kSyncAuto = 0, kSyncBarrier = 1, kSyncStamped = 2, kSyncGather = 3, kSyncTiledGather = 4, kSyncBits = 5,
       kSyncStream = 6 };

// Auto mode picks a bitmask plan (uniform g only) over tile/gather plans when
// the density is at least 1 / kBitsMinDensityInv.
enum { kBitsMinDensityInv = 16 };

// Auto mode picks a tiled gather plan over a barrier plan when the mean degree
// is at most this (rows too short to fill a warp per chunk once split by tiles).
enum { kGatherMaxMeanDegree = 384 };

// Stream plans are for edges that do not stay on chip.  Auto mode takes them
//   - with the whole V_dend array as one share (up to about 50,000 cells), except
//     for one conductance at a density of kStreamMaxDensity or more,
//     where a bit per pair is shorter than 16 bits per edge by more than the
//     walk of the bits costs;
//   - with the senders shared by a cluster's CTAs for rows of at least
//     kStreamMinDegree edges on average (shorter rows spend more on the
//     exchange of partial sums than the tiles cost), unless they are dense
//     with one conductance (bitmask plans).
// A stamped plan (edges on chip, V_dend word by word from its publishers) gives
// way to a stream plan when a CTA polls more than kStampedMaxWords words or owns
// more than kStampedMaxCells cells.  Microseconds per step, stamped against
// stream: 6,000 cells x 60 senders (2,800 words) 2.85 / 3.5; 10,000 x 40 (3,300)
// 3.30 / 3.53; 20,000 x 30 (132 cells, 3,900) 3.73 / 3.65; 4,000 at 20 % (4,000)
// 3.85 / 4.52; 10,000 x 100 (4,850) 4.29 / 3.86; 6,000 x 200 (5,300) 3.97 / 3.79;
// 20,000 x 100 (9,700) 6.82 / 4.30; 30,000 x 8 (198 cells, 1,600 words) 4.56 /
// 3.51; 150 x 150 grid (148 cells) 4.33 / 4.94; 200 x 200 grid (264 cells) 5.33 /
// 4.95; 48,000 x 33 (316 cells, 9,400) 7.84 / 4.66.
enum { kStampedMaxWords = 4500, kStampedMaxCells = 192 };
enum { kStreamMinDegree = 16 };
constexpr double kStreamMaxDensity = 0.45;

// A vector whose resize() leaves new elements as they are: the threads that fill
// a large table touch its pages first.
template <class T>
struct UnclearedAllocator : std::allocator<T> {
  template <class U>
  struct rebind {
    using other = UnclearedAllocator<U>;
  };
  template <class U>
  void construct(U*) noexcept {}
  template <class U, class A, class... B>
  void construct(U* p, A&& a, B&&... b) {
    ::new ((void*)p) U(std::forward<A>(a), std::forward<B>(b)...);
  }
};
template <class T>
using Uncleared = std::vector<T, UnclearedAllocator<T>>;

struct Plan {
  int grid = 0, threads = 0, tile_cap = 0, nbuf = 1, max_slots = 0;
  SmemShape shape{};                  // shared-memory shape of the launch
  size_t smem_bytes = 0;
  std::vector<CtaWork> cta;
  std::vector<TileDesc> tiles;
  std::vector<ChunkDesc> chunks;
  std::vector<CellSlots> cell_slots;  // [n]
  Uncleared<uint16_t> edges;
  Uncleared<float> edge_g;            // empty unless per-edge g
  std::vector<int> probes;            // stamped mode: progress-probe cells
  std::vector<int2_t> gdesc;          // stamped mode: {slot, recv} per lane-chunk, 32 per group
  std::vector<int32_t> gcol;          // gather mode: sender ids, column by column per CTA;
                                      // tiled gather: entries per (tile, receiver);
                                      // bitmask plans: the rows' bit words
  std::vector<int32_t> perm;          // relabelled plans: perm[plan cell] = caller's cell
                                      // (empty: the caller's order); every table above
                                      // uses plan cell ids
};

// Shared-memory bytes the step kernel needs for a plan's parameters.
size_t plan_smem_bytes(int tile_cap, int nbuf, int threads, int cells_cap, int max_slots, int kahan);

// Returns false and sets *err on failure.
bool make_plan(const PlanInput& in, Plan* out, std::string* err);

// Locality-preserving cell order for `parts` CTAs of at most `threads`
// cells: order[new] = old and the CTA starts in the new order (parts + 1
// entries).  Empty when no such order was found.
std::vector<int> locality_order(const PlanInput& in, int parts, int threads, std::vector<int>* starts);

}  // namespace infoli
