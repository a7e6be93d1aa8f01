// Work decomposition shared by the host planner (infoli_plan.cpp) and the
// persistent step kernel (infoli_kernels.cu).  Plain-old-data only.
//
// A network (or a batch of independent networks laid side by side) is a set
// of receiver cells with CSR neighbour lists into one global V_dend array.
// The planner cuts it into CTA work items:
//   * a CTA owns a contiguous run of cells (<= its thread count); one thread
//     per owned cell runs the fused compartment update, state in registers;
//   * the senders its receivers read form one or more "tiles": contiguous,
//     16-byte-aligned ranges of the V_dend array that are staged into shared
//     memory by a bulk async copy each step;
//   * the edges of a (receiver, tile) pair are cut into chunks of at most
//     kChunkEdges edges (a multiple of it for dense networks, whose slots
//     would not fit in shared memory otherwise); one warp reduces one chunk
//     into one partial-sum slot; the update thread adds its receiver's slots
//     in sender order.
// Edge entries are 16-bit offsets from the tile start (a tile is at most
// 65536 floats), so one gather from shared memory per edge.
//
// Two ways of exchanging V_dend between the steps of such plans:
//   * barrier mode: V_dend double buffer in global memory, one grid barrier
//     per step, tiles staged by bulk async copies (any window size);
//   * stamped mode (every CTA's window fits in shared memory at once): every
//     cell publishes (V_dend, step) as one 64-bit word into a two-slot array;
//     a CTA polls exactly the words it reads -- its window, the sorted list of
//     its receivers' unique senders, kept in the plan's gcol table at
//     CtaWork::tile_begin (n_tiles entries; stamped plans have no tiles) --
//     plus one word of every CTA that reads it without being read by it, so
//     no slot is overwritten before its readers are done, until their stamps
//     show the step it needs.  No grid barrier: each CTA waits only for its
//     own neighbourhood.
// Networks whose edges do not stay on chip have plans of their own (SmemShape::
// gather): gathers through L2 or from staged tiles, adjacency bits, or entry lists
// streamed over shares of V_dend (StreamLayout), all with the grid barrier.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
namespace infoli {
#endif

enum { kChunkEdges = 128, kMaxChunkEdges = 8192 };

// Packed layout of stamped plans.  A lane-chunk is up to `lane_edges` (8, 16
// or 32, one number per plan) edges of one receiver reduced by ONE lane; 32
// lane-chunks form a group handled by one warp.  Entries are stored transposed
// in 4-entry quads so lane l reads its next four entries with one 8-byte load:
//   entry k of lane l in group g at ((g * lane_edges / 4 + k / 4) * 32 + l) * 4 + k % 4
// Each entry is the byte offset, from the start of dynamic shared memory, of
// the sender's V_dend; padding entries address the receiver's own V_dend.
enum { kMaxLaneEdges = 32 };
// Stamped plans: words that a thread polls in one round of loads where the
// largest window allows it (StepArgs, SmemShape::poll_words).
enum { kPollBatchSmall = 3 };

typedef struct {
  int cell_begin;   // first owned cell (index into the V_dend / state arrays)
  int n_cells;      // owned cells, <= threads per CTA
  int tile_begin;   // first tile of this CTA in the tile table
  int n_tiles;      // tiles this CTA stages each step
  int slot_begin;   // partial slots of this CTA: chunk ids slot_begin.. (absolute)
  int n_slots;      // number of chunks == number of partial slots
  int probe_begin;  // stamped-exchange mode: cells of CTAs that read this CTA's
  int n_probes;     //   cells but are not read by it (progress probes)
  int group_begin;  // stamped mode: first lane-chunk group of this CTA (absolute)
  int n_groups;     //   number of groups
  int pad0, pad1;
} CtaWork;

typedef struct {
  int lo;           // first V_dend index of the tile (multiple of 4)
  int nfloats;      // tile length in floats (multiple of 4)
  int chunk_begin;  // chunks of this tile: [chunk_begin, chunk_end), absolute
  int chunk_end;
} TileDesc;

typedef struct {
  int slot;         // partial slot, relative to the CTA's slot_begin (first: the
  int recv;         //   kernel loads {slot, recv} as one 8-byte word)
                    // receiver, relative to the CTA's cell_begin
  int edge_begin;   // absolute index into the edge-offset (and per-edge g) arrays
  int count;        // edges in this chunk, 1 .. the plan's chunk length
} ChunkDesc;

#if defined(__CUDACC__)
#define INFOLI_HD __host__ __device__
#else
#define INFOLI_HD
#endif

// Sizes that fix the step kernel's dynamic shared memory.  When res_chunks
// is non-zero the CTA's static work (tile and chunk descriptors, edge
// offsets, per-edge conductances) is copied into shared memory once per
// launch ("resident" plan) instead of being re-read from global memory
// every step.
typedef struct {
  int tile_cap;    // floats per tile buffer
  int nbuf;        // tile buffers (1 or 2)
  int threads;     // threads per CTA
  int cells_cap;   // owned cells per CTA (max over CTAs, multiple of 32)
  int max_slots;   // partial-sum slots per CTA
  int kahan;       // compensated sums (second slot array)
  int res_tiles;   // resident tile descriptors per CTA (0: not resident); stamped
                   // plans keep the window's sender ids there, four per slot
  int res_chunks;  // resident chunk descriptors per CTA (stamped: lane-chunks, 16 B each)
  int res_edges;   // resident edge offsets per CTA
  int edge_g;      // per-edge conductances present
  int stamped;     // stamped exchange (the whole window resident at once, nbuf = 1)
  int dup_words;   // stamped: second copy of the window starts this many floats in
                   // (a multiple of 32 plus 16, so each word sits in two banks 16
                   // apart); 0 = single copy
  int gather;      // 1: gather plan, one thread per receiver reads its senders' V_dend
                   // through L2; edges column by column per CTA (CtaWork::slot_begin
                   // = first entry, pad0 = padded row length); no dynamic shared memory.
                   // 2: tiled gather plan, V_dend staged tile by tile in shared memory
                   // (nbuf x tile_cap floats, then 2 mbarriers), one thread per
                   // receiver; per tile, entries column by column (16-bit offsets from
                   // the tile start; TileDesc::chunk_begin = first entry, chunk_end =
                   // padded row length) and per-receiver counts at CtaWork::slot_begin
                   // + tile * n_cells + receiver.
                   // 3: bitmask plan (uniform g), V_dend staged tile by tile as above;
                   // receivers' adjacency rows as bits (bit 31 of word w = sender 32 w),
                   // word w of local receiver t at CtaWork::slot_begin + w * n_cells + t,
                   // two zero words after each row (CtaWork::pad0 = words per row);
                   // tiles cover whole 32-sender columns (TileDesc::chunk_begin /
                   // chunk_end = first / end column); `slices` threads share a row
                   // 4: stream plan (see StreamLayout): one or more CTAs per receiver group,
                   // each staging its share of V_dend whole (tile_cap floats) and
                   // streaming its lane-chunks' entries from global memory
  int slices;      // bitmask plan: threads per receiver (column slices)
  int lane_edges;  // stamped: entries per lane-chunk (8, 16 or 32)
  int poll_words;  // stamped: the most words one CTA polls per step (window
                   // senders + progress probes); picks the poll batch size
  int cluster;     // stream plan: CTAs per cluster (sender shares)
  int rows_cap;    // stream plan with cluster > 1: staged V_dend of the cluster's receivers
  int block;       // stream plan: entries per lane taken at a time (8, or 16 for long lane-chunks)
  int plain;       // stream plan: differences of V_dend itself, not of V_dend x kVScale
  int byte_off;    // stream plan: entries are byte offsets (the staged floats fit in 64 KB), else float indices
} SmemShape;

static inline INFOLI_HD size_t tgather_smem_bytes(SmemShape s) {
  const size_t tiles = (((size_t)s.nbuf * (size_t)s.tile_cap * sizeof(float) + 15) & ~(size_t)15);
  // bitmask plans: per-slice partial sums (and compensations) of the receivers
  const size_t part =
      s.gather == 3 ? ((size_t)s.slices * 2 + 1) * (size_t)s.cells_cap * sizeof(float) : 0;  // + V_dend
  return tiles + part + 2 * sizeof(uint64_t);
}

// Number of per-cell float arrays kept in shared memory: V_dend, V_soma,
// V_axon and the nine gate-unit currents.
enum { kCellArrays = 13 };
// Stamped plans: cell array 12 holds V_dend x kVScale of the CTA's own cells
// (the window copy holds scaled values too; padding entries read it).
enum { kScaledVArray = 12 };
// Per-cell gate state in shared memory: 17 float fields (indexed like the
// device state arrays) plus the FP64 Ca2+ concentration.
enum { kGateFloats = 17 };

// Dynamic shared-memory layout of the step kernel (byte offsets):
//   [tile buffers: nbuf x tile_cap floats]
//   [cell arrays: kCellArrays x cells_cap floats]
//   [gate state: cells_cap doubles (Ca2+), kGateFloats x cells_cap floats]
//   [partial sums: max_slots floats][Kahan compensations: max_slots floats,
//    16-byte aligned]
//   [2 mbarriers, 16-byte aligned]
//   resident plans only: [tile descs][chunk descs][per-edge g][edge offsets]
typedef struct {
  size_t tiles, vown, gates, gca, part, partc, mbar, tdesc, chunks, eg, edges, total;
} SmemLayout;

static inline INFOLI_HD SmemLayout smem_layout(SmemShape s) {
  SmemLayout L;
  size_t off = 0;
  L.tiles = off;
  off += (size_t)s.nbuf * (size_t)s.tile_cap * sizeof(float);
  L.vown = off;
  off += (size_t)kCellArrays * (size_t)s.cells_cap * sizeof(float);
  off = (off + 7) & ~(size_t)7;
  L.gca = off;
  off += (size_t)s.cells_cap * sizeof(double);
  L.gates = off;
  off += (size_t)kGateFloats * (size_t)s.cells_cap * sizeof(float);
  off = (off + 15) & ~(size_t)15;  // stamped plans read partial slots as float4
  L.part = off;
  off += (size_t)s.max_slots * sizeof(float);
  off = (off + 15) & ~(size_t)15;  // stamped Kahan plans read compensations as float4
  L.partc = off;
  if (s.kahan) off += (size_t)s.max_slots * sizeof(float);
  off = (off + 15) & ~(size_t)15;
  L.mbar = off;
  off += 2 * sizeof(uint64_t);
  L.tdesc = off;
  off += (size_t)s.res_tiles * sizeof(TileDesc);
  L.chunks = off;
  off += (size_t)s.res_chunks * sizeof(ChunkDesc);
  L.eg = off;
  if (s.edge_g) off += (size_t)s.res_edges * sizeof(float);
  L.edges = off;
  off += (size_t)s.res_edges * sizeof(uint16_t);
  off = (off + 15) & ~(size_t)15;
  L.total = off;
  return L;
}

// Stream plans.  A cluster of `cluster` CTAs owns a contiguous run of
// receivers (rows CtaWork::tile_begin .. + n_tiles); every CTA of it owns a
// contiguous part of them (cell_begin, n_cells: one thread per cell runs the
// cell update) and holds one share of the senders, tile_cap consecutive
// V_dend, in shared memory (share k: cells k * tile_cap ..).  The rows'
// entries in that share are cut into lane-chunks, one lane each; 32 chunks of
// like length form a group, a warp walks the groups assigned to it
// (probes[pad0 + warp] .. probes[pad0 + warp + 1], relative to group_begin).
// Group i: gdesc[i] = {first quad row, quads per lane}, a quad row being 32
// lanes x 4 entries; gcol[32 i + lane] = row | slot << 16.  Entry k of lane l
// lies at (first * 128) + (k / 8) * 256 + l * 8 + k % 8 in the edge array while
// whole 8-entry pairs last (16-byte loads), the odd quad after them at
// + l * 4 + k % 4; its conductance at (first * 128) + (k / 4) * 128 + l * 4 + k % 4.
// An entry is the place of a float from the start of dynamic shared memory, in
// bytes where all of them lie within 64 KB (one instruction less per entry),
// else in floats; padding entries name the row's own V_dend (a term of exactly 0).  Partial
// sums: cell_slots[cell * cluster + k] = its slots in CTA k of the cluster.
//   [share of V_dend][cluster > 1: the rows' V_dend][partial sums][the own
//   cells' sums by CTA of the cluster][mbarrier][the rows' slots: first |
//   count << 16][the own cells' stimulus of the step]
// (slots and stimulus in shared memory: read from L2 after the coupling, the
// last warp's loads stood in the step's way: 11.7 against 11.0 us per step at
// 100,000 cells x 100 senders with conductances, 6.96 against 6.80 at 6,007 x
// 1,500, 4.17 against 4.10 at 48,017 x 33)
// 24 warps, not 32: 80 registers a thread keep the loads of the coupling and
// the gate units unspilled (16 bytes spill with conductances per edge), which is
// worth more than the warps (13.1 -> 11.7 us per step at 100,000 cells x 100
// senders with conductances, 8.9 -> 8.3 at 10,000 x 2,000, 4.4 -> 4.15 at 48,017
// x 33).
enum { kStreamThreads = 768, kStreamWarps = 24, kStreamMaxCluster = 4 };
typedef struct {
  size_t rows, part, sums, mbar, slots, app, total;
} StreamLayout;

static inline INFOLI_HD StreamLayout stream_layout(SmemShape s) {
  StreamLayout L;
  size_t off = (size_t)s.tile_cap * sizeof(float);
  L.rows = off;
  off += (size_t)s.rows_cap * sizeof(float);
  off = (off + 15) & ~(size_t)15;
  L.part = off;
  off += (size_t)s.max_slots * sizeof(float);
  L.sums = off;
  off += (size_t)s.cluster * (size_t)s.cells_cap * sizeof(float);
  off = (off + 15) & ~(size_t)15;
  L.mbar = off;
  off += 16;
  L.slots = off;
  off += (size_t)(s.cluster > 1 ? s.rows_cap : s.cells_cap) * sizeof(uint32_t);
  L.app = off;
  off += (size_t)s.cells_cap * sizeof(float);
  L.total = off;
  return L;
}

#ifdef __cplusplus
}  // namespace infoli
#endif
