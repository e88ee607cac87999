// mtc_gather.hpp -- argument blocks and launchers of the forest, compaction
// and diff-assembly kernels (gather_kernels.cu) and of the map maintenance
// kernels.  Internal to the library.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "mtc_common.cuh"
#include "mtc_internal.hpp"

namespace mtc {

enum : int { APPROACH_TREE = 0, APPROACH_LIST = 1, APPROACH_BASIC = 2 };
constexpr uint32_t kSortTile = 4096;

// Device-resident description of one assembled diff.  Offsets are relative to
// the first header byte, which sits at stage + pad (pad makes the data section
// 16-byte aligned in device memory).
struct Layout {
  uint32_t F, S, P, num_distinct;  // FO entries, shift entries, source checkpoints, valid FO regions
  uint64_t chunk_counter;          // chunk slots in the data section
  uint64_t pad, data_off, table_off, pairs_off, diff_len;
  uint64_t size_data, size_meta;   // the reference's datasizes pair
  uint32_t root_fo, max_key, ok, nkeys;  // nkeys: distinct sort keys of the shift entries
  uint32_t sort_n, sort_tiles;            // nkeys * sort tiles; tiles of kSortTile shift entries
};

// The canonical (serial push) order of a tree's nodes.
struct RootOrder {
  int ascending;   // 0 = deeper levels first, 1 = ascending node id
  uint32_t D;      // depth of node M-1
  uint64_t sizeD;  // nodes on depth D
};

struct ForestArgs {
  Digest* tree;
  uint8_t* labels;
  uint8_t* rflag;  // root flags at canonical positions (M-1 bytes)
  DigestMap map;
  const StepParams* sp;  // cur, epochs (device)
  uint32_t* err;
  int hash_kind;
  RootOrder order;
  // Incremental checkpoints: word that is 0 when no leaf was demoted to a
  // shifted duplicate of a digest first seen in this checkpoint.  Then no
  // shifted pair can hash to a digest inserted by the first-occurrence pass
  // (its leaves would share a digest with a first occurrence, whose digest is
  // new), so both passes run in one traversal.  Null: two passes.
  const uint32_t* fuse_gate;
  uint32_t* ins_queue;  // first-occurrence nodes awaiting their map insert (N entries)
  uint32_t* ins_count;
  uint32_t* span_done;  // forest_done_words(N) counters, zero between passes
  uint32_t* zero_found; // set by pass 3 when a shift test succeeds
};

// Position of node x (>= 1) in the canonical root order.
__host__ __device__ __forceinline__ uint64_t canon_pos(const ForestArgs& a, uint32_t x) {
  if (a.order.ascending) return (uint64_t)x - 1;
#ifdef __CUDA_ARCH__
  const uint32_t d = 31 - __clz(x + 1);
#else
  uint32_t d = 0;
  while (((2ull << d) - 1) <= (uint64_t)x) d++;
#endif
  const uint64_t fp = d == a.order.D ? 0 : a.order.sizeD + ((1ull << a.order.D) - (2ull << d));
  return fp + (x - ((1ull << d) - 1));
}

struct GatherArgs {
  int approach;
  const uint8_t* data;
  uint64_t len;
  uint32_t cs, N, M;
  const StepParams* sp;   // cur, baseline_id (device)
  uint32_t k_cap;         // capacity of hist / rep / rank (checkpoint ids + 1)
  const Digest* digests;  // tree heap (by node) or hash list (by chunk)
  DigestMap map;
  uint32_t* err;
  uint64_t* clk;          // phase times (may be null)
  uint32_t* counters;     // COUNT_*
  // what is compacted: root flags at canonical positions (tree) or the chunks'
  // labels, padded to whole 16-byte words
  uint8_t* flags;
  uint64_t n_flags;
  const uint8_t* labels;  // tree: node labels
  RootOrder order;
  int all_own;            // a baseline of an empty map: every first occurrence owns its digest
  uint64_t *tile_counts, *tile_regions;  // per tile of flags
  uint32_t* fo_list;
  uint32_t* sh_list;
  uint64_t* fo_val;       // tree: regions and chunks before the entry in its tile, bit 63 if it is a region
  uint32_t* fo_tile;      // tree: the entry's tile
  uint32_t *reg_chunk, *reg_slot;
  uint32_t *sh_key, *sh_prev;
  uint32_t *hist, *rep, *rank;
  uint64_t* sort_mat;
  uint64_t *scan_scratch2, *scan_total2;
  // inserts queued by a fused forest pass (fuse_gate as in ForestArgs)
  const uint32_t* fuse_gate;
  const uint32_t *ins_queue, *ins_count;
  uint8_t* stage;
  uint64_t stage_cap;
  Layout* lay;
  Readback results;       // written by the last launch
  uint32_t n_emit, n_sort, n_drain, n_copy, sort_scan;  // set by launch_assemble
};

// One forest pass.  pass 0 = first-occurrence forest, 1 = duplicate forest, 3 =
// both of a baseline whose digests count as cleared (baseline = 1), which
// launch_forest_inserts completes.
size_t forest_done_words(uint32_t N);
cudaError_t launch_forest(const ForestArgs& a, int pass, int baseline, uint32_t N, cudaStream_t s);
// The inserts of pass 3: all of them, or only if its shift test found the zero
// digest (its shifted roots may then be interior nodes, which the root lookups
// need in the map), or only if it did not (no lookup then waits for them).  No
// buffer with a zero digest is known (a zero leaf counts as unchanged, and no 32
// bytes hash to zero with Murmur3), so the second kind is there for the rule's
// sake and returns at once.  Launched ahead of the third on another stream, it
// also lets the root count's blocks start before the inserts fill the GPU:
// without it a baseline of 4 GiB in 512-byte chunks takes 3.30 instead of 3.24 ms,
// with the inserts behind the root lookups 3.39.
enum : int { INSERT_ALWAYS = 0, INSERT_IF_ZERO = 1, INSERT_UNLESS_ZERO = 2 };
cudaError_t launch_forest_inserts(const ForestArgs& a, int when, uint32_t N, cudaStream_t s);
// Roots listed and the diff assembled into g.stage; max_entries bounds F and S
// (N + 1).  whole: most chunks are expected in the diff (a baseline).  join: the
// last launch waits for this event too (may be null).
cudaError_t launch_assemble(GatherArgs g, uint64_t max_entries, bool whole, cudaEvent_t join, cudaStream_t s);
// Rebuild `from` into the empty table `to` (capacity change), preserving values.
cudaError_t launch_map_rehash(const DigestMap& from, uint64_t from_cap, const DigestMap& to, uint32_t* err,
                              cudaStream_t s);
// Every entry's epoch set to 0 (before the epoch counter restarts).
cudaError_t launch_map_rebase(const DigestMap& m, uint64_t cap, cudaStream_t s);

}  // namespace mtc
