// gather_kernels.cu -- everything between the leaf kernel and the finished
// incremental checkpoint in HBM:
//   * Merkle forest passes, several tree levels per launch (src/tree_approach.cpp
//     :124-227 baseline, :378-477 incremental; both incremental passes in
//     one traversal when no leaf was demoted);
//   * deterministic compaction of region roots in the order a serial backend
//     pushes them (replaces the atomic Vector::push, include/kokkos_vector.hpp:37-40);
//   * diff assembly: region sizes, repeat-count table, stable sort of the
//     shifted duplicates by source checkpoint, metadata and the chunk gather
//     (src/tree_approach.cpp:512-710, src/list_approach.cpp:79-247,
//     src/basic_approach.cpp:52-143).
#include <algorithm>
#include <cstdio>

#include "mtc_common.cuh"
#include "mtc_gather.hpp"
#include "mtc_scan.cuh"

namespace mtc {

namespace {

constexpr uint32_t kSortFastKeys = 1024;  // distinct source checkpoints per diff

inline uint32_t grid_for(uint64_t n, int threads, int per_sm = 8) {
  uint64_t g = (n + threads - 1) / threads;
  uint64_t cap = (uint64_t)num_sms() * per_sm;
  if (g > cap) g = cap;
  if (g == 0) g = 1;
  return (uint32_t)g;
}

// ---------------------------------------------------------------------------
// Forest passes
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint8_t child_flag(uint8_t lab) {
  return (lab == FIXED_DUPL || lab == DONE) ? ROOT_NONE : (lab == SHIFT_DUPL ? ROOT_SHIFT : ROOT_FO);
}

// Passes.  0: first-occurrence forest (src/tree_approach.cpp:378-404); 1:
// duplicate forest (:413-477); 2: both incremental passes in one traversal
// (ForestArgs::fuse_gate); 3: both passes of a baseline (:115-227) whose
// digests count as cleared in one traversal, which hashes every node and leaves the inserts to
// forest_insert_all_kernel.
//
// Pass 3.  A node is a first occurrence in the baseline's second pass exactly
// when it is one in the first (both only look at the leaves' labels), with the
// same digest, so its second hash and insert change nothing.  The shift test
// reads a digest that is still zero, so it asks one question of the map:
// whether it holds the all-zero digest.  Which of the passes a node's insert
// belongs to is kept in its epoch, and a map entry keeps the lowest (epoch,
// priority), so the inserts may follow in any order.  4 GiB in 512-byte
// chunks: the two passes took 2.10 ms (bottom 0.23, inserts 1.16, a barrier
// per level with a second hash and insert of every node 0.71).
//
// Launches.  A pass is one launch.  Block b of forest_kernel owns the 12 lowest
// levels below one node; the last block to finish below a node nine levels up
// goes on with those nine levels, and so on to the root, so that no level
// waits for a launch (the upper levels as launches of their own took 5-8 us of
// a 47 us labelling of 2^19 chunks, and as much again for the duplicate pass
// that usually returns at once).  Trees of at most 2048 leaves are one block.
constexpr uint32_t kSpanLevels = 9;     // 256 nodes on the bottom level of a span
constexpr uint32_t kBottomLevels = 12;  // bottom span: 16 leaves per thread, 4096 per block
constexpr uint32_t kSmallLeaves = 2048; // forest_small_kernel

__device__ __forceinline__ bool forest_fused(const ForestArgs& a) { return a.fuse_gate && *a.fuse_gate == 0; }

// First-occurrence nodes of a span, collected in shared memory as positions in
// the subtree of the span's root r: position h at relative depth k = log2 h is
// node h - 1 + (r << k).  `off` is (r << k) - 1 of the level being computed.
struct IdSink {
  uint16_t* ids;
  uint32_t* n;
  uint32_t off;
};
__device__ __forceinline__ void sink_level(IdSink& sink, uint64_t r, int k) { sink.off = (uint32_t)((r << k) - 1); }
__device__ __forceinline__ void queue_insert(IdSink& sink, uint32_t n) {
  sink.ids[atomicAdd(sink.n, 1u)] = (uint16_t)(n - sink.off);
}
// The span's inserts, by its block: issued at once when the duplicate pass is
// still to come and will look them up; queued when the passes are fused (a
// fused pass looks nothing up that they could add), for launches that have
// other work to hide them (drain_inserts).  Each node's digest is new, as its
// leaves' are; the serial-order rule does not depend on the inserts' order.
__device__ __forceinline__ void flush_sink(const ForestArgs& a, bool fused, uint64_t r, const IdSink& sink,
                                           uint32_t* base) {
  __syncthreads();
  const uint32_t cnt = *sink.n;
  auto node = [&](uint32_t k) {
    const uint32_t h = sink.ids[k];
    return (uint32_t)(h - 1 + (r << (31 - __clz(h))));
  };
  if (fused) {
    if (cnt && threadIdx.x == 0) *base = atomicAdd(a.ins_count, cnt);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x) a.ins_queue[*base + k] = node(k);
  } else {
    const uint32_t cur_id = a.sp->cur, epoch_fo = a.sp->epoch + 1;
    uint32_t created = 0;
    for (uint32_t k = threadIdx.x; k < cnt; k += blockDim.x)
      created += map_insert_serial(a.map, ld_digest(a.tree + node(k)), node(k), cur_id, epoch_fo, false, a.err);
    count_new_entries(a.map, created);
  }
  __syncthreads();
  if (threadIdx.x == 0) *sink.n = 0;
}

// One interior node n of a baseline's duplicate pass on digests that are not
// cleared (a second checkpoint under id 0): tests the not-yet-hashed digest,
// then hashes and inserts every interior node (:155-227).
__device__ __forceinline__ uint8_t forest_node(const ForestArgs& a, uint64_t n, uint8_t ll, uint8_t lr,
                                               uint32_t cur_id, uint32_t epoch_all) {
  const uint32_t l = 2 * (uint32_t)n + 1, rr = l + 1;
  uint8_t lab_n = DONE, fl = ROOT_NONE, fr = ROOT_NONE;
  if (ll != lr) {
    fl = child_flag(ll);
    fr = child_flag(lr);
  } else if (ll == FIXED_DUPL || ll == FIRST_OCUR) {
    lab_n = ll;
  } else if (ll == SHIFT_DUPL) {
    if (map_find(a.map, ld_digest(a.tree + n), a.err) >= 0) lab_n = SHIFT_DUPL;
    else fl = fr = ROOT_SHIFT;
  }
  if (fl != ROOT_NONE) a.rflag[canon_pos(a, l)] = fl;
  if (fr != ROOT_NONE) a.rflag[canon_pos(a, rr)] = fr;
  const Digest dg = hash_pair(a.hash_kind, ld_digest(a.tree + l), ld_digest(a.tree + rr));
  st_digest(a.tree + n, dg);
  if (map_insert_serial(a.map, dg, (uint32_t)n, cur_id, epoch_all, true, a.err)) atomicAdd(a.map.size, 1u);
  a.labels[n] = lab_n;
  return lab_n;
}

// Levels d_bot .. d_top of the subtree rooted at depth d_top for that pass,
// node labels in shared memory, one barrier per level: its shift test must
// see every insert of the levels below it.
__global__ void __launch_bounds__(256) forest_span_kernel(ForestArgs a, uint32_t N, uint32_t d_top, uint32_t d_bot) {
  pdl_enter();
  __shared__ uint8_t lab[2][2 << (kSpanLevels - 1)];
  const uint32_t cur_id = a.sp->cur, epoch_all = a.sp->epoch + 2;
  const uint64_t r = ((1ull << d_top) - 1) + blockIdx.x;
  const uint64_t last_interior = (uint64_t)N - 2, M = 2ull * N - 1;
  if (r > last_interior) return;
  const uint32_t wb = 1u << (d_bot - d_top);
  uint8_t* child = lab[0];
  uint8_t* cur = lab[1];
  {
    const uint64_t cfirst = (r + 1) * (2ull * wb) - 1;  // subtree nodes at depth d_bot + 1
    for (uint32_t i = threadIdx.x; i < 2 * wb; i += blockDim.x) {
      const uint64_t n = cfirst + i;
      child[i] = n < M ? a.labels[n] : DONE;
    }
  }
  __syncthreads();
  for (int d = (int)d_bot; d >= (int)d_top; d--) {
    const uint32_t width = 1u << (d - d_top);
    const uint64_t first = (r + 1) * width - 1;
    for (uint32_t i = threadIdx.x; i < width; i += blockDim.x) {
      const uint64_t n = first + i;
      cur[i] = n > last_interior ? (n < M ? a.labels[n] : (uint8_t)DONE)
                                 : forest_node(a, n, child[2 * i], child[2 * i + 1], cur_id, epoch_all);
    }
    __syncthreads();
    uint8_t* t = child;
    child = cur;
    cur = t;
  }
}

// Whether a node's digest is read by its parent in a pass: first-occurrence
// pairs are hashed in the first pass, shifted-duplicate pairs in the second,
// both in the fused pass 2.
__device__ __forceinline__ bool digest_wanted(int pass, uint8_t lab) {
  return pass == 0 ? lab == FIRST_OCUR : pass == 1 ? lab == SHIFT_DUPL : (lab == FIRST_OCUR || lab == SHIFT_DUPL);
}

// One interior node n of a pass given its children's labels and digests; `dg`
// receives n's digest when n is hashed.  First occurrences go to the block's
// sink; n's label is written when `store` is set (the top of a span); only
// flags other than ROOT_NONE are written, the flag array being clear before
// the first pass.  BASE: pass 3, every node hashed and its label kept for the
// inserts that follow.
template <int HK, bool BASE>
__device__ __forceinline__ uint8_t span_node(const ForestArgs& a, int pass, uint32_t n, uint8_t ll, uint8_t lr,
                                             const Digest& dl, const Digest& dr, Digest& dg, bool store,
                                             IdSink& sink) {
  const uint32_t l = 2 * n + 1, rr = l + 1;
  uint8_t lab_n = DONE;
  uint8_t fl = ROOT_NONE, fr = ROOT_NONE;
  if (!BASE && pass == 0) {
    if (ll == FIRST_OCUR && lr == FIRST_OCUR) {
      lab_n = FIRST_OCUR;
      dg = hash_pair(HK, dl, dr);
      st_digest(a.tree + n, dg);
      queue_insert(sink, n);
    }
  } else {
    if (ll != lr) {
      fl = child_flag(ll);
      fr = child_flag(lr);
    } else if (ll == FIXED_DUPL) {
      lab_n = FIXED_DUPL;
    } else if (ll == SHIFT_DUPL) {
      if (!BASE) {
        dg = hash_pair(HK, dl, dr);
        st_digest(a.tree + n, dg);
      }
      if (map_find(a.map, BASE ? Digest{{0, 0, 0, 0}} : dg, a.err) >= 0) {
        lab_n = SHIFT_DUPL;
        if (BASE) atomicOr(a.zero_found, 1u);
      } else {
        fl = fr = ROOT_SHIFT;
      }
    } else if (ll == FIRST_OCUR) {
      lab_n = FIRST_OCUR;
      if (!BASE && pass == 2) {
        dg = hash_pair(HK, dl, dr);
        st_digest(a.tree + n, dg);
        queue_insert(sink, n);
      }
    }  // both first duplicates, or both done: DONE
    if (fl != ROOT_NONE) a.rflag[canon_pos(a, l)] = fl;
    if (fr != ROOT_NONE) a.rflag[canon_pos(a, rr)] = fr;
  }
  if (BASE) {
    dg = hash_pair(HK, dl, dr);
    st_digest(a.tree + n, dg);
  }
  if (BASE || store) a.labels[n] = lab_n;
  return lab_n;
}

// Node n on the deepest interior level: a leaf there (a ragged last level)
// keeps its label and stored digest; an interior node is computed.
template <int HK, bool BASE>
__device__ __forceinline__ uint8_t span_label(const ForestArgs& a, int pass, uint64_t n, uint64_t last_interior,
                                              uint64_t M, uint8_t ll, uint8_t lr, const Digest& dl,
                                              const Digest& dr, Digest& dg, IdSink& sink) {
  if (n > last_interior) {
    const uint8_t lab = n < M ? a.labels[n] : DONE;
    if (BASE ? n < M : digest_wanted(pass, lab)) dg = ld_digest(a.tree + n);
    return lab;
  }
  return span_node<HK, BASE>(a, pass, (uint32_t)n, ll, lr, dl, dr, dg, false, sink);
}

__device__ __forceinline__ Digest shfl_digest(const Digest& d, int src) {
  constexpr unsigned kFull = 0xffffffffu;
  return Digest{{__shfl_sync(kFull, d.w[0], src), __shfl_sync(kFull, d.w[1], src), __shfl_sync(kFull, d.w[2], src),
                 __shfl_sync(kFull, d.w[3], src)}};
}

// The levels of an L-level span above its bottom one, from one node per thread
// (relative depth L - 1, node (r+1) * 2^(L-1) - 1 + threadIdx.x, label `lab`,
// digest `dg`, threads below 2^(L-1)): up to five inside each warp (children's
// labels and digests by shuffle), then up to three in warp 0 from the eight
// warps' results.  Stores r's label (L > 1).  Every node here is interior.
template <int HK, bool BASE>
__device__ __forceinline__ void upper_levels(const ForestArgs& a, int pass, uint64_t r, uint32_t L, uint8_t lab,
                                             Digest dg, IdSink& sink, uint8_t* top8, Digest* topdg) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t w = 1u << (L - 1);
  constexpr unsigned kFull = 0xffffffffu;
  const uint32_t in_warp = L - 1 < 5 ? L - 1 : 5;
#pragma unroll 1
  for (uint32_t step = 1; step <= in_warp; step++) {
    const int sl = (2 * lane) & 31, sr = (2 * lane + 1) & 31;
    const uint8_t cl = (uint8_t)__shfl_sync(kFull, lab, sl);
    const uint8_t cr = (uint8_t)__shfl_sync(kFull, lab, sr);
    Digest dl{{0, 0, 0, 0}}, dr{{0, 0, 0, 0}};
    if (BASE || __any_sync(kFull, digest_wanted(pass, lab))) {
      dl = shfl_digest(dg, sl);
      dr = shfl_digest(dg, sr);
    }
    const uint32_t width = 32u >> step, i = warp * width + lane;
    if (lane < width && i < (w >> step)) {
      sink_level(sink, r, (int)(L - 1 - step));
      const uint64_t n = (r + 1) * (w >> step) - 1 + i;
      lab = span_node<HK, BASE>(a, pass, (uint32_t)n, cl, cr, dl, dr, dg, step == L - 1, sink);
    }
  }
  if (L <= 6) return;
  if (lane == 0) {
    top8[warp] = lab;
    topdg[warp] = dg;
  }
  __syncthreads();
  if (warp == 0) {
    lab = lane < 8 ? top8[lane] : DONE;
    if (lane < 8) dg = topdg[lane];
#pragma unroll 1
    for (uint32_t step = 6; step <= L - 1; step++) {
      const int sl = (2 * lane) & 31, sr = (2 * lane + 1) & 31;
      const uint8_t cl = (uint8_t)__shfl_sync(kFull, lab, sl);
      const uint8_t cr = (uint8_t)__shfl_sync(kFull, lab, sr);
      const Digest dl = shfl_digest(dg, sl), dr = shfl_digest(dg, sr);
      if (lane < (w >> step)) {
        sink_level(sink, r, (int)(L - 1 - step));
        const uint64_t n = (r + 1) * (w >> step) - 1 + lane;
        lab = span_node<HK, BASE>(a, pass, (uint32_t)n, cl, cr, dl, dr, dg, step == L - 1, sink);
      }
    }
  }
}

// The spans above the block's own, whose root is node i of depth d: the last
// block to finish below a span's root takes the span.  The counters return to
// zero for the next pass.  Thread 0 wrote the label and digest of the block's
// root, so its fence publishes them; they are read past the L1.
template <int HK, bool BASE>
__device__ __forceinline__ void upper_spans(const ForestArgs& a, int pass, bool fused, uint32_t d, uint32_t i,
                                            IdSink& sink, uint32_t* base, uint8_t* top8, Digest* topdg,
                                            uint32_t* s_last) {
  uint32_t* done = a.span_done;
#pragma unroll 1
  while (d > 0) {
    const uint32_t L = d < kSpanLevels ? d : kSpanLevels, p = i >> L;
    d -= L;
    if (threadIdx.x == 0) {
      __threadfence();
      const bool last = atomicAdd(&done[p], 1u) + 1 == (1u << L);
      if (last) done[p] = 0;
      __threadfence();
      *s_last = last ? 1u : 0u;
    }
    __syncthreads();
    if (!*s_last) return;
    const uint64_t r = ((1ull << d) - 1) + p;
    const uint32_t w = 1u << (L - 1);
    uint8_t lab = DONE;
    Digest dg{{0, 0, 0, 0}};
    if (threadIdx.x < w) {
      const uint64_t n = (r + 1) * w - 1 + threadIdx.x, c = 2 * n + 1;
      const uint8_t ll = __ldcg(a.labels + c), lr = __ldcg(a.labels + c + 1);
      Digest dl{{0, 0, 0, 0}}, dr{{0, 0, 0, 0}};
      if (BASE || (ll == lr && digest_wanted(pass, ll))) {
        const uint4 vl = __ldcg(reinterpret_cast<const uint4*>(a.tree + c)),
                    vr = __ldcg(reinterpret_cast<const uint4*>(a.tree + c + 1));
        dl = Digest{{vl.x, vl.y, vl.z, vl.w}};
        dr = Digest{{vr.x, vr.y, vr.z, vr.w}};
      }
      sink_level(sink, r, (int)L - 1);
      lab = span_node<HK, BASE>(a, pass, (uint32_t)n, ll, lr, dl, dr, dg, L == 1, sink);
    }
    upper_levels<HK, BASE>(a, pass, r, L, lab, dg, sink, top8, topdg);
    if (!BASE && pass != 1) flush_sink(a, fused, r, sink, base);
    __syncthreads();
    done += 1ull << d;
    i = p;
  }
}

// Byte-parallel labelling of four (left, right) pairs per 32-bit word, the
// rules of span_node: P receives the parents' labels, FL / FR the children's
// root flags (duplicate passes), XF the pairs to hash and insert
// (first-occurrence passes), XS the pairs to hash and look up (duplicate
// passes; their parents read SHIFT_DUPL until resolved).  Bytes are 0xff in
// the X masks.
constexpr uint32_t kB1 = 0x01010101u;
__device__ __forceinline__ uint32_t child_flags4(uint32_t x) {
  const uint32_t sh = __vcmpeq4(x, SHIFT_DUPL * kB1);
  const uint32_t none = __vcmpeq4(x, FIXED_DUPL * kB1) | __vcmpeq4(x, DONE * kB1);
  return (sh & (ROOT_SHIFT * kB1)) | (~sh & ~none & (ROOT_FO * kB1));
}
__device__ __forceinline__ void label_pairs4(int pass, uint32_t L, uint32_t R, uint32_t& P, uint32_t& FL,
                                             uint32_t& FR, uint32_t& XF, uint32_t& XS) {
  const uint32_t eq = __vcmpeq4(L, R);
  const uint32_t fo = eq & __vcmpeq4(L, FIRST_OCUR * kB1);
  P = (DONE * kB1) & ~fo;  // FIRST_OCUR is 0
  FL = FR = XS = 0;
  XF = pass != 1 ? fo : 0;
  if (pass != 0) {
    const uint32_t fix = eq & __vcmpeq4(L, FIXED_DUPL * kB1);
    const uint32_t sh = eq & __vcmpeq4(L, SHIFT_DUPL * kB1);
    P = (P & ~(fix | sh)) | (fix & (FIXED_DUPL * kB1)) | (sh & (SHIFT_DUPL * kB1));
    FL = ~eq & child_flags4(L);
    FR = ~eq & child_flags4(R);
    XS = sh;
  }
}
__device__ __forceinline__ void set_byte(uint32_t& w, int b, uint32_t v) {
  w = (w & ~(0xffu << (8 * b))) | (v << (8 * b));
}

// A thread's four levels below node (r+1)*256-1+t when its 8 nodes on the
// deepest interior level are all interior: the 16 children's labels in c[4]
// (byte j = child j).  Returns the label of the thread's top node and its
// digest in dg when a parent reads it.
template <int HK, bool BASE>
__device__ __forceinline__ uint8_t thread_levels_bytewise(const ForestArgs& a, int pass, uint64_t r, uint32_t t,
                                                          uint32_t c[4], IdSink& sink, Digest (*work)[256],
                                                          Digest& dg) {
  uint64_t nb = (r + 1) * 2048 - 1 + 8ull * t;  // first parent of the level
#pragma unroll 1
  for (int lvl = 0; lvl < 4; lvl++) {
    uint32_t P[2], FL[2], FR[2], XF[2], XS[2];
    sink_level(sink, r, (int)kBottomLevels - 1 - lvl);
#pragma unroll
    for (int q = 0; q < 2; q++)
      label_pairs4(pass, __byte_perm(c[2 * q], c[2 * q + 1], 0x6420), __byte_perm(c[2 * q], c[2 * q + 1], 0x7531),
                   P[q], FL[q], FR[q], XF[q], XS[q]);
    // pairs that hash: ascending, so work[i] is written after its children
    // work[2i], work[2i+1] of the level below were read
#pragma unroll
    for (int q = 0; q < 2; q++) {
      uint32_t X = XF[q] | XS[q];
      if (BASE) X = lvl == 0 ? ~0u : q == 1 ? 0u : lvl == 1 ? ~0u : lvl == 2 ? 0xffffu : 0xffu;  // every node
      while (X) {
        const int b = (__ffs(X) - 1) >> 3;
        X &= ~(0xffu << (8 * b));
        const uint32_t i = 4 * q + b;
        const uint64_t n = nb + i;
        Digest dl, dr;
        if (lvl == 0) {
          dl = ld_digest(a.tree + 2 * n + 1);
          dr = ld_digest(a.tree + 2 * n + 2);
        } else {
          dl = work[2 * i][t];
          dr = work[2 * i + 1][t];
        }
        const Digest d = hash_pair(HK, dl, dr);
        if (BASE) {
          if ((XS[q] >> (8 * b)) & 1) {
            if (map_find(a.map, Digest{{0, 0, 0, 0}}, a.err) >= 0) {
              atomicOr(a.zero_found, 1u);
            } else {
              set_byte(P[q], b, DONE);
              set_byte(FL[q], b, ROOT_SHIFT);
              set_byte(FR[q], b, ROOT_SHIFT);
            }
          }
          st_digest(a.tree + n, d);
          a.labels[n] = (uint8_t)(P[q] >> (8 * b));
          work[i][t] = d;
          continue;
        }
        st_digest(a.tree + n, d);
        if ((XF[q] >> (8 * b)) & 1) {
          queue_insert(sink, (uint32_t)n);
          work[i][t] = d;
        } else if (map_find(a.map, d, a.err) >= 0) {
          work[i][t] = d;  // parent stays SHIFT_DUPL
        } else {
          set_byte(P[q], b, DONE);
          set_byte(FL[q], b, ROOT_SHIFT);
          set_byte(FR[q], b, ROOT_SHIFT);
        }
      }
    }
    // children's root flags, children in order at consecutive canonical positions
    if ((FL[0] | FR[0] | FL[1] | FR[1]) != 0) {
      const uint64_t cp0 = canon_pos(a, (uint32_t)(2 * nb + 1));
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const uint32_t f4[2] = {__byte_perm(FL[q], FR[q], 0x5140), __byte_perm(FL[q], FR[q], 0x7362)};
#pragma unroll
        for (int k = 0; k < 2; k++) {
          uint32_t f = f4[k];
          while (f) {
            const int b = (__ffs(f) - 1) >> 3;
            a.rflag[cp0 + 8 * q + 4 * k + b] = (uint8_t)(f >> (8 * b));
            f &= ~(0xffu << (8 * b));
          }
        }
      }
    }
    c[0] = P[0];
    c[1] = P[1];
    c[2] = c[3] = DONE * kB1;  // pairs past the level's width: DONE, no flags
    nb = (nb - 1) / 2;
  }
  const uint8_t lab = (uint8_t)c[0];
  if (BASE || digest_wanted(pass, lab)) dg = work[0][t];
  return lab;
}

// A pass over a tree of more than kSmallLeaves leaves.  Bottom span: 12 levels,
// 4096 leaves per block.  Each thread reads the labels of its 16 children with
// one aligned 16-byte load (the first byte comes from the lane before) and
// computes its 8, 4, 2 and 1 nodes in a loop, labels packed in a 64-bit word,
// digests in shared memory; a thread whose 16 children are all unchanged
// (fixed duplicates) has nothing to hash, flag or insert.  upper_levels does
// the rest of the span, upper_spans the rest of the tree.  Loops rather than
// unrolled levels keep the kernel small enough for the instruction cache.
// The duplicate pass (1) has nothing left to do when the passes were fused: it
// is launched as one wave, whose blocks return or take several subtrees.
template <int HK, bool BASE>
__global__ void __launch_bounds__(256) forest_kernel(ForestArgs a, int pass, uint32_t N, uint32_t d_top,
                                                     uint32_t count) {
  pdl_enter();
  __shared__ uint8_t top8[8];
  __shared__ Digest topdg[8];
  __shared__ uint16_t ids[BASE ? 1 : 4096];
  __shared__ uint32_t ids_n, ids_base, s_last;
  __shared__ Digest work[8][256];  // [node of the thread's level][thread]: 16-byte lanes, no bank conflicts
  const bool fused = forest_fused(a);
  if (fused) {
    if (pass == 1) return;
    pass = 2;
  }
  const uint64_t last_interior = (uint64_t)N - 2, M = 2ull * N - 1;
  const uint32_t t = threadIdx.x, lane = t & 31;
  constexpr unsigned kFull = 0xffffffffu;
  if (t == 0) ids_n = 0;
  __syncthreads();
  IdSink sink{ids, &ids_n, 0};
#pragma unroll 1
  for (uint32_t blk = blockIdx.x; blk < count; blk += gridDim.x) {
    const uint64_t r = ((1ull << d_top) - 1) + blk;
    // children (relative depth 12) cb .. cb+15; cb + 1 is a multiple of 16
    const uint64_t cb = (r + 1) * 4096 - 1 + 16ull * t;
    uint4 v;
    if (cb + 17 <= M) {
      v = *reinterpret_cast<const uint4*>(a.labels + cb + 1);
    } else {
      uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 16; j++) {
        const uint64_t c = cb + 1 + j;
        w[j >> 2] |= (uint32_t)(c < M ? a.labels[c] : DONE) << (8 * (j & 3));
      }
      v = make_uint4(w[0], w[1], w[2], w[3]);
    }
    uint32_t first = __shfl_up_sync(kFull, v.w, 1) >> 24;  // byte 15 of the lane before = child cb
    if (lane == 0) first = cb < M ? a.labels[cb] : DONE;
    // child j's label is byte j of (lo, hi)
    uint64_t lo = ((uint64_t)((v.y << 8) | (v.x >> 24)) << 32) | ((v.x << 8) | first);
    uint64_t hi = ((uint64_t)((v.w << 8) | (v.z >> 24)) << 32) | ((v.y >> 24) | (v.z << 8));
    const uint64_t nb1 = (r + 1) * 2048 - 1 + 8ull * t;  // relative depth 11: the deepest interior level
    uint8_t lab;
    Digest dg{{0, 0, 0, 0}};
    constexpr uint64_t kFixed8 = 0x0101010101010101ull * FIXED_DUPL;
    if (!BASE && lo == kFixed8 && hi == kFixed8 && nb1 + 7 <= last_interior) {
      lab = pass == 0 ? DONE : FIXED_DUPL;
    } else if (nb1 + 7 <= last_interior) {
      uint32_t c[4] = {(uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32)};
      lab = thread_levels_bytewise<HK, BASE>(a, pass, r, t, c, sink, work, dg);
    } else {
      uint64_t nb = nb1;
      uint32_t width = 8;
#pragma unroll 1
      for (int lvl = 0; lvl < 4; lvl++) {
        uint64_t out = 0;
        sink_level(sink, r, (int)kBottomLevels - 1 - lvl);
#pragma unroll 1
        for (uint32_t i = 0; i < width; i++) {
          const uint32_t j = 2 * i;
          const uint8_t ll = (uint8_t)((j < 8 ? lo >> (8 * j) : hi >> (8 * (j - 8))) & 0xff);
          const uint8_t lr = (uint8_t)((j + 1 < 8 ? lo >> (8 * (j + 1)) : hi >> (8 * (j - 7))) & 0xff);
          const uint64_t n = nb + i;
          Digest dl{{0, 0, 0, 0}}, dr{{0, 0, 0, 0}}, d{{0, 0, 0, 0}};
          if (BASE || (ll == lr && digest_wanted(pass, ll))) {
            if (lvl == 0) {
              if (n <= last_interior) {
                dl = ld_digest(a.tree + 2 * n + 1);
                dr = ld_digest(a.tree + 2 * n + 2);
              }
            } else {
              dl = work[j][t];
              dr = work[j + 1][t];
            }
          }
          const uint8_t l = lvl == 0 ? span_label<HK, BASE>(a, pass, n, last_interior, M, ll, lr, dl, dr, d, sink)
                                     : span_node<HK, BASE>(a, pass, (uint32_t)n, ll, lr, dl, dr, d, false, sink);
          // read back only at the next level, from a higher index
          if (BASE || digest_wanted(pass, l)) work[i][t] = d;
          out |= (uint64_t)l << (8 * i);
          if (lvl == 3) dg = d;
        }
        lo = out;
        hi = 0;
        nb = (nb - 1) / 2;  // parent of the level's first node
        width >>= 1;
      }
      lab = (uint8_t)lo;
    }
    upper_levels<HK, BASE>(a, pass, r, kSpanLevels, lab, dg, sink, top8, topdg);
    if (!BASE && pass != 1) flush_sink(a, fused, r, sink, &ids_base);
    upper_spans<HK, BASE>(a, pass, fused, d_top, blk, sink, &ids_base, top8, topdg, &s_last);
    __syncthreads();
  }
}

// A pass over a tree of at most kSmallLeaves leaves, by one block: labels in
// shared memory, a barrier per level.
template <int HK, bool BASE>
__global__ void __launch_bounds__(512) forest_small_kernel(ForestArgs a, int pass, uint32_t N, uint32_t dmax) {
  pdl_enter();
  __shared__ uint8_t lab[2 * kSmallLeaves];
  __shared__ uint16_t ids[BASE ? 1 : kSmallLeaves];
  __shared__ uint32_t ids_n, ids_base;
  const bool fused = forest_fused(a);
  if (fused) {
    if (pass == 1) return;
    pass = 2;
  }
  if (threadIdx.x == 0) ids_n = 0;
  for (uint32_t n = N - 1 + threadIdx.x; n < 2 * N - 1; n += blockDim.x) lab[n] = a.labels[n];
  __syncthreads();
  IdSink sink{ids, &ids_n, 0};
  for (int d = (int)dmax; d >= 0; d--) {
    const uint32_t first = (1u << d) - 1, last = min(2 * first, N - 2);
    sink_level(sink, 0, d);
    for (uint32_t n = first + threadIdx.x; n <= last; n += blockDim.x) {
      const uint8_t ll = lab[2 * n + 1], lr = lab[2 * n + 2];
      Digest dl{{0, 0, 0, 0}}, dr{{0, 0, 0, 0}}, dg;
      if (BASE || (ll == lr && digest_wanted(pass, ll))) {
        dl = ld_digest(a.tree + 2 * n + 1);
        dr = ld_digest(a.tree + 2 * n + 2);
      }
      lab[n] = span_node<HK, BASE>(a, pass, n, ll, lr, dl, dr, dg, d == 0, sink);
    }
    __syncthreads();
  }
  if (!BASE && pass != 1) flush_sink(a, fused, 0, sink, &ids_base);
}

// The queued first-occurrence inserts of a fused pass, one thread per node, by
// nblk blocks.
__device__ __forceinline__ void drain_inserts(const GatherArgs& g, uint32_t blk, uint32_t nblk) {
  const uint32_t n = *g.ins_count;
  const uint32_t cur_id = g.sp->cur, epoch_fo = g.sp->epoch + 1;
  uint32_t created = 0;
  for (uint32_t k = blk * blockDim.x + threadIdx.x; k < n; k += nblk * blockDim.x) {
    const uint32_t node = g.ins_queue[k];
    created += map_insert_owner(g.map, ld_digest(g.digests + node), node, cur_id, epoch_fo, g.err);
  }
  count_new_entries(g.map, created);
}
// After pass 3: every interior node's digest into the map.  First occurrences
// carry the first pass's epoch, the others the second's, among which equal
// digests abound (runs of equal chunks): those of a warp insert once.  Bound by the
// random accesses (two operations on each line).
__global__ void __launch_bounds__(256) forest_insert_all_kernel(ForestArgs a, int when, uint32_t n_interior) {
  pdl_enter();
  if (when != INSERT_ALWAYS && (*a.zero_found != 0) != (when == INSERT_IF_ZERO)) return;
  const uint32_t cur_id = a.sp->cur, epoch = a.sp->epoch;
  const uint32_t lane = threadIdx.x & 31;
  uint32_t created = 0;
  for (uint64_t nw = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); nw < n_interior;
       nw += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t n = (uint32_t)nw + lane;
    const bool in = nw + lane < n_interior;
    const bool fo = in && a.labels[n] == FIRST_OCUR;
    Digest d{{0, 0, 0, 0}};
    if (in) d = ld_digest(a.tree + n);
    if (fo) created += map_insert_owner(a.map, d, n, cur_id, epoch + 1, a.err);
    if (__any_sync(0xffffffffu, in && !fo))
      created += warp_insert_serial(a.map, in && !fo, d, n, cur_id, epoch + 2, a.err);
  }
  count_new_entries(a.map, created);
}
// ---------------------------------------------------------------------------
// Root compaction in serial push order, and what the diff's layout needs to
// know of each root.  Tree: the flag bytes lie at canonical positions, so the
// lists are a stable compaction of one byte array.  List and basic: the same of
// the chunks' labels.
//
// From here to the finished diff there are four launches, each a chain of a few
// dependent accesses, so the time is mostly latency and launches: 64 MiB in
// 128-byte chunks spent 44 us of an increment in the eleven launches (counts,
// roots, lookups, region sums, layout, metadata, four for the sort, copy,
// results) that these replace.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t node_at(const RootOrder& a, uint64_t p) {
  if (a.ascending) return (uint32_t)p + 1;
  if (p < a.sizeD) return (uint32_t)(((1ull << a.D) - 1) + p);
  // levels D-1, D-2, ... follow with sizes 2^(D-1), 2^(D-2), ...: position q
  // past level D lies on level d with x = 2^D - q in (2^d, 2^(d+1)]
  const uint64_t x = (1ull << a.D) - (p - a.sizeD);
  const int d = 63 - __clzll((long long)(x - 1));
  return (uint32_t)(((1ull << d) - 1) + ((2ull << d) - x));
}

// 16 contiguous flags per thread, 8 Ki flags per tile: a tile's roots are
// looked up by its block, so many small tiles keep a dense diff's lookups
// spread over the GPU.
constexpr uint64_t kRootPerThread = 16;
constexpr uint64_t kRootTile = kRootPerThread * kScanThreads;
constexpr uint32_t kRootReduceTiles = 4096;  // up to here blocks sum the tiles before theirs

// Masks (0x01 per byte) of the first occurrences and shifted duplicates among
// four flags or labels.
template <int APPROACH>
__device__ __forceinline__ void kinds4(uint32_t w, uint32_t& fo, uint32_t& sh) {
  constexpr uint32_t one = 0x01010101u;
  if (APPROACH == APPROACH_TREE) {
    static_assert(ROOT_FO == 1 && ROOT_SHIFT == 2, "flag bytes told apart by bit");
    fo = w & one;
    sh = (w >> 1) & one;
  } else if (APPROACH == APPROACH_LIST) {
    fo = __vcmpeq4(w, FIRST_OCUR * one) & one;
    sh = __vcmpeq4(w, SHIFT_DUPL * one) & one;
  } else {
    fo = __vcmpeq4(w, one) & one;
    sh = 0;
  }
}

// The thread's 16 flags at p (a multiple of 16; the arrays are padded to whole
// words): masks per word, none at or past n.
template <int APPROACH>
__device__ __forceinline__ uint64_t load_kinds(const uint8_t* f, uint64_t p, uint64_t n, uint32_t fo[4], uint32_t sh[4]) {
  uint64_t c = 0;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (p < n) v = *reinterpret_cast<const uint4*>(f + p);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    kinds4<APPROACH>(w[q], fo[q], sh[q]);
    const uint64_t at = p + 4 * q;
    const uint32_t in = at + 4 <= n ? ~0u : at >= n ? 0u : (1u << (8 * (uint32_t)(n - at))) - 1;
    fo[q] &= in;
    sh[q] &= in;
    c += (uint64_t)__popc(fo[q]) | ((uint64_t)__popc(sh[q]) << 32);
  }
  return c;
}

// Block-wide: exclusive prefix in place over n words, their total returned.
__device__ __forceinline__ uint64_t scan_in_place(uint64_t* v, uint32_t n, uint64_t* sh) {
  const uint32_t per = (n + blockDim.x - 1) / blockDim.x;
  const uint32_t lo = min(threadIdx.x * per, n), hi = min(lo + per, n);
  uint64_t s = 0;
  for (uint32_t i = lo; i < hi; i++) s += __ldcg(v + i);
  uint64_t total;
  uint64_t ex = block_excl_scan(s, sh, &total);
  for (uint32_t i = lo; i < hi; i++) {
    const uint64_t x = __ldcg(v + i);
    v[i] = ex;
    ex += x;
  }
  return total;
}

// True in every thread of the last block of a part of `nblocks` blocks to get
// here; what the others wrote before is visible to it past the L1.
__device__ __forceinline__ bool last_block(uint32_t* done, uint32_t nblocks, uint32_t* s_last) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    *s_last = atomicAdd(done, 1u) + 1 == nblocks ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  return *s_last != 0;
}

// Flags per tile, packed as (shift << 32) | fo.  The root itself is pushed only
// for N >= 2 in the incremental and baseline passes
// (src/tree_approach.cpp:384-393); the serial reference inserts it whenever it
// is a first occurrence (include/reference_impl.hpp:105-106).
template <int APPROACH>
__global__ void __launch_bounds__(kScanThreads) root_count_kernel(GatherArgs g) {
  pdl_enter();
  __shared__ uint64_t sh[33];
  if (APPROACH == APPROACH_BASIC) stamp(g.clk, CLK_LEAVES_DONE);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const bool root = APPROACH == APPROACH_TREE && g.labels[0] == FIRST_OCUR && (g.order.ascending || g.N >= 2);
    g.lay->root_fo = root ? 1 : 0;
    if (root) g.fo_list[0] = 0;
  }
  const uint64_t p = (uint64_t)blockIdx.x * kRootTile + (uint64_t)threadIdx.x * kRootPerThread;
  uint32_t fo[4], shf[4];
  const uint64_t c = load_kinds<APPROACH>(g.flags, p, g.n_flags, fo, shf);
  uint64_t total;
  block_excl_scan(c, sh, &total);
  if (threadIdx.x == 0) g.tile_counts[blockIdx.x] = total;
}

// First-occurrence root: (1 << 32) | chunks if it owns its digest, else 0.  A
// first-occurrence leaf owns its digest: the leaf pass demotes every other one
// (same checkpoint id, another owner).  The inserts of a fused pass may still
// wait: a digest that is not in the map then is the root's own.  In a baseline
// of an empty map every first occurrence owns its digest: its leaves own
// theirs, and no second pair of the same leaves is a first occurrence.  The
// inserts check both (map_insert_owner).
__device__ __forceinline__ uint64_t fo_region(const GatherArgs& g, uint32_t node, bool fused, uint32_t cur) {
  bool owner = node >= g.N - 1 || g.all_own;
  if (!owner) {
    const int64_t slot = map_find(g.map, ld_digest(g.digests + node), g.err);
    const NodeIdDev prev = slot_value(g.map, slot);
    owner = slot < 0 ? fused : prev.node == node && prev.tree == cur;
  }
  return owner ? (1ull << 32) | num_leaf_descendents(node, g.M) : 0;
}

// One block, once every root is listed: repeat-count table, layout, header; bin
// representatives for the list approach's BinOp1D.  The tiles' region sums
// become offsets in place.
template <int APPROACH>
__device__ void build_layout(const GatherArgs& g, uint32_t ntiles, uint64_t* sh) {
  volatile Layout* lay = g.lay;
  const uint32_t F = lay->F, S = lay->S;
  uint64_t regions = ((uint64_t)F << 32) | F;  // list / basic: one chunk per entry
  if (APPROACH == APPROACH_TREE) regions = scan_in_place(g.tile_regions, ntiles, sh);
  const uint32_t nd = (uint32_t)(regions >> 32), chunks = (uint32_t)regions;
  const uint32_t cur = g.sp->cur;
  const uint32_t K = cur + 1, tid = threadIdx.x, nt = blockDim.x;
  constexpr bool kMeta = APPROACH != APPROACH_BASIC;
  // P = number of source checkpoints that occur; max_key = largest of them
  __shared__ uint32_t smax;
  if (tid == 0) smax = 0;
  __syncthreads();
  uint32_t P = 0;
  if (kMeta && S)
    for (uint32_t b = 0; b < K; b += nt) {
      const uint32_t k = b + tid;
      const bool nz = k < K && __ldcg(g.hist + k) > 0;
      P += (uint32_t)__syncthreads_count(nz);
      if (nz) atomicMax(&smax, k);
    }
  __syncthreads();
  const uint32_t max_key = smax;
  const uint64_t fo_off = 32;
  const uint64_t data_off = fo_off + 4ull * F + (kMeta ? 8ull * P + 8ull * S : 0);
  const uint64_t pad = (16 - (data_off & 15)) & 15;
  const uint64_t diff_len = data_off + (uint64_t)chunks * g.cs;
  const bool ok = pad + diff_len <= g.stage_cap;
  const uint64_t table_off = fo_off + 4ull * nd;
  // sort representative of each key: stable sort by BinOp1D bin equals stable
  // sort by the smallest key sharing the bin
  const uint32_t nbins = APPROACH == APPROACH_TREE ? cur : S;
  const double range = (double)(APPROACH == APPROACH_TREE ? cur : max_key);
  const bool plain = range <= (double)nbins;  // every key is its own bin
  uint8_t* diff = g.stage + pad;
  if (tid == 0) {
    lay->num_distinct = nd;
    lay->chunk_counter = chunks;
    lay->P = P;
    lay->pad = pad;
    lay->data_off = data_off;
    lay->table_off = table_off;
    lay->pairs_off = table_off + 8ull * P;
    lay->nkeys = plain ? P : 0;
    lay->sort_n = 0;
    lay->sort_tiles = 0;
    lay->diff_len = ok ? diff_len : 0;
    lay->ok = ok ? 1 : 0;
    if (!ok) atomicOr(g.err, DERR_CAPACITY);
    // datasizes as the reference's collect_diff returns them
    if (APPROACH == APPROACH_TREE) {
      const uint64_t meta = 4ull * F + 8ull * P + 8ull * S;
      lay->size_data = diff_len - meta;  // src/tree_approach.cpp:707-709
      lay->size_meta = meta;
    } else {
      // src/list_approach.cpp:241-246; src/basic_approach.cpp:141-142 (32-bit product)
      const uint64_t dsz = APPROACH == APPROACH_LIST ? (uint64_t)g.cs * F : (uint64_t)(uint32_t)(F * g.cs);
      lay->size_data = dsz;
      lay->size_meta = diff_len - dsz;
    }
    if (ok) {
      // header_t, include/utils.hpp:29-37
      uint32_t* h32 = reinterpret_cast<uint32_t*>(diff);
      h32[0] = g.sp->baseline_id;
      h32[1] = cur;
      h32[2] = (uint32_t)g.len;
      h32[3] = (uint32_t)(g.len >> 32);
      h32[4] = g.cs;
      h32[5] = F;
      h32[6] = P;
      h32[7] = kMeta ? S : 0;
    }
  }
  if (!kMeta) return;
  // zero bytes that the reference leaves at zero when F != num_distinct
  if (ok)
    for (uint64_t b = 32 + 4ull * nd + 8ull * P + 8ull * S + tid; b < data_off; b += nt) diff[b] = 0;
  if (!S) return;
  // (checkpoint id, count) table in ascending id (src/tree_approach.cpp:657-665),
  // each key's dense index, and the histogram cleared for the next checkpoint
  uint32_t base = 0;
  for (uint32_t b = 0; b < K; b += nt) {
    const uint32_t k = b + tid;
    const uint32_t h = k < K ? __ldcg(g.hist + k) : 0;
    uint64_t t;
    const uint32_t at = base + (uint32_t)block_excl_scan(h > 0 ? 1 : 0, sh, &t);
    if (h > 0) {
      if (ok) {
        uint32_t* e = reinterpret_cast<uint32_t*>(diff + table_off + 8ull * at);
        e[0] = k;
        e[1] = h;
      }
      g.hist[k] = 0;
    }
    if (k < K) {
      if (plain) {
        g.rep[k] = at;
      } else {
        const double mul = (double)nbins / range;
        const int bk = (int)(mul * (double)k);
        // the bin's smallest key: bins ascend with the keys, so it lies next to
        // bk / mul (stepping down from k took most of a 1.6 ms list series with
        // few shift entries after some thousand checkpoints; now 0.29 ms)
        uint32_t rep = min(k, (uint32_t)((double)bk / mul));
        while (rep > 0 && (int)(mul * (double)(rep - 1)) == bk) rep--;
        while ((int)(mul * (double)rep) < bk) rep++;
        g.rep[k] = rep | (h > 0 ? 0x80000000u : 0u);
        g.rank[k] = 0;
      }
    }
    base += (uint32_t)t;
  }
  uint32_t nkeys = P;
  if (!plain) {
    // dense index of each representative that some present key maps to
    __syncthreads();
    for (uint32_t k = tid; k < K; k += nt)
      if (g.rep[k] >> 31) g.rank[g.rep[k] & 0x7fffffffu] = 1;
    __syncthreads();
    nkeys = 0;
    for (uint32_t b = 0; b < K; b += nt) {
      const uint32_t k = b + tid;
      const uint64_t v = k < K ? __ldcg(g.rank + k) : 0;
      uint64_t t;
      const uint64_t ex = block_excl_scan(v, sh, &t);
      if (k < K) g.rank[k] = nkeys + (uint32_t)ex;
      nkeys += (uint32_t)t;
    }
    __syncthreads();
    for (uint32_t k = tid; k < K; k += nt)
      if (g.rep[k] >> 31) g.rep[k] = __ldcg(g.rank + (g.rep[k] & 0x7fffffffu));
  }
  if (tid == 0) {
    const uint32_t T = (S + kSortTile - 1) / kSortTile;
    lay->nkeys = nkeys;
    lay->sort_tiles = T;
    lay->sort_n = nkeys * T;
    if (nkeys > kSortFastKeys) atomicOr(g.err, DERR_SORTKEYS);
  }
}

// Emits the roots in serial push order (the tile offset is the sum of the
// earlier tiles' counts, or with kReduce false a scanned offset: a block that
// scans them for the others takes 2-6 us longer), clears the flags, and looks up the tile's own roots: region sizes of the first
// occurrences, prefixed within the tile, and (source checkpoint, source node)
// of the shifted duplicates with a histogram of their sources (warp-aggregated:
// most share a few).  The last block lays the diff out.
template <int APPROACH, bool kReduce>
__global__ void __launch_bounds__(kScanThreads) root_emit_kernel(GatherArgs g) {
  pdl_enter();
  stamp(g.clk, CLK_ROOTS_DONE);
  __shared__ uint64_t sh[33];
  __shared__ uint32_t s_last;
  constexpr bool kTree = APPROACH == APPROACH_TREE;
  const uint32_t tile = blockIdx.x, tid = threadIdx.x;
  const uint64_t p = (uint64_t)tile * kRootTile + (uint64_t)tid * kRootPerThread;
  uint32_t fo[4], shf[4];
  const uint64_t c = load_kinds<APPROACH>(g.flags, p, g.n_flags, fo, shf);
  uint64_t off = 0;
  if (kReduce) {
    uint64_t part = 0;
    for (uint32_t k = tid; k < tile; k += blockDim.x) part += g.tile_counts[k];
    block_excl_scan(part, sh, &off);
  } else {
    off = g.tile_counts[tile];
  }
  uint64_t total;
  uint64_t ex = block_excl_scan(c, sh, &total) + off;
  const uint32_t root = g.lay->root_fo;
  if (tile == gridDim.x - 1 && tid == 0) {
    g.lay->F = root + (uint32_t)(off + total);
    g.lay->S = (uint32_t)((off + total) >> 32);
  }
  if (c) {
    // cleared for the next checkpoint
    if (kTree) *reinterpret_cast<uint4*>(g.flags + p) = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      uint32_t w = fo[q] | shf[q];
      while (w) {
        const int bit = __ffs(w) - 1;  // byte order = serial order
        const uint64_t pos = p + 4 * q + (bit >> 3);
        const uint32_t id = kTree ? node_at(g.order, pos) : (uint32_t)pos;
        if ((fo[q] >> bit) & 1) { g.fo_list[root + (uint32_t)ex] = id; ex += 1; }
        else { g.sh_list[(uint32_t)(ex >> 32)] = id; ex += 1ull << 32; }
        w &= w - 1;
      }
    }
  }
  __syncthreads();
  const uint32_t cur = g.sp->cur;
  if (kTree) {
    // the tile's first occurrences, the root ahead of tile 0's
    const bool fused = g.fuse_gate && *g.fuse_gate == 0;
    const uint32_t f0 = tile == 0 ? 0 : root + (uint32_t)off, f1 = root + (uint32_t)off + (uint32_t)total;
    uint64_t carry = 0;
    for (uint32_t b = f0; b < f1; b += blockDim.x) {
      const uint32_t i = b + tid;
      const uint64_t v = i < f1 ? fo_region(g, g.fo_list[i], fused, cur) : 0;
      uint64_t t;
      const uint64_t before = carry + block_excl_scan(v, sh, &t);
      if (i < f1) {
        g.fo_val[i] = before | (v ? 1ull << 63 : 0);
        g.fo_tile[i] = tile;
      }
      carry += t;
    }
    if (tid == 0) g.tile_regions[tile] = carry;
  }
  if (APPROACH != APPROACH_BASIC) {
    const uint32_t s0 = (uint32_t)(off >> 32), s1 = s0 + (uint32_t)(total >> 32);
    const uint32_t lane = tid & 31;
    for (uint32_t b = s0; b < s1; b += blockDim.x) {
      const uint32_t i = b + tid;
      uint32_t key = 0xffffffffu;
      if (i < s1) {
        const int64_t slot = map_find(g.map, ld_digest(g.digests + g.sh_list[i]), g.err);
        NodeIdDev prev = slot_value(g.map, slot);
        if (slot < 0 || prev.tree > cur) { atomicOr(g.err, DERR_MISSING); prev.tree = 0; prev.node = 0; }
        g.sh_key[i] = prev.tree;
        g.sh_prev[i] = prev.node;
        key = prev.tree;
      }
      const uint32_t peers = __match_any_sync(0xffffffffu, key);
      if (key != 0xffffffffu && lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&g.hist[key], (uint32_t)__popc(peers));
    }
  }
  if (last_block(g.counters + COUNT_ROOTS_DONE, gridDim.x, &s_last)) build_layout<APPROACH>(g, gridDim.x, sh);
}

// ---------------------------------------------------------------------------
// Diff assembly
// ---------------------------------------------------------------------------
// First-occurrence entries: metadata and regions, by entry.
__device__ __forceinline__ void emit_regions(const GatherArgs& g, uint32_t blk, uint32_t nblk) {
  const uint32_t F = g.lay->F;
  const bool ok = g.lay->ok;
  uint8_t* meta = g.stage + g.lay->pad + 32;
  for (uint64_t i = (uint64_t)blk * blockDim.x + threadIdx.x; i < F; i += (uint64_t)nblk * blockDim.x) {
    const uint32_t node = g.fo_list[i];
    uint32_t r = (uint32_t)i, slot = (uint32_t)i, chunk = node;
    if (g.approach == APPROACH_TREE) {
      const uint64_t v = g.fo_val[i];
      if (!(v >> 63)) continue;
      const uint64_t ex = (v & ~(1ull << 63)) + g.tile_regions[g.fo_tile[i]];
      r = (uint32_t)(ex >> 32);
      slot = (uint32_t)ex;
      chunk = leftmost_leaf(node, g.M) - (g.N - 1);
    }
    g.reg_slot[r] = slot;
    g.reg_chunk[r] = chunk;
    // FO metadata: node ids (tree) or chunk ids (list, basic), 4-byte aligned
    if (ok) *reinterpret_cast<uint32_t*>(meta + 4ull * r) = node;
  }
}

// Stable counting sort of the shift entries by representative key.
// Tile t counts its keys; matrix[key * T + t] (key-major).
__device__ __forceinline__ void sort_count(const GatherArgs& g, uint32_t blk, uint32_t nblk, uint32_t* cnt) {
  const uint32_t K = g.lay->nkeys, S = g.lay->S, T = g.lay->sort_tiles;
  if (K > kSortFastKeys) return;
  for (uint32_t t = blk; t < T; t += nblk) {
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    const uint64_t b = (uint64_t)t * kSortTile;
    // every load of the tile issued before the first count
    constexpr int kPer = kSortTile / 256;
    uint32_t key[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const uint64_t i = b + threadIdx.x + 256ull * j;
      key[j] = i < S ? g.sh_key[i] : 0xffffffffu;
    }
#pragma unroll
    for (int j = 0; j < kPer; j++) key[j] = key[j] != 0xffffffffu ? g.rep[key[j]] : 0xffffffffu;
#pragma unroll
    for (int j = 0; j < kPer; j++)
      if (key[j] != 0xffffffffu) atomicAdd(&cnt[key[j]], 1u);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) g.sort_mat[(uint64_t)k * T + t] = cnt[k];
    __syncthreads();
  }
}

// Metadata and regions (the first n_emit blocks) beside the sort's counts (the
// others, whose last block turns the counts into positions unless the matrix
// is large: sort_scan false).
__global__ void __launch_bounds__(256) emit_count_kernel(GatherArgs g) {
  pdl_enter();
  extern __shared__ uint32_t cnt[];
  __shared__ uint64_t sh[33];
  __shared__ uint32_t s_last;
  if (blockIdx.x < g.n_emit) {
    emit_regions(g, blockIdx.x, g.n_emit);
    return;
  }
  const uint32_t nblk = gridDim.x - g.n_emit;
  sort_count(g, blockIdx.x - g.n_emit, nblk, cnt);
  if (g.sort_scan && last_block(g.counters + COUNT_SORT_DONE, nblk, &s_last) && g.lay->nkeys <= kSortFastKeys)
    scan_in_place(g.sort_mat, g.lay->sort_n, sh);
}

struct MatVal {
  const uint64_t* m;
  __device__ __forceinline__ uint64_t operator()(uint64_t i) const { return m[i]; }
};
struct MatEmit {
  uint64_t* m;
  __device__ __forceinline__ void operator()(uint64_t i, uint64_t ex, uint64_t) const { m[i] = ex; }
};
// Stable placement of the shift entries of one 4096-entry tile: 8 warps each
// rank a contiguous 512-entry slice in order (per-warp key counters in shared
// memory), then the per-key counts of earlier warps and the tile's global
// base (key-major scan of sort_mat) give each entry its position.
constexpr int kSortWarps = 8;
struct SortShared {
  uint16_t keys[kSortTile], lrank[kSortTile];
};
static_assert(kSortFastKeys <= 0x10000 && kSortTile <= 0x10000, "keys and ranks kept in 16 bits");
__device__ __forceinline__ void sort_scatter(const GatherArgs& g, uint32_t blk, uint32_t nblk, SortShared& sm,
                                             uint32_t* cnt) {  // cnt: [kSortWarps][K]
  const uint32_t K = g.lay->nkeys, S = g.lay->S, T = g.lay->sort_tiles;
  if (!g.lay->ok || K > kSortFastKeys) return;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr uint32_t kSlice = kSortTile / kSortWarps;
  uint8_t* pairs = g.stage + g.lay->pad + g.lay->pairs_off;
  for (uint32_t t = blk; t < T; t += nblk) {
    const uint64_t b = (uint64_t)t * kSortTile;
    if (b >= S) break;
    const uint32_t n = (uint32_t)(S - b < kSortTile ? S - b : kSortTile);
    constexpr int kPer = kSortTile / 256;
    {
      uint32_t kk[kPer];
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + 256u * j;
        kk[j] = i < n ? g.sh_key[b + i] : 0;
      }
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + 256u * j;
        if (i < n) sm.keys[i] = (uint16_t)g.rep[kk[j]];
      }
    }
    for (uint32_t k = threadIdx.x; k < kSortWarps * K; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    uint32_t* wc = cnt + warp * K;
    for (uint32_t i0 = warp * kSlice; i0 < (warp + 1) * kSlice && i0 < n; i0 += 32) {
      const uint32_t i = i0 + lane;
      const bool v = i < n && i < (warp + 1) * kSlice;
      const uint32_t key = v ? sm.keys[i] : 0xffffffffu;
      const uint32_t peers = __match_any_sync(0xffffffffu, key);
      const uint32_t rank = __popc(peers & ((1u << lane) - 1));
      uint32_t base = v ? wc[key] : 0;
      __syncwarp();
      if (v) {
        sm.lrank[i] = (uint16_t)(base + rank);
        if (lane == (uint32_t)(__ffs(peers) - 1)) wc[key] = base + __popc(peers);
      }
      __syncwarp();
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) {
      uint32_t run = (uint32_t)g.sort_mat[(uint64_t)k * T + t];
      for (int w = 0; w < kSortWarps; w++) {
        uint32_t c = cnt[w * K + k];
        cnt[w * K + k] = run;
        run += c;
      }
    }
    __syncthreads();
    {
      uint32_t nd[kPer], pv[kPer];
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + 256u * j;
        nd[j] = i < n ? g.sh_list[b + i] : 0;
        pv[j] = i < n ? g.sh_prev[b + i] : 0;
      }
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        const uint32_t i = threadIdx.x + 256u * j;
        if (i >= n) continue;
        const uint32_t pos = cnt[(i / kSlice) * K + sm.keys[i]] + sm.lrank[i];
        uint32_t* e = reinterpret_cast<uint32_t*>(pairs + 8ull * pos);  // 4-byte aligned only
        e[0] = nd[j];
        e[1] = pv[j];
      }
    }
    __syncthreads();
  }
}

// Chunk gather into the data section.  Regions (reg_chunk, reg_slot) are
// sorted by slot; every 16-byte unit of the data section is written once, by
// one 16-byte store (the section starts on a 16-byte boundary).
//
// Bound by HBM (the chunks read once, written once).  A tile is 32 KiB of the
// data section, or 256 slots of chunks shorter than 128 bytes; a block owns a
// contiguous range of tiles, so it searches the region list once and then
// carries its position along.  Per tile the regions are staged in shared
// memory and every slot's chunk is found there once, so a unit costs a lookup
// in shared memory whatever the regions' lengths: threads that walked the
// list one region at a time took 372 us for 3.1 M regions of one 64-byte
// chunk and 1481 us for one region of 4 GiB, a search per byte 819 us for
// 64 MB in chunks of 100 bytes.
constexpr uint32_t kCopyTileUnits = 2048;
constexpr uint32_t kCopySlots = 256 + 2;  // slots that a tile can touch
constexpr int kCopyPer = 4;               // units in flight per thread

// Words of 16 bytes from address A: byte i of the result is the byte at A + i
// for i in [lo, hi).  Loads only aligned words that hold one of these bytes.
__device__ __forceinline__ uint4 load_window(uint64_t A, uint32_t lo, uint32_t hi) {
  const uint32_t d = (uint32_t)(A & 15);
  const uint4* w = reinterpret_cast<const uint4*>(A - d);
  uint4 w0 = make_uint4(0, 0, 0, 0), w1 = make_uint4(0, 0, 0, 0);
  if (lo + d < 16) w0 = __ldg(w);
  if (hi + d > 16) w1 = __ldg(w + 1);
  return cut16(w0, w1, d);
}
// mask of the bytes of word q (bytes 4q .. 4q + 3) that lie below n
__device__ __forceinline__ uint32_t bytes_below(int n, int q) {
  const int k = n - 4 * q;
  return k <= 0 ? 0u : k >= 4 ? ~0u : (1u << (8 * k)) - 1;
}

// kVec: chunks of whole 16-byte words from a 16-byte aligned buffer, one load
// per unit.  Otherwise a unit is cut out of the aligned words around each of
// its pieces (one piece, or two where it crosses into a slot of another
// region; more only for chunks shorter than 16 bytes).
struct CopyShared {
  uint32_t rs[kCopySlots + 1], rc[kCopySlots + 1], ch[kCopySlots];
  uint32_t r;     // region of the tile's first slot
  uint32_t j[2];  // region (from the tile's first) of the last slot, of the slot after it
};
template <bool kVec>
__device__ __forceinline__ void copy_tiles(const GatherArgs& g, uint32_t blk, uint32_t nblk, CopyShared& sm) {
  if (!g.lay->ok) return;
  const uint32_t R = g.lay->num_distinct;
  const uint64_t nslots = g.lay->chunk_counter;
  if (R == 0 || nslots == 0) return;
  uint32_t* rs = sm.rs;
  uint32_t* rc = sm.rc;
  uint32_t* ch = sm.ch;
  uint8_t* dst = g.stage + g.lay->pad + g.lay->data_off;
  const uint64_t cs = g.cs;
  const uint32_t tid = threadIdx.x;
  const uint64_t nbytes = nslots * cs;
  const uint64_t nunits = (nbytes + 15) / 16;
  const uint32_t ut = cs >= 128 ? kCopyTileUnits : 16 * (uint32_t)cs;
  const uint64_t ntiles = (nunits + ut - 1) / ut;
  const uint64_t per_block = (ntiles + nblk - 1) / nblk;
  const uint64_t tile0 = (uint64_t)blk * per_block;
  const uint64_t tile1 = tile0 + per_block < ntiles ? tile0 + per_block : ntiles;
  if (tile0 >= tile1) return;
  const int lg = (cs & (cs - 1)) == 0 ? __ffsll((long long)cs) - 1 : -1;
  // slot of byte x, counted from the tile's first slot (x < cs + 32 KiB: at
  // most one slot on for chunks longer than a tile)
  auto slot_of = [&](uint64_t x) -> uint32_t {
    if (x < cs) return 0;
    if (cs > 16 * kCopyTileUnits) return 1;
    return lg >= 0 ? (uint32_t)(x >> lg) : (uint32_t)x / (uint32_t)cs;
  };
  if (tid < 32) {
    const uint32_t s0 = (uint32_t)(tile0 * ut * 16 / cs);
    uint32_t lo = 0, hi = R - 1;  // last region that starts at or before s0
    if (R == nslots) lo = hi = s0;
    while (lo < hi) {
      const uint32_t step = (hi - lo) / 32 + 1;
      const uint64_t p = (uint64_t)lo + (uint64_t)tid * step;
      const uint32_t b = __ballot_sync(0xffffffffu, p <= hi && g.reg_slot[p] <= s0);
      lo += (31 - __clz(b)) * step;
      if ((uint64_t)lo + step - 1 < hi) hi = lo + step - 1;
    }
    if (tid == 0) sm.r = lo;
  }
  __syncthreads();
  for (uint64_t tile = tile0; tile < tile1; tile++) {
    const uint64_t u0 = tile * ut;
    const uint32_t nu = (uint32_t)(nunits - u0 < ut ? nunits - u0 : ut);
    const uint64_t b0 = u0 * 16, b1 = b0 + 16ull * nu < nbytes ? b0 + 16ull * nu : nbytes;
    const uint32_t s0 = (uint32_t)(lg >= 0 ? b0 >> lg : b0 / cs);
    const uint64_t rel = b0 - s0 * cs;
    const uint32_t ns = slot_of(rel + (b1 - 1 - b0)) + 1;
    const uint32_t r0 = sm.r;
    const uint32_t m = R - r0 < ns + 1 ? R - r0 : ns + 1;
    for (uint32_t i = tid; i < m; i += 256) {
      rs[i] = g.reg_slot[r0 + i];
      rc[i] = g.reg_chunk[r0 + i];
    }
    __syncthreads();
    for (uint32_t i = tid; i <= ns; i += 256) {
      uint32_t lo = 0, hi = m - 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (rs[mid] <= s0 + i) lo = mid; else hi = mid - 1;
      }
      if (i < ns) ch[i] = rc[lo] + (s0 + i - rs[lo]);
      if (i + 1 >= ns) sm.j[i + 1 - ns] = lo;
    }
    __syncthreads();
    // the next tile starts in this tile's last slot, or in the one after it
    if (tid == 0) sm.r = r0 + sm.j[rel + (b1 - b0) >= ns * cs ? 1 : 0];
    uint4* out = reinterpret_cast<uint4*>(dst) + u0;
    for (uint32_t k0 = tid; k0 < nu; k0 += 256 * kCopyPer) {
      uint4 v[kCopyPer];
#pragma unroll
      for (int q = 0; q < kCopyPer; q++) {
        const uint32_t k = k0 + 256u * q;
        v[q] = make_uint4(0, 0, 0, 0);
        if (k >= nu) continue;
        const uint64_t x = rel + 16ull * k;
        uint32_t si = slot_of(x);
        if (kVec) {
          // bytes past the end of the buffer stay zero (the reference reads
          // out of bounds there)
          const uint64_t off = ch[si] * cs + (x - si * cs);
          if (off + 16 <= g.len) {
            v[q] = __ldcs(reinterpret_cast<const uint4*>(g.data + off));
          } else if (off < g.len) {
            // an aligned word of the buffer's allocation
            const int hi = (int)(g.len - off);
            const uint4 w = __ldcs(reinterpret_cast<const uint4*>(g.data + off));
            v[q] = make_uint4(w.x & bytes_below(hi, 0), w.y & bytes_below(hi, 1), w.z & bytes_below(hi, 2),
                              w.w & bytes_below(hi, 3));
          }
        } else {
          uint32_t pos = 0;
          uint64_t within = x - si * cs;
          const uint32_t want = (uint32_t)(nbytes - (b0 + 16ull * k) < 16 ? nbytes - (b0 + 16ull * k) : 16);
          while (pos < want) {
            const uint64_t off = ch[si] * cs + within;  // source of byte pos
            uint32_t end = cs - within < want - pos ? pos + (uint32_t)(cs - within) : want;
            const uint32_t s1 = si;
            if (end < want && cs >= 16 && ch[si + 1] == ch[si] + 1) end = want;  // one run of bytes
            uint32_t hi = off >= g.len ? pos : g.len - off < end - pos ? pos + (uint32_t)(g.len - off) : end;
            if (hi > pos) {
              const uint4 w = load_window(reinterpret_cast<uint64_t>(g.data) + off - pos, pos, hi);
              v[q].x |= w.x & bytes_below(hi, 0) & ~bytes_below(pos, 0);
              v[q].y |= w.y & bytes_below(hi, 1) & ~bytes_below(pos, 1);
              v[q].z |= w.z & bytes_below(hi, 2) & ~bytes_below(pos, 2);
              v[q].w |= w.w & bytes_below(hi, 3) & ~bytes_below(pos, 3);
            }
            pos = end;
            si = s1 + 1;
            within = 0;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kCopyPer; q++) {
        const uint32_t k = k0 + 256u * q;
        if (k >= nu) continue;
        const uint64_t left = nbytes - (b0 + 16ull * k);
        if (kVec || left >= 16) {
          __stcs(out + k, v[q]);
        } else {
#pragma unroll
          for (uint32_t b = 0; b < 15; b++) {
            const uint32_t w = b < 4 ? v[q].x : b < 8 ? v[q].y : b < 12 ? v[q].z : v[q].w;
            if (b < left) reinterpret_cast<uint8_t*>(out + k)[b] = (uint8_t)(w >> (8 * (b & 3)));
          }
        }
      }
    }
    __syncthreads();
  }
}

// The gather of a whole checkpoint, a block per tile, in a launch of its own:
// counting 2^17 finished blocks (below) would cost more than the launch.
template <bool kVec>
__global__ void __launch_bounds__(256, 5) copy_kernel(GatherArgs g) {
  pdl_enter();
  __shared__ CopyShared sm;
  copy_tiles<kVec>(g, blockIdx.x, gridDim.x, sm);
}

// The rest of a checkpoint in one launch, by block: the sorted shift entries
// (n_sort blocks), the map inserts a fused forest pass has queued (n_drain:
// only later checkpoints read them, and the copy hides their random accesses),
// the chunk gather (the others).  The last block to finish writes the results
// to pinned host memory.
template <bool kVec>
__global__ void __launch_bounds__(256, 5) final_kernel(GatherArgs g) {
  pdl_enter();
  extern __shared__ uint32_t cnt[];
  __shared__ union {
    SortShared sort;
    CopyShared copy;
  } sm;
  __shared__ uint32_t s_last;
  const uint32_t blk = blockIdx.x;
  if (blk < g.n_sort) sort_scatter(g, blk, g.n_sort, sm.sort, cnt);
  else if (blk < g.n_sort + g.n_drain) drain_inserts(g, blk - g.n_sort, g.n_drain);
  else if (g.n_copy) copy_tiles<kVec>(g, blk - g.n_sort - g.n_drain, g.n_copy, sm.copy);
  if (last_block(g.counters + COUNT_FINAL_DONE, gridDim.x, &s_last)) readback(g.results);
}

// Entries of a table moved into a larger one (keys are stored already
// mapped, and unique, so every claim is new).
__global__ void map_rehash_kernel(DigestMap from, uint64_t from_cap, DigestMap to, uint32_t* err) {
  uint32_t created = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < from_cap; i += (uint64_t)gridDim.x * blockDim.x) {
    const MapSlot& s = from.slots[i];
    const uint4 v = *reinterpret_cast<const uint4*>(s.key);
    if (key_empty(v)) continue;
    uint64_t slot;
    if (map_claim(to, Digest{{v.x, v.y, v.z, v.w}}, false, &slot, err) != INS_NEW) continue;
    to.slots[slot].win = s.win;
    to.slots[slot].tree = s.tree;
    created++;
  }
  count_new_entries(to, created);
}

// Epochs of every entry set to 0, before the engine's epoch counter restarts.
__global__ void map_rebase_kernel(DigestMap m, uint64_t cap) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (uint64_t)gridDim.x * blockDim.x) {
    MapSlot& s = m.slots[i];
    if (s.win != kWinEmpty) s.win &= (1ull << kPrioBits) - 1;
  }
}

}  // namespace

cudaError_t launch_map_rehash(const DigestMap& from, uint64_t from_cap, const DigestMap& to, uint32_t* err,
                              cudaStream_t s) {
  map_rehash_kernel<<<grid_for(from_cap, 256), 256, 0, s>>>(from, from_cap, to, err);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_map_rebase(const DigestMap& m, uint64_t cap, cudaStream_t s) {
  map_rebase_kernel<<<grid_for(cap, 256), 256, 0, s>>>(m, cap);
  note_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------
size_t forest_done_words(uint32_t N) { return ((size_t)N >> 19) + 16; }

cudaError_t launch_forest(const ForestArgs& a, int pass, int baseline, uint32_t N, cudaStream_t s) {
  if (N < 2) return cudaSuccess;
  // deepest interior depth: that of node N-2
  uint32_t dmax = 0;
  while (((2ull << dmax) - 1) <= (uint64_t)(N - 2)) dmax++;
  const bool md5 = a.hash_kind == HASH_MD5;
  if (pass == 1 && baseline) {
    for (int bot = (int)dmax; bot >= 0; bot -= kSpanLevels) {
      const uint32_t top = bot >= (int)kSpanLevels - 1 ? (uint32_t)bot - (kSpanLevels - 1) : 0;
      const uint64_t first = (1ull << top) - 1;
      const uint64_t count = std::min<uint64_t>(1ull << top, (uint64_t)N - 1 - first);
      launch_k(forest_span_kernel, (uint32_t)count, 256, 0, s, a, N, top, (uint32_t)bot);
      note_launch();
    }
    return cudaGetLastError();
  }
  // the first pass follows the leaf inserts and starts after them: its blocks
  // beside theirs leave the inserts little L1 (a baseline of 64 MiB in 128-byte
  // chunks with a fifth of them duplicates: 218 against 195 us, an increment 88
  // against 84)
  const bool beside = pass == 1;
  if (N <= kSmallLeaves) {
    auto k = pass == 3 ? (md5 ? forest_small_kernel<HASH_MD5, true> : forest_small_kernel<HASH_MURMUR3, true>)
                       : (md5 ? forest_small_kernel<HASH_MD5, false> : forest_small_kernel<HASH_MURMUR3, false>);
    launch_with(beside, k, 1, 512, 0, s, a, pass, N, dmax);
  } else {
    auto k = pass == 3 ? (md5 ? forest_kernel<HASH_MD5, true> : forest_kernel<HASH_MURMUR3, true>)
                       : (md5 ? forest_kernel<HASH_MD5, false> : forest_kernel<HASH_MURMUR3, false>);
    const uint32_t top = dmax - (kBottomLevels - 1), count = 1u << top;
    launch_with(beside, k, pass == 1 ? std::min<uint32_t>(count, (uint32_t)num_sms() * 5) : count, 256, 0, s, a,
                pass, N, top, count);
  }
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_forest_inserts(const ForestArgs& a, int when, uint32_t N, cudaStream_t s) {
  if (N < 2) return cudaSuccess;
  launch_k(forest_insert_all_kernel, grid_for(N - 1, 256), 256, 0, s, a, when, N - 1);
  note_launch();
  return cudaGetLastError();
}

cudaError_t launch_assemble(GatherArgs g, uint64_t max_entries, bool whole, cudaEvent_t join, cudaStream_t s) {
  const uint32_t tiles = (uint32_t)std::max<uint64_t>(1, (g.n_flags + kRootTile - 1) / kRootTile);
  const bool reduce = tiles <= std::min<uint32_t>(kRootReduceTiles, 2 * reduce_tile_limit());
  const bool tree = g.approach == APPROACH_TREE, basic = g.approach == APPROACH_BASIC;
  auto count = tree ? root_count_kernel<APPROACH_TREE>
               : basic ? root_count_kernel<APPROACH_BASIC> : root_count_kernel<APPROACH_LIST>;
  auto emit = tree ? (reduce ? root_emit_kernel<APPROACH_TREE, true> : root_emit_kernel<APPROACH_TREE, false>)
              : basic ? (reduce ? root_emit_kernel<APPROACH_BASIC, true> : root_emit_kernel<APPROACH_BASIC, false>)
                      : (reduce ? root_emit_kernel<APPROACH_LIST, true> : root_emit_kernel<APPROACH_LIST, false>);
  launch_k(count, tiles, kScanThreads, 0, s, g);
  if (!reduce) {
    launch_k(scan_tile_offsets_kernel, 1, 1024, 0, s, g.tile_counts, tiles, (uint64_t*)nullptr);
    note_launch();
  }
  launch_k(emit, tiles, kScanThreads, 0, s, g);

  // metadata, regions, and the sort's counts.  Bound on the distinct keys
  // (source checkpoints): at most k_cap, which covers every checkpoint id that
  // this launch sequence can see
  const uint32_t K = std::min<uint32_t>(g.k_cap, kSortFastKeys);
  const uint32_t T = (uint32_t)((max_entries + kSortTile - 1) / kSortTile) + 1;
  const uint32_t emit_cap = 4 * num_sms();
  g.n_emit = whole ? (uint32_t)std::min<uint64_t>((max_entries + 255) / 256, emit_cap) : sparse_grid(max_entries, emit_cap);
  // tiles of the actual shift entries, read on the device: small grids
  g.n_sort = basic ? 0 : std::min<uint32_t>(T, 2 * num_sms());
  // one block scans the counts of all tiles; for larger matrices two launches
  // over the whole GPU
  g.sort_scan = (uint64_t)K * T <= (1u << 18) ? 1 : 0;
  launch_k(emit_count_kernel, g.n_emit + g.n_sort, 256, basic ? 0 : sizeof(uint32_t) * (size_t)K, s, g);
  note_launch(3);
  if (!basic && !g.sort_scan) {
    cudaError_t e = grid_scan(MatVal{g.sort_mat}, MatEmit{g.sort_mat}, &g.lay->sort_n, (uint64_t)K * T, g.scan_scratch2,
                              g.scan_total2, s);
    if (e != cudaSuccess) return e;
  }

  const bool vec = (g.cs % 16 == 0) && ((reinterpret_cast<uintptr_t>(g.data) & 15) == 0);
  static const bool reg = (register_input_kernel(reinterpret_cast<const void*>(final_kernel<true>), INPUT_GATHER),
                           register_input_kernel(reinterpret_cast<const void*>(final_kernel<false>), INPUT_GATHER), true);
  (void)reg;
  auto k = vec ? final_kernel<true> : final_kernel<false>;
  const size_t smem = basic ? 0 : sizeof(uint32_t) * (size_t)K * kSortWarps;
  if (smem > 16 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(sizeof(uint32_t) * kSortFastKeys * kSortWarps));
    if (e != cudaSuccess) return e;
  }
  // A first or whole checkpoint gathers (nearly) every chunk: a block per tile
  // keeps the copy at the bandwidth of a plain one (4 GiB: 1.21 ms against
  // 1.46 ms for a persistent grid).  An incremental one gathers a few percent
  // and gets one wave of blocks at most: a block per possible tile costs more
  // to launch than the copy takes.
  const uint64_t tile_bytes = 16ull * (g.cs >= 128 ? kCopyTileUnits : 16 * g.cs);
  const uint64_t ctiles = ((uint64_t)g.N * g.cs + tile_bytes - 1) / tile_bytes;
  const uint32_t wave = (uint32_t)num_sms() * 5;
  uint32_t copies = whole ? (uint32_t)std::min<uint64_t>(ctiles, 1u << 20) : sparse_grid(256 * ctiles, wave);
  if (whole && copies > wave) {  // never in a captured sequence
    launch_k(vec ? copy_kernel<true> : copy_kernel<false>, copies, 256, 0, s, g);
    note_launch();
    copies = 0;
  }
  g.n_drain = g.fuse_gate ? sparse_grid(g.N, 2 * num_sms()) : 0;
  if (join) {
    const cudaError_t e = cudaStreamWaitEvent(s, join, 0);
    if (e != cudaSuccess) return e;
  }
  g.n_copy = copies;
  const uint32_t grid = std::max(1u, g.n_sort + g.n_drain + copies);
  launch_k(k, grid, 256, smem, s, g);
  note_launch();
  return cudaGetLastError();
}

}  // namespace mtc
