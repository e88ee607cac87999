// leaf_kernels.cu -- chunk hashing and per-chunk classification.
//
// One thread owns one chunk (Murmur3 and MD5 are serial over a chunk).  On the
// fast path the chunk bytes reach shared memory through TMA tiled loads: the
// buffer is viewed as a 2-D tensor [n_full rows x cs bytes]; each stage moves a
// box of 128 (Murmur3) or 256 (MD5) rows x W bytes (W = 128, 64, 32 or 16) with
// the matching TMA swizzle so that the consumer threads, one per row, read their
// rows without bank conflicts.  A dedicated producer warp keeps STAGES boxes in flight; full/empty
// mbarriers hand stages between producer and consumers; one more warp hashes a
// partial last chunk.  Buffers off a 16-byte boundary are tiled from the boundary
// before them.  Other short chunks come as whole tiles by untiled bulk
// copies, longer ones in panels through a staged kernel, the rest (and many
// word-aligned chunks) through a thread-per-chunk kernel that reads global
// memory directly.  All end in the
// same epilogue, which restates the leaf loops of the reference:
//   tree  -- src/tree_approach.cpp:57-94 (baseline) and :309-351
//   list  -- src/list_approach.cpp:38-61
//   basic -- src/basic_approach.cpp:25-46
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <mutex>
#include <utility>

#include "mtc_common.cuh"
#include "mtc_internal.hpp"
#include "mtc_tma.cuh"

namespace mtc {

namespace {
// R (template) = consumer threads = chunks per tile = TMA box rows; one
// producer warp more per CTA
constexpr int kStages = 3;    // boxes in flight per CTA

template <int W>
__device__ __forceinline__ uint32_t swz(uint32_t logical) {
  constexpr uint32_t mask = W == 128 ? 7u : W == 64 ? 3u : W == 32 ? 1u : 0u;
  return logical ^ (((logical >> 7) & mask) << 4);
}

// Appends a changed chunk to the list the map inserts read (warp-aggregated).
__device__ __forceinline__ void append_changed(const LeafArgs& a, bool changed, uint32_t c) {
  const unsigned act = __activemask();
  const unsigned b = __ballot_sync(act, changed);
  if (!b) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(b) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(a.changed_count, (uint32_t)__popc(b));
  base = __shfl_sync(act, base, leader);
  if (changed) a.changed_list[base + __popc(b & ((1u << lane) - 1))] = c;
}

// A warp's changed chunks gathered in shared memory and appended 32 at a time:
// with a few percent of the chunks changed, most warps append one or two a
// tile, and each then waits for the counter, whose line takes one atomic after
// the other.  Hashing an increment, one append per warp and tile against this:
// 200 MB in 64-byte chunks 59 -> 47 us, 64 MiB in 32 35 -> 23, in 16 63 -> 38.
// Chunks of 128 bytes and more meet the counter too seldom, and their few warps
// per SM feel the extra steps (64 MiB in 128-byte chunks 16.0 -> 16.8 us, 4 GiB
// in 512 648 -> 677).  Whole warps call it.
struct ChangedBuf {
  uint32_t* buf;  // 64 entries of the warp's own
  uint32_t n;     // entries in it, below 32 between calls
  __device__ __forceinline__ void add(const LeafArgs& a, bool changed, uint32_t c) {
    const unsigned b = __ballot_sync(0xffffffffu, changed);
    if (!b) return;
    const uint32_t lane = threadIdx.x & 31;
    if (changed) buf[n + __popc(b & ((1u << lane) - 1))] = c;
    n += __popc(b);
    __syncwarp();
    if (n < 32) return;
    const uint32_t out = buf[lane], rest = buf[32 + lane];
    __syncwarp();
    buf[lane] = rest;
    n -= 32;
    put(a, out, 32);
    __syncwarp();
  }
  __device__ __forceinline__ void flush(const LeafArgs& a) {
    if (n) put(a, buf[threadIdx.x & 31], n);
  }
  __device__ __forceinline__ void put(const LeafArgs& a, uint32_t c, uint32_t count) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(a.changed_count, count);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lane < count) a.changed_list[base + lane] = c;
  }
};
template <int EPI>
__device__ __forceinline__ bool appends(const LeafArgs& a) {
  return (EPI == EPI_TREE || EPI == EPI_LIST) && !a.fresh;
}

// Streaming part of the per-chunk work: compare with the previous digest,
// store the new one; true where it changed (tree, list).  Map inserts happen in
// leaf_insert_kernel so that the hashing pipeline never waits on random memory
// accesses.
template <int EPI>
__device__ __forceinline__ bool leaf_store(const LeafArgs& a, bool valid, uint32_t c, const Digest& dg,
                                           const Digest& old) {
  if (EPI == EPI_HASH) {
    if (valid) st_digest(a.out + c, dg);
    return false;
  }
  if (EPI == EPI_BASIC) {
    if (!valid) return false;
    uint8_t changed = 1;
    if (!a.basic_first && digest_eq(dg, old)) changed = 0;
    if (changed || a.fresh) st_digest(a.prev + c, dg);
    a.labels[c] = changed;
    return false;
  }
  // tree (src/tree_approach.cpp:326-349) and list (src/list_approach.cpp:50-59)
  bool changed = false;
  if (valid) {
    changed = !digest_eq(dg, old);
    if (changed || a.fresh) st_digest(a.prev + c, dg);
    // a changed chunk is a first occurrence until the insert pass finds its
    // digest held by another
    a.labels[c] = changed ? FIRST_OCUR : (EPI == EPI_TREE ? FIXED_DUPL : DONE);
    // A FIXED_DUPL leaf's insert() always finds its digest (every earlier
    // leaf digest was inserted) and changes nothing, so it is not repeated.
  }
  return changed;
}
template <int EPI>
__device__ __forceinline__ void leaf_epilogue(const LeafArgs& a, bool valid, uint32_t c, const Digest& dg,
                                              const Digest& old) {
  const bool changed = leaf_store<EPI>(a, valid, c, dg, old);
  if (appends<EPI>(a)) append_changed(a, changed, c);
}

// Map insert of one changed chunk (src/tree_approach.cpp:325-369,
// src/list_approach.cpp:50-59): new digest -> first occurrence; a digest
// inserted by this launch too -> first occurrence of the lowest chunk, shifted
// duplicates of the others; an older digest -> shifted duplicate, except (tree)
// one whose entry carries this checkpoint's id, which an id that was not
// advanced (the header overload) leaves in place: the reference lowers its
// node there too and keeps the chunk that has it a first occurrence.
// Every insert lowers the entry's win word to its own, and the word it gets
// back tells who lost: itself, where that is lower, else the chunk it names.  So
// each loser is marked once by whoever passes it, in any order.  A second pass over
// notes of the duplicates took a launch more (a 1 MB increment 63 against 58 us) and
// an append to one list per duplicate (a list baseline of 256 MB in 64-byte
// chunks, half of them copies: 799 against 586 us).  Labels only ever go from
// first occurrence to shifted duplicate here.
// Lanes of a warp that hold one digest (runs of equal chunks) insert it once,
// through their first lane and with their lowest chunk, as if the lowest had
// come first.  The slot is read before it is claimed only once the block has
// met a digest that was there already (and for each thread's first chunk):
// with random accesses the bound, new digests save the read.
template <int EPI>
__global__ void __launch_bounds__(256) leaf_insert_kernel(LeafArgs a) {
  pdl_enter();
  stamp(a.clk, CLK_LEAVES_DONE);
  __shared__ volatile uint32_t s_dups;
  const uint32_t n = a.fresh ? a.n_chunks : *a.changed_count;
  const uint32_t cur = a.sp->cur, epoch = a.sp->epoch;
  const uint32_t lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_dups = 0;
  __syncthreads();
  bool first = true, lost = false;
  uint32_t created = 0;
  // whole warps step together
  for (uint64_t kw = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); kw < n;
       kw += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = kw + lane;
    bool in = k < n;
    const uint32_t c = !in ? 0xffffffffu : a.fresh ? (uint32_t)k : a.changed_list[k];
    // (only a chunk that has been inserted is ever marked by another)
    if (a.fresh) in = in && a.labels[c] == FIRST_OCUR;
    Digest dg{{0, 0, 0, 0}};
    if (in) dg = map_key(ld_digest(a.prev + c));
    const unsigned act = __ballot_sync(0xffffffffu, in);
    unsigned peers = 1u << lane;
    uint32_t low = c;
    const unsigned like = in ? __match_any_sync(act, dg.w[0]) : 0;
    if (like & (like - 1)) {
      const int src = __ffs(like) - 1;
      const uint32_t w1 = __shfl_sync(like, dg.w[1], src), w2 = __shfl_sync(like, dg.w[2], src),
                     w3 = __shfl_sync(like, dg.w[3], src);
      const bool same = dg.w[1] == w1 && dg.w[2] == w2 && dg.w[3] == w3;
      const unsigned all = __ballot_sync(like, same);
      if (same) {
        peers = all;
        low = __reduce_min_sync(all, c);
      }
    }
    const int lead = __ffs(peers) - 1;
    int r = INS_FAILED;
    // the entry is this launch's (or, tree, carries this checkpoint's id), and
    // the lowest of these chunks has it so far
    bool ours = false, wins = false;
    if (in && (int)lane == lead) {
      const uint32_t node = EPI == EPI_TREE ? a.leaf_base + low : low;
      unsigned long long w = win_of(epoch, node), old = kWinEmpty;
      uint64_t slot = 0;
      r = map_claim(a.map, dg, first || s_dups != 0, &slot, a.err);
      MapSlot* s = &a.map.slots[slot];
      bool older = false;
      if (r == INS_NEW) {
        old = slot_init(s, w, cur);
        ours = true;
        created++;
      } else if (r == INS_EXISTING) {
        old = win_min(s, w);
        older = old != kWinEmpty && win_epoch(old) != epoch;
        ours = !older || (EPI == EPI_TREE && __ldcg(&s->tree) == cur);
        if (older && ours) {
          // lowest node within the older entry (the reference's atomic_min,
          // src/tree_approach.cpp:337-339): the entry's high bits (epoch and
          // serial level) are fixed, since every insert of this launch carries
          // a larger epoch and leaves them alone, so lowering the whole word
          // lowers exactly its node
          w = (old & ~0xffffffffull) | node;
          if (old > w) old = win_min(s, w);
        }
      }
      wins = ours && old >= w;
      if (wins && old > w && old != kWinEmpty) {
        // the chunk that had it; an older entry's owner is one of this launch's
        // only if it is a changed chunk with this digest
        const uint32_t was = win_node(old) - (EPI == EPI_TREE ? a.leaf_base : 0u);
        if (!older || (win_node(old) >= a.leaf_base && a.labels[was] == FIRST_OCUR &&
                       digest_eq(map_key(ld_digest(a.prev + was)), dg))) {
          a.labels[was] = SHIFT_DUPL;
          lost = true;
        }
      }
    }
    first = false;
    if (__any_sync(0xffffffffu, r == INS_EXISTING) && lane == 0) s_dups = 1;
    ours = __shfl_sync(0xffffffffu, (int)ours, lead) != 0;
    wins = __shfl_sync(0xffffffffu, (int)wins, lead) != 0;
    const bool dup = in && !(wins && c == low);
    if (dup) a.labels[c] = SHIFT_DUPL;
    lost |= dup && ours;
  }
  // one store per block: with one per warp the word was what a baseline with
  // duplicates all over it waited for
  if (EPI == EPI_TREE && a.demoted && __syncthreads_or(lost) && threadIdx.x == 0) *a.demoted = 1;
  count_new_entries(a.map, created);
}

template <int EPI>
__device__ __forceinline__ bool needs_old(const LeafArgs& a) {
  return EPI != EPI_HASH && !a.fresh && !(EPI == EPI_BASIC && a.basic_first);
}

// ---------------------------------------------------------------------------
// TMA pipeline kernel.  A partial last chunk is hashed from global memory by one
// more warp of the last block: a launch of its own took 3-4 us, as long as the
// hashing of a 1 MB buffer, and a lane of the producer warp hashes it before the
// block's first box, since the warp's branches run one after the other.
// ---------------------------------------------------------------------------
// Digest of `len` bytes at a 16-byte aligned address, one thread: a serial
// chain, so what bounds it is the wait for its bytes.  They are loaded 64 bytes
// ahead of the hashing, from L2.  Digests of 1.4 MB in chunks of 4096 bytes with
// a tail of 3743: Murmur3 89 -> 36 us, MD5 127 -> 63 us; without
// the tail 31 and 58 us.
// kShift: they start d bytes past p.
template <int HK, bool kShift>
__device__ __noinline__ Digest hash_tail(const uint4* p, uint32_t d, uint32_t len) {
  constexpr uint32_t kWords = 4, kPiece = 16 * kWords;
  uint4 v[kWords];
  const uint64_t stop = (uint64_t)len + (kShift ? d : 0);  // from p
  auto word = [&](uint64_t at) { return at < stop ? __ldg(p + at / 16) : make_uint4(0, 0, 0, 0); };
  auto load = [&](uint64_t off) {
#pragma unroll
    for (uint32_t q = 0; q < kWords; q++) v[q] = word(off + 16 * q);
    if (kShift) {
      const uint4 after = word(off + kPiece);
#pragma unroll
      for (uint32_t q = 0; q < kWords; q++) v[q] = cut16(v[q], q + 1 < kWords ? v[q + 1] : after, d);
    }
  };
  Md5State md;
  Murmur3State mm;
  if (HK == HASH_MD5) md.init(); else mm.init();
  uint32_t X[4 * kWords];
  load(0);
  uint64_t off = 0;
  while (true) {
#pragma unroll
    for (uint32_t q = 0; q < kWords; q++) {
      X[4 * q] = v[q].x; X[4 * q + 1] = v[q].y; X[4 * q + 2] = v[q].z; X[4 * q + 3] = v[q].w;
    }
    if (off + kPiece > len) break;
    load(off + kPiece);
    if (HK == HASH_MD5) {
      md.block(X);
    } else {
#pragma unroll
      for (uint32_t q = 0; q < kWords; q++) mm.block(X[4 * q], X[4 * q + 1], X[4 * q + 2], X[4 * q + 3]);
    }
    off += kPiece;
  }
  const uint32_t rem = (uint32_t)(len - off);
#pragma unroll
  for (uint32_t i = 0; i < 4 * kWords; i++) {  // zero past the end
    const int k = (int)rem - 4 * (int)i;
    X[i] &= k <= 0 ? 0u : k >= 4 ? ~0u : (1u << (8 * k)) - 1;
  }
  if (HK == HASH_MD5) return md.finish(X, rem, len);
  uint64_t t0 = 0, t1 = 0;
#pragma unroll
  for (uint32_t q = 0; q < kWords; q++) {
    if (16 * q + 16 <= rem) {
      mm.block(X[4 * q], X[4 * q + 1], X[4 * q + 2], X[4 * q + 3]);
    } else if (16 * q < rem) {
      t0 = ((uint64_t)X[4 * q + 1] << 32) | X[4 * q];
      t1 = ((uint64_t)X[4 * q + 3] << 32) | X[4 * q + 2];
    }
  }
  mm.tail(t0, t1, rem & 15);
  return mm.finish(len);
}

// kShift: a buffer off a 16-byte boundary is tiled from the boundary before it, so
// chunk r starts d bytes into row r and ends d bytes into row r + 1.  Each 16
// bytes are cut out of two words; the last word of a box waits for the next box,
// and the first word of the next row is read with the row's first box (from
// global memory for a tile's last row).  Against the staged kernel (64-byte
// chunks: direct reads), 4 bytes off: 1 GiB in 4096-byte chunks 369 -> 216 us
// (Murmur3), 480 -> 269 (MD5); 256 MiB in 128-byte chunks 107 -> 67, 168 -> 111; in
// 64-byte chunks 150 -> 75, 221 -> 138.  On a boundary the 128-byte ones take 60.
template <int HK, int EPI, int W, int kRows, bool kShift>
__global__ void __launch_bounds__(kRows + 64, 2) leaf_tma_kernel(const __grid_constant__ CUtensorMap tmap, LeafArgs a,
                                                              uint32_t n_full) {
  pdl_enter();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr uint32_t kStageBytes = kRows * W;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  uint64_t* empty = full + kStages;
  const int tid = threadIdx.x;
  const uint32_t xsteps = a.cs / W;
  const uint32_t ntiles = (n_full + kRows - 1) / kRows;
  const uint32_t limit = a.spin_limit ? a.spin_limit : kMbarSpinLimit;
  static_assert(!kShift || W >= 64, "whole MD5 blocks per box");
  const uint32_t d = kShift ? (uint32_t)(reinterpret_cast<uintptr_t>(a.data) & 15) : 0;

  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kRows / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (tid >= kRows) {
    if (tid >= kRows + 32) {  // launched only with a partial last chunk
      if (blockIdx.x != gridDim.x - 1) return;
      const uint8_t* tail = a.data + (uint64_t)n_full * a.cs;
      const uint32_t nb = (uint32_t)(a.len - (uint64_t)n_full * a.cs);
      for (uint64_t at = 128ull * (tid - kRows - 32); at < nb; at += 32 * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(tail + at));
      if (tid != kRows + 32) return;
      Digest old{{0, 0, 0, 0}};
      if (needs_old<EPI>(a)) old = ld_digest(a.prev + n_full);
      const Digest dg = hash_tail<HK, kShift>(reinterpret_cast<const uint4*>(tail - d), d, nb);
      leaf_epilogue<EPI>(a, true, n_full, dg, old);
      return;
    }
    // producer warp: one elected lane issues every box in consumption order
    if (tid == kRows) {
      tma_prefetch_desc(&tmap);
      uint32_t it = 0;
      bool ok = !a.stall;  // injected fault: no copy is ever issued
      for (uint32_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        for (uint32_t xs = 0; xs < xsteps; xs++, it++) {
          const uint32_t s = it % kStages, ph = (it / kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, limit)) { raise_err(a.err, DERR_SPIN); ok = false; break; }
          mbar_arrive_expect_tx(&full[s], kStageBytes);
          tma_load_2d(smem + s * kStageBytes, &tmap, (int32_t)(xs * W), (int32_t)(tile * kRows), &full[s]);
        }
      }
      // drain: every issued box must land before the CTA may exit
      uint32_t first = it > (uint32_t)kStages ? it - kStages : 0;
      for (uint32_t j = first; j < it; j++) mbar_wait(&full[j % kStages], (j / kStages) & 1);
    }
    return;
  }

  const uint32_t lane = tid & 31;
  constexpr bool kGather = W < 128 && (EPI == EPI_TREE || EPI == EPI_LIST);
  __shared__ uint32_t changed_buf[kGather ? kRows / 32 : 1][64];
  ChangedBuf list{changed_buf[kGather ? tid >> 5 : 0], 0};
  uint32_t it = 0;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t c = tile * kRows + tid;
    const bool valid = c < n_full;
    Digest old{{0, 0, 0, 0}};
    if (valid && needs_old<EPI>(a)) old = ld_digest(a.prev + c);
    Murmur3State mm;
    Md5State md;
    if (HK == HASH_MD5) md.init(); else mm.init();
    uint32_t X[16];
    uint4 carry = make_uint4(0, 0, 0, 0), next = carry;  // kShift
    for (uint32_t xs = 0; xs < xsteps; xs++, it++) {
      const uint32_t s = it % kStages, ph = (it / kStages) & 1;
      if (!mbar_wait(&full[s], ph, limit)) { raise_err(a.err, DERR_SPIN); return; }
      const uint8_t* stage = smem + s * kStageBytes;
      const uint32_t rowbase = (uint32_t)tid * W;
      // the row into registers, then the stage goes back to the producer
      // before any hashing: the refill overlaps this thread's hash work
      uint4 row[W / 16];
#pragma unroll
      for (int q = 0; q < W / 16; q++) row[q] = *reinterpret_cast<const uint4*>(stage + swz<W>(rowbase + q * 16));
      if (kShift && xs == 0 && valid) {
        if (tid + 1 < kRows && c + 1 < n_full) next = *reinterpret_cast<const uint4*>(stage + swz<W>(rowbase + W));
        else next = __ldg(reinterpret_cast<const uint4*>(a.data - d + (uint64_t)(c + 1) * a.cs));
      }
      // release the stage: this thread's reads before the refill's TMA write
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (kShift) {
        auto put = [&](int slot, const uint4& v) {  // the next 16 bytes; MD5: fourth `slot` of its block
          if (HK == HASH_MD5) {
            X[4 * slot] = v.x; X[4 * slot + 1] = v.y; X[4 * slot + 2] = v.z; X[4 * slot + 3] = v.w;
            if (slot == 3) md.block(X);
          } else {
            mm.block(v.x, v.y, v.z, v.w);
          }
        };
        if (xs) put(3, cut16(carry, row[0], d));
#pragma unroll
        for (int q = 0; q + 1 < W / 16; q++) put(q & 3, cut16(row[q], row[q + 1], d));
        carry = row[W / 16 - 1];
        if (xs + 1 == xsteps) put(3, cut16(carry, next, d));
      } else if (HK == HASH_MD5) {
        if (W >= 64) {
#pragma unroll
          for (int blk = 0; blk < W / 64; blk++) {
#pragma unroll
            for (int q = 0; q < 4; q++) {
              const uint4 v = row[blk * 4 + q];
              X[4 * q] = v.x; X[4 * q + 1] = v.y; X[4 * q + 2] = v.z; X[4 * q + 3] = v.w;
            }
            md.block(X);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 16; i++) X[i] = 0;
#pragma unroll
          for (int q = 0; q < W / 16; q++) {
            const uint4 v = row[q];
            X[4 * q] = v.x; X[4 * q + 1] = v.y; X[4 * q + 2] = v.z; X[4 * q + 3] = v.w;
          }
        }
      } else {
#pragma unroll
        for (int q = 0; q < W / 16; q++) mm.block(row[q].x, row[q].y, row[q].z, row[q].w);
      }
    }
    Digest dg;
    if (HK == HASH_MD5) {
      if (W >= 64) {
#pragma unroll
        for (int i = 0; i < 16; i++) X[i] = 0;
        dg = md.finish(X, 0, a.cs);
      } else {
        dg = md.finish(X, a.cs, a.cs);
      }
    } else {
      dg = mm.finish(a.cs);
    }
    const bool changed = leaf_store<EPI>(a, valid, c, dg, old);
    if (!appends<EPI>(a)) continue;
    if (kGather) list.add(a, changed, c); else append_changed(a, changed, c);
  }
  if (kGather && appends<EPI>(a)) list.flush(a);
}

// ---------------------------------------------------------------------------
// Thread-per-chunk kernel reading global memory directly, for chunks
// [c0, c1).
// ---------------------------------------------------------------------------
template <int EPI>
__global__ void leaf_direct_kernel(LeafArgs a, uint32_t c0, uint32_t c1) {
  pdl_enter();
  for (uint64_t c = c0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; c < c1; c += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t off = c * (uint64_t)a.cs;
    uint64_t nb = a.cs;
    if (c == a.n_chunks - 1) nb = a.len - off;
    Digest old{{0, 0, 0, 0}};
    if (needs_old<EPI>(a)) old = ld_digest(a.prev + c);
    Digest dg = hash_bytes(a.hash_kind, a.data + off, nb);
    leaf_epilogue<EPI>(a, true, (uint32_t)c, dg, old);
  }
}

// ---------------------------------------------------------------------------
// Staged kernel for what the tiled copies and whole tiles cannot take: longer chunk
// sizes, and multiples of 32 bytes, that are no supported box width.  One thread hashes
// one chunk, 128 chunks per tile, in panels of 128 bytes that come through
// shared memory: a thread that reads its own chunk from global memory touches
// a line per lane.  Rows of a panel start on 16 bytes of shared memory whatever
// the chunk's address, so the copies are as wide as that allows (cp.async of 16,
// 8 or 4 bytes) and a thread reads its row in 16-byte words, without bank
// conflicts at a stride of 144 bytes; an address off a 4-byte boundary is
// shifted in registers.  kStageBufs panels in flight per block.  They leave room
// for 16 warps per SM, which wait for their own instructions: 441-byte chunks use
// 63 % of the issue slots and 61 % of the integer pipe with Murmur3, 73 % of the
// pipe with MD5, and a quarter of the bandwidth.  1 GiB in 4096-byte chunks 4 bytes off a boundary: 376 us (MD5 486), with
// direct loads 1054 us (991).
// ---------------------------------------------------------------------------
constexpr int kStageRows = 128;
constexpr int kStageBufs = 3;
constexpr uint32_t kPanel = 128;                       // bytes of a chunk per step
constexpr uint32_t kRowStride = kPanel + 16;
constexpr uint32_t kStagedBytes = kStageRows * kRowStride;  // one buffer

template <int B>
__device__ __forceinline__ void cp_async(uint32_t smem, uint64_t gmem) {
  if (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem), "l"(gmem), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Copies of one panel: each warp its own 32 rows, 128 / B lanes a row.  p0: the
// panel's first byte in the warp's first row; n_rows of the warp's rows exist;
// nb: bytes of a whole chunk in the panel; end: of the buffer.  Only words that
// hold a byte of a chunk are read.  With B = 4 a row starts at the word that
// holds its first byte, and may need a 33rd word.
template <int B>
__device__ __forceinline__ void stage_panel(uint32_t sm, uint64_t p0, uint64_t cs, uint32_t n_rows, uint32_t nb,
                                            uint64_t end) {
  constexpr uint32_t kLanes = kPanel / B, kRows = 32 / kLanes;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t sub = lane / kLanes, w = lane % kLanes;
#pragma unroll 4
  for (uint32_t r = sub; r < n_rows; r += kRows) {
    const uint64_t p = p0 + r * cs, lo = p & ~(uint64_t)(B - 1);
    const uint64_t stop = p + nb < end ? p + nb : end, at = lo + w * B;
    if (at < stop) cp_async<B>(sm + r * kRowStride + w * B, at);
  }
  if (B == 4 && lane < n_rows) {
    const uint64_t p = p0 + lane * cs, at = (p & ~3ull) + kPanel;
    const uint64_t stop = p + nb < end ? p + nb : end;
    if (at < stop) cp_async<B>(sm + lane * kRowStride + kPanel, at);
  }
}

template <int HK, int EPI>
__global__ void __launch_bounds__(kStageRows, 4) leaf_staged_kernel(LeafArgs a, uint32_t c0, uint32_t c1) {
  pdl_enter();
  extern __shared__ __align__(16) uint8_t sm_raw[];
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint64_t cs = a.cs;
  const uint64_t base = reinterpret_cast<uint64_t>(a.data), end = base + a.len;
  const uint32_t steps = (uint32_t)((cs + kPanel - 1) / kPanel);
  const uint32_t ntiles = (c1 - c0 + kStageRows - 1) / kStageRows;
  const uint32_t mine = blockIdx.x < ntiles ? (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
  const uint64_t total = (uint64_t)mine * steps;  // steps of this block, tile by tile
  const uint32_t align = (uint32_t)(base | cs) & 15;  // of every row
  const uint32_t sm0 = smem_u32(sm_raw);

  uint32_t ld_tile = blockIdx.x, ld_step = 0;
  auto load = [&](uint32_t buf) {
    const uint64_t row0 = (uint64_t)c0 + (uint64_t)ld_tile * kStageRows + warp * 32;
    const uint32_t n_rows = row0 >= c1 ? 0 : c1 - row0 < 32 ? (uint32_t)(c1 - row0) : 32;
    const uint64_t done = (uint64_t)ld_step * kPanel;
    const uint32_t nb = cs - done < kPanel ? (uint32_t)(cs - done) : kPanel;
    const uint64_t p0 = base + row0 * cs + done;
    const uint32_t sm = sm0 + buf * kStagedBytes + warp * 32 * kRowStride;
    if (align == 0) stage_panel<16>(sm, p0, cs, n_rows, nb, end);
    else if ((align & 7) == 0) stage_panel<8>(sm, p0, cs, n_rows, nb, end);
    else stage_panel<4>(sm, p0, cs, n_rows, nb, end);
    if (++ld_step == steps) {
      ld_step = 0;
      ld_tile += gridDim.x;
    }
  };

  uint64_t issued = 0;
#pragma unroll
  for (int k = 0; k < kStageBufs - 1; k++) {
    if (issued < total) load((uint32_t)(issued % kStageBufs));
    issued++;
    cp_async_commit();
  }
  Murmur3State mm;
  Md5State md;
  Digest old{{0, 0, 0, 0}};
  uint32_t tile = blockIdx.x, step = 0, buf = 0;
  for (uint64_t k = 0; k < total; k++) {
    const uint64_t c = (uint64_t)c0 + (uint64_t)tile * kStageRows + tid;
    const bool valid = c < c1;
    if (step == 0) {
      if (HK == HASH_MD5) md.init(); else mm.init();
      old = Digest{{0, 0, 0, 0}};
      if (valid && needs_old<EPI>(a)) old = ld_digest(a.prev + c);
    }
    // a warp reads only the rows it has copied itself
    cp_async_wait<kStageBufs - 2>();
    __syncwarp();
    if (issued < total) load(buf == 0 ? kStageBufs - 1 : buf - 1);  // the buffer of step k - 1
    issued++;
    cp_async_commit();
    if (valid) {
      const uint4* src = reinterpret_cast<const uint4*>(sm_raw + buf * kStagedBytes + tid * kRowStride);
      const uint64_t nb = min(cs, a.len - c * cs);  // bytes of the chunk
      const uint64_t done = (uint64_t)step * kPanel;
      const uint32_t rem = nb <= done ? 0 : nb - done < kPanel ? (uint32_t)(nb - done) : kPanel;
      const uint32_t sh = ((uint32_t)(base + c * cs) & 3) * 8;
      uint32_t y[33];
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const uint4 v = src[q];
        y[4 * q] = v.x; y[4 * q + 1] = v.y; y[4 * q + 2] = v.z; y[4 * q + 3] = v.w;
      }
      if (sh) {
        y[32] = src[8].x;
#pragma unroll
        for (int i = 0; i < 32; i++) y[i] = __funnelshift_r(y[i], y[i + 1], sh);
      }
      if (rem < kPanel) {  // words past the chunk's end read as zero
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const int left = (int)rem - 4 * i;
          if (left < 4) y[i] &= left <= 0 ? 0u : (1u << (8 * left)) - 1;
        }
      }
      const bool last = done < nb && nb <= done + kPanel;  // the chunk ends in this step
      if (HK == HASH_MD5) {
        if (rem >= 64) md.block(y);
        if (rem == kPanel) md.block(y + 16);
        if (last) {
          // the final partial block: nothing, or the bytes after the last whole one
          uint32_t X[16];
          const uint32_t part = rem & 63;
#pragma unroll
          for (int i = 0; i < 16; i++) X[i] = part == 0 ? 0 : rem < 64 ? y[i] : y[16 + i];
          const Digest dg = md.finish(X, part, nb);
          leaf_epilogue<EPI>(a, true, (uint32_t)c, dg, old);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 8; q++)
          if (16u * (q + 1) <= rem) mm.block(y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]);
        if (last) {
          const uint32_t part = rem & 15, q = rem >> 4;
          uint32_t t[4] = {0, 0, 0, 0};
#pragma unroll
          for (int i = 0; i < 8; i++)
            if ((uint32_t)i == q && part) {
              t[0] = y[4 * i]; t[1] = y[4 * i + 1]; t[2] = y[4 * i + 2]; t[3] = y[4 * i + 3];
            }
          mm.tail(((uint64_t)t[1] << 32) | t[0], ((uint64_t)t[3] << 32) | t[2], part);
          leaf_epilogue<EPI>(a, true, (uint32_t)c, mm.finish(nb), old);
        }
      }
    }
    __syncwarp();  // the row is read before the warp refills this buffer
    if (++step == steps) {
      step = 0;
      tile += gridDim.x;
    }
    buf = buf + 1 == kStageBufs ? 0 : buf + 1;
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// Short chunks that no box fits: the 128 chunks of a tile are contiguous, so one
// untiled bulk copy of 128 * cs bytes (from the 16-byte boundary before them to
// the one after) brings a tile in whatever its chunk size and alignment, and a
// producer lane keeps two in flight.  A thread reads its row word by word: an
// odd multiple of four bytes apart, rows lie in different banks.  100-byte chunks
// use two thirds of the issue slots (hashing, and realigning words) and of the
// bandwidth with Murmur3, 77 % of the integer pipe with MD5.  Two stages, for more CTAs per SM
// (three: 250-byte chunks 73 us for 256 MiB, two 62).  Whole calls, two stages
// against the kernels before: 400 MB in chunks of 100 bytes 130 -> 91 us
// (Murmur3), 183 -> 174 (MD5); 256 MiB in 300 bytes 131 -> 69 and 166 -> 106.
// ---------------------------------------------------------------------------
constexpr uint32_t kRowTile = 128;
constexpr int kRowStages = 2;
constexpr uint32_t kRowsMax = 440;
__host__ __device__ constexpr uint32_t row_stage_bytes(uint32_t cs) { return (kRowTile * cs + 30) & ~15u; }
// barriers, stages, and what a row's last words are read past its end (masked)
__host__ __device__ constexpr uint32_t row_smem_bytes(uint32_t cs) {
  return 128 + kRowStages * row_stage_bytes(cs) + 128;
}

template <int HK, int EPI>
__global__ void __launch_bounds__(kRowTile + 32, HK == HASH_MD5 ? 5 : 8) leaf_rows_kernel(LeafArgs a, uint32_t c0,
                                                                                        uint32_t c1) {
  pdl_enter();
  extern __shared__ __align__(128) uint8_t row_smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(row_smem);
  uint64_t* empty = full + kRowStages;
  uint8_t* stages = row_smem + 128;
  constexpr bool kLists = EPI == EPI_TREE || EPI == EPI_LIST;
  __shared__ uint32_t changed_buf[kLists ? kRowTile / 32 : 1][64];
  const uint32_t tid = threadIdx.x, cs = a.cs, stage_bytes = row_stage_bytes(cs);
  const uint32_t ntiles = (c1 - c0 + kRowTile - 1) / kRowTile;
  const uint32_t limit = a.spin_limit ? a.spin_limit : kMbarSpinLimit;
  const uint64_t base = reinterpret_cast<uint64_t>(a.data) + (uint64_t)c0 * cs;
  const uint64_t end = reinterpret_cast<uint64_t>(a.data) + min(a.len, (uint64_t)c1 * cs);
  if (tid == 0) {
    for (int s = 0; s < kRowStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kRowTile / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (tid >= kRowTile) {
    if (tid != kRowTile) return;
    uint32_t it = 0;
    bool ok = !a.stall;  // injected fault: no copy is ever issued
    for (uint32_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, it++) {
      const uint32_t s = it % kRowStages, ph = (it / kRowStages) & 1;
      if (!mbar_wait(&empty[s], ph ^ 1, limit)) { raise_err(a.err, DERR_SPIN); ok = false; break; }
      const uint64_t p0 = (base + (uint64_t)tile * kRowTile * cs) & ~15ull;
      const uint64_t p1 = min(end, base + (uint64_t)(tile + 1) * kRowTile * cs);
      const uint32_t bytes = (uint32_t)(p1 - p0 + 15) & ~15u;
      mbar_arrive_expect_tx(&full[s], bytes);
      bulk_load(stages + s * stage_bytes, reinterpret_cast<const void*>(p0), bytes, &full[s]);
    }
    // drain: every issued copy must land before the CTA may exit
    for (uint32_t j = it > (uint32_t)kRowStages ? it - kRowStages : 0; j < it; j++)
      mbar_wait(&full[j % kRowStages], (j / kRowStages) & 1);
    return;
  }

  const uint32_t lane = tid & 31;
  ChangedBuf list{changed_buf[kLists ? tid >> 5 : 0], 0};
  uint32_t it = 0;
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
    const uint64_t c = (uint64_t)c0 + (uint64_t)tile * kRowTile + tid;
    const bool valid = c < c1;
    Digest old{{0, 0, 0, 0}};
    if (valid && needs_old<EPI>(a)) old = ld_digest(a.prev + c);
    const uint32_t s = it % kRowStages, ph = (it / kRowStages) & 1;
    if (!mbar_wait(&full[s], ph, limit)) { raise_err(a.err, DERR_SPIN); return; }
    const uint32_t nb = !valid ? 0 : (uint32_t)min((uint64_t)cs, a.len - c * cs);
    const uint32_t o = (uint32_t)((base + (uint64_t)tile * kRowTile * cs) & 15) + tid * cs;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(stages + s * stage_bytes) + (o >> 2);
    const uint32_t sh = (o & 3) * 8;
    constexpr uint32_t kWords = HK == HASH_MD5 ? 16 : 4;
    Md5State md;
    Murmur3State mm;
    if (HK == HASH_MD5) md.init(); else mm.init();
    uint32_t X[kWords];
    uint32_t left = nb;
#pragma unroll 1
    while (true) {
      if (valid) {
        uint32_t lo = w[0];
#pragma unroll
        for (uint32_t i = 0; i < kWords; i++) {
          // past a short last chunk's copy the words are whatever the stage holds
          const uint32_t hi = w[i + 1];
          X[i] = __funnelshift_r(lo, hi, sh);
          lo = hi;
        }
      }
      if (left < 4 * kWords) break;
      if (HK == HASH_MD5) md.block(X); else mm.block(X[0], X[1], X[2], X[3]);
      left -= 4 * kWords;
      w += kWords;
    }
    // the rows go back before the epilogue
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
#pragma unroll
    for (uint32_t i = 0; i < kWords; i++) {  // zero past the end
      const int k = (int)left - 4 * (int)i;
      X[i] &= k <= 0 ? 0u : k >= 4 ? ~0u : (1u << (8 * k)) - 1;
    }
    Digest dg;
    if (HK == HASH_MD5) {
      dg = md.finish(X, left, nb);
    } else {
      mm.tail(((uint64_t)X[1] << 32) | X[0], ((uint64_t)X[3 % kWords] << 32) | X[2], left);
      dg = mm.finish(nb);
    }
    const bool changed = leaf_store<EPI>(a, valid, (uint32_t)c, dg, old);
    if (appends<EPI>(a)) list.add(a, changed, (uint32_t)c);
  }
  if (appends<EPI>(a)) list.flush(a);
}

// ---------------------------------------------------------------------------
// One persistent launch for the leaf pass of many deduplicators (a batch).
// A device work queue holds (member, tile) items; each CTA's producer lane
// claims the next item with one atomicAdd and streams its boxes through the
// same full/empty mbarrier pipeline as leaf_tma_kernel, announcing in a small
// per-stage record which member, tile and column step each box belongs to.
// Members differ in chunk size (box width 64 or 128 bytes), digest and
// approach; every consumer thread owns one row of the current item and ends
// with that member's epilogue.  Items are ordered largest first.  A producer
// that finds the queue empty drains its copies, then sends one record
// without data that stops the CTA's consumers.
// ---------------------------------------------------------------------------
struct BatchStageMeta {
  uint32_t member, tile, xs, flags;  // flags: kMetaFirst | kMetaLast | kMetaDone
};
constexpr uint32_t kMetaFirst = 1, kMetaLast = 2, kMetaDone = 4;
constexpr uint32_t kBatchStageBytes = kBatchRows * 128;

__device__ __forceinline__ bool needs_old_rt(const LeafArgs& a) {
  return a.epi != EPI_HASH && !a.fresh && !(a.epi == EPI_BASIC && a.basic_first);
}

__global__ void __launch_bounds__(kBatchRows + 32, 3) batch_leaf_kernel(BatchLeafParams p) {
  pdl_enter();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * kBatchStageBytes);
  uint64_t* empty = full + kStages;
  BatchStageMeta* meta = reinterpret_cast<BatchStageMeta*>(empty + kStages);
  const int tid = threadIdx.x;
  const uint32_t limit = p.spin_limit ? p.spin_limit : kMbarSpinLimit;
  if (tid == 0) {
    for (int s = 0; s < kStages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kBatchRows / 32);
    }
    mbar_fence_init();
  }
  __syncthreads();

  if (tid >= kBatchRows) {
    if (tid == kBatchRows) {
      uint32_t it = 0;
      uint32_t* err = p.members[0].la.err;
      bool ok = true;
      while (ok) {
        const uint32_t k = atomicAdd(p.head, 1u);
        if (k >= p.nitems) break;
        const uint2 item = p.items[k];
        const uint32_t m = item.x, tile = item.y;
        const uint32_t xsteps = p.members[m].xsteps, W = p.members[m].W;
        err = p.members[m].la.err;
        for (uint32_t xs = 0; xs < xsteps; xs++, it++) {
          const uint32_t s = it % kStages, ph = (it / kStages) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, limit)) {
            raise_err(err, DERR_SPIN);
            ok = false;
            break;
          }
          meta[s] = BatchStageMeta{m, tile, xs, (xs == 0 ? kMetaFirst : 0u) | (xs + 1 == xsteps ? kMetaLast : 0u)};
          mbar_arrive_expect_tx(&full[s], kBatchRows * W);
          tma_load_2d(smem + s * kBatchStageBytes, &p.members[m].map, (int32_t)(xs * W), (int32_t)(tile * kBatchRows),
                      &full[s]);
        }
      }
      // drain: every issued box lands before the CTA exits (before the stop
      // record, which reuses the slot of the oldest of them)
      const uint32_t first = it > (uint32_t)kStages ? it - kStages : 0;
      for (uint32_t j2 = first; j2 < it; j2++) mbar_wait(&full[j2 % kStages], (j2 / kStages) & 1, limit);
      if (ok) {
        // the stop record: no data, the arrive alone completes the phase
        const uint32_t s = it % kStages, ph = (it / kStages) & 1;
        if (mbar_wait(&empty[s], ph ^ 1, limit)) {
          meta[s] = BatchStageMeta{0, 0, 0, kMetaDone};
          mbar_arrive(&full[s]);
        } else {
          raise_err(err, DERR_SPIN);
        }
      }
    }
    return;
  }

  const uint32_t lane = tid & 31;
  Murmur3State mm;
  Md5State md;
  mm.init();
  md.init();
  Digest old{{0, 0, 0, 0}};
  uint32_t c = 0;
  bool valid = false;
  for (uint32_t it = 0;; it++) {
    const uint32_t s = it % kStages, ph = (it / kStages) & 1;
    if (!mbar_wait(&full[s], ph, limit)) {
      raise_err(p.members[0].la.err, DERR_SPIN);
      return;
    }
    const BatchStageMeta mt = meta[s];
    if (mt.flags & kMetaDone) return;
    const MemberLeaf& ml = p.members[mt.member];
    const LeafArgs& a = ml.la;
    const uint32_t W = ml.W;
    const bool md5 = a.hash_kind == HASH_MD5;
    if (mt.flags & kMetaFirst) {
      c = mt.tile * kBatchRows + tid;
      valid = c < ml.n_full;
      old = Digest{{0, 0, 0, 0}};
      if (valid && needs_old_rt(a)) old = ld_digest(a.prev + c);
      mm.init();
      md.init();
    }
    // the row into registers, then the stage goes back to the producer
    const uint8_t* stage = smem + s * kBatchStageBytes;
    uint4 row[8];
    if (W == 128) {
#pragma unroll
      for (int q = 0; q < 8; q++) row[q] = *reinterpret_cast<const uint4*>(stage + swz<128>((uint32_t)tid * 128 + q * 16));
    } else {
#pragma unroll
      for (int q = 0; q < 4; q++) row[q] = *reinterpret_cast<const uint4*>(stage + swz<64>((uint32_t)tid * 64 + q * 16));
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    const int nblk = W == 128 ? 2 : 1;
    if (md5) {
      uint32_t X[16];
      for (int blk = 0; blk < nblk; blk++) {
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const uint4 v = row[blk * 4 + q];
          X[4 * q] = v.x; X[4 * q + 1] = v.y; X[4 * q + 2] = v.z; X[4 * q + 3] = v.w;
        }
        md.block(X);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (q < 4 * nblk) mm.block(row[q].x, row[q].y, row[q].z, row[q].w);
    }
    if (mt.flags & kMetaLast) {
      Digest dg;
      if (md5) {
        uint32_t X[16];
#pragma unroll
        for (int i = 0; i < 16; i++) X[i] = 0;
        dg = md.finish(X, 0, a.cs);
      } else {
        dg = mm.finish(a.cs);
      }
      switch (a.epi) {
        case EPI_TREE: leaf_epilogue<EPI_TREE>(a, valid, c, dg, old); break;
        case EPI_LIST: leaf_epilogue<EPI_LIST>(a, valid, c, dg, old); break;
        case EPI_BASIC: leaf_epilogue<EPI_BASIC>(a, valid, c, dg, old); break;
        default: leaf_epilogue<EPI_HASH>(a, valid, c, dg, old); break;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Warp-per-chunk kernel: the lanes of a warp load one chunk together into
// shared memory (coalesced 4-byte words), then lane 0 hashes it.  The digests
// are serial chains (each 16-byte Murmur3 block and each 64-byte MD5 block
// depends on the state left by the previous one), so the other lanes cannot
// share the hashing; this shape exists for the autotuner to compare against
// the thread-per-chunk pipelines.
// ---------------------------------------------------------------------------
constexpr uint32_t kWarpChunkMax = 4096;
template <int EPI>
__global__ void leaf_warp_kernel(LeafArgs a, uint32_t c0, uint32_t c1) {
  pdl_enter();
  extern __shared__ uint32_t wsm[];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t stride_w = (a.cs + 64 + 3) / 4;  // words per warp buffer, zero padding included
  uint32_t* buf = wsm + warp * stride_w;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const bool al4 = (reinterpret_cast<uintptr_t>(a.data) & 3) == 0 && (a.cs & 3) == 0;
  for (uint64_t c = c0 + (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); c < c1; c += nwarps) {
    const uint64_t off = c * (uint64_t)a.cs;
    const uint32_t nb = c == a.n_chunks - 1 ? (uint32_t)(a.len - off) : a.cs;
    const uint32_t nw = (nb + 64 + 3) / 4;
    for (uint32_t i = lane; i < nw; i += 32) {
      uint32_t v = 0;
      if (al4 && 4 * i + 4 <= nb) v = __ldg(reinterpret_cast<const uint32_t*>(a.data + off) + i);
      else v = ld_word_any(a.data + off, 4 * (uint64_t)i, nb);
      buf[i] = v;
    }
    __syncwarp();
    if (lane == 0) {
      Digest old{{0, 0, 0, 0}};
      if (needs_old<EPI>(a)) old = ld_digest(a.prev + c);
      const Digest dg = hash_words(a.hash_kind, buf, nb);
      leaf_epilogue<EPI>(a, true, (uint32_t)c, dg, old);
    }
    __syncwarp();
  }
}

template <int EPI>
cudaError_t launch_warp(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  if (c1 <= c0) return cudaSuccess;
  const uint32_t warps_per_block = 8;
  const size_t smem = (size_t)warps_per_block * 4 * ((a.cs + 64 + 3) / 4);
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(leaf_warp_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(warps_per_block * 4 * ((kWarpChunkMax + 64 + 3) / 4)));
    if (e != cudaSuccess) return e;
    attr_set.store(true, std::memory_order_release);
  }
  uint64_t grid = (c1 - c0 + warps_per_block - 1) / warps_per_block;
  const uint64_t cap = (uint64_t)num_sms() * 8;
  if (grid > cap) grid = cap;
  static const bool reg =
      (register_input_kernel(reinterpret_cast<const void*>(leaf_warp_kernel<EPI>), INPUT_LEAF_DIRECT), true);
  (void)reg;
  launch_k(leaf_warp_kernel<EPI>, (uint32_t)grid, warps_per_block * 32, smem, s, a, c0, c1);
  note_launch();
  return cudaGetLastError();
}

cudaError_t dispatch_warp(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_warp<EPI_TREE>(a, c0, c1, s);
    case EPI_LIST: return launch_warp<EPI_LIST>(a, c0, c1, s);
    case EPI_BASIC: return launch_warp<EPI_BASIC>(a, c0, c1, s);
    default: return launch_warp<EPI_HASH>(a, c0, c1, s);
  }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

int tma_width(uint32_t cs) {
  if (cs % 128 == 0) return 128;
  if (cs == 64 || cs == 32 || cs == 16) return (int)cs;
  return 0;
}

bool make_tmap(TmaCache* c, const uint8_t* data, uint64_t len, uint32_t cs, int W, int rows, uint32_t n_full) {
  if (c->ptr == data && c->len == len && c->cs == cs && c->width == W && c->rows == rows) return true;
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {cs, n_full};
  cuuint64_t strides[1] = {cs};
  cuuint32_t box[2] = {(cuuint32_t)W, (cuuint32_t)rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapSwizzle sw = W == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                        : W == 64  ? CU_TENSOR_MAP_SWIZZLE_64B
                        : W == 32  ? CU_TENSOR_MAP_SWIZZLE_32B
                                   : CU_TENSOR_MAP_SWIZZLE_NONE;
  CUresult r = fn(&c->map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(data), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { c->ptr = nullptr; return false; }
  c->ptr = data; c->len = len; c->cs = cs; c->width = W; c->rows = rows;
  return true;
}

template <int HK, int EPI, int W, int R, bool kShift = false>
cudaError_t launch_tma_t(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int ctas_per_sm, cudaStream_t s) {
  auto k = leaf_tma_kernel<HK, EPI, W, R, kShift>;
  static const bool reg = (register_input_kernel(reinterpret_cast<const void*>(k), INPUT_LEAF_TMA), true);
  (void)reg;
  const size_t smem = 1024 + (size_t)kStages * R * W + 2 * kStages * sizeof(uint64_t);
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set.store(true, std::memory_order_release);
  }
  const uint32_t ntiles = (n_full + R - 1) / R;
  // resident CTAs per SM that fit in 227 KB of shared memory, at most 3 by default
  const int fit = (int)((227u * 1024u) / smem);
  int per_sm = ctas_per_sm > 0 ? ctas_per_sm : 3;
  if (per_sm > fit) per_sm = fit > 0 ? fit : 1;
  uint32_t grid = (uint32_t)(num_sms() * per_sm);
  if (grid > ntiles) grid = ntiles;
  launch_k(k, grid, n_full < a.n_chunks ? R + 64 : R + 32, smem, s, m, a, n_full);
  note_launch();
  return cudaGetLastError();
}

template <int HK, int EPI, int R>
cudaError_t launch_tma_w(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int W, int per_sm, cudaStream_t s) {
  switch (W) {
    case 128: return launch_tma_t<HK, EPI, 128, R>(a, m, n_full, per_sm, s);
    case 64: return launch_tma_t<HK, EPI, 64, R>(a, m, n_full, per_sm, s);
    case 32: return launch_tma_t<HK, EPI, 32, R>(a, m, n_full, per_sm, s);
    default: return launch_tma_t<HK, EPI, 16, R>(a, m, n_full, per_sm, s);
  }
}

template <int EPI>
cudaError_t launch_tma_e(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int W, const LeafTune& t,
                         cudaStream_t s) {
  if (t.rows == 128) {
    if (a.hash_kind == HASH_MD5) return launch_tma_w<HASH_MD5, EPI, 128>(a, m, n_full, W, t.ctas_per_sm, s);
    return launch_tma_w<HASH_MURMUR3, EPI, 128>(a, m, n_full, W, t.ctas_per_sm, s);
  }
  if (a.hash_kind == HASH_MD5) return launch_tma_w<HASH_MD5, EPI, 256>(a, m, n_full, W, t.ctas_per_sm, s);
  return launch_tma_w<HASH_MURMUR3, EPI, 256>(a, m, n_full, W, t.ctas_per_sm, s);
}

// Buffers off a 16-byte boundary, with the digest's default tile
template <int EPI>
cudaError_t launch_shift(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int W, int per_sm, cudaStream_t s) {
  if (a.hash_kind == HASH_MD5)
    return W == 128 ? launch_tma_t<HASH_MD5, EPI, 128, 256, true>(a, m, n_full, per_sm, s)
                    : launch_tma_t<HASH_MD5, EPI, 64, 256, true>(a, m, n_full, per_sm, s);
  return W == 128 ? launch_tma_t<HASH_MURMUR3, EPI, 128, 128, true>(a, m, n_full, per_sm, s)
                  : launch_tma_t<HASH_MURMUR3, EPI, 64, 128, true>(a, m, n_full, per_sm, s);
}
cudaError_t dispatch_shift(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int W, int per_sm, cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_shift<EPI_TREE>(a, m, n_full, W, per_sm, s);
    case EPI_LIST: return launch_shift<EPI_LIST>(a, m, n_full, W, per_sm, s);
    case EPI_BASIC: return launch_shift<EPI_BASIC>(a, m, n_full, W, per_sm, s);
    default: return launch_shift<EPI_HASH>(a, m, n_full, W, per_sm, s);
  }
}

template <int EPI>
cudaError_t launch_direct(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  if (c1 <= c0) return cudaSuccess;
  uint64_t n = c1 - c0;
  uint32_t grid = (uint32_t)((n + 127) / 128);
  uint32_t cap = (uint32_t)num_sms() * 16;
  if (grid > cap) grid = cap;
  static const bool reg =
      (register_input_kernel(reinterpret_cast<const void*>(leaf_direct_kernel<EPI>), INPUT_LEAF_DIRECT), true);
  (void)reg;
  launch_k(leaf_direct_kernel<EPI>, grid, 128, 0, s, a, c0, c1);
  note_launch();
  return cudaGetLastError();
}

template <int HK, int EPI>
cudaError_t launch_staged_t(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  auto k = leaf_staged_kernel<HK, EPI>;
  constexpr size_t smem = (size_t)kStageBufs * kStagedBytes;
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set.store(true, std::memory_order_release);
  }
  static const bool reg = (register_input_kernel(reinterpret_cast<const void*>(k), INPUT_LEAF_DIRECT), true);
  (void)reg;
  const uint32_t ntiles = (c1 - c0 + kStageRows - 1) / kStageRows;
  const uint32_t cap = (uint32_t)num_sms() * 4;
  launch_k(k, ntiles < cap ? ntiles : cap, kStageRows, smem, s, a, c0, c1);
  note_launch();
  return cudaGetLastError();
}
template <int EPI>
cudaError_t launch_staged(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  return a.hash_kind == HASH_MD5 ? launch_staged_t<HASH_MD5, EPI>(a, c0, c1, s)
                                 : launch_staged_t<HASH_MURMUR3, EPI>(a, c0, c1, s);
}
cudaError_t dispatch_staged(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_staged<EPI_TREE>(a, c0, c1, s);
    case EPI_LIST: return launch_staged<EPI_LIST>(a, c0, c1, s);
    case EPI_BASIC: return launch_staged<EPI_BASIC>(a, c0, c1, s);
    default: return launch_staged<EPI_HASH>(a, c0, c1, s);
  }
}

template <int HK, int EPI>
cudaError_t launch_rows_t(const LeafArgs& a, cudaStream_t s) {
  auto k = leaf_rows_kernel<HK, EPI>;
  static const bool reg = (register_input_kernel(reinterpret_cast<const void*>(k), INPUT_LEAF_DIRECT), true);
  (void)reg;
  const size_t smem = row_smem_bytes(a.cs);
  static std::atomic<bool> attr_set{false};
  if (!attr_set.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)row_smem_bytes(kRowsMax));
    if (e != cudaSuccess) return e;
    attr_set.store(true, std::memory_order_release);
  }
  const uint32_t fit = (uint32_t)((227u * 1024u) / (smem + 2048));
  const uint32_t per_sm = std::min<uint32_t>(fit, HK == HASH_MD5 ? 5 : 8);
  const uint32_t tiles = (a.n_chunks + kRowTile - 1) / kRowTile;
  launch_k(k, std::min<uint32_t>(tiles, num_sms() * per_sm), kRowTile + 32, smem, s, a, 0u, a.n_chunks);
  note_launch();
  return cudaGetLastError();
}
template <int EPI>
cudaError_t launch_rows(const LeafArgs& a, cudaStream_t s) {
  return a.hash_kind == HASH_MD5 ? launch_rows_t<HASH_MD5, EPI>(a, s) : launch_rows_t<HASH_MURMUR3, EPI>(a, s);
}
cudaError_t dispatch_rows(const LeafArgs& a, cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_rows<EPI_TREE>(a, s);
    case EPI_LIST: return launch_rows<EPI_LIST>(a, s);
    case EPI_BASIC: return launch_rows<EPI_BASIC>(a, s);
    default: return launch_rows<EPI_HASH>(a, s);
  }
}

cudaError_t dispatch_direct(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_direct<EPI_TREE>(a, c0, c1, s);
    case EPI_LIST: return launch_direct<EPI_LIST>(a, c0, c1, s);
    case EPI_BASIC: return launch_direct<EPI_BASIC>(a, c0, c1, s);
    default: return launch_direct<EPI_HASH>(a, c0, c1, s);
  }
}
cudaError_t dispatch_tma(const LeafArgs& a, const CUtensorMap& m, uint32_t n_full, int W, const LeafTune& t,
                         cudaStream_t s) {
  switch (a.epi) {
    case EPI_TREE: return launch_tma_e<EPI_TREE>(a, m, n_full, W, t, s);
    case EPI_LIST: return launch_tma_e<EPI_LIST>(a, m, n_full, W, t, s);
    case EPI_BASIC: return launch_tma_e<EPI_BASIC>(a, m, n_full, W, t, s);
    default: return launch_tma_e<EPI_HASH>(a, m, n_full, W, t, s);
  }
}
}  // namespace

namespace {
// A fixed table (no heap allocation, so that launch sites reached from the
// allocation-free entry point allocate nothing either): one entry per kernel
// instantiation that reads the input, well below the capacity.
constexpr int kMaxInputKernels = 256;
std::mutex g_input_mu;
std::pair<const void*, int> g_input_kernels[kMaxInputKernels];
int g_input_count = 0;
}  // namespace
void register_input_kernel(const void* func, int kind) {
  std::lock_guard<std::mutex> lk(g_input_mu);
  if (g_input_count < kMaxInputKernels) g_input_kernels[g_input_count++] = {func, kind};
}
int input_kernel_kind(const void* func) {
  std::lock_guard<std::mutex> lk(g_input_mu);
  for (int i = 0; i < g_input_count; i++)
    if (g_input_kernels[i].first == func) return g_input_kernels[i].second;
  return INPUT_NONE;
}

namespace {
thread_local int t_pdl_suppress = 0;
}  // namespace
PdlSuppress::PdlSuppress() { t_pdl_suppress++; }
PdlSuppress::~PdlSuppress() { t_pdl_suppress--; }
bool pdl_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("MTCHECK_PDL");
    return !(e && e[0] == '0');
  }();
  return on && t_pdl_suppress == 0;
}

static std::atomic<uint64_t> g_launches{0};
void note_launch(uint32_t n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

static int shift_rows(int hash_kind) { return hash_kind == HASH_MD5 ? 256 : 128; }

bool input_tmap(TmaCache* c, const uint8_t* data, uint64_t len, uint32_t cs, int hash_kind, const LeafTune& tune) {
  const uint32_t n_full = (uint32_t)(len / cs);
  const int W = tma_width(cs);
  int rows = tune.rows != 128 ? 256 : 128;
  if (!W || n_full == 0) return false;
  const uint32_t d = (uint32_t)(reinterpret_cast<uintptr_t>(data) & 15);
  if (d) {
    if (W < 64) return false;
    rows = shift_rows(hash_kind);
  }
  return make_tmap(c, data - d, len, cs, W, rows, n_full);
}

// Chunks without a tiled copy whose tiles are copied whole (leaf_rows_kernel): up
// to 440 bytes, where two stages of two CTAs still fit an SM (256 MiB in chunks
// of 436 bytes: 70 us, staged 125; of 24 bytes: 106, direct 124; of 63: 70 and
// 208); not multiples of 32 bytes, whose rows share banks (64 MiB in 128-byte
// chunks, before shifted boxes took them: 97 us, staged 33); not MD5 of less than a
// block, which wants the direct kernel's warps (256 MiB in 56 bytes: 199, 174).
bool rows_fit(const LeafArgs& a) {
  return a.cs <= kRowsMax && a.cs % 32 != 0 && (a.hash_kind != HASH_MD5 || a.cs >= 64);
}
// Of the others, chunks up to here are read directly: a warp's 32 chunks share
// their lines in L1, and a panel is mostly padding (400 MB in 100-byte chunks: 140 us
// direct, 226 staged; 256 MiB in 128-byte chunks off a boundary: 282 direct, 117
// staged; both before other kernels took them).
constexpr uint32_t kDirectMax = 100;
// Of the longer ones, chunks of whole 4-byte words at word addresses that are read
// directly all the same.  The direct kernel's 1536 threads per SM have three
// times as many chunks in flight as the staged one's 512 (a wave), and a word
// costs it no copy; the staged kernel's narrow copies take it one instruction per
// 4 or 8 bytes, and a chunk's last panel is copied and hashed around whole.
// Staged against direct, 4-byte aligned: MD5 1.0-1.5 from half a wave on; Murmur3
// 0.3-0.95 up to half a wave, 1.0-1.25 from there to three waves (chunks above
// about 1 KiB: from one and a half), 0.8-1.0 beyond, but 1.05-1.3 where the panels
// are a sixth longer than the chunk (160, 288, 516 bytes).  8-byte aligned: MD5
// 0.95-1.1 up to a wave, 1.0-1.2 beyond (but 0.9 for multiples of 16 above half a
// KiB), Murmur3 0.6-1.05.  Multiples of 64 bytes (0.6-1.0: direct reads of a warp's
// chunks meet in few L1 sets) and 16-byte aligned chunks (0.4-0.9) are always
// staged.
bool direct_words(const LeafArgs& a) {
  const uint64_t align = reinterpret_cast<uintptr_t>(a.data) | a.cs;
  if ((align & 3) != 0 || (align & 15) == 0 || a.cs % 64 == 0) return false;
  const uint64_t n = a.n_chunks, wave = 512ull * num_sms();
  const bool half8 = (align & 7) == 0;
  if (a.hash_kind == HASH_MD5) return half8 ? n > wave && (a.cs % 16 != 0 || a.cs < 512) : n > wave / 2;
  if (half8) return false;
  const uint64_t panels = ((uint64_t)a.cs + kPanel - 1) / kPanel * kPanel;
  if (6 * panels > 7ull * a.cs) return n > wave / 2;
  return n > (a.cs < 1100 ? 3 * wave / 4 : 3 * wave / 2) && n <= 3 * wave;
}

cudaError_t launch_leaves(const LeafArgs& a, TmaCache* cache, cudaStream_t s, const LeafTune& tune) {
  if (a.n_chunks == 0) return cudaSuccess;
  const uint32_t n_full = (uint32_t)(a.len / a.cs);
  const int W = tma_width(a.cs);
  const bool aligned = (reinterpret_cast<uintptr_t>(a.data) & 15) == 0;
  LeafTune t = tune;
  if (t.rows != 128) t.rows = 256;
  if (t.threads_per_chunk == 32 && a.cs <= kWarpChunkMax) return dispatch_warp(a, 0, a.n_chunks, s);
  if (!t.direct && (W >= 64 || (W && aligned)) && n_full > 0 && cache &&
      input_tmap(cache, a.data, a.len, a.cs, a.hash_kind, t))
    return aligned ? dispatch_tma(a, cache->map, n_full, W, t, s)
                   : dispatch_shift(a, cache->map, n_full, W, t.ctas_per_sm, s);
  if (!t.direct && rows_fit(a)) return dispatch_rows(a, s);
  if (!t.direct && a.cs > kDirectMax && !direct_words(a)) return dispatch_staged(a, 0, a.n_chunks, s);
  return dispatch_direct(a, 0, a.n_chunks, s);
}

bool batch_leaf_member(MemberLeaf* out, const LeafArgs& a) {
  const int W = tma_width(a.cs);
  const uint32_t n_full = (uint32_t)(a.len / a.cs);
  if ((W != 64 && W != 128) || n_full == 0 || (reinterpret_cast<uintptr_t>(a.data) & 15) != 0) return false;
  TmaCache cache;
  if (!make_tmap(&cache, a.data, a.len, a.cs, W, kBatchRows, n_full)) return false;
  std::memcpy(&out->map, &cache.map, sizeof(CUtensorMap));
  out->la = a;
  out->n_full = n_full;
  out->W = (uint32_t)W;
  out->xsteps = a.cs / (uint32_t)W;
  out->pad = 0;
  return true;
}

cudaError_t launch_leaf_range(const LeafArgs& a, uint32_t c0, uint32_t c1, cudaStream_t s) {
  return dispatch_direct(a, c0, c1, s);
}

static size_t batch_leaf_smem() {
  return 1024 + (size_t)kStages * kBatchStageBytes + 2 * kStages * sizeof(uint64_t) + kStages * sizeof(BatchStageMeta);
}

cudaError_t batch_leaf_node_params(const BatchLeafParams& p, cudaKernelNodeParams* kp, void** args) {
  static std::atomic<bool> attr_set{false};
  const size_t smem = batch_leaf_smem();
  if (!attr_set.load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(batch_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set.store(true, std::memory_order_release);
  }
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_leaf_kernel, kBatchRows + 32, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 3) per_sm = 3;
  uint32_t grid = (uint32_t)(num_sms() * per_sm);
  if (grid > p.nitems && p.nitems > 0) grid = p.nitems;
  args[0] = const_cast<BatchLeafParams*>(&p);
  kp->func = reinterpret_cast<void*>(batch_leaf_kernel);
  kp->gridDim = dim3(grid);
  kp->blockDim = dim3(kBatchRows + 32);
  kp->sharedMemBytes = (unsigned)smem;
  kp->kernelParams = args;
  kp->extra = nullptr;
  return cudaSuccess;
}

cudaError_t launch_leaf_inserts(const LeafArgs& a, cudaStream_t s) {
  const uint32_t wave = (uint32_t)num_sms() * 6;
  const uint32_t grid = a.fresh ? wave : sparse_grid(a.n_chunks, wave);
  // not while the hashing kernel still holds its SMs: blocks that start beside
  // it run with the little L1 its shared memory leaves (2^23 inserts into a
  // 2 GiB map: 0.16 ms slower, 1 GiB MD5 increments 6 us)
  if (a.epi == EPI_TREE) launch_with(false, leaf_insert_kernel<EPI_TREE>, grid, 256, 0, s, a);
  else launch_with(false, leaf_insert_kernel<EPI_LIST>, grid, 256, 0, s, a);
  note_launch();
  return cudaGetLastError();
}

}  // namespace mtc
