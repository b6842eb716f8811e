// Two-CTA variant of the batched tcgen05 GEMM: a cluster of two CTAs (one SM pair)
// computes one 256 x 256 tile with tcgen05.mma.cta_group::2.  Each CTA loads its own
// 128 rows of A and only HALF of B (128 of the tile's 256 columns), so shared-memory
// fill traffic per FLOP drops by a third against the one-CTA kernel and a stage shrinks
// from 48 KB to 32 KB: six stages fit where four did.
//
// Roles per CTA: warp 0 = TMA producer for this CTA's operands; warp 1 = in the leader
// CTA (cluster rank 0) the MMA issuer (idle in the other CTA); warps 2-9 = epilogue of this
// CTA's 128 accumulator rows (the epilogue code is shared with the one-CTA kernel); warp 10 = in a plan
// of several products the reporter of stored tiles; warp 11 = the scheduler, which hands out tiles.  Every
// TMA load is a per-CTA load into the CTA's own shared memory (no multicast); both CTAs' loads
// of a stage complete on ONE barrier, in the leader, which the .cta_group::2 form of the copy
// permits; only the leader's producer announces the pair's byte count on it.  The other
// cluster-wide operations are the epilogues' mbarrier arrives on the leader's barriers, the
// tcgen05.commit that arrives in both CTAs and the two cluster barriers that bracket the
// kernel.  Arrives on a peer's barrier use the default (CTA-scope) semantics: a
// `.release.cluster` arrive once per stage cost about 0.5 us each and held the whole
// pipeline to a third of its rate.
//
// Measured on a B200 against the one-CTA kernel (same call, alternating runs): the Gram iteration
// of 18 blocks of 3584 x 4096 takes 13.6-14.4 ms instead of 15.7-16.8, the whole Llama-3-8B-shaped
// optimizer step 97.5-100.5 ms instead of 100.0-103.1.  It is the default; DIONW_GEMM_CTA_PAIRS=0
// selects the one-CTA kernel.
//
// A launch runs a PLAN: one product, or the whole Newton-Schulz iterations of up to six batches (chains of
// up to 18 products that depend on one another, matrix by matrix).  In a plan of several products the tiles
// of all of them form one sequence, ordered by position in the chain and then by chain, which the pairs draw
// from a counter; `progress[b]` counts what has been stored for matrix b, and a tile's loads start once
// everything its product reads from matrix b is there.  What that buys, against one launch per product: pairs
// that run out of tiles of one product go on with the next one's, so only the last product of a plan ends in a
// part-filled wave; the start of a product (launch, descriptor fetch, first loads) and the end of the one
// before (last epilogue, teardown) overlap across matrices; and the host makes one launch where it made 15 to 18.
// Measured, an iteration as one launch per product against one plan, replayed from a graph: 16 blocks of 1024^2
// 443 -> 325 us, 16 of 1024 x 4096 810 -> 700 us, 1 of 256 x 1024 137 -> 108 us; the four batches of a 12-layer 768-wide
// language model 1108 -> 893 us, the six of a 1100-wide image encoder 964 -> 271 us, a 4-layer 4096-wide
// one's four 7.5 -> 7.1 ms.  A plan's matrices need not lie in L2 for that: running them in cohorts of two
// waves of tiles, each through all its products, changed nothing.
//
// What bounds it now, with clocks read inside the kernel, in cycles per tile (main loop / whole): K = 3584 29700 / 31800
// (530 per k-block of 512), K = 1024 8900 / 11000, K = 768 6400 / 9200.  On long main loops that is the tensor cores'
// rate at the clock the 1 kW cap leaves (1.25 GHz); on short ones the rest is the epilogue of products with a second
// term (8300 cycles of latencies, eight warps deep) and the way to the next tile's first load.  Even 16 x 1024^2 and
// 48 x 768^2 run into the cap (1.4 GHz): a cycle saved there is worth about half.  Sixteen epilogue warps, each with half
// the columns, were 10 to 25 % slower (96 registers a thread: spills); five stages instead of six cost 1 %.
//
// Why a plan cannot deadlock, whatever else runs on the GPU: tiles are drawn in order by pairs that are
// already running, and a tile depends only on tiles before it.  The earliest unfinished tile is therefore
// held by a running pair whose wait is over.
//
// Every spin-wait is bounded, as in the one-CTA kernel.
#pragma once

#include "cluster.cuh"
#include "gemm_sm100.cuh"

namespace dionw {
namespace gemm2 {

using gemm::Params;
using gemm::Tile;

constexpr int kPairM = 256;                        // rows of a pair's tile
constexpr int kBM = 128;                           // rows per CTA
constexpr int kBN = 256;
constexpr int kBK = 64;
constexpr int kStages = 6;
constexpr int kEpilogueWarps = 8;
constexpr int kReporterWarp = 2 + kEpilogueWarps;
constexpr int kSchedulerWarp = kReporterWarp + 1;
constexpr int kThreads = 32 * (kSchedulerWarp + 1);
constexpr uint32_t kBarrierBytes = 832;
constexpr uint32_t kABytes = kBM * kBK * 2;        // 16 KB
constexpr uint32_t kBBytes = (kBN / 2) * kBK * 2;  // 16 KB: the half of B's columns that each CTA loads
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kPanelBytes = 64 * kBK * 2;     // one 64-column panel of an MN-major operand
constexpr size_t kSmemBytes = size_t(kStages) * kStageBytes + 1024 + kBarrierBytes +
                              kEpilogueWarps * 2 * gemm::kPieceBytes;

__device__ __forceinline__ void remote_arrive(uint32_t cluster_address) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}

// Relaxed arrive that is issued once `loaded`, made of the results of one or more loads, is there: the arrive is
// predicated on the value, which is never kNoTile.  (Relaxed, so the memory model does not order the loads before
// it; the dependency does, since an instruction is not issued before its predicate is known.  The comparison is
// with the largest integer because no branch on the sign of an entry's step decides it.)
constexpr int kNoTile = 0x7FFFFFFF;   // no step, number of k-blocks or map
__device__ __forceinline__ void remote_arrive_after(uint32_t cluster_address, int loaded) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.s32 p, %1, %2;\n"
               "@p mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];\n}\n"
               ::"r"(cluster_address), "r"(loaded), "n"(kNoTile) : "memory");
}

// An entry of the tile ring: the product of the plan (negative: no more tiles), the tile of it, and what the
// loads and the main loop need to know about the two (see entry_of), so that neither waits for the parameters of a
// product it has not met yet: read from the kernel's arguments they took 700 cycles between tile and first load.
struct alignas(16) Entry {
  int step, batch, tm, tn;
  int k_blocks, a_end, b_end, flags;
  int map_a, map_b, map_a_mn, map_b_mn;
};
constexpr int kSharedFlag = 1, kWideFlag = 2;
constexpr int kEntryWords = sizeof(Entry) / sizeof(int4);

// Stores an entry in the peer's shared memory and counts its bytes on a barrier there, which releases it: the
// sender waits for nothing.  (A store and an arrive with release at cluster scope took the sender 1700 cycles.)
__device__ __forceinline__ void send_entry(uint32_t cluster_address, uint32_t cluster_bar, const Entry& e) {
  const int4* words = reinterpret_cast<const int4*>(&e);
#pragma unroll
  for (int i = 0; i < kEntryWords; ++i)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(cluster_address + 16 * i), "r"(words[i].x), "r"(words[i].y), "r"(words[i].z), "r"(words[i].w),
                 "r"(cluster_bar) : "memory");
}

// Word i of an entry; one instruction, so what depends on one of its fields depends on all of them.
__device__ __forceinline__ void load_entry_word(const Entry* from, int i, Entry& e) {
  int4& w = reinterpret_cast<int4*>(&e)[i];
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(gemm::smem_u32(from) + 16 * i) : "memory");
}
// The entry, but for its last word(s) where they are not needed; the tile itself is in the first, which is read last.
template <int kWords>
__device__ __forceinline__ Entry load_entry(const Entry* from) {
  Entry e{};
#pragma unroll
  for (int i = kWords - 1; i >= 0; --i) load_entry_word(from, i, e);
  return e;
}

__device__ __forceinline__ bool mbar_try_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(gemm::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait with the acquire at cluster scope (see gemm::mbar_wait for the protocol).
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                                  uint64_t limit_ns) {
  uint32_t spins = 0;
  uint64_t start = 0;
  while (!mbar_try_cluster(bar, parity)) {
    if ((++spins & 1023u) == 0) {
      if (*abort_flag != 0) return false;
      const uint64_t now = gemm::global_ns();
      if (start == 0) start = now;
      else if (now - start > limit_ns) {
        *abort_flag = 1;
        if (status != nullptr) atomicExch(status, gemm::kWaitCode);
        return false;
      }
    }
  }
  return true;
}

// TMA load into this CTA's shared memory whose completion is signalled on a barrier of the
// pair's leader CTA (the .cta_group::2 form allows the barrier to be the peer's).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t smem_dst, const CUtensorMap* map, uint32_t leader_bar, int c0,
                                                 int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tmem_alloc2(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(gemm::smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc2(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

__device__ __forceinline__ void umma2_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on the barrier at this offset in BOTH CTAs once the pair's MMAs issued so far have completed.
__device__ __forceinline__ void umma2_commit_both(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          gemm::smem_u32(bar)),
      "h"(mask)
      : "memory");
}

// Instruction descriptor: fp32 accumulate, M = 256 (128 rows in each CTA), N = 256 or 128.
template <typename T>
__device__ __forceinline__ uint32_t make_idesc2(bool a_major_mn, bool b_major_mn, int tile_n) {
  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  uint32_t d = 0;
  d |= 1u << 4;
  d |= fmt << 7;
  d |= fmt << 10;
  d |= (a_major_mn ? 1u : 0u) << 15;
  d |= (b_major_mn ? 1u : 0u) << 16;
  d |= uint32_t(tile_n >> 3) << 17;
  d |= uint32_t(kPairM >> 4) << 24;
  return d;
}

// ----------------------------------------------------------------------------
// plans
// ----------------------------------------------------------------------------
struct Step {
  Params p;               // tiles_m, tiles_n, tiles_per_batch count tiles of 256 x tile_n
  short map_a, map_b;     // indices into the plan's maps
  short map_a_t, map_b_t; // of a lower operand: the map for the blocks that are read transposed
  int first_tile;         // tiles of the plan before this product
  unsigned need;          // progress of a matrix from which on this product may read it
  unsigned* progress;     // of the chain's matrices: zero at the start of the launch (null: one product only)
  short tile_n;           // 256 or 128
  bool symmetric;         // only tiles on and below the diagonal
  bool a_major_mn, b_major_mn;
  bool a_lower, b_lower;  // the operand is a symmetric matrix of which only the 256 x 256 blocks up to the diagonal are stored
  bool same_operands;     // a tile on the diagonal has the same rows of A and of B
  bool out_bf16;          // the result is bf16 although the operands are fp16
};

template <int kMaps, int kSteps>
struct Plan {
  CUtensorMap maps[kMaps];
  Step steps[kSteps];
  int count;
  int total_tiles;
  int* tile_counter;      // {next tile, pairs done} in global memory, or null for a fixed stride (one product only)
  DecayJob* job;          // streaming job the epilogue warps work on while they wait, or null
  int* status;
  uint64_t wait_ns;
};
constexpr unsigned kReportsPerTile = 2;   // each CTA reports its half

// General: groups of 4 tile rows sweep the columns.
__device__ __forceinline__ Tile general_tile(int t, const Params& p) {
  Tile tile;
  tile.batch = t / p.tiles_per_batch;
  int r = t - tile.batch * p.tiles_per_batch;
  const int group_rows = 4;
  const int per_group = group_rows * p.tiles_n;
  const int g = r / per_group;
  const int first = g * group_rows;
  const int rows_here = min(group_rows, p.tiles_m - first);
  r -= g * per_group;
  tile.tm = first + r % rows_here;
  tile.tn = r / rows_here;
  return tile;
}

// Symmetric: tile row i needs the columns up to its own end, (i + 1) * per_row tiles (per_row = 256 / tile_n);
// per_row * i(i+1)/2 tiles precede row i.  (Walking the triangle in groups of four tile rows swept by
// columns, as the general schedule does, was measured and dropped: 18 blocks of 3584^2, K = 3584,
// 664 / 707 / 801 / 804 us against 646 / 733 / 776 / 740 us for A A^T plain / with Cin / with two
// outputs / with B != A -- no better on balance.)
__device__ __forceinline__ Tile sym_tile(int t, const Params& p, int per_row) {
  Tile tile;
  tile.batch = t / p.tiles_per_batch;
  const int r = t - tile.batch * p.tiles_per_batch;
  const int u = r / per_row;
  int i = int((sqrtf(8.0f * float(u) + 1.0f) - 1.0f) * 0.5f);
  while (i * (i + 1) / 2 > u) --i;
  while ((i + 1) * (i + 2) / 2 <= u) ++i;
  tile.tm = i;
  tile.tn = r - per_row * (i * (i + 1) / 2);
  return tile;
}

__device__ __forceinline__ Tile tile_of(int t, const Step& step) {
  return step.symmetric ? gemm2::sym_tile(t, step.p, kBN / step.tile_n) : gemm2::general_tile(t, step.p);
}

// How a tile's k-blocks are read: A in rows (K-major) up to a_end and B up to b_end <= a_end, and in columns
// (MN-major) from there on; with kSharedFlag A's rows serve as B's.  Of a symmetric matrix that a product of the plan left, only the 256 x 256 blocks up to the
// diagonal exist: what lies right of the diagonal in a row is read from the column it is equal to.  The tensor
// cores take either order, so nothing is stored twice: a mirrored copy was half of all bytes the products wrote,
// and the write path, at 20 to 25 bytes per cycle and SM, what their epilogues waited for (1300 to 2900 of 2500 to
// 4600 cycles per 32-column chunk).
__device__ __forceinline__ Entry entry_of(const Step& step, int at, const Tile& tile) {
  constexpr int kPerBlock = kPairM / kBK;
  const int k_blocks = (step.p.kdim + kBK - 1) / kBK;
  const int column_block = step.tile_n == kBN ? tile.tn : tile.tn >> 1;
  const bool shared = step.same_operands && step.tile_n == kBN && tile.tm == tile.tn;
  Entry e;
  e.step = at;
  e.batch = tile.batch;
  e.tm = tile.tm;
  e.tn = tile.tn;
  e.k_blocks = k_blocks;
  e.a_end = step.a_major_mn ? 0 : step.a_lower ? min(k_blocks, (tile.tm + 1) * kPerBlock) : k_blocks;
  e.b_end = step.b_major_mn ? 0 : step.b_lower ? min(k_blocks, (column_block + 1) * kPerBlock) : k_blocks;
  e.flags = (shared ? kSharedFlag : 0) | (step.tile_n == kBN ? kWideFlag : 0);
  e.map_a = step.map_a;
  e.map_b = step.map_b;
  e.map_a_mn = step.a_lower ? step.map_a_t : step.map_a;
  e.map_b_mn = step.b_lower ? step.map_b_t : step.map_b;
  return e;
}

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void add_release(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// One lane of a converged warp, as the compiler understands it.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
  return one != 0;
}

// Orders this thread's accesses to global memory through the generic proxy (ordinary loads and stores) with those of
// the async proxy (TMA) on both sides.
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// Bounded wait until the progress of a matrix has reached `need`.
__device__ __forceinline__ bool progress_wait(const unsigned* progress, unsigned need, volatile int* abort_flag,
                                              int* status, uint64_t limit_ns) {
  uint32_t spins = 0;
  uint64_t start = 0;
  while (load_acquire(progress) < need) {
    if ((++spins & 255u) == 0) {
      if (*abort_flag != 0) return false;
      const uint64_t now = gemm::global_ns();
      if (start == 0) start = now;
      else if (now - start > limit_ns) {
        *abort_flag = 1;
        if (status != nullptr) atomicExch(status, gemm::kWaitCode);
        return false;
      }
    }
  }
  return true;
}

// ----------------------------------------------------------------------------
// tile hand-out
// ----------------------------------------------------------------------------
// A pair takes its tiles either in a fixed stride (tile = pair, pair + pairs, ...: no shared state)
// or from a counter in global memory, one atomicAdd per tile (Plan::tile_counter non-null).  The
// second form is for products that run beside other kernels (NCCL's, another stream's): a pair whose
// CTAs become resident late, or not before the others are done, simply takes fewer tiles, where the
// fixed stride makes the whole product wait for it.
//
// A warp of its own in each CTA, the scheduler, does the hand-out, ahead of the loads.  The leader's draws the
// index, finds the product and the tile that it stands for, and publishes them to every consumer of the pair
// through a ring of kTileSlots entries kept in BOTH CTAs' shared memory: it writes its own copy and arrives on
// the slot's `tile_full` barrier, and sends the peer's, where the bytes themselves complete the phase that the
// peer's scheduler has armed.  Consumers -- the leader's MMA issuer, the producer and the epilogue warps
// of each CTA, the peer's scheduler -- wait on their own
// CTA's `tile_full` (acquire at cluster scope), read the entry and arrive on the LEADER's `tile_empty`
// barrier of the slot; the scheduler reuses a slot after all of them have done so.  A negative step ends the pair's work.
// When a pair has drawn its end it adds one to a second counter; the pair that brings that to the number
// of pairs knows that nobody will draw again and clears both counters for the next launch on the stream.
// In a plan of several products each CTA's scheduler then waits for what the tile depends on, and tells its
// own CTA's producer and its epilogue warps, which read Cin, through the slot's `ready` barrier.  (Waiting before the tile is
// published, so that the ring itself carries the news, put the ring's two cluster-scope hops on the path
// from one product to the next.)  Who waits for `ready` reports the slot as read only then, so
// that the barrier is never more than one phase ahead of it.
//
// When the leader draws its next tile: once what the current one reads is there, and not before the current
// one's loads are within kDrawAhead k-blocks of their end (its first tile, which waits for nothing while other
// pairs may not have started: at their end).  Earlier, a pair that waits for a product's inputs would take two of
// its tiles while other pairs get none, and a product of 66 tiles on 74 pairs take two tiles' time (1 block of
// 2816 x 2927: 788 us so, 514 without).  Later, the way from the draw to the first load is not hidden behind the
// current tile: when the producer itself drew, decoded, published, waited and loaded in turn, the tensor pipe had
// nothing to do for 4500 of the 15000 cycles of a 1024-deep tile.
//
// A CTA's half of a tile is reported by a warp of its own, once the eight epilogue warps have arrived on the
// slot's `stored` barrier: the release at GPU scope waits until the stores have reached L2, and took an
// epilogue warp 2700 cycles of every tile.  The reporter, too, reports the slot as read only then.
// For the same reason the arrivals on `tile_empty` are relaxed: they have to follow the read of the slot, which
// their predicate depends on, and not the stores of the tile before (as a release at cluster scope each cost
// the warp 2000 cycles per tile).
constexpr int kTileSlots = 8;
constexpr uint32_t kTileConsumers = 2 + 2 * (1 + kEpilogueWarps);   // and the reporters, in a plan of several products
constexpr int kDrawAhead = 24;

// ----------------------------------------------------------------------------
// the kernel (launched as clusters of two CTAs)
// ----------------------------------------------------------------------------
template <typename InT, int kMaps, int kSteps>
__global__ void __launch_bounds__(kThreads, 1)
gemm2_kernel(const __grid_constant__ Plan<kMaps, kSteps> plan) {
  using namespace gemm;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + size_t(kStages) * kStageBytes);  // leader's: both CTAs' stage landed
  uint64_t* empty_bar = full_bar + kStages;   // both: the pair's MMAs on this stage completed
  uint64_t* acc_full = empty_bar + kStages;   // [2] both: accumulator complete
  uint64_t* acc_empty = acc_full + 2;         // [2] leader only: both CTAs' epilogues drained it
  uint64_t* tile_full = acc_empty + 2;        // [kTileSlots] both: the slot's tile index is written
  uint64_t* tile_empty = tile_full + kTileSlots;  // [kTileSlots] leader only: every consumer has read the slot
  uint64_t* ready = tile_empty + kTileSlots;      // [kTileSlots] both: what the slot's tile reads is there
  uint64_t* stored = ready + kTileSlots;          // [kTileSlots] both: this CTA's half of the slot's tile is stored
  Entry* tile_ring = reinterpret_cast<Entry*>(stored + kTileSlots);  // [kTileSlots] both
  uint64_t* may_draw = reinterpret_cast<uint64_t*>(tile_ring + kTileSlots);   // leader's: its scheduler may draw again
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(may_draw + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* mirror_stage = smem + size_t(kStages) * kStageBytes + kBarrierBytes;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();       // 0 = leader
  const int pair = blockIdx.x >> 1;
  const int pairs = gridDim.x >> 1;
  const int total_tiles = plan.total_tiles;
  const bool dynamic = kSteps > 1 || plan.tile_counter != nullptr;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);   // the leader's producer arrives once with the pair's byte count
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 2 * kEpilogueWarps);
    }
    for (int s = 0; s < kTileSlots; ++s) {
      mbar_init(&tile_full[s], 1);
      mbar_init(&tile_empty[s], kTileConsumers + (kSteps > 1 ? 2 : 0));
      mbar_init(&ready[s], 1);
      mbar_init(&stored[s], kEpilogueWarps);
    }
    mbar_init(may_draw, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 2 && lane < (kMaps < 32 ? kMaps : 32)) prefetch_map(&plan.maps[lane]);
  if (warp == 1) tmem_alloc2(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // both CTAs' barriers exist before anyone arrives on a peer's
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  gemm::griddep_wait();     // set-up above overlaps the tail of the previous product; global memory from here on
  gemm::griddep_launch();

  // All lanes of a warp wait; false for all of them when one gave up.
  auto warp_wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, plan.status, plan.wait_ns)) != 0;
  };
  auto warp_wait_cluster = [&](uint64_t* bar, uint32_t parity) -> bool {
    return __all_sync(0xffffffffu, mbar_wait_cluster(bar, parity, abort_flag, plan.status, plan.wait_ns)) != 0;
  };
  // The n-th tile of this pair for a consumer; its step is -1 when the pair is done and -2 when the wait gave up.
  // Called by whole warps: every lane waits and reads, and one reports the slot as read once all of them have.
  // (Where one lane handed the entry to the others by shuffles the first load of a tile came 650 cycles later.)
  const uint32_t leader_tile_empty = peer_address(&tile_empty[0], 0);
  auto take_tile = [&](uint32_t n, bool when_ready, auto words) -> Entry {
    Entry none{};
    none.step = -1;
    if (!dynamic) {
      const long long t = (long long)pair + (long long)n * pairs;
      if (t >= total_tiles) return none;
      return entry_of(plan.steps[0], 0, tile_of(int(t), plan.steps[0]));
    }
    none.step = -2;
    const uint32_t slot = n % kTileSlots, phase = (n / kTileSlots) & 1u;
    if (!warp_wait_cluster(&tile_full[slot], phase)) return none;
    const Entry e = load_entry<decltype(words)::value>(&tile_ring[slot]);
    if (kSteps > 1 && when_ready && e.step >= 0 && !warp_wait(&ready[slot], phase)) return none;
    // a value of every load of every lane
    constexpr int kWords = decltype(words)::value;
    const bool none_there = e.step == kNoTile || (kWords > 1 && e.k_blocks == kNoTile) || (kWords > 2 && e.map_a == kNoTile);
    const int seen = __any_sync(0xffffffffu, none_there) ? kNoTile : 0;
    if (lane == 0) remote_arrive_after(leader_tile_empty + slot * uint32_t(sizeof(uint64_t)), seen);
    return e;
  };
  const std::integral_constant<int, 1> kTileOnly{};
  const std::integral_constant<int, 2> kTileAndRanges{};
  const std::integral_constant<int, 3> kWholeEntry{};

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    // A whole warp of which one elected lane issues, as in the MMA issuer.
    int s = 0;                 // stage of the ring, and the parity that its slot's next release has
    uint32_t released = 1;
    bool ok = true;
    const uint32_t ring = smem_u32(smem), leader_full = peer_address(full_bar, 0);
    for (uint32_t n = 0; ok; ++n) {
      const Entry tile = take_tile(n, true, kWholeEntry);
      if (tile.step < 0) break;
      const bool shared = (tile.flags & kSharedFlag) != 0;
      const int tile_n = (tile.flags & kWideFlag) != 0 ? kBN : kBN / 2, half_n = tile_n / 2;
      const int m0 = tile.tm * kPairM + int(rank) * kBM;
      const int n0 = tile.tn * tile_n + int(rank) * half_n;
      // the k-block after whose loads this pair's next tile may be drawn
      const int draw_at = !dynamic || rank != 0 ? -1 : n == 0 ? tile.k_blocks - 1 : max(0, tile.k_blocks - kDrawAhead);
      const uint32_t pair_bytes = 2 * (kABytes + (shared ? 0u : uint32_t(half_n) * kBK * 2));
      // The layout of the operands is a constant inside the loop.
      auto load_loop = [&](int begin, int end, auto a_major_mn, auto b_major_mn) {
        constexpr bool kAMN = decltype(a_major_mn)::value, kBMN = decltype(b_major_mn)::value;
        if (!ok || begin >= end) return;
        const CUtensorMap* map_a = &plan.maps[kAMN ? tile.map_a_mn : tile.map_a];
        const CUtensorMap* map_b = &plan.maps[kBMN ? tile.map_b_mn : tile.map_b];
        for (int kb = begin; kb < end; ++kb) {
          if (!warp_wait(&empty_bar[s], released)) { ok = false; break; }
          const uint32_t a_dst = ring + uint32_t(s) * kStageBytes, b_dst = a_dst + kABytes;
          const uint32_t landed = leader_full + uint32_t(s) * uint32_t(sizeof(uint64_t));
          const int k0 = kb * kBK;
          if (elect_one()) {
            // The peer's bytes may land before the leader has announced them: the phase still
            // cannot complete before the leader's arrive, and the peer cannot run a phase ahead
            // because its empty barrier is released by the MMAs that consumed this one.
            if (rank == 0) mbar_expect_tx(&full_bar[s], pair_bytes);
            if constexpr (kAMN) {
#pragma unroll
              for (int panel = 0; panel < kBM / 64; ++panel)
                tma_load_3d_pair(a_dst + panel * kPanelBytes, map_a, landed, m0 + panel * 64, k0, tile.batch);
            } else {
              tma_load_3d_pair(a_dst, map_a, landed, k0, m0, tile.batch);
            }
            if (!shared) {
              if constexpr (kBMN) {
                tma_load_3d_pair(b_dst, map_b, landed, n0, k0, tile.batch);
                if (half_n > 64) tma_load_3d_pair(b_dst + kPanelBytes, map_b, landed, n0 + 64, k0, tile.batch);
              } else {
                tma_load_3d_pair(b_dst, map_b, landed, k0, n0, tile.batch);
              }
            }
            if (kb == draw_at) mbar_arrive(may_draw);
          }
          __syncwarp();
          if (++s == kStages) s = 0, released ^= 1u;
        }
      };
      load_loop(0, tile.b_end, std::false_type(), std::false_type());
      load_loop(tile.b_end, tile.a_end, std::false_type(), std::true_type());
      load_loop(tile.a_end, tile.k_blocks, std::true_type(), std::true_type());
    }
  } else if (warp == 1) {
    if (rank == 0) {   // the second CTA's MMA warp has nothing to issue
      // ------------------------------------------------------------ MMA issuer (leader)
      // The whole warp goes through the loop and one elected lane issues: the descriptors of an MMA are uniform
      // registers, which the compiler can only keep there where the warp is converged.  Issued by a thread of its own,
      // an MMA took 140 to 190 cycles to issue and 128 to run (64 on a tile of 128 columns).
      int s = 0;                 // stage of the ring, and the parity that its next load completes
      uint32_t loaded = 0;
      bool ok = true;
      const uint32_t ring = smem_u32(smem);
      for (uint32_t local = 0; ok; ++local) {
        const Entry tile = take_tile(local, false, kTileAndRanges);
        if (tile.step < 0) break;
        const uint32_t acc = local & 1u;
        const uint32_t acc_phase = (local >> 1) & 1u;
        if (!warp_wait(&acc_empty[acc], acc_phase ^ 1u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * uint32_t(kBN);
        const uint32_t b_offset = (tile.flags & kSharedFlag) != 0 ? 0u : kABytes;
        const int tile_n = (tile.flags & kWideFlag) != 0 ? kBN : kBN / 2;
        // The layout of the operands is a constant inside the loop.
        auto main_loop = [&](int begin, int end, auto a_major_mn, auto b_major_mn) {
          constexpr bool kAMN = decltype(a_major_mn)::value, kBMN = decltype(b_major_mn)::value;
          if (!ok) return;
          const uint32_t idesc = make_idesc2<InT>(kAMN, kBMN, tile_n);
          for (int kb = begin; kb < end; ++kb) {
            if (!warp_wait(&full_bar[s], loaded)) { ok = false; break; }
            tc_fence_after();
            const uint32_t a_addr = ring + uint32_t(s) * kStageBytes;
            const uint32_t b_addr = a_addr + b_offset;
            const uint64_t a_desc = make_smem_desc(a_addr, kAMN ? kPanelBytes : 16, 1024);
            const uint64_t b_desc = make_smem_desc(b_addr, kBMN ? kPanelBytes : 16, 1024);
            if (elect_one()) {
#pragma unroll
              for (int j = 0; j < kBK / kUmmaK; ++j) {
                const uint64_t k_step = uint64_t((j * kUmmaK * 2) >> 4), mn_step = uint64_t((j * kUmmaK * 128) >> 4);
                umma2_f16(tmem_d, a_desc + (kAMN ? mn_step : k_step), b_desc + (kBMN ? mn_step : k_step), idesc,
                          (kb > 0 || j > 0) ? 1u : 0u);
              }
              umma2_commit_both(&empty_bar[s]);
            }
            __syncwarp();
            if (++s == kStages) s = 0, loaded ^= 1u;
          }
        };
        main_loop(0, tile.b_end, std::false_type(), std::false_type());
        main_loop(tile.b_end, tile.a_end, std::false_type(), std::true_type());
        main_loop(tile.a_end, tile.k_blocks, std::true_type(), std::true_type());
        if (ok && elect_one()) umma2_commit_both(&acc_full[acc]);
        __syncwarp();
      }
    }
  } else if (warp == kReporterWarp) {
    // ------------------------------------------------------------ reporter (both CTAs)
    if (kSteps > 1 && lane == 0) {
      for (uint32_t n = 0;; ++n) {
        const uint32_t slot = n % kTileSlots, phase = (n / kTileSlots) & 1u;
        if (!mbar_wait_cluster(&tile_full[slot], phase, abort_flag, plan.status, plan.wait_ns)) break;
        const Entry tile = load_entry<1>(&tile_ring[slot]);
        if (tile.step < 0) break;
        unsigned* progress = &plan.steps[tile.step].progress[tile.batch];
        if (!mbar_wait(&stored[slot], phase, abort_flag, plan.status, plan.wait_ns)) break;
        // The tile's stores are there for later tiles once it is counted (their producers order the
        // proxies: the stores went through the generic one, TMA reads through the async one).
        add_release(progress, 1u);
        remote_arrive_after(leader_tile_empty + slot * uint32_t(sizeof(uint64_t)), tile.step);
      }
    }
  } else if (warp == kSchedulerWarp) {
    // ------------------------------------------------------------ scheduler (both CTAs)
    if (dynamic && lane == 0) {
      if (rank != 0) mbar_expect_tx(&tile_full[0], sizeof(Entry));
      int at = 0;   // the product of the last tile drawn: tiles only ever grow
      for (uint32_t n = 0;; ++n) {
        const uint32_t slot = n % kTileSlots, phase = (n / kTileSlots) & 1u;
        Entry e;
        if (rank == 0) {
          if (n != 0 && !mbar_wait(may_draw, (n - 1) & 1u, abort_flag, plan.status, plan.wait_ns)) break;
          const int t = atomicAdd(plan.tile_counter, 1);
          if (t < total_tiles) {
            if constexpr (kSteps > 1) {
              while (at + 1 < plan.count && t >= plan.steps[at + 1].first_tile) ++at;
            }
            e = entry_of(plan.steps[at], at, tile_of(t - plan.steps[at].first_tile, plan.steps[at]));
          } else {
            e = Entry{};
            e.step = -1;
          }
          if (!mbar_wait_cluster(&tile_empty[slot], phase ^ 1u, abort_flag, plan.status, plan.wait_ns)) break;
          send_entry(peer_address(&tile_ring[slot], 1), peer_address(&tile_full[slot], 1), e);
          tile_ring[slot] = e;
          mbar_arrive(&tile_full[slot]);
          if (e.step < 0) {
            // nobody of this pair draws again; the last pair to get here clears the counters
            if (atomicAdd(plan.tile_counter + 1, 1) == pairs - 1) {
              plan.tile_counter[0] = 0;
              plan.tile_counter[1] = 0;
              __threadfence();
            }
            break;
          }
        } else {
          if (!mbar_wait_cluster(&tile_full[slot], phase, abort_flag, plan.status, plan.wait_ns)) break;
          e = load_entry<1>(&tile_ring[slot]);
          remote_arrive_after(leader_tile_empty + slot * uint32_t(sizeof(uint64_t)), e.step);
          if (e.step < 0) break;
          mbar_expect_tx(&tile_full[(n + 1) % kTileSlots], sizeof(Entry));   // its last phase is over: this thread has seen it
        }
        if constexpr (kSteps > 1) {
          const Step& step = plan.steps[e.step];
          if (step.need != 0) {
            if (!progress_wait(&step.progress[e.batch], step.need, abort_flag, plan.status, plan.wait_ns)) break;
            proxy_fence();   // what the tile reads was stored through the generic proxy, by other SMs
          }
          mbar_arrive(&ready[slot]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (both CTAs)
    const int ew = warp - 2;
    const int sub = warp & 3;
    uint8_t* stage = mirror_stage + ew * 2 * kPieceBytes;
    const uint32_t leader_empty[2] = {peer_address(&acc_empty[0], 0), peer_address(&acc_empty[1], 0)};
    for (uint32_t local = 0;; ++local) {
      const Entry tile = take_tile(local, true, kTileOnly);
      if (tile.step < 0) break;
      const Step& step = plan.steps[tile.step];
      const Params& p = step.p;
      const int chunks = step.tile_n / (32 * kEpilogueWarps / 4);
      const int first_chunk = (ew >> 2) * chunks;
      const uint32_t acc = local & 1u;
      const uint32_t acc_phase = (local >> 1) & 1u;
      // The streaming job rides on products whose main loop is long enough to hide a row behind it.
      if (plan.job != nullptr && p.kdim >= 24 * kBK) {
        // The accumulator of this tile is still being summed: take rows of the streaming job
        // meanwhile, at most `per_wait` of them, one at a time, looking at the barrier in between.
        const int limit = plan.job->per_wait;
        for (int taken = 0; taken < limit; ++taken) {
          long long row = -1;
          if (lane == 0 && !mbar_try(&acc_full[acc], acc_phase)) row = atomicAdd(&plan.job->cursor, 1);
          row = __shfl_sync(0xffffffffu, row, 0);
          if (row < 0 || row >= plan.job->total_rows) break;
          decay_job_row(plan.job, row, lane);
        }
      }
      const int m_base = tile.tm * kPairM + int(rank) * kBM, n_base = tile.tn * step.tile_n;
      const uint32_t tmem_acc = tmem_base + acc * uint32_t(kBN);
      auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) remote_arrive(leader_empty[acc]);
      };
      auto epilogue = [&](auto symmetric) {
        return epilogue_tile<InT, decltype(symmetric)::value>(
            p, tile.batch, m_base, n_base, tmem_acc, &acc_full[acc], acc_phase, abort_flag, stage, sub, lane, first_chunk,
            chunks, step.out_bf16, release);
      };
      const bool done = step.symmetric ? epilogue(std::true_type()) : epilogue(std::false_type());
      if (!done) break;
      if constexpr (kSteps > 1) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&stored[local % kTileSlots]);
      }
    }
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0 && threadIdx.x == 0) {
    const uint64_t start = global_ns();
    while (global_ns() - start < 200000ull) {
    }
  }
  cluster_sync();   // the peer may still be reading this CTA's shared memory through the pair's MMAs
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc2(tmem_base, kTmemCols);
  }
}

}  // namespace gemm2
}  // namespace dionw
