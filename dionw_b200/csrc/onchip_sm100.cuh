// The Gram iteration of a batch whose shorter side m is at most 256, as one launch in which a matrix never
// leaves the SMs that work on it: a cluster of 1 to 8 SM pairs per matrix of the batch.  Every pair computes
// G = X X^T over all of X and the whole chain of m x m products on it; only Q X, whose n columns are split,
// is shared.  What pairs repeat costs no time (the other SMs have nothing to do) and saves every exchange
// but one: a cluster barrier between X <- Q X and the next X X^T.
//
// A pair holds the three m x m matrices that are alive at a time in shared memory.  Each CTA has 128 rows of
// every matrix, 64 KB, in the K-major layout that the tensor cores read: its rows are its half of A, and as
// the matrices are symmetric also its half of B.  A product is up to 16 steps of tcgen05.mma.cta_group::2
// (256 x 256 x 16) into TMEM, from where the epilogue warps write the result over a matrix that is no longer
// read.  X passes through a ring that lies over matrices which are dead meanwhile.  Same instructions on the
// same values in the same order as gemm2_kernel, the same rounding and the same lower triangle mirrored:
// the same bits.
//
// Roles per CTA: warp 0 = in the leader the MMA issuer, in the second CTA the forwarder of its news; warps 1-16 =
// epilogue, warp w has the 32 rows of TMEM sub-partition w % 4 and one or two of their 32-column pieces up
// to the diagonal (of Q X warps 1-8 have the even tiles and warps 9-16 the odd ones, four pieces a warp); warp 17 =
// TMA producer.  A product begins when the columns up to 128 of its operands are there, which are all warps'
// first pieces.  What it reads from its ninth step on follows meanwhile: the second CTA's second pieces, and in
// the leader's rows the mirror images of the second CTA's first ones: two warps put 64 rows of those together,
// and a bulk copy takes them there.
//
// Bounded by the latency of the chain, 14 dependent products.  With clocks read inside the kernel (1965 MHz) one takes
// 5100 to 5900 cycles from its operands' first half to the next one's for m = 256, 2048 of them MMA and the rest epilogue and
// signals, which nothing hides; 4300 to 4800 for m = 192, 3100 for 128, 2600 for 96.  X X^T takes 523 cycles per 64 columns and
// 4300 besides, twice.  As a plan (gemm2_sm100.cuh) a product of one 256 x 256 matrix took 12600 cycles, most of them the
// way through L2: stores, report, flag, first loads.
#pragma once

#include "gemm2_sm100.cuh"

namespace dionw {
namespace onchip {

using namespace gemm;

constexpr int kSide = 256;                           // largest m
constexpr int kRows = 128;                           // rows per CTA
constexpr uint32_t kPanelBytes = kRows * 128;        // 64 columns of a matrix
constexpr uint32_t kMatrixBytes = 4 * kPanelBytes;
constexpr int kSlots = 3;
constexpr int kMaxOps = 10;
constexpr int kStages = 8;                           // of the ring: two slots
constexpr uint32_t kStageBytes = kRows * gemm2::kBK * 2;
constexpr int kEpilogueWarps = 16;
constexpr int kTileWarps = 8;                        // of them, on a tile of Q X
constexpr int kProducerWarp = 1 + kEpilogueWarps;
constexpr int kThreads = 32 * (kProducerWarp + 1);
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kBarrierBytes = 320;
constexpr uint32_t kNowhereBytes = 32 * 16;
// (Clusters above 8 CTAs are not portable, and only taken where the device says that all of them run at a time: 1 block of
// 256 x 2048 82 -> 79 us with up to 8 pairs instead of 4, of 256 x 6000 134 -> 123.)
constexpr int kMaxPairs = 8;
constexpr size_t kSmemBytes = 1024 + size_t(kSlots) * kMatrixBytes + kBarrierBytes + kEpilogueWarps * kPieceBytes + kNowhereBytes;
static_assert(kStages * kStageBytes == 2 * kMatrixBytes, "the ring lies over two slots");

// out = alpha A B + beta Cin; matrices are slots.  `out` may be a slot that is read: it is written once the
// accumulator is complete, and each piece of Cin is read by the warp that writes it.  The first of a part
// is X X^T: no operands, no Cin.
struct Op {
  int8_t a, b, cin, out, out2;   // out2: out + diag on the diagonal; -1: none
  float alpha, beta, diag;
};
// Twice: X X^T -> slot 0, the chain, slot 2 times X.
struct Iteration {
  CUtensorMap x[2][2];           // X of each part, boxes of 128 and of 64 rows
  Op ops[2][kMaxOps];
  int count[2];
  Params result[2];              // Q X
  bool result_bf16[2];
  bool tall;                     // X is n x m: X^T X and X Q
  int m, n;
  int pairs;                     // of a cluster
  int* status;
  uint64_t wait_ns;
};

// Arrives on the barrier at this offset in both CTAs of the pair once the pair's MMAs issued so far have completed.
__device__ __forceinline__ void commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t t;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t) : "r"(v));
  return t;
}

// Copies `bytes` (a multiple of 16) from this CTA's shared memory to another's; they count on a barrier there.
__device__ __forceinline__ void copy_to_peer(uint32_t cluster_dst, const void* src, uint32_t bytes, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(cluster_dst), "r"(smem_u32(src)), "r"(bytes), "r"(cluster_bar) : "memory");
}

// Orders this thread's ordinary accesses to its CTA's shared memory with the tensor cores' and copies'.
__device__ __forceinline__ void shared_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Byte offset of element (row of this CTA, column) in a slot: 128-byte rows of a panel, whose 16-byte units lie
// at unit ^ (row % 8).  `column` is a multiple of 8.
__device__ __forceinline__ uint32_t offset_of(int row, int column) {
  return uint32_t(column >> 6) * kPanelBytes + uint32_t(row) * 128 + (uint32_t((column >> 3) & 7) ^ uint32_t(row & 7)) * 16;
}

__global__ void __launch_bounds__(kThreads, 1)
iteration_kernel(const __grid_constant__ Iteration it) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kSlots * kMatrixBytes);   // [kStages] leader's: both CTAs' stage landed
  uint64_t* empty = full + kStages;       // [kStages] both: the pair's MMAs on this stage completed
  uint64_t* acc_full = empty + kStages;   // [2] both: accumulator complete
  uint64_t* acc_empty = acc_full + 2;     // [2] leader's: a tile's epilogues drained it
  uint64_t* ring_free = acc_empty + 2;    // both: the MMAs that read the slots under the ring completed
  // both: this CTA's warps have written their own rows, up to column 128 and from there on (the leader's: and the
  // peer's theirs; it has no own pieces in the right half)
  uint64_t* written_left = ring_free + 1;
  uint64_t* written_right = written_left + 1;
  uint64_t* mirrored = written_right + 1; // leader's: the peer's mirror images have landed there
  uint64_t* half_image = mirrored + 1;    // [8] the second warp of an image has written its half
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(half_image + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* staging = smem + kSlots * kMatrixBytes + kBarrierBytes;
  uint8_t* nowhere_at = staging + kEpilogueWarps * kPieceBytes;   // written by every warp, read by none

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_rank();
  const uint32_t rank = cta & 1u, leader = cta & ~1u;   // rank in the pair; 0 = leader
  const int pair = int(cta >> 1), pairs = it.pairs;
  const int batch = int(blockIdx.x / cluster_size());
  const int m = it.m, n = it.n;
  const int k_steps = (m + kUmmaK - 1) / kUmmaK;          // of an m x m product: nothing past them is read
  const int k_blocks = (m + gemm2::kBK - 1) / gemm2::kBK;
  const int n_blocks = (n + gemm2::kBK - 1) / gemm2::kBK;
  const int tiles = (n + kSide - 1) / kSide;              // of Q X; this pair's are pair, pair + pairs, ...

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 2 * kTileWarps);
    }
    mbar_init(ring_free, 1);
    mbar_init(written_left, kEpilogueWarps + (rank == 0 ? 1 : 0));
    mbar_init(written_right, rank == 0 ? 1 : kEpilogueWarps);
    mbar_init(mirrored, 1);
    for (int i = 0; i < 8; ++i) mbar_init(&half_image[i], 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1 && lane < 4) prefetch_map(&it.x[lane >> 1][lane & 1]);
  if (warp == 0) gemm2::tmem_alloc2(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  cluster_sync();   // every CTA's barriers exist
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  griddep_wait();
  griddep_launch();

  // What each role keeps from part to part.
  bool ok = true;
  uint32_t stage = 0;                 // producer, issuer: stages of the ring so far
  uint32_t news = 0;                  // issuer, forwarder: products whose rows were waited for
  uint32_t uses[2] = {0, 0};          // issuer, epilogue: products and tiles through each accumulator
  uint32_t freed = 0;                 // producer: waits for the ring so far
  uint32_t emptied[2] = {0, 0};       // issuer: waits for each accumulator so far
  uint32_t landed = 0;                // issuer: products whose mirror images were waited for
  uint32_t images_made = 0;           // epilogue: mirror images put together

#pragma unroll 1
  for (int part = 0; part < 2; ++part) {
    if (warp == kProducerWarp) {
      // ---------------------------------------------------------- TMA producer (both CTAs)
      if (lane == 0) {
        if (part != 0) gemm2::proxy_fence();   // X was stored through the generic proxy, by this cluster
        auto wait_for_ring = [&] {
          ok = ok && mbar_wait(ring_free, freed & 1u, abort_flag, it.status, it.wait_ns);
          ++freed;
        };
        // one stage: `rows` = 128 rows of 64 columns at (column, row), else 64 rows of 128 columns
        auto load = [&](uint8_t* ring, bool rows, int column, int row) {
          const int s = stage % kStages;
          ok = ok && mbar_wait(&empty[s], ((stage / kStages) & 1u) ^ 1u, abort_flag, it.status, it.wait_ns);
          if (!ok) return;
          const uint32_t to = smem_u32(ring) + uint32_t(s) * kStageBytes;
          const uint32_t bar = peer_address(&full[s], leader);
          if (rank == 0) mbar_expect_tx(&full[s], 2 * kStageBytes);
          if (rows) {
            gemm2::tma_load_3d_pair(to, &it.x[part][0], bar, column, row, batch);
          } else {
            gemm2::tma_load_3d_pair(to, &it.x[part][1], bar, column, row, batch);
            gemm2::tma_load_3d_pair(to + kStageBytes / 2, &it.x[part][1], bar, column + 64, row, batch);
          }
          ++stage;
        };
        if (part != 0) wait_for_ring();
        const int own = int(rank) * kRows;
        for (int kb = 0; kb < n_blocks && ok; ++kb) {
          if (it.tall) load(smem + kMatrixBytes, false, own, kb * 64);
          else load(smem + kMatrixBytes, true, kb * 64, own);
        }
        wait_for_ring();
        for (int t = pair; t < tiles && ok; t += pairs)
          for (int kb = 0; kb < k_blocks && ok; ++kb) {
            if (it.tall) load(smem, true, kb * 64, t * kSide + own);
            else load(smem, false, t * kSide + own, kb * 64);
          }
      }
    } else if (warp == 0) {
      if (rank == 0) {
        // -------------------------------------------------------- MMA issuer (leader): a whole warp, as in gemm2_kernel
        const uint16_t both = uint16_t(3u << leader);
        const uint32_t slots = smem_u32(smem);
        // 64 rows of the peer's in 32 columns at a time
        const uint32_t image_bytes = m <= kRows ? 0u : uint32_t((m - kRows + 63) / 64) * 4 * 2 * kPieceBytes;
        auto arm = [&](int op) {
          if (image_bytes == 0) return;
          if (gemm2::elect_one()) mbar_expect_tx(mirrored, it.ops[part][op].out2 >= 0 ? 2 * image_bytes : image_bytes);
        };
        // All lanes wait; false for all of them when one gave up.
        auto wait = [&](uint64_t* bar, uint32_t phase) {
          ok = ok && __all_sync(0xffffffffu, mbar_wait(bar, phase & 1u, abort_flag, it.status, it.wait_ns)) != 0;
        };
        auto wait_cluster = [&](uint64_t* bar, uint32_t phase) {
          ok = ok && __all_sync(0xffffffffu, gemm2::mbar_wait_cluster(bar, phase & 1u, abort_flag, it.status, it.wait_ns)) != 0;
        };
        // what the last product left up to column 128 ...
        auto left_half = [&] {
          wait_cluster(written_left, news);
          tc_fence_after();
        };
        // ... and from there on: in the leader's rows that is mirror images
        auto right_half = [&] {
          if (image_bytes != 0) {
            wait_cluster(written_right, news);
            wait_cluster(mirrored, landed);
            tc_fence_after();
            ++landed;
          }
          ++news;
        };
        auto landed_stage = [&]() -> uint32_t {
          const int s = stage % kStages;
          wait(&full[s], stage / kStages);
          tc_fence_after();
          return uint32_t(s);
        };
        const uint32_t rows_idesc = gemm2::make_idesc2<__half>(false, false, kSide);
        // X X^T: this CTA's rows are its half of A and of B
        arm(0);
        auto gram = [&](auto tall) {
          constexpr bool kTall = decltype(tall)::value;
          const uint32_t idesc = gemm2::make_idesc2<__half>(kTall, kTall, kSide);
          for (int kb = 0; kb < n_blocks; ++kb, ++stage) {
            const uint32_t s = landed_stage();
            if (!ok) break;
            const uint64_t desc = make_smem_desc(slots + kMatrixBytes + s * kStageBytes, kTall ? kStageBytes / 2 : 16, 1024);
            if (gemm2::elect_one()) {
#pragma unroll
              for (int j = 0; j < gemm2::kBK / kUmmaK; ++j) {
                const uint64_t at = desc + uint64_t((kTall ? j * kUmmaK * 128 : j * kUmmaK * 2) >> 4);
                gemm2::umma2_f16(tmem_base, at, at, idesc, (kb > 0 || j > 0) ? 1u : 0u);
              }
              commit_pair(&empty[s], both);
            }
            __syncwarp();
          }
        };
        if (it.tall) gram(std::true_type());
        else gram(std::false_type());
        if (ok && gemm2::elect_one()) commit_pair(&acc_full[0], both);
        __syncwarp();
        // the chain
        for (int op = 1; op < it.count[part] && ok; ++op) {
          left_half();
          if (!ok) break;
          const uint32_t acc = tmem_base + uint32_t(op & 1) * 256;   // the other one is still being read
          const uint32_t a = slots + uint32_t(it.ops[part][op].a) * kMatrixBytes;
          const uint32_t b = slots + uint32_t(it.ops[part][op].b) * kMatrixBytes;
          auto steps = [&](int first, int last) {
            if (gemm2::elect_one()) {
#pragma unroll 8
              for (int k = first; k < last; ++k) {
                const uint32_t at = uint32_t(k >> 2) * kPanelBytes + uint32_t(k & 3) * (kUmmaK * 2);
                gemm2::umma2_f16(acc, make_smem_desc(a + at, 16, 1024), make_smem_desc(b + at, 16, 1024), rows_idesc, k > 0 ? 1u : 0u);
              }
            }
            __syncwarp();
          };
          steps(0, min(k_steps, kRows / kUmmaK));
          right_half();
          if (!ok) break;
          steps(kRows / kUmmaK, k_steps);
          arm(op);   // nothing is copied before this product's accumulator is complete
          if (gemm2::elect_one()) commit_pair(&acc_full[op & 1], both);
          __syncwarp();
        }
        // The ring may lie over slots 0 and 1 from here on: the last product's epilogue, which is still to come, reads
        // and writes slot 2 only (run_on_chip checks the schedule for that).
        if (ok && gemm2::elect_one()) commit_pair(ring_free, both);
        __syncwarp();
        // Q X (X Q of a tall block)
        left_half();
        right_half();
        int i = 0;
        auto tile = [&](auto tall, int acc) {
          constexpr bool kTall = decltype(tall)::value;
          const uint32_t idesc = gemm2::make_idesc2<__half>(false, !kTall, kSide);
          for (int kb = 0; kb < k_blocks; ++kb, ++stage) {
            const uint32_t s = landed_stage();
            if (!ok) break;
            const uint64_t q_desc = make_smem_desc(slots + 2 * kMatrixBytes + uint32_t(kb) * kPanelBytes, 16, 1024);
            const uint64_t x_desc = make_smem_desc(slots + s * kStageBytes, kTall ? 16 : kStageBytes / 2, 1024);
            const int steps = min(gemm2::kBK / kUmmaK, k_steps - kb * (gemm2::kBK / kUmmaK));
            if (gemm2::elect_one()) {
#pragma unroll
              for (int j = 0; j < gemm2::kBK / kUmmaK; ++j) {
                if (j >= steps) break;
                const uint64_t q = q_desc + uint64_t((j * kUmmaK * 2) >> 4);
                const uint64_t x = x_desc + uint64_t((kTall ? j * kUmmaK * 2 : j * kUmmaK * 128) >> 4);
                gemm2::umma2_f16(tmem_base + uint32_t(acc) * 256, kTall ? x : q, kTall ? q : x, idesc, (kb > 0 || j > 0) ? 1u : 0u);
              }
              commit_pair(&empty[s], both);
            }
            __syncwarp();
          }
          if (ok && gemm2::elect_one()) commit_pair(&acc_full[acc], both);
          __syncwarp();
        };
        for (int t = pair; t < tiles && ok; t += pairs, ++i) {
          const int acc = i & 1;
          if (i >= 2) {
            wait(&acc_empty[acc], emptied[acc]);
            ++emptied[acc];
            if (!ok) break;
            tc_fence_after();
          }
          if (it.tall) tile(std::true_type(), acc);
          else tile(std::false_type(), acc);
        }
        // A later part waits for no accumulator: the barrier below follows their epilogues.
        for (int acc = 0; acc < 2; ++acc) emptied[acc] += uint32_t(i > acc ? 1 : 0);
        if (ok && gemm2::elect_one()) commit_pair(ring_free, both);
        __syncwarp();
      } else if (lane == 0) {
        // The second CTA's news, as one arrive.  What it tells of lies in that CTA's own shared memory, fenced for the
        // tensor cores by the warps that wrote it (with release at cluster scope the arrive took 1200 cycles).
        const uint32_t leader_left = peer_address(written_left, leader), leader_right = peer_address(written_right, leader);
        for (int op = 0; op < it.count[part]; ++op, ++news) {
          if (!mbar_wait(written_left, news & 1u, abort_flag, it.status, it.wait_ns)) break;
          gemm2::remote_arrive(leader_left);
          if (m <= kRows) continue;
          if (!mbar_wait(written_right, news & 1u, abort_flag, it.status, it.wait_ns)) break;
          gemm2::remote_arrive(leader_right);
        }
      }
    } else {
      // ---------------------------------------------------------- epilogue (both CTAs)
      const int sub = warp & 3, group = (warp - 1) >> 2;
      const uint32_t slots = smem_u32(smem);
      const uint32_t leader_slots = peer_address(smem, leader);
      const uint32_t leader_mirrored = peer_address(mirrored, leader);
      const int local_row0 = sub * 32, row0 = int(rank) * kRows + local_row0;
      // A mirror image of 64 rows of the second CTA, 32 rows of a panel as they lie in the leader's slot, is put
      // together by two warps and copied as one.
      const int half = sub >> 1;
      uint8_t* const image_stage = staging + (group * 2 + half) * 2 * kPieceBytes;
      const uint32_t image_at = uint32_t(2 + half) * kPanelBytes + uint32_t(group) * 32 * 128;   // in the leader's slot
      // For the four 8 x 8 matrices of a stmatrix or ldmatrix this lane gives the address of row lane % 8 of matrix
      // lane / 8, at rows 16h + 8 * (lane / 8 % 2) and columns 16 * side + 8 * (lane / 16) of the piece: from these
      // offsets h is 2048 bytes and side flips bit 5; in the mirror image it is the other way round.
      const uint32_t own_base = offset_of(local_row0 + ((lane >> 3) & 1) * 8 + (lane & 7), (lane >> 4) * 8);
      const uint32_t image_base = offset_of((lane >> 4) * 8 + (lane & 7), (sub & 1) * 32 + ((lane >> 3) & 1) * 8);
      const uint32_t nowhere = smem_u32(nowhere_at) + uint32_t(lane) * 16;
      for (int op = 0; ok && op < it.count[part]; ++op) {
        const Op& o = it.ops[part][op];
        const uint32_t acc = uint32_t(op & 1);
        ok = mbar_wait(&acc_full[acc], (acc == 0 ? uses[0] : uses[1]) & 1u, abort_flag, it.status, it.wait_ns);
        if (acc == 0) ++uses[0];
        else ++uses[1];
        if (!ok) break;
        tc_fence_after();
        auto piece = [&](int c) {
          const int col0 = 32 * c;
          if (col0 > row0 || row0 >= m) return;   // uniform over the warp; left of the diagonal is also inside the matrix
          uint32_t v[32];
          const uint32_t taddr = tmem_base + acc * 256 + (uint32_t(sub * 32) << 16) + uint32_t(col0);
          tmem_load_16x32(taddr, v);
          tmem_load_16x32(taddr + (16u << 16), v + 16);
          uint32_t r[16];   // [half of the rows][pair of column blocks][row block in the half + 2 * column block in the pair]
          const uint32_t own = (own_base ^ uint32_t((c & 1) << 6)) + uint32_t(c >> 1) * kPanelBytes;
          if (o.cin >= 0) {
            const uint32_t cin = slots + uint32_t(o.cin) * kMatrixBytes;
            uint32_t ci[16];
#pragma unroll
            for (int f = 0; f < 16; f += 4)
              ldmatrix4(cin + (own ^ uint32_t(((f >> 2) & 1) << 5)) + uint32_t(f >> 3) * 2048, ci[f], ci[f + 1], ci[f + 2],
                        ci[f + 3]);
            tmem_wait(v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float2 cf = unpack2<__half>(ci[j]);
              r[j] = pack2<__half>(fmaf(o.beta, cf.x, o.alpha * __uint_as_float(v[2 * j])),
                                   fmaf(o.beta, cf.y, o.alpha * __uint_as_float(v[2 * j + 1])));
            }
          } else {
            tmem_wait(v);
#pragma unroll
            for (int j = 0; j < 16; ++j)
              r[j] = pack2<__half>(o.alpha * __uint_as_float(v[2 * j]), o.alpha * __uint_as_float(v[2 * j + 1]));
          }
          const bool diagonal = row0 == col0;
          if (diagonal) {
            // The blocks on the diagonal: what lies above it comes from below it.
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 4; i += 3) {
                uint32_t& w = r[8 * h + 4 * h + i];
                const uint32_t t = transpose_8x8(w);
                const int row = lane >> 2, column = 2 * (lane & 3);
                uint32_t mask = 0;
                if (column > row) mask |= 0x0000FFFFu;
                if (column + 1 > row) mask |= 0xFFFF0000u;
                w = (w & ~mask) | (t & mask);
              }
          }
          const bool remote = rank != 0 && col0 < kRows;   // the mirror image is the leader's
          const uint32_t image = remote ? smem_u32(image_stage) + image_base
                                        : image_base + uint32_t(row0 >> 6) * kPanelBytes + uint32_t(c & 3) * 32 * 128;
          auto store = [&](uint32_t slot, bool with_image) {
            const uint32_t image_slot = remote ? 0u : slot;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int side = 0; side < 2; ++side) {
                const uint32_t* f = r + 8 * h + 4 * side;
                uint32_t at = slot + (own ^ uint32_t(side << 5)) + uint32_t(h) * 2048;
                uint32_t to = image_slot + (image ^ uint32_t(h << 5)) + uint32_t(side) * 2048;
                if (diagonal) {
                  // Blocks above the diagonal are the mirror images of those below it.
                  const int block = 2 * h + ((lane >> 3) & 1), column_block = 2 * side + (lane >> 4);
                  if (block < column_block) at = nowhere;
                  if (block <= column_block) to = nowhere;
                }
                stmatrix4(at, f[0], f[1], f[2], f[3]);
                if (with_image) stmatrix4_trans(to, f[0], f[1], f[2], f[3]);
              }
          };
          store(slots + uint32_t(o.out) * kMatrixBytes, true);
          if (remote) {
            shared_fence();
            __syncwarp();
            uint64_t* const other_half = &half_image[group * 2 + half];
            if ((sub & 1) != 0) {
              if (lane == 0) mbar_arrive(other_half);
            } else if (lane == 0 && (row0 + 32 >= m || mbar_wait(other_half, images_made & 1u, abort_flag, it.status, it.wait_ns))) {
              copy_to_peer(leader_slots + uint32_t(o.out) * kMatrixBytes + image_at, image_stage, 2 * kPieceBytes, leader_mirrored);
              if (o.out2 >= 0)
                copy_to_peer(leader_slots + uint32_t(o.out2) * kMatrixBytes + image_at, image_stage, 2 * kPieceBytes, leader_mirrored);
            }
          }
          if (o.out2 >= 0) {
            if (diagonal) {
              const int row = lane >> 2, column = 2 * (lane & 3);
#pragma unroll
              for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 4; i += 3) {
                  uint32_t& w = r[8 * h + 4 * h + i];
                  const float2 f = unpack2<__half>(w);
                  if (column == row) w = pack2<__half>(f.x + o.diag, f.y);
                  if (column + 1 == row) w = pack2<__half>(f.x, f.y + o.diag);
                }
            }
            store(slots + uint32_t(o.out2) * kMatrixBytes, !remote);
          }
        };
        auto report = [&](uint64_t* bar) {
          tc_fence_before();
          shared_fence();   // written through the generic proxy, read by the tensor cores
          __syncwarp();
          if (lane == 0) mbar_arrive(bar);
        };
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
          if (side != 0 && (rank == 0 || m <= kRows)) break;
          piece(group + 4 * side);
          report(side == 0 ? written_left : written_right);
        }
        ++images_made;
      }
      // tiles of Q X
      {
        Params p = it.result[part];
        p.cin = nullptr;
        const int own = warp <= kTileWarps ? 0 : 1;   // the accumulator whose tiles this warp has
        const uint32_t leader_empty = peer_address(&acc_empty[own], leader);
        auto release = [&] {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) gemm2::remote_arrive(leader_empty);
        };
        int i = 0;
#pragma unroll 1
        for (int t = pair; t < tiles; t += pairs, ++i) {
          if ((i & 1) != own || !ok) continue;
          const uint32_t phase = ((own == 0 ? uses[0] : uses[1]) + uint32_t(i >> 1)) & 1u;
          const int m_base = (it.tall ? t * kSide : 0) + int(rank) * kRows, n_base = it.tall ? 0 : t * kSide;
          ok = epilogue_tile<__half, false>(p, batch, m_base, n_base, tmem_base + uint32_t(own) * 256, &acc_full[own], phase,
                                            abort_flag, staging + (warp - 1) * kPieceBytes, sub, lane, (group & 1) * 4, 4,
                                            it.result_bf16[part], release);
        }
        uses[0] += uint32_t((i + 1) / 2);
        uses[1] += uint32_t(i / 2);
        gemm2::proxy_fence();   // read by the next part's copies
      }
    }
    __syncwarp();
    if (part == 0) cluster_sync();   // X is stored, and every accumulator drained
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0 && threadIdx.x == 0) {
    const uint64_t start = global_ns();
    while (global_ns() - start < 200000ull) {
    }
  }
  cluster_sync();   // nobody reaches into a peer's shared memory any more
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    gemm2::tmem_dealloc2(tmem_base, kTmemCols);
  }
}

}  // namespace onchip
}  // namespace dionw
