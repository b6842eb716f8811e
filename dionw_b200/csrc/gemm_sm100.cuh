// Batched tcgen05 GEMM for sm_100a: TMA-fed shared-memory ring, accumulators in
// TMEM, a persistent tile loop with three warp roles (TMA producer, MMA issuer,
// eight epilogue warps).  Two tile schedules: every tile of a general product,
// or only the tiles on and below the diagonal of a symmetric product, whose
// strictly-lower 128x128 sub-blocks are also stored transposed.
//
// Tile 128 x 256 x 64 (one tcgen05.mma is 128 x 256 x 16), cta_group::1,
// 4-stage ring (48 KB per stage), two 256-column accumulators so the epilogue
// of tile t overlaps the main loop of tile t+1.  No cluster multicast anywhere.
//
// Every spin-wait is bounded; when one runs out the kernel stores a code in the
// device status word and leaves through the common teardown (TMEM is freed).
#pragma once

#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "decay_job.cuh"

namespace dionw {
namespace gemm {

constexpr int kBM = 128;
constexpr int kBN = 256;
constexpr int kBK = 64;
constexpr int kStages = 4;
constexpr int kUmmaK = 16;
constexpr int kThreads = 320;  // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-9: epilogue
constexpr int kEpilogueThreads = 256;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kABytes = kBM * kBK * 2;        // 16 KB
constexpr uint32_t kBBytes = kBN * kBK * 2;        // 32 KB
constexpr uint32_t kStageBytes = kABytes + kBBytes;
constexpr uint32_t kPanelBytes = 64 * kBK * 2;     // one 64-column panel of an MN-major stage
constexpr uint32_t kPieceBytes = 32 * 32 * 2;      // one 32 x 32 piece of the output, 64 bytes a row
constexpr uint32_t kMirrorBytes = 8 * 2 * kPieceBytes;  // per epilogue warp: a piece as it lies and its transpose
constexpr size_t kSmemBytes =
    size_t(kStages) * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/ + kMirrorBytes;

constexpr int kWaitCode = 0x7001;
constexpr uint64_t kWaitLimitNs = 2000000000ull;   // default limit of a bounded wait: two seconds

struct Params {
  // epilogue operands (element pointers; strides in elements)
  const void* cin;       // nullable
  void* out;
  void* out2;            // nullable: out + diag on the diagonal (symmetric schedule only)
  int64_t ldc, ldo;
  int64_t cin_batch, out_batch;
  float alpha, beta, diag;
  // problem
  int m, n, kdim;        // output m x n, reduction length kdim
  int batches;
  int tiles_m, tiles_n, tiles_per_batch;
  int mirror_diagonal;   // symmetric schedule with B != A: also mirror inside the diagonal sub-blocks
  int lower_only;        // symmetric schedule: no mirror image outside the 256 x 256 blocks on the diagonal
  float* rowsq;          // nullable, general products only: [batches, m, rowsq_parts] partial row sums of out^2
  int rowsq_parts;       // = 2 * tiles_n: one partial per 128 columns, written once each, summed by the reader
  int* status;           // device status word (may be null: the code is then not recorded)
  uint64_t wait_ns;      // limit of every bounded wait, in nanoseconds of %globaltimer
};

// ----------------------------------------------------------------------------
// PTX wrappers
// ----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Programmatic dependent launch: the host launches every product with the stream-serialization
// attribute, so the CTAs of the next product may become resident, and run their set-up, as soon as
// CTAs of this one exit.  Nothing of global memory is read or written before griddep_wait()
// returns, which it does once the previous kernel of the stream has completed and its writes are
// visible; griddep_launch() then allows the kernel after this one to start the same way.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait: gives up after `limit_ns` (two seconds unless the launch says otherwise), flags
// the failure in the device status word and tells the rest of the CTA to stop through `abort_flag`.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, uint64_t limit_ns = kWaitLimitNs) {
  uint32_t spins = 0;
  uint64_t start = 0;   // the timer is first read after 1024 failed tries: a wait that ends soon never pays for it
  while (!mbar_try(bar, parity)) {
    if ((++spins & 1023u) == 0) {
      if (*abort_flag != 0) return false;
      const uint64_t now = global_ns();
      if (start == 0) start = now;
      else if (now - start > limit_ns) {
        *abort_flag = 1;
        if (status != nullptr) atomicExch(status, kWaitCode);
        return false;
      }
    }
  }
  return true;
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0,
                                            int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// Brings a kernel argument's tensor map into the descriptor cache; touches no data of the operands.
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives on `bar` once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 16 accumulator rows x 32 columns in the layout of an mma.m16n8 result: register 4g + q of lane l is
// row l / 4 + 8 * (q / 2), column 8g + 2 * (l % 4) + q % 2.  Valid after tmem_wait.
__device__ __forceinline__ void tmem_load_16x32(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// The registers pass through the wait, so that no use of them can be moved in front of it.
__device__ __forceinline__ void tmem_wait(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
      : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
        "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
        "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
        "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
      :
      : "memory");
}

// Four 8 x 8 matrices of 2-byte elements between registers (mma layout) and shared memory; lane l gives
// the address of row l % 8 of matrix l / 8.  The transposing store writes column l % 8 there instead.
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stmatrix4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void stmatrix4_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Shared-memory matrix descriptor, 128-byte swizzle, version 1 (Blackwell).
//   K-major operand  (rows of 64 elements = 128 B): SBO = 1024 B between 8-row groups, LBO unused (1).
//   MN-major operand (64-element panels, one 128 B row per k): LBO = bytes between
//   panels, SBO = 1024 B between 8-k groups.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((addr >> 4) & 0x3FFFu);
  d |= uint64_t((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= uint64_t(1) << 46;  // descriptor version
  d |= uint64_t(2) << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16: fp32 accumulate, M = 128, N = 256.
template <typename T, bool kAMajorMN, bool kBMajorMN>
__device__ __forceinline__ uint32_t make_idesc() {
  constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
  uint32_t d = 0;
  d |= 1u << 4;                       // D format f32
  d |= fmt << 7;                      // A format
  d |= fmt << 10;                     // B format
  d |= (kAMajorMN ? 1u : 0u) << 15;   // A major
  d |= (kBMajorMN ? 1u : 0u) << 16;   // B major
  d |= uint32_t(kBN >> 3) << 17;      // N
  d |= uint32_t(kBM >> 4) << 24;      // M
  return d;
}

// ----------------------------------------------------------------------------
// tile schedules
// ----------------------------------------------------------------------------
struct Tile {
  int batch, tm, tn;
};

// General product: groups of 8 tile rows sweep the tile columns, so that one
// wave of CTAs reuses a band of A and the whole of B from L2.
__device__ __forceinline__ Tile general_tile(int t, const Params& p) {
  Tile tile;
  tile.batch = t / p.tiles_per_batch;
  int r = t - tile.batch * p.tiles_per_batch;
  const int group_rows = 8;
  const int per_group = group_rows * p.tiles_n;
  const int g = r / per_group;
  const int first = g * group_rows;
  const int rows_here = min(group_rows, p.tiles_m - first);
  r -= g * per_group;
  tile.tm = first + r % rows_here;
  tile.tn = r / rows_here;
  return tile;
}

// Symmetric product: tile row i (128 rows) needs tile columns 0..i/2 (256
// columns each).  Rows 2q and 2q+1 hold q+1 tiles each, q(q+1) tiles precede them.
__device__ __forceinline__ Tile sym_tile(int t, const Params& p) {
  Tile tile;
  tile.batch = t / p.tiles_per_batch;
  const int r = t - tile.batch * p.tiles_per_batch;
  int q = int((sqrtf(4.0f * float(r) + 1.0f) - 1.0f) * 0.5f);
  while (q * (q + 1) > r) --q;
  while ((q + 1) * (q + 2) <= r) ++q;
  const int rem = r - q * (q + 1);
  if (rem <= q) {
    tile.tm = 2 * q;
    tile.tn = rem;
  } else {
    tile.tm = 2 * q + 1;
    tile.tn = rem - (q + 1);
  }
  return tile;
}

// Two values as one word of the 2-byte type (the first in the low half), and back.
template <typename T>
__device__ __forceinline__ uint32_t pack2(float a, float b);
template <>
__device__ __forceinline__ uint32_t pack2<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w);
template <>
__device__ __forceinline__ float2 unpack2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <>
__device__ __forceinline__ float2 unpack2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
}

// ----------------------------------------------------------------------------
// epilogue of one accumulator: 128 rows (m_base ..) x tile_n columns (n_base ..) of batch
// ``batch``, read from TMEM at ``tmem_acc`` by the warp that owns sub-partition ``sub``;
// this warp handles `chunks` of the tile's 32-column chunks from first_chunk on.  `release` is called once,
// when the warp has read all it needs of the accumulator.  Returns false when the bounded wait for the
// accumulator ran out.
//
// A warp works on 32 x 32 pieces.  The accumulator is read in the mma result layout, because
// stmatrix turns that into rows of the piece and, with .trans, into rows of its mirror image at four
// instructions each; global memory is read and written in "piece order" (lane l holds the 8
// consecutive elements at row 8*it + l/4, column 8*(l%4), it = 0..3), so one instruction touches
// 8 rows x 64 contiguous bytes.  The two staging tiles keep 16-byte units at unit ^ (row/2 & 3):
// stmatrix, ldmatrix and the 16-byte accesses all go without bank conflicts.  Every class of piece
// takes this one path: matrix edges only guard the final 16-byte accesses.
//
// What bounds it: in products of one or two waves (small matrices) nothing hides this chain, in
// longer ones it runs under the next tile's main loop.  The first version read the accumulator row
// by row, transposed with 2-byte gathers and sent diagonal pieces of B != A and all edge pieces
// through per-element loops: a 256^3 mirrored product with Cin took 15.7 us in a chain of products,
// this takes 8.1; 6 blocks of 517^3 17.8 us against 12.6.
// ----------------------------------------------------------------------------
template <typename InT, bool kSym, typename Release>
__device__ __forceinline__ bool epilogue_tile(const Params& p, int batch, int m_base, int n_base, uint32_t tmem_acc,
                                              uint64_t* acc_full_bar, uint32_t acc_phase, volatile int* abort_flag,
                                              uint8_t* stage, int sub, int lane, int first_chunk, int chunks,
                                              bool to_bf16, Release&& release) {
  // A general product of fp16 operands has a bf16 result where `to_bf16` says so.  (As a template argument the
  // second general form cost the kernel that holds all of them its registers.)
  auto pack_out = [&](float a, float b) -> uint32_t {
    if constexpr (kSym || std::is_same<InT, __nv_bfloat16>::value) return pack2<InT>(a, b);
    return to_bf16 ? pack2<__nv_bfloat16>(a, b) : pack2<InT>(a, b);
  };
  auto unpack_out = [&](uint32_t w) -> float2 {
    if constexpr (kSym || std::is_same<InT, __nv_bfloat16>::value) return unpack2<InT>(w);
    return to_bf16 ? unpack2<__nv_bfloat16>(w) : unpack2<InT>(w);
  };
  const uint16_t* cin = p.cin ? reinterpret_cast<const uint16_t*>(p.cin) + size_t(batch) * p.cin_batch : nullptr;
  uint16_t* out = reinterpret_cast<uint16_t*>(p.out) + size_t(batch) * p.out_batch;
  uint16_t* out2 = kSym && p.out2 ? reinterpret_cast<uint16_t*>(p.out2) + size_t(batch) * p.out_batch : nullptr;
  // What every piece needs, held in registers: the parameters themselves lie where a load takes a while.
  const int m = p.m, n = p.n;
  const int64_t ldo = p.ldo, ldc = p.ldc;
  const float alpha = p.alpha, beta = p.beta, diag = p.diag;
  const int row0 = m_base + sub * 32;
  // Class of the 32 x 32 piece at (row0, col0) under the symmetric schedule:
  // 0 stored as it is (also below the diagonal, outside of its 256 x 256 blocks, where readers want no mirror
  // image); 1 strictly below the diagonal: stored and stored transposed;
  // 2 strictly above: skipped (its mirror image writes it); 3 on the diagonal of a product with
  // B != A, which is symmetric only up to rounding: the lower triangle is stored and mirrored, so
  // that the stored matrix is exactly symmetric.
  auto class_of = [&](int col0) -> int {
    if constexpr (!kSym) return 0;
    if (col0 + 32 <= row0) return p.lower_only != 0 && (col0 ^ row0) >= 256 ? 0 : 1;
    if (col0 >= row0 + 32) return 2;
    return p.mirror_diagonal != 0 ? 3 : 0;
  };
  // Chunks past the matrix, and under the symmetric schedule those above the diagonal, come last.
  int end_chunk = first_chunk;
  while (end_chunk < first_chunk + chunks && n_base + end_chunk * 32 < n && row0 < m &&
         class_of(n_base + end_chunk * 32) != 2)
    ++end_chunk;
  const bool out_aligned = (ldo & 7) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0 &&
                           (reinterpret_cast<uintptr_t>(out2) & 15u) == 0;
  const bool cin_aligned = (ldc & 7) == 0 && (reinterpret_cast<uintptr_t>(cin) & 15u) == 0;
  const int piece_row = lane >> 2, piece_unit = lane & 3, piece_col = piece_unit * 8;
  // 16 bytes of Cin at (r, c): elements outside the matrix read as zero.  Read from L2: in a plan of
  // several products the bytes were written by another SM during this launch.
  auto get = [&](int r, int c) -> uint4 {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r >= m || c >= n) return v;
    const uint16_t* at = cin + size_t(r) * ldc + c;
    if (cin_aligned && c + 8 <= n) return __ldcg(reinterpret_cast<const uint4*>(at));
    uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c + j < n) w[j >> 1] |= uint32_t(__ldcg(at + j)) << (16 * (j & 1));
    return make_uint4(w[0], w[1], w[2], w[3]);
  };
  auto put = [&](uint16_t* base, int r, int c, const uint4& v) {
    if (r >= m || c >= n) return;
    uint16_t* at = base + size_t(r) * ldo + c;
    if (out_aligned && c + 8 <= n) {
      *reinterpret_cast<uint4*>(at) = v;
      return;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (c + j < n) at[j] = uint16_t(w[j >> 1] >> (16 * (j & 1)));
  };
  auto unit_at = [](int row, int unit) -> uint32_t { return uint32_t(row * 64 + ((unit ^ ((row >> 1) & 3)) << 4)); };
  // Places in the staging tiles, from one base each: 16 rows on are 1024 bytes, which leaves the swizzle
  // alone, and two units on are the same place with bit 5 flipped.
  uint8_t* const my_piece = stage + unit_at(piece_row, piece_unit);   // + 512 * it
  uint8_t* const my_mirror = my_piece + kPieceBytes;
  // This lane's row addresses for the four matrices of one ldmatrix / stmatrix: rows 16h + 8 * (i % 2),
  // columns 16 * pair + 8 * (i / 2) of the piece, i = lane / 8; and their places in the mirror image.
  const uint32_t matrix_base = smem_u32(stage) + unit_at(((lane >> 3) & 1) * 8 + (lane & 7), lane >> 4);
  const uint32_t mirror_base = smem_u32(stage) + kPieceBytes + unit_at((lane >> 4) * 8 + (lane & 7), (lane >> 3) & 1);
  auto matrix_at = [&](int h, int pair) { return (matrix_base ^ uint32_t(pair << 5)) + uint32_t(h << 10); };
  auto mirror_at = [&](int h, int pair) { return (mirror_base ^ uint32_t(h << 5)) + uint32_t(pair << 10); };

  // The Cin piece of the next chunk is requested before the current chunk is worked on.
  // (Whole pieces, which are nearly all, from one pointer and a row stride: with bounds and address worked out per
  // 16 bytes the request took 550 of a chunk's 2000 cycles.)
  uint4 ahead[4];
  const bool rows_whole = row0 + 32 <= m;   // uniform over the warp, like all that decides on a whole piece
  const uint16_t* const cin_at = cin + int64_t(row0 + piece_row) * ldc + (n_base + piece_col);
  auto prefetch = [&](int chunk) {
    const int col0 = n_base + chunk * 32;
    if (cin == nullptr || chunk >= end_chunk) return;
    if (rows_whole && cin_aligned && col0 + 32 <= n) {
      const uint16_t* at = cin_at + chunk * 32;
#pragma unroll
      for (int it = 0; it < 4; ++it) ahead[it] = __ldcg(reinterpret_cast<const uint4*>(at + it * 8 * ldc));
      return;
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) ahead[it] = get(row0 + 8 * it + piece_row, col0 + piece_col);
  };
  prefetch(first_chunk);   // does not depend on the accumulator: overlaps the wait below
  if (!mbar_wait(acc_full_bar, acc_phase, abort_flag, p.status, p.wait_ns)) return false;
  tc_fence_after();
  if (end_chunk == first_chunk) release();
  // Sums of the squares of the rounded results over the warp's columns, for NorMuon: the values are
  // in registers here, so the row statistics need no second pass over the output.  Lane l sums its
  // columns of rows l/4 + 8i; the four lanes of a row are added at the end: the order is fixed.
  const bool want_sq = !kSym && p.rowsq != nullptr;   // 256-column tiles only
  float sq[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 1
  for (int chunk = first_chunk; chunk < end_chunk; ++chunk) {
    const int col0 = n_base + chunk * 32;
    const int cls = class_of(col0);   // uniform over the warp
    // (Requesting the next chunk's accumulator before this one is stored was measured: 1-2 % slower.)
    uint32_t v[32];
    const uint32_t taddr = tmem_acc + (uint32_t(sub * 32) << 16) + uint32_t(chunk * 32);
    tmem_load_16x32(taddr, v);
    tmem_load_16x32(taddr + (16u << 16), v + 16);
    uint32_t r[16];               // [half of the rows][column group of 8][row / 8 in the half]
    if (cin != nullptr) {
#pragma unroll
      for (int it = 0; it < 4; ++it)
        *reinterpret_cast<uint4*>(my_piece + 512 * it) = ahead[it];
      prefetch(chunk + 1);
      __syncwarp();
      tmem_wait(v);
      if (chunk + 1 == end_chunk) release();
#pragma unroll
      for (int f = 0; f < 16; f += 4) {   // (h, pair) = (f / 8, f / 4 % 2)
        uint32_t c[4];
        ldmatrix4(matrix_at(f >> 3, (f >> 2) & 1), c[0], c[1], c[2], c[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 cf = unpack2<InT>(c[j]);
          r[f + j] = pack_out(fmaf(beta, cf.x, alpha * __uint_as_float(v[2 * (f + j)])),
                                 fmaf(beta, cf.y, alpha * __uint_as_float(v[2 * (f + j) + 1])));
        }
      }
      __syncwarp();               // every lane has its part of Cin: the staging tile is free
    } else {
      tmem_wait(v);
      if (chunk + 1 == end_chunk) release();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        r[j] = pack_out(alpha * __uint_as_float(v[2 * j]), alpha * __uint_as_float(v[2 * j + 1]));
    }
    if (want_sq) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int column = col0 + (j >> 1 & 3) * 8 + (lane & 3) * 2;
        const float2 f = unpack_out(r[j]);
        float& sum = sq[2 * (j >> 3) + (j & 1)];
        if (column < n) sum = fmaf(f.x, f.x, sum);
        if (column + 1 < n) sum = fmaf(f.y, f.y, sum);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int pair = 0; pair < 2; ++pair) {
        const uint32_t* f = r + 8 * h + 4 * pair;
        stmatrix4(matrix_at(h, pair), f[0], f[1], f[2], f[3]);
        if (kSym && cls != 0) stmatrix4_trans(mirror_at(h, pair), f[0], f[1], f[2], f[3]);
      }
    __syncwarp();
    // Whole pieces, which are nearly all, go out with plain 16-byte stores, the four loads first.
    const bool whole = out_aligned && rows_whole && col0 + 32 <= n;
    uint4 piece[4];
#pragma unroll
    for (int it = 0; it < 4; ++it)
      piece[it] = *reinterpret_cast<const uint4*>(my_piece + 512 * it);
    if constexpr (kSym) {
      if (cls != 0) {
        uint4 other[4];
#pragma unroll
        for (int it = 0; it < 4; ++it)
          other[it] = *reinterpret_cast<const uint4*>(my_mirror + 512 * it);
        if (cls == 1) {
          if (whole) {
            const size_t at = size_t(col0 + piece_row) * ldo + row0 + piece_col;
#pragma unroll
            for (int it = 0; it < 4; ++it) *reinterpret_cast<uint4*>(out + at + size_t(8 * it) * ldo) = other[it];
            if (out2 != nullptr) {
#pragma unroll
              for (int it = 0; it < 4; ++it) *reinterpret_cast<uint4*>(out2 + at + size_t(8 * it) * ldo) = other[it];
            }
          } else {
#pragma unroll
            for (int it = 0; it < 4; ++it) {
              put(out, col0 + 8 * it + piece_row, row0 + piece_col, other[it]);
              if (out2 != nullptr) put(out2, col0 + 8 * it + piece_row, row0 + piece_col, other[it]);
            }
          }
        } else {
          // elements above the diagonal come from the mirror image; here row0 == col0
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            uint32_t* w = reinterpret_cast<uint32_t*>(&piece[it]);
            const uint32_t o[4] = {other[it].x, other[it].y, other[it].z, other[it].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t mask = 0;
              if (piece_col + 2 * j > 8 * it + piece_row) mask |= 0x0000FFFFu;
              if (piece_col + 2 * j + 1 > 8 * it + piece_row) mask |= 0xFFFF0000u;
              w[j] = (w[j] & ~mask) | (o[j] & mask);
            }
          }
        }
      }
    }
    const size_t at = size_t(row0 + piece_row) * ldo + col0 + piece_col;
    if (whole) {
#pragma unroll
      for (int it = 0; it < 4; ++it) *reinterpret_cast<uint4*>(out + at + size_t(8 * it) * ldo) = piece[it];
    } else {
#pragma unroll
      for (int it = 0; it < 4; ++it) put(out, row0 + 8 * it + piece_row, col0 + piece_col, piece[it]);
    }
    if constexpr (kSym) {
      if (out2 != nullptr) {
        if (row0 == col0) {       // the piece on the diagonal: pieces and diagonal are both 32-aligned
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            uint32_t* w = reinterpret_cast<uint32_t*>(&piece[it]);
            const int d = 8 * it + piece_row - piece_col;   // its position inside the 8 elements
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 f = unpack_out(w[j]);
              if (d == 2 * j) w[j] = pack_out(f.x + diag, f.y);
              if (d == 2 * j + 1) w[j] = pack_out(f.x, f.y + diag);
            }
          }
        }
        if (whole) {
#pragma unroll
          for (int it = 0; it < 4; ++it) *reinterpret_cast<uint4*>(out2 + at + size_t(8 * it) * ldo) = piece[it];
        } else {
#pragma unroll
          for (int it = 0; it < 4; ++it) put(out2, row0 + 8 * it + piece_row, col0 + piece_col, piece[it]);
        }
      }
    }
    __syncwarp();                 // the staging tiles are read: the next chunk may write them
  }
  if (want_sq) {
    const int part = 2 * (n_base / kBN) + first_chunk / (kBN / 64);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 1);
      sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 2);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = row0 + 8 * i + piece_row;
      if (piece_unit == 0 && row < m) p.rowsq[(size_t(batch) * m + row) * p.rowsq_parts + part] = sq[i];
    }
  }
  return true;
}

// ----------------------------------------------------------------------------
// the kernel
// ----------------------------------------------------------------------------
// kSym with kBMajorMN is X^T X: both operands are the row-major [kdim, m] matrix, read MN-major.
template <typename InT, typename OutT, bool kBMajorMN, bool kSym>
__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params p) {
  constexpr bool kAMajorMN = kSym && kBMajorMN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + size_t(kStages) * kStageBytes);
  uint64_t* empty_bar = full_bar + kStages;
  uint64_t* acc_full = empty_bar + kStages;   // [2]
  uint64_t* acc_empty = acc_full + 2;         // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* mirror_stage = smem + size_t(kStages) * kStageBytes + 256;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int total_tiles = p.tiles_per_batch * p.batches;
  const int k_blocks = (p.kdim + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], kEpilogueThreads);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    prefetch_map(&map_a);
    prefetch_map(&map_b);
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  griddep_wait();
  griddep_launch();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const Tile tile = kSym ? sym_tile(t, p) : general_tile(t, p);
        const int m0 = tile.tm * kBM, n0 = tile.tn * kBN;
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t phase = (it / kStages) & 1u;
          if (!mbar_wait(&empty_bar[s], phase ^ 1u, abort_flag, p.status, p.wait_ns)) { ok = false; break; }
          uint8_t* a_dst = smem + size_t(s) * kStageBytes;
          uint8_t* b_dst = a_dst + kABytes;
          mbar_expect_tx(&full_bar[s], kStageBytes);
          if constexpr (kAMajorMN) {
#pragma unroll
            for (int panel = 0; panel < kBM / 64; ++panel)
              tma_load_3d(a_dst + panel * kPanelBytes, &map_a, &full_bar[s], m0 + panel * 64, kb * kBK, tile.batch);
          } else {
            tma_load_3d(a_dst, &map_a, &full_bar[s], kb * kBK, m0, tile.batch);
          }
          if constexpr (kBMajorMN) {
#pragma unroll
            for (int panel = 0; panel < kBN / 64; ++panel)
              tma_load_3d(b_dst + panel * kPanelBytes, &map_b, &full_bar[s], n0 + panel * 64, kb * kBK, tile.batch);
          } else {
            tma_load_3d(b_dst, &map_b, &full_bar[s], kb * kBK, n0, tile.batch);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = make_idesc<InT, kAMajorMN, kBMajorMN>();
      uint32_t it = 0, local = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
        const uint32_t acc = local & 1u;
        const uint32_t acc_phase = (local >> 1) & 1u;
        if (!mbar_wait(&acc_empty[acc], acc_phase ^ 1u, abort_flag, p.status, p.wait_ns)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * uint32_t(kBN);
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
          const int s = it % kStages;
          const uint32_t phase = (it / kStages) & 1u;
          if (!mbar_wait(&full_bar[s], phase, abort_flag, p.status, p.wait_ns)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + size_t(s) * kStageBytes);
          const uint32_t b_addr = a_addr + kABytes;
          const uint64_t a_desc = kAMajorMN ? make_smem_desc(a_addr, kPanelBytes, 1024)
                                            : make_smem_desc(a_addr, 16, 1024);
          const uint64_t b_desc = kBMajorMN ? make_smem_desc(b_addr, kPanelBytes, 1024)
                                            : make_smem_desc(b_addr, 16, 1024);
#pragma unroll
          for (int j = 0; j < kBK / kUmmaK; ++j) {
            // K-major: 16 elements = 32 B further along each 128 B row.
            // MN-major: 16 k-rows of 128 B further.
            const uint64_t k_step = uint64_t((j * kUmmaK * 2) >> 4), mn_step = uint64_t((j * kUmmaK * 128) >> 4);
            const uint64_t a_step = kAMajorMN ? mn_step : k_step;
            const uint64_t b_step = kBMajorMN ? mn_step : k_step;
            umma_f16(tmem_d, a_desc + a_step, b_desc + b_step, idesc, (kb > 0 || j > 0) ? 1u : 0u);
          }
          umma_commit(&empty_bar[s]);
        }
        if (ok) umma_commit(&acc_full[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Eight warps: two per TMEM sub-partition (a warp may only read the 32 lanes
    // 32 * (warp % 4) ...), each taking four of the tile's eight 32-column chunks.
    const int ew = warp - 2;                  // 0..7
    const int sub = warp & 3;                 // TMEM lanes 32*sub .. 32*sub+31
    const int first_chunk = (ew >> 2) * (kBN / 64);
    uint8_t* stage = mirror_stage + ew * 2 * kPieceBytes;
    uint32_t local = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local) {
      const Tile tile = kSym ? sym_tile(t, p) : general_tile(t, p);
      const uint32_t acc = local & 1u;
      const uint32_t acc_phase = (local >> 1) & 1u;
      auto release = [&] {
        tc_fence_before();
        mbar_arrive(&acc_empty[acc]);
      };
      if (!epilogue_tile<InT, kSym>(p, tile.batch, tile.tm * kBM, tile.tn * kBN, tmem_base + acc * uint32_t(kBN),
                                    &acc_full[acc], acc_phase, abort_flag, stage, sub, lane, first_chunk, kBN / 64,
                                    std::is_same<OutT, __nv_bfloat16>::value, release)) {
        ok = false;
        break;
      }
    }
  }

  // ------------------------------------------------------------ teardown
  __syncthreads();
  if (*abort_flag != 0 && threadIdx.x == 0) {
    // Give copies that may still be in flight time to land before the CTA's
    // shared memory is released.
    const uint64_t start = global_ns();
    while (global_ns() - start < 200000ull) {
    }
  }
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace gemm
}  // namespace dionw
