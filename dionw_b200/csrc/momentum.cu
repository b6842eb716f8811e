// HBM-bound passes over bucketed momentum: accumulate + row scores, row
// selection, error-feedback decay + pack to the Newton-Schulz operand.
//
// Every byte these kernels touch is used once per step, so their loads and stores carry
// the streaming (evict-first) hint: they run next to the tensor-core products on another
// stream and must not push the products' operands out of L2.
//
// Row kernels give one warp to one row.  The row is walked in chunks of 1024
// elements; lane t of the warp owns the float4 slots t, t+32, ..., t+224 of a
// chunk, i.e. the "score lanes" 4(t+32q)+i of the documented 1024-lane order,
// so the fold below reproduces that order exactly: lanes are combined by
// halving (512, 256, 128 inside a thread; 64..4 by shuffles; 2, 1 inside
// thread 0).
#include <algorithm>
#include <type_traits>

#include "cluster.cuh"
#include "common.cuh"

namespace dionw {
namespace {

constexpr int kTable = 64;
constexpr int kWarpsPerBlock = 8;

struct RowTable {
  const void* ptr[kTable];
  long long row_end[kTable];  // exclusive prefix of rows, relative to the launch
  int n;
};

__device__ __forceinline__ int find_tensor(const RowTable& tab, long long row) {
  int lo = 0, hi = tab.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (row < tab.row_end[mid]) hi = mid; else lo = mid + 1;
  }
  return lo;
}

template <typename G>
__device__ __forceinline__ void load4(const G* p, bool vec, long long e, long long cols, float (&out)[4]);

template <>
__device__ __forceinline__ void load4<float>(const float* p, bool vec, long long e, long long cols, float (&out)[4]) {
  if (vec) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p + e));
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (e + i < cols) ? p[e + i] : 0.0f;
  }
}
template <>
__device__ __forceinline__ void load4<__half>(const __half* p, bool vec, long long e, long long cols, float (&out)[4]) {
  if (vec) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p + e);
    const __half2 a = *reinterpret_cast<const __half2*>(&raw.x);
    const __half2 b = *reinterpret_cast<const __half2*>(&raw.y);
    out[0] = __low2float(a); out[1] = __high2float(a); out[2] = __low2float(b); out[3] = __high2float(b);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (e + i < cols) ? __half2float(p[e + i]) : 0.0f;
  }
}
template <>
__device__ __forceinline__ void load4<__nv_bfloat16>(const __nv_bfloat16* p, bool vec, long long e, long long cols,
                                                      float (&out)[4]) {
  if (vec) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p + e);
    out[0] = __uint_as_float(raw.x << 16); out[1] = __uint_as_float(raw.x & 0xFFFF0000u);
    out[2] = __uint_as_float(raw.y << 16); out[3] = __uint_as_float(raw.y & 0xFFFF0000u);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (e + i < cols) ? __bfloat162float(p[e + i]) : 0.0f;
  }
}

__device__ __forceinline__ void load4f(const float* p, bool vec, long long e, long long cols, float (&out)[4]) {
  if (vec) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p + e));
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = (e + i < cols) ? p[e + i] : 0.0f;
  }
}

__device__ __forceinline__ void store4f(float* p, bool vec, long long e, long long cols, const float (&v)[4]) {
  if (vec) {
    __stcs(reinterpret_cast<float4*>(p + e), make_float4(v[0], v[1], v[2], v[3]));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e + i < cols) p[e + i] = v[i];
  }
}

// The same, but for a line that is read again soon.
__device__ __forceinline__ void store4f_kept(float* p, bool vec, long long e, long long cols, const float (&v)[4]) {
  if (vec) {
    *reinterpret_cast<float4*>(p + e) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (e + i < cols) p[e + i] = v[i];
  }
}

// Folds the 8 x 4 per-thread lane accumulators of a warp into one value, in
// the documented order.  The result is valid in lane 0.
__device__ __forceinline__ float fold_lanes(float (&acc)[8][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc[0][i] = __fadd_rn(acc[0][i], acc[4][i]);
    acc[1][i] = __fadd_rn(acc[1][i], acc[5][i]);
    acc[2][i] = __fadd_rn(acc[2][i], acc[6][i]);
    acc[3][i] = __fadd_rn(acc[3][i], acc[7][i]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc[0][i] = __fadd_rn(acc[0][i], acc[2][i]);
    acc[1][i] = __fadd_rn(acc[1][i], acc[3][i]);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[0][i] = __fadd_rn(acc[0][i], acc[1][i]);
#pragma unroll
  for (int delta = 16; delta >= 1; delta >>= 1) {
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[0][i] = __fadd_rn(acc[0][i], __shfl_down_sync(0xffffffffu, acc[0][i], delta));
  }
  const float a = __fadd_rn(acc[0][0], acc[0][2]);
  const float b = __fadd_rn(acc[0][1], acc[0][3]);
  return __fadd_rn(a, b);
}

// ---------------------------------------------------------------------------
// teams: a CTA to a row, or to two or four short ones
// ---------------------------------------------------------------------------
// Warp q of the eight holds the float4 slots 32q .. 32q + 31 of each 1024-element chunk of a row, i.e. what a lone
// warp holds in its q-th registers, so the same fold gives the same sums.  Four chunks (of one row, of two or of four)
// are requested before the first is used.  Against a warp to a row that keeps as many bytes in flight with four times
// the registers, the rows being worked on lie close together in memory and twice as many loads are under way: scores
// of four 14336 x 4096 tensors 457 -> 409 us (6.9 TB/s), of a 4-layer 4096-wide model 1726 -> 1509; copies of twelve
// 768 x 2304 69 -> 58.
constexpr int kTeamThreads = kWarpsPerBlock * 32;
constexpr int kTeamChunks = 4;
// From how many columns on a team is the faster: for scores, for copies, for packing, and for packing in accesses of
// less than 16 bytes.  A warp to a row against a team, us: scores 32 x 1024 x 512 65 and 77, 12 x 3072 x 768 79 and 85,
// 6 x 1100 x 1100 30 and 26; copies 32 x 1024 x 512 71 and 75, 12 x 3072 x 768 93 and 89; packing all of 12 x 768 x 2304 31
// and 34, a quarter of 4 x 2048 x 2560 18.4 and 16.4, of 4 x 1024 x 4096 20 and 14; odd rows, a quarter of 8 x 700 x 701
// 16 and 18, of 6 x 2930 x 1101 22 and 20.
constexpr int kTeamScoreColumns = 1025, kTeamCopyColumns = 768, kTeamPackColumns = 2560, kTeamOddColumns = 1024;
// Whole blocks: a warp takes its row from L2, where the copying pass has left it, in the time that a CTA needs to come and
// go, so the more rows there are the longer they have to be, and longer still for bf16, whose three roundings hold a CTA up.
// After the copying pass, a warp to a row against a team, us.  16-byte accesses: 5859 x 2560 18.7 and 17.5 (bf16 19.8 and 20.6),
// 12695 x 2560 34 and 37, 10579 x 3072 36 and 35 (38 and 42), 15258 x 4096 69 and 65 (71 and 76), 36621 x 4096 162 and 163 (165
// and 184), 24414 x 6144 164 and 151 (167 and 173), 10172 x 6144 (74 and 72).  Shorter ones: 2724 x 1101 9.0 and 8.0, 5449 x 1101 12.2
// and 13.9, 20435 x 1101 37 and 49; 5002 x 1999 17.7 and 15.5, 11255 x 1999 33 and 33 (33 and 35), 31265 x 1999 78 and 97; 4164 x
// 2401 18 and 14; 22305 x 2802 87 and 81.
inline int team_whole_columns(int span, bool bf16, long long rows) {
  if (span != 4) return rows <= 4096 ? kTeamOddColumns : rows <= 8192 ? 1600 : 2560;
  return rows <= 8192 ? kTeamPackColumns : rows <= 16384 ? (bf16 ? 4096 : 3072) : bf16 ? 6144 : 4096;
}
// Four rows at a time only where they go in 16-byte accesses: in shorter ones a thread has four times the addresses and
// bounds, and copies of fp32 take, warps / four rows / two, us: 4000 x 1001 17.9 / 24.0 / 16.1, 30000 x 770 88 / 110 / 84,
// 1500 x 1024 off the boundary 8.4 / 11.2 / 7.7; of bf16 30000 x 1001 189 / 157 / 126.
inline int team_rows(long long cols, bool vec) { return cols <= 1024 && vec ? 4 : cols <= 2048 ? 2 : 1; }

// Runs of six to eight rows an SM: one even wave of warps, eight to an SM, but the beginning of a second wave of teams.
// fp32, a warp to a row against a team, us: copies of 1024 x 1024 4.5 and 5.1, 1184 x 1022 5.5 and 7.3, 1100 x 1999 9.9
// and 10.8, scores of 1100 x 1202 6.1 and 7.0; 860 x 1022 5.2 and 4.7, 1200 x 1022 8.6 and 7.4; 1024 x 1280 (16-byte accesses) 6.0 and
// 5.9.  (16-bit gradients 1000 x 1001 8.6 and 7.7.)
inline bool one_wave_of_warps(int grad_dtype, bool vec, long long cols, long long rows) {
  return cols <= (vec ? 1024 : 2048) && grad_dtype == DIONW_F32 && rows > 6 * sm_count() && rows <= 8 * sm_count();
}

// Calls fn(std::integral_constant<int, rows at a time>).
template <typename Fn>
auto with_team_rows(long long cols, bool vec, Fn&& fn) {
  switch (team_rows(cols, vec)) {
    case 4: return fn(std::integral_constant<int, 4>());
    case 2: return fn(std::integral_constant<int, 2>());
    default: return fn(std::integral_constant<int, 1>());
  }
}

// The sums of `kSums` sets of lane accumulators, each spread over the team: warp s folds set s and hands it to
// write(s, sum) in lane 0.
template <int kSums, typename Write>
__device__ __forceinline__ void fold_team(const float4 (&part)[kSums], Write&& write) {
  __shared__ float4 parts[kSums][kWarpsPerBlock][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < kSums; ++i) parts[i][warp][lane] = part[i];
  __syncthreads();
  if (warp < kSums) {
    float acc[kWarpsPerBlock][4];
#pragma unroll
    for (int q = 0; q < kWarpsPerBlock; ++q) {
      const float4 v = parts[warp][q][lane];
      acc[q][0] = v.x; acc[q][1] = v.y; acc[q][2] = v.z; acc[q][3] = v.w;
    }
    const float sum = fold_lanes(acc);
    if (lane == 0) write(warp, sum);
  }
}

// Rows row0 .. row0 + kRows - 1 of a run: their gradients, and whether they exist.
template <typename G, int kRows>
struct TeamRows {
  const G* g[kRows];
  bool there[kRows];
  __device__ __forceinline__ TeamRows(const RowTable& tab, long long row0, long long total_rows, long long cols) {
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const long long row = row0 + r;
      there[r] = row < total_rows;
      const int t = find_tensor(tab, there[r] ? row : total_rows - 1);
      g[r] = reinterpret_cast<const G*>(tab.ptr[t]) + (row - (t == 0 ? 0 : tab.row_end[t - 1])) * cols;
    }
  }
};

template <typename G, int kRows>
__global__ void __launch_bounds__(kTeamThreads, kRows == 1 ? 4 : 3)
team_accumulate_row_l1_kernel(const RowTable tab, float* __restrict__ momentum, float* __restrict__ scores,
                              float* __restrict__ sumsq, long long cols, long long total_rows, bool vec) {
  after_previous();
  constexpr int kChunks = kTeamChunks / kRows;
  const long long row0 = (long long)blockIdx.x * kRows;
  const TeamRows<G, kRows> rows(tab, row0, total_rows, cols);
  float sums[2 * kRows][4] = {};   // |m|, m^2
  for (long long base = 4 * threadIdx.x; base < cols; base += 1024 * kChunks) {
    float gv[kRows][kChunks][4], mv[kRows][kChunks][4];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const long long e = base + 1024 * c;
        if (rows.there[r] && e < cols) {
          load4<G>(rows.g[r], vec, e, cols, gv[r][c]);
          load4f(momentum + (row0 + r) * cols, vec, e, cols, mv[r][c]);
        }
      }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const long long e = base + 1024 * c;
        if (rows.there[r] && e < cols) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float v = __fadd_rn(mv[r][c][i], gv[r][c][i]);
            mv[r][c][i] = v;
            // Elements past the row end were loaded as zero and add nothing.
            sums[2 * r][i] = __fadd_rn(sums[2 * r][i], fabsf(v));
            sums[2 * r + 1][i] = __fadd_rn(sums[2 * r + 1][i], __fmul_rn(v, v));
          }
          store4f(momentum + (row0 + r) * cols, vec, e, cols, mv[r][c]);
        }
      }
  }
  float4 part[2 * kRows];
#pragma unroll
  for (int i = 0; i < 2 * kRows; ++i) part[i] = make_float4(sums[i][0], sums[i][1], sums[i][2], sums[i][3]);
  fold_team<2 * kRows>(part, [&](int i, float sum) {
    const long long row = row0 + (i >> 1);
    if (row < total_rows) ((i & 1) == 0 ? scores : sumsq)[row] = sum;
  });
}

template <typename G, int kRows>
__global__ void __launch_bounds__(kTeamThreads, kRows == 1 ? 4 : 3)
team_accumulate_copy_decay_kernel(const RowTable tab, float* __restrict__ momentum, float* __restrict__ u,
                                  float* __restrict__ sumsq, long long cols, long long total_rows, float decay,
                                  bool nesterov, bool vec) {
  after_previous();
  constexpr int kChunks = kTeamChunks / kRows;
  const long long row0 = (long long)blockIdx.x * kRows;
  const TeamRows<G, kRows> rows(tab, row0, total_rows, cols);
  float sums[kRows][4] = {};
  for (long long base = 4 * threadIdx.x; base < cols; base += 1024 * kChunks) {
    float gv[kRows][kChunks][4], mv[kRows][kChunks][4];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const long long e = base + 1024 * c;
        if (rows.there[r] && e < cols) {
          load4<G>(rows.g[r], vec, e, cols, gv[r][c]);
          load4f(momentum + (row0 + r) * cols, vec, e, cols, mv[r][c]);
        }
      }
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const long long e = base + 1024 * c;
        if (rows.there[r] && e < cols) {
          float uv[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float sum = __fadd_rn(mv[r][c][i], gv[r][c][i]);
            const float decayed = __fmul_rn(sum, decay);
            mv[r][c][i] = decayed;
            uv[i] = nesterov ? __fadd_rn(gv[r][c][i], decayed) : sum;
            sums[r][i] = __fadd_rn(sums[r][i], __fmul_rn(uv[i], uv[i]));
          }
          store4f(momentum + (row0 + r) * cols, vec, e, cols, mv[r][c]);
          store4f_kept(u + (row0 + r) * cols, vec, e, cols, uv);
        }
      }
  }
  float4 part[kRows];
#pragma unroll
  for (int i = 0; i < kRows; ++i) part[i] = make_float4(sums[i][0], sums[i][1], sums[i][2], sums[i][3]);
  fold_team<kRows>(part, [&](int i, float sum) {
    if (row0 + i < total_rows) sumsq[row0 + i] = sum;
  });
}

// M += G; scores = sum |M|; sumsq = sum M^2 per row.
template <typename G>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
accumulate_row_l1_kernel(const RowTable tab, float* __restrict__ momentum, float* __restrict__ scores,
                         float* __restrict__ sumsq, long long cols, long long total_rows, bool vec) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= total_rows) return;
  const int t = find_tensor(tab, row);
  const long long first = t == 0 ? 0 : tab.row_end[t - 1];
  const G* g = reinterpret_cast<const G*>(tab.ptr[t]) + (row - first) * cols;
  float* m = momentum + row * cols;
  float l1[8][4], sq[8][4];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) l1[q][i] = sq[q][i] = 0.0f;
  for (long long base = 0; base < cols; base += 1024) {
    float gv[8][4], mv[8][4];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long e = base + 4 * (lane + 32 * q);
      if (e < cols) {
        load4<G>(g, vec, e, cols, gv[q]);
        load4f(m, vec, e, cols, mv[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long e = base + 4 * (lane + 32 * q);
      if (e < cols) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float v = __fadd_rn(mv[q][i], gv[q][i]);
          mv[q][i] = v;
          // Elements past the row end were loaded as zero and add nothing.
          l1[q][i] = __fadd_rn(l1[q][i], fabsf(v));
          sq[q][i] = __fadd_rn(sq[q][i], __fmul_rn(v, v));
        }
        store4f(m, vec, e, cols, mv[q]);
      }
    }
  }
  const float s1 = fold_lanes(l1);
  const float s2 = fold_lanes(sq);
  if (lane == 0) {
    scores[row] = s1;
    sumsq[row] = s2;
  }
}

// m = M + G; M = decay m; u = m or G + decay m; sumsq = sum u^2 per row.
template <typename G>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
accumulate_copy_decay_kernel(const RowTable tab, float* __restrict__ momentum, float* __restrict__ u,
                             float* __restrict__ sumsq, long long cols, long long total_rows, float decay,
                             bool nesterov, bool vec) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= total_rows) return;
  const int t = find_tensor(tab, row);
  const long long first = t == 0 ? 0 : tab.row_end[t - 1];
  const G* g = reinterpret_cast<const G*>(tab.ptr[t]) + (row - first) * cols;
  float* m = momentum + row * cols;
  float* out = u + row * cols;
  float sq[8][4];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) sq[q][i] = 0.0f;
  for (long long base = 0; base < cols; base += 1024) {
    float gv[8][4], mv[8][4];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long e = base + 4 * (lane + 32 * q);
      if (e < cols) {
        load4<G>(g, vec, e, cols, gv[q]);
        load4f(m, vec, e, cols, mv[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const long long e = base + 4 * (lane + 32 * q);
      if (e < cols) {
        float uv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float sum = __fadd_rn(mv[q][i], gv[q][i]);
          const float decayed = __fmul_rn(sum, decay);
          mv[q][i] = decayed;
          uv[i] = nesterov ? __fadd_rn(gv[q][i], decayed) : sum;
          sq[q][i] = __fadd_rn(sq[q][i], __fmul_rn(uv[i], uv[i]));
        }
        store4f(m, vec, e, cols, mv[q]);
        store4f_kept(out, vec, e, cols, uv);
      }
    }
  }
  const float s2 = fold_lanes(sq);
  if (lane == 0) sumsq[row] = s2;
}

// ---------------------------------------------------------------------------
// row selection
// ---------------------------------------------------------------------------
constexpr int kSelectThreads = 1024;

__device__ __forceinline__ uint32_t order_key(float v) {
  const uint32_t bits = __float_as_uint(v);
  return (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
}

// One cluster of up to eight CTAs per block: radix-select the k-th largest score, then list the chosen
// rows in ascending order (rows equal to the threshold are taken lowest first).  Every CTA owns a
// consecutive range of rows, the first kKeep rows per thread in registers; a pass counts them into the
// CTA's own histogram and sums the cluster's through distributed shared memory.
//
// Bounded by latency: four dependent passes over a few tens of kilobytes.  One CTA per block walked 28672
// rows in 28 dependent steps per pass: the four selections of a one-layer 8192-wide model took 254 us, on
// clusters they take 141.  A CTA per 1024 rows, because below that a pass is one step and a larger cluster
// only adds barriers.
//
// A launch takes the blocks of up to six runs (launch_together): the selections of a step are some 10 us of latency each on a few SMs,
// and side by side they take the time of one.  Every run keeps the cluster that its own rows ask for (the first CTAs of
// the launch's), so that its sums have one order.
constexpr int kKeep = 4;

struct SelectRun {
  const float* scores;
  const float* sumsq;
  int32_t* index;
  int32_t* rowmap;
  float* frob;
  int rows, k;
  unsigned ctas;         // of a cluster that work on a block
  unsigned blocks;
  unsigned first_block;  // blocks of the runs before
};
template <int kRuns>
struct SelectTable {
  SelectRun run[kRuns];
  int n;
};

template <int kRuns>
__global__ void __launch_bounds__(kSelectThreads)
select_rows_kernel(const __grid_constant__ SelectTable<kRuns> tab) {
  after_previous();
  __shared__ uint32_t hist[4][256];
  __shared__ uint32_t s_prefix, s_remaining;
  __shared__ uint32_t warp_totals[32];
  __shared__ uint32_t s_gt, s_eq;          // this CTA's rows above and at the threshold
  __shared__ float partial[kSelectThreads];
  const int tid = threadIdx.x;
  const uint32_t rank = cluster_rank();
  const unsigned block = blockIdx.x / cluster_size();
  int at = 0;   // a constant, and with it where the run's values lie, for a run on its own
  if constexpr (kRuns > 1) {
    while (at + 1 < tab.n && block >= tab.run[at + 1].first_block) ++at;
  }
  const SelectRun& run = tab.run[at];
  const int rows = run.rows, k = run.k;
  const uint32_t ctas = kRuns > 1 ? run.ctas : cluster_size();
  int32_t* __restrict__ const index = run.index;
  int32_t* __restrict__ const rowmap = run.rowmap;
  const long long b = block - run.first_block;
  const float* ss = run.sumsq + b * rows;
  const float* sc = run.scores + b * rows;
  const int per = (rows + int(ctas) - 1) / int(ctas);
  const int first = min(rows, int(rank) * per), last = min(rows, first + per);

  const int warp = tid >> 5, lane = tid & 31;
  // Rows past the end get the lowest key and are told apart by their number.
  uint32_t kept[kKeep];
#pragma unroll
  for (int i = 0; i < kKeep; ++i) {
    const int r = first + i * kSelectThreads + tid;
    kept[i] = r < last ? order_key(sc[r]) : 0u;
  }
  for (int i = tid; i < 4 * 256; i += kSelectThreads) hist[0][i] = 0;
  if (tid == 0) s_gt = s_eq = 0;
  __syncthreads();

  // Calls visit(row, key) for each of the CTA's rows, the whole block in step; row >= last: no row.
  auto each_row = [&](auto&& visit) {
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      if (first + i * kSelectThreads < last) visit(first + i * kSelectThreads + tid, kept[i]);
    }
    for (int start = first + kKeep * kSelectThreads; start < last; start += kSelectThreads) {
      const int r = start + tid;
      visit(r, r < last ? order_key(sc[r]) : 0u);
    }
  };

  uint32_t prefix = 0, mask = 0, remaining = uint32_t(k);
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    // Scores of one block share sign and exponent, so in the first passes nearly every key
    // falls into one bin: the lanes of a warp that hit the same bin add once, together.
    each_row([&](int r, uint32_t key) {
      uint32_t bin = 256;   // not a candidate (or past the end)
      if (r < last && (key & mask) == prefix) bin = (key >> shift) & 255u;
      const uint32_t peers = __match_any_sync(0xffffffffu, bin);
      if (bin < 256 && lane == __ffs(peers) - 1) atomicAdd(&hist[pass][bin], uint32_t(__popc(peers)));
    });
    cluster_sync();
    // The highest bin whose count, added to the counts above it, reaches `remaining`: lane l of
    // warp 0 holds bins 8l..8l+7, a suffix sum over the lanes finds the lane, which finds the bin.
    if (warp == 0) {
      uint32_t cnt[8], own = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) cnt[i] = 0;
      for (uint32_t c = 0; c < ctas; ++c) {
#pragma unroll
        for (int i = 0; i < 8; ++i) cnt[i] += peer_load(&hist[pass][lane * 8 + i], c);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) own += cnt[i];
      uint32_t incl = own;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_down_sync(0xffffffffu, incl, d);
        if (lane + d < 32) incl += v;
      }
      uint32_t above = incl - own;   // candidates in the bins of higher lanes
      if (above < remaining && remaining <= incl) {
        int found = 0;
        bool open = true;
#pragma unroll
        for (int i = 7; i > 0; --i) {
          if (open && above + cnt[i] >= remaining) {
            found = i;
            open = false;
          }
          if (open) above += cnt[i];
        }
        s_prefix = prefix | (uint32_t(lane * 8 + found) << shift);
        s_remaining = remaining - above;
      }
    }
    __syncthreads();
    prefix = s_prefix;
    remaining = s_remaining;
    mask |= 255u << shift;
    __syncthreads();
  }
  const uint32_t threshold = prefix;     // key of the k-th largest score
  const uint32_t take_equal = remaining; // rows equal to it that are still needed

  // Rows above and at the threshold in the CTAs before this one.
  each_row([&](int r, uint32_t key) {
    const uint32_t gt = __popc(__ballot_sync(0xffffffffu, r < last && key > threshold));
    const uint32_t eq = __popc(__ballot_sync(0xffffffffu, r < last && key == threshold));
    if (lane == 0 && gt != 0) atomicAdd(&s_gt, gt);
    if (lane == 0 && eq != 0) atomicAdd(&s_eq, eq);
  });
  cluster_sync();
  uint32_t base_gt = 0, base_eq = 0;
  for (uint32_t c = 0; c < rank; ++c) {
    base_gt += peer_load(&s_gt, c);
    base_eq += peer_load(&s_eq, c);
  }
  float local = 0.0f;
  each_row([&](int r, uint32_t key) {
    const bool gt = r < last && key > threshold, eq = r < last && key == threshold;
    const uint32_t gt_ballot = __ballot_sync(0xffffffffu, gt);
    const uint32_t eq_ballot = __ballot_sync(0xffffffffu, eq);
    const uint32_t below = (1u << lane) - 1u;
    uint32_t gt_before = __popc(gt_ballot & below);
    uint32_t eq_before = __popc(eq_ballot & below);
    if (lane == 0) warp_totals[warp] = (__popc(gt_ballot) << 16) | __popc(eq_ballot);
    __syncthreads();
    uint32_t gt_total = 0, eq_total = 0;
    for (int w = 0; w < 32; ++w) {
      const uint32_t packed = warp_totals[w];
      if (w < warp) {
        gt_before += packed >> 16;
        eq_before += packed & 0xFFFFu;
      }
      gt_total += packed >> 16;
      eq_total += packed & 0xFFFFu;
    }
    if (r < last) {
      const uint32_t eq_rank = base_eq + eq_before;
      const bool chosen = gt || (eq && eq_rank < take_equal);
      int32_t pos = -1;
      if (chosen) {
        const uint32_t eq_taken_before = eq_rank < take_equal ? eq_rank : take_equal;
        pos = int32_t(base_gt + gt_before + eq_taken_before);
        index[b * k + pos] = r;
        local = __fadd_rn(local, ss[r]);
      }
      rowmap[b * rows + r] = pos;
    }
    base_gt += gt_total;
    base_eq += eq_total;
    __syncthreads();
  });
  partial[tid] = local;
  __syncthreads();
  for (int width = kSelectThreads / 2; width >= 1; width >>= 1) {
    if (tid < width) partial[tid] = __fadd_rn(partial[tid], partial[tid + width]);
    __syncthreads();
  }
  cluster_sync();
  if (rank == 0 && tid == 0) {
    float total = 0.0f;
    for (uint32_t c = 0; c < ctas; ++c) total = __fadd_rn(total, __uint_as_float(peer_load(&partial[0], c)));
    run.frob[b] = sqrtf(total);
  }
  cluster_sync();   // the other CTAs' shared memory stays until rank 0 has read it
}

__global__ void __launch_bounds__(kSelectThreads)
block_norms_kernel(const float* __restrict__ sumsq, int rows, float* __restrict__ frob) {
  after_previous();
  __shared__ float partial[kSelectThreads];
  const int tid = threadIdx.x;
  const float* ss = sumsq + (long long)blockIdx.x * rows;
  float local = 0.0f;
  for (int r = tid; r < rows; r += kSelectThreads) local = __fadd_rn(local, ss[r]);
  partial[tid] = local;
  __syncthreads();
  for (int width = kSelectThreads / 2; width >= 1; width >>= 1) {
    if (tid < width) partial[tid] = __fadd_rn(partial[tid], partial[tid + width]);
    __syncthreads();
  }
  if (tid == 0) frob[blockIdx.x] = sqrtf(partial[0]);
}

// ---------------------------------------------------------------------------
// decay + pack
// ---------------------------------------------------------------------------
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <bool kBf16>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
pack_rows_kernel(float* __restrict__ src, const int32_t* __restrict__ index, const float* __restrict__ frob,
                 long long rows, long long k, long long cols, long long total, float decay, bool decay_rows,
                 float eps, float norm_scale, uint16_t* __restrict__ x, long long ldx, bool vec) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long long place = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (place >= total) return;
  // Copies of whole blocks from their end on: what the accumulating pass wrote last is still in L2 (packing a 12-layer
  // 768-wide model: 97 us so, 107 with the copies streamed past L2 and read from their start).
  const long long item = index ? place : total - 1 - place;
  const long long b = item / k;
  const long long source_row = index ? (long long)index[item] : (item - b * k);
  float* m = src + (b * rows + source_row) * cols;
  uint16_t* dst = x + item * ldx;
  float denom;
  if (kBf16) {
    // The bf16 iterations normalise in bf16: norm, scaled norm and sum are each rounded.
    denom = bf16_round(bf16_round(bf16_round(frob[b]) * norm_scale) + eps);
  } else {
    denom = __fadd_rn(frob[b], eps);
  }
  // Four 16-byte loads per lane are requested before the first is used: a warp keeps 2 KB of
  // the row in flight, which is what the stream needs to approach the memory rate.
  constexpr int kUnroll = 4;
  for (long long e0 = 4LL * lane; e0 < cols; e0 += 128 * kUnroll) {
    float v[kUnroll][4];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long e = e0 + 128LL * u;
      if (e < cols) load4f(m, vec, e, cols, v[u]);
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long e = e0 + 128LL * u;
      if (e >= cols) break;
      uint16_t h[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (kBf16) {
          const __nv_bfloat16 r = __float2bfloat16_rn(__fdiv_rn(bf16_round(v[u][i]), denom));
          h[i] = *reinterpret_cast<const uint16_t*>(&r);
        } else {
          const __half r = __float2half_rn(__fdiv_rn(v[u][i], denom));
          h[i] = *reinterpret_cast<const uint16_t*>(&r);
        }
      }
      if (vec) {
        uint2 packed;
        packed.x = uint32_t(h[0]) | (uint32_t(h[1]) << 16);
        packed.y = uint32_t(h[2]) | (uint32_t(h[3]) << 16);
        __stcs(reinterpret_cast<uint2*>(dst + e), packed);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (e + i < cols) dst[e + i] = h[i];
      }
      if (decay_rows) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[u][i] = __fmul_rn(v[u][i], decay);
        store4f(m, vec, e, cols, v[u]);
      }
    }
  }
  // Zero the padding columns so that they add nothing to any product.
  for (long long e = cols + lane; e < ldx; e += 32) dst[e] = 0;
}

// The same with a team to a row, kSpan elements to an access: a quarter of 1024 x 4096 18 -> 10 us, of 4 x 4099 x 4099
// (rows in accesses of 4 bytes) 59 -> 41, of 4 x 14336 x 4096 109 -> 100 (5.9 TB/s).
template <bool kBf16, int kSpan>
__global__ void __launch_bounds__(kTeamThreads, 6)
team_pack_rows_kernel(float* __restrict__ src, const int32_t* __restrict__ index, const float* __restrict__ frob,
                      long long rows, long long k, long long cols, float decay, bool decay_rows, float eps,
                      float norm_scale, uint16_t* __restrict__ x, long long ldx) {
  after_previous();
  constexpr int kChunks = 16 / kSpan, kStep = kTeamThreads * kSpan;
  const long long item = index ? blockIdx.x : gridDim.x - 1 - blockIdx.x, b = item / k;   // see pack_rows_kernel
  float* const m = src + (b * rows + (index ? (long long)index[item] : item - b * k)) * cols;
  uint16_t* const dst = x + item * ldx;
  const float norm = frob[b];
  // The bf16 iterations normalise in bf16: norm, scaled norm and sum are each rounded.
  const float denom = kBf16 ? bf16_round(bf16_round(bf16_round(norm) * norm_scale) + eps) : __fadd_rn(norm, eps);
  for (long long base = kSpan * threadIdx.x; base < cols; base += kStep * kChunks) {
    float v[kChunks][kSpan];
#pragma unroll
    for (int c = 0; c < kChunks; ++c)
      if (base + kStep * c < cols) Span<kSpan>::load(m + base + kStep * c, v[c]);
#pragma unroll
    for (int c = 0; c < kChunks; ++c) {
      const long long e = base + kStep * c;
      if (e >= cols) break;
      uint32_t h[kSpan];
#pragma unroll
      for (int i = 0; i < kSpan; ++i) {
        if (kBf16) {
          const __nv_bfloat16 q = __float2bfloat16_rn(__fdiv_rn(bf16_round(v[c][i]), denom));
          h[i] = *reinterpret_cast<const uint16_t*>(&q);
        } else {
          const __half q = __float2half_rn(__fdiv_rn(v[c][i], denom));
          h[i] = *reinterpret_cast<const uint16_t*>(&q);
        }
      }
      Span<kSpan>::store(dst + e, h);
      if (decay_rows) {
#pragma unroll
        for (int i = 0; i < kSpan; ++i) v[c][i] = __fmul_rn(v[c][i], decay);
        Span<kSpan>::store(m + e, v[c]);
      }
    }
  }
  for (long long e = cols + threadIdx.x; e < ldx; e += kTeamThreads) dst[e] = 0;   // adds nothing to any product
}

// ---------------------------------------------------------------------------
// normalise + pack a caller's own batch
// ---------------------------------------------------------------------------
// 16 bytes of a row as floats: 4 elements of a 4-byte type, 8 of a 2-byte type.
template <typename S>
struct Quad;
template <>
struct Quad<float> {
  static constexpr int kCount = 4;
  static __device__ __forceinline__ void unpack(const uint4& raw, float (&out)[4]) {
    out[0] = __uint_as_float(raw.x); out[1] = __uint_as_float(raw.y);
    out[2] = __uint_as_float(raw.z); out[3] = __uint_as_float(raw.w);
  }
};
template <>
struct Quad<__half> {
  static constexpr int kCount = 8;
  static __device__ __forceinline__ void unpack(const uint4& raw, float (&out)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      out[2 * i] = f.x; out[2 * i + 1] = f.y;
    }
  }
};
template <>
struct Quad<__nv_bfloat16> {
  static constexpr int kCount = 8;
  static __device__ __forceinline__ void unpack(const uint4& raw, float (&out)[8]) {
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      out[2 * i] = __uint_as_float(w[i] << 16); out[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
};

// A row in steps of 4 x 16 bytes per lane, all four requested before the first is used; `use` gets the
// position of the first element and up to kCount elements (`count` of them; 0 past the row end).
template <typename S, typename Use>
__device__ __forceinline__ void walk_row(const S* __restrict__ row, long long cols, bool vec, int lane, Use&& use) {
  constexpr int kUnroll = 4, kCount = Quad<S>::kCount;
  for (long long e0 = kCount * lane; e0 < cols; e0 += 32 * kCount * kUnroll) {
    if (vec) {
      uint4 raw[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const long long e = e0 + 32LL * kCount * u;
        if (e < cols) raw[u] = *reinterpret_cast<const uint4*>(row + e);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const long long e = e0 + 32LL * kCount * u;
        if (e >= cols) break;
        float v[kCount];
        Quad<S>::unpack(raw[u], v);
        use(e, v, kCount);
      }
    } else {
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const long long e = e0 + 32LL * kCount * u;
        if (e >= cols) break;
        float v[kCount];
#pragma unroll
        for (int i = 0; i < kCount; ++i) v[i] = e + i < cols ? to_float<S>(row[e + i]) : 0.0f;
        use(e, v, cols - e < kCount ? int(cols - e) : kCount);
      }
    }
  }
}

// Row sums of squares (of the values rounded to bf16 first for the bf16 iterations), for a caller that has no
// norms, and the normalised 2-byte operand, straight from the caller's dtype.  HBM-bound: two reads of the
// source (the norm needs the whole block before the first division) and one write of the operand are all the
// traffic.  A conversion to fp32 in front of norm and pack moved 18 bytes per bf16 element instead of 6: 16
// blocks of 4096 x 14336 spent 5.4 ms of a 38.7 ms call in conversion, norm and pack.
template <typename S, bool kBf16>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
source_sumsq_kernel(const S* __restrict__ src, long long total_rows, long long cols, float* __restrict__ sumsq,
                    bool vec) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= total_rows) return;
  float acc[Quad<S>::kCount] = {};
  walk_row<S>(src + row * cols, cols, vec, lane, [&](long long, const float* v, int) {
#pragma unroll
    for (int i = 0; i < Quad<S>::kCount; ++i) {
      const float x = kBf16 ? bf16_round(v[i]) : v[i];
      acc[i] = fmaf(x, x, acc[i]);
    }
  });
  float sum = 0.0f;
#pragma unroll
  for (int width = Quad<S>::kCount / 2; width >= 1; width >>= 1)
#pragma unroll
    for (int i = 0; i < width; ++i) acc[i] += acc[i + width];
  sum = acc[0];
#pragma unroll
  for (int delta = 16; delta >= 1; delta >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, delta);
  if (lane == 0) sumsq[row] = sum;
}

template <typename S, bool kBf16>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
source_pack_kernel(const S* __restrict__ src, const float* __restrict__ frob, long long total_rows, long long rows,
                   long long cols, float eps, float norm_scale, uint16_t* __restrict__ x, long long ldx, bool vec) {
  after_previous();
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5);
  if (row >= total_rows) return;
  const float norm = frob[row / rows];
  // The bf16 iterations normalise in bf16: norm, scaled norm and sum are each rounded.
  const float denom = kBf16 ? bf16_round(bf16_round(bf16_round(norm) * norm_scale) + eps) : __fadd_rn(norm, eps);
  uint16_t* dst = x + row * ldx;
  walk_row<S>(src + row * cols, cols, vec, lane, [&](long long e, const float* v, int count) {
    constexpr int kCount = Quad<S>::kCount;
    uint32_t w[kCount / 2];
#pragma unroll
    for (int i = 0; i < kCount / 2; ++i) {
      float2 q;
      q.x = __fdiv_rn(kBf16 ? bf16_round(v[2 * i]) : v[2 * i], denom);
      q.y = __fdiv_rn(kBf16 ? bf16_round(v[2 * i + 1]) : v[2 * i + 1], denom);
      if (kBf16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(q.x, q.y);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
      } else {
        const __half2 h = __floats2half2_rn(q.x, q.y);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
      }
    }
    if (vec) {
      if constexpr (kCount == 8) *reinterpret_cast<uint4*>(dst + e) = make_uint4(w[0], w[1], w[2], w[3]);
      else *reinterpret_cast<uint2*>(dst + e) = make_uint2(w[0], w[1]);
    } else {
#pragma unroll
      for (int i = 0; i < kCount; ++i)
        if (i < count) dst[e + i] = uint16_t(w[i >> 1] >> (16 * (i & 1)));
    }
  });
  for (long long e = cols + lane; e < ldx; e += 32) dst[e] = 0;   // padding adds nothing to any product
}

template <typename S, bool kBf16>
int source_pack(const void* src, int64_t blocks, int64_t rows, int64_t cols, float eps, float norm_scale, void* x,
                int64_t ldx, float* sumsq, float* frob, cudaStream_t stream) {
  const long long total = blocks * rows;
  const unsigned grid = unsigned((total + kWarpsPerBlock - 1) / kWarpsPerBlock);
  const S* typed = static_cast<const S*>(src);
  const bool vec = cols % Quad<S>::kCount == 0 && aligned16(src) && aligned16(x);   // ldx is a multiple of 8
  if (sumsq != nullptr) {
    launch_dependent(source_sumsq_kernel<S, kBf16>, grid, kWarpsPerBlock * 32, stream, typed, total, cols, sumsq, vec);
    int st = launch_status("source_sumsq_kernel");
    if (st != DIONW_OK) return st;
    launch_dependent(block_norms_kernel, unsigned(blocks), kSelectThreads, stream, sumsq, int(rows), frob);
    st = launch_status("block_norms_kernel");
    if (st != DIONW_OK) return st;
  }
  launch_dependent(source_pack_kernel<S, kBf16>, grid, kWarpsPerBlock * 32, stream, typed, frob, total, rows, cols, eps, norm_scale,
                                                                         static_cast<uint16_t*>(x), ldx, vec);
  return launch_status("source_pack_kernel");
}

__global__ void transpose_2byte_kernel(const uint16_t* __restrict__ in, uint16_t* __restrict__ out, long long rows,
                                       long long cols, long long ld_in, long long ld_out) {
  __shared__ uint16_t tile[64][66];
  const long long b = blockIdx.z;
  const uint16_t* src = in + b * rows * ld_in;
  uint16_t* dst = out + b * cols * ld_out;
  const long long r0 = (long long)blockIdx.y * 64, c0 = (long long)blockIdx.x * 64;
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const long long r = r0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const long long c = c0 + j;
      tile[i][j] = (r < rows && c < cols) ? src[r * ld_in + c] : uint16_t(0);
    }
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const long long c = c0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const long long r = r0 + j;
      if (c < cols && r < rows) dst[c * ld_out + r] = tile[j][i];
    }
  }
  // padding columns of the output rows
  if (blockIdx.y == 0) {
    for (int i = threadIdx.y; i < 64; i += blockDim.y) {
      const long long c = c0 + i;
      if (c < cols)
        for (long long p = rows + threadIdx.x; p < ld_out; p += blockDim.x) dst[c * ld_out + p] = 0;
    }
  }
}

template <typename Fn>
int for_each_table(const void* const* ptrs, const int64_t* rows_per_tensor, int n_tensors, Fn&& launch_one) {
  long long done_rows = 0;
  for (int start = 0; start < n_tensors; start += kTable) {
    RowTable tab;
    tab.n = (n_tensors - start < kTable) ? n_tensors - start : kTable;
    long long acc = 0;
    for (int i = 0; i < tab.n; ++i) {
      tab.ptr[i] = ptrs[start + i];
      acc += rows_per_tensor[start + i];
      tab.row_end[i] = acc;
    }
    const int st = launch_one(tab, done_rows, acc);
    if (st != DIONW_OK) return st;
    done_rows += acc;
  }
  return DIONW_OK;
}

bool table_vectorizable(const void* const* ptrs, int n, int64_t cols) {
  if (cols % 4 != 0) return false;
  for (int i = 0; i < n; ++i)
    if (!aligned16(ptrs[i])) return false;
  return true;
}

}  // namespace
}  // namespace dionw

using namespace dionw;

extern "C" int dionw_accumulate_row_l1_run(const void* const* grads, int grad_dtype, const int64_t* rows_per_tensor,
                                           int n_tensors, float* momentum, float* scores, float* sumsq, int64_t cols,
                                           void* stream_ptr) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  DIONW_REQUIRE(n_tensors > 0 && cols > 0, "accumulate_row_l1_run: empty run");
  DIONW_REQUIRE(grad_dtype >= DIONW_F32 && grad_dtype <= DIONW_BF16, "accumulate_row_l1_run: bad gradient dtype");
  const bool vec = table_vectorizable(grads, n_tensors, cols) && aligned16(momentum);
  return for_each_table(grads, rows_per_tensor, n_tensors, [&](const RowTable& tab, long long row0, long long nrows) {
    if (nrows == 0) return DIONW_OK;
    const unsigned grid = unsigned((nrows + kWarpsPerBlock - 1) / kWarpsPerBlock);
    float* m = momentum + row0 * cols;
    if (cols >= kTeamScoreColumns && !one_wave_of_warps(grad_dtype, vec, cols, nrows)) {
      auto launch = [&](auto g) {
        with_team_rows(cols, vec, [&](auto n) {
          constexpr int kRows = decltype(n)::value < 2 ? 1 : 2;   // of the kernel and of its grid; four need too many sums
          launch_dependent(team_accumulate_row_l1_kernel<decltype(g), kRows>, unsigned((nrows + kRows - 1) / kRows), kTeamThreads, stream, tab,
                           m, scores + row0, sumsq + row0, cols, nrows, vec);
        });
      };
      if (grad_dtype == DIONW_F32) launch(float());
      else if (grad_dtype == DIONW_F16) launch(__half());
      else launch(__nv_bfloat16());
      return launch_status("team_accumulate_row_l1_kernel");
    }
    if (grad_dtype == DIONW_F32)
      launch_dependent(accumulate_row_l1_kernel<float>, grid, kWarpsPerBlock * 32, stream, tab, m, scores + row0, sumsq + row0, cols, nrows, vec);
    else if (grad_dtype == DIONW_F16)
      launch_dependent(accumulate_row_l1_kernel<__half>, grid, kWarpsPerBlock * 32, stream, tab, m, scores + row0, sumsq + row0, cols, nrows, vec);
    else
      launch_dependent(accumulate_row_l1_kernel<__nv_bfloat16>, grid, kWarpsPerBlock * 32, stream, tab, m, scores + row0, sumsq + row0, cols, nrows, vec);
    return launch_status("accumulate_row_l1_kernel");
  });
}

extern "C" int dionw_accumulate_copy_decay_run(const void* const* grads, int grad_dtype,
                                               const int64_t* rows_per_tensor, int n_tensors, float* momentum,
                                               float* u, float* sumsq, int64_t cols, float decay, int nesterov,
                                               void* stream_ptr) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  DIONW_REQUIRE(n_tensors > 0 && cols > 0, "accumulate_copy_decay_run: empty run");
  DIONW_REQUIRE(grad_dtype >= DIONW_F32 && grad_dtype <= DIONW_BF16, "accumulate_copy_decay_run: bad gradient dtype");
  const bool vec = table_vectorizable(grads, n_tensors, cols) && aligned16(momentum) && aligned16(u);
  return for_each_table(grads, rows_per_tensor, n_tensors, [&](const RowTable& tab, long long row0, long long nrows) {
    if (nrows == 0) return DIONW_OK;
    const unsigned grid = unsigned((nrows + kWarpsPerBlock - 1) / kWarpsPerBlock);
    float* m = momentum + row0 * cols;
    float* out = u + row0 * cols;
    const bool nest = nesterov != 0;
    if (cols >= kTeamCopyColumns && !one_wave_of_warps(grad_dtype, vec, cols, nrows)) {
      auto launch = [&](auto g) {
        with_team_rows(cols, vec, [&](auto n) {
          launch_dependent(team_accumulate_copy_decay_kernel<decltype(g), decltype(n)::value>, unsigned((nrows + n - 1) / n), kTeamThreads, stream, tab,
                           m, out, sumsq + row0, cols, nrows, decay, nest, vec);
        });
      };
      if (grad_dtype == DIONW_F32) launch(float());
      else if (grad_dtype == DIONW_F16) launch(__half());
      else launch(__nv_bfloat16());
      return launch_status("team_accumulate_copy_decay_kernel");
    }
    if (grad_dtype == DIONW_F32)
      launch_dependent(accumulate_copy_decay_kernel<float>, grid, kWarpsPerBlock * 32, stream, tab, m, out, sumsq + row0, cols, nrows, decay, nest, vec);
    else if (grad_dtype == DIONW_F16)
      launch_dependent(accumulate_copy_decay_kernel<__half>, grid, kWarpsPerBlock * 32, stream, tab, m, out, sumsq + row0, cols, nrows, decay, nest, vec);
    else
      launch_dependent(accumulate_copy_decay_kernel<__nv_bfloat16>, grid, kWarpsPerBlock * 32, stream, tab, m, out, sumsq + row0, cols, nrows, decay, nest, vec);
    return launch_status("accumulate_copy_decay_kernel");
  });
}

extern "C" int dionw_select_rows_group(int n, const float* const* scores, const float* const* sumsq, const int64_t* blocks,
                                       const int64_t* rows, const int64_t* k, int32_t* const* index, int32_t* const* rowmap,
                                       float* const* frob, void* stream_ptr) {
  DIONW_REQUIRE(n >= 1 && n <= kGroupRuns, "select_rows_group: takes 1 to %d runs (got %d)", kGroupRuns, n);
  SelectRun runs[kGroupRuns];
  for (int i = 0; i < n; ++i) {
    DIONW_REQUIRE(blocks[i] > 0 && rows[i] > 0 && k[i] > 0 && k[i] <= rows[i], "select_rows: need 0 < k <= rows and blocks > 0");
    DIONW_REQUIRE(rows[i] < (1LL << 30) && blocks[i] < (1LL << 31), "select_rows: too many rows or blocks");
    runs[i] = SelectRun{scores[i], sumsq[i], index[i], rowmap[i], frob[i], int(rows[i]), int(k[i]),
                        cluster_for(blocks[i], rows[i], kSelectThreads), unsigned(blocks[i]), 0};
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  return launch_together(runs, n, 3, [&](const SelectRun* run, int count, unsigned total, unsigned cluster) {
    count_launch();
    if (count == 1)
      return check_cuda(launch_clusters(select_rows_kernel<1>, total, cluster, kSelectThreads, stream, SelectTable<1>{{*run}, 1}),
                        "select_rows_kernel");
    SelectTable<kGroupRuns> tab;
    std::copy(run, run + count, tab.run);
    tab.n = count;
    return check_cuda(launch_clusters(select_rows_kernel<kGroupRuns>, total, cluster, kSelectThreads, stream, tab), "select_rows_kernel");
  });
}

extern "C" int dionw_select_rows(const float* scores, const float* sumsq, int64_t blocks, int64_t rows, int64_t k,
                                 int32_t* index, int32_t* rowmap, float* frob, void* stream_ptr) {
  return dionw_select_rows_group(1, &scores, &sumsq, &blocks, &rows, &k, &index, &rowmap, &frob, stream_ptr);
}

extern "C" int dionw_block_norms(const float* sumsq, int64_t blocks, int64_t rows, float* frob, void* stream_ptr) {
  DIONW_REQUIRE(blocks > 0 && rows > 0, "block_norms: empty problem");
  launch_dependent(block_norms_kernel, unsigned(blocks), kSelectThreads, static_cast<cudaStream_t>(stream_ptr), sumsq, int(rows), frob);
  return launch_status("block_norms_kernel");
}

extern "C" int dionw_pack_rows(float* src, const int32_t* index, const float* frob, int64_t blocks, int64_t rows,
                               int64_t k, int64_t cols, float decay, int decay_rows, float eps, float norm_scale,
                               void* x, int x_dtype, int64_t ldx, void* stream_ptr) {
  DIONW_REQUIRE(blocks > 0 && rows > 0 && k > 0 && k <= rows && cols > 0, "pack_rows: empty problem");
  DIONW_REQUIRE(x_dtype == DIONW_F16 || x_dtype == DIONW_BF16, "pack_rows: x must be F16 or BF16");
  DIONW_REQUIRE(ldx >= cols, "pack_rows: ldx must be >= cols");
  const long long total = blocks * k;
  const bool vec = cols % 4 == 0 && ldx % 4 == 0 && aligned16(src) && aligned16(x);
  const unsigned grid = unsigned((total + kWarpsPerBlock - 1) / kWarpsPerBlock);
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  const int span = span_of(cols, ldx);
  const int team_columns = index == nullptr ? team_whole_columns(span, x_dtype == DIONW_BF16, total) : span == 4 ? kTeamPackColumns : kTeamOddColumns;
  if (aligned16(src) && aligned16(x) && cols >= team_columns && total <= 0x7FFFFFFFll) {
    auto launch = [&](auto bf16, auto n) {
      launch_dependent(team_pack_rows_kernel<decltype(bf16)::value, decltype(n)::value>, unsigned(total), kTeamThreads, stream, src, index, frob,
                       rows, k, cols, decay, decay_rows != 0, eps, norm_scale, static_cast<uint16_t*>(x), ldx);
    };
    auto with_span = [&](auto bf16) {
      if (span == 4) launch(bf16, std::integral_constant<int, 4>());
      else if (span == 2) launch(bf16, std::integral_constant<int, 2>());
      else launch(bf16, std::integral_constant<int, 1>());
    };
    if (x_dtype == DIONW_BF16) with_span(std::true_type());
    else with_span(std::false_type());
    return launch_status("team_pack_rows_kernel");
  }
  if (x_dtype == DIONW_BF16)
    launch_dependent(pack_rows_kernel<true>, grid, kWarpsPerBlock * 32, stream, src, index, frob, rows, k, cols, total, decay,
                                                                      decay_rows != 0, eps, norm_scale,
                                                                      static_cast<uint16_t*>(x), ldx, vec);
  else
    launch_dependent(pack_rows_kernel<false>, grid, kWarpsPerBlock * 32, stream, src, index, frob, rows, k, cols, total, decay,
                                                                       decay_rows != 0, eps, norm_scale,
                                                                       static_cast<uint16_t*>(x), ldx, vec);
  return launch_status("pack_rows_kernel");
}

extern "C" int dionw_normalize_pack(const void* src, int src_dtype, int64_t blocks, int64_t rows, int64_t cols,
                                    float eps, float norm_scale, void* x, int x_dtype, int64_t ldx, float* sumsq,
                                    float* frob, void* stream_ptr) {
  DIONW_REQUIRE(blocks > 0 && rows > 0 && cols > 0, "normalize_pack: empty problem");
  DIONW_REQUIRE(rows < (1LL << 30), "normalize_pack: too many rows");
  DIONW_REQUIRE(src_dtype >= DIONW_F32 && src_dtype <= DIONW_BF16, "normalize_pack: bad source dtype");
  DIONW_REQUIRE(x_dtype == DIONW_F16 || x_dtype == DIONW_BF16, "normalize_pack: x must be F16 or BF16");
  DIONW_REQUIRE(ldx >= cols && ldx % 8 == 0, "normalize_pack: ldx must be >= cols and a multiple of 8");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
#define DIONW_SOURCE(type)                                                                                       \
  return x_dtype == DIONW_BF16                                                                                   \
             ? source_pack<type, true>(src, blocks, rows, cols, eps, norm_scale, x, ldx, sumsq, frob, stream)    \
             : source_pack<type, false>(src, blocks, rows, cols, eps, norm_scale, x, ldx, sumsq, frob, stream)
  if (src_dtype == DIONW_F32) DIONW_SOURCE(float);
  if (src_dtype == DIONW_F16) DIONW_SOURCE(__half);
  DIONW_SOURCE(__nv_bfloat16);
#undef DIONW_SOURCE
}

extern "C" int dionw_transpose_2byte(const void* in, void* out, int64_t blocks, int64_t rows, int64_t cols,
                                     int64_t ld_in, int64_t ld_out, void* stream_ptr) {
  DIONW_REQUIRE(blocks > 0 && rows > 0 && cols > 0, "transpose_2byte: empty problem");
  DIONW_REQUIRE(ld_in >= cols && ld_out >= rows, "transpose_2byte: leading dimensions too small");
  DIONW_REQUIRE(blocks <= 65535, "transpose_2byte: more than 65535 blocks in one call");
  const dim3 grid(unsigned((cols + 63) / 64), unsigned((rows + 63) / 64), unsigned(blocks));
  transpose_2byte_kernel<<<grid, dim3(32, 8), 0, static_cast<cudaStream_t>(stream_ptr)>>>(
      static_cast<const uint16_t*>(in), static_cast<uint16_t*>(out), rows, cols, ld_in, ld_out);
  return launch_status("transpose_2byte_kernel");
}
