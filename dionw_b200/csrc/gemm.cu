// Host side of the tcgen05 GEMMs: tensor maps, launches, and the Newton-Schulz
// product schedules built from them.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <map>
#include <mutex>
#include <utility>

#include "gemm2_sm100.cuh"
#include "onchip_sm100.cuh"
#include "products.cuh"

namespace dionw {

// Products, and the other kernels of a step (cluster.cuh), are launched with programmatic stream serialization:
// they wait with griddepcontrol.wait before they touch global memory.  DIONW_GEMM_PDL=0 turns that off.
// Measured on the Llama-3-8B-shaped step, for the products when each was a launch of its own (about 290 per
// step): 95.1-96.2 ms with it, 98.3-99.0 ms without.
bool use_dependent_launch() {
  static const bool on = [] {
    const char* v = std::getenv("DIONW_GEMM_PDL");
    return v == nullptr || v[0] != '0';
  }();
  return on;
}

namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver entry point is looked up at run time so that the library itself
// links against the CUDA runtime only and still loads on a machine without a GPU.
EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess &&
        res == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeFn>(ptr);
    }
  });
  return fn;
}

// 3-D map over a batch of row-major 2-byte matrices: (inner, rows, batch).
int make_map(CUtensorMap* map, const void* base, int dtype, int64_t inner, int64_t rows, int64_t batches,
             int64_t ld, int64_t batch_stride, uint32_t box_inner, uint32_t box_rows) {
  EncodeFn fn = encode_fn();
  if (fn == nullptr) {
    set_error("cuTensorMapEncodeTiled is not available from this driver");
    return DIONW_ERR_CUDA;
  }
  DIONW_REQUIRE(aligned16(base), "matrix base address must be 16-byte aligned");
  DIONW_REQUIRE(ld % 8 == 0 && batch_stride % 8 == 0,
                "leading dimension (%lld) and batch stride (%lld) must be multiples of 8 elements",
                (long long)ld, (long long)batch_stride);
  cuuint64_t dims[3] = {cuuint64_t(inner), cuuint64_t(rows), cuuint64_t(batches)};
  cuuint64_t strides[2] = {cuuint64_t(ld) * 2, cuuint64_t(batch_stride) * 2};
  if (batches == 1) strides[1] = cuuint64_t(ld) * 2 * cuuint64_t(rows);
  cuuint32_t box[3] = {box_inner, box_rows, 1};
  cuuint32_t elem[3] = {1, 1, 1};
  const CUtensorMapDataType type = dtype == DIONW_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                       : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult res = fn(map, type, 3, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed with code %d (inner=%lld rows=%lld batches=%lld ld=%lld)", int(res),
              (long long)inner, (long long)rows, (long long)batches, (long long)ld);
    return DIONW_ERR_CUDA;
  }
  return DIONW_OK;
}

constexpr int kMaxDevices = 64;

// Ordinal of the current device, clamped into the per-device tables.
int current_device() {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) device = 0;
  return device;
}

template <typename InT, typename OutT, bool kBMajorMN, bool kSym>
int launch(const CUtensorMap& map_a, const CUtensorMap& map_b, const gemm::Params& p, cudaStream_t stream) {
  auto kernel = gemm::gemm_kernel<InT, OutT, kBMajorMN, kSym>;
  static std::atomic<bool> configured[kMaxDevices];   // the attribute is per device
  const int device = current_device();
  if (!configured[device].load(std::memory_order_acquire)) {
    DIONW_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm::kSmemBytes)));
    configured[device].store(true, std::memory_order_release);
  }
  const int total = p.tiles_per_batch * p.batches;
  if (total == 0) return DIONW_OK;
  const int grid = total < sm_count() ? total : sm_count();
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(grid));
  config.blockDim = dim3(gemm::kThreads);
  config.dynamicSmemBytes = gemm::kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = use_dependent_launch() ? 1 : 0;
  count_launch();
  return check_cuda(cudaLaunchKernelEx(&config, kernel, map_a, map_b, p), "gemm_kernel launch");
}

// ---- tile counters of the two-CTA kernel's dynamic hand-out ------------------------------------
// One {next tile, pairs done} pair per (device, stream) that has launched a product with the dynamic
// hand-out: launches of one stream run one after the other and each leaves its counters at zero,
// launches of different streams may overlap and must not share.  The counters live in the library's
// device image (zero at load); their address on a device is looked up once.
constexpr int kCounterSlots = 1024;
__device__ int g_tile_counters[kCounterSlots][2];

std::mutex g_counter_mutex;
std::map<std::pair<int, cudaStream_t>, int> g_counter_slot;   // guarded by g_counter_mutex
int g_counter_next[kMaxDevices];                              // guarded by g_counter_mutex
int* g_counter_base[kMaxDevices];                             // guarded by g_counter_mutex

// Process-wide switch (dionw_gemm_dynamic_tiles): off by default.  A product launched with it on
// draws its tiles from a counter; see gemm2_sm100.cuh.
std::atomic<int> g_dynamic_tiles{-1};

bool use_dynamic_tiles() {
  int mode = g_dynamic_tiles.load(std::memory_order_relaxed);
  if (mode < 0) {
    const char* v = std::getenv("DIONW_GEMM_DYNAMIC_TILES");
    mode = (v != nullptr && v[0] == '1') ? 1 : 0;
    g_dynamic_tiles.store(mode, std::memory_order_relaxed);
  }
  return mode != 0;
}

// The counters of `stream` on the current device, or null when they cannot be had (the product then
// takes its tiles in the fixed stride).
int* tile_counters(cudaStream_t stream) {
  const int device = current_device();
  std::lock_guard<std::mutex> lock(g_counter_mutex);
  if (g_counter_base[device] == nullptr) {
    void* address = nullptr;
    if (cudaGetSymbolAddress(&address, g_tile_counters) != cudaSuccess) return nullptr;
    g_counter_base[device] = static_cast<int*>(address);
  }
  const auto key = std::make_pair(device, stream);
  auto found = g_counter_slot.find(key);
  if (found == g_counter_slot.end()) {
    if (g_counter_next[device] >= kCounterSlots) return nullptr;
    found = g_counter_slot.emplace(key, g_counter_next[device]++).first;
  }
  return g_counter_base[device] + 2 * found->second;
}

// The streaming job (decay_job.cuh) that products launched by this thread carry, or null.
thread_local DecayJob* t_side_job = nullptr;

// Two-CTA tiles (clusters of two CTAs) unless the environment says DIONW_GEMM_CTA_PAIRS=0,
// which selects the one-CTA kernel.
bool use_cta_pairs() {
  static const bool on = [] {
    const char* v = std::getenv("DIONW_GEMM_CTA_PAIRS");
    return v == nullptr || v[0] != '0';
  }();
  return on;
}

// Runs a filled plan as clusters of two CTAs.
template <typename InT, int kMaps, int kSteps>
int launch_plan(const gemm2::Plan<kMaps, kSteps>& plan, cudaStream_t stream) {
  static_assert(sizeof(plan) <= 32764, "kernel parameters are limited to 32764 bytes");
  auto kernel = gemm2::gemm2_kernel<InT, kMaps, kSteps>;
  static std::atomic<bool> configured[kMaxDevices];   // the attribute is per device
  const int device = current_device();
  if (!configured[device].load(std::memory_order_acquire)) {
    DIONW_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm2::kSmemBytes)));
    configured[device].store(true, std::memory_order_release);
  }
  const int pairs_max = sm_count() / 2;
  const int pairs = plan.total_tiles < pairs_max ? plan.total_tiles : pairs_max;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(2 * pairs));
  config.blockDim = dim3(gemm2::kThreads);
  config.dynamicSmemBytes = gemm2::kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  // A plan of several products follows the clearing of its counters, which is no kernel.
  config.numAttrs = kSteps == 1 && use_dependent_launch() ? 2 : 1;
  count_launch();
  return check_cuda(cudaLaunchKernelEx(&config, kernel, plan), "gemm2_kernel launch");
}

// The epilogue's side of a product; the tile counts are the caller's.
gemm::Params params_of(const Product& product) {
  gemm::Params p{};
  p.cin = product.cin.base;
  p.out = const_cast<void*>(product.out.base);
  p.out2 = product.out2;
  p.ldc = product.cin.ld;
  p.ldo = product.out.ld;
  p.cin_batch = product.cin.batch;
  p.out_batch = product.out.batch;
  p.alpha = product.alpha;
  p.beta = product.beta;
  p.diag = product.diag;
  p.m = int(product.m);
  p.n = int(product.n);
  p.kdim = int(product.k);
  p.batches = int(product.blocks);
  p.mirror_diagonal = product.same_operands ? 0 : 1;
  p.lower_only = 0;
  p.rowsq = product.rowsq;
  p.rowsq_parts = int(2 * ((product.n + gemm::kBN - 1) / gemm::kBN));
  p.status = device_status_word();
  p.wait_ns = gemm::kWaitLimitNs;
  return p;
}

// Operand A is stored [m, k] (or [k, m]: a_mn), B is stored [n, k] (or [k, n]: b_mn).
int operand_map(CUtensorMap* map, const Operand& x, int dtype, bool mn, int64_t outer, int64_t k, int64_t blocks,
                uint32_t box_outer) {
  if (mn) return make_map(map, x.base, dtype, outer, k, blocks, x.ld, x.batch, 64, gemm::kBK);
  return make_map(map, x.base, dtype, k, outer, blocks, x.ld, x.batch, gemm::kBK, box_outer);
}

int run_one_cta(const Product& product, int dtype, cudaStream_t stream) {
  const int64_t blocks = product.blocks;
  CUtensorMap map_a, map_b;
  int st = operand_map(&map_a, product.a, dtype, product.a_mn, product.m, product.k, blocks, gemm::kBM);
  if (st != DIONW_OK) return st;
  st = operand_map(&map_b, product.b, dtype, product.b_mn, product.n, product.k, blocks, gemm::kBN);
  if (st != DIONW_OK) return st;
  gemm::Params p = params_of(product);
  p.tiles_m = (p.m + gemm::kBM - 1) / gemm::kBM;
  p.tiles_n = (p.n + gemm::kBN - 1) / gemm::kBN;
  const int q = p.tiles_m / 2;
  p.tiles_per_batch = product.symmetric ? q * (q + 1) + ((p.tiles_m & 1) ? q + 1 : 0) : p.tiles_m * p.tiles_n;
  const bool f16 = dtype == DIONW_F16, same = product.out_dtype == dtype;
  if (product.symmetric) {
    if (product.b_mn)
      return f16 ? launch<__half, __half, true, true>(map_a, map_b, p, stream)
                 : launch<__nv_bfloat16, __nv_bfloat16, true, true>(map_a, map_b, p, stream);
    return f16 ? launch<__half, __half, false, true>(map_a, map_b, p, stream)
               : launch<__nv_bfloat16, __nv_bfloat16, false, true>(map_a, map_b, p, stream);
  }
  if (product.b_mn) {
    if (f16 && same) return launch<__half, __half, true, false>(map_a, map_b, p, stream);
    if (f16) return launch<__half, __nv_bfloat16, true, false>(map_a, map_b, p, stream);
    return launch<__nv_bfloat16, __nv_bfloat16, true, false>(map_a, map_b, p, stream);
  }
  if (f16 && same) return launch<__half, __half, false, false>(map_a, map_b, p, stream);
  if (f16) return launch<__half, __nv_bfloat16, false, false>(map_a, map_b, p, stream);
  return launch<__nv_bfloat16, __nv_bfloat16, false, false>(map_a, map_b, p, stream);
}

// Tiles of 256 x 256.
int64_t wide_tiles(const Product& product) {
  const int64_t tm = (product.m + gemm2::kPairM - 1) / gemm2::kPairM, tn = (product.n + gemm2::kBN - 1) / gemm2::kBN;
  return product.blocks * (product.symmetric ? tm * (tm + 1) / 2 : tm * tn);
}

// Width of the tiles of a product that runs beside products of `tiles` 256-wide tiles in all (its own
// among them).  256 columns are the better use of the memory system (a k-block of a 256 x 256 tile brings
// 32 KB into each SM, one of two 256 x 128 tiles 24 KB each), so they are taken wherever they fill the GPU.
// Where they would leave half of the SM pairs without a tile, twice as many pairs with half the columns each
// finish sooner: main loop and epilogue are then half as long.  Row sums come in parts of 128 columns per
// warp: 256-wide tiles.  In a chain, 128 against 256 columns: 1 block of 256^3 with Cin 7.1 against 8.0 us,
// with two outputs 8.1 against 10.7; 1 block of 2048^3 18.0 against 26.5 us.
int tile_width(const Product& product, int64_t tiles) {
  if (product.rowsq != nullptr) return gemm2::kBN;
  if (product.n <= gemm2::kBN / 2) return gemm2::kBN / 2;
  return 2 * tiles <= sm_count() / 2 ? gemm2::kBN / 2 : gemm2::kBN;
}

// Tiles on and below the diagonal of an n x n product (gemm2::sym_tile): tile row i holds those up to its own
// end.  The last 128-wide one of the last row lies past the matrix where the row's first 128 columns hold it
// all: for n up to 128 it was every second tile (1000 blocks of 64^2: an iteration of 15 products 1016 us with it, 691 without).
int symmetric_tiles(int64_t n, int tile_n) {
  const int64_t rows = (n + gemm2::kPairM - 1) / gemm2::kPairM, per_row = gemm2::kBN / tile_n;
  const int64_t tiles = per_row * (rows * (rows + 1) / 2);
  return int(n <= rows * gemm2::kPairM - tile_n ? tiles - 1 : tiles);
}

// Fills a plan with `count` products.  `counters` (device memory, see plan_counter_bytes) is needed for more
// than one; a single product draws its tiles from the stream's own counters when that is switched on.
template <typename InT, int kMaps, int kSteps>
int run_plan(const Product* const* products, int count, int dtype, unsigned* counters, cudaStream_t stream) {
  gemm2::Plan<kMaps, kSteps> plan;
  struct Mapped {
    Operand x;
    int64_t inner, rows;
    uint32_t box;
  } mapped[kMaps];
  int maps = 0;
  int64_t tiles = 0;
  int64_t matrices = 0;
  uint64_t done[kMaxChains] = {}, need[kMaxChains] = {};   // reports of a matrix: by the products so far; before this one
  for (int i = 0; i < count; ++i) {
    const Product& product = *products[i];
    const int64_t blocks = product.blocks;
    // the products that run at the same time: the neighbours at the same position of other chains
    int64_t together = 0;
    for (int j = i; j >= 0 && (j == i || products[j]->chain < products[j + 1]->chain); --j) together += wide_tiles(*products[j]);
    for (int j = i + 1; j < count && products[j]->chain > products[j - 1]->chain; ++j) together += wide_tiles(*products[j]);
    gemm2::Step& step = plan.steps[i];
    // One map serves an operand in several products: the dimensions are those of memory, and boxes of 64
    // rows suit both an MN-major operand and the half of B that a CTA loads of a 128-wide tile.
    auto map_of = [&](const Operand& x, bool mn, int64_t outer, uint32_t box, short* index) {
      const int64_t inner = mn ? outer : product.k, rows = mn ? product.k : outer;
      for (int j = 0; j < maps; ++j)
        if (mapped[j].x.base == x.base && mapped[j].x.ld == x.ld && mapped[j].x.batch == x.batch &&
            mapped[j].inner == inner && mapped[j].rows == rows && mapped[j].box == box) {
          *index = short(j);
          return int(DIONW_OK);
        }
      if (maps == kMaps) {
        set_error("a plan of %d products needs more than %d tensor maps", count, kMaps);
        return int(DIONW_ERR_UNSUPPORTED);
      }
      const int st = operand_map(&plan.maps[maps], x, dtype, mn, outer, product.k, blocks, box);
      if (st != DIONW_OK) return st;
      mapped[maps] = {x, inner, rows, box};
      *index = short(maps++);
      return int(DIONW_OK);
    };
    step.tile_n = short(tile_width(product, together));
    int st = map_of(product.a, product.a_mn, product.m, product.a_mn ? 64 : gemm2::kBM, &step.map_a);
    if (st != DIONW_OK) return st;
    st = map_of(product.b, product.b_mn, product.n, product.b_mn ? 64 : step.tile_n / 2, &step.map_b);
    if (st != DIONW_OK) return st;
    if (product.a_lower) st = map_of(product.a, true, product.m, 64, &step.map_a_t);
    if (st != DIONW_OK) return st;
    if (product.b_lower) st = map_of(product.b, true, product.n, 64, &step.map_b_t);
    if (st != DIONW_OK) return st;
    DIONW_REQUIRE((!product.a_lower || (!product.a_mn && product.m == product.k)) &&
                      (!product.b_lower || (!product.b_mn && product.n == product.k)),
                  "a lower operand is square and read in rows");
    step.p = params_of(product);
    step.p.lower_only = product.out_lower ? 1 : 0;
    step.p.tiles_m = (step.p.m + gemm2::kPairM - 1) / gemm2::kPairM;
    step.p.tiles_n = (step.p.n + step.tile_n - 1) / step.tile_n;
    step.p.tiles_per_batch = product.symmetric ? symmetric_tiles(product.n, step.tile_n) : step.p.tiles_m * step.p.tiles_n;
    step.symmetric = product.symmetric;
    step.a_major_mn = product.a_mn;
    step.b_major_mn = product.b_mn;
    step.a_lower = product.a_lower;
    step.b_lower = product.b_lower;
    step.same_operands = product.symmetric && product.same_operands;
    step.out_bf16 = product.out_dtype == DIONW_BF16;
    if (!product.beside_previous) need[product.chain] = done[product.chain];
    done[product.chain] += uint64_t(step.p.tiles_per_batch) * gemm2::kReportsPerTile;
    step.need = unsigned(need[product.chain]);
    step.progress = counters != nullptr ? counters + 2 + product.first_block : nullptr;
    if (product.first_block + blocks > matrices) matrices = product.first_block + blocks;
    step.first_tile = int(tiles);
    tiles += int64_t(step.p.tiles_per_batch) * blocks;
    DIONW_REQUIRE(tiles < (1LL << 31) && done[product.chain] < (1ULL << 32), "the products of one launch have too many tiles");
  }
  for (int i = maps; i < kMaps; ++i) plan.maps[i] = plan.maps[0];   // every map is prefetched
  if (tiles == 0) return DIONW_OK;
  plan.count = count;
  plan.total_tiles = int(tiles);
  plan.job = t_side_job;
  plan.status = device_status_word();
  plan.wait_ns = gemm::kWaitLimitNs;
  if (count > 1) {
    plan.tile_counter = reinterpret_cast<int*>(counters);
    DIONW_CUDA(cudaMemsetAsync(counters, 0, plan_counter_bytes(matrices), stream));
  } else {
    // Tiles from a counter only where a pair takes more than one: a one-wave product gains nothing
    // from it and would pay the hand-out's latency on its critical path.
    plan.tile_counter = (use_dynamic_tiles() && tiles > sm_count() / 2) ? tile_counters(stream) : nullptr;
  }
  return launch_plan<InT>(plan, stream);
}

}  // namespace

size_t plan_counter_bytes(int64_t blocks) { return blocks <= kMaxPlanBlocks ? size_t(blocks + 2) * sizeof(unsigned) : 0; }

int run_products(const Product* products, int count, int dtype, void* counters, cudaStream_t stream) {
  const bool f16 = dtype == DIONW_F16;
  // position in the chain first, then the chain
  const Product* ordered[kMaxChains * kMaxChainProducts];
  int position[kMaxChains * kMaxChainProducts], seen[kMaxChains] = {};
  int64_t matrices = 0;
  int chains = 0;
  DIONW_REQUIRE(count <= kMaxChains * kMaxChainProducts, "products: too many in one call");
  for (int i = 0; i < count; ++i) {
    DIONW_REQUIRE(products[i].blocks > 0, "products: empty batch");
    position[i] = seen[products[i].chain]++;
    matrices = std::max(matrices, products[i].first_block + products[i].blocks);
    chains = std::max(chains, products[i].chain + 1);
  }
  int n = 0;
  for (int level = 0; level < kMaxChainProducts; ++level)
    for (int i = 0; i < count; ++i)
      if (position[i] == level) ordered[n++] = products + i;
  DIONW_REQUIRE(n == count, "products: a chain is too long");
  if (use_cta_pairs() && count > 1 && matrices <= kMaxPlanBlocks && counters != nullptr) {
    unsigned* c = static_cast<unsigned*>(counters);
    constexpr int kMaps = kMaxChainMaps, kSteps = kMaxChainProducts;
    if (chains == 1)
      return f16 ? run_plan<__half, kMaps, kSteps>(ordered, count, dtype, c, stream)
                 : run_plan<__nv_bfloat16, kMaps, kSteps>(ordered, count, dtype, c, stream);
    return f16 ? run_plan<__half, kMaxChains * kMaps, kMaxChains * kSteps>(ordered, count, dtype, c, stream)
               : run_plan<__nv_bfloat16, kMaxChains * kMaps, kMaxChains * kSteps>(ordered, count, dtype, c, stream);
  }
  for (int i = 0; i < count; ++i) {
    int st;
    if (!use_cta_pairs()) st = run_one_cta(products[i], dtype, stream);
    else if (f16) st = run_plan<__half, 4, 1>(ordered + i, 1, dtype, nullptr, stream);
    else st = run_plan<__nv_bfloat16, 4, 1>(ordered + i, 1, dtype, nullptr, stream);
    if (st != DIONW_OK) return st;
  }
  return DIONW_OK;
}

namespace {

// Clusters of `pairs` SM pairs that the current device runs at a time, 0 where it cannot be told (asked again then).
int onchip_clusters(int pairs) {
  static std::atomic<int> known[kMaxDevices][onchip::kMaxPairs + 1];   // + 1; zero: not known yet
  std::atomic<int>& slot = known[current_device()][pairs];
  int value = slot.load(std::memory_order_acquire);
  if (value != 0) return value - 1;
  int clusters = 0;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(2 * pairs));
  config.blockDim = dim3(onchip::kThreads);
  config.dynamicSmemBytes = onchip::kSmemBytes;
  cudaLaunchAttribute attribute;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = unsigned(2 * pairs);
  attribute.val.clusterDim.y = 1;
  attribute.val.clusterDim.z = 1;
  config.attrs = &attribute;
  config.numAttrs = 1;
  if (cudaFuncSetAttribute(onchip::iteration_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(onchip::kSmemBytes)) != cudaSuccess ||
      cudaFuncSetAttribute(onchip::iteration_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&clusters, onchip::iteration_kernel, &config) != cudaSuccess) {
    cudaGetLastError();   // not an error of the call: the plan takes the batch
    return 0;
  }
  slot.store(clusters + 1, std::memory_order_release);
  return clusters;
}

// As many pairs to a matrix as it has column blocks, while all clusters run at the same time.
int pairs_per_matrix(int64_t blocks, int64_t tiles) {
  for (int pairs = int(std::min<int64_t>(tiles, onchip::kMaxPairs)); pairs > 1; --pairs)
    if (blocks <= onchip_clusters(pairs)) return pairs;
  return 1;
}

}  // namespace

// On chip a chain of products takes 14 x 2.8 us (m = 256) whatever the rest of the GPU does, but every pair sums the whole
// Gram matrix (0.27 us per 64 columns of n, twice) and a batch takes whole waves of clusters.  Iteration as a plan against on
// chip, us, m = 256: 1 block of n = 1024 105 and 69, 4096 126 and 102, 6144 140 and 125; 37 blocks of 1024 129 and 83, 4096
// 189 and 162; 74 blocks (one wave) 178 and 91, 310 and 223; 160 (two and a bit) of 1024 303 and 257.  m = 96: 1 block of 1024
// 82 and 42; 160 of 1024 190 and 155.  The lines were drawn where, with four pairs to a matrix, the two met; with eight it is
// still ahead behind them: 1 block of 8192 154 and 147, 74 of 8192 529 and 425, 160 of 2048 418 and 340.
constexpr int64_t kOnChipColumns = 6144, kOnChipColumnsInWaves = 1024;

int on_chip_pairs(int64_t blocks, int64_t m, int64_t n) {
  if (!use_cta_pairs() || m > onchip::kSide) return 0;
  const int wave = onchip_clusters(1);
  if (wave <= 0 || n > (blocks <= wave ? kOnChipColumns : kOnChipColumnsInWaves)) return 0;
  return pairs_per_matrix(blocks, (n + onchip::kSide - 1) / onchip::kSide);
}

int run_on_chip(const Product* list, const int* chain_length, const ChainSlot* slots, int n_slots, bool tall, int pairs,
                cudaStream_t stream) {
  auto slot_of = [&](const void* base) -> int {
    for (int i = 0; i < n_slots; ++i)
      if (slots[i].base == base) return slots[i].slot;
    return -1;
  };
  onchip::Iteration it{};
  const int64_t blocks = list[0].blocks, m = list[0].m, n = list[0].k;
  it.tall = tall;
  it.m = int(m);
  it.n = int(n);
  it.status = device_status_word();
  it.wait_ns = gemm::kWaitLimitNs;
  for (int part = 0; part < 2; ++part) {
    const Product& gram = *list++;
    const int64_t cols = tall ? m : n, rows = tall ? n : m;
    const uint32_t boxes[2] = {uint32_t(onchip::kRows), 64};
    for (int box = 0; box < 2; ++box) {
      const int st = make_map(&it.x[part][box], gram.a.base, DIONW_F16, cols, rows, blocks, gram.a.ld, gram.a.batch, 64, boxes[box]);
      if (st != DIONW_OK) return st;
    }
    it.count[part] = 1 + chain_length[part];
    DIONW_REQUIRE(it.count[part] <= onchip::kMaxOps, "a chain has at most %d products", onchip::kMaxOps - 1);
    it.ops[part][0] = {-1, -1, -1, 0, -1, gram.alpha, 0.0f, 0.0f};
    DIONW_REQUIRE(slot_of(gram.out.base) == 0, "the Gram matrix is the first slot's");
    for (int i = 1; i < it.count[part]; ++i) {
      const Product& p = *list++;
      onchip::Op& op = it.ops[part][i];
      op.a = int8_t(slot_of(p.a.base));
      op.b = int8_t(slot_of(p.b.base));
      op.cin = int8_t(slot_of(p.cin.base));
      op.out = int8_t(slot_of(p.out.base));
      op.out2 = int8_t(p.out2 != nullptr ? slot_of(p.out2) : -1);
      op.alpha = p.alpha;
      op.beta = p.beta;
      op.diag = p.diag;
      DIONW_REQUIRE(p.symmetric && p.m == m && p.n == m && p.k == m && op.a >= 0 && op.b >= 0 && op.cin >= 0 && op.out >= 0 &&
                        (p.out2 == nullptr || op.out2 >= 0),
                    "a chain is of symmetric products of one size on known matrices");
    }
    const Product& result = *list++;
    DIONW_REQUIRE(slot_of(tall ? result.b.base : result.a.base) == 2, "Q is the third slot's");
    // X is loaded over the other two as soon as the chain's last product has been summed, while its epilogue still runs.
    const onchip::Op& last = it.ops[part][it.count[part] - 1];
    DIONW_REQUIRE(last.out == 2 && (last.cin == 2 || last.cin == -1) && (last.out2 == 2 || last.out2 == -1),
                  "the epilogue of a chain's last product keeps to the third slot");
    it.result[part] = params_of(result);
    it.result_bf16[part] = result.out_dtype == DIONW_BF16;
  }
  it.pairs = pairs;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(unsigned(2 * it.pairs * blocks));
  config.blockDim = dim3(onchip::kThreads);
  config.dynamicSmemBytes = onchip::kSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = unsigned(2 * it.pairs);
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = use_dependent_launch() ? 2 : 1;
  count_launch();
  return check_cuda(cudaLaunchKernelEx(&config, onchip::iteration_kernel, it), "iteration_kernel launch");
}

}  // namespace dionw

extern "C" int dionw_symmetric_product(const void* a, const void* b, int64_t blocks, int64_t m, int64_t kdim,
                                       int64_t lda, int64_t ldb, const void* cin, int64_t ldc, float alpha,
                                       float beta, void* out, int64_t ldo, void* out2, float diag, int dtype,
                                       void* stream) {
  using namespace dionw;
  DIONW_REQUIRE(dtype == DIONW_F16 || dtype == DIONW_BF16, "symmetric_product: dtype must be F16 or BF16");
  DIONW_REQUIRE(blocks > 0 && m > 0 && kdim > 0, "symmetric_product: empty problem");
  Product product;
  product.a = {a, lda, m * lda};
  product.same_operands = b == nullptr || b == a;
  product.b = b == nullptr ? product.a : Operand{b, ldb, m * ldb};
  product.symmetric = true;
  product.cin = {cin, ldc, m * ldc};
  product.alpha = alpha;
  product.beta = beta;
  product.out = {out, ldo, m * ldo};
  product.out2 = out2;
  product.diag = diag;
  product.m = product.n = m;
  product.k = kdim;
  product.out_dtype = dtype;
  product.blocks = blocks;
  return run_products(&product, 1, dtype, nullptr, static_cast<cudaStream_t>(stream));
}

extern "C" int dionw_batched_gemm(const void* a, int64_t lda, const void* b, int64_t ldb, int b_is_nk,
                                  const void* cin, int64_t ldc, float beta, void* out, int64_t ldo, int64_t blocks,
                                  int64_t m, int64_t n, int64_t kdim, int in_dtype, int out_dtype, void* stream) {
  using namespace dionw;
  DIONW_REQUIRE(in_dtype == DIONW_F16 || in_dtype == DIONW_BF16, "batched_gemm: input dtype must be F16 or BF16");
  DIONW_REQUIRE(out_dtype == DIONW_F16 || out_dtype == DIONW_BF16, "batched_gemm: output dtype must be F16 or BF16");
  DIONW_REQUIRE(blocks > 0 && m > 0 && n > 0 && kdim > 0, "batched_gemm: empty problem");
  if (in_dtype == DIONW_BF16 && out_dtype != DIONW_BF16) {
    set_error("batched_gemm: bf16 inputs with an fp16 output are not supported");
    return DIONW_ERR_UNSUPPORTED;
  }
  Product product;
  product.a = {a, lda, m * lda};
  product.b = {b, ldb, (b_is_nk ? n : kdim) * ldb};
  product.b_mn = b_is_nk == 0;
  product.cin = {cin, ldc, m * ldc};
  product.beta = beta;
  product.out = {out, ldo, m * ldo};
  product.m = m;
  product.n = n;
  product.k = kdim;
  product.out_dtype = out_dtype;
  product.blocks = blocks;
  return run_products(&product, 1, in_dtype, nullptr, static_cast<cudaStream_t>(stream));
}

namespace dionw {
// After a wait that ran out a product may have left its tile counters in any state: put them back to
// zero on the current device (called by dionw_check_device when it reports a failure).
void reset_tile_counters() {
  void* address = nullptr;
  if (cudaGetSymbolAddress(&address, g_tile_counters) == cudaSuccess)
    cudaMemset(address, 0, sizeof(int) * 2 * kCounterSlots);
}
}  // namespace dionw

extern "C" void dionw_gemm_side_job(void* job) { dionw::t_side_job = static_cast<dionw::DecayJob*>(job); }

extern "C" int dionw_gemm_dynamic_tiles(int on) {
  const int before = dionw::use_dynamic_tiles() ? 1 : 0;
  if (on >= 0) dionw::g_dynamic_tiles.store(on != 0 ? 1 : 0, std::memory_order_relaxed);
  return before;
}

// ---------------------------------------------------------------------------
// Self-test of the bounded wait.  One CTA of one warp initialises an mbarrier on
// which nothing ever arrives (no TMA, no TMEM, no other CTA) and waits on it with
// the products' own mbar_wait and a limit of `limit_ns`.  The wait runs out, the
// kernel stores the wait code in the device status word and returns normally: the
// context stays usable and the host reads the code with dionw_check_device().
// ---------------------------------------------------------------------------
namespace dionw {
namespace {

__global__ void __launch_bounds__(32)
wait_selftest_kernel(int* status, uint64_t limit_ns, int* gave_up) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    gemm::mbar_init(&bar, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    const bool ok = gemm::mbar_wait(&bar, 0u, &abort_flag, status, limit_ns);
    if (gave_up != nullptr) *gave_up = ok ? 0 : 1;
  }
}

}  // namespace
}  // namespace dionw

extern "C" int dionw_selftest_wait_timeout(int64_t limit_us, int* gave_up, void* stream) {
  using namespace dionw;
  DIONW_REQUIRE(limit_us > 0 && limit_us <= 100000, "selftest_wait_timeout: the limit must be 1 .. 100000 us (got %lld)",
                (long long)limit_us);
  wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(device_status_word(),
                                                                        uint64_t(limit_us) * 1000ull, gave_up);
  return launch_status("wait_selftest_kernel");
}
