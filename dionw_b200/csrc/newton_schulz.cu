// The Newton-Schulz product schedules: which products, in which order.  gemm.cu runs them, all of one
// iteration as one launch.
#include <algorithm>

#include "products.cuh"

namespace dionw {
namespace {

struct Coeff {
  double a, b, c;
};

// Polar Express coefficients divided by the safety factor 1.05, 1.05^3, 1.05^5:
// the table the reference's Gram iteration uses.
constexpr double kS = 1.05;
const Coeff kGram[5] = {
    {8.28721201814563 / kS, -23.595886519098837 / (kS * kS * kS), 17.300387312530933 / (kS * kS * kS * kS * kS)},
    {4.107059111542203 / kS, -2.9478499167379106 / (kS * kS * kS), 0.5448431082926601 / (kS * kS * kS * kS * kS)},
    {3.9486908534822946 / kS, -2.908902115962949 / (kS * kS * kS), 0.5518191394370137 / (kS * kS * kS * kS * kS)},
    {3.3184196573706015 / kS, -2.488488024314874 / (kS * kS * kS), 0.51004894012372 / (kS * kS * kS * kS * kS)},
    {2.300652019954817 / kS, -1.6689039845747493 / (kS * kS * kS), 0.4188073119525673 / (kS * kS * kS * kS * kS)},
};
const Coeff kPolarExpress[5] = {
    {8.156554524902461, -22.48329292557795, 15.878769915207462},
    {4.042929935166739, -2.808917465908714, 0.5000178451051316},
    {3.8916678022926607, -2.772484153217685, 0.5060648178503393},
    {3.285753657755655, -2.3681294933425376, 0.46449024233003106},
    {2.3465413258596377, -1.7097828382687081, 0.42323551169305323},
};
const Coeff kKeller[5] = {
    {3.4445, -4.7750, 2.0315}, {3.4445, -4.7750, 2.0315}, {3.4445, -4.7750, 2.0315},
    {3.4445, -4.7750, 2.0315}, {3.4445, -4.7750, 2.0315},
};
constexpr int kRestart = 2;

inline int64_t round_up(int64_t v, int64_t to) { return (v + to - 1) / to * to; }
inline size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// A block is rows x cols as it lies in memory; m is its shorter side, n its longer one.
struct Layout {
  int64_t m, n;
  int64_t ldg;          // leading dimension of the m x m scratch matrices
  size_t x_bytes;       // one [blocks, rows, ldx] operand
  size_t g_bytes;       // one [blocks, m, ldg] matrix
  bool gram;            // the iteration on the Gram matrix (blocks that are not square)
};

Layout layout_of(int64_t blocks, int64_t rows, int64_t cols, int64_t ldx, int kind) {
  Layout l;
  l.m = rows < cols ? rows : cols;
  l.n = rows < cols ? cols : rows;
  l.ldg = round_up(l.m, 8);
  l.x_bytes = align256(size_t(blocks) * rows * ldx * 2);
  l.g_bytes = align256(size_t(blocks) * l.m * l.ldg * 2);
  l.gram = (kind == DIONW_NS_GRAM || kind == DIONW_NS_GRAM_FULL) && l.n > l.m;
  return l;
}

size_t bytes_of(const Layout& l) {
  // Gram iteration: X1 + {G, Z, Q0, Q1, RZ}.  Standard iteration: X1, X2 + {G, P}.
  return l.gram ? l.x_bytes + 5 * l.g_bytes : 2 * l.x_bytes + 2 * l.g_bytes;
}

// A batch of rows x cols blocks and where its result goes.
struct Problem {
  void* x;
  void* out;
  int64_t blocks, rows, cols, ldx;
  int kind;
  float* rowsq;
};

// The schedule on a batch of either orientation, as it lies: appends its products to `list`.  A wide block is
// multiplied from the left (G = X X^T, X <- Q X), a tall one from the right (G = X^T X, X <- X Q): every
// matrix among G, Q and the polynomials is stored exactly symmetric, so Q serves as the K-major second
// operand of X Q as it is, and the only product that needs transposed reads is X^T X, which takes both
// operands MN-major.  Value for value the same as iterating the transposed copy of a tall block, without
// the two transposing passes, which took 102 us each on 12 blocks of 3072 x 768.
void append_products(const Problem& problem, int chain, int64_t first_block, const Layout& l, uint8_t* ws, Product* list,
                     int& count) {
  void* const x = problem.x;
  void* const out = problem.out;
  const int64_t blocks = problem.blocks, rows = problem.rows, cols = problem.cols, ldx = problem.ldx;
  const int kind = problem.kind;
  float* const rowsq = problem.rowsq;
  const bool gram = kind == DIONW_NS_GRAM || kind == DIONW_NS_GRAM_FULL;
  const int dt = gram ? DIONW_F16 : DIONW_BF16;
  // Every m x m matrix of the Gram schedule is a polynomial in one symmetric G, so the
  // products among them are symmetric too: GRAM computes their lower tiles only, GRAM_FULL
  // computes them as general products, as the reference's cuBLAS calls do.
  const bool mirror = kind == DIONW_NS_GRAM;
  // Where every m x m product is on the triangle, nothing reads past the diagonal.
  const bool lower = kind != DIONW_NS_GRAM_FULL || !l.gram;
  const bool tall = rows > cols;
  const int64_t m = l.m, n = l.n;
  const int64_t xb = rows * ldx;    // batch strides in elements
  const int64_t gb = m * l.ldg;
  const int64_t ldg = l.ldg;
  auto next_product = [&]() -> Product& {
    Product& p = list[count++];
    p.blocks = blocks;
    p.chain = chain;
    p.first_block = first_block;
    return p;
  };
  auto small = [&](const void* base) { return Operand{base, ldg, gb}; };   // an m x m matrix
  auto block = [&](const void* base) { return Operand{base, ldx, xb}; };   // a rows x cols matrix
  // to = X X^T (wide), X^T X (tall)
  auto gram_of = [&](const void* from, void* to) {
    Product& p = next_product();
    p.a = p.b = block(from);
    p.a_mn = p.b_mn = tall;
    p.symmetric = p.same_operands = true;
    p.out_lower = lower;
    p.out = small(to);
    p.m = p.n = m;
    p.k = n;
    p.out_dtype = dt;
  };
  // to = alpha A B + beta A-or-B's polynomial `cin`, all m x m and symmetric; a == b: the square of a matrix
  auto combine = [&](const void* a, const void* b, double alpha, const void* cin, double beta, void* to) -> Product& {
    Product& p = next_product();
    p.a = small(a);
    p.b = small(b);
    p.symmetric = a == b || mirror;
    p.same_operands = a == b;
    p.a_lower = p.b_lower = p.out_lower = lower;
    p.alpha = float(alpha);
    p.cin = small(cin);
    p.beta = float(beta);
    p.out = small(to);
    p.m = p.n = p.k = m;
    p.out_dtype = dt;
    return p;
  };
  // to = S from + beta from (wide), from S + beta from (tall) with a symmetric S; beta = 0: no second term
  auto multiply = [&](const void* s, const void* from, double beta, void* to, int out_dtype, float* sums) {
    Product& p = next_product();
    p.a = tall ? block(from) : small(s);
    p.b = tall ? small(s) : block(from);
    p.b_mn = !tall;
    p.a_lower = lower && !tall;
    p.b_lower = lower && tall;
    if (beta != 0.0) p.cin = block(from);
    p.beta = float(beta);
    p.out = block(to);
    p.m = rows;
    p.n = cols;
    p.k = m;
    p.out_dtype = out_dtype;
    p.rowsq = sums;
  };

  if (l.gram) {
    void* x1 = ws;
    void* g = ws + l.x_bytes;
    void* z = ws + l.x_bytes + l.g_bytes;
    void* q = ws + l.x_bytes + 2 * l.g_bytes;
    void* qnext = ws + l.x_bytes + 3 * l.g_bytes;
    void* rz = ws + l.x_bytes + 4 * l.g_bytes;
    const void* xcur = x;
    gram_of(xcur, g);
    for (int i = 0; i < 5; ++i) {
      const Coeff k = kGram[i];
      if (i == kRestart) {   // X <- Q X and its Gram matrix
        multiply(q, xcur, 0.0, x1, dt, nullptr);
        xcur = x1;
        gram_of(xcur, g);
      }
      // Z = c G G^T + b G; on a fresh start also Q = Z + a I.  The diagonal is round(fp32(Z) + fp32(a)),
      // as the reference's compiled GPU step forms `z + a * eye` (its eager CPU run rounds `a` to
      // fp16 first, which costs 4e-3 of accuracy on 256 x 4096 operands).
      const bool fresh_q = i == 0 || i == kRestart;
      Product& zp = combine(g, g, k.c, g, k.b, z);
      if (fresh_q) {
        zp.out2 = q;
        zp.diag = float(k.a);
      }
      if (!fresh_q) {
        // Q <- a Q + Q Z
        combine(q, z, 1.0, q, k.a, qnext);
        void* t = q;
        q = qnext;
        qnext = t;
      }
      if (i < 4 && i + 1 != kRestart) {
        // RZ = a G + G Z, which does not touch Q; G <- a RZ + Z RZ.  (RZ is stored exactly symmetric by the
        // mirrored products only, so the full ones read it as the [k, n] operand that it is.)
        combine(g, z, 1.0, g, k.a, rz).beside_previous = !fresh_q;
        combine(z, rz, 1.0, rz, k.a, g).b_mn = !mirror;
      }
    }
    multiply(q, xcur, 0.0, out, DIONW_BF16, rowsq);   // out = Q X
  } else {
    // Standard iteration: X <- a X + (b G + c G^2) X with G = X X^T.
    const Coeff* table = gram ? kGram : (kind == DIONW_NS_POLAR_EXPRESS ? kPolarExpress : kKeller);
    void* x1 = ws;
    void* x2 = ws + l.x_bytes;
    void* g = ws + 2 * l.x_bytes;
    void* poly = ws + 2 * l.x_bytes + l.g_bytes;
    const void* cur = x;
    for (int i = 0; i < 5; ++i) {
      const Coeff k = table[i];
      void* next = i == 4 ? out : (cur == x1 ? x2 : x1);
      gram_of(cur, g);
      combine(g, g, k.c, g, k.b, poly);
      multiply(poly, cur, k.a, next, i == 4 ? DIONW_BF16 : dt, i == 4 ? rowsq : nullptr);
      cur = next;
    }
  }
}

// A batch of blocks up to this wide on their shorter side goes product by product.  The line was drawn when a producer drew
// its own tiles and a plan of them was the slower one: 1 block of 64^2 92 us against 74, 1000 of them 691 against 588.  With
// tiles handed out ahead a plan takes 53 against 68 us (16 of 64 x 1024 83 against 111, 1000 of 64^2 500 against 513): it is
// the faster one here too.
constexpr int64_t kStepwiseSide = 64;

size_t group_bytes(const Problem* problems, int n) {
  int64_t matrices = 0;
  size_t bytes = 0;
  for (int i = 0; i < n; ++i) {
    matrices += problems[i].blocks;
    bytes += bytes_of(layout_of(problems[i].blocks, problems[i].rows, problems[i].cols, problems[i].ldx, problems[i].kind));
  }
  return bytes + align256(plan_counter_bytes(matrices));
}

// The list that append_products makes of a Gram iteration, on chip: products 1 to 5 and 8 to 16 are on m x m matrices.
int iterate_on_chip(const Product* list, int count, bool tall, int pairs, cudaStream_t stream) {
  const int lengths[2] = {5, 9};
  DIONW_REQUIRE(count == 4 + lengths[0] + lengths[1], "newton_schulz: the Gram schedule has 18 products");
  // G and RZ, Z, both Qs: RZ is written from G and G from RZ, each for the last time
  const ChainSlot slots[] = {{list[0].out.base, 0}, {list[2].out.base, 0}, {list[1].out.base, 1}, {list[1].out2, 2}, {list[5].out.base, 2}};
  return run_on_chip(list, lengths, slots, 5, tall, pairs, stream);
}

// SM pairs to a matrix with which a batch on its own is iterated on chip; 0: as a plan or product by product.
int pairs_on_chip(const Problem& p, bool stepwise) {
  if (stepwise || p.kind != DIONW_NS_GRAM || std::min(p.rows, p.cols) <= kStepwiseSide || plan_counter_bytes(p.blocks) == 0) return 0;
  const Layout l = layout_of(p.blocks, p.rows, p.cols, p.ldx, p.kind);
  return l.gram ? on_chip_pairs(p.blocks, l.m, l.n) : 0;
}

// Up to kMaxChains batches that are iterated in the same dtype, as one launch, or product by product.
int iterate(const Problem* problems, int n, bool stepwise, void* workspace, size_t workspace_bytes, cudaStream_t stream) {
  uint8_t* ws = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  const size_t lost = size_t(ws - reinterpret_cast<uint8_t*>(workspace));
  const size_t need = group_bytes(problems, n);
  if (workspace == nullptr || workspace_bytes < need + lost) {
    set_error("newton_schulz: workspace of %zu bytes is smaller than the %zu needed", workspace_bytes, need + lost);
    return DIONW_ERR_WORKSPACE;
  }
  int64_t matrices = 0;
  for (int i = 0; i < n; ++i) matrices += problems[i].blocks;
  const size_t counter_bytes = align256(plan_counter_bytes(matrices));
  const bool small = n == 1 && std::min(problems[0].rows, problems[0].cols) <= kStepwiseSide;
  void* counters = counter_bytes != 0 && !stepwise && !small ? ws : nullptr;
  ws += counter_bytes;
  Product list[kMaxChains * kMaxChainProducts];
  int count = 0;
  int64_t first_block = 0;
  for (int i = 0; i < n; ++i) {
    const Layout l = layout_of(problems[i].blocks, problems[i].rows, problems[i].cols, problems[i].ldx, problems[i].kind);
    append_products(problems[i], i, first_block, l, ws, list, count);
    ws += bytes_of(l);
    first_block += problems[i].blocks;
  }
  const bool gram = problems[0].kind == DIONW_NS_GRAM || problems[0].kind == DIONW_NS_GRAM_FULL;
  const int pairs = n == 1 ? pairs_on_chip(problems[0], stepwise) : 0;
  if (pairs > 0) return iterate_on_chip(list, count, problems[0].rows > problems[0].cols, pairs, stream);
  return run_products(list, count, gram ? DIONW_F16 : DIONW_BF16, counters, stream);
}

bool known_kind(int kind) {
  kind &= ~DIONW_NS_STEPWISE;
  return kind == DIONW_NS_GRAM || kind == DIONW_NS_POLAR_EXPRESS || kind == DIONW_NS_KELLER || kind == DIONW_NS_GRAM_FULL;
}

}  // namespace
}  // namespace dionw

namespace dionw {
// Part of dionw_newton_schulz_workspace_bytes that is not operands (newton_schulz_static.cu keeps it apart).
size_t newton_schulz_counter_bytes(int64_t blocks) { return align256(plan_counter_bytes(blocks)); }
}  // namespace dionw

extern "C" size_t dionw_newton_schulz_workspace_bytes(int64_t blocks, int64_t m, int64_t n, int kind) {
  using namespace dionw;
  if (blocks <= 0 || m <= 0 || n <= 0) return 0;
  const Problem problem{nullptr, nullptr, blocks, m, n, round_up(n, 8), kind & ~DIONW_NS_STEPWISE, nullptr};
  return group_bytes(&problem, 1) + 256;
}

extern "C" int dionw_newton_schulz_on_chip_pairs(int64_t blocks, int64_t rows, int64_t cols, int kind) {
  using namespace dionw;
  if (blocks <= 0 || rows <= 0 || cols <= 0) return 0;
  const Problem problem{nullptr, nullptr, blocks, rows, cols, round_up(cols, 8), kind & ~DIONW_NS_STEPWISE, nullptr};
  return pairs_on_chip(problem, (kind & DIONW_NS_STEPWISE) != 0);
}

extern "C" int64_t dionw_newton_schulz_rowsq_parts(int64_t n) { return n <= 0 ? 0 : 2 * ((n + 255) / 256); }

extern "C" int dionw_newton_schulz(void* x, void* out, int64_t blocks, int64_t m, int64_t n, int64_t ldx, int kind,
                                   void* workspace, size_t workspace_bytes, float* rowsq, void* stream_ptr) {
  using namespace dionw;
  DIONW_REQUIRE(known_kind(kind), "newton_schulz: unknown kind %d", kind);
  DIONW_REQUIRE(blocks > 0 && m > 0 && n >= m, "newton_schulz: needs blocks > 0 and 0 < m <= n (got %lld, %lld, %lld)",
                (long long)blocks, (long long)m, (long long)n);
  DIONW_REQUIRE(ldx >= n && ldx % 8 == 0, "newton_schulz: ldx must be >= n and a multiple of 8");
  DIONW_REQUIRE(aligned16(x) && aligned16(out), "newton_schulz: x and out must be 16-byte aligned");
  const Problem problem{x, out, blocks, m, n, ldx, kind & ~DIONW_NS_STEPWISE, rowsq};
  return iterate(&problem, 1, (kind & DIONW_NS_STEPWISE) != 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream_ptr));
}

extern "C" size_t dionw_newton_schulz_tall_workspace_bytes(int64_t blocks, int64_t rows, int64_t cols, int kind) {
  using namespace dionw;
  if (blocks <= 0 || rows <= 0 || cols <= 0) return 0;
  const Problem problem{nullptr, nullptr, blocks, rows, cols, round_up(cols, 8), kind & ~DIONW_NS_STEPWISE, nullptr};
  return group_bytes(&problem, 1) + 256;
}

extern "C" int dionw_newton_schulz_tall(void* x, void* out, int64_t blocks, int64_t rows, int64_t cols, int64_t ldx,
                                        int kind, void* workspace, size_t workspace_bytes, float* rowsq,
                                        void* stream) {
  using namespace dionw;
  DIONW_REQUIRE(known_kind(kind), "newton_schulz_tall: unknown kind %d", kind);
  DIONW_REQUIRE(blocks > 0 && cols > 0 && rows > cols,
                "newton_schulz_tall: needs blocks > 0 and 0 < cols < rows (got %lld, %lld, %lld)", (long long)blocks,
                (long long)rows, (long long)cols);
  DIONW_REQUIRE(ldx >= cols && ldx % 8 == 0, "newton_schulz_tall: ldx must be >= cols and a multiple of 8");
  DIONW_REQUIRE(aligned16(x) && aligned16(out), "newton_schulz_tall: x and out must be 16-byte aligned");
  const Problem problem{x, out, blocks, rows, cols, ldx, kind & ~DIONW_NS_STEPWISE, rowsq};
  return iterate(&problem, 1, (kind & DIONW_NS_STEPWISE) != 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

namespace dionw {
namespace {
// Fills `problems`; the message says what is wrong with a bad group.
int read_group(int n, const int64_t* blocks, const int64_t* rows, const int64_t* cols, const int* kinds, Problem* problems) {
  DIONW_REQUIRE(n >= 1 && n <= kMaxChains, "newton_schulz_group: takes 1 to %d batches (got %d)", kMaxChains, n);
  auto is_gram = [](int kind) { return kind == DIONW_NS_GRAM || kind == DIONW_NS_GRAM_FULL; };
  for (int i = 0; i < n; ++i) {
    DIONW_REQUIRE(known_kind(kinds[i]) && (kinds[i] & DIONW_NS_STEPWISE) == 0, "newton_schulz_group: unknown kind %d", kinds[i]);
    DIONW_REQUIRE(is_gram(kinds[i]) == is_gram(kinds[0]), "newton_schulz_group: fp16 and bf16 iterations in one group");
    DIONW_REQUIRE(blocks[i] > 0 && rows[i] > 0 && cols[i] > 0, "newton_schulz_group: empty batch");
    problems[i] = Problem{nullptr, nullptr, blocks[i], rows[i], cols[i], round_up(cols[i], 8), kinds[i], nullptr};
  }
  return DIONW_OK;
}
}  // namespace
}  // namespace dionw

extern "C" size_t dionw_newton_schulz_group_workspace_bytes(int n, const int64_t* blocks, const int64_t* rows,
                                                            const int64_t* cols, const int* kinds) {
  using namespace dionw;
  Problem problems[kMaxChains];
  if (read_group(n, blocks, rows, cols, kinds, problems) != DIONW_OK) return 0;
  return group_bytes(problems, n) + 256;
}

extern "C" int dionw_newton_schulz_group(int n, void* const* x, void* const* out, const int64_t* blocks,
                                         const int64_t* rows, const int64_t* cols, const int* kinds, void* workspace,
                                         size_t workspace_bytes, float* const* rowsq, void* stream) {
  using namespace dionw;
  Problem problems[kMaxChains];
  const int st = read_group(n, blocks, rows, cols, kinds, problems);
  if (st != DIONW_OK) return st;
  for (int i = 0; i < n; ++i) {
    DIONW_REQUIRE(aligned16(x[i]) && aligned16(out[i]), "newton_schulz_group: x and out must be 16-byte aligned");
    problems[i].x = x[i];
    problems[i].out = out[i];
    problems[i].rowsq = rowsq != nullptr ? rowsq[i] : nullptr;
  }
  return iterate(problems, n, false, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}
