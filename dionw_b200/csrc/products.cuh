// Batched tensor-core products as the host describes them (gemm.cu runs them).
#pragma once

#include "common.cuh"

namespace dionw {

// A batch of row-major 2-byte matrices; strides in elements.
struct Operand {
  const void* base = nullptr;
  int64_t ld = 0;
  int64_t batch = 0;
};

// out = alpha A B + beta Cin, [m, n], reduced over k.
struct Product {
  Operand a, b;                  // A stored [m, k]; B stored [n, k]
  bool a_mn = false;             // A stored [k, m] (symmetric products of one operand only: A^T A)
  bool b_mn = false;             // B stored [k, n]
  bool symmetric = false;        // known to be symmetric: lower tiles + mirror
  // An operand or the result is symmetric and only its 256 x 256 blocks up to the diagonal are stored.  (The
  // one-CTA kernel stores mirror images everywhere and reads whole matrices.)
  bool a_lower = false, b_lower = false, out_lower = false;
  bool same_operands = false;    // symmetric: A and B are the same matrix, so diagonal tiles come out symmetric
  Operand cin;                   // base null: no second term
  float alpha = 1.0f, beta = 0.0f;
  Operand out;
  void* out2 = nullptr;          // symmetric: out + diag on the diagonal
  float diag = 0.0f;
  int64_t m = 0, n = 0, k = 0;
  int out_dtype = DIONW_F16;
  float* rowsq = nullptr;        // general: [blocks, m, 2 * ceil(n / 256)] partial row sums of out^2
  bool beside_previous = false;  // reads nothing that the product of its chain before it writes (nor writes what it reads)
  int64_t blocks = 0;            // matrices of the batch
  // A chain is a sequence of products on one batch, each of which may read what the ones before it wrote.
  // Products of different chains have nothing to do with one another.
  int chain = 0;
  int64_t first_block = 0;       // matrices of the chains before this one
};

// What runs as one launch: chains, products and tensor maps (two box sizes of seven operands) of a chain, and
// matrices in all.
constexpr int kMaxChains = 6;
constexpr int kMaxChainProducts = 18;
constexpr int kMaxChainMaps = 14;
constexpr int64_t kMaxPlanBlocks = 16384;
// Device memory that run_products uses to hand out tiles; 0 for batches that run product by product.
size_t plan_counter_bytes(int64_t blocks);

// Runs the products, of one or several chains, in an order that keeps every chain's own.  One launch when
// `counters` (plan_counter_bytes of all chains' matrices, 4-byte aligned) is given and the limits hold.
int run_products(const Product* products, int count, int dtype, void* counters, cudaStream_t stream);

// The Gram schedule of a batch on chip (onchip_sm100.cuh): X X^T, a chain of fp16 symmetric products, Q X, twice.
// Each m x m matrix is in one of three places; several may share a place where the one is no longer read when the
// other is written.
struct ChainSlot {
  const void* base;
  int slot;
};
// SM pairs to a matrix on the current device where that is the faster way; 0 where it is not.
int on_chip_pairs(int64_t blocks, int64_t m, int64_t n);
int run_on_chip(const Product* list, const int* chain_length, const ChainSlot* slots, int n_slots, bool tall, int pairs,
                cudaStream_t stream);

}  // namespace dionw
