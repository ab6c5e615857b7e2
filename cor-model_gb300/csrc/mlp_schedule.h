// mlp_schedule.h -- the order of the products of the window network's row
// kernel (mlp.cu) and what each of them waits for.  Plain constant functions,
// so that tests/test_network_order.py can check on the CPU that no buffer is
// written while it may still be read.
//
// A cluster of `split` CTAs takes a tile of rows.  A hidden layer's output is
// exchanged as the four K blocks of the next product's A operand: each CTA
// computes kBlocks / split of them and copies them to its peers.  A CTA has one
// accumulator.
#pragma once

#ifdef __CUDACC__
#define MLP_HD __host__ __device__
#else
#define MLP_HD
#endif

namespace mlp {

constexpr int kBlocks = 4;   // K blocks of a hidden layer's output

// Products in order: layers 1 .. 5 forward, then back through W5^T, W4^T, W3^T, W2^T.
constexpr int kFwdProducts = 5, kProducts = 9;
MLP_HD constexpr int product_blocks(int p) { return p == 0 || p == 5 ? 1 : kBlocks; }

// The output of hidden product p (0 .. 3 forward, 5 .. 7 back) is exchange p or
// p - 1, into A buffer exchange % a_sets; the two products before and after the
// output layer read the single block that every CTA fills itself.
MLP_HD constexpr int exchange_into(int p) { return p == 0 || p == 5 ? -1 : p < 5 ? p - 1 : p - 2; }
MLP_HD constexpr int exchange_out(int p) { return p < 4 ? p : p - 1; }

// Exchanges that a CTA has room for.  Peers write theirs while this CTA may
// still read the one before; a CTA alone writes after its own product.
MLP_HD constexpr int a_sets(int split) { return split == 1 ? 1 : 2; }

MLP_HD constexpr int block_owner(int split, int block) { return block / (kBlocks / split); }

// Whether CTA `rank` waits for `block` of the exchange that product p reads
// before it issues the product's K block kb.  The block that kb reads; and
// before the first, which starts to overwrite the accumulator, this CTA's own
// blocks: its epilogue threads arrive there once they have read the product
// before out of the accumulator.  (A peer's block says nothing about that.)
MLP_HD constexpr bool waits_for(int split, int rank, int kb, int block) {
    return block == kb || (kb == 0 && block_owner(split, block) == rank);
}

}  // namespace mlp
