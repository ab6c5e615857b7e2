// print_schedule.cpp -- TEST INFRASTRUCTURE: csrc/mlp_schedule.h as text, for
// tests/test_network_order.py.
#include <cstdio>

#include "../../cor-model_gb300/csrc/mlp_schedule.h"

using namespace mlp;

int main() {
    printf("products %d %d\n", kFwdProducts, kProducts);
    for (int p = 0; p < kProducts; p++) printf("product %d %d %d\n", product_blocks(p), exchange_into(p), exchange_out(p));
    for (int split = 1; split <= kBlocks; split *= 2) printf("sets %d %d\n", split, a_sets(split));
    for (int split = 1; split <= kBlocks; split *= 2)
        for (int block = 0; block < kBlocks; block++) printf("owner %d %d %d\n", split, block, block_owner(split, block));
    for (int split = 1; split <= kBlocks; split *= 2)
        for (int rank = 0; rank < split; rank++)
            for (int kb = 0; kb < kBlocks; kb++)
                for (int block = 0; block < kBlocks; block++)
                    if (waits_for(split, rank, kb, block)) printf("waits %d %d %d %d\n", split, rank, kb, block);
}
