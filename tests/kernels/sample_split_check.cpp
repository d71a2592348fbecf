// sa_split over a loop of sampled steps, printed a line a step: rounds spans shared own
//   sample_split_check SHARED OWN_FIRST STEPS GQA SAMPLES KV_HEADS MAX_SLICES SMS
#include <cstdio>
#include <cstdlib>

#include "sample_split.h"

int main(int argc, char** argv) {
    if (argc != 9) return 2;
    int a[8];
    for (int i = 0; i < 8; ++i) a[i] = atoi(argv[1 + i]);
    const cd::SaBlocks blocks{a[3], a[4]};
    for (int k = 0; k < a[2]; ++k) {
        const cd::SaSplit s = cd::sa_split(a[0], a[0] + a[1] + k, blocks, a[5], a[6], a[7]);
        printf("%d %d %d %d %d\n", s.id(), s.rounds, s.spans, s.shared, s.own);
    }
    printf("%d %d\n", blocks.count(), blocks.per_block());
    return 0;
}
