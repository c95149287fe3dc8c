// prints the tokens of a product's tiles and whether it reads its rows itself:  probe <N> <groups> <rows of each> <K>, for each line of standard input
#include <stdio.h>

#include "tc_tiles.h"

int main() {
    uint32_t n, g, e, k;
    while (scanf("%u %u %u %u", &n, &g, &e, &k) == 4) printf("%u %d\n", nb::tc_tile_tokens(e), nb::tc_reads_rows(n, g, e, k) ? 1 : 0);
    return 0;
}
