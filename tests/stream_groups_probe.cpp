// prints the query heads of an attention item and its splits:  probe <kv heads> <query heads of each> <head size> <Q4K> <keys> <SMs>
#include <stdio.h>
#include <stdlib.h>

#include "stream_groups.h"

int main(int, char **argv) {
    const auto n = [&](int i) { return (uint32_t)strtoul(argv[i], nullptr, 10); };
    const uint32_t h = nb::st_group_heads(n(1), n(2), n(3), n(4) != 0, n(5), n(6));
    printf("%u %u\n", h, nb::st_splits(n(1) * (n(2) / h), n(6)));
    return 0;
}
