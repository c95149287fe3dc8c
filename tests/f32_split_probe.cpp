// prints how many blocks share a tile's depth:  probe <col tiles> <rows> <groups> <K> <SMs>
#include <stdio.h>
#include <stdlib.h>

#include "f32_split.h"

int main(int, char **argv) {
    const auto n = [&](int i) { return (uint32_t)strtoul(argv[i], nullptr, 10); };
    printf("%u\n", nb::f32_split(n(1), n(2), n(3), n(4), n(5)));
    return 0;
}
