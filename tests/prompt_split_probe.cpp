// prints, for every depth that the arguments ask for, how the parts of csrc/prompt_split.h cover it:  probe <max depth>
#include <stdio.h>
#include <stdlib.h>

#include "prompt_split.h"

int main(int, char **argv) {
    const uint32_t most = (uint32_t)atoi(argv[1]);
    const uint32_t gss[] = {32, 64, 128, 256};
    for (uint32_t gs : gss)
        for (uint32_t n = gs; n <= most; n += gs) {
            if (n % 16u) continue;
            for (uint32_t ks = 1; ks <= 8; ks *= 2) {
                uint32_t groups = 0, steps = 0;
                for (uint32_t p = 0; p < ks; p++) {
                    const nb::PromptPart a = nb::prompt_part(true, n, 0, gs, ks, p);
                    if (a.g0 != groups || a.groups > n / gs || (a.steps && a.s0 != steps)) { printf("q80 n %u gs %u ks %u part %u: groups [%u, +%u), stages [%u, +%u)\n", n, gs, ks, p, a.g0, a.groups, a.s0, a.steps); return 1; }
                    groups += a.groups; steps += a.steps;
                }
                if (groups != n / gs || steps * 128u < n) { printf("q80 n %u gs %u ks %u: %u groups, %u stages\n", n, gs, ks, groups, steps); return 1; }
            }
        }
    for (uint32_t np = 64; np <= most; np += 64)
        for (uint32_t ks = 1; ks <= 8; ks *= 2) {
            uint32_t steps = 0;
            for (uint32_t p = 0; p < ks; p++) {
                const nb::PromptPart a = nb::prompt_part(false, np, np, 0, ks, p);
                if (a.steps && a.s0 != steps) { printf("f32 np %u ks %u part %u: stages [%u, +%u)\n", np, ks, p, a.s0, a.steps); return 1; }
                steps += a.steps;
            }
            if (steps != np / 64u) { printf("f32 np %u ks %u: %u stages\n", np, ks, steps); return 1; }
        }
    printf("ok\n");
    return 0;
}
