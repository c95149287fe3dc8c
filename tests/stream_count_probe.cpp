// launches of the streaming kernel, some of them refused, through csrc/stream_count.h, against a counter that moves as the device's does
#include <stdio.h>

#include "stream_count.h"

int main() {
    nb::StreamCount c;
    uint32_t device = 0xffffff00u, first_free = 1;          // the barrier's counter, about to wrap; epochs below this one may have been published
    c.bar = device;
    c.epoch = first_free;
    for (uint32_t i = 0; i < 1000; i++) {
        const uint32_t steps = 1 + i % 7, epochs = steps * 120, arrivals = steps * 148;
        const bool refused = i % 3 == 1 || i % 11 == 0;
        const int r = c.run(epochs, arrivals, [&](uint32_t epoch, uint32_t bar) -> int {
            if (refused) return -4;
            if (bar != device) { printf("launch %u waits for %u arrivals more than the counter will have\n", i, bar - device); return 1; }
            if (epoch < first_free) { printf("launch %u uses epochs again\n", i); return 1; }
            device += arrivals; first_free = epoch + epochs;
            return 0;
        });
        if (r == 1) return 1;
        if (r != (refused ? -4 : 0)) { printf("launch %u: its answer is lost\n", i); return 1; }
    }
    printf("ok\n");
    return 0;
}
