// stream_count.h -- what launches of the streaming decode kernel have used up: epochs of its exchanges and arrivals at its grid barrier, whose counter is never reset
#pragma once
#include <stdint.h>

namespace nb {

// The host's copy of two numbers that only the device moves.  A launch that is refused arrives nowhere: it must leave them as they are, or the launch after it would wait
// for arrivals that never come.
struct StreamCount {
    uint32_t epoch = 0, bar = 0;          // epochs handed out so far; what the barrier's counter stands at (modulo 2^32)
    // launch(epoch, bar) puts a kernel that uses so many epochs and arrivals on the stream; 0: it is there
    template <typename Launch>
    int run(uint32_t epochs, uint32_t arrivals, Launch &&launch) {
        const int r = launch(epoch, bar);
        if (r == 0) { epoch += epochs; bar += arrivals; }
        return r;
    }
};

}  // namespace nb
