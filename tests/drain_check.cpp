// Drives csrc/drain.h against a model of a ring of mbarriers: load i may start once load i - depth has landed, a wait on a parity returns
// at once where the phase of that parity is the one before the running one, and lands a load that is in flight.  Prints "ok".
#include <cstdio>
#include <vector>

#include "../bi-mamba2_b200/csrc/drain.h"

int main() {
    for (int depth = 1; depth <= 6; ++depth)
        for (int issued = 0; issued <= 3 * depth + 1; ++issued)
            for (int flying = 0; flying < 1 << depth; ++flying) {        // barriers whose last load has not landed
                std::vector<int> phase(depth, 0), pending(depth, 0);     // phases completed; loads in flight
                for (int i = 0; i < issued; ++i) {
                    const bool last = i + depth >= issued;
                    if (last && (flying >> (i % depth) & 1)) pending[i % depth] = 1;
                    else ++phase[i % depth];
                }
                bool stuck = false;
                bissd::drain_ring(issued, depth, [&](int bar, int parity) {
                    if ((phase[bar] & 1) != parity) return;              // that phase is over
                    if (!pending[bar]) stuck = true;                     // nothing will ever end it
                    ++phase[bar];
                    pending[bar] = 0;
                });
                bool left = false;
                for (int p : pending) left = left || p;
                if (stuck || left) {
                    std::printf("depth %d, issued %d, in flight %x: %s\n", depth, issued, flying, stuck ? "a wait without end" : "left in flight");
                    return 1;
                }
            }
    std::puts("ok");
    return 0;
}
