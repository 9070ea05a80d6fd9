// Drives csrc/drain.h against a model of a ring of mbarriers: load i may start once load i - depth has landed, a wait on a parity returns
// at once where the phase of that parity is the one before the running one, and lands a load that is in flight.  And tile_asked
// against the order in which a tile of csrc/tc_scan_tma.cuh asks for its slabs and x pieces, with any of its waits running out.  Prints "ok".
#include <cstdio>
#include <vector>

#include "../bi-mamba2_b200/csrc/drain.h"

// The waits of one tile in their order, the one numbered `bad` running out: what it had asked for, and what it noted.
struct Tile {
    int slabs = 0, pieces = 0, where = 0, waits = 0, bad;
    bool wait() { return waits++ != bad; }
    bool products(int ns, int nx) {
        slabs = ns > 1 ? 2 : 1;
        if (ns == 1) pieces = nx ? 2 : 0;
        for (int k = 0; k < ns; ++k) {
            if (!wait()) { where = 1 + k; return false; }               // slab k
            if (k >= 1) {
                if (!wait()) { where = 1 + k; return false; }           // slab k - 1 has been read
                if (k + 1 < ns) ++slabs;
                else pieces = nx ? 2 : 0;
            }
        }
        return true;
    }
    void run(int ns, int nx) {
        bool ok = products(ns, nx) && wait();                           // the products are done
        for (int it = 0; it < nx; ++it) {
            if (it >= 2 && ok) ok = wait();                             // the stage's buffers are free
            if (!ok) {
                if (!where) where = bissd::kStages + it;
                return;
            }
            if (it >= 2) ++pieces;
            if (!wait()) { where = bissd::kStages + it + 1; ok = false; }   // its piece of x
        }
        if (ok) wait();                                                 // the last product
    }
};

int main() {
    for (int ns = 1; ns <= 4; ++ns)
        for (int nx = 0; nx <= 4; nx += 2)                              // chunks of 128 and 256; 0: a tile without x
            for (int bad = 0, last = 1; bad < last; ++bad) {
                Tile t;
                t.bad = bad;
                t.run(ns, nx);
                last = t.waits + 1;
                const bissd::Asked a = bissd::tile_asked(t.where, ns, nx);
                if (a.slabs != t.slabs || a.pieces != t.pieces) {
                    std::printf("%d slabs, %d pieces, wait %d: %d, %d asked for\n", ns, nx, bad, t.slabs, t.pieces);
                    return 1;
                }
            }
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
