// drain_check.cpp -- the order of MMAs, commits and waits of a training tile (swpathtracer_b200/csrc/
// guiding_tc.cu) on a model of the mbarrier, with the wait of every layer and pass running out in turn:
// after spt::tc::drain no MMA may be in flight.
#include <cstdio>
#include <string>
#include <vector>

#include "mma_drain.h"

namespace {

constexpr int kLayers = 5;

// MMAs complete in order, and only when a wait of the drain lets time pass; a commit arrives when every
// MMA before it has completed.
struct Model {
    std::vector<std::string> flight;   // MMAs and commits, oldest first
    unsigned parity = 0;               // of the phase that is still open
    void mma(const std::string& name) { flight.push_back(name); }
    void commit() { flight.push_back("commit"); }
    // phase `p` complete?  `run`: time passes until the next commit arrives.
    bool wait(unsigned p, bool run) {
        if (parity != p) return true;
        while (run && !flight.empty()) {
            const std::string head = flight.front();
            flight.erase(flight.begin());
            if (head == "commit") {
                parity ^= 1u;
                return true;
            }
        }
        return false;
    }
};

// One tile; the wait number `fails` runs out.  True when every MMA had completed before the columns went.
bool tile(int fails, bool& reached) {
    Model m;
    unsigned phase = 0;
    int waits = 0;
    bool ok = true;
    auto wait = [&] {
        const bool out = waits++ == fails;
        ok = out ? false : m.wait(phase, true);
        phase ^= 1u;
    };
    for (int l = 0; l < kLayers && ok; ++l) {
        m.mma("forward " + std::to_string(l));
        m.commit();
        wait();
    }
    for (int l = kLayers - 1; l >= 0 && ok; --l) {
        m.mma("dX " + std::to_string(l));
        if (l > 0) m.commit();
        m.mma("dW " + std::to_string(l));
        if (l == 0) m.commit();
        wait();
    }
    reached = !ok;
    if (ok) return m.flight.empty();
    const bool drained = spt::tc::drain(phase ^ 1u, [&](unsigned p) { return m.wait(p, true); }, [&] { m.commit(); });
    return drained && m.flight.empty();
}

// The same with thread 0's wait satisfied and another thread's run out: the drain starts with its phase
// complete.
bool tile_other_thread(int fails, bool& reached) {
    Model m;
    unsigned phase = 0;
    int waits = 0;
    reached = false;
    auto wait = [&] {
        m.wait(phase, true);
        phase ^= 1u;
        reached = waits++ == fails;
    };
    for (int l = 0; l < kLayers && !reached; ++l) {
        m.mma("forward");
        m.commit();
        wait();
    }
    for (int l = kLayers - 1; l >= 0 && !reached; --l) {
        m.mma("dX");
        if (l > 0) m.commit();
        m.mma("dW");
        if (l == 0) m.commit();
        wait();
    }
    if (!reached) return m.flight.empty();
    const bool drained = spt::tc::drain(phase ^ 1u, [&](unsigned p) { return m.wait(p, true); }, [&] { m.commit(); });
    return drained && m.flight.empty();
}

}  // namespace

int main() {
    int bad = 0, ends = 0;
    for (int fails = 0; fails <= 2 * kLayers; ++fails)
        for (int other = 0; other < 2; ++other) {
            bool reached = false;
            const bool good = other ? tile_other_thread(fails, reached) : tile(fails, reached);
            ends += reached;
            if (!good) std::printf("wait %d%s: MMAs in flight\n", fails, other ? " (another thread's)" : ""), ++bad;
        }
    if (ends != 4 * kLayers) std::printf("%d waits ran out, expected %d\n", ends, 4 * kLayers), ++bad;
    // an MMA that never completes: the drain gives up without a second commit
    int commits = 0;
    if (spt::tc::drain(0, [](unsigned) { return false; }, [&] { ++commits; }) || commits) std::puts("stuck"), ++bad;
    if (!bad) std::puts("ok");
    return bad != 0;
}
