// Host-side check of a batch's block arena (cuopo3d_b200/csrc/block_arena.h), compiled and run by
// tests/test_block_arena.py; no GPU needed.
//
// Device and pinned memory are counted address ranges.  Instances of random sizes are
// admitted (whenever the blocks in use leave the budget room, as the batch does) and
// retired in random order: every admission must be served, the device memory held must never
// exceed the budget, not even during a move, idle memory must stay within its bound unless the
// budget left no room for the moves, and every block must keep its contents.  A second form
// makes device allocations fail at random: an admission may then be refused, but no block
// may lose its contents.
#include "../../cuopo3d_b200/csrc/block_arena.h"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>

namespace {

constexpr size_t MB = (size_t)1 << 20;

struct Block {
    size_t bytes;
    uint64_t tag;
};

struct World {
    std::map<void *, size_t> device, host;  // allocations
    size_t now = 0, peak = 0, moves = 0, spills = 0;
    std::map<char *, Block> live;
    std::mt19937_64 rng{7};
    double fail = 0;
    bool failing() { return std::uniform_real_distribution<>(0, 1)(rng) < fail; }
};

// The contents of the block at p: one value (the addresses have no storage).
uint64_t &word(World &w, const void *p)
{
    static std::map<const void *, uint64_t> store;
    for (auto *m : {&w.device, &w.host}) {
        auto it = m->upper_bound(const_cast<void *>(p));
        if (it != m->begin() && (size_t)((const char *)p - (const char *)(--it)->first) < it->second) return store[p];
    }
    std::printf("FAIL: access outside every allocation\n");
    std::exit(1);
}

struct Mem {
    World *w;
    static char *reserve(size_t n)
    {
        static uintptr_t next = (uintptr_t)1 << 40;
        const uintptr_t p = next;
        next += (n + MB) / MB * MB;
        return reinterpret_cast<char *>(p);
    }
    void *alloc(size_t n)
    {
        if (w->failing()) return nullptr;
        void *p = reserve(n);
        w->device[p] = n;
        w->now += n;
        w->peak = std::max(w->peak, w->now);
        return p;
    }
    void free(void *p)
    {
        w->now -= w->device.at(p);
        w->device.erase(p);
    }
    void *alloc_host(size_t n)
    {
        void *p = reserve(n);
        w->host[p] = n;
        return p;
    }
    void free_host(void *p) { w->host.erase(w->host.find(p)); }
    bool copy(void *to, const void *from, size_t)
    {
        word(*w, to) = word(*w, from);
        return true;
    }
    void moved(void *from, void *to, size_t n)
    {
        auto it = w->live.find(static_cast<char *>(from));
        if (it == w->live.end()) return;
        const Block b = it->second;
        if (b.bytes != n) {
            std::printf("FAIL: moved %zu bytes of %zu\n", n, b.bytes);
            std::exit(1);
        }
        w->live.erase(it);
        w->live[static_cast<char *>(to)] = b;
        w->moves++;
        w->spills += w->host.count(to);
    }
};

int fails = 0;
void expect(bool ok, const char *what, int step)
{
    if (ok || fails++ > 10) return;
    std::printf("FAIL: %s at step %d\n", what, step);
}

void random_run(unsigned seed, size_t budget, double fail)
{
    World w;
    w.rng.seed(seed);
    w.fail = fail;
    {
        opo::BlockArena<Mem> arena(Mem{&w});
        uint64_t tag = 1;
        size_t used = 0;
        const size_t sizes[] = {2 * MB, 5 * MB, 9 * MB, 32 * MB, 33 * MB, 100 * MB, 300 * MB, budget / 2, budget - 40 * MB};
        for (int step = 0; step < 4000; step++) {
            const bool phase = (step / 200) % 2;  // many small ones, then few large ones
            if (std::uniform_int_distribution<>(0, 99)(w.rng) < 55) {
                const size_t need = sizes[phase ? std::uniform_int_distribution<>(3, 8)(w.rng)
                                                : std::uniform_int_distribution<>(0, 4)(w.rng)];
                if (used + need <= budget) {
                    void *p = arena.take(need, 20, budget);
                    expect(p || fail > 0, "an admissible instance was refused", step);
                    if (p) {
                        word(w, p) = tag;
                        w.live[static_cast<char *>(p)] = Block{need, tag++};
                        used += need;
                    }
                }
            } else if (!w.live.empty()) {
                auto it = w.live.begin();
                std::advance(it, std::uniform_int_distribution<size_t>(0, w.live.size() - 1)(w.rng));
                char *p = it->first;
                used -= it->second.bytes;
                w.live.erase(it);
                arena.give(p, budget);
                // (a slab's blocks in use, all of which a move copies, are less than 256 MB)
                expect(fail > 0 || arena.idle() <= opo::BlockArena<Mem>::kIdleBytes || arena.held() + 256 * MB > budget,
                       "idle memory kept beyond its bound", step);
            }
            for (auto &l : w.live) expect(word(w, l.first) == l.second.tag, "a block lost its contents", step);
            expect(w.now == arena.held() && w.now <= budget, "held beyond the budget", step);
        }
        expect(w.peak <= budget, "held beyond the budget during a move", -1);
        if (fail == 0) expect(w.moves > 0 && w.spills == 0, "the run made no move", -1);
    }
    expect(w.device.empty() && w.host.empty(), "memory not given back", -1);
    std::printf("seed %u budget %zu MB fail %.2f: peak %zu MB, %zu moves, %zu to the host\n", seed, budget / MB, fail,
                w.peak / MB, w.moves, w.spills);
}

// 64 instances of 32 MB, seven of each slab's eight retired, then one of 3500 MB in 4096.
void survivors()
{
    World w;
    opo::BlockArena<Mem> arena(Mem{&w});
    const size_t budget = 4096 * MB;
    std::vector<char *> p;
    for (int k = 0; k < 64; k++) {
        char *q = static_cast<char *>(arena.take(32 * MB, 63 - k, budget));
        word(w, q) = 100 + k;
        w.live[q] = Block{32 * MB, 100u + k};
        p.push_back(q);
    }
    expect(w.device.size() == 8, "slabs of eight", 0);
    for (int k = 0; k < 64; k++)
        if (k % 8 != 3) {
            // (a survivor may have moved: find the instance by its tag)
            for (auto &l : w.live)
                if (l.second.tag == 100u + k) {
                    char *q = l.first;
                    w.live.erase(q);
                    arena.give(q, budget);
                    break;
                }
        }
    expect(w.live.size() == 8 && arena.idle() <= opo::BlockArena<Mem>::kIdleBytes, "idle memory kept beyond its bound", 1);
    expect(arena.take(3500 * MB, 0, budget) != nullptr, "an admissible instance was refused", 2);
    expect(w.peak <= budget && w.now <= budget, "held beyond the budget", 3);
    for (auto &l : w.live) expect(word(w, l.first) == l.second.tag, "a block lost its contents", 4);
}

}  // namespace

int main()
{
    survivors();
    for (unsigned seed = 1; seed <= 6; seed++)
        for (size_t mb : {400, 700, 2000}) {
            random_run(seed, mb * MB, 0);
            random_run(seed, mb * MB, 0.2);
        }
    return fails ? 1 : 0;
}
