// Device memory of a batch's instances (batch.cu): blocks out of slabs of up to eight, kept for
// the next instance of the same size.
//
// A cudaMalloc of an instance's size takes 0.32 ms, its cudaFree 0.29 ms, and a slab of eight
// no longer than one block, so a slab costs an eighth per instance.  What is held stays
// within the batch's HBM budget whatever the order of sizes: a request that the budget has
// room for gets the idle blocks' memory.  Wholly idle slabs go back to the driver; of a slab with
// blocks still in use, those move into memory of their own first (dissolve).  Idle memory is
// kept up to kIdleBytes and given back beyond that (short of room for the moves, the
// budget remains its bound), everything with the arena.
//
// Mem supplies the memory: alloc / free (device), alloc_host / free_host (pinned host memory
// that kernels can address), copy (after the work on the blocks so far, complete on return),
// and moved(from, to, bytes): the instance whose block was at `from` has it at `to` now.
// alloc* return null when there is none.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace opo {

template <typename Mem> class BlockArena {
public:
    static constexpr size_t kIdleBytes = (size_t)256 << 20;

    explicit BlockArena(Mem m) : mem_(m) {}
    BlockArena(const BlockArena &) = delete;
    BlockArena &operator=(const BlockArena &) = delete;
    ~BlockArena()
    {
        for (Slab &s : slabs_) release(s);
    }

    // A block of `need` bytes for an instance that the budget has room for (the blocks in use
    // and this one are within it); up to `more` further instances may follow.  Null: out of
    // memory.  Blocks in use may move.
    void *take(size_t need, int more, size_t budget)
    {
        for (Slab &s : slabs_)
            if (s.block == need)
                for (Part &b : s.parts)
                    if (!b.used) {
                        b.used = true;
                        return b.p;
                    }
        while (held_ + need > budget)
            if (!give_back(budget, true)) return nullptr;
        size_t n = std::min<size_t>({8, (size_t)more + 1, (budget - held_) / need,
                                     1 + (kIdleBytes - std::min(kIdleBytes, idle())) / need});
        void *p = mem_.alloc(n * need);
        while (!p && (n > 1 || give_back(budget, true))) {
            n = 1;
            p = mem_.alloc(need);
        }
        if (!p) return nullptr;
        add(p, need, n, false);
        slabs_.back().parts[0].used = true;
        return p;
    }

    // The block at p is idle.  Blocks in use may move.
    void give(const void *p, size_t budget)
    {
        for (Slab &s : slabs_)
            for (Part &b : s.parts)
                if (b.p == p) b.used = false;
        for (size_t k = 0; k < slabs_.size(); k++)  // spilled to the host: not kept
            if (slabs_[k].host && !slabs_[k].used()) drop(k--);
        while (idle() > kIdleBytes && give_back(budget, false)) {}
    }

    size_t held() const { return held_; }
    size_t idle() const
    {
        size_t n = 0;
        for (const Slab &s : slabs_) n += s.host ? 0 : (s.parts.size() - s.used()) * s.block;
        return n;
    }

private:
    struct Part {
        char *p;
        bool used;
    };
    struct Slab {
        void *p;
        size_t block;  // bytes of each part
        bool host;
        std::vector<Part> parts;
        size_t used() const
        {
            return (size_t)std::count_if(parts.begin(), parts.end(), [](const Part &b) { return b.used; });
        }
        size_t bytes() const { return block * parts.size(); }
    };

    void add(void *p, size_t block, size_t n, bool host)
    {
        Slab s{p, block, host, {}};
        for (size_t k = 0; k < n; k++) s.parts.push_back({static_cast<char *>(p) + k * block, false});
        if (!host) held_ += s.bytes();
        slabs_.push_back(s);
    }
    void release(Slab &s)
    {
        if (s.host) mem_.free_host(s.p);
        else mem_.free(s.p);
    }
    void drop(size_t k)
    {
        if (!slabs_[k].host) held_ -= slabs_[k].bytes();
        release(slabs_[k]);
        slabs_.erase(slabs_.begin() + (std::ptrdiff_t)k);
    }

    // Gives the idle memory of one slab back: of one that is wholly idle, or else of the one with
    // the least in use beside idle blocks.  False: there is none, or it cannot be done.
    bool give_back(size_t budget, bool through_host)
    {
        size_t best = slabs_.size(), least = 0;
        for (size_t k = 0; k < slabs_.size(); k++) {
            const size_t used = slabs_[k].used();
            if (slabs_[k].host || used == slabs_[k].parts.size()) continue;
            if (best == slabs_.size() || used * slabs_[k].block < least) {
                best = k;
                least = used * slabs_[k].block;
            }
        }
        if (best == slabs_.size()) return false;
        if (least) return dissolve(best, budget, through_host);
        drop(best);
        return true;
    }

    // Moves the blocks in use of slab k into allocations of their own and frees it: by device
    // copies where the budget and the device have room for both, else (through_host) by way of
    // pinned host memory.  A block whose memory is gone when it comes back (taken by another
    // process meanwhile) stays in that host memory, which kernels can use: none is ever lost.
    bool dissolve(size_t k, size_t budget, bool through_host)
    {
        std::vector<char *> from;
        for (const Part &b : slabs_[k].parts)
            if (b.used) from.push_back(b.p);
        const size_t block = slabs_[k].block, n = from.size();
        std::vector<void *> to;
        if (held_ + n * block <= budget && copies(from, block, to, false)) {
            for (size_t i = 0; i < n; i++) settle(from[i], to[i], block, false);
            drop(k);
            return true;
        }
        if (!through_host || !copies(from, block, to, true)) return false;
        drop(k);
        for (size_t i = 0; i < n; i++) {
            void *p = mem_.alloc(block);
            if (p && !mem_.copy(p, to[i], block)) {
                mem_.free(p);
                p = nullptr;
            }
            settle(from[i], p ? p : to[i], block, !p);
            if (p) mem_.free_host(to[i]);
        }
        return true;
    }
    // Copies of the blocks at `from` in new memory; none when one cannot be made.
    bool copies(const std::vector<char *> &from, size_t block, std::vector<void *> &to, bool host)
    {
        to.clear();
        bool ok = true;
        for (size_t i = 0; i < from.size() && ok; i++) {
            void *p = host ? mem_.alloc_host(block) : mem_.alloc(block);
            ok = p != nullptr;
            if (p) to.push_back(p);
            ok = ok && mem_.copy(p, from[i], block);
        }
        if (ok) return true;
        for (void *p : to) {
            if (host) mem_.free_host(p);
            else mem_.free(p);
        }
        to.clear();
        return false;
    }
    void settle(void *from, void *to, size_t block, bool host)
    {
        add(to, block, 1, host);
        slabs_.back().parts[0].used = true;
        mem_.moved(from, to, block);
    }

    Mem mem_;
    std::vector<Slab> slabs_;
    size_t held_ = 0;
};

}  // namespace opo
