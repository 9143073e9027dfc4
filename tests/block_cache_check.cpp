// CPU check of boat_b200/csrc/cuda/block_cache.h against a source that hands out addresses only.
#include "block_cache.h"
#include <stdio.h>
#include <stdlib.h>
#include <vector>

using boatcu::BlockCache;

#define CHECK(c)                                                                              \
    do {                                                                                      \
        if (!(c)) {                                                                           \
            printf("%s:%d: %s\n", __FILE__, __LINE__, #c);                                    \
            exit(1);                                                                          \
        }                                                                                     \
    } while (0)

struct Addresses : BlockCache::Source {
    std::map<uintptr_t, size_t> slabs;
    uintptr_t next = (uintptr_t)1 << 32;
    size_t bytes = 0, room = SIZE_MAX;
    int taken = 0, given = 0, waits = 0;
    void* take(size_t n) override {
        if (n > room || bytes > room - n) return nullptr;
        const uintptr_t at = next;
        next += n + 4096;
        slabs[at] = n;
        bytes += n;
        ++taken;
        return (void*)at;
    }
    void give(void* p) override {
        const auto it = slabs.find((uintptr_t)p);
        CHECK(it != slabs.end());
        bytes -= it->second;
        slabs.erase(it);
        ++given;
    }
    bool wait() override { return ++waits, true; }
    bool holds(uintptr_t p, size_t n) const {
        auto it = slabs.upper_bound(p);
        if (it == slabs.begin()) return false;
        --it;
        return p + n <= it->first + it->second;
    }
};

// Blocks of all sizes taken and freed at random on three streams: none overlaps another, all lie in slabs that
// are held, and memory last used on another stream comes back only after a wait.
static void random_use(unsigned seed) {
    srand(seed);
    Addresses src;
    BlockCache cache(src, (size_t)256 << 20);
    struct Use { size_t bytes; };
    std::map<uintptr_t, Use> live;
    std::map<uintptr_t, std::pair<uintptr_t, uint64_t>> last;     // freed ranges: begin -> end, stream
    int waits = 0;
    uint64_t stream = 0;
    size_t used = 0;
    for (int step = 0; step < 20000; ++step) {
        if (rand() % 200 == 0) stream = rand() % 3;
        if (src.waits != waits) { waits = src.waits; last.clear(); }
        if (live.size() < 40 && rand() % 2) {
            const int kind = rand() % 3;
            const size_t n = kind == 0 ? 1 + rand() % 5000 : kind == 1 ? 1 + rand() % (3 << 20) : ((size_t)(1 + rand() % 60) << 20) + rand() % 4096;
            const uintptr_t p = (uintptr_t)cache.get(n, stream);
            CHECK(p && p % 512 == 0 && src.holds(p, n));
            if (src.waits != waits) { waits = src.waits; last.clear(); }
            auto after = live.lower_bound(p);
            CHECK(after == live.end() || p + n <= after->first);
            if (after != live.begin()) { --after; CHECK(after->first + after->second.bytes <= p); }
            for (auto it = last.begin(); it != last.end();) {
                if (it->first < p + n && it->second.first > p) {
                    CHECK(it->second.second == stream);
                    it = last.erase(it);
                } else {
                    ++it;
                }
            }
            live[p] = Use{n};
            used += n;
        } else if (!live.empty()) {
            auto it = live.begin();
            std::advance(it, rand() % live.size());
            const uintptr_t p = it->first, n = it->second.bytes;
            last[p] = {p + n, stream};
            used -= n;
            live.erase(it);
            CHECK(cache.put((void*)p, stream));
            CHECK(!cache.put((void*)p, stream));
            for (auto k = last.begin(); k != last.end();) k = src.holds(k->first, 1) ? std::next(k) : last.erase(k);
        }
        CHECK(cache.used_bytes() == used && cache.held_bytes() == src.bytes);
    }
    for (auto& l : live) CHECK(cache.put((void*)l.first, stream));
    cache.trim(0, stream);
    CHECK(cache.idle_bytes() == 0 && cache.held_bytes() == 0 && src.slabs.empty() && src.taken == src.given);
}

static void limits() {
    Addresses src;
    BlockCache cache(src, (size_t)100 << 20);
    std::vector<void*> b;
    for (int i = 0; i < 8; ++i) b.push_back(cache.get((size_t)32 << 20, 0));
    CHECK(cache.held_bytes() == (size_t)256 << 20);
    for (void* p : b) cache.put(p, 0);
    CHECK(cache.idle_bytes() == (size_t)96 << 20 && cache.held_bytes() == cache.idle_bytes());      // the newest three stay
    // short memory: what is idle, on whatever stream, makes room; nothing is left in a state that a later call trips over
    Addresses small;
    small.room = (size_t)96 << 20;
    BlockCache c2(small, SIZE_MAX);
    void* x = c2.get((size_t)32 << 20, 1);
    void* y = c2.get((size_t)32 << 20, 2);
    CHECK(x && y);
    c2.put(x, 1);
    c2.put(y, 2);
    void* z = c2.get((size_t)90 << 20, 3);
    CHECK(z && small.waits == 1);
    CHECK(!c2.get((size_t)32 << 20, 3) && !c2.get(SIZE_MAX - 3, 3));
    c2.put(z, 3);
    CHECK(c2.get((size_t)32 << 20, 3));
    // a slab that does not fit as a whole is taken as large as it has to be
    Addresses odd;
    odd.room = ((size_t)33 << 20) + 512;
    BlockCache c3(odd, SIZE_MAX);
    CHECK(c3.get(((size_t)33 << 20) + 5, 0));
    CHECK(!c3.get(512, 0));
    // a small block never holds a large slab
    Addresses two;
    BlockCache c4(two, SIZE_MAX);
    void* big = c4.get((size_t)64 << 20, 0);
    c4.put(big, 0);
    CHECK(c4.get(100, 0) && c4.idle_bytes() >= (size_t)64 << 20);
    CHECK(c4.get((size_t)64 << 20, 0) == big);
}

// The allocations of one forward and backward of an attention layer on T rows of width H (BF16), in its order.
struct Layer {
    std::vector<void*> state;
    void step(BlockCache& c, size_t T, size_t H) {
        const size_t act = T * H * 2;
        for (void* p : state) c.put(p, 0);
        state.clear();
        for (int i = 0; i < 4; ++i) state.push_back(c.get(act, 0));
        state.push_back(c.get(T * 64, 0));
        void* out = c.get(act, 0);
        void* dout = c.get(act, 0);
        std::vector<void*> gin, temp;
        for (int i = 0; i < 3; ++i) gin.push_back(c.get(act, 0));
        for (int i = 0; i < 4; ++i) temp.push_back(c.get(act, 0));
        temp.push_back(c.get(2 * act + T * 128, 0));
        for (void* p : temp) c.put(p, 0);
        c.put(out, 0);
        c.put(dout, 0);
        for (void* p : gin) c.put(p, 0);
    }
};

// Lengths that change with every step settle: from the third round on nothing is taken or given.
static void changing_lengths() {
    Addresses src;
    BlockCache cache(src, (size_t)8 << 30);
    Layer layer;
    int moves = 0;
    for (int round = 0; round < 6; ++round) {
        if (round == 3) moves = src.taken + src.given;
        for (size_t i = 0; i < 10; ++i) layer.step(cache, 4 * (300 + 170 * ((i * 7) % 10)), 1024);
    }
    printf("changing lengths: %d slabs taken, %d given back, %.0f MB held\n", src.taken, src.given, cache.held_bytes() / 1048576.0);
    CHECK(src.taken + src.given == moves);
}

int main() {
    for (unsigned seed = 1; seed <= 10; ++seed) random_use(seed);
    limits();
    changing_lengths();
    printf("ok\n");
    return 0;
}
