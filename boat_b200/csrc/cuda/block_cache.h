// block_cache.h - idle device memory kept by the library between a free and the next allocation, in pieces of
// larger slabs.  Host code without a CUDA call in it: the memory comes from a Source.
//
// A freed piece first waits in a bin for a request of the very size that it was handed out for: a step that
// repeats finds all its blocks there, without cutting or joining (nine launches of a 2 x 64 x 64 step took 2 us longer
// with both at every call).  A request that finds its bin empty has all binned pieces joined with their idle
// neighbours, and takes the smallest idle piece that holds it and leaves the rest idle.  So a program whose sizes change from step to step - batches of uneven length, one
// encoder block after another - finds its memory in what the last sizes left, which a cache of whole blocks by
// size does not: fresh memory costs the driver 6 to 40 us per MB on B200, a piece of a slab a look-up.
//
// Order is the stream's: a piece may be written by whatever is launched next on the stream on which it was
// freed.  Pieces freed on another stream than the current one are not handed out and not joined with others until
// everything on the device has been waited for, which only happens when memory is short.  A stream is named by
// the id that the runtime gives it, which is never used twice, so nothing here refers to a stream that the caller may
// have destroyed since.
//
// Requests up to kSmall live in slabs of their own: a bias that lives as long as its layer must not hold a
// large slab.  Slabs grow by the step in which the driver's pool grows.  When no idle piece is large enough, whole
// idle slabs are first given back, oldest first and as many bytes as are about to be asked for: the driver's pool
// joins what lies side by side without mapping anything (3 us where a fresh 384 MB take milliseconds).
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <map>
#include <set>
#include <unordered_map>
#include <vector>

namespace boatcu {

class BlockCache {
public:
    struct Source {
        virtual void* take(size_t bytes) = 0;     // NULL when there is no such block
        virtual void give(void* slab) = 0;        // in the order of the current stream
        virtual bool wait() = 0;                  // until the device is idle
        virtual ~Source() {}
    };
    static constexpr size_t kUnit = 512, kSmall = (size_t)1 << 20, kSmallSlab = (size_t)2 << 20, kSlab = (size_t)32 << 20;

    BlockCache(Source& source, size_t idle_limit) : source_(source), limit_(idle_limit) {}

    // A block of at least `bytes` (> 0) for use on `stream`; NULL when the source has none.
    void* get(size_t bytes, uint64_t stream) {
        const size_t want = round_up(bytes, kUnit);
        if (want < bytes) return nullptr;
        Piece* p = from_bin(want, stream);
        if (!p) p = cut(want, stream);
        if (!p) return nullptr;
        p->want = want;
        p->asked = bytes;
        used_ += bytes;
        live_[p->ptr] = p;
        return p->ptr;
    }

    // Ends the use of a block on `stream`; false when it is not one of this cache's.
    bool put(void* ptr, uint64_t stream) {
        const auto found = live_.find(ptr);
        if (found == live_.end()) return false;
        Piece* p = found->second;
        live_.erase(found);
        used_ -= p->asked;
        p->stream = stream;
        if (stream != bins_stream_) empty_bins();
        bins_stream_ = stream;
        bins_[p->want].push_back(p);
        binned_ += p->bytes;
        if (idle_bytes() > limit_) trim(limit_, stream);
        return true;
    }

    bool owns(void* ptr) const { return live_.count(ptr) != 0; }
    size_t used_bytes() const { return used_; }         // as asked for
    size_t idle_bytes() const { return idle_bytes_ + binned_; }
    size_t held_bytes() const { return held_; }         // all slabs

    // Gives whole idle slabs back, oldest first (binned pieces count as new), until at most `limit` bytes are idle or
    // none is left.
    void trim(size_t limit, uint64_t stream) {
        empty_bins();
        give_back(limit, stream);
        if (idle_bytes_ <= limit) return;
        bool foreign = false;
        for (Piece* p : idle_) foreign = foreign || p->stream != stream;
        if (!foreign || !source_.wait()) return;
        adopt(stream);
        give_back(limit, stream);
    }

private:
    struct Slab {
        size_t bytes;
        bool large;
    };
    struct Piece {
        char* ptr;
        size_t bytes, want, asked;                // its own, and those of the request it serves or last served
        Slab* slab;
        Piece *prev, *next;                       // neighbours in the slab
        uint64_t stream;                          // on which it was freed
        uint64_t age;                             // of a slab that is idle as a whole
        bool idle;                                // and listed; a piece in a bin is not
    };
    struct Less {
        bool operator()(const Piece* a, const Piece* b) const {
            if (a->slab->large != b->slab->large) return b->slab->large;
            if (a->stream != b->stream) return a->stream < b->stream;
            if (a->bytes != b->bytes) return a->bytes < b->bytes;
            return a->ptr < b->ptr;
        }
    };
    typedef std::set<Piece*, Less> IdleSet;

    static size_t round_up(size_t n, size_t unit) { return (n + unit - 1) / unit * unit; }

    // A piece that last served a request of this size, as it is.
    Piece* from_bin(size_t want, uint64_t stream) {
        if (stream != bins_stream_) return nullptr;
        const auto bin = bins_.find(want);
        if (bin == bins_.end() || bin->second.empty()) return nullptr;
        Piece* p = bin->second.back();
        bin->second.pop_back();
        binned_ -= p->bytes;
        return p;
    }

    void empty_bins() {
        if (binned_ == 0) return;
        binned_ = 0;
        for (auto& bin : bins_)
            for (Piece* p : bin.second) {
                p->idle = true;
                list(join(p));
            }
        bins_.clear();
    }

    // The smallest idle piece that holds `want`, less what is left over.
    Piece* cut(size_t want, uint64_t stream) {
        const bool large = want > kSmall;
        empty_bins();
        auto it = find(want, large, stream);
        if (it == idle_.end()) {
            if (!grow(want, large, stream)) return nullptr;
            it = find(want, large, stream);
        }
        Piece* p = *it;
        unlist(p);
        p->idle = false;
        if (p->bytes - want >= (large ? kSmall : kUnit)) {
            Piece* rest = new Piece{p->ptr + want, p->bytes - want, 0, 0, p->slab, p, p->next, p->stream, 0, true};
            if (p->next) p->next->prev = rest;
            p->next = rest;
            p->bytes = want;
            list(rest);
        }
        return p;
    }

    // The smallest idle piece of at least `want` bytes that may be used on `stream`.
    IdleSet::iterator find(size_t want, bool large, uint64_t stream) {
        Slab kind{0, large};
        Piece key{nullptr, want, 0, 0, &kind, nullptr, nullptr, stream, 0, true};
        const auto it = idle_.lower_bound(&key);
        return it != idle_.end() && (*it)->slab->large == large && (*it)->stream == stream ? it : idle_.end();
    }

    void list(Piece* p) {
        idle_.insert(p);
        idle_bytes_ += p->bytes;
        if (p->bytes == p->slab->bytes) whole_[p->age = ++clock_] = p;
    }

    void unlist(Piece* p) {
        idle_.erase(p);
        idle_bytes_ -= p->bytes;
        if (p->age) whole_.erase(p->age);
        p->age = 0;
    }

    // `p` (idle, not listed) as one piece with its idle neighbours of the same stream.
    Piece* join(Piece* p) {
        Piece* n = p->next;
        if (n && n->idle && n->stream == p->stream) {
            unlist(n);
            p->bytes += n->bytes;
            p->next = n->next;
            if (n->next) n->next->prev = p;
            delete n;
        }
        Piece* b = p->prev;
        if (b && b->idle && b->stream == p->stream) {
            unlist(b);
            b->bytes += p->bytes;
            b->next = p->next;
            if (p->next) p->next->prev = b;
            delete p;
            p = b;
        }
        return p;
    }

    void drop(Piece* whole) {
        unlist(whole);
        held_ -= whole->bytes;
        source_.give(whole->ptr);
        delete whole->slab;
        delete whole;
    }

    void give_back(size_t limit, uint64_t stream) {
        for (auto it = whole_.begin(); it != whole_.end() && idle_bytes_ > limit;) {
            Piece* p = (it++)->second;
            if (p->stream == stream) drop(p);
        }
    }

    // The device is idle: every idle piece is free for `stream`.
    void adopt(uint64_t stream) {
        IdleSet all;
        all.swap(idle_);
        whole_.clear();
        idle_bytes_ = 0;
        for (Piece* p : all) {                    // `all` keeps its order: only re-listed below
            p->age = 0;
            p->idle = false;
        }
        std::set<Piece*> left(all.begin(), all.end());
        all.clear();
        while (!left.empty()) {
            Piece* p = *left.begin();
            left.erase(left.begin());
            p->stream = stream;
            p->idle = true;
            list(join(p));                        // neighbours still in `left` are not idle yet and join later
        }
    }

    bool grow(size_t want, bool large, uint64_t stream) {
        size_t bytes = large ? round_up(want, kSlab) : kSmallSlab;
        if (large) {
            size_t given = 0;
            for (auto it = whole_.begin(); it != whole_.end() && given < bytes;) {
                Piece* p = (it++)->second;
                if (!p->slab->large || p->stream != stream) continue;
                given += p->bytes;
                drop(p);
            }
        }
        void* base = source_.take(bytes);
        if (!base) {
            trim(0, stream);                      // what is kept idle here may be what is missing
            if (find(want, large, stream) != idle_.end()) return true;
            base = source_.take(bytes);
        }
        if (!base && bytes > want) base = source_.take(bytes = want);
        if (!base) return false;
        held_ += bytes;
        list(new Piece{(char*)base, bytes, 0, 0, new Slab{bytes, large}, nullptr, nullptr, stream, 0, true});
        return true;
    }

    Source& source_;
    const size_t limit_;
    IdleSet idle_;
    std::map<uint64_t, Piece*> whole_;            // slabs idle as a whole, oldest first
    std::unordered_map<void*, Piece*> live_;
    std::unordered_map<size_t, std::vector<Piece*>> bins_;        // by the size of the request, freed on bins_stream_
    uint64_t bins_stream_ = 0;
    size_t binned_ = 0;
    size_t used_ = 0, idle_bytes_ = 0, held_ = 0;
    uint64_t clock_ = 0;
};

}  // namespace boatcu
