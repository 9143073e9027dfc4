// launch_order.h - which kernel launch may run beside the ones before it.  Bookkeeping alone: it makes no CUDA call and takes no
// lock, so that it can be checked on the CPU.
//
// A launch names the memory that it reads and writes.  It may run beside the launches that may still be running when none of that
// memory matters to them.  The table knows the launches it is told of, nothing else, so it only takes the last of them for the
// predecessor on the stream within one SEQUENCE: a stretch in which one thread issues launches of this library and nothing else, as
// the body of a layer's forward or backward does.  What a program or another library puts on the stream comes before the first
// launch of a sequence or after its last one; the first launch of a sequence, and every launch outside one, waits for whatever is
// before it.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace boatcu {

class LaunchOrder {
public:
    // What a launch belongs to.  Launches of different places never run beside one another.
    struct Place {
        uint64_t sequence;       // 0: none, the launch stands alone
        const void* stream;
        bool per_thread;         // the handle stands for another stream in every thread: nothing follows from it
        uint64_t capture;        // of the stream, while it is being captured: what goes into a graph does not run now
        bool alone() const { return sequence == 0 || per_thread; }
        bool operator==(const Place& o) const {
            return sequence == o.sequence && stream == o.stream && per_thread == o.per_thread && capture == o.capture;
        }
    };

    // One launch: begin, name() for all that it touches, beside(), end - which is told whether it got onto the stream.
    void begin(const Place& place) {
        if (place.alone() || !(place == place_)) count_ = 0;
        place_ = place;
        before_ = count_;
        named_ = overflow_ = beside_ = false;
    }
    void name(const void* p, size_t bytes, bool written) {
        named_ = true;
        if (!p || bytes == 0) return;
        if (count_ == kMaxRanges) overflow_ = true;
        else ranges_[count_++] = Range{(uintptr_t)p, (uintptr_t)p + bytes, written};
    }
    // Whether the launch may run beside the ones before it; without this question it waits for them.
    bool beside() {
        beside_ = before_ > 0 && !overflow_;
        for (int i = before_; i < count_ && beside_; ++i)
            for (int j = 0; j < before_ && beside_; ++j)
                beside_ = ranges_[i].hi <= ranges_[j].lo || ranges_[j].hi <= ranges_[i].lo || !(ranges_[i].written || ranges_[j].written);
        return beside_;
    }
    void end(bool launched) {
        if (!launched || !named_ || overflow_ || place_.alone()) {
            count_ = 0;
        } else if (!beside_) {                  // the launches before are complete once this one lets its successors go
            for (int i = before_; i < count_; ++i) ranges_[i - before_] = ranges_[i];
            count_ -= before_;
        }
    }
    // Something that names nothing comes next on the stream: the launch after it waits.
    void interrupt() { count_ = 0; }

private:
    struct Range {
        uintptr_t lo, hi;
        bool written;
    };
    static constexpr int kMaxRanges = 96;
    Range ranges_[kMaxRanges];   // of the launches that may still be running: the last that waited, and those beside it
    int count_ = 0;              // 0: the next launch waits
    int before_ = 0;             // ranges of the launches before the present one
    bool named_ = false, overflow_ = false, beside_ = false;
    Place place_ = {0, nullptr, false, 0};
};

}  // namespace boatcu
