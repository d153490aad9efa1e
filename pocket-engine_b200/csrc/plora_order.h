// What a launch of the path has to know about the launches before it: plain logic, kept apart from the CUDA runtime.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

// The step's grouping kernel lets its successors start early, so nothing that it writes (launch records, unit counts) may be read
// by a kernel that has not waited. A kernel that did wait lets its own successors start only afterwards: from then on launches
// of the same stream may read records ahead of their wait. Calls name a stream each, so this is known per stream: the first
// launch of a step on any stream waits first, whatever other streams did. A stream that captures counts as another one for
// each capture: what is captured is not behind what was launched before, nor what is launched later behind what was captured.
class LaunchOrder {
public:
    struct Stream {
        uint64_t handle, capture;  // capture: the runtime's id of the capture, 0 outside of one
        bool operator==(const Stream& o) const { return handle == o.handle && capture == o.capture; }
    };
    struct Launch {
        bool pdl;   // overlaps the kernel before it (programmatic launch)
        bool late;  // ... and reads nothing that the grouping wrote before its dependency wait
    };
    // The tile words were touched, or a launch did not follow the rules above: the next launch on every stream is a plain one.
    void reset() {
        past_.clear();
        grouped_ = false;
    }
    // The step's grouping was launched.
    void grouped() {
        past_.clear();
        grouped_ = true;
    }
    // How the next kernel on a stream is launched; can_wait: it has a form that waits before it reads.
    Launch next(Stream stream, bool can_wait) const {
        for (const Stream& s : past_)
            if (s == stream) return {true, false};
        return {grouped_ && can_wait, grouped_ && can_wait};
    }
    // That kernel was launched.
    void launched(Stream stream) {
        for (const Stream& s : past_)
            if (s == stream) return;
        if (past_.size() == kMost) past_.erase(past_.begin());  // (that stream's next launch waits once more than it has to)
        past_.push_back(stream);
    }

private:
    static constexpr size_t kMost = 32;
    std::vector<Stream> past_;  // streams with a launch since
    bool grouped_ = false;
};

// Whether a layer's tile shrink may run beside the cluster kernel launched right before it, reading x at once: only if that
// kernel lets it start after its own wait (release 0 is at kernel start), or the caller vouched for x. waits_first: the
// cluster kernel is the first of its step on the stream and waits before anything else.
inline bool tile_shrink_beside(bool tile_late, bool early_x, int release, bool waits_first) { return tile_late && (early_x || release != 0 || waits_first); }
