// Buffers of a handle's calls, kept from call to call: a call takes what it
// needs and gives all of it back at its end.
//
// What is kept is bounded by twice what the largest of the last calls took (at
// least kFloor): every call counts for the kWindow to 2 kWindow calls after it,
// so small calls between large ones (a read-out after every update) do not give
// the large one's buffers away, and a structure that has stopped being used
// that way does.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace cgb {

class KeptBuffers {
  public:
    static constexpr size_t kFloor = 64u << 20;
    static constexpr uint32_t kWindow = 64;

    // A buffer of at least `bytes` bytes: the smallest free one that wastes no
    // more than three quarters of itself, else a new one.  alloc(n): n bytes or
    // nullptr; then the free buffers go first, and nullptr is returned if that
    // does not help.
    template <class Alloc, class Free>
    void* take(size_t bytes, Alloc alloc, Free release) {
        Buf* best = nullptr;
        for (Buf& b : bufs_)
            if (!b.used && b.bytes >= bytes && b.bytes <= 4 * bytes + (1u << 20) && (!best || b.bytes < best->bytes)) best = &b;
        if (!best) {
            size_t room = bytes + bytes / 4;
            void* p = alloc(room);
            if (!p) {
                auto first = std::partition(bufs_.begin(), bufs_.end(), [](const Buf& b) { return b.used; });
                for (auto b = first; b != bufs_.end(); ++b) release(b->p);
                bufs_.erase(first, bufs_.end());
                p = alloc(room = bytes);
            }
            if (!p) return nullptr;
            bufs_.push_back({p, room, false});
            best = &bufs_.back();
        }
        best->used = true;
        call_ += best->bytes;
        return best->p;
    }

    // The call's end, and the start of the next (a call that failed left its
    // buffers out).  Nothing taken and nothing out: not a call.
    template <class Free>
    void give_back(Free release) {
        if (call_ == 0) return;
        size_t total = 0;
        for (Buf& b : bufs_) {
            b.used = false;
            total += b.bytes;
        }
        now_ = std::max(now_, call_);
        call_ = 0;
        const size_t keep = std::max(2 * std::max(now_, before_), kFloor);
        if (++calls_ == kWindow) {
            calls_ = 0;
            before_ = now_;
            now_ = 0;
        }
        if (total <= keep) return;
        std::sort(bufs_.begin(), bufs_.end(), [](const Buf& x, const Buf& y) { return x.bytes < y.bytes; });
        while (total > keep) {  // the largest go first
            total -= bufs_.back().bytes;
            release(bufs_.back().p);
            bufs_.pop_back();
        }
    }

    template <class Free>
    void release_all(Free release) {
        for (Buf& b : bufs_) release(b.p);
        bufs_.clear();
        call_ = now_ = before_ = 0;
        calls_ = 0;
    }

  private:
    struct Buf {
        void* p;
        size_t bytes;
        bool used;
    };
    std::vector<Buf> bufs_;
    size_t call_ = 0;                // taken in the current call
    size_t now_ = 0, before_ = 0;    // most taken by a call of this window, of the one before
    uint32_t calls_ = 0;             // in this window
};

}  // namespace cgb
