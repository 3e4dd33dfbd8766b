// Page-locked staging kept between calls.  A call takes the buffer, queues
// copies out of it and into it, and gives it back at its end.  What it queued
// must have run by then: the next call writes the buffer from the host, with a
// layout of its own.  So a call that returns early, on an error, waits for its
// stream first; one that has waited after its last copy says so (settled) and
// does not wait again.
#pragma once

#include <cstddef>
#include <cstdint>

namespace vrg {

struct Staging {
    uint8_t *ptr = nullptr;
    size_t bytes = 0;
};

// Mem: uint8_t *alloc(size_t) (null: none to be had), void release(uint8_t *), void wait()
template <class Mem>
class StagingLease {
public:
    // keep: the size up to which the buffer stays for the next call
    StagingLease(Staging &b, Mem m, size_t keep) : buf(b), mem(m), kept(keep) {}
    StagingLease(const StagingLease &) = delete;
    StagingLease &operator=(const StagingLease &) = delete;
    ~StagingLease() {
        if (queued) mem.wait();
        if (buf.bytes > kept) drop();
    }
    // the buffer with at least n bytes, or null; copies may be queued from here on
    uint8_t *take(size_t n) {
        if (buf.bytes < n) {
            drop();
            buf.ptr = mem.alloc(n);
            buf.bytes = buf.ptr ? n : 0;
        }
        queued = buf.ptr != nullptr;
        return buf.ptr;
    }
    void settled() { queued = false; }

private:
    void drop() {
        if (buf.ptr) mem.release(buf.ptr);
        buf = Staging{};
    }
    Staging &buf;
    Mem mem;
    size_t kept;
    bool queued = false;
};

}  // namespace vrg
