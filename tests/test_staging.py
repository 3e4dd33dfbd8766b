"""The staging buffer a flush keeps (csrc/staging.h), on the host with a stream
that runs its copies only when it is waited for: the copies that an early
return leaves queued still read what their call wrote, although the next call
writes the same buffer with another layout; a call that has waited does not
wait again; the buffer grows, is kept up to its bound and given back above it."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vulkan-voxel-restir-gi_gb300",
                    "csrc")

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <cstring>
#include <functional>
#include <vector>

#include "staging.h"
using namespace vrg;

std::vector<std::function<void()>> stream;
int waits = 0, allocated = 0, released = 0;
bool none = false;
struct Mem {
    uint8_t *alloc(size_t n) { return none ? nullptr : (allocated++, new uint8_t[n]); }
    void release(uint8_t *p) { released++; delete[] p; }
    void wait() {
        waits++;
        for (auto &f : stream) f();
        stream.clear();
    }
};

// a flush of n bytes: copies them to the device, then its plan (the last 8
// bytes); fails: an error return between the plan's copy and the last wait
bool flush(Staging &b, size_t n, uint8_t fill, bool fails, std::vector<uint8_t> &device, size_t keep = 64) {
    StagingLease<Mem> lease(b, Mem{}, keep);
    uint8_t *h = lease.take(n);
    if (!h) return false;
    device.assign(n, 0);
    memset(h, fill, n - 8);
    memset(h + n - 8, fill ^ 0xFF, 8);
    stream.push_back([h, n, &device] { memcpy(device.data(), h, n); });
    if (fails) return false;
    Mem{}.wait();
    lease.settled();
    return true;
}

bool holds(const std::vector<uint8_t> &d, uint8_t fill) {
    for (size_t i = 0; i < d.size(); i++)
        if (d[i] != (i + 8 < d.size() ? fill : (uint8_t)(fill ^ 0xFF))) return false;
    return !d.empty();
}

int main() {
    Staging b;
    std::vector<uint8_t> d0, d1, d2;
    assert(flush(b, 64, 1, false, d0) && holds(d0, 1) && waits == 1 && allocated == 1);
    assert(!flush(b, 32, 2, true, d1));                       // its copies wait in the stream ...
    assert(flush(b, 48, 3, false, d2));                       // ... and the retry has more chunks
    assert(holds(d1, 2) && holds(d2, 3) && waits == 3 && allocated == 1 && released == 0);
    assert(!flush(b, 500, 4, true, d1) && holds(d1, 4));      // above the bound: waited for, then given back
    assert(b.ptr == nullptr && b.bytes == 0 && allocated == 2 && released == 2);
    none = true;
    assert(!flush(b, 16, 5, false, d0) && b.ptr == nullptr && waits == 4);
    none = false;
    assert(flush(b, 16, 6, false, d0) && holds(d0, 6) && b.bytes == 16);
    assert(flush(b, 20, 7, false, d0) && holds(d0, 7) && b.bytes == 20);  // grows
    puts("staging ok");
}
"""


def test_staging_outlives_what_was_queued(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "staging ok" in r.stdout, r.stdout + r.stderr
