// pinned.h - the host ranges pinned through mdg_pin_host and the GPU's addresses of them (hostio.cu).  Host code
// alone, no CUDA.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <map>

namespace mdg {

class PinnedRanges {
public:
    void add(const void* p, size_t bytes, void* device) {
        ranges_[(uintptr_t)p] = {bytes, (uintptr_t)device};
    }
    void remove(const void* p) { ranges_.erase((uintptr_t)p); }
    // The GPU's address of host address p, and into `room` how many of the `bytes` from p on lie in p's range;
    // nullptr and 0 when p is in none.
    void* find(const void* p, size_t bytes, size_t& room) const {
        room = 0;
        const uintptr_t a = (uintptr_t)p;
        auto it = ranges_.upper_bound(a);
        if (it == ranges_.begin()) return nullptr;
        --it;
        const size_t off = a - it->first;
        if (off >= it->second.bytes) return nullptr;
        room = std::min(bytes, it->second.bytes - off);
        return (void*)(it->second.device + off);
    }

private:
    struct Range {
        size_t bytes;
        uintptr_t device;
    };
    std::map<uintptr_t, Range> ranges_;
};

}  // namespace mdg
