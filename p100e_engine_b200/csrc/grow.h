// A buffer that grows: a request that does not fit gets a new allocation, the old one stays where it is (work in flight may use it).
#pragma once
#include <algorithm>
#include <cstddef>

namespace b200 {

struct grow_buffer {
    void * p = nullptr;
    size_t cap = 0;
    size_t refused = (size_t) -1;   // smallest size that could not be had

    // At least `bytes`.  Grows by half, so that a context that gets longer call by call does not allocate in each of them, but not beyond `limit` for
    // that alone.  A size that was refused once is not asked for again: the attempt costs a call milliseconds and may be repeated in every call.
    // alloc(size) returns nullptr on failure.
    template <typename Alloc> bool need(size_t bytes, size_t limit, Alloc alloc) {
        if (bytes <= cap) return true;
        for (const size_t want : {std::max(bytes, std::min(cap + cap / 2, limit)), bytes}) {
            if (want >= refused) continue;
            if (void * q = alloc(want)) {
                p = q;
                cap = want;
                return true;
            }
            refused = want;
        }
        return false;
    }
};

}  // namespace b200
