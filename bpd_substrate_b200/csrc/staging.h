// Host memory that only grows, from a source that may refuse (host code without CUDA).
#pragma once
#include <cstddef>
#include <cstdint>

namespace bpdq {

struct Staging {
    uint8_t* base = nullptr;
    size_t bytes = 0;

    // Whether there are `need` bytes: take(n) gives new memory or null, give(p) takes the old back.  What is refused leaves everything as it was.
    template <class Take, class Give>
    bool reserve(size_t need, Take take, Give give)
    {
        if (need <= bytes) return true;
        uint8_t* more = static_cast<uint8_t*>(take(need));
        if (!more) return false;
        if (base) give(base);
        base = more;
        bytes = need;
        return true;
    }
};

}  // namespace bpdq
