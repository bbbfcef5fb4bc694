// spare.cuh — scratch that a call can do without (it has another way): kept between calls, and given back when something that has no other way finds no
// room.  Plain arithmetic (compiled by the host compiler in tests/test_spare_host.py).
#pragma once
#include <algorithm>
#include <cstddef>

// alloc(): 0, or an error.  give_back(): frees the scratch, false if there was none.
template <typename Alloc, typename GiveBack> inline int alloc_or_give_back(Alloc alloc, GiveBack give_back) {
    const int e = alloc();
    return e && give_back() ? alloc() : e;
}

// What scratch of `have` bytes grows to for `want` (have < want <= most): at least twice what it was, so that a conversation whose portions ask for a little
// more each time allocates (and waits for the device) a few times in all; never above `most`.
inline size_t grown(size_t have, size_t want, size_t most) { return std::min(most, std::max(want, 2 * have)); }

// When scratch that found no room is asked for again.  Asking costs 0.3 ms where there is none, more than a small step takes (eight sequences through two 2048-wide layers
// on a full device: 582 us when every step asked, 250 without): so not at every call, but after 1, 2, 4, .. 64 calls without it.
struct SpareRetry {
    int wait = 0, next = 1;
    bool due() { return wait == 0 || --wait == 0; }
    void failed() {
        wait = next + 1;
        next = std::min(64, 2 * next);
    }
    void got() {
        wait = 0;
        next = 1;
    }
};
