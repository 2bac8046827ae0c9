// fk_workspace.h -- growing a context's device block, and the choice between a
// request's larger and smaller workspace.  Host code only (no CUDA): a CPU test
// drives it with an allocator that refuses.
#pragma once
#include <stddef.h>

namespace fk {

// Size of a block grown to hold `need`: a quarter more, so that slightly larger requests fit too.
inline size_t grown_size(size_t need) { return need + need / 4 + (1u << 20); }

// Replaces the block (base, cap) by one of at least `need` bytes.  The old block is given back
// first; where the new one cannot be had with room to spare it is tried without, and when that
// fails too the old size is taken again, so that what fitted before still does.
// alloc(size_t) returns nullptr when it fails; release(void*).  True: cap >= need.
template <class Alloc, class Release>
bool grow_block(void*& base, size_t& cap, size_t need, Alloc alloc, Release release) {
    const size_t old = cap, sizes[3] = {grown_size(need), need, old};
    if (base) release(base);
    base = nullptr;
    cap = 0;
    for (size_t s : sizes) {
        if (!s || !(base = alloc(s))) continue;
        cap = s;
        break;
    }
    return cap >= need;
}

// Runs a request of FP64 (two_sizes) with its larger workspace where that can be had, else with
// the smaller one.  need(bool larger): bytes; can_hold(bytes): whether trying is worth while;
// ensure(bytes): a status, `ok` for success, `nomem` when memory is short (the smaller one
// is tried then).  Returns ensure's last status; `larger` is the choice.
template <class Status, class Need, class CanHold, class Ensure>
Status choose_workspace(bool two_sizes, bool& larger, Status nomem, Need need, CanHold can_hold, Ensure ensure) {
    if (two_sizes) {
        larger = true;
        const size_t n = need(true);
        if (can_hold(n)) {
            const Status s = ensure(n);
            if (s != nomem) return s;
        }
    }
    larger = false;
    return ensure(need(false));
}

}  // namespace fk
