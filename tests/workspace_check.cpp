// CPU check of csrc/fk_workspace.h with an allocator that refuses blocks above a
// limit (a fragmented device, or another process that took the memory between the
// query and the allocation): a request with two workspace sizes falls back to the
// smaller one, and the old block is there again when nothing larger can be had.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "fk_workspace.h"

namespace {

enum Status { OK, NOMEM, OTHER };

struct Device {
    size_t limit, in_use = 0;
    std::map<void*, size_t> live;
    void* alloc(size_t n) {
        if (in_use + n > limit) return nullptr;
        void* p = std::malloc(1);
        live[p] = n;
        in_use += n;
        return p;
    }
    void release(void* p) {
        in_use -= live.at(p);
        live.erase(p);
        std::free(p);
    }
};

struct Context {
    Device& d;
    void* base = nullptr;
    size_t cap = 0;
    Status ensure(size_t need) {
        if (cap >= need) return OK;
        return fk::grow_block(base, cap, need, [&](size_t n) { return d.alloc(n); }, [&](void* p) { d.release(p); }) ? OK
                                                                                                             : NOMEM;
    }
    // a request of FP64: `can` is what the memory query said
    Status request(size_t small, size_t large, bool can, bool& larger) {
        return fk::choose_workspace(
            true, larger, NOMEM, [&](bool l) { return l ? large : small; }, [&](size_t n) { return cap >= n || can; },
            [&](size_t n) { return ensure(n); });
    }
};

int fail(const char* what) {
    std::printf("FAIL %s\n", what);
    return 1;
}

}  // namespace

int main() {
    const size_t MB = 1u << 20;
    bool larger = false;
    {
        Device d{1000 * MB};
        Context c{d};
        if (c.request(10 * MB, 100 * MB, true, larger) != OK || !larger) return fail("plenty: the larger workspace");
        if (c.cap != fk::grown_size(100 * MB)) return fail("plenty: with room to spare");
        if (c.request(20 * MB, 110 * MB, false, larger) != OK || !larger) return fail("what is there is used");
        if (d.live.size() != 1) return fail("one block at a time");
    }
    {
        Device d{120 * MB};
        Context c{d};
        if (c.request(10 * MB, 110 * MB, true, larger) != OK || !larger || c.cap != 110 * MB)
            return fail("no room to spare: the exact size");
    }
    {
        // the query says yes, the allocation says no: the smaller workspace, not an error
        Device d{60 * MB};
        Context c{d};
        if (c.request(10 * MB, 100 * MB, true, larger) != OK || larger || c.cap < 10 * MB)
            return fail("refused: the smaller workspace");
        const size_t before = c.cap;
        if (c.request(8 * MB, 200 * MB, true, larger) != OK || larger) return fail("refused again");
        if (c.cap != before || d.in_use != before) return fail("the old block is there again");
        if (c.request(80 * MB, 200 * MB, true, larger) != NOMEM) return fail("neither fits: out of memory");
        if (c.cap != before) return fail("and the old block is still there");
        if (c.request(8 * MB, 200 * MB, false, larger) != OK || larger) return fail("the query says no");
    }
    {
        // any other failure is returned as it is
        const Status s = fk::choose_workspace(
            true, larger, NOMEM, [](bool) { return size_t(1); }, [](size_t) { return true; }, [](size_t) { return OTHER; });
        if (s != OTHER || !larger) return fail("other failures are not retried");
    }
    std::printf("ok\n");
    return 0;
}
