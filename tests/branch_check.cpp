// CPU check of csrc/fk_branch.h with calls that fail: work on the side stream is
// ordered before what follows join(), or join() reports an error.
#include <cstdio>
#include <string>
#include <vector>

#include "fk_branch.h"

namespace {

struct Fake {
    std::vector<std::string> log;
    int fail_record = -1, fail_wait = -1;  // which call of the kind fails (0: the first)
    int records = 0, waits = 0;
    bool capture = false;
};
using Handle = const char*;

struct Api {
    using Stream = Handle;
    using Event = Handle;
    using Error = int;
    Fake* f;
    int record(Event e, Stream s) {
        if (f->records++ == f->fail_record) return 1;
        f->log.push_back(std::string("record ") + e + " " + s);
        return 0;
    }
    int wait(Stream s, Event e) {
        if (f->waits++ == f->fail_wait) return 2;
        f->log.push_back(std::string("wait ") + s + " " + e);
        return 0;
    }
    int synchronize(Stream s) {
        f->log.push_back(std::string("synchronize ") + s);
        return 0;
    }
    bool capturing(Stream) { return f->capture; }
    void clear() {}
};

std::string go(Fake f, bool side, int* err) {
    Handle current = "main";
    fk::Branch<Api> b(Api{&f}, current, side ? "side" : nullptr, "fork", "joined");
    b.run([&] { f.log.push_back(std::string("work ") + current); });
    *err = b.join();
    f.log.push_back(std::string("then ") + current);
    std::string s;
    for (auto& l : f.log) s += l + "; ";
    return s;
}

int fails = 0;
void want(const char* what, const Fake& f, bool side, const std::string& expect, int expect_err) {
    int err = 0;
    const std::string got = go(f, side, &err);
    if (got == expect && err == expect_err) return;
    std::printf("FAIL %s: %s (%d)\n", what, got.c_str(), err);
    ++fails;
}

}  // namespace

int main() {
    Fake f;
    want("no side stream", f, false, "work main; then main; ", 0);
    want("all well", f, true, "record fork main; wait side fork; work side; record joined side; wait main joined; then main; ", 0);
    f.fail_record = 0;
    want("fork not recorded", f, true, "work main; then main; ", 0);
    f = Fake{};
    f.fail_wait = 0;
    want("fork not waited for", f, true, "record fork main; work main; then main; ", 0);
    f = Fake{};
    f.fail_record = 1;
    want("join not recorded", f, true, "record fork main; wait side fork; work side; synchronize side; then main; ", 0);
    f.capture = true;
    want("join not recorded, capture", f, true, "record fork main; wait side fork; work side; then main; ", 1);
    f = Fake{};
    f.fail_wait = 1;
    want("join not waited for", f, true,
         "record fork main; wait side fork; work side; record joined side; synchronize side; then main; ", 0);
    f.capture = true;
    want("join not waited for, capture", f, true,
         "record fork main; wait side fork; work side; record joined side; then main; ", 2);
    if (!fails) std::printf("ok\n");
    return fails;
}
