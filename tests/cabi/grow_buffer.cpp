// The growth rule of the library's prefill scratch against an allocator that refuses what is too large.
#include "grow.h"

#include <cstdio>
#include <vector>

int main() {
    using b200::grow_buffer;
    size_t room = 1000;
    std::vector<size_t> asked;
    std::vector<char *> kept;
    auto alloc = [&](size_t n) -> void * {
        asked.push_back(n);
        if (n > room) return nullptr;
        kept.push_back(new char[n]);
        return kept.back();
    };
    int bad = 0;
    auto expect = [&](bool ok, const char * what) { if (!ok) { printf("wrong: %s\n", what); ++bad; } };

    grow_buffer b;
    expect(b.need(100, 600, alloc) && b.cap == 100, "the first request gets what it asks for");
    void * first = b.p;
    expect(b.need(80, 600, alloc) && b.p == first && asked.size() == 1, "what fits allocates nothing");
    expect(b.need(101, 600, alloc) && b.cap == 150, "growth by half");
    expect(b.need(160, 160, alloc) && b.cap == 160, "growth for its own sake stops at the limit");
    expect(b.need(700, 160, alloc) && b.cap == 700, "a request beyond the limit is met");
    room = 900;
    asked.clear();
    expect(b.need(800, 5000, alloc) && b.cap == 800 && asked.size() == 2 && asked[0] == 1050, "the request itself where half as much again cannot be had");
    asked.clear();
    expect(!b.need(1000, 5000, alloc) && asked.size() == 1 && asked[0] == 1000, "a size above a refused one is not asked for");
    asked.clear();
    for (int i = 0; i < 5; ++i) expect(!b.need(1000, 5000, alloc), "refused");
    expect(asked.empty(), "a refused size is not asked for again");
    expect(b.cap == 800 && b.need(500, 5000, alloc), "the buffer stays");
    expect(b.need(850, 5000, alloc) && b.cap == 850, "a smaller size than the refused one still works");
    for (char * p : kept) delete[] p;
    printf(bad ? "failed\n" : "ok\n");
    return bad != 0;
}
