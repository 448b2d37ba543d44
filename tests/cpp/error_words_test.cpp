// ErrorWords (csrc/error_words.h) with a host allocator: distinct zeroed words,
// one page kept, further ones given back, pages that a device reset took away,
// several threads.
#include <stdio.h>
#include <stdlib.h>

#include <set>
#include <thread>

#include "error_words.h"

static std::mutex m;
static std::set<int *> live;
static int allocs = 0;

int main()
{
    bool reset = false;
    int *gone = nullptr;
    auto alloc = [&](size_t bytes) {
        std::lock_guard<std::mutex> lock(m);
        ++allocs;
        int *p = (int *)malloc(bytes);
        live.insert(p);
        return p;
    };
    auto release = [&](int *p) {
        std::lock_guard<std::mutex> lock(m);
        if (!live.erase(p)) exit(3);
        free(p);
    };
    auto alive = [&](int *p) { return !(reset && p == gone); };
    lgd::ErrorWords<decltype(alloc), decltype(release), decltype(alive)> words(alloc, release, alive);

    for (int i = 0; i < 1000; ++i) {            // handles made and destroyed one after the other
        int *p = words.take();
        if (*p != 0) return 4;
        *p = 1;
        words.give(p);
    }
    if (allocs != 1 || live.size() != 1) return 5;
    std::vector<int *> taken;                   // many at once: more pages, given back but for one
    for (int i = 0; i < 200; ++i) taken.push_back(words.take());
    if (std::set<int *>(taken.begin(), taken.end()).size() != 200 || live.size() != 4) return 6;
    for (int *p : taken) words.give(p);
    if (live.size() != 1) return 7;
    int *a = words.take();                      // a reset while a handle is alive
    gone = *live.begin();
    reset = true;
    live.erase(gone);
    int *b = words.take();
    if (b == a || live.size() != 1 || *b != 0) return 8;
    words.give(a);                              // of the page that is gone: not released
    words.give(b);
    reset = false;
    if (live.size() != 1) return 9;
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t) {
        threads.emplace_back([&] {
            for (int i = 0; i < 3000; ++i) {
                int *p = words.take(), *q = words.take();
                if (p == q || *p || *q) exit(10);
                *p = *q = 1;
                words.give(p);
                words.give(q);
            }
        });
    }
    for (std::thread& t : threads) t.join();
    if (live.size() != 1) return 11;
    puts("ok");
    return 0;
}
