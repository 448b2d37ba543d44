// allocate_all (csrc/alloc_all.h) with an allocator that fails at a given call:
// nothing is kept, no pointer stays set, and the next attempt starts over.
#include <stdio.h>
#include <stdlib.h>

#include <set>

#include "alloc_all.h"

int main()
{
    const int n = 9;
    for (int fail_at = 0; fail_at <= n; ++fail_at) {
        void *p[n] = {};
        std::set<void *> live;
        std::vector<lgd::BufferRequest> list;
        for (int i = 0; i < n; ++i) list.push_back({&p[i], (size_t)(16 * (i + 1))});
        for (int attempt = 0; attempt < 3; ++attempt) {
            int calls = 0;
            const bool works = attempt == 2;
            const int rc = lgd::allocate_all(
                list,
                [&](void **out, size_t bytes) {
                    if (!works && calls++ == fail_at) {
                        *out = (void *)0x10;            // a failing allocator may leave anything
                        return 2;
                    }
                    *out = malloc(bytes);
                    live.insert(*out);
                    return 0;
                },
                [&](void *q) {
                    if (!live.erase(q)) exit(3);        // not ours, or twice
                    free(q);
                });
            const bool expect_ok = works || fail_at == n;
            if ((rc == 0) != expect_ok) return 4;
            int set = 0;
            for (int i = 0; i < n; ++i) set += p[i] != nullptr;
            if (set != (expect_ok ? n : 0) || live.size() != (size_t)set) return 5;
            if (expect_ok) break;
        }
        for (int i = 0; i < n; ++i) free(p[i]);
    }
    puts("ok");
    return 0;
}
