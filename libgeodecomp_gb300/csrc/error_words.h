// Error words of handles in mapped host memory.  Allocating and freeing one per
// handle took 300 us, twice what the rest of a small grid's create takes; the pool
// hands out words of a page and keeps one page when all have come back.
#ifndef LGD_ERROR_WORDS_H
#define LGD_ERROR_WORDS_H

#include <stddef.h>

#include <mutex>
#include <vector>

namespace lgd {

// ALLOC(bytes) returns memory or throws, RELEASE(p) frees it, ALIVE(p) tells
// whether it still is what ALLOC returned (a device reset takes it away).
template<typename ALLOC, typename RELEASE, typename ALIVE>
class ErrorWords {
public:
    static constexpr int STRIDE = 16;       // ints: a line of 64 bytes per word
    static constexpr int WORDS = 64;        // per page

    ErrorWords(ALLOC alloc, RELEASE release, ALIVE alive) : alloc(alloc), release(release), alive(alive) {}

    // a word that holds 0
    int *take()
    {
        std::lock_guard<std::mutex> lock(mutex);
        for (size_t i = 0; i < pages.size();) {
            if (!alive(pages[i].base)) {
                pages[i].dead = true;
                if (pages[i].used == 0) {
                    pages.erase(pages.begin() + i);
                    continue;
                }
            }
            if (!pages[i].dead && pages[i].used != ~0ull) return word(pages[i]);
            ++i;
        }
        pages.push_back({alloc(sizeof(int) * STRIDE * WORDS), 0, false});
        return word(pages.back());
    }

    // no kernel may write it any more
    void give(int *p)
    {
        std::lock_guard<std::mutex> lock(mutex);
        for (size_t i = 0; i < pages.size(); ++i) {
            const ptrdiff_t at = p - pages[i].base;
            if (pages[i].base > p || at >= STRIDE * WORDS) continue;
            pages[i].used &= ~(1ull << (at / STRIDE));
            if (pages[i].used == 0 && (pages[i].dead || pages.size() > 1)) {
                if (!pages[i].dead) release(pages[i].base);
                pages.erase(pages.begin() + i);
            }
            return;
        }
    }

private:
    struct Page {
        int *base;
        unsigned long long used;
        bool dead;
    };

    static int *word(Page& page)
    {
        int i = 0;
        while (page.used >> i & 1) ++i;
        page.used |= 1ull << i;
        int *p = page.base + i * STRIDE;
        *p = 0;
        return p;
    }

    ALLOC alloc;
    RELEASE release;
    ALIVE alive;
    std::mutex mutex;
    std::vector<Page> pages;
};

}  // namespace lgd

#endif
