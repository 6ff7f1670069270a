// Single 32-bit words out of pages that are expensive to get (pinned host memory: about 2 ms a page).  Every taker has a word of
// its own; a page whose words have all come back is given back, except the last one.  No CUDA in here: `get(words)` returns a
// zeroed page or NULL, `put(page)` frees it.
#pragma once
#include <cstdint>
#include <memory>
#include <mutex>
#include <vector>

namespace wick {

template <class Get, class Put, uint32_t WORDS = 1024>
class WordPool {
    struct Page {
        uint32_t* base;
        std::vector<uint32_t> unused;  // indexes; capacity WORDS from the start, so that giving back cannot fail
    };
    std::mutex lock;
    std::vector<std::unique_ptr<Page>> pages;
    Get get;
    Put put;

public:
    WordPool(Get g, Put p) : get(g), put(p) {}

    // NULL: no memory.
    uint32_t* take() {
        std::lock_guard<std::mutex> hold(lock);
        Page* from = nullptr;
        for (auto& p : pages)
            if (!p->unused.empty()) from = p.get();
        if (!from) {
            std::unique_ptr<Page> p(new Page());
            p->unused.reserve(WORDS);
            for (uint32_t i = WORDS; i > 0; i--) p->unused.push_back(i - 1);
            pages.reserve(pages.size() + 1);
            if (!(p->base = get(WORDS))) return nullptr;
            from = p.get();
            pages.push_back(std::move(p));
        }
        const uint32_t i = from->unused.back();
        from->unused.pop_back();
        return from->base + i;
    }

    void give_back(uint32_t* w) {
        std::lock_guard<std::mutex> hold(lock);
        for (size_t n = 0; w && n < pages.size(); n++) {
            Page& p = *pages[n];
            if (w < p.base || w >= p.base + WORDS) continue;
            *w = 0;
            p.unused.push_back((uint32_t)(w - p.base));
            if (p.unused.size() == WORDS && pages.size() > 1) {
                put(p.base);
                pages.erase(pages.begin() + (long)n);
            }
            return;
        }
    }
};

}  // namespace wick
