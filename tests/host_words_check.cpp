// Replays takes and gives of page-locked words (csrc/host_words.h) against a fake
// of the allocator that hands out the same addresses again after a reset: no two
// live contexts share words, no page is used after its device's reset, and a
// reset of one device leaves the other's words alone.
#include <algorithm>
#include <cstdio>
#include <set>
#include <vector>

#include "host_words.h"

struct Fake {
    uint64_t next = 7, epochs[2] = {1, 2};
    int device = 0;
    std::vector<std::vector<double>> blocks[2];
    std::set<double*> live[2];
    bool fail = false;
    int epoch(int d, uint64_t* e) {
        device = d;
        *e = epochs[d];
        return 0;
    }
    int alloc(double** p, size_t n) {
        if (fail) return 2;
        for (auto& b : blocks[device])
            if (b.size() == n && !live[device].count(b.data())) {  // the same address again
                *p = b.data();
                live[device].insert(*p);
                return 0;
            }
        blocks[device].emplace_back(n);
        *p = blocks[device].back().data();
        live[device].insert(*p);
        return 0;
    }
    int free(double* p) { return live[device].erase(p) == 1 ? 0 : 1; }
    void reset(int d) {
        live[d].clear();
        epochs[d] = next++;
    }
    bool valid(const khrr::HostWords& w) const {
        for (double* p : live[w.device])
            if (w.slot < 0 ? p == w.p : (w.p >= p && w.p < p + 16 * 32)) return true;
        return false;
    }
};

#define CHECK(x) do { if (!(x)) { std::printf("failed: %s (line %d)\n", #x, __LINE__); return 1; } } while (0)

int main() {
    using Pool = khrr::HostWordPool<Fake>;
    Fake api;
    api.blocks[0].reserve(100);
    api.blocks[1].reserve(100);
    Pool pool;
    khrr::HostWords a, b, c, d;
    // One device: a context that lives across a reset gives nothing into the new page.
    CHECK(pool.take(api, 0, &a) == 0 && api.valid(a));
    api.reset(0);
    CHECK(pool.take(api, 0, &b) == 0 && api.valid(b) && b.p == a.p);  // the address is used again
    pool.give(api, a);
    CHECK(pool.take(api, 0, &c) == 0 && api.valid(c) && c.p != b.p);
    // Two devices: a reset of the first leaves the second's words alone.
    CHECK(pool.take(api, 1, &d) == 0 && api.valid(d));
    api.reset(0);
    CHECK(api.valid(d));
    CHECK(pool.take(api, 1, &a) == 0 && api.valid(a) && a.p != d.p && a.device == 1);
    pool.give(api, b);
    pool.give(api, c);
    pool.give(api, d);
    pool.give(api, a);
    // More than a page's contexts, given back in another order and taken again.
    std::vector<khrr::HostWords> held(20);
    for (int round = 0; round < 3; ++round) {
        std::set<double*> seen;
        for (auto& w : held) CHECK(pool.take(api, 0, &w) == 0 && api.valid(w) && seen.insert(w.p).second);
        CHECK(std::count_if(held.begin(), held.end(), [](const khrr::HostWords& w) { return w.slot < 0; }) == 4);
        for (int k = 0; k < 20; ++k) pool.give(api, held[(7 * k + round) % 20]);
        CHECK(api.live[0].size() == 1);  // the page alone
    }
    // An allocation that fails leaves the pool as it was.
    api.reset(0);
    api.fail = true;
    CHECK(pool.take(api, 0, &a) == 2);
    api.fail = false;
    CHECK(pool.take(api, 0, &a) == 0 && api.valid(a));
    std::printf("ok\n");
    return 0;
}
