// Page-locked words for contexts, kWords doubles each.  Allocating and freeing
// page-locked memory takes 2 ms or more, a context's creation without it 3 ms:
// the slots of one page per device, kept for the process, serve up to kSlots
// contexts at a time, and any more allocate their own.
//
// A page belongs to the device's primary context, and goes with it when the
// program resets the device.  So each slot carries the context's identity
// (`epoch`): a page of another one is forgotten, and a slot of another one is
// not given back into the page that may stand at the same address now.
//
// Api: epoch(device, uint64_t*), alloc(double**, size_t doubles) and
// free(double*), each 0 on success, for the current device.
#pragma once

#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>

namespace khrr {

struct HostWords {
    double* p = nullptr;
    int device = 0;
    uint64_t epoch = 0;
    int slot = -1;  // -1: an allocation of its own
};

template <class Api>
class HostWordPool {
public:
    static constexpr size_t kWords = 32;
    static constexpr int kSlots = 16;

    int take(Api& api, int device, HostWords* out) {
        std::lock_guard<std::mutex> lock(mutex_);
        HostWords w;
        w.device = device;
        if (const int e = api.epoch(device, &w.epoch)) return e;
        Page& page = pages_[device];
        if (page.p && page.epoch != w.epoch) page = Page{};
        if (!page.p) {
            if (const int e = api.alloc(&page.p, kSlots * kWords)) {
                page = Page{};
                return e;
            }
            page.epoch = w.epoch;
        }
        for (int k = 0; k < kSlots && w.slot < 0; ++k)
            if (!(page.used >> k & 1u)) w.slot = k;
        if (w.slot >= 0) {
            page.used |= 1u << w.slot;
            w.p = page.p + w.slot * kWords;
        } else if (const int e = api.alloc(&w.p, kWords)) {
            return e;
        }
        *out = w;
        return 0;
    }

    // After the context's last work on its stream has ended.
    void give(Api& api, const HostWords& w) {
        if (!w.p) return;
        std::lock_guard<std::mutex> lock(mutex_);
        uint64_t now = 0;
        if (api.epoch(w.device, &now) || now != w.epoch) return;  // its memory went with a reset
        if (w.slot < 0) api.free(w.p);
        else if (Page& page = pages_[w.device]; page.epoch == w.epoch) page.used &= ~(1u << w.slot);
    }

private:
    struct Page {
        double* p = nullptr;
        unsigned used = 0;  // one bit per slot
        uint64_t epoch = 0;
    };
    std::mutex mutex_;
    std::map<int, Page> pages_;
};

}  // namespace khrr
