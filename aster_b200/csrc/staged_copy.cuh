// Results to pageable host memory through a page-locked slab (host code; no CUDA
// here, the caller passes the copies and the allocation).
//
// A copy from the device into pageable memory goes through the driver's staging
// on one thread, which also takes the page faults of a caller's freshly
// allocated array: 19 MB (three arrays of 262,153 bodies) took 1.1 to 4.5 ms on
// different hosts, and up to 2.4 more with the faults. Here the bytes come through
// a page-locked slab in 1 MB pieces, and several threads copy them on (on the
// slower host, memory reused / fresh: 4.5 -> 1.4 and 6.9 -> 1.6 ms; 75 MB of 2^20
// bodies 13.0 -> 3.7 and 21.3 -> 5.0; two threads 2.5 and 8.1 ms). The slab is the process's (16 MB,
// allocated by the first large copy, freed with the last context); a copy that
// finds it in use takes the driver's way.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace staged {

constexpr size_t kPiece = (size_t)1 << 20;
constexpr int kSlots = 16;
constexpr int kTeam = 8;  // threads at most (with 2 of the host's left over)
// Below this the driver's copy is used: starting the threads costs some 0.2 ms,
// as much as 2.4 MB take on a fast host.
constexpr size_t kLeast = (size_t)6 << 20;

// The slab. Host: static void* alloc(size_t) (null: none), static void free(void*).
template <class Host>
class Slab {
public:
    char* take() {  // null: in use, or there is none
        std::lock_guard<std::mutex> lock(mu_);
        if (busy_ || failed_) return nullptr;
        if (!base_ && !(base_ = Host::alloc(kPiece * kSlots))) {
            failed_ = true;
            return nullptr;
        }
        busy_ = true;
        return static_cast<char*>(base_);
    }
    void give_back() {
        std::lock_guard<std::mutex> lock(mu_);
        busy_ = false;
        if (contexts_ == 0) drop();
    }
    void contexts(int by) {  // a context more (1) or fewer (-1) that keeps the slab
        std::lock_guard<std::mutex> lock(mu_);
        contexts_ += by;
        if (contexts_ == 0 && !busy_) drop();
    }

private:
    void drop() {  // (the next contexts may have the memory that these did not get)
        if (base_) Host::free(base_);
        base_ = nullptr;
        failed_ = false;
    }
    std::mutex mu_;
    void* base_ = nullptr;
    bool busy_ = false, failed_ = false;
    int contexts_ = 0;
};

struct Piece {
    char* dst;
    const char* src;
    size_t bytes;
};

// The pieces of those arrays whose destination is pageable (null destinations
// skipped): the others take one direct copy each.
inline std::vector<Piece> pieces_of(void* const* dst, const void* const* src, const size_t* bytes, const bool* pageable,
                                    int count) {
    std::vector<Piece> p;
    for (int k = 0; k < count; ++k)
        for (size_t o = 0; dst[k] && pageable[k] && o < bytes[k]; o += kPiece)
            p.push_back({(char*)dst[k] + o, (const char*)src[k] + o, std::min(kPiece, bytes[k] - o)});
    return p;
}

// The pieces through the slab, in order. Dev: bool issue(slot, to, piece) starts
// the copy of a piece's bytes to `to`, bool wait(slot) returns when it has
// arrived; false: failed. Returns whether all have arrived at their
// destinations; after a failure copies may still be on their way to the slab.
template <class Dev>
bool copy(Dev& dev, const std::vector<Piece>& pieces, char* slab) {
    const int n = (int)pieces.size();
    std::atomic<int> ready{0}, taken{0};
    std::atomic<bool> stop{false};
    std::vector<std::atomic<bool>> done(n);
    for (auto& d : done) d.store(false, std::memory_order_relaxed);
    auto copy_next = [&](bool wait) -> bool {  // one piece; false: none left (or, without wait, none ready)
        int k = taken.load();
        do {
            if (k >= n || (!wait && k >= ready.load())) return false;
        } while (!taken.compare_exchange_weak(k, k + 1));
        while (ready.load(std::memory_order_acquire) <= k) {
            if (stop.load()) return false;
            std::this_thread::yield();
        }
        std::memcpy(pieces[k].dst, slab + (size_t)(k % kSlots) * kPiece, pieces[k].bytes);
        done[k].store(true, std::memory_order_release);
        return true;
    };
    std::vector<std::thread> team;
    bool ok = true;
    int issued = 0, arrived = 0;
    auto issue = [&]() {
        for (; issued < n && ok && (issued < kSlots || done[issued - kSlots].load(std::memory_order_acquire)); ++issued)
            ok = dev.issue(issued % kSlots, slab + (size_t)(issued % kSlots) * kPiece, pieces[issued]);
    };
    issue();
    const unsigned hw = std::thread::hardware_concurrency();
    const int want = std::min<int>({n - 1, (int)(hw > 2 ? hw - 2 : 0), kTeam - 1});
    try {
        team.reserve(std::max(want, 0));
        for (int k = 0; k < want; ++k)
            team.emplace_back([&]() {
                while (copy_next(true)) {
                }
            });
    } catch (const std::exception&) {  // no thread or no memory for one: those that run do the work with this one
    }
    while (arrived < n && ok) {
        issue();
        if (!ok) break;
        if (arrived < issued) {
            ok = dev.wait(arrived % kSlots);
            if (ok) ready.store(++arrived, std::memory_order_release);
        } else if (!copy_next(false)) {
            std::this_thread::yield();  // every slot is being copied on
        }
    }
    if (!ok) stop.store(true);
    while (ok && copy_next(true)) {
    }
    for (std::thread& t : team) t.join();
    return ok;
}

}  // namespace staged
