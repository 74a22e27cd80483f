// The staged copy (aster_b200/csrc/staged_copy.cuh) with copies made here instead
// of by a device, and allocations that can be made to fail. One command a run:
//   memory N   for k = 0, 1, ..: the k-th allocation after the first copy was
//              issued fails; every copy of N pieces must arrive whole all the same
//   slab 0     the slab's life: refused, in use, given back, freed with the last context
//   pieces 0   which arrays are cut, and how
//   device N   for k = 0, 1, ..: the k-th copy, then the k-th wait, fails: reported
// Prints "ok" and exits 0, or says what was wrong.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <string>

#include "../../aster_b200/csrc/staged_copy.cuh"

static std::atomic<long> g_left{-1};  // allocations until one fails (-1: none does)
void* operator new(size_t n) {
    if (g_left.load() >= 0 && g_left.fetch_sub(1) == 0) throw std::bad_alloc();
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

struct Fake {
    long arm = -1, bad_issue = -1, bad_wait = -1;
    long issued = 0, waited = 0;
    struct {
        char* to;
        staged::Piece p;
    } slot[staged::kSlots];
    bool issue(int s, char* to, const staged::Piece& p) {
        if (issued == 0) g_left.store(arm);
        if (issued++ == bad_issue) return false;
        slot[s] = {to, p};
        return true;
    }
    bool wait(int s) {
        if (waited++ == bad_wait) return false;
        std::memcpy(slot[s].to, slot[s].p.src, slot[s].p.bytes);
        return true;
    }
};

static bool g_refuse = false;
static int g_held = 0;
struct FakeHost {
    static void* alloc(size_t n) {
        if (g_refuse) return nullptr;
        ++g_held;
        return std::malloc(n);
    }
    static void free(void* p) {
        --g_held;
        std::free(p);
    }
};
static int slab_life() {
#define WANT(x)                                              \
    do {                                                     \
        if (!(x)) return std::printf("not so: %s\n", #x), 1; \
    } while (0)
    staged::Slab<FakeHost> s;
    s.contexts(1);
    s.contexts(1);
    WANT(s.take() && g_held == 1);
    WANT(!s.take());  // in use
    s.contexts(-1);
    s.give_back();
    WANT(g_held == 1 && s.take());
    s.contexts(-1);
    WANT(g_held == 1);  // still in use
    s.give_back();
    WANT(g_held == 0);
    g_refuse = true;
    s.contexts(1);
    WANT(!s.take());
    g_refuse = false;
    WANT(!s.take());  // not asked for again by these contexts
    s.contexts(-1);
    s.contexts(1);
    WANT(s.take() && g_held == 1);  // by the next ones it is
    s.give_back();
    s.contexts(-1);
    WANT(g_held == 0);
    std::printf("ok\n");
    return 0;
}

static int pieces_of_arrays() {
    static char a[3 * staged::kPiece], b[10], x[3 * staged::kPiece], y[10];
    void* const dst[4] = {x, y, nullptr, x};
    const void* const src[4] = {a, b, a, a};
    const size_t bytes[4] = {2 * staged::kPiece + 5, 10, 7, 2 * staged::kPiece};
    for (int m = 0; m < 16; ++m) {
        const bool pageable[4] = {(m & 1) != 0, (m & 2) != 0, (m & 4) != 0, (m & 8) != 0};
        size_t got[4] = {0, 0, 0, 0}, want = 0, sum = 0;
        const auto p = staged::pieces_of(dst, src, bytes, pageable, 4);
        int at = 0;  // pieces come in the arrays' order
        for (const auto& q : p) {
            while (at < 4 && (!pageable[at] || !dst[at] || got[at] == bytes[at])) ++at;
            WANT(at < 4 && q.dst == (char*)dst[at] + got[at] && q.src == (const char*)src[at] + got[at]);
            WANT(q.bytes > 0 && q.bytes <= staged::kPiece);
            got[at] += q.bytes;
            sum += q.bytes;
        }
        for (int k = 0; k < 4; ++k)
            if (pageable[k] && dst[k]) want += bytes[k];
        WANT(sum == want);
    }
    std::printf("ok\n");
    return 0;
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    const std::string what = argv[1];
    const int n = std::atoi(argv[2]);
    if (what == "slab") return slab_life();
    if (what == "pieces") return pieces_of_arrays();
    const size_t bytes = (size_t)n * staged::kPiece - 12345;
    std::vector<char> src(bytes), dst(bytes), slab(staged::kPiece * staged::kSlots);
    for (size_t k = 0; k < bytes; ++k) src[k] = (char)(k * 2654435761u >> 11);
    std::vector<staged::Piece> pieces;
    for (size_t o = 0; o < bytes; o += staged::kPiece)
        pieces.push_back({&dst[o], &src[o], std::min(staged::kPiece, bytes - o)});
    auto whole = [&]() { return std::memcmp(src.data(), dst.data(), bytes) == 0; };
    if (what == "memory") {
        for (long k = -1; k < 12; ++k) {
            std::memset(dst.data(), 0, bytes);
            Fake dev;
            dev.arm = k;
            const bool ok = staged::copy(dev, pieces, slab.data());
            g_left.store(-1);
            if (!ok || !whole()) return std::printf("allocation %ld: not whole\n", k), 1;
        }
    } else {
        for (long k = 0; k < n; ++k)
            for (int q = 0; q < 2; ++q) {
                Fake dev;
                (q ? dev.bad_wait : dev.bad_issue) = k;
                if (staged::copy(dev, pieces, slab.data())) return std::printf("%s %ld: not reported\n", q ? "wait" : "copy", k), 1;
            }
    }
    std::printf("ok\n");
    return 0;
}
