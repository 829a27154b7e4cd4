// Sessions that map and unmap host rows in threads, and copies from and beside them in others: no page is unmapped under a copy, none is
// mapped twice, and all threads end.  Prints OK.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <random>
#include <thread>

#include "../../paraselect_b200/csrc/mapped_rows.h"

using namespace psb;

// Stands in for the driver: which pages are registered, and by which registration.
struct Fake {
    static constexpr uintptr_t kBase = 1 << 20, kPages = 64;
    static std::atomic<int> owner[kPages];   // 0: not registered
    static std::atomic<int> next, maps, wrong;
    struct Reg { uintptr_t begin, end; int id; };
    static std::mutex mu;
    static std::vector<Reg> regs;
    static uintptr_t page(uintptr_t a) { return (a - kBase) / 4096; }
    static Mapping map(const void* p, size_t bytes, int* code) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(p);
        if (bytes == 12345) { *code = 7; return Mapping::kNot; }
        for (uintptr_t x = page(b); x <= page(b + bytes - 1); ++x) if (bytes == 5000 && owner[x]) return Mapping::kOthers;   // as the driver may
        const int id = ++next;
        ++maps;
        std::this_thread::sleep_for(std::chrono::microseconds(id % 5 * 20));
        for (uintptr_t x = page(b); x <= page(b + bytes - 1); ++x) { int none = 0; if (!owner[x].compare_exchange_strong(none, id)) ++wrong; }   // mapped twice
        std::lock_guard<std::mutex> lk(mu);
        regs.push_back({b, b + bytes, id});
        return Mapping::kMapped;
    }
    static void unmap(void* p) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(p);
        std::this_thread::sleep_for(std::chrono::microseconds(next % 3 * 20));
        std::lock_guard<std::mutex> lk(mu);
        for (size_t i = 0; i < regs.size(); ++i) {
            if (regs[i].begin != b) continue;
            for (uintptr_t x = page(b); x <= page(regs[i].end - 1); ++x) owner[x] = 0;
            regs.erase(regs.begin() + (long)i);
            return;
        }
        ++wrong;
    }
};
std::atomic<int> Fake::owner[Fake::kPages], Fake::next, Fake::maps, Fake::wrong;
std::mutex Fake::mu;
std::vector<Fake::Reg> Fake::regs;

int main() {
    MappedRows<Fake> rows;
    auto at = [](uintptr_t off) { return reinterpret_cast<const void*>(Fake::kBase + off); };
    int code = 0;
    bool ok = true;
    // one thread: counted, views, overlaps, neighbours in one page are not overlaps to the counting but share pages
    ok = ok && rows.take(at(100), 9000, &code) == Mapping::kMapped && rows.take(at(200), 50, &code) == Mapping::kMapped;
    ok = ok && rows.take(at(50), 100, &code) == Mapping::kOverlaps;
    rows.give(at(100), 9000);
    ok = ok && Fake::owner[1] != 0;
    rows.give(at(200), 50);
    ok = ok && Fake::owner[0] == 0 && Fake::owner[1] == 0;
    ok = ok && rows.take(at(0), 12345, &code) == Mapping::kNot && code == 7 && rows.take(at(0), 4096, &code) == Mapping::kMapped;
    rows.give(at(0), 4096);
    rows.give(at(0), 4096);   // not there: nothing happens
    ok = ok && rows.take(at(100), 8192, &code) == Mapping::kMapped && rows.take(at(8300), 5000, &code) == Mapping::kOverlaps;   // begins in the last page
    rows.give(at(100), 8192);
    if (!ok) { std::printf("single thread\n"); return 1; }

    std::atomic<bool> stop{false};
    std::atomic<long> copies{0}, sessions{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 5; ++t)
        threads.emplace_back([&, t] {   // sessions over one of three arrays, which share no page
            std::mt19937 rng(t);
            while (!stop) {
                const uintptr_t a = rng() % 3 * 20 * 4096 + 64;
                const size_t n = 15 * 4096;
                int c = 0;
                if (rows.take(at(a), n, &c) != Mapping::kMapped) { ++Fake::wrong; continue; }
                std::this_thread::sleep_for(std::chrono::microseconds(rng() % 100));
                rows.give(at(a), n);
                ++sessions;
            }
        });
    for (int t = 0; t < 4; ++t)
        threads.emplace_back([&, t] {   // copies of the rows, of a part, and of memory in the last page of the one and the first of the next
            std::mt19937 rng(100 + t);
            while (!stop) {
                const uintptr_t a = rng() % 3 * 20 * 4096, b = rng() % 3 * 20 * 4096 + 15 * 4096 + 100;
                MappedRows<Fake>::Copies c(rows, {{at(a + 64), 3 * 4096}, {at(b), 64}, {nullptr, 5}, {at(a), 0}});
                const uintptr_t p0 = Fake::page(Fake::kBase + a + 64), p1 = Fake::page(Fake::kBase + b);
                const int was0 = Fake::owner[p0], was1 = Fake::owner[p1];
                std::this_thread::sleep_for(std::chrono::microseconds(rng() % 60));
                if ((was0 && Fake::owner[p0] != was0) || (was1 && Fake::owner[p1] != was1)) ++Fake::wrong;   // unmapped under the copy
                ++copies;
            }
        });
    std::this_thread::sleep_for(std::chrono::milliseconds(1500));
    stop = true;
    for (auto& t : threads) t.join();
    ok = Fake::wrong == 0 && copies > 100 && sessions > 100 && Fake::maps > 20 && Fake::regs.empty();
    if (!ok) std::printf("wrong %d copies %ld sessions %ld maps %d left %zu\n", Fake::wrong.load(), copies.load(), sessions.load(), Fake::maps.load(), Fake::regs.size());
    else std::printf("OK\n");
    return ok ? 0 : 1;
}
