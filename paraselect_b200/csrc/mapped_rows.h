// Host rows that sessions have mapped for the device, and the copies of host memory that are under way.  Host side only; Rt maps and unmaps.
#pragma once

#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <initializer_list>
#include <list>
#include <mutex>
#include <utility>
#include <vector>

namespace psb {

// Ranges are counted over the sessions that read them: several sessions may lie over one array (a session per query thread, or per view of
// it), and the mapping ends with the last of them, whichever made it.  A copy between the device and host memory that shares a page with a
// mapped range may be a transfer straight from these pages; were they unmapped meanwhile, it would fault.  So the copies of every call are noted
// while they may be under way, an unmapping waits for those over its pages, and a call that would begin one meanwhile waits for the unmapping.
// Mapping and unmapping, which take seconds for large arrays, hold up nobody else.
//   Rt::map(begin, bytes, code)   kMapped; kOthers: the caller itself has the range registered, which is then the caller's to end; kNot: *code says why
//   Rt::unmap(begin)
enum class Mapping { kMapped, kOthers, kNot, kOverlaps };   // kOverlaps: of MappedRows::take, only some of the rows' pages are mapped
template <typename Rt>
class MappedRows {
    struct Range { uintptr_t begin, end; int users; enum { kComing, kHere, kGoing } state; };
    struct Span { uintptr_t begin, end; };
    static constexpr uintptr_t kPage = 4096;
    static Span pages(uintptr_t b, uintptr_t e) { return {b / kPage * kPage, (e + kPage - 1) / kPage * kPage}; }
    static bool meet(const Span& a, const Span& b) { return a.begin < b.end && b.begin < a.end; }
public:
    // give() has to follow kMapped, and nothing else.  Not while this thread has Copies.
    Mapping take(const void* rows, size_t bytes, int* code) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(rows), e = b + bytes;
        std::unique_lock<std::mutex> lk(mu_);
        for (bool again = true; again;) {
            again = false;
            for (Range& r : ranges_) {
                if (!meet(pages(r.begin, r.end), pages(b, e))) continue;
                if (r.state != Range::kHere) { change_.wait(lk); again = true; break; }
                if (r.begin <= b && e <= r.end) { ++r.users; return Mapping::kMapped; }
                if (r.begin < e && b < r.end) return Mapping::kOverlaps;
            }
        }
        ranges_.push_back(Range{b, e, 1, Range::kComing});
        const auto mine = std::prev(ranges_.end());
        lk.unlock();
        const Mapping got = Rt::map(rows, bytes, code);
        lk.lock();
        if (got == Mapping::kMapped) mine->state = Range::kHere;
        else ranges_.erase(mine);
        change_.notify_all();
        if (got == Mapping::kOthers)   // unless the registration that was met is one of these, of an array that ends or begins in the same page
            for (const Range& r : ranges_) if (meet(pages(r.begin, r.end), pages(b, e))) return Mapping::kOverlaps;
        return got;
    }
    void give(const void* rows, size_t bytes) {
        const uintptr_t b = reinterpret_cast<uintptr_t>(rows), e = b + bytes;
        std::unique_lock<std::mutex> lk(mu_);
        for (auto r = ranges_.begin(); r != ranges_.end(); ++r) {
            if (r->state != Range::kHere || b < r->begin || r->end < e) continue;
            if (--r->users > 0) return;
            r->state = Range::kGoing;
            change_.wait(lk, [&] {
                for (const Span& c : copies_) if (meet(c, pages(r->begin, r->end))) return false;
                return true;
            });
            lk.unlock();
            Rt::unmap(reinterpret_cast<void*>(r->begin));
            lk.lock();
            ranges_.erase(r);
            change_.notify_all();
            return;
        }
    }
    // The host memory that a call copies to or from, from before its first copy until its last has ended; all of it at once, for a call
    // that waited with some noted could wait for itself.
    class Copies {
    public:
        Copies(MappedRows& all, std::initializer_list<std::pair<const void*, size_t>> spans) : all_(all) {
            std::vector<Span> want;
            for (const auto& s : spans)
                if (s.first && s.second) want.push_back(pages(reinterpret_cast<uintptr_t>(s.first), reinterpret_cast<uintptr_t>(s.first) + s.second));
            if (want.empty()) return;
            std::unique_lock<std::mutex> lk(all_.mu_);
            all_.change_.wait(lk, [&] {
                for (const Range& r : all_.ranges_)
                    if (r.state == Range::kGoing)
                        for (const Span& s : want) if (meet(s, pages(r.begin, r.end))) return false;
                return true;
            });
            for (const Span& s : want) { all_.copies_.push_back(s); mine_.push_back(std::prev(all_.copies_.end())); }
        }
        Copies(const Copies&) = delete;
        Copies& operator=(const Copies&) = delete;
        ~Copies() {
            if (mine_.empty()) return;
            { std::lock_guard<std::mutex> lk(all_.mu_); for (auto at : mine_) all_.copies_.erase(at); }
            all_.change_.notify_all();
        }
        bool any() const { return !mine_.empty(); }
    private:
        MappedRows& all_;
        std::vector<typename std::list<Span>::iterator> mine_;
    };
private:
    std::mutex mu_;
    std::condition_variable change_;   // of ranges_ or copies_
    std::list<Range> ranges_;
    std::list<Span> copies_;
};

}  // namespace psb
