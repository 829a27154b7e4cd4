// How a batch is cut into sub-batches, and where each sub-batch's range of row slots is noted.  Plain arithmetic, host side only.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace psb {

// Queries per sub-batch: `parts` equal ones, or more where a sub-batch's lookup tables (table_bytes per query; 0: none) would pass 16 GiB.
inline int part_rows(int n, int parts, double table_bytes) {
    if (table_bytes > 0.0) parts = std::max(parts, (int)std::ceil((double)n * table_bytes / (16.0 * 1024 * 1024 * 1024)));
    parts = std::min(parts, std::max(n, 1));
    return (n + parts - 1) / parts;
}

// First query of each sub-batch of `rows` queries, then n.
inline std::vector<int> even_cuts(int n, int rows) {
    std::vector<int> cuts;
    for (long long p0 = 0; p0 < n; p0 += rows) cuts.push_back((int)p0);
    cuts.push_back(n);
    return cuts;
}

// The slot marks of a batch of so many parts.  On the device: the number of slots claimed so far, then 0, then the end of each part's
// range, so that part p's range is words p + 1 and p + 2.  On the host: the two words of each part.  Both arrays are as long as the batch
// has parts: 65,537 queries with 4,096 tables of 64 KiB each are 1,025 parts, and nothing bounds them from above.
struct PartMarks {
    static constexpr size_t device_words(size_t parts) { return parts + 2; }
    static constexpr size_t host_words(size_t parts) { return 2 * parts; }
    static constexpr size_t device_begin(size_t part) { return part + 1; }   // and the word after it, the end
    static constexpr size_t host_begin(size_t part) { return 2 * part; }
};

}  // namespace psb
