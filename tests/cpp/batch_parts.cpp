// Sub-batches of a batch, and the marks of their slot ranges, at the ends of their range.  Prints OK.
#include <cstdio>

#include "../../paraselect_b200/csrc/batch_parts.h"

using namespace psb;

static bool check(int n, int want, double table_bytes, int at_least) {
    const std::vector<int> cuts = even_cuts(n, part_rows(n, want, table_bytes));
    const size_t parts = cuts.size() - 1;
    bool ok = cuts.front() == 0 && cuts.back() == n && parts >= (size_t)at_least;
    std::vector<int> device(PartMarks::device_words(parts), 0), host(PartMarks::host_words(parts), 0);
    for (size_t p = 0; p < parts && ok; ++p) {
        const size_t d = PartMarks::device_begin(p), h = PartMarks::host_begin(p);
        ok = cuts[p] < cuts[p + 1] && (cuts[p + 1] - cuts[p]) * table_bytes <= 17179869184.0 * 1.01 + table_bytes && d >= 1 && d + 1 < device.size() &&
             h + 1 < host.size();
        if (ok) { ++device[d + 1]; ++host[h]; ++host[h + 1]; }   // each part has an end and a pair of its own
    }
    for (size_t i = 2; i < device.size(); ++i) ok = ok && device[i] == 1;
    for (int v : host) ok = ok && v == 1;
    if (!ok) std::printf("n %d want %d bytes %.0f: %zu parts\n", n, want, table_bytes, parts);
    return ok;
}

int main() {
    bool ok = true;
    for (int want : {1, 4, 32}) {
        for (int n : {1, 2, 3, 31, 2048, 2600, 10000, 65537, 1000003}) ok = check(n, want, 0.0, n >= 1000 * want ? want : 1) && ok;
        ok = check(65537, want, 4096.0 * 64 * 256 * 4, 1025) && ok;       // a table per (query, probe): more than 1,024 parts
        ok = check(200000, want, 4096.0 * 128 * 256 * 4, 6000) && ok;
        ok = check(5, want, 4.0e10, 5) && ok;                             // one query above the limit: a part each
    }
    if (ok) std::printf("OK\n");
    return ok ? 0 : 1;
}
