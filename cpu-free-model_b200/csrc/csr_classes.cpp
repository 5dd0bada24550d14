// Bound: one read of the matrix on the host.  On one thread this took longer than a solve
// saves (128^3 7-point, 14.6 million entries, 16 host threads); here every thread takes
// a chunk of the rows.
#include "csr_classes.h"

#include <omp.h>

#include <algorithm>
#include <atomic>
#include <cstring>

namespace cfm {

namespace {

constexpr int MAX_THREADS = 16;
constexpr int ROWS_PER_THREAD = 1 << 15;  // fewer are not worth a thread

int thread_count(long long items, int asked) {
    const int most = std::min(asked > 0 ? asked : omp_get_max_threads(), MAX_THREADS);
    return asked > 0 ? most : (int)std::min<long long>(most, items / ROWS_PER_THREAD + 1);
}

struct Rows {
    const int *rp, *col;
    const double *val;  // nullptr: offsets alone

    bool same(int i, int j) const {
        const int m = rp[i + 1] - rp[i];
        if (rp[j + 1] - rp[j] != m) return false;
        const int a = rp[i], b = rp[j], d = i - j;
        for (int k = 0; k < m; ++k)
            if (col[a + k] - d != col[b + k]) return false;
        return !val || m == 0 || std::memcmp(val + a, val + b, sizeof(double) * m) == 0;
    }
    unsigned long long hash(int i) const {
        unsigned long long h = (unsigned long long)(rp[i + 1] - rp[i]) + 1;
        auto mix = [&](unsigned long long v) { h = (h ^ v) * 0x9E3779B97F4A7C15ull, h ^= h >> 29; };
        for (int k = rp[i]; k < rp[i + 1]; ++k) {
            mix((unsigned)(col[k] - i));
            if (val) {
                unsigned long long b;
                std::memcpy(&b, val + k, sizeof(b));
                mix(b);
            }
        }
        return h;
    }
};

// Classes found so far, an open-addressed table of their first rows.
struct Table {
    static constexpr int SLOTS = 4 * CLS_MAX;
    int slot[SLOTS], reps[CLS_MAX], count = 0;
    Table() { std::fill(slot, slot + SLOTS, -1); }

    // Class of row i, a new one if it is like none before; -1 when there are too many.
    int find(const Rows &r, int i) {
        int s = (int)(r.hash(i) % SLOTS);
        while (slot[s] >= 0 && !r.same(i, reps[slot[s]])) s = (s + 1) % SLOTS;
        if (slot[s] < 0) {
            if (count == CLS_MAX) return -1;
            slot[s] = count;
            reps[count++] = i;
        }
        return slot[s];
    }
};

// Every chunk's rows into the chunk's own table, then the tables in chunk order into one,
// so classes are numbered by their first rows whatever the chunks.
bool classify(int n, const Rows &r, int threads, RowClasses *out) {
    std::vector<Table> tables(threads);
    std::vector<unsigned char> &cls = out->cls;
    std::atomic<bool> bad{false};
    auto first = [&](int t) { return (int)((long long)n * t / threads); };
#pragma omp parallel for num_threads(threads) schedule(static, 1) if (threads > 1)
    for (int t = 0; t < threads; ++t) {
        Table &tab = tables[t];
        int last = -1;
        for (int i = first(t), e = first(t + 1); i < e; ++i) {
            // a row is compared with its predecessor's class before it is looked up
            if (last < 0 || !r.same(i, tab.reps[last])) {
                if (r.rp[i + 1] - r.rp[i] > CLS_MAXLEN || (last = tab.find(r, i)) < 0) bad = true;
                if (bad.load(std::memory_order_relaxed)) break;
            }
            cls[i] = (unsigned char)last;
        }
    }
    if (bad) return false;
    Table all;
    std::vector<unsigned char> to(threads * CLS_MAX);
    for (int t = 0; t < threads; ++t)
        for (int c = 0; c < tables[t].count; ++c) {
            const int id = all.find(r, tables[t].reps[c]);
            if (id < 0) return false;
            to[t * CLS_MAX + c] = (unsigned char)id;
        }
#pragma omp parallel for num_threads(threads) schedule(static, 1) if (threads > 1)
    for (int t = 1; t < threads; ++t)
        for (int i = first(t), e = first(t + 1); i < e; ++i) cls[i] = to[t * CLS_MAX + cls[i]];
    out->reps.assign(all.reps, all.reps + all.count);
    return true;
}

}  // namespace

RowClasses find_row_classes(int n, const int *rowptr, const int *col, const double *val, int threads) {
    RowClasses out;
    out.cls.resize(n);
    threads = thread_count(n, threads);
    if (classify(n, {rowptr, col, val}, threads, &out))
        out.kind = 2;
    else if (classify(n, {rowptr, col, nullptr}, threads, &out))
        out.kind = 1;
    return out;
}

const char *csr_fault(int n, long long nnz, const int *rowptr, const int *col, int base) {
    bool falls = false, outside = false;
    const int tr = thread_count(n, 0), tc = thread_count(nnz, 0);
#pragma omp parallel for num_threads(tr) schedule(static) reduction(|| : falls) if (tr > 1)
    for (int i = 0; i < n; ++i) falls = falls || rowptr[i + 1] < rowptr[i];
    if (falls) return "rowptr must be non-decreasing";
#pragma omp parallel for num_threads(tc) schedule(static) reduction(|| : outside) if (tc > 1)
    for (long long k = 0; k < nnz; ++k) outside = outside || col[k] < base || col[k] - base >= n;
    return outside ? "column index out of range" : nullptr;
}

void rebase(const int *src, long long count, int base, int *dst) {
    const int t = thread_count(count, 0);
#pragma omp parallel for num_threads(t) schedule(static) if (t > 1)
    for (long long k = 0; k < count; ++k) dst[k] = src[k] - base;
}

}  // namespace cfm
