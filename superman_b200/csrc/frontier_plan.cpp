// Host planning of the row-by-row expansion (frontier.cu): the order of the
// rows, the index bits of the open columns and where the two halves meet.
#include "frontier.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace spb {
namespace frontier {
namespace {

// The planning loops count bits by the ten thousand: with the instruction
// (every x86-64 host of a CUDA 12 GPU has it), not the compiler's table walk.
#if defined(__x86_64__)
#define SPB_POPCNT __attribute__((target("popcnt")))
#else
#define SPB_POPCNT
#endif

SPB_POPCNT inline int popc(uint64_t x) { return __builtin_popcountll(x); }

// Orders the lines (rows as masks of their columns) greedily: after `start`,
// always the line that leaves the fewest columns open, then the one that opens
// the fewest, then the lowest index.  Returns the number of states of all
// prefixes, 2^(open columns) each, stopping early above `limit`.
SPB_POPCNT double greedy(const std::vector<uint64_t>& line, const std::vector<uint64_t>& cross, int start, double limit,
              std::vector<int>* order)
{
    const int n = (int)line.size();
    uint64_t left = (1ull << n) - 1, open = 0, last = 0;  // last: columns with one line left
    int remain[kMaxRows];
    for (int c = 0; c < n; ++c) {
        remain[c] = popc(cross[c]);
        if (remain[c] == 1) last |= 1ull << c;
    }
    order->clear();
    double states = 0.0;
    int next = start;
    while (true) {
        order->push_back(next);
        left &= ~(1ull << next);
        open = (open | line[next]) & ~(line[next] & last);  // `last` columns close with it
        for (uint64_t m = line[next]; m; m &= m - 1) {
            const int c = __builtin_ctzll(m);
            --remain[c];
            if (remain[c] == 1) last |= 1ull << c;
            else last &= ~(1ull << c);
        }
        states += (double)(1ull << popc(open));
        if (!left || states > limit) return states;
        int best = 1 << 30;
        for (uint64_t m = left; m; m &= m - 1) {
            const int i = __builtin_ctzll(m);
            const int wide = popc(open | line[i]), key = ((wide - popc(line[i] & last)) << 12) | (wide << 6) | i;
            if (key < best) { best = key; next = i; }
        }
    }
}

// Simulates the steps of `rows` (in that order) and fills them at `st`;
// `*front` ends as the open columns in index-bit order.  False past the limits.
bool simulate(const std::vector<uint64_t>& line, const std::vector<uint64_t>& cross, const std::vector<int>& rows,
              const std::vector<double>& val, Plan* p, Step* st, int* entry, std::vector<int>* front)
{
    uint64_t left = 0;
    for (size_t i = 0; i < line.size(); ++i) left |= 1ull << i;
    front->clear();
    int used = 0;
    for (size_t t = 0; t < rows.size(); ++t, ++st) {
        const int r = rows[t];
        left &= ~(1ull << r);
        st->kb = (uint8_t)front->size();
        uint64_t have = 0;
        for (int c : *front) have |= 1ull << c;
        for (uint64_t m = line[r] & ~have; m; m &= m - 1) front->push_back(__builtin_ctzll(m));
        if (front->size() > 31 || *entry + popc(line[r]) > kMaxEntries) return false;
        st->entry = (uint16_t)*entry;
        st->entries = (uint8_t)popc(line[r]);
        st->used = (uint8_t)++used;
        st->closed = 0;
        std::vector<int> rest;
        for (size_t b = 0; b < front->size(); ++b) {
            const int c = (*front)[b];
            if ((line[r] >> c) & 1ull) {
                p->bit[*entry] = (uint8_t)b;
                p->val[*entry] = val[r * line.size() + c];
                ++*entry;
            }
            if (cross[c] & left) rest.push_back(c);
            else { st->closed |= 1u << b; --used; }
        }
        *front = rest;
        st->ka = (uint8_t)front->size();
        if (st->ka > kMaxWidth) return false;
        p->width = std::max(p->width, (int)st->ka);
        p->states += std::ldexp(1.0, st->ka);
    }
    return true;
}

// Augments a matching of rows to columns from row r (columns of `seen` tried).
bool augment(const std::vector<uint64_t>& line, int r, uint64_t* seen, std::vector<int>* row_of)
{
    while (uint64_t m = line[r] & ~*seen) {
        const int c = __builtin_ctzll(m);
        *seen |= 1ull << c;
        if ((*row_of)[c] < 0 || augment(line, (*row_of)[c], seen, row_of)) {
            (*row_of)[c] = r;
            return true;
        }
    }
    return false;
}

}  // namespace

bool has_matching(const double* a, int n)
{
    std::vector<uint64_t> line(n, 0);
    for (int r = 0; r < n; ++r)
        for (int c = 0; c < n; ++c)
            if (a[(size_t)r * n + c] != 0.0) line[r] |= 1ull << c;
    std::vector<int> row_of(n, -1);
    for (int r = 0; r < n; ++r) {
        uint64_t seen = 0;
        if (!augment(line, r, &seen, &row_of)) return false;
    }
    return true;
}

bool make_plan(const double* a, int n, Plan* p, double max_states)
{
    if (n < 2 || n > kMaxRows) return false;
    std::memset(p, 0, sizeof(*p));
    std::vector<uint64_t> rm(n, 0), cm(n, 0);
    for (int r = 0; r < n; ++r)
        for (int c = 0; c < n; ++c)
            if (a[(size_t)r * n + c] != 0.0) {
                rm[r] |= 1ull << c;
                cm[c] |= 1ull << r;
            }
    // the lines with the fewest entries of each orientation as starts
    constexpr int kStarts = 4;
    std::vector<int> order, best_order;
    double best = std::min(max_states, std::ldexp(1.0, kMaxWidth + 4));
    bool transpose = false;
    for (int o = 0; o < 2; ++o) {
        // (a start past the limit leaves no order: the rest rarely differ by
        // enough, and a dense pattern is given up after a few steps)
        const std::vector<uint64_t>&line = o ? cm : rm, &cross = o ? rm : cm;
        std::vector<int> by(n);
        for (int i = 0; i < n; ++i) by[i] = i;
        std::stable_sort(by.begin(), by.end(), [&](int x, int y) { return popc(line[x]) < popc(line[y]); });
        for (int s = 0; s < std::min(n, kStarts); ++s) {
            const double c = greedy(line, cross, by[s], best, &order);
            if (c < best && (int)order.size() == n) {
                best = c;
                best_order = order;
                transpose = o == 1;
            } else if (best_order.empty()) {
                break;
            }
        }
    }
    if (best_order.empty()) return false;
    const std::vector<uint64_t>&line = transpose ? cm : rm, &cross = transpose ? rm : cm;

    // lines scaled by powers of two to a largest entry in [0.5, 1)
    std::vector<double> val((size_t)n * n);
    p->abs_bound = 1.0;
    for (int r = 0; r < n; ++r) {
        double* row = val.data() + (size_t)r * n;
        double mx = 0.0, sum = 0.0;
        for (int c = 0; c < n; ++c) {
            row[c] = transpose ? a[(size_t)c * n + r] : a[(size_t)r * n + c];
            mx = std::max(mx, std::fabs(row[c]));
        }
        int e = 0;
        if (mx > 0.0) std::frexp(mx, &e);
        for (uint64_t m = line[r]; m; m &= m - 1) {
            double& v = row[__builtin_ctzll(m)];
            v = std::ldexp(v, -e);
            sum += std::fabs(v);
        }
        p->exp_sum += e;
        p->abs_bound *= sum;
    }

    // open columns at each cut (after t lines); the halves meet where the
    // wide steps of the longer half are fewest, then where the cut is narrowest
    std::vector<int> open(n + 1, 0);
    uint64_t left = 0, seen = 0;
    for (int i = 0; i < n; ++i) left |= 1ull << i;
    for (int t = 0; t < n; ++t) {
        left &= ~(1ull << best_order[t]);
        seen |= line[best_order[t]];
        for (uint64_t m = seen; m; m &= m - 1) open[t + 1] += (cross[__builtin_ctzll(m)] & left) ? 1 : 0;
    }
    int cut = 0, cost = 1 << 30;
    for (int t = 1; t < n; ++t) {
        int wf = 0, wb = 0;
        for (int i = 1; i <= t; ++i) wf += open[i] > kNarrow;
        for (int i = t; i < n; ++i) wb += open[i] > kNarrow;
        // (the back half's table after the lines n-1 .. i holds the columns open at i)
        const int key = (std::max(wf, wb) << 12) | (std::max(t, n - t) << 6) | std::min(open[t], 63);
        if (key < cost) { cost = key; cut = t; }
    }
    p->n = n;
    p->nf = cut;
    p->nb = n - cut;
    std::vector<int> rows(best_order.begin(), best_order.begin() + cut), ff, bf;
    int entry = 0;
    if (!simulate(line, cross, rows, val, p, p->step, &entry, &ff)) return false;
    rows.assign(best_order.rbegin(), best_order.rbegin() + (n - cut));
    if (!simulate(line, cross, rows, val, p, p->step + cut, &entry, &bf)) return false;
    p->total = entry;
    while (p->hf < p->nf && p->step[p->hf].ka <= kNarrow) ++p->hf;
    while (p->hb < p->nb && p->step[p->nf + p->hb].ka <= kNarrow) ++p->hb;
    p->kcut = (int)ff.size();
    if (ff.size() != bf.size()) return false;
    for (size_t i = 0; i < ff.size(); ++i) {
        const auto it = std::find(bf.begin(), bf.end(), ff[i]);
        if (it == bf.end()) return false;
        p->back_bit[i] = (uint8_t)(it - bf.begin());
    }
    return true;
}

}  // namespace frontier
}  // namespace spb
