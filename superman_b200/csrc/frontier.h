// Row-by-row expansion of a sparse real permanent (frontier.cu): the plan the
// kernel takes as its parameter, and the host entry.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "superman_b200.h"

namespace spb {
struct DeviceContext;
namespace frontier {

constexpr int kMaxRows = 63;
constexpr int kMaxEntries = 1024;  // nonzeros a plan holds (9 KB of kernel parameters)
constexpr int kMaxWidth = 22;      // widest state table: 2^22 double-doubles, 64 MiB
// The first steps of a half, while their tables have at most 2^kNarrow states,
// are run by one CTA in shared memory behind block barriers; wider ones by the whole grid behind grid barriers.
constexpr int kNarrow = 11;

struct Step {
    uint32_t closed;   // bits (of the full index) of the columns this row closes
    uint16_t entry;    // first entry of the row in Plan::bit / Plan::val
    uint8_t kb, ka;    // index bits before and after the step
    uint8_t entries;   // nonzeros of the row
    uint8_t used;      // columns of the full index used in a live state
};

// Rows 0 .. nf-1 of the order are taken from the front, rows n-1 .. nf from the
// back; both halves meet at the cut, whose kcut open columns a front state M
// and the back state of the complement share.
struct Plan {
    int n, nf, nb, hf, hb;  // steps of each half, and how many of its first are narrow
    int kcut;
    int total;              // entries
    int exp_sum;            // sum of the row scaling exponents
    int width;              // widest table (index bits)
    double states;          // states visited over all steps
    double abs_bound;       // product of the scaled rows' absolute sums
    Step step[kMaxRows];    // front steps, then back steps
    uint8_t back_bit[24];   // cut column i of the front index -> its bit in the back index
    uint8_t bit[kMaxEntries];  // entry's bit in the step's full index
    double val[kMaxEntries];   // its value, rows scaled to a maximum in [0.5, 1)
};
static_assert(kMaxWidth <= 24 && offsetof(Plan, bit) % 4 == 0 && offsetof(Plan, val) % 8 == 0,
              "the kernel copies the plan in 4-byte words");

// Plans the expansion of the row-major n x n matrix a (finite entries).
// False when a plan does not fit the limits above or visits more states than
// max_states (given up after an order of either orientation).
bool make_plan(const double* a, int n, Plan* plan, double max_states = 1e300);

// States that take the kernel `seconds`, whatever the plan.
double expansion_states(double seconds);

// Estimated device time of the expansion, in seconds.
double expansion_seconds(const Plan& plan);

// Whether the nonzeros of the n x n matrix a hold a perfect matching, n <= 63.
bool has_matching(const double* a, int n);

// Runs the plan; *launched is false when its tables could not be allocated or
// its launch was refused, in which case nothing ran and a walk can.
int run(const Plan& plan, const spb_options* opt, spb_result* out, DeviceContext* own_ctx, bool* launched);

}  // namespace frontier
}  // namespace spb
