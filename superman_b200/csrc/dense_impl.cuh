// Dense walk kernels (real and complex), shared between the driver in
// dense.cu and the per-n instantiation units dense_walk_{real,complex}.cu.
#pragma once

#include <cuda_runtime.h>

#include "spb_common.cuh"

namespace spb {
namespace dense {

constexpr int kMaxN = 63;
// Smallest n of the derivative walk in whole-GPU calls.  Below, picking the
// pivot and dividing by it cost the call more than the walk saves (FP64 calls
// on one B200, plain against derivative: real n=20 43.6 and 47.1 us, n=22 51.0 and
// 52.0, n=23 with double-double 45.6 and 48.2 of device time, n=24 75.5 and 70.5; complex n=21
// 95.4 and 97.4, n=23 133.5 and 130.9).
constexpr int kMinDerivReal = 24, kMinDerivComplex = 22;

// Everything the host reads back after a call, contiguous so that one copy
// brings it over: a call costs one host round trip, the double-double
// refinement included (its threshold is picked on the device).
struct Readback {
    dd res[2];                  // [comps] the walk's total
    dd corr[2];                 // [comps] the refinement's correction
    unsigned long long list_n;  // units listed for the refinement
    unsigned long long count;   // units the histogram puts at or above thr
    double err;                 // SPB_PREC_DD: expected relative error of the unrefined units;
                                // SPB_PREC_FP32: the walk's sum of squared terms
    int thr;                    // refinement bin
    int from_list;              // 1: the walk's own list holds every unit at or above thr
    int exp_sum;                // sum of the row scaling exponents
    int pivot;                  // derivative walk: the column the rows are divided by; -1: plain walk
    dd scale[2];                // derivative walk: [comps] product of the pivots' mantissas
    int scale_exp;              // and the sum of their exponents
    int pad;
    // Nanosecond stamps of the device's global timer: the call's first kernel
    // begins, the walk begins, the walk ends, the readback is complete.  Calls of
    // up to kStampedMaxN take their device times from them: events around the
    // kernels and the queries of their times cost such a call 5 to 12 us.
    unsigned long long stamp[4];
};
constexpr int kStampedMaxN = 26;

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Device-side description of one permanent: sizes plus pointers into the
// scratch arena written by setup_kernel.
struct Problem {
    int n, comps, w, g, grid, threads;
    int na;                    // rows that vary within a unit: n (dense walk) or the
                               // active rows of the row-compacted walk (sparse_impl.cuh)
    unsigned long long units;  // 2^(n-1-w) Gray units of 2^w terms each (the derivative walk
                               // takes half of them, eff_units)
    int deriv;                 // 1: the derivative walk runs if the matrix has a pivot column
                               // (rb->pivot, set by the setup kernel); 0: the plain walk
    double* x0_hi;             // [comps][n] NW start vector, double-double
    double* x0_lo;
    double* de_hi;             // [comps][2^w/G][n][G] low-column subset sums
    double* de_lo;             // rounding residues of de_hi
    float* de32;               // SPB_PREC_FP32: de_hi rounded to float (else null)
    int f32;                   // 1: the FP32-product walk runs (tables include de32)
    double* mt;                // [comps][ntop][n] high columns
    double* mt_lo;             // their low words (derivative walk)
    dd* partials;              // [comps][grid] per-CTA sums
    unsigned* ticket;          // last-CTA election counter (reset by the kernel)
    dd* result;                // [comps] grid total (rb->res; rb->corr for the refinement)
    int* exp_sum;              // sum of the row scaling exponents (&rb->exp_sum)
    Readback* rb;
    Readback* rb_host;         // the device's address of the host's page-locked copy of *rb; the
                               // call's last kernel fills it (null in the others, and where the
                               // host copies the readback itself)
    int timed;                 // nonzero: the kernels stamp their times (2: fetch_kernel takes the first)
    double tol;                // SPB_PREC_DD: relative tolerance of the threshold
    // Double-double refinement (SPB_PREC_DD); unused when mode == 0.
    int mode;                  // 0 walk, 1 walk + unit-bound histogram, 2 scan only
    int thr_bin;               // mode 2: list the units whose bound bin >= thr_bin
    double* bnd;               // real [2][n] min/max of DE over d; complex [n] max |DE|
    double* hist_s2;           // [kHistBins] sum of squared terms of the units per bin
    unsigned long long* hist_cnt;  // [kHistBins] units per bin
    unsigned long long* list_n;    // number of listed units (&rb->list_n)
    unsigned long long list_cap;
    unsigned long long* list_u;    // [list_cap] unit index
    double* list_x;                // [list_cap][comps][2][n] unit base, hi then lo
    unsigned short* tmax;          // [grid*threads] highest bound bin of each thread's units
    // Mode 1 direct listing: bound_walk counts the units per bound bin
    // (pre_cnt), pick_list_bin sets *list_bin to the lowest bin whose tail fits
    // raw_cap, and the walk appends every unit at or above it (raw_*).
    unsigned* pre_cnt;             // [kHistBins]
    int* list_bin;
    unsigned long long* raw_n;
    unsigned long long raw_cap;
    unsigned long long* raw_u;     // [raw_cap] unit index
    unsigned short* raw_b;         // [raw_cap] its bound bin
};

// Capacity of the mode-1 list (units; 10 bytes each, 21 MB).  A walk of at
// most kRawCap / 2 units (real n <= 29, complex n <= 28 at the default unit
// width) lists every unit and needs no bound pass; larger walks list from
// the bin pick_list_bin chooses, aiming at kRawTarget units, far below the
// capacity so that bins computed by the walk and by bound_walk may differ at
// bin edges.  The units the refinement takes (a few hundred to a few thousand
// from n = 27 to 32) fit that target many times over, and every listed unit
// costs the walk an append.
constexpr unsigned long long kRawCap = 1ull << 21;
constexpr unsigned long long kRawTarget = 1ull << 14;
constexpr int kListNone = 0x7f7f7f7f;  // a list bin above every bin

// Derivative walk.  The permanent is linear in a column; expanded along
// column c it is the sum over rows r of a_rc times the minor without r and c,
// and one Nijenhuis-Wilf walk over the other n-1 columns (2^(n-2) subsets, half
// of the plain walk's) evaluates all minors together: with every row divided
// by its pivot a_rc,
//   perm(A) = prod_r a_rc * (4((n-1)%2)-2) * sum_S (-1)^|S| q_S,
//   q_S = sum_r prod_{r' != r} x_r'(S),
// the derivative of prod_r (x_r + t) at t = 0.  The chain q <- q x + p, p <- p x
// costs an add, a multiply and a fused multiply-add per row where the two
// plain terms it stands for cost two adds and two multiplies: 3/4 of the FP64
// instructions, with the same or a smaller rounding error.  The quotients are
// kept in double-double wherever the plain walk holds exact entries (start
// vector, subset sums, high columns).
// Where the high columns' low words lie during the walk: beside the columns in
// shared memory, or, at sizes whose tables and per-thread words leave no room
// there without taking threads from the CTA, in global memory.  They are read
// once per unit of 64 or 128 terms, mostly the same column by all threads.  One
// B200: real n=40 2292 ms with the words in shared memory and 480 threads, 2198 ms
// here with 512 (plain walk 3014 ms); complex n=37 994 ms with 224 threads, 804 ms
// with 256 (1045 ms).
__host__ __device__ constexpr bool deriv_low_far(int n, int comps) { return n >= (comps == 1 ? 40 : 37); }
// Whether the derivative walk runs; the same for every thread of a call.
__device__ __forceinline__ bool deriv_on(const Problem& pb) { return pb.deriv != 0 && pb.rb->pivot >= 0; }
__device__ __forceinline__ int eff_ntop(const Problem& pb, bool deriv) { return pb.n - 1 - pb.w - (deriv ? 1 : 0); }
__device__ __forceinline__ unsigned long long eff_units(const Problem& pb, bool deriv)
{
    return deriv ? pb.units >> 1 : pb.units;
}

// a + m, the sum normalised, low words added first: about 2^-105 off.
__device__ __forceinline__ dd dd_step(dd a, double mh, double ml)
{
    const dd s = two_sum(a.hi, mh);
    return fast_two_sum(s.hi, add_rn(s.lo, add_rn(a.lo, ml)));
}

// Pivot column of an n x n matrix whose rows are scaled to maxima in [0.5, 1);
// mag(r, j) is entry (r, j)'s magnitude (complex: the larger of its parts).
// The column whose smallest magnitude is largest; -1 when every column holds a
// zero or a non-finite entry, or when dividing by the pivots could take what the
// walk forms out of the FP64 range.  A row value of the walk is below n, n over
// its pivot after the division, so a term is below n 2^bits, with `bits` the
// pivots' exponents and log2 n added up over the rows.  Without refinement
// (`squares` false) terms are only added up, 2^62 of them at most: 900 bits.  The
// refinement sums their squares and squares the total: 420 bits (terms below
// 2^426, squares 2^852, their sum 2^914, the total's square 2^976).  Called by
// one full warp; every lane returns the same.
template <class Mag>
__device__ __forceinline__ int pick_pivot(int n, bool squares, Mag mag)
{
    const int lane = threadIdx.x & 31;
    const int log2n = 32 - __clz(n), most = squares ? 420 : 900;
    double best = 0.0;
    int col = -1;
    for (int j = lane; j < n; j += 32) {
        double lo = INFINITY;
        int bits = 0;
        bool ok = true;
        for (int r = 0; r < n; ++r) {
            const double m = mag(r, j);
            const int em = (__double2hiint(m) >> 20) & 0x7ff;
            ok = ok && em != 0 && em != 0x7ff;
            bits += 1023 + log2n - em;
            lo = fmin(lo, m);
        }
        if (ok && bits <= most && lo > best) {
            best = lo;
            col = j;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double b = __shfl_xor_sync(0xffffffffu, best, off);
        const int c = __shfl_xor_sync(0xffffffffu, col, off);
        if (b > best || (b == best && c >= 0 && (col < 0 || c < col))) {
            best = b;
            col = c;
        }
    }
    return col;
}
// The same on a row-major array of scaled entries, COMPS interleaved.
template <int COMPS>
__device__ __forceinline__ int pick_pivot(const double* a, int n, bool squares)
{
    return pick_pivot(n, squares, [&](int r, int j) {
        const double* e = a + ((size_t)r * n + j) * COMPS;
        return COMPS == 1 ? fabs(e[0]) : fmax(fabs(e[0]), fabs(e[COMPS - 1]));
    });
}

struct ddc {
    dd re, im;
};
__device__ __forceinline__ ddc ddc_mul(ddc a, ddc b)
{
    return {dd_add(dd_mul(a.re, b.re), dd_neg(dd_mul(a.im, b.im))),
            dd_add(dd_mul(a.re, b.im), dd_mul(a.im, b.re))};
}

// Product of the n pivots as mantissa and exponent, formed by a full warp (every
// lane returns it); get(r) is row r's pivot as {re, im}.
struct DerivScale {
    ddc v;
    int e;
};
template <int COMPS, class Get>
__device__ __forceinline__ DerivScale deriv_scale(int n, Get get)
{
    const int lane = threadIdx.x & 31;
    DerivScale s{{{1.0, 0.0}, {0.0, 0.0}}, 0};
    for (int r = lane; r < n; r += 32) {
        const double2 d = get(r);
        int e = 0;
        if (COMPS == 1) {
            const double m = frexp(d.x, &e);
            s.v.re = dd_mul(s.v.re, dd{m, 0.0});
        } else {
            frexp(fmax(fabs(d.x), fabs(d.y)), &e);
            s.v = ddc_mul(s.v, ddc{{ldexp(d.x, -e), 0.0}, {ldexp(d.y, -e), 0.0}});
        }
        s.e += e;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const ddc o = {shfl_xor_dd(s.v.re, off), shfl_xor_dd(s.v.im, off)};
        if (COMPS == 1) s.v.re = dd_mul(s.v.re, o.re);
        else s.v = ddc_mul(s.v, o);
        s.e += __shfl_xor_sync(0xffffffffu, s.e, off);
    }
    return s;
}

// x / d as a double-double (to about 2^-105), d not zero.
__device__ __forceinline__ dd quotient(double x, double d)
{
    const double h = __ddiv_rn(x, d);
    return dd{h, __ddiv_rn(__fma_rn(-h, d, x), d)};
}

// (xr + i xi) / (dr + i di) in double-double, to about 2^-102 of its magnitude.
// Both are first scaled by the power of two that takes the divisor's larger
// part to [0.5, 1): of a divisor below 2^-460 the squares and their errors
// would leave the FP64 range.
__device__ __forceinline__ ddc quotient_c(double xr, double xi, double dr, double di)
{
    int e = 0;
    frexp(fmax(fabs(dr), fabs(di)), &e);
    dr = ldexp(dr, -e);
    di = ldexp(di, -e);
    xr = ldexp(xr, -e);
    xi = ldexp(xi, -e);
    auto prod = [](double a, double b) {
        const double p = __dmul_rn(a, b);
        return dd{p, __fma_rn(a, b, -p)};
    };
    auto div = [](dd a, dd b) {
        const double h = __ddiv_rn(a.hi, b.hi);
        const dd r = dd_add(a, dd_neg(dd_mul(dd{h, 0.0}, b)));
        return fast_two_sum(h, __ddiv_rn(r.hi, b.hi));
    };
    const dd den = dd_add(prod(dr, dr), prod(di, di));
    return {div(dd_add(prod(xr, dr), prod(xi, di)), den), div(dd_add(prod(xi, dr), dd_neg(prod(xr, di))), den)};
}

// Appends unit u (bound bin b) to the mode-1 list when b >= lbin.  The
// appending lanes of a warp take their slots with one atomic (a leader
// reserves popc of them), not one each.
__device__ __forceinline__ void raw_list_add(const Problem& pb, int lbin, unsigned long long u, int b)
{
    const unsigned act = __activemask();
    const bool want = b >= lbin;
    const unsigned m = __ballot_sync(act, want);
    if (!want) return;
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(pb.raw_n, (unsigned long long)__popc(m));
    base = __shfl_sync(m, base, leader);
    const unsigned long long k = base + (unsigned long long)__popc(m & ((1u << lane) - 1u));
    if (k < pb.raw_cap) {
        pb.raw_u[k] = u;
        pb.raw_b[k] = (unsigned short)b;
    }
}

// Unit-bound histogram: bin = (ilogb(U) + 1024) / 4, i.e. four octaves per bin.
constexpr int kHistBins = 512;

__device__ __forceinline__ int hist_bin(double u)
{
    if (!(u > 0.0)) return 0;
    if (!isfinite(u)) return kHistBins - 1;
    int b = (ilogb(u) + 1024) >> 2;
    return b < 0 ? 0 : (b >= kHistBins ? kHistBins - 1 : b);
}

// Shared memory the histogram needs (reserved in every mode so the walk and
// the scan run with the same launch shape, hence the same unit split).  Per
// bin: the sum of squared terms as a float scaled by 2^(-8(b-256)) (bin b
// holds bounds below 2^(4(b-256)+4), so a unit adds at most 2^(w+8)), and a
// 32-bit count; both have native shared-memory atomics.
constexpr size_t kHistSmemBytes = kHistBins * (sizeof(float) + sizeof(unsigned));
// Shared memory for the per-row bound terms (two per row, real or complex).
__host__ __device__ constexpr size_t bound_smem_bytes(int n) { return sizeof(double) * 2 * n; }

// 2^(4(b-256)) for bins 1..511 (bin 0 holds zero bounds, whose terms are 0),
// built from the exponent field; the histogram scale is its square.
__device__ __forceinline__ double hist_half_scale(int bin)
{
    const int b = bin < 1 ? 1 : bin;
    return __hiloint2double((1023 + 4 * (b - 256)) << 20, 0);
}
__device__ __forceinline__ double hist_half_unscale(int bin)
{
    const int b = bin < 1 ? 1 : bin;
    return __hiloint2double((1023 - 4 * (b - 256)) << 20, 0);
}

// Per-thread cache of the histogram: shared-memory atomics are issued only
// when a thread's bin changes from one unit to the next.
struct HistCache {
    int bin = -1;
    double s2 = 0.0;
    unsigned cnt = 0;
    __device__ __forceinline__ void add(int b, double v, float* s_hist, unsigned* s_cnt)
    {
        if (b != bin) {
            flush(s_hist, s_cnt);
            bin = b;
        }
        s2 += v;
        ++cnt;
    }
    __device__ __forceinline__ void flush(float* s_hist, unsigned* s_cnt)
    {
        if (cnt) {
            const double h = hist_half_unscale(bin);
            atomicAdd(&s_hist[bin], __double2float_rn((s2 * h) * h));
            atomicAdd(&s_cnt[bin], cnt);
        }
        s2 = 0.0;
        cnt = 0;
    }
};

// Flushes a CTA's shared histogram into the global one (double, 64-bit).
__device__ __forceinline__ void flush_hist(const float* s_hist, const unsigned* s_cnt, const Problem& pb)
{
    for (int i = threadIdx.x; i < kHistBins; i += blockDim.x)
        if (s_cnt[i]) {
            atomicAdd(&pb.hist_cnt[i], (unsigned long long)s_cnt[i]);
            const double h = hist_half_scale(i);
            atomicAdd(&pb.hist_s2[i], ((double)s_hist[i] * h) * h);
        }
}

// Thread caps keep the x vector (2 registers per double) plus the product
// chains under the per-thread register budget the cap implies
// (65536 / threads), so the walk never spills at the sizes that matter.
__host__ __device__ constexpr int RealMaxThreads(int n) { return n <= 40 ? 512 : 256; }
__host__ __device__ constexpr int ComplexMaxThreads(int n) { return n <= 10 ? 512 : (n <= 20 ? 384 : 256); }

template <int N>
struct RealCfg {
    static constexpr int G = N >= 3 ? 4 : (N == 2 ? 2 : 1);
    static constexpr int kMaxThreads = RealMaxThreads(N);
};

// Complex groups: four independent term chains per component while the
// x vector leaves room for them in registers (n <= 32), two beyond.
__host__ __device__ constexpr int ComplexGroup(int n) { return (n >= 3 && n <= 32) ? 4 : (n >= 2 ? 2 : 1); }

template <int N>
struct ComplexCfg {
    static constexpr int G = ComplexGroup(N);
    static constexpr int kMaxThreads = ComplexMaxThreads(N);
};

__device__ __forceinline__ dd ldcg_dd(const dd* p)
{
    return {__ldcg(&p->hi), __ldcg(&p->lo)};
}

// p[lane] + p[lane + 32] + ... over the entries below count, added in that
// order; the loads (through L2) are issued eight at a time ahead of the adds,
// so a lane waits for one round trip per eight entries, not one per entry.
__device__ __forceinline__ dd lane_sum_dd(const dd* p, int count, int lane)
{
    dd v = {0.0, 0.0};
    for (int b0 = lane; b0 < count; b0 += 32 * 8) {
        dd x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = b0 + 32 * k < count ? ldcg_dd(p + b0 + 32 * k) : dd{0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (b0 + 32 * k < count) v = dd_add(v, x[k]);
    }
    return v;
}

// Copies the finished readback to the host's page-locked copy (mapped into
// the device's address space), reading it through L2: its fields were
// written by other CTAs and kernels (and by lane 0 of this warp).  The host then
// needs no copy after the call.  Called by a full warp, a word per lane: the
// stores leave for the host link together, where one thread's 22 of them took
// the fused call 2 to 4 us longer (n=20 FP64 21.7 -> 18.8 us of kernel time).
__device__ __forceinline__ void publish(const Problem& pb, Readback* host)
{
    if (!host) return;
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        if (pb.timed) pb.rb->stamp[3] = global_ns();
        __threadfence();
    }
    __syncwarp();
    constexpr int kWords = (int)(sizeof(Readback) / sizeof(unsigned long long));
    static_assert(sizeof(Readback) % sizeof(unsigned long long) == 0 && kWords <= 32, "an 8-byte word per lane");
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(pb.rb);
    if (lane < kWords) reinterpret_cast<unsigned long long*>(host)[lane] = __ldcg(src + lane);
}

// Warp -> block -> grid double-double reduction of C components.  The last
// CTA to finish (ticket election) sums the per-CTA partials in index order,
// so the result does not depend on CTA completion order.
template <int C>
__device__ __forceinline__ void grid_reduce(dd (&tot)[C], const Problem& pb)
{
    __shared__ dd s_warp[C][32];
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int c = 0; c < C; ++c) tot[c] = warp_sum_dd(tot[c]);
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) s_warp[c][wid] = tot[c];
    }
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
            dd v = lane < nw ? s_warp[c][lane] : dd{0.0, 0.0};
            v = warp_sum_dd(v);
            if (lane == 0) pb.partials[c * pb.grid + blockIdx.x] = v;
        }
        if (lane == 0) {
            __threadfence();
            unsigned prev = atomicAdd(pb.ticket, 1u);
            s_last = (prev == gridDim.x - 1) ? 1 : 0;
        }
    }
    __syncthreads();
    if (s_last && wid == 0) {
        __threadfence();
#pragma unroll
        for (int c = 0; c < C; ++c) {
            dd v = lane_sum_dd(pb.partials + c * pb.grid, (int)gridDim.x, lane);
            v = warp_sum_dd(v);
            if (lane == 0) pb.result[c] = v;
        }
        if (lane == 0) {
            *pb.ticket = 0u;
            if (pb.timed && pb.result == pb.rb->res) pb.rb->stamp[2] = global_ns();  // the walk's end
        }
        publish(pb, pb.rb_host);
    }
}

// ---------------------------------------------------------------- real ----
// Sum over one unit: sum_d (-1)^popc(d) prod_r (xh_r + DE[d][r]).
// With STATS, also returns sum_d term_d^2 in *s2 (one FMA per term; sizes the
// double-double refinement).
template <int N, int G, bool STATS = false>
__device__ __forceinline__ double unit_sum_real(const double (&xh)[N], const double* __restrict__ s_de,
                                                int nq, double* s2 = nullptr)
{
    double acc = 0.0, sq[G];
#pragma unroll
    for (int i = 0; i < G; ++i) sq[i] = 0.0;
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
        const double* de = s_de + q * (N * G);
        double p[G];
        if constexpr (G == 4) {
            double2 v0 = reinterpret_cast<const double2*>(de)[0];
            double2 v1 = reinterpret_cast<const double2*>(de)[1];
            p[0] = add_rn(xh[0], v0.x);
            p[1] = add_rn(xh[0], v0.y);
            p[2] = add_rn(xh[0], v1.x);
            p[3] = add_rn(xh[0], v1.y);
#pragma unroll
            for (int r = 1; r < N; ++r) {
                double2 a = reinterpret_cast<const double2*>(de + r * 4)[0];
                double2 b = reinterpret_cast<const double2*>(de + r * 4)[1];
                p[0] = mul_rn(p[0], add_rn(xh[r], a.x));
                p[1] = mul_rn(p[1], add_rn(xh[r], a.y));
                p[2] = mul_rn(p[2], add_rn(xh[r], b.x));
                p[3] = mul_rn(p[3], add_rn(xh[r], b.y));
            }
        } else {
#pragma unroll
            for (int i = 0; i < G; ++i) p[i] = add_rn(xh[0], de[i]);
#pragma unroll
            for (int r = 1; r < N; ++r) {
#pragma unroll
                for (int i = 0; i < G; ++i) p[i] = mul_rn(p[i], add_rn(xh[r], de[r * G + i]));
            }
        }
        double gs;
        if constexpr (G == 4) gs = sub_rn(sub_rn(p[0], p[1]), sub_rn(p[2], p[3]));  // + - - +
        else if constexpr (G == 2) gs = sub_rn(p[0], p[1]);
        else gs = p[0];
        acc = (__popc(q) & 1) ? sub_rn(acc, gs) : add_rn(acc, gs);
        if constexpr (STATS) {
#pragma unroll
            for (int i = 0; i < G; ++i) sq[i] = __fma_rn(p[i], p[i], sq[i]);
        }
    }
    if constexpr (STATS) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < G; ++i) t += sq[i];
        *s2 = t;
    }
    return acc;
}

// The same for the derivative walk: sum_d (-1)^popc(d) q_d, one pass over the
// rows per group (see deriv_on).  Twelve FP64 instructions per row and group
// of four terms against two 16-byte shared loads; eight independent chains.
// group_sum_deriv_rt (refine_impl.cuh) replays a group's operations.
template <int N, int G, bool STATS = false>
__device__ __forceinline__ double unit_sum_deriv(const double (&xh)[N], const double* __restrict__ s_de,
                                                 int nq, double* s2 = nullptr)
{
    double acc = 0.0, sq[G];
#pragma unroll
    for (int i = 0; i < G; ++i) sq[i] = 0.0;
#pragma unroll 1
    for (int k = 0; k < nq; ++k) {
        const double* de = s_de + k * (N * G);
        double p[G], q[G];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            double v[G];
            if constexpr (G == 4) {
                const double2 a = reinterpret_cast<const double2*>(de + r * 4)[0];
                const double2 b = reinterpret_cast<const double2*>(de + r * 4)[1];
                v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
            } else {
#pragma unroll
                for (int i = 0; i < G; ++i) v[i] = de[r * G + i];
            }
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const double x = add_rn(xh[r], v[i]);
                if (r == 0) {
                    p[i] = x;
                } else {
                    q[i] = r == 1 ? add_rn(x, p[i]) : __fma_rn(q[i], x, p[i]);
                    if (r + 1 < N) p[i] = mul_rn(p[i], x);
                }
            }
        }
        double gs;
        if constexpr (G == 4) gs = sub_rn(sub_rn(q[0], q[1]), sub_rn(q[2], q[3]));  // + - - +
        else if constexpr (G == 2) gs = sub_rn(q[0], q[1]);
        else gs = q[0];
        acc = (__popc(k) & 1) ? sub_rn(acc, gs) : add_rn(acc, gs);
        if constexpr (STATS) {
#pragma unroll
            for (int i = 0; i < G; ++i) sq[i] = __fma_rn(q[i], q[i], sq[i]);
        }
    }
    if constexpr (STATS) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < G; ++i) t += sq[i];
        *s2 = t;
    }
    return acc;
}

// Upper bound of |term| over a unit: prod_r f_r, f_r = max |xh_r + DE[d][r]| with
// bnd [2][n] the range of DE over d; for the derivative sum_r prod_{r' != r} f_r'.
template <int N, bool D>
__device__ __forceinline__ double unit_bound_real(const double (&xh)[N], const double* bnd)
{
    double p = 1.0, q = 0.0;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const double f = fmax(fabs(add_rn(xh[r], bnd[r])), fabs(add_rn(xh[r], bnd[N + r])));
        if (D) q = __fma_rn(q, f, p);
        p = mul_rn(p, f);
    }
    return D ? q : p;
}

// First unit base of each thread (one component), built cooperatively by its
// warp from the NW start vector (x0h, x0l) and the high columns s_mt; every lane of the
// warp calls this (it shuffles), whether it owns units or not.
// The lanes' first units u0 lie in one range [ulo, uhi] (balanced_range is
// monotonic in the thread index), so the Gray bits above P, the highest bit
// where ulo and uhi differ, are the same for every lane.  Lane r adds the
// high columns j > P selected by those common bits to x0_r (double-double,
// ascending j) for rows r and r + 32, the warp broadcasts the N results,
// and each lane adds its own columns j <= P (ascending), four rows at a time
// (independent chains, the same operations per row).  Hi words go to xh,
// lo words to the thread's shared slots s_lo[r * bd + tid].  Compared with
// every lane adding all of its columns, this saves most of the double-double
// adds when threads own few units (n <= 26).
// D: the derivative walk, whose high columns have low words (s_ml).
template <int N, bool D>
__device__ __forceinline__ void first_base(const double* __restrict__ x0h, const double* __restrict__ x0l,
                                           const double* __restrict__ s_mt, const double* __restrict__ s_ml,
                                           double* s_lo, int ntop,
                                           unsigned long long u0, unsigned long long u1, int tid, int bd,
                                           double (&xh)[N])
{
    const unsigned full = 0xffffffffu;
    const int lane = tid & 31;
    const unsigned act = __ballot_sync(full, u0 < u1);
    if (act == 0u) return;  // warp-uniform
    const int last = 31 - __clz(act);
    const unsigned long long ulo = __shfl_sync(full, u0, 0), uhi = __shfl_sync(full, u0, last);
    const int P = ulo == uhi ? -1 : 63 - __clzll(ulo ^ uhi);
    const unsigned long long gc = gray_of(ulo);
    auto plus = [&](dd x, int i) { return D ? dd_step(x, s_mt[i], s_ml[i]) : dd_add_d(x, s_mt[i]); };
    dd c0 = {0.0, 0.0}, c1 = {0.0, 0.0};
    if (lane < N) {
        c0 = dd{x0h[lane], x0l[lane]};
        if (N > 32 && lane + 32 < N) c1 = dd{x0h[lane + 32], x0l[lane + 32]};
        for (int j = P + 1; j < ntop; ++j)
            if ((gc >> j) & 1ull) {
                c0 = plus(c0, j * N + lane);
                if (N > 32 && lane + 32 < N) c1 = plus(c1, j * N + lane + 32);
            }
    }
    const bool own = u0 < u1;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const double h = __shfl_sync(full, r < 32 ? c0.hi : c1.hi, r & 31);
        const double l = __shfl_sync(full, r < 32 ? c0.lo : c1.lo, r & 31);
        xh[r] = h;
        if (own) s_lo[r * bd + tid] = l;
    }
    if (!own) return;
    const unsigned long long g0 = gray_of(u0);
    const int jp = P + 1 < ntop ? P + 1 : ntop;  // private columns 0 .. jp-1
#pragma unroll
    for (int r0 = 0; r0 < N; r0 += 4) {
        dd x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r0 + k < N) x[k] = dd{xh[r0 + k], s_lo[(r0 + k) * bd + tid]};
        for (int j = 0; j < jp; ++j)
            if ((g0 >> j) & 1ull) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (r0 + k < N) x[k] = plus(x[k], j * N + r0 + k);
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r0 + k < N) {
                xh[r0 + k] = x[k].hi;
                s_lo[(r0 + k) * bd + tid] = x[k].lo;
            }
    }
}

template <int N, bool D>
__device__ __forceinline__ void walk_real_body(const Problem& pb)
{
    constexpr int G = RealCfg<N>::G;
    extern __shared__ __align__(16) double smem[];
    const int w = pb.w;
    const int terms = 1 << w;
    const int nq = terms / G;
    const int ntop = N - 1 - (D ? 1 : 0) - w;
    const int tid = threadIdx.x, bd = blockDim.x;
    double* s_de = smem;
    double* s_mt = s_de + terms * N;
    constexpr bool kFar = deriv_low_far(N, 1);
    const int ntp = ntop > 0 ? ntop : 0;
    double* s_ml = kFar ? pb.mt_lo : s_mt + ntp * N;  // derivative walk: the high columns' low words
    double* s_lo = s_mt + (D && !kFar ? 2 : 1) * ntp * N;
    float* s_hist = reinterpret_cast<float*>(s_lo + N * bd);  // mode 1
    unsigned* s_cnt = reinterpret_cast<unsigned*>(s_hist + kHistBins);
    // DE range per row, [2][N] (min, max).  Two scalar loads per row: a paired
    // 16-byte load keeps more registers live and makes the n=32 walk spill.
    double* s_bnd = reinterpret_cast<double*>(s_cnt + kHistBins);
    for (int i = tid; i < terms * N; i += bd) s_de[i] = pb.de_hi[i];
    for (int i = tid; i < ntop * N; i += bd) {
        s_mt[i] = pb.mt[i];
        if (D && !kFar) s_ml[i] = pb.mt_lo[i];
    }
    const int mode = pb.mode;
    if (mode != 0)
        for (int i = tid; i < 2 * N; i += bd) s_bnd[i] = pb.bnd[i];
    if (mode == 1)
        for (int i = tid; i < kHistBins; i += bd) { s_hist[i] = 0.0f; s_cnt[i] = 0u; }
    __syncthreads();

    const unsigned long long T = (unsigned long long)gridDim.x * bd;
    const unsigned long long t = (unsigned long long)blockIdx.x * bd + tid;
    unsigned long long u0, u1;
    balanced_range(eff_units(pb, D), T, t, &u0, &u1);
    // The scan only walks threads that own a unit at or above the threshold.
    if (mode == 2 && (int)pb.tmax[t] < pb.thr_bin) u1 = u0;
    dd tot[1] = {{0.0, 0.0}};
    HistCache hc;
    const int lbin = mode == 1 ? __ldcg(pb.list_bin) : 0;
    int bmax = 0;
    double xh[N];
    // First unit base: x0 plus the selected high columns, the warp's common
    // ones first (the refinement rebuilds bases in plain index order; the hi
    // words agree unless a row value lies within ~2^-100 of a rounding
    // midpoint, and then only that unit's correction carries one FP64 rounding).
    first_base<N, D>(pb.x0_hi, pb.x0_lo, s_mt, s_ml, s_lo, ntop, u0, u1, tid, bd, xh);
    if (u0 < u1) {
        unsigned long long u = u0;
        while (true) {
            int b = 0;
            if (mode != 0) {
                // the scan recomputes the bound bit for bit to select the same units
                b = hist_bin(unit_bound_real<N, D>(xh, s_bnd));
                bmax = b > bmax ? b : bmax;
                if (mode == 2 && b >= pb.thr_bin) {
                    unsigned long long k = atomicAdd(pb.list_n, 1ull);
                    if (k < pb.list_cap) {
                        pb.list_u[k] = u;
                        double* dst = pb.list_x + k * (2 * N);
#pragma unroll
                        for (int r = 0; r < N; ++r) { dst[r] = xh[r]; dst[N + r] = s_lo[r * bd + tid]; }
                    }
                }
            }
            if (mode == 0) {
                const double us = D ? unit_sum_deriv<N, G>(xh, s_de, nq) : unit_sum_real<N, G>(xh, s_de, nq);
                tot[0] = dd_add_d(tot[0], (u & 1ull) ? -us : us);
            } else if (mode == 1) {
                double sq;
                const double us = D ? unit_sum_deriv<N, G, true>(xh, s_de, nq, &sq)
                                    : unit_sum_real<N, G, true>(xh, s_de, nq, &sq);
                tot[0] = dd_add_d(tot[0], (u & 1ull) ? -us : us);
                hc.add(b, sq, s_hist, s_cnt);  // actual sum of squared terms, keyed by the bound
                raw_list_add(pb, lbin, u, b);
            }
            if (++u >= u1) break;
            const int j = __ffsll((long long)u) - 1;
            const bool add = (gray_of(u) >> j) & 1ull;
            const double* col = s_mt + j * N;
#pragma unroll
            for (int r = 0; r < N; ++r) {
                double m = add ? col[r] : -col[r];
                dd s = two_sum(xh[r], m);
                double l = s_lo[r * bd + tid];
                if (D) l = add ? add_rn(l, s_ml[j * N + r]) : sub_rn(l, s_ml[j * N + r]);
                dd z = fast_two_sum(s.hi, add_rn(s.lo, l));
                xh[r] = z.hi;
                s_lo[r * bd + tid] = z.lo;
            }
        }
    }
    if (mode == 1) {
        pb.tmax[t] = (unsigned short)bmax;
        hc.flush(s_hist, s_cnt);
        __syncthreads();
        flush_hist(s_hist, s_cnt, pb);
    }
    if (mode != 2) grid_reduce<1>(tot, pb);
}

// The derivative walk where the matrix has a pivot column, else the plain
// walk; the branch is the same for the whole grid.
template <int N>
__global__ void __launch_bounds__(RealCfg<N>::kMaxThreads, 1) walk_real(Problem pb)
{
    if (pb.timed && blockIdx.x == 0 && threadIdx.x == 0) pb.rb->stamp[1] = global_ns();
    if constexpr (N >= kMinDerivReal) {
        if (deriv_on(pb)) {
            walk_real_body<N, true>(pb);
            return;
        }
    }
    walk_real_body<N, false>(pb);
}

// ------------------------------------------------------------- complex ----
template <int N, int G, bool STATS = false>
__device__ __forceinline__ void unit_sum_complex(const double (&xr)[N], const double (&xi)[N],
                                                 const double* __restrict__ s_de_re,
                                                 const double* __restrict__ s_de_im, int nq,
                                                 double& acc_re, double& acc_im, double* s2 = nullptr)
{
    double ar = 0.0, ai = 0.0, sq[G];
#pragma unroll
    for (int i = 0; i < G; ++i) sq[i] = 0.0;
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
        const double* dr = s_de_re + q * (N * G);
        const double* di = s_de_im + q * (N * G);
        double pr[G], pi[G];
#pragma unroll
        for (int i = 0; i < G; ++i) {
            pr[i] = add_rn(xr[0], dr[i]);
            pi[i] = add_rn(xi[0], di[i]);
        }
#pragma unroll
        for (int r = 1; r < N; ++r) {
            double vr[G], vi[G];
            if constexpr (G == 4) {
                double2 a0 = reinterpret_cast<const double2*>(dr + r * 4)[0];
                double2 a1 = reinterpret_cast<const double2*>(dr + r * 4)[1];
                double2 b0 = reinterpret_cast<const double2*>(di + r * 4)[0];
                double2 b1 = reinterpret_cast<const double2*>(di + r * 4)[1];
                vr[0] = a0.x; vr[1] = a0.y; vr[2] = a1.x; vr[3] = a1.y;
                vi[0] = b0.x; vi[1] = b0.y; vi[2] = b1.x; vi[3] = b1.y;
            } else if constexpr (G == 2) {
                double2 a = reinterpret_cast<const double2*>(dr + r * 2)[0];
                double2 b = reinterpret_cast<const double2*>(di + r * 2)[0];
                vr[0] = a.x; vr[1] = a.y; vi[0] = b.x; vi[1] = b.y;
            } else {
#pragma unroll
                for (int i = 0; i < G; ++i) { vr[i] = dr[r * G + i]; vi[i] = di[r * G + i]; }
            }
#pragma unroll
            for (int i = 0; i < G; ++i) {
                double yr = add_rn(xr[r], vr[i]);
                double yi = add_rn(xi[r], vi[i]);
                double t1 = mul_rn(pi[i], yi);
                double t2 = mul_rn(pi[i], yr);
                double nr = __fma_rn(pr[i], yr, -t1);
                double ni = __fma_rn(pr[i], yi, t2);
                pr[i] = nr;
                pi[i] = ni;
            }
        }
        double gr, gi;
        if constexpr (G == 4) {  // + - - +
            gr = sub_rn(sub_rn(pr[0], pr[1]), sub_rn(pr[2], pr[3]));
            gi = sub_rn(sub_rn(pi[0], pi[1]), sub_rn(pi[2], pi[3]));
        } else if constexpr (G == 2) { gr = sub_rn(pr[0], pr[1]); gi = sub_rn(pi[0], pi[1]); }
        else { gr = pr[0]; gi = pi[0]; }
        if (__popc(q) & 1) { ar = sub_rn(ar, gr); ai = sub_rn(ai, gi); }
        else { ar = add_rn(ar, gr); ai = add_rn(ai, gi); }
        if constexpr (STATS) {
#pragma unroll
            for (int i = 0; i < G; ++i) sq[i] = __fma_rn(pi[i], pi[i], __fma_rn(pr[i], pr[i], sq[i]));
        }
    }
    acc_re = ar;
    acc_im = ai;
    if constexpr (STATS) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < G; ++i) t += sq[i];
        *s2 = t;
    }
}

// The derivative walk's complex terms (unit_sum_deriv): two at a time out of the
// table's groups of G, so that p and q of each fit the registers beside x.
// Ten FP64 instructions per row and term where the two plain terms it stands
// for take twelve.
template <int N, int G, bool STATS = false>
__device__ __forceinline__ void unit_sum_complex_deriv(const double (&xr)[N], const double (&xi)[N],
                                                       const double* __restrict__ s_de_re,
                                                       const double* __restrict__ s_de_im, int nq,
                                                       double& acc_re, double& acc_im, double* s2 = nullptr)
{
    static_assert(G % 2 == 0, "pairs of terms");
    double ar = 0.0, ai = 0.0, sq[2] = {0.0, 0.0};
#pragma unroll 1
    for (int k = 0; k < nq * (G / 2); ++k) {
        const double* dr = s_de_re + (k / (G / 2)) * (N * G) + 2 * (k % (G / 2));
        const double* di = s_de_im + (k / (G / 2)) * (N * G) + 2 * (k % (G / 2));
        double pr[2], pi[2], qr[2], qi[2];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            const double2 a = *reinterpret_cast<const double2*>(dr + r * G);
            const double2 b = *reinterpret_cast<const double2*>(di + r * G);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const double yr = add_rn(xr[r], i ? a.y : a.x);
                const double yi = add_rn(xi[r], i ? b.y : b.x);
                if (r == 0) {
                    pr[i] = yr;
                    pi[i] = yi;
                } else {
                    if (r == 1) {
                        qr[i] = add_rn(yr, pr[i]);
                        qi[i] = add_rn(yi, pi[i]);
                    } else {
                        const double t = __fma_rn(-qi[i], yi, pr[i]);
                        const double u = __fma_rn(qi[i], yr, pi[i]);
                        qi[i] = __fma_rn(qr[i], yi, u);
                        qr[i] = __fma_rn(qr[i], yr, t);
                    }
                    if (r + 1 < N) {
                        const double t1 = mul_rn(pi[i], yi), t2 = mul_rn(pi[i], yr);
                        pi[i] = __fma_rn(pr[i], yi, t2);
                        pr[i] = __fma_rn(pr[i], yr, -t1);
                    }
                }
            }
        }
        const double gr = sub_rn(qr[0], qr[1]), gi = sub_rn(qi[0], qi[1]);
        if (__popc(k) & 1) { ar = sub_rn(ar, gr); ai = sub_rn(ai, gi); }
        else { ar = add_rn(ar, gr); ai = add_rn(ai, gi); }
        if constexpr (STATS) {
#pragma unroll
            for (int i = 0; i < 2; ++i) sq[i] = __fma_rn(qi[i], qi[i], __fma_rn(qr[i], qr[i], sq[i]));
        }
    }
    acc_re = ar;
    acc_im = ai;
    if constexpr (STATS) *s2 = sq[0] + sq[1];
}

// Upper bound of |term| over a unit (unit_bound_real), with |x_r| <= |xtop_r| +
// max_d |DE[d][r]| (triangle inequality), bnd [N] the latter.
template <int N, bool D>
__device__ __forceinline__ double unit_bound_complex(const double (&xr)[N], const double (&xi)[N], const double* bnd)
{
    double p = 1.0, q = 0.0;
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const double f = add_rn(__dsqrt_rn(__fma_rn(xr[r], xr[r], mul_rn(xi[r], xi[r]))), bnd[r]);
        if (D) q = __fma_rn(q, f, p);
        p = mul_rn(p, f);
    }
    return D ? q : p;
}

template <int N, bool D>
__device__ __forceinline__ void walk_complex_body(const Problem& pb)
{
    constexpr int G = ComplexCfg<N>::G;
    extern __shared__ __align__(16) double smem[];
    const int w = pb.w;
    const int terms = 1 << w;
    const int nq = terms / G;
    const int ntop = N - 1 - (D ? 1 : 0) - w;
    const int ntp = ntop > 0 ? ntop : 0;
    const int tid = threadIdx.x, bd = blockDim.x;
    double* s_de = smem;                        // [2][terms*N]
    double* s_mt = s_de + 2 * terms * N;        // [2][ntop*N]
    constexpr bool kFar = deriv_low_far(N, 2);
    double* s_ml = kFar ? pb.mt_lo : s_mt + 2 * ntp * N;  // [2][ntop*N] low words (derivative walk)
    double* s_lo = s_mt + (D && !kFar ? 4 : 2) * ntp * N;  // [2][N][bd]
    float* s_hist = reinterpret_cast<float*>(s_lo + 2 * N * bd);  // mode 1
    unsigned* s_cnt = reinterpret_cast<unsigned*>(s_hist + kHistBins);
    double* s_bnd = reinterpret_cast<double*>(s_cnt + kHistBins);  // [N]
    for (int i = tid; i < 2 * terms * N; i += bd) s_de[i] = pb.de_hi[i];
    for (int i = tid; i < 2 * ntp * N; i += bd) {
        s_mt[i] = pb.mt[i];
        if (D && !kFar) s_ml[i] = pb.mt_lo[i];
    }
    const int mode = pb.mode;
    if (mode != 0)
        for (int i = tid; i < N; i += bd) s_bnd[i] = pb.bnd[i];
    if (mode == 1)
        for (int i = tid; i < kHistBins; i += bd) { s_hist[i] = 0.0f; s_cnt[i] = 0u; }
    __syncthreads();
    const double* s_mt_re = s_mt;
    const double* s_mt_im = s_mt + ntp * N;
    double* s_lo_re = s_lo;
    double* s_lo_im = s_lo + N * bd;

    const unsigned long long T = (unsigned long long)gridDim.x * bd;
    const unsigned long long t = (unsigned long long)blockIdx.x * bd + tid;
    unsigned long long u0, u1;
    balanced_range(eff_units(pb, D), T, t, &u0, &u1);
    if (mode == 2 && (int)pb.tmax[t] < pb.thr_bin) u1 = u0;
    dd tot[2] = {{0.0, 0.0}, {0.0, 0.0}};
    HistCache hc;
    const int lbin = mode == 1 ? __ldcg(pb.list_bin) : 0;
    int bmax = 0;
    double xr[N], xi[N];
    first_base<N, D>(pb.x0_hi, pb.x0_lo, s_mt_re, s_ml, s_lo_re, ntop, u0, u1, tid, bd, xr);
    first_base<N, D>(pb.x0_hi + N, pb.x0_lo + N, s_mt_im, s_ml + ntp * N, s_lo_im, ntop, u0, u1, tid, bd, xi);
    if (u0 < u1) {
        unsigned long long u = u0;
        while (true) {
            int b = 0;
            if (mode != 0) {
                b = hist_bin(unit_bound_complex<N, D>(xr, xi, s_bnd));
                bmax = b > bmax ? b : bmax;
                if (mode == 2 && b >= pb.thr_bin) {
                    unsigned long long k = atomicAdd(pb.list_n, 1ull);
                    if (k < pb.list_cap) {
                        pb.list_u[k] = u;
                        double* dst = pb.list_x + k * (4 * N);
#pragma unroll
                        for (int r = 0; r < N; ++r) {
                            dst[r] = xr[r];
                            dst[N + r] = s_lo_re[r * bd + tid];
                            dst[2 * N + r] = xi[r];
                            dst[3 * N + r] = s_lo_im[r * bd + tid];
                        }
                    }
                }
            }
            if (mode != 2) {
                double ur, ui, sq = 0.0;
                if constexpr (D) {
                    if (mode == 0) unit_sum_complex_deriv<N, G>(xr, xi, s_de, s_de + terms * N, nq, ur, ui);
                    else unit_sum_complex_deriv<N, G, true>(xr, xi, s_de, s_de + terms * N, nq, ur, ui, &sq);
                } else {
                    if (mode == 0) unit_sum_complex<N, G>(xr, xi, s_de, s_de + terms * N, nq, ur, ui);
                    else unit_sum_complex<N, G, true>(xr, xi, s_de, s_de + terms * N, nq, ur, ui, &sq);
                }
                if (u & 1ull) { ur = -ur; ui = -ui; }
                tot[0] = dd_add_d(tot[0], ur);
                tot[1] = dd_add_d(tot[1], ui);
                if (mode == 1) {
                    hc.add(b, sq, s_hist, s_cnt);
                    raw_list_add(pb, lbin, u, b);
                }
            }
            if (++u >= u1) break;
            const int j = __ffsll((long long)u) - 1;
            const bool add = (gray_of(u) >> j) & 1ull;
#pragma unroll
            for (int r = 0; r < N; ++r) {
                double mr = add ? s_mt_re[j * N + r] : -s_mt_re[j * N + r];
                double mi = add ? s_mt_im[j * N + r] : -s_mt_im[j * N + r];
                double lr = s_lo_re[r * bd + tid], li = s_lo_im[r * bd + tid];
                if (D) {
                    const double er = s_ml[j * N + r], ei = s_ml[(ntp + j) * N + r];
                    lr = add ? add_rn(lr, er) : sub_rn(lr, er);
                    li = add ? add_rn(li, ei) : sub_rn(li, ei);
                }
                dd s = two_sum(xr[r], mr);
                dd z = fast_two_sum(s.hi, add_rn(s.lo, lr));
                xr[r] = z.hi;
                s_lo_re[r * bd + tid] = z.lo;
                s = two_sum(xi[r], mi);
                z = fast_two_sum(s.hi, add_rn(s.lo, li));
                xi[r] = z.hi;
                s_lo_im[r * bd + tid] = z.lo;
            }
        }
    }
    if (mode == 1) {
        pb.tmax[t] = (unsigned short)bmax;
        hc.flush(s_hist, s_cnt);
        __syncthreads();
        flush_hist(s_hist, s_cnt, pb);
    }
    if (mode != 2) grid_reduce<2>(tot, pb);
}

// The derivative walk where the matrix has a pivot column, else the plain
// walk; the branch is the same for the whole grid.
template <int N>
__global__ void __launch_bounds__(ComplexCfg<N>::kMaxThreads, 1) walk_complex(Problem pb)
{
    if (pb.timed && blockIdx.x == 0 && threadIdx.x == 0) pb.rb->stamp[1] = global_ns();
    if constexpr (N >= kMinDerivComplex) {
        if (deriv_on(pb)) {
            walk_complex_body<N, true>(pb);
            return;
        }
    }
    walk_complex_body<N, false>(pb);
}

// Double-double refinement (dense_refine.cu), all stream-ordered after the
// mode-1 walk with no host round trip in between:
//   launch_threshold   picks rb->thr / rb->count / rb->err from the
//                      histogram and decides the listing path (rb->from_list);
//   launch_listing     lists the units whose bin >= rb->thr: from the walk's
//                      own list when rb->from_list, else from the walk's
//                      per-thread maxima (pb.tmax), one warp per thread
//                      range, bases rebuilt from scratch;
//   launch_refine      re-evaluates the listed units in double-double and
//                      writes sum(double-double unit sum - the walk's FP64
//                      unit sum) to rb->corr, a worker of one or more warps
//                      per unit; it refines nothing unless
//                      rb->list_n == rb->count <= pb.list_cap.
// bound_walk + pick_list_bin run before the walk and set the bin from which
// the walk lists its units.  A mode-2 walk (same launch shape as mode 1)
// replays the listing with the walk's own bases (pb.list_x) when the host
// finds the count check failed.
int launch_threshold(const Problem& pb, cudaStream_t s);
int launch_refine(const Problem& pb, int blocks, Readback* rb_host, cudaStream_t s);  // rb_host: Problem::rb_host
int launch_bound_pass(const Problem& pb, int blocks, cudaStream_t s);
int launch_listing(const Problem& pb, cudaStream_t s);
// Dynamic shared memory of the refinement at `threads` threads per CTA: both
// words of every part's table, per-warp bases and group sums, high columns.
size_t refine_smem_bytes(const Problem& pb, int threads);

// FP32-product walks (f32_impl.cuh), n <= kMaxF32N.  A result whose
// estimated relative error exceeds opt.rel_tol (kF32DefaultBound when unset,
// the library's accuracy bar) comes back with SPB_ERR_ACCURACY.
constexpr int kMaxF32N = 40;
constexpr double kF32DefaultBound = 1e-12;
int launch_walk_f32(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s);
size_t walk_f32_smem_bytes(const Problem& pb, int threads);
int walk_f32_max_threads(int n, int comps);

// Per-n dispatch (defined in the instantiation units).
int launch_walk_real(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s);
int launch_walk_complex(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s);

// Row-compacted walk on NA = pb.na active rows (sparse_walk.cu).
int launch_walk_sparse(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s);

inline int launch_walk(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s)
{
    if (pb.na < pb.n) return launch_walk_sparse(pb, blocks, threads, smem, s);
    return pb.comps == 1 ? launch_walk_real(pb, blocks, threads, smem, s)
                         : launch_walk_complex(pb, blocks, threads, smem, s);
}

int walk_max_threads(int n, int comps);

}  // namespace dense
}  // namespace spb

// X-macro over n = 1..63.
#define SPB_FOR_EACH_N(X)                                                                  \
    X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15)       \
    X(16) X(17) X(18) X(19) X(20) X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29)    \
    X(30) X(31) X(32) X(33) X(34) X(35) X(36) X(37) X(38) X(39) X(40) X(41) X(42) X(43)    \
    X(44) X(45) X(46) X(47) X(48) X(49) X(50) X(51) X(52) X(53) X(54) X(55) X(56) X(57)    \
    X(58) X(59) X(60) X(61) X(62) X(63)
