// Exact 0/1 permanent by the Nijenhuis–Wilf form of Ryser's formula in
// integers.  With x'_r(S) = 2 a_{r,n-1} - rowsum_r + 2 sum_{j in S} a_rj
// (twice the NW row value, an integer in [-n, n]) over the subsets S of
// columns 0..n-2,
//   Sigma = sum_S (-1)^|S| prod_r x'_r(S) = 2^(n-1) * (+-) perm(A)
// (+ for odd n, - for even), computed in wrap-around integer arithmetic
// modulo 2^(32L).  The host picks L from a Bregman-Minc bound so that
// |Sigma| < 2^(32L-1), then shifts Sigma right by n-1 bits: the result is
// exact.  Half the subsets of plain Ryser, for n - 1 more accumulator bits.
//
// The reference has no integer path: 0/1 input goes through its FP64 NW
// walk (IO/IO.h:441-443 feeding Algorithms/GPU/Dense/dpSingleGPU.cuh), whose
// result is off by ~1e-10 relative at n=30.
//
// Layout mirrors the dense walk: the w low columns are enumerated from a
// shared table DEI[d][r] = twice the number of ones of row r among the
// columns of d (grouped [d/4][r][d%4], so one 16-byte broadcast load serves
// four terms); the n-1-w high columns form a unit index walked in Gray order
// per thread with the integer unit base xtop_r in registers.  Each term
// multiplies its row values in words of up to K rows (n^K < 2^32: the word's
// magnitude is an exact unsigned 32-bit integer), folds the word magnitudes
// into L 32-bit limbs with 32x32->64 multiply-adds over only the limbs the
// bit widths so far can reach, and applies the sign (the xor of the words')
// once.  Unit sums and the grid reduction are exact, so the result does not
// depend on the launch shape.
//
// Expanded walk (walk_binary<N, L, true>).  The permanent is expanded along one
// column c with m ones, whose rows the host puts first:
//   perm(A) = sum_{r < m} perm(A without row r and column c).
// All m minors share the columns, so one NW walk over the other n-1 columns
// (2^(n-2) subsets, half of the plain walk's) evaluates them together: a term
// is sum_{r < m} prod_{r' != r} x'_r', the first derivative of prod_r (x'_r + t)
// over the rows r < m, times the other rows' product.  Per row below m that
// takes one more multiply-add (q <- q x + p beside p <- p x), per row above m
// nothing more, so two plain terms' work of 4 operations per row becomes 3 or 2.
// The host picks the line (column, or row by transposing) with the fewest
// ones.  Sigma = sum_S (-1)^|S| term = 2^(n-2) * (+-) perm(A) (+ for even n).
// On one B200 at 1965 MHz, Bernoulli(0.5) entries with the identity: n=36
// 203.4 -> 120 ms with 12 ones in the line, 140 ms with 14.
// Bound, as the plain walk, by the instructions it issues: with 32-bit words as
// there (a sign and a magnitude per word) n=36 took 146 ms at 16 warps per SM and
// 183 ms at 8, one term at a time with these 64-bit words 134 ms.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "spb_common.cuh"

namespace spb {
namespace binary {

constexpr int kMaxN = 63;
constexpr int kMaxLimbs = 12;   // accumulator limbs (the result needs at most 10)

struct Problem {
    int n, w, limbs, grid;
    int m;                     // expanded walk: ones of the expanded column (rows 0..m-1); 0 = plain walk
    unsigned long long units;  // 2^(n-1-w) Gray units of 2^w terms each (expanded walk: 2^(n-2-w))
    const int* x0;             // [n] 2 a_{r,n-1} - rowsum_r
    const int* dei;            // [2^w/4][n][4] twice the low-column row counts
    const int8_t* mt;          // [ntop][n] high columns, doubled (0/2)
    uint32_t* partials;        // [grid][limbs]
    unsigned* ticket;          // last-CTA election (reset by the kernel)
    uint32_t* result;          // [limbs] sum over subsets, mod 2^(32*limbs)
};

// Rows per word: the largest K with n^K < 2^32, so a word's magnitude fits
// an unsigned 32-bit integer (|x'_r| <= n).  Its first K-1 rows multiply in
// signed 32-bit arithmetic (n^(K-1) < 2^31: exact); the last row's magnitude
// multiplies the magnitude of that product, unsigned.
__host__ __device__ constexpr int rows_per_word(int n)
{
    int k = 1;
    const unsigned long long b = (unsigned long long)(n > 1 ? n : 2);
    unsigned long long p = b;
    while (p * b < (1ull << 32) && k < 16) {
        p *= b;
        ++k;
    }
    return k;
}

// Bit width of n^k, the largest magnitude of a word of k rows.
__host__ __device__ constexpr int word_bits(int n, int k)
{
    unsigned long long p = 1;
    for (int i = 0; i < k; ++i) p *= (unsigned long long)n;
    int b = 0;
    while (b < 63 && (1ull << b) <= p) ++b;
    return b;
}

// Limbs that can be nonzero in the product of words 0..g (at most L): the
// bit widths of the words so far, summed, in 32-bit limbs.
__host__ __device__ constexpr int limbs_after(int n, int g, int L)
{
    const int K = rows_per_word(n);
    int bits = 0;
    for (int h = 0; h <= g; ++h) {
        const int rows = n - h * K < K ? n - h * K : K;
        bits += word_bits(n, rows);
    }
    const int l = (bits + 31) / 32;
    return l < L ? l : L;
}

template <int L>
__device__ __forceinline__ void limb_add(uint32_t (&a)[L], const uint32_t (&b)[L])
{
    uint64_t c = 0;
#pragma unroll
    for (int i = 0; i < L; ++i) {
        uint64_t t = (uint64_t)a[i] + b[i] + c;
        a[i] = (uint32_t)t;
        c = t >> 32;
    }
}

template <int L>
__device__ __forceinline__ void limb_sub(uint32_t (&a)[L], const uint32_t (&b)[L])
{
    uint64_t br = 0;
#pragma unroll
    for (int i = 0; i < L; ++i) {
        uint64_t t = (uint64_t)a[i] - b[i] - br;
        a[i] = (uint32_t)t;
        br = (t >> 63) & 1ull;
    }
}

// Word g of a term (rows g*K .. g*K + rows - 1): the signed product of its
// first rows, then the unsigned product of the magnitudes with its last row;
// its sign bit is xor-ed into sg and its magnitude multiplied into the limbs
// that the bit widths of words 0..g-1 can reach (a compile-time count), the
// carry out of the top one landing in the next (dropped past L: mod 2^(32L)).
// Recurses over g so that every count is a constant.
template <int N, int L, int G, int g>
__device__ __forceinline__ void term_word(const int (&xt)[N], const int* __restrict__ de, int i,
                                          uint32_t (&p)[L], uint32_t& sg)
{
    constexpr int K = rows_per_word(N);
    constexpr int NG = (N + K - 1) / K;
    constexpr int r0 = g * K, rows = N - r0 < K ? N - r0 : K;
    uint32_t m;
    if constexpr (rows == 1) {
        const int x = xt[r0] + de[r0 * G + i];
        sg ^= (uint32_t)x;
        m = (uint32_t)(x < 0 ? -x : x);
    } else {
        int sw = xt[r0] + de[r0 * G + i];
#pragma unroll
        for (int k = 1; k < rows - 1; ++k) sw *= xt[r0 + k] + de[(r0 + k) * G + i];
        const int x = xt[r0 + rows - 1] + de[(r0 + rows - 1) * G + i];
        sg ^= (uint32_t)sw ^ (uint32_t)x;
        m = (uint32_t)(sw < 0 ? -sw : sw) * (uint32_t)(x < 0 ? -x : x);
    }
    if constexpr (g == 0) {
        p[0] = m;
    } else {
        constexpr int nb = limbs_after(N, g - 1, L);
        uint64_t c = 0;
#pragma unroll
        for (int l = 0; l < nb; ++l) {
            const uint64_t t = (uint64_t)p[l] * m + c;
            p[l] = (uint32_t)t;
            c = t >> 32;
        }
        if constexpr (nb < L) p[nb] = (uint32_t)c;
    }
    if constexpr (g + 1 < NG) term_word<N, L, G, g + 1>(xt, de, i, p, sg);
}

// |prod_r x'_r| mod 2^(32L) for one term (x'_r = xt[r] + de(r), signed) into
// p; returns a word whose bit 31 is the product's sign (the xor of the
// factors' signs).
template <int N, int L, int G>
__device__ __forceinline__ uint32_t term_product(const int (&xt)[N], const int* __restrict__ de, int i,
                                                 uint32_t (&p)[L])
{
#pragma unroll
    for (int l = 0; l < L; ++l) p[l] = 0u;
    uint32_t sg = 0u;
    term_word<N, L, G, 0>(xt, de, i, p, sg);
    return sg;
}

// a += p when mask is 0, a -= p when mask is all ones, modulo 2^(32L).
template <int L>
__device__ __forceinline__ void limb_add_masked(uint32_t (&a)[L], const uint32_t (&p)[L], uint32_t mask)
{
    uint64_t c = mask & 1u;
#pragma unroll
    for (int l = 0; l < L; ++l) {
        const uint64_t t = (uint64_t)a[l] + (p[l] ^ mask) + c;
        a[l] = (uint32_t)t;
        c = t >> 32;
    }
}

// ------------------------------------------------------- expanded walk ----
// Rows multiply in halves of up to K rows, signed 32-bit integers, and two
// halves make a signed 64-bit word (one 32x32->64 multiply), so that a term
// takes a sign and a magnitude per 2K rows instead of one per K.  The words
// with rows of the expanded column carry the derivative q beside the product.
constexpr int kExpandHalves = 4;  // halves that may hold rows of the expanded column
// Smallest n of the expanded walk.  Below, a call waits for its launch and copies
// and the longer chain of a term only adds to it (wall time, plain and expanded:
// n=12 61.4 and 65.1 us, n=16 63.5 and 67.2, n=21 70.6 and 73.4, n=23 90.1 and 80.0).
constexpr int kMinExpand = 22;

// Rows per half: the largest K with (n-1)^K < 2^31 and K (n-1)^(K-1) < 2^31 (the
// half's product and its derivative; row values are at most n-1 in magnitude).
__host__ __device__ constexpr int half_rows(int n)
{
    const unsigned long long b = (unsigned long long)(n - 1 > 1 ? n - 1 : 2);
    int k = 1;
    unsigned long long p = b;  // b^k
    while (p * b < (1ull << 31) && (unsigned long long)(k + 1) * p < (1ull << 31) && k < 16) {
        p *= b;
        ++k;
    }
    return k;
}
__host__ __device__ constexpr int rows_in_half(int n, int h)
{
    const int left = n - h * half_rows(n);
    return left <= 0 ? 0 : (left < half_rows(n) ? left : half_rows(n));
}

// Limbs that can be nonzero after words 0..g: a product of R rows is at most
// (n-1)^R, a sum of m <= n products of R-1 rows at most n (n-1)^(R-1): one bit more.
__host__ __device__ constexpr int expand_limbs_after(int n, int g, int L)
{
    int bits = 1;
    for (int h = 0; h <= 2 * g + 1; ++h)
        if (rows_in_half(n, h) > 0) bits += word_bits(n - 1, rows_in_half(n, h));
    const int l = (bits + 31) / 32;
    return l < L ? l : L;
}

// Terms evaluated side by side.  Two share each table load (8 bytes: with the
// branches on m the loads of separate terms are not merged) and give the
// scheduler two chains; four would not fit the registers.  One term at a time
// spent a table load per row (the load pipe 40 % busy): n=36 141.6 -> 122.7 ms,
// n=33 15.4 -> 13.9 ms, n=30 1.91 -> 1.64 ms.
constexpr int kPair = 2;

// Row r's values of terms i and i + 1.
__device__ __forceinline__ void row_values(int xt, const int* __restrict__ de, int (&x)[kPair])
{
    const int2 d = *reinterpret_cast<const int2*>(de);
    x[0] = xt + d.x;
    x[1] = xt + d.y;
}

// Half h: the product p of its rows' values.
template <int N, int G, int h>
__device__ __forceinline__ void half_plain(const int (&xt)[N], const int* __restrict__ de, int i, int (&p)[kPair])
{
    constexpr int r0 = h * half_rows(N), rows = rows_in_half(N, h);
#pragma unroll
    for (int k = 0; k < rows; ++k) {
        int x[kPair];
        row_values(xt[r0 + k], de + (r0 + k) * G + i, x);
#pragma unroll
        for (int t = 0; t < kPair; ++t) p[t] = k == 0 ? x[t] : p[t] * x[t];
    }
}

// The same with its derivative q over the rows below m.  ALL: all of them are.
template <int N, int G, int h, bool ALL>
__device__ __forceinline__ void half_dual(const int (&xt)[N], const int* __restrict__ de, int i, int m, int (&p)[kPair],
                                          int (&q)[kPair])
{
    constexpr int r0 = h * half_rows(N), rows = rows_in_half(N, h);
#pragma unroll
    for (int k = 0; k < rows; ++k) {
        int x[kPair];
        row_values(xt[r0 + k], de + (r0 + k) * G + i, x);
#pragma unroll
        for (int t = 0; t < kPair; ++t) {
            if (k == 0) {
                p[t] = x[t];
                q[t] = 1;  // the half holds a row below m
            } else {
                q[t] = ALL && k == 1 ? x[t] + p[t] : q[t] * x[t] + (ALL || r0 + k < m ? p[t] : 0);
                p[t] *= x[t];
            }
        }
    }
}

template <int N, int G, int h>
__device__ __forceinline__ void half_any(const int (&xt)[N], const int* __restrict__ de, int i, int m, int (&p)[kPair],
                                         int (&q)[kPair])
{
    if (m >= h * half_rows(N) + rows_in_half(N, h)) half_dual<N, G, h, true>(xt, de, i, m, p, q);
    else half_dual<N, G, h, false>(xt, de, i, m, p, q);
}

// Word g: the product W of its rows, its derivative Q when it holds rows below m.
template <int N, int G, int g>
__device__ __forceinline__ void word_plain(const int (&xt)[N], const int* __restrict__ de, int i, long long (&W)[kPair])
{
    int a[kPair], b[kPair];
    half_plain<N, G, 2 * g>(xt, de, i, a);
    if constexpr (rows_in_half(N, 2 * g + 1) > 0) half_plain<N, G, 2 * g + 1>(xt, de, i, b);
#pragma unroll
    for (int t = 0; t < kPair; ++t) {
        if constexpr (rows_in_half(N, 2 * g + 1) > 0) W[t] = (long long)a[t] * b[t];
        else W[t] = a[t];
    }
}
template <int N, int G, int g>
__device__ __forceinline__ void word_dual(const int (&xt)[N], const int* __restrict__ de, int i, int m,
                                          long long (&W)[kPair], long long (&Q)[kPair])
{
    int pa[kPair], qa[kPair];
    half_any<N, G, 2 * g>(xt, de, i, m, pa, qa);
    if constexpr (rows_in_half(N, 2 * g + 1) == 0) {
#pragma unroll
        for (int t = 0; t < kPair; ++t) {
            W[t] = pa[t];
            Q[t] = qa[t];
        }
    } else {
        int pb[kPair], qb[kPair];
        if (m > (2 * g + 1) * half_rows(N)) {
            half_any<N, G, 2 * g + 1>(xt, de, i, m, pb, qb);
            // at most 2K (n-1)^(2K-1) < 2^63: 2K <= n rows, (n-1)^(2K) < 2^62
#pragma unroll
            for (int t = 0; t < kPair; ++t) Q[t] = (long long)qa[t] * pb[t] + (long long)pa[t] * qb[t];
        } else {
            half_plain<N, G, 2 * g + 1>(xt, de, i, pb);
#pragma unroll
            for (int t = 0; t < kPair; ++t) Q[t] = (long long)qa[t] * pb[t];
        }
#pragma unroll
        for (int t = 0; t < kPair; ++t) W[t] = (long long)pa[t] * pb[t];
    }
}

__device__ __forceinline__ unsigned long long magnitude(long long v, uint32_t& sg)
{
    const long long s = v >> 63;
    sg ^= (uint32_t)s;
    return (unsigned long long)((v ^ s) - s);
}

// p (nb limbs) times w, into min(nb + 2, L) limbs (mod 2^(32L)).
template <int L, int nb>
__device__ __forceinline__ void fold64(uint32_t (&p)[L], unsigned long long w)
{
    const uint32_t w0 = (uint32_t)w, w1 = (uint32_t)(w >> 32);
    uint32_t r[L];
    uint64_t c = 0;
#pragma unroll
    for (int l = 0; l < nb; ++l) {
        const uint64_t t = (uint64_t)p[l] * w0 + c;
        r[l] = (uint32_t)t;
        c = t >> 32;
    }
    if constexpr (nb < L) r[nb] = (uint32_t)c;
    c = 0;
#pragma unroll
    for (int l = 0; l < nb && l + 1 < L; ++l) {
        const uint64_t t = (uint64_t)p[l] * w1 + r[l + 1] + c;
        r[l + 1] = (uint32_t)t;
        c = t >> 32;
    }
    if constexpr (nb + 1 < L) r[nb + 1] = (uint32_t)c;
#pragma unroll
    for (int l = 0; l < nb + 2 && l < L; ++l) p[l] = r[l];
}

// Words g, g+1, ... of two terms, none with rows of the expanded column.
template <int N, int L, int G, int g>
__device__ __forceinline__ void plain_words(const int (&xt)[N], const int* __restrict__ de, int i,
                                            uint32_t (&p)[kPair][L], uint32_t (&sg)[kPair])
{
    if constexpr (rows_in_half(N, 2 * g) > 0) {
        long long W[kPair];
        word_plain<N, G, g>(xt, de, i, W);
#pragma unroll
        for (int t = 0; t < kPair; ++t) fold64<L, expand_limbs_after(N, g - 1, L)>(p[t], magnitude(W[t], sg[t]));
        plain_words<N, L, G, g + 1>(xt, de, i, p, sg);
    }
}

// |Q0 W1 + W0 Q1|, 128 bits (4K rows below (2^31)^4), into p; the sign to sg.
template <int L>
__device__ __forceinline__ void join_words(long long W0, long long Q0, long long W1, long long Q1, uint32_t (&p)[L],
                                           uint32_t& sg)
{
    const unsigned long long a = (unsigned long long)Q0 * (unsigned long long)W1;
    const unsigned long long b = (unsigned long long)W0 * (unsigned long long)Q1;
    const unsigned long long lo = a + b;
    const long long hi = (long long)((unsigned long long)__mul64hi(Q0, W1) + (unsigned long long)__mul64hi(W0, Q1) +
                                     (lo < a ? 1ull : 0ull));
    const unsigned long long s = (unsigned long long)(hi >> 63);
    sg ^= (uint32_t)s;
    const unsigned long long l0 = (lo ^ s) - s, h0 = ((unsigned long long)hi ^ s) + (s && l0 == 0 ? 1ull : 0ull);
    p[0] = (uint32_t)l0;
    p[1] = (uint32_t)(l0 >> 32);
    p[2] = (uint32_t)h0;
    p[3] = (uint32_t)(h0 >> 32);
}

// |(Q0 c + W0 q) d| with a half's product c and derivative q and another's
// product d: 96 bits (3K rows below 2^94), then one 32-bit factor.
template <int L>
__device__ __forceinline__ void join_half(long long W0, long long Q0, int c, int q, int d, uint32_t (&p)[L],
                                          uint32_t& sg)
{
    const int sc = c >> 31;  // c's sign moves to sg and q
    sg ^= (uint32_t)sc;
    const uint32_t cm = (uint32_t)((c ^ sc) - sc);
    const int qs = (q ^ sc) - sc;
    const unsigned long long al = (unsigned long long)(uint32_t)Q0 * cm;
    const long long ah = (Q0 >> 32) * (long long)cm + (long long)(al >> 32);
    const long long bl = (long long)(uint32_t)W0 * (long long)qs;
    const long long bh = (W0 >> 32) * (long long)qs + (bl >> 32);
    const unsigned long long lo = (unsigned long long)(uint32_t)al + (uint32_t)bl;
    const long long hi = ah + bh + (long long)(lo >> 32);
    const uint32_t s = (uint32_t)(hi >> 63);
    const unsigned long long l0 = (unsigned long long)((uint32_t)lo ^ s) + (s & 1u);
    const unsigned long long h0 = ((unsigned long long)hi ^ (unsigned long long)(hi >> 63)) + (l0 >> 32);
    const int sd = d >> 31;
    sg ^= s ^ (uint32_t)sd;
    const uint32_t dm = (uint32_t)((d ^ sd) - sd);
    const unsigned long long t0 = (unsigned long long)(uint32_t)l0 * dm;
    const unsigned long long t1 = (unsigned long long)(uint32_t)h0 * dm + (t0 >> 32);
    const unsigned long long t2 = (h0 >> 32) * dm + (t1 >> 32);
    p[0] = (uint32_t)t0;
    p[1] = (uint32_t)t1;
    p[2] = (uint32_t)t2;
    p[3] = (uint32_t)(t2 >> 32);
}

// |sum_{r < m} prod_{r' != r} x'_r'| mod 2^(32L) for terms i and i + 1 into p;
// bit 31 of sg[t] is term t's sign.  1 <= m <= kExpandHalves * K.  The branches
// on m are the same for every thread of the grid.  Bernoulli(0.5) columns at
// n = 36 mostly hold 11 to 14 ones, two or three halves.
template <int N, int L, int G>
__device__ __forceinline__ void terms_expanded(const int (&xt)[N], const int* __restrict__ de, int i, int m,
                                               uint32_t (&p)[kPair][L], uint32_t (&sg)[kPair])
{
#pragma unroll
    for (int t = 0; t < kPair; ++t) {
#pragma unroll
        for (int l = 0; l < L; ++l) p[t][l] = 0u;
        sg[t] = 0u;
    }
    long long W0[kPair], Q0[kPair];
    word_dual<N, G, 0>(xt, de, i, m, W0, Q0);
    if (rows_in_half(N, 2) > 0 && m > 3 * half_rows(N)) {
        if constexpr (rows_in_half(N, 2) > 0) {
            long long W1[kPair], Q1[kPair];
            word_dual<N, G, 1>(xt, de, i, m, W1, Q1);
#pragma unroll
            for (int t = 0; t < kPair; ++t) join_words<L>(W0[t], Q0[t], W1[t], Q1[t], p[t], sg[t]);
        }
    } else if (rows_in_half(N, 2) > 0 && m > 2 * half_rows(N)) {
        if constexpr (rows_in_half(N, 2) > 0) {
            int c[kPair], q[kPair], d[kPair] = {1, 1};
            half_any<N, G, 2>(xt, de, i, m, c, q);
            if constexpr (rows_in_half(N, 3) > 0) half_plain<N, G, 3>(xt, de, i, d);
#pragma unroll
            for (int t = 0; t < kPair; ++t) join_half<L>(W0[t], Q0[t], c[t], q[t], d[t], p[t], sg[t]);
        }
    } else {
#pragma unroll
        for (int t = 0; t < kPair; ++t) {
            const unsigned long long q = magnitude(Q0[t], sg[t]);
            p[t][0] = (uint32_t)q;
            p[t][1] = (uint32_t)(q >> 32);
        }
        if constexpr (rows_in_half(N, 2) > 0) {
            long long W1[kPair];
            word_plain<N, G, 1>(xt, de, i, W1);
#pragma unroll
            for (int t = 0; t < kPair; ++t) fold64<L, 2>(p[t], magnitude(W1[t], sg[t]));
        }
    }
    plain_words<N, L, G, 2>(xt, de, i, p, sg);
}

// Sum over one unit: sum_d (-1)^popc(d) prod_r (xt_r + DEI[d][r]), or with X
// the expanded walk's terms.
template <int N, int L, bool X>
__device__ __forceinline__ void unit_sum_bin(const int (&xt)[N], const int* __restrict__ s_de, int nq, int m,
                                             uint32_t (&acc)[L])
{
    constexpr int G = 4;
#pragma unroll
    for (int l = 0; l < L; ++l) acc[l] = 0u;
#pragma unroll 1
    for (int q = 0; q < nq; ++q) {
        const int* de = s_de + q * (N * G);
        // signs: the product's (bit 31 of the returned word) and the group
        // pattern + - - + relative to popc(q); an all-ones mask subtracts
        const uint32_t flip = (__popc(q) & 1) ? 0x80000000u : 0u;
        if constexpr (X) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {  // + - then - +
                uint32_t p[kPair][L], sg[kPair];
                terms_expanded<N, L, G>(xt, de, 2 * h, m, p, sg);
                const uint32_t f = flip ^ (h ? 0x80000000u : 0u);
                limb_add_masked<L>(acc, p[0], (uint32_t)((int32_t)(sg[0] ^ f) >> 31));
                limb_add_masked<L>(acc, p[1], (uint32_t)((int32_t)(sg[1] ^ f ^ 0x80000000u) >> 31));
            }
            continue;
        }
        uint32_t p[L];
        uint32_t sg = term_product<N, L, G>(xt, de, 0, p);
        limb_add_masked<L>(acc, p, (uint32_t)((int32_t)(sg ^ flip) >> 31));
        sg = term_product<N, L, G>(xt, de, 1, p);
        limb_add_masked<L>(acc, p, (uint32_t)((int32_t)(sg ^ flip ^ 0x80000000u) >> 31));
        sg = term_product<N, L, G>(xt, de, 2, p);
        limb_add_masked<L>(acc, p, (uint32_t)((int32_t)(sg ^ flip ^ 0x80000000u) >> 31));
        sg = term_product<N, L, G>(xt, de, 3, p);
        limb_add_masked<L>(acc, p, (uint32_t)((int32_t)(sg ^ flip) >> 31));
    }
}

template <int L>
__device__ __forceinline__ void shfl_add(uint32_t (&v)[L], int m)
{
    uint32_t o[L];
#pragma unroll
    for (int l = 0; l < L; ++l) o[l] = __shfl_xor_sync(0xffffffffu, v[l], m);
    limb_add<L>(v, o);
}

// Threads per CTA.  Plain walk: 512 (128 registers) keeps 4 limbs spill-free up
// to n = 28; larger n or more limbs get 255 registers at 256 threads.  Expanded
// walk, which holds fewer limbs at a time: 512 up to n = 40 (126 registers at
// n = 36 with 5 limbs; n = 37 and 38 spill, and still take 393 and 798 ms
// against 436 and 854 at 384 threads), 384 (168 registers) up to n = 44, then 256.
__host__ __device__ constexpr int bin_max_threads(int n, int limbs, bool x)
{
    if (x) return n <= 40 ? 512 : (n <= 44 ? 384 : 256);
    return (limbs <= 4 && n <= 28) ? 512 : 256;
}

template <int N, int L, bool X>
__global__ void __launch_bounds__(bin_max_threads(N, L, X), 1) walk_binary(Problem pb)
{
    constexpr int G = 4;
    extern __shared__ __align__(16) int smem_i[];
    const int w = pb.w, terms = 1 << w, nq = terms / G, ntop = N - 1 - (X ? 1 : 0) - w;
    const int tid = threadIdx.x, bd = blockDim.x;
    int* s_de = smem_i;
    int8_t* s_mt = reinterpret_cast<int8_t*>(s_de + terms * N);
    for (int i = tid; i < terms * N; i += bd) s_de[i] = pb.dei[i];
    for (int i = tid; i < ntop * N; i += bd) s_mt[i] = pb.mt[i];
    __syncthreads();

    const unsigned long long T = (unsigned long long)gridDim.x * bd;
    const unsigned long long t = (unsigned long long)blockIdx.x * bd + tid;
    unsigned long long u0, u1;
    balanced_range(pb.units, T, t, &u0, &u1);
    uint32_t tot[L];
#pragma unroll
    for (int l = 0; l < L; ++l) tot[l] = 0u;
    if (u0 < u1) {
        int xt[N];
        const unsigned long long g0 = gray_of(u0);
#pragma unroll
        for (int r = 0; r < N; ++r) xt[r] = pb.x0[r];
        for (int j = 0; j < ntop; ++j) {  // columns outermost, rows independent
            if (!((g0 >> j) & 1ull)) continue;
#pragma unroll
            for (int r = 0; r < N; ++r) xt[r] += s_mt[j * N + r];
        }
        unsigned long long u = u0;
        while (true) {
            uint32_t us[L];
            unit_sum_bin<N, L, X>(xt, s_de, nq, X ? pb.m : 0, us);
            if (u & 1ull) limb_sub<L>(tot, us);
            else limb_add<L>(tot, us);
            if (++u >= u1) break;
            const int j = __ffsll((long long)u) - 1;
            const int sg = ((gray_of(u) >> j) & 1ull) ? 1 : -1;
            const int8_t* col = s_mt + j * N;
#pragma unroll
            for (int r = 0; r < N; ++r) xt[r] += sg * col[r];
        }
    }
    // warp -> block -> grid (exact; order only affects speed)
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) shfl_add<L>(tot, m);
    __shared__ uint32_t s_warp[16][kMaxLimbs];
    __shared__ int s_last;
    const int lane = tid & 31, wid = tid >> 5, nw = bd >> 5;
    if (lane == 0)
#pragma unroll
        for (int l = 0; l < L; ++l) s_warp[wid][l] = tot[l];
    __syncthreads();
    if (wid == 0) {
        uint32_t v[L];
#pragma unroll
        for (int l = 0; l < L; ++l) v[l] = lane < nw ? s_warp[lane][l] : 0u;
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) shfl_add<L>(v, m);
        if (lane == 0) {
#pragma unroll
            for (int l = 0; l < L; ++l) pb.partials[blockIdx.x * L + l] = v[l];
            __threadfence();
            unsigned prev = atomicAdd(pb.ticket, 1u);
            s_last = (prev == gridDim.x - 1) ? 1 : 0;
        }
    }
    __syncthreads();
    if (s_last && wid == 0) {
        __threadfence();
        uint32_t v[L];
#pragma unroll
        for (int l = 0; l < L; ++l) v[l] = 0u;
        for (int b = lane; b < (int)gridDim.x; b += 32) {
            uint32_t o[L];
#pragma unroll
            for (int l = 0; l < L; ++l) o[l] = __ldcg(pb.partials + b * L + l);
            limb_add<L>(v, o);
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) shfl_add<L>(v, m);
        if (lane == 0) {
#pragma unroll
            for (int l = 0; l < L; ++l) pb.result[l] = v[l];
            *pb.ticket = 0u;
        }
    }
}

// Launches walk_binary<pb.n, pb.limbs, pb.m > 0>; with per_sm set, launches nothing
// and stores the CTAs per SM that the launch shape allows.
int launch_binary(const Problem& pb, int blocks, int threads, size_t smem, cudaStream_t s, int* per_sm = nullptr);

}  // namespace binary
}  // namespace spb
