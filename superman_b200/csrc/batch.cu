// Many small permanents in one launch: one warp per matrix, a CTA or a cluster
// each where there are too few matrices for that (choose_split).
//
// The whole-GPU walk (dense_impl.cuh) spreads one permanent over every SM;
// for n <= 24 a permanent is too small for that (2^(n-1) terms, a few
// microseconds of FP64 work) and launch latency dominates.  Here each warp
// takes a matrix of the batch (grid-stride over the batch), builds its row
// scaling, double-double NW start vector, low-column subset-sum table and
// high columns in the warp's slice of shared memory, then its 32 lanes split
// the Gray units of that matrix exactly as the threads of the big walk do
// (same unit evaluators; the double-double unit bases live in registers), and
// their sums are added up in double-double, in one order whatever the launch's
// split (kLeaves).  A matrix with a pivot column
// (dense_impl.cuh) takes the derivative walk, half the subsets at 3/4 (complex
// 5/6) of the FP64 instructions, the others the plain walk; the choice is the
// warp's own.  The permanent of matrix m
// is written as (hi, lo) per component: out[m*2*comps + 2*c + {0, 1}].
//
// Device pointers only, no allocation, no host synchronisation: the serving
// loop captures one launch per batch shape in a CUDA graph, and the
// decomposition path runs its independent pieces through it.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>

#include "batch.h"
#include "dense_impl.cuh"
#include "per_device.h"
#include "spb_common.cuh"

namespace cg = cooperative_groups;

namespace spb {
namespace batch {

constexpr int kWarpsPerCta = 4;
constexpr int kMaxCluster = 8;  // CTAs that may share a matrix (the portable cluster size)

// D: the derivative walk; T: threads that share the slice.
template <int N, int C, bool D, int T>
struct Cfg {
    static constexpr int NC = N - (D ? 1 : 0);           // walked columns
    // low column bits per unit.  A unit's base costs about 10 operations per row,
    // a tenth of a real unit's work at 32 terms, 6 % of a complex one's.  Real
    // matrices of n >= 18 take 64 terms (three CTAs per SM stay, the registers'
    // limit): 4096 x n=20 4825 -> 4533 us, 1500 x n=24 34.6 -> 32.3 ms, errors as
    // before.  Complex ones would leave room for one CTA per SM.
    static constexpr int LOW = C == 1 && N >= 18 ? 6 : 5;
    static constexpr int W = NC - 1 < LOW ? NC - 1 : LOW;
    static constexpr int G = C == 1 ? (W >= 2 ? 4 : (W == 1 ? 2 : 1)) : (W >= 1 ? 2 : 1);
    static constexpr int TERMS = 1 << W;
    static constexpr int NTOP = NC - 1 - W;
    static constexpr int NTP = NTOP > 0 ? NTOP : 0;
    // Unit-base lo words: registers, except complex n >= 21, where hi and lo
    // of both parts (4n doubles) would spill; there they sit in a lane-private
    // slot of the shared slice.  (With 32 terms per unit the slot's
    // per-unit traffic costs more than it saves wherever registers suffice.)
    static constexpr bool LO_SMEM = C == 2 && N >= 21;
    static constexpr int LO_DOUBLES = LO_SMEM ? T * N * C : 0;
    // doubles per slice: DE table, walked columns (with low words in the
    // derivative walk), x0 hi/lo, lo words, row exponents (as doubles),
    // rounded up to 32 bytes: the unit evaluator reads the DE table with
    // 16-byte vector loads, so every slice must start aligned.
    static constexpr int SMEM_DOUBLES =
        (TERMS * N * C + (D ? 2 : 1) * NC * N * C + 2 * N * C + LO_DOUBLES + N + 3) / 4 * 4;
    static_assert(SMEM_DOUBLES % 4 == 0, "shared slice must keep 32-byte alignment");
};

// Sizes that have a derivative walk, and the slice that holds either walk.
// Below n = 11 the pivot and the quotients cost a matrix more than the walk saves
// (4096 matrices on one B200, plain against derivative: n=8 real 25.6 and 27.7 us,
// complex 60.7 and 64.0; n=12 real 52.4 and 46.2, n=14 complex 347 and 295).
__host__ __device__ constexpr bool has_deriv(int n) { return n >= 11; }
template <int N, int C, int T>
constexpr int slice_doubles()
{
    constexpr int p = Cfg<N, C, false, T>::SMEM_DOUBLES;
    if constexpr (has_deriv(N)) {
        constexpr int d = Cfg<N, C, true, T>::SMEM_DOUBLES;
        return d > p ? d : p;
    }
    return p;
}

// The threads that share a matrix's tables: one warp, or (CTA) a whole CTA.
template <bool CTA>
struct Team {
    static constexpr int kSize = CTA ? kWarpsPerCta * 32 : 32;
    __device__ __forceinline__ static int rank() { return CTA ? threadIdx.x : (threadIdx.x & 31); }
    __device__ __forceinline__ static void sync()
    {
        if (CTA) __syncthreads();
        else __syncwarp();
    }
    // sync, and whether v holds for any of the threads (a warp's vote orders no
    // memory by itself)
    __device__ __forceinline__ static bool any(bool v)
    {
        if (CTA) return __syncthreads_or(v) != 0;
        v = __any_sync(0xffffffffu, v) != 0;
        __syncwarp();
        return v;
    }
};

// The order of a matrix's sum (n >= 16, where launches differ in how they split a
// matrix).  Its units fall into kLeaves runs of equal length (fewer where there
// are fewer units); a run's unit sums are added one after the other, the runs'
// sums pairwise as a binary tree over the runs in their order.  A thread owns a
// power of two of neighbouring runs, a warp's, a CTA's and a cluster's threads
// neighbouring ranges, so every split adds up the same tree, and a permanent's
// bits do not depend on how many matrices are launched with it.  (A row value
// carried from unit to unit and one built anew differ by 2^-100: the bits agree
// unless one lies that close to a rounding boundary.)  A thread's
// own levels of the tree (five of them, one warp per matrix) cost little: 4096 x
// n=16 292 -> 297 us against sums in each split's own order, n=17 567 -> 574 us,
// n=20 4532 -> 4548 us, 148 x n=24 3213 -> 3228 us.
constexpr int kLeaves = kMaxCluster * kWarpsPerCta * 32;

template <int C>
struct RunTree {
    dd level[C][6];  // sums of 2^l runs, waiting for their neighbours
    // Adds the thread's run number i, whose sum is tot; the sum of all runs so far
    // is then in tot when i + 1 is a power of two, else tot is to start at zero.
    __device__ __forceinline__ void add(unsigned i, bool last, dd (&tot)[C])
    {
        int l = 0;
        for (; (i >> l) & 1u; ++l)
#pragma unroll
            for (int c = 0; c < C; ++c) tot[c] = dd_add(level[c][l], tot[c]);
        if (last) return;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            level[c][l] = tot[c];
            tot[c] = {0.0, 0.0};
        }
    }
};

// Neighbouring lanes first (dd_add gives both of them the same bits).
__device__ __forceinline__ dd warp_tree_dd(dd v)
{
#pragma unroll
    for (int m = 1; m <= 16; m <<= 1) v = dd_add(v, shfl_xor_dd(v, m));
    return v;
}

// The sum of count (a power of two) values, pairwise in order; v is overwritten.
__device__ __forceinline__ dd tree_dd(dd* v, int count)
{
    for (int step = 1; step < count; step *= 2)
        for (int i = 0; i + step < count; i += 2 * step) v[i] = dd_add(v[i], v[i + step]);
    return v[0];
}

// One matrix, its rows' scaling exponents in s_exp: tables in the team's slice,
// then the walk over part `part` of `parts` teams' units; the warp's total (in
// every lane).  pivot: the derivative walk's column.
template <int N, int C, bool D, bool CTA>
__device__ __forceinline__ void walk_matrix(const double* __restrict__ A, const int* s_exp, int pivot, double* slice,
                                            int part, int parts, dd (&tot)[C])
{
    using TM = Team<CTA>;
    const int rank = TM::rank();
    using Q = Cfg<N, C, D, TM::kSize>;
    constexpr int G = Q::G, TERMS = Q::TERMS, NTOP = Q::NTOP, NTP = Q::NTP, W = Q::W, NC = Q::NC;
    double* s_de = slice;                    // [C][TERMS/G][N][G]
    double* s_col = s_de + TERMS * N * C;    // [C][NC][N] walked columns: entries or quotients
    double* s_cl = s_col + NC * N * C;       // their low words (derivative walk)
    double* s_x0h = s_cl + (D ? NC * N * C : 0);  // [C][N]
    double* s_x0l = s_x0h + N * C;           // [C][N]
    double* s_lo = s_x0l + N * C;            // [C][N][threads] thread-private lo words (LO_SMEM)
    const double* s_mt = s_col + W * N;      // high columns of part c at + c * NC * N
    const double* s_ml = s_cl + W * N;
    for (int idx = rank; idx < NC * N; idx += TM::kSize) {
        const int j = idx / N, r = idx % N, src = D && j >= pivot ? j + 1 : j;
        const double* row = A + (size_t)r * N * C;
        if constexpr (!D) {
#pragma unroll
            for (int c = 0; c < C; ++c) s_col[c * NC * N + idx] = ldexp(row[src * C + c], -s_exp[r]);
        } else if constexpr (C == 1) {
            const dd v = dense::quotient(ldexp(row[src], -s_exp[r]), ldexp(row[pivot], -s_exp[r]));
            s_col[idx] = v.hi;
            s_cl[idx] = v.lo;
        } else {
            const dense::ddc v = dense::quotient_c(
                ldexp(row[2 * src], -s_exp[r]), ldexp(row[2 * src + 1], -s_exp[r]), ldexp(row[2 * pivot], -s_exp[r]),
                ldexp(row[2 * pivot + 1], -s_exp[r]));
            s_col[idx] = v.re.hi;
            s_cl[idx] = v.re.lo;
            s_col[NC * N + idx] = v.im.hi;
            s_cl[NC * N + idx] = v.im.lo;
        }
    }
    TM::sync();
    auto plus = [&](dd x, int i) { return D ? dense::dd_step(x, s_col[i], s_cl[i]) : dd_add_d(x, s_col[i]); };
    // NW start vector (double-double)
    for (int rr = rank; rr < N * C; rr += TM::kSize) {
        const int r = rr / C, part = rr % C;
        dd s = {0.0, 0.0};
        for (int j = 0; j < NC; ++j) s = plus(s, (part * NC + j) * N + r);
        dd h = {-0.5 * s.hi, -0.5 * s.lo};
        dd x = plus(h, (part * NC + NC - 1) * N + r);
        s_x0h[part * N + r] = x.hi;
        s_x0l[part * N + r] = x.lo;
    }
    // low-column subset sums, grouped [part][d/G][r][d%G]
    for (int idx = rank; idx < TERMS * N * C; idx += TM::kSize) {
        const int part = idx / (TERMS * N), rem = idx % (TERMS * N);
        const int d = rem / N, r = rem % N;
        dd s = {0.0, 0.0};
        for (int j = 0; j < W; ++j)
            if ((d >> j) & 1) s = plus(s, (part * NC + j) * N + r);
        s_de[part * TERMS * N + ((d / G) * N + r) * G + (d % G)] = s.hi;
    }
    TM::sync();

    unsigned long long u0, u1;
    balanced_range(1ull << NTP, (unsigned long long)parts * TM::kSize, (unsigned long long)part * TM::kSize + rank, &u0,
                   &u1);
#pragma unroll
    for (int c = 0; c < C; ++c) tot[c] = {0.0, 0.0};
    constexpr unsigned long long UNITS = 1ull << NTP, RUN = UNITS > kLeaves ? UNITS / kLeaves : 1;
    RunTree<C> tree;
    if (u0 < u1) {
        // unit base: hi words in registers; lo words in registers or in the
        // thread's shared slot (element (c, r) at [(c * N + r) * LS + rank])
        double xh[C][N];
        double xlr[Q::LO_SMEM ? 1 : C * N];
        double* xl = Q::LO_SMEM ? s_lo + rank : xlr;
        constexpr int LS = Q::LO_SMEM ? TM::kSize : 1;  // stride between elements
        const unsigned long long g0 = gray_of(u0);
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int r = 0; r < N; ++r) {
                dd x = {s_x0h[c * N + r], s_x0l[c * N + r]};
                for (int j = 0; j < NTOP; ++j)
                    if ((g0 >> j) & 1ull) x = plus(x, (c * NC + W + j) * N + r);
                xh[c][r] = x.hi;
                xl[(c * N + r) * LS] = x.lo;
            }
        unsigned long long u = u0;
        while (true) {
            if constexpr (C == 1) {
                const double us = D ? dense::unit_sum_deriv<N, G>(xh[0], s_de, TERMS / G)
                                    : dense::unit_sum_real<N, G>(xh[0], s_de, TERMS / G);
                tot[0] = dd_add_d(tot[0], (u & 1ull) ? -us : us);
            } else {
                double ur, ui;
                if constexpr (D)
                    dense::unit_sum_complex_deriv<N, G>(xh[0], xh[C - 1], s_de, s_de + TERMS * N, TERMS / G, ur, ui);
                else
                    dense::unit_sum_complex<N, G>(xh[0], xh[C - 1], s_de, s_de + TERMS * N, TERMS / G, ur, ui);
                if (u & 1ull) { ur = -ur; ui = -ui; }
                tot[0] = dd_add_d(tot[0], ur);
                tot[C - 1] = dd_add_d(tot[C - 1], ui);
            }
            if (N >= 16 && ((u + 1) & (RUN - 1)) == 0) tree.add((unsigned)((u - u0) / RUN), u + 1 >= u1, tot);
            if (++u >= u1) break;
            const int j = __ffsll((long long)u) - 1;
            const bool add = (gray_of(u) >> j) & 1ull;
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int r = 0; r < N; ++r) {
                    const double v = s_mt[(c * NC + j) * N + r];
                    dd s = two_sum(xh[c][r], add ? v : -v);
                    double l = xl[(c * N + r) * LS];
                    if (D) {
                        const double m = s_ml[(c * NC + j) * N + r];
                        l = add ? add_rn(l, m) : sub_rn(l, m);
                    }
                    dd z = fast_two_sum(s.hi, add_rn(s.lo, l));
                    xh[c][r] = z.hi;
                    xl[(c * N + r) * LS] = z.lo;
                }
        }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) tot[c] = warp_tree_dd(tot[c]);
}

// Matrix m of a batch starts at mats + m*N*N*C, or, with an offset table, at
// mats + offs[m] * kOffsetUnit doubles (the serving loop's device pool).

// With `src` (the serving loop's page-locked host mirror, mapped into the
// device's address space, at the same offsets), each warp first copies its
// matrix from src into its place in mats, so every matrix crosses the host
// link once, in coalesced reads that overlap the other warps' work.
// SPLIT: a matrix is one CTA's, or shared by the CTAs of a cluster (part of the
// units each, tables of its own); else one warp's.  A split matrix's CTAs meet in
// distributed shared memory (no workspace, so the launch still allocates nothing).
template <int N, int C, bool SPLIT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) batch_walk(double* __restrict__ mats,
                                                                 const unsigned* __restrict__ offs,
                                                                 const double* __restrict__ src,
                                                                 int count, double* __restrict__ out)
{
    using TM = Team<SPLIT>;
    constexpr int SLICE = slice_doubles<N, C, TM::kSize>();
    extern __shared__ __align__(16) double smem[];
    __shared__ dd s_part[C][kWarpsPerCta];  // SPLIT: the CTA's warps' totals, then (first CTA) ...
    __shared__ dd s_cta[C][kMaxCluster];    // ... the cluster's CTAs' totals
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, rank = TM::rank();
    double* slice = smem + (SPLIT ? 0 : (size_t)wid * SLICE);
    int* s_exp = reinterpret_cast<int*>(slice + SLICE - N);  // [N], past either walk's arrays
    cg::cluster_group cluster = cg::this_cluster();
    const int parts = SPLIT ? (int)cluster.num_blocks() : 1, part = SPLIT ? (int)cluster.block_rank() : 0;

    // A CTA's shared memory may be written by another of its cluster only once it
    // has started: each arrives here and waits before the first such write.
    if constexpr (SPLIT) cluster.barrier_arrive();
    bool started = false;
    const int teams = SPLIT ? gridDim.x / parts : gridDim.x * kWarpsPerCta;
    for (int m = SPLIT ? blockIdx.x / parts : blockIdx.x * kWarpsPerCta + wid; m < count; m += teams) {
        const size_t base = offs ? (size_t)offs[m] * kOffsetUnit : (size_t)m * N * N * C;
        const double* A = mats + base;
        if constexpr (SPLIT) {
            // each CTA stages the matrix for itself; the first also brings a
            // source matrix into its place
            double* stage = slice + SLICE;
            const double* from = src ? src + base : A;
            for (int i = rank; i < N * N * C; i += TM::kSize) {
                const double v = from[i];
                stage[i] = v;
                if (src && part == 0) mats[base + i] = v;
            }
            A = stage;
            TM::sync();
        } else if (src) {
            for (int i = rank; i < N * N * C; i += TM::kSize) mats[base + i] = src[base + i];
            TM::sync();  // orders the warp's writes before its reads below
        }
        // row exponents: row max scaled into [0.5, 1)
        bool any = false;  // a nonzero (or NaN) entry
        for (int r = rank; r < N; r += TM::kSize) {
            double mx = 0.0;
            for (int j = 0; j < N * C; ++j) {
                const double v = A[r * N * C + j];
                mx = fmax(mx, fabs(v));
                any |= v != 0.0;
            }
            int e = 0;
            if (mx > 0.0 && isfinite(mx)) frexp(mx, &e);
            s_exp[r] = e;
        }
        // A matrix of zeros (the serving loop fills its batches up with them)
        // takes no walk, which would be the plain one, the slower.
        any = TM::any(any);
        dd tot[C];
#pragma unroll
        for (int c = 0; c < C; ++c) tot[c] = {0.0, 0.0};
        int pivot = -1;
        if constexpr (has_deriv(N)) {
            pivot = dense::pick_pivot(N, false, [&](int r, int j) {
                const double* e = A + ((size_t)r * N + j) * C;
                return ldexp(C == 1 ? fabs(e[0]) : fmax(fabs(e[0]), fabs(e[C - 1])), -s_exp[r]);
            });
            if (pivot >= 0) walk_matrix<N, C, true, SPLIT>(A, s_exp, pivot, slice, part, parts, tot);
        }
        if (pivot < 0 && any) walk_matrix<N, C, false, SPLIT>(A, s_exp, pivot, slice, part, parts, tot);
        if constexpr (SPLIT) {
            if (lane == 0)
#pragma unroll
                for (int c = 0; c < C; ++c) s_part[c][wid] = tot[c];
            __syncthreads();
            if (!started) cluster.barrier_wait();  // long since complete: no CTA is waited for
            started = true;
            if (threadIdx.x == 0)
#pragma unroll
                for (int c = 0; c < C; ++c)
                    *cluster.map_shared_rank(&s_cta[c][part], 0) = tree_dd(s_part[c], kWarpsPerCta);
            cluster.sync();
            if (part == 0 && wid == 0)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    dd v[kMaxCluster];
#pragma unroll
                    for (int b = 0; b < kMaxCluster; ++b) v[b] = b < parts ? s_cta[c][b] : dd{0.0, 0.0};
                    tot[c] = tree_dd(v, kMaxCluster);  // (adding the zeros changes nothing)
                }
        }
        if (part == 0 && (!SPLIT || wid == 0)) {
            int es = 0;
            for (int r = 0; r < N; ++r) es += s_exp[r];
            bool odd = N % 2 != 0;  // perm = (4(nc%2)-2) * total over nc walked columns
            if constexpr (has_deriv(N))
                if (pivot >= 0) {  // times the product of the pivots
                    const dense::DerivScale sc = dense::deriv_scale<C>(N, [&](int r) {
                        const double* d = A + ((size_t)r * N + pivot) * C;
                        return make_double2(ldexp(d[0], -s_exp[r]), ldexp(d[C - 1], -s_exp[r]));
                    });
                    if constexpr (C == 1) {
                        tot[0] = dd_mul(tot[0], sc.v.re);
                    } else {
                        const dense::ddc t = dense::ddc_mul(dense::ddc{tot[0], tot[1]}, sc.v);
                        tot[0] = t.re;
                        tot[1] = t.im;
                    }
                    es += sc.e;
                    odd = !odd;
                }
            if (lane == 0) {
                const double sgn = odd ? 1.0 : -1.0;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    out[(size_t)m * 2 * C + 2 * c] = sgn * ldexp(tot[c].hi, es + 1);
                    out[(size_t)m * 2 * C + 2 * c + 1] = sgn * ldexp(tot[c].lo, es + 1);
                }
            }
        }
        // the slice and the totals are rewritten for the next matrix (and no CTA
        // of a cluster leaves while another may still write to it)
        if (SPLIT) cluster.sync();
        else __syncwarp();
    }
}

// CTAs per matrix: 0 for a warp per matrix, else a power of two up to
// kMaxCluster, by the walks that the busiest SM is given.  An SM's FP64 pipe is
// 0.6 busy with one CTA of four warps and little busier with more, so what counts
// is how evenly the parts fill the SMs: `rounds` CTAs of 1/c of a matrix, where a
// warp per matrix hands them out four matrices at a time.  Every CTA builds
// tables of its own: kTables of the walk at n=16, where the whole is 8 us of the
// pipe, less in proportion at larger n.  Clusters of 4 and 8 leave some SMs of a
// GPC over.  On one B200 (all with 32 terms
// per unit) the choice takes 1024 x n=20 from 1448 us (a warp each) to 1248 us,
// 700 x n=22 from 6324 to 3851 us, complex 24488 to 12531 us, 16 x n=16 from 33
// to 27 us (one CTA each, four).  top: high column bits, 2^top units.
int choose_split(int n, int top, int count, int sms)
{
    constexpr double kTables = 0.43, kShared = 0.92;  // kShared: a round's time beside other CTAs
    const double tables = kTables * 16.0 / n * std::ldexp(1.0, 16 - n);
    auto cost = [&](double ctas, double on, double work) {
        const double rounds = std::ceil(ctas / on);
        return rounds * work * (rounds > 1.0 ? kShared : 1.0);
    };
    double best = cost(std::ceil((double)count / kWarpsPerCta), sms, kWarpsPerCta);
    int split = 0;
    for (int c = 1; c <= kMaxCluster && (1ll << top) >= (long long)c * kWarpsPerCta * 32; c *= 2) {
        const double on = sms * (c == 8 ? 13.0 / 16.0 : c == 4 ? 15.0 / 16.0 : 1.0);
        const double t = cost((double)count * c, on, 1.0 / c + tables);
        if (t < best) {
            best = t;
            split = c;
        }
    }
    return split;
}

template <int N, int C, bool SPLIT>
int launch_split(double* mats, const unsigned* offs, const double* src, int count, double* out, int blocks,
                 int cluster, cudaStream_t s)
{
    constexpr size_t smem =
        sizeof(double) *
        (SPLIT ? slice_doubles<N, C, kWarpsPerCta * 32>() + N * N * C : slice_doubles<N, C, 32>() * kWarpsPerCta);
    if (smem > 48 * 1024) {
        static OncePerDevice<cudaError_t> ready;
        int dev = 0;
        SPB_CUDA_TRY(cudaGetDevice(&dev));
        SPB_CUDA_TRY(ready(dev, [] {
            return cudaFuncSetAttribute(batch_walk<N, C, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem);
        }));
    }
    if constexpr (!SPLIT) {
        batch_walk<N, C, false><<<blocks, kWarpsPerCta * 32, smem, s>>>(mats, offs, src, count, out);
        SPB_CUDA_TRY(cudaGetLastError());
        return SPB_OK;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kWarpsPerCta * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    SPB_CUDA_TRY(cudaLaunchKernelEx(&cfg, batch_walk<N, C, SPLIT>, mats, offs, src, count, out));
    return SPB_OK;
}

template <int N, int C>
int launch_n(double* mats, const unsigned* offs, const double* src, int count, double* out, int sms,
             cudaStream_t s)
{
    if constexpr (N >= 16) {
        const int c = choose_split(N, Cfg<N, C, has_deriv(N), 32>::NTOP, count, sms);
        if (c > 0) return launch_split<N, C, true>(mats, offs, src, count, out, count * c, c, s);
    }
    int blocks = (count + kWarpsPerCta - 1) / kWarpsPerCta;
    const int cap = sms * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return launch_split<N, C, false>(mats, offs, src, count, out, blocks, 1, s);
}

int dispatch(double* mats, const unsigned* offs, const double* src, int n, int is_complex, int count, double* out,
             int sms, cudaStream_t s)
{
    const int key = n * 2 + (is_complex ? 1 : 0);
    switch (key) {
#define SPB_BCASE(N)                                                               \
    case 2 * N: return launch_n<N, 1>(mats, offs, src, count, out, sms, s);        \
    case 2 * N + 1: return launch_n<N, 2>(mats, offs, src, count, out, sms, s);
        SPB_BCASE(1) SPB_BCASE(2) SPB_BCASE(3) SPB_BCASE(4) SPB_BCASE(5) SPB_BCASE(6) SPB_BCASE(7)
        SPB_BCASE(8) SPB_BCASE(9) SPB_BCASE(10) SPB_BCASE(11) SPB_BCASE(12) SPB_BCASE(13)
        SPB_BCASE(14) SPB_BCASE(15) SPB_BCASE(16) SPB_BCASE(17) SPB_BCASE(18) SPB_BCASE(19)
        SPB_BCASE(20) SPB_BCASE(21) SPB_BCASE(22) SPB_BCASE(23) SPB_BCASE(24)
#undef SPB_BCASE
    default:
        spb_set_error("batched walk: unsupported n=%d", n);
        return SPB_ERR_INVALID;
    }
}

int launch_gathered(const double* src, double* dst, const unsigned* d_offs, int n, int is_complex, int count,
                    double* d_out, cudaStream_t s)
{
    if (n < 1 || n > kMaxN || count < 0) {
        spb_set_error("batched walk: n=%d outside 1..%d or negative count", n, kMaxN);
        return SPB_ERR_INVALID;
    }
    if (count == 0) return SPB_OK;
    int dev = 0, sms = 0;
    SPB_CUDA_TRY(cudaGetDevice(&dev));
    SPB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return dispatch(dst, d_offs, src, n, is_complex, count, d_out, sms, s);
}

}  // namespace batch
}  // namespace spb

extern "C" int spb_perm_batch_dev(const double* d_mats, int n, int is_complex, int count, double* d_out,
                                  void* stream)
{
    using namespace spb::batch;
    if (!d_mats || !d_out || count < 0) {
        spb_set_error("spb_perm_batch_dev: null pointer or negative count");
        return SPB_ERR_INVALID;
    }
    if (n < 1 || n > kMaxN) {
        spb_set_error("spb_perm_batch_dev: n=%d outside 1..%d (larger n: the whole-GPU entry points)", n, kMaxN);
        return SPB_ERR_INVALID;
    }
    if (count == 0) return SPB_OK;
    int dev = 0, sms = 0;
    SPB_CUDA_TRY(cudaGetDevice(&dev));
    SPB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // the matrices are read in place (the cast drops const: with no source
    // the kernel only reads them)
    return dispatch(const_cast<double*>(d_mats), nullptr, nullptr, n, is_complex, count, d_out, sms, s);
}
