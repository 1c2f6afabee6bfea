// Sparse real permanents by expansion row by row (spb_perm_sparse_f64, and the
// dense entry point on host matrices with zeros).
//
// Reference behaviour: spSingleGPU (Algorithms/GPU/Sparse/spSingleGPU.cuh:45-234)
// walks all 2^(n-1) subsets whatever the pattern.  When few columns are open
// at a time, i.e. have nonzeros both in rows already taken and in rows still
// to come, the permanent is far cheaper by the expansion
//   T_t[M] = sum over j in row t's columns within M of a_tj T_{t-1}[M - j],
// T_t[M] the sum of products over the ways rows 0..t can use exactly the
// column set M.  Only sets that hold every closed column (its last row taken)
// can lead to a perfect matching, so a set is indexed by the bits of the open
// columns alone: a step reads a table of 2^kb states and writes one of 2^ka,
// with no subset of 2^n ever formed.  Terms are added with their own signs
// only, so for non-negative entries nothing cancels (Ryser's sum does); all
// arithmetic is double-double in every precision mode.
//
// The plan (frontier_plan.cpp) orders the rows so that few columns are open
// (n=30, permutation plus three per row: 13-18; 1e5-2e6 states in all, against
// 2^29 Gray terms) and splits the order in two halves that advance at the
// same time, front rows forwards and back rows backwards, which halves the
// chain of dependent steps; at the cut the permanent is
//   sum_M front[M] back[open columns - M].
//
// What bounds it: the chain of steps, each a grid barrier (~1.3 us) and a round
// trip to L2 for its dependent loads, not bandwidth (2^18 states are 4 MB in
// L2) and not the FP64 pipe.  So the first, narrow steps of a half are run by
// one CTA in shared memory, the plan travels as the kernel's parameter
// (no copy before it), and the result is written into page-locked host memory
// (no copy after it).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "context.h"
#include "frontier.h"
#include "spb_common.cuh"

namespace cg = cooperative_groups;

namespace spb {
namespace frontier {
namespace {

constexpr int kThreads = 1024;
constexpr int kMaxCluster = 8;  // the portable cluster size
constexpr size_t kSmem = sizeof(double2) * 2 << kNarrow;  // 64 KB

// What the host reads: the total, and the device's global timer (ns) as the
// kernel began and ended.
struct Outcome {
    dd total;
    unsigned long long begin, end;
};

struct Tables {
    double2* t[2][2];    // [half][parity]: step s of a half writes parity s & 1
    dd* partials;        // [grid]
    unsigned* ticket;    // last-CTA election
    unsigned long long* begin;
    Outcome* out;        // page-locked host memory, mapped
};

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// A double-double sum of products a * t: the high words by TwoSum in order, all
// rounding errors and low words in one FP64 sum beside it (they are 2^-53 of the
// high words, so its own rounding is of the order of the result's).  The chain
// from entry to entry is one addition, not a normalised double-double one.
struct Sum {
    double hi = 0.0, lo = 0.0;
    __device__ __forceinline__ void add(double a, double2 t)
    {
        const double p = __dmul_rn(a, t.x);
        const double e = __fma_rn(a, t.y, __fma_rn(a, t.x, -p));
        const dd s = two_sum(hi, p);
        hi = s.hi;
        lo = add_rn(lo, add_rn(s.lo, e));
    }
    __device__ __forceinline__ double2 value() const
    {
        const dd v = two_sum(hi, lo);  // after cancellation lo may be the larger
        return make_double2(v.hi, v.lo);
    }
};

// State `idx` of the table after step `st`, from the table before it.  Four
// entries' states are loaded before the first is added, so a state waits for
// one round trip per four entries.  G: the table is in global memory, read
// through L2 (other CTAs wrote it), else in shared memory.
template <bool G>
__device__ __forceinline__ double2 advance(const Plan& P, const Step& st, const double2* from, unsigned idx)
{
    // the full index: `idx` with a one inserted at every closed column's bit
    unsigned full = idx;
    for (unsigned m = st.closed; m; m &= m - 1) {
        const unsigned low = (m & (0u - m)) - 1u;
        full = (full & low) | ((full & ~low) << 1) | (low + 1u);
    }
    Sum acc;
    if (__popc(full) == st.used) {
        for (int e0 = 0; e0 < st.entries; e0 += 4) {
            double2 t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                t[k] = make_double2(0.0, 0.0);
                if (e0 + k < st.entries) {
                    const unsigned bit = 1u << P.bit[st.entry + e0 + k], old = full ^ bit;
                    // the column is in the set, and no column this row opens is left in it
                    if ((full & bit) && (old >> st.kb) == 0u) t[k] = G ? __ldcg(from + old) : from[old];
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (e0 + k < st.entries) acc.add(P.val[st.entry + e0 + k], t[k]);
        }
    }
    return acc.value();
}

__device__ __forceinline__ dd dd_mul_dd(double2 a, double2 b) { return dd_mul(dd{a.x, a.y}, dd{b.x, b.y}); }

// COOP: the grid is launched cooperatively, else it is one cluster, whose
// barrier is several times cheaper and whose launch needs no residency check.
template <bool COOP>
__global__ void __launch_bounds__(kThreads, 1) expand_rows(const __grid_constant__ Plan A, const Tables T)
{
    auto sync_all = [] {
        if constexpr (COOP) cg::this_grid().sync();
        else cg::this_cluster().sync();
    };
    if (blockIdx.x == 0 && threadIdx.x == 0) *T.begin = global_ns();
    // The plan's used part goes to shared memory at once: read in place, every
    // step's first look at its row missed the constant cache anew (about 2 us
    // a step).
    __shared__ Plan P;
    {
        const unsigned* from = reinterpret_cast<const unsigned*>(&A);
        unsigned* to = reinterpret_cast<unsigned*>(&P);
        constexpr int head = offsetof(Plan, bit) / 4, bits = offsetof(Plan, val) / 4;
        const int nb = (A.total + 3) / 4, nw = head + nb + 2 * A.total;
        for (int i = threadIdx.x; i < nw; i += kThreads) {
            const int w = i < head + nb ? i : bits + (i - head - nb);
            to[w] = from[w];
        }
        __syncthreads();
    }
    extern __shared__ __align__(16) double2 s_tab[];  // [2][2^kNarrow]
    __shared__ dd s_warp[kThreads / 32];
    __shared__ int s_last;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;

    // narrow first steps, in shared memory: CTA 0 the front half, CTA 1 the
    // back half.  The state before the first step is the empty set, "written"
    // as step -1; the last table goes to global memory for the grid.
    if (blockIdx.x == 0 && tid == 0) *T.ticket = 0u;
    if (blockIdx.x < 2) {
        const int h = blockIdx.x, ns = h ? P.hb : P.hf;
        if (tid == 0) s_tab[1 << kNarrow] = make_double2(1.0, 0.0);
        if (ns == 0 && tid == 0) __stcg(T.t[h][1], make_double2(1.0, 0.0));
        for (int s = 0; s < ns; ++s) {
            __syncthreads();
            const Step& st = P.step[(h ? P.nf : 0) + s];
            const double2* from = s_tab + (((s + 1) & 1) << kNarrow);
            for (unsigned i = tid; i < (1u << st.ka); i += kThreads) {
                const double2 v = advance<false>(P, st, from, i);
                if (s + 1 < ns) s_tab[((s & 1) << kNarrow) + i] = v;
                else __stcg(T.t[h][s & 1] + i, v);
            }
        }
    }
    sync_all();
    // the remaining steps, one of each half at a time, over the whole grid
    const int wf = P.nf - P.hf, wb = P.nb - P.hb, wide = wf > wb ? wf : wb;
    const unsigned g = blockIdx.x * kThreads + tid, G = gridDim.x * kThreads;
    for (int k = 0; k < wide; ++k) {
        const unsigned cf = k < wf ? 1u << P.step[P.hf + k].ka : 0u;
        const unsigned cb = k < wb ? 1u << P.step[P.nf + P.hb + k].ka : 0u;
        for (unsigned i = g; i < cf + cb; i += G) {
            const int h = i < cf ? 0 : 1, s = (h ? P.hb : P.hf) + k;
            const unsigned at = h ? i - cf : i;
            __stcg(T.t[h][s & 1] + at, advance<true>(P, P.step[(h ? P.nf : 0) + s], T.t[h][(s + 1) & 1], at));
        }
        sync_all();
    }
    // the cut: front set M meets the back set of the other open columns
    const double2* front = T.t[0][(P.nf + 1) & 1];
    const double2* back = T.t[1][(P.nb + 1) & 1];
    dd sum = {0.0, 0.0};
    for (unsigned i = g; i < (1u << P.kcut); i += G) {
        const double2 f = __ldcg(front + i);
        if (f.x == 0.0 && f.y == 0.0) continue;
        unsigned j = 0;
        for (int b = 0; b < P.kcut; ++b) j |= ((~i >> b) & 1u) << P.back_bit[b];
        sum = dd_add(sum, dd_mul_dd(f, __ldcg(back + j)));
    }
    sum = warp_sum_dd(sum);
    if (lane == 0) s_warp[wid] = sum;
    __syncthreads();
    if (tid == 0) {
        dd v = s_warp[0];
        for (int w = 1; w < kThreads / 32; ++w) v = dd_add(v, s_warp[w]);
        T.partials[blockIdx.x] = v;
        __threadfence();
        s_last = atomicAdd(T.ticket, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (s_last && wid == 0) {  // the last CTA adds the CTAs' sums in a fixed order
        __threadfence();
        dd v = {0.0, 0.0};
        for (unsigned b = lane; b < gridDim.x; b += 32)
            v = dd_add(v, dd{__ldcg(&T.partials[b].hi), __ldcg(&T.partials[b].lo)});
        v = warp_sum_dd(v);
        if (lane == 0) *T.out = Outcome{v, __ldcg(T.begin), global_ns()};
    }
}

}  // namespace

// Fitted on one B200 to kernel times of 15 us (n=20, 10 narrow steps a half), 20 us
// (n=30, 15), 38 us (n=20, 10 and 3 wide), 59 us (n=34, 9 and 10), 109 us (n=30, 11
// wide, 4.4 million states) and 205 us (n=34, 13 wide, 10.5 million).
constexpr double kLaunch = 7e-6, kState = 13e-12;
double expansion_seconds(const Plan& p)
{
    const int wide = std::max(p.nf - p.hf, p.nb - p.hb);
    return kLaunch + 0.9e-6 * std::max(p.hf, p.hb) + 4e-6 * wide + kState * p.states;
}
double expansion_states(double seconds) { return (seconds - kLaunch) / kState; }

int run(const Plan& p, const spb_options* opt, spb_result* out, DeviceContext* own_ctx, bool* launched)
{
    *launched = false;
    const double t0 = wall_seconds();
    int st = SPB_OK;
    DeviceContext* ctx = own_ctx ? own_ctx : get_context(opt->device, &st);
    if (!ctx) return out->status = st;
    std::lock_guard<std::mutex> lk(ctx->mu);
    SPB_CUDA_TRY(cudaSetDevice(ctx->device));
    cudaStream_t stream = call_stream(ctx, opt);

    // one CTA per SM, fewer when the widest pair of steps does not fill them;
    // at least one per half
    double most = std::ldexp(1.0, p.kcut);
    for (int k = 0; k < std::max(p.nf - p.hf, p.nb - p.hb); ++k) {
        double c = 0.0;
        if (p.hf + k < p.nf) c += std::ldexp(1.0, p.step[p.hf + k].ka);
        if (p.hb + k < p.nb) c += std::ldexp(1.0, p.step[p.nf + p.hb + k].ka);
        most = std::max(most, c);
    }
    int blocks = (int)std::min((double)ctx->sm_count, std::ceil(most / kThreads));
    if (blocks < 2) blocks = 2;
    // One cluster while a step's states give its threads two each at most,
    // above that the whole GPU (n=24 with 3 more per row: 53 us on a cooperative
    // grid of as many CTAs, 33 us as a cluster; n=30 with 2: 39 and 20 us).
    const bool coop = most > 2.0 * kMaxCluster * kThreads;
    if (!coop) {
        int c = 2;
        while (c < blocks && c < kMaxCluster) c *= 2;
        blocks = c;
    }
    static std::mutex mu;
    static signed char fits[64];  // per device: 1 a CTA per SM stays resident, -1 not
    {
        std::lock_guard<std::mutex> lk2(mu);
        signed char& f = fits[ctx->device & 63];
        if (f == 0) {
            int can = 0, per_sm = 0;
            SPB_CUDA_TRY(cudaFuncSetAttribute(expand_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
            SPB_CUDA_TRY(cudaFuncSetAttribute(expand_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
            SPB_CUDA_TRY(cudaDeviceGetAttribute(&can, cudaDevAttrCooperativeLaunch, ctx->device));
            SPB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, expand_rows<true>, kThreads, kSmem));
            f = can && per_sm >= 1 && ctx->sm_count >= 2 ? 1 : -1;
        }
        if (f < 0) return SPB_OK;
    }

    size_t off = 0;
    auto take = [&](size_t bytes) { size_t o = off; off = align_up(off + bytes, 256); return o; };
    const size_t o_tick = take(sizeof(unsigned)), o_begin = take(sizeof(unsigned long long));
    const size_t o_part = take(sizeof(dd) * blocks);
    size_t o_t[2][2];
    for (int h = 0; h < 2; ++h)
        for (int q = 0; q < 2; ++q) {
            int w = 0;  // widest table of this parity (parity 1 also holds the start)
            for (int s = q; s < (h ? p.nb : p.nf); s += 2) w = std::max(w, (int)p.step[(h ? p.nf : 0) + s].ka);
            o_t[h][q] = take(sizeof(double2) << w);
        }
    // no room for the tables (up to 256 MiB): a walk needs far less
    if (ensure_scratch(ctx, off) != SPB_OK || ensure_pinned(ctx, sizeof(Outcome)) != SPB_OK) return SPB_OK;
    if (!ctx->pinned_dev) return SPB_OK;
    char* base = static_cast<char*>(ctx->scratch);
    Tables t{};
    for (int h = 0; h < 2; ++h)
        for (int q = 0; q < 2; ++q) t.t[h][q] = reinterpret_cast<double2*>(base + o_t[h][q]);
    t.ticket = reinterpret_cast<unsigned*>(base + o_tick);
    t.partials = reinterpret_cast<dd*>(base + o_part);
    t.begin = reinterpret_cast<unsigned long long*>(base + o_begin);
    t.out = static_cast<Outcome*>(ctx->pinned_dev);

    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    if (coop) {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    } else {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = (unsigned)blocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    }
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // (refused launches, a grid that cannot be resident beside what else runs,
    // leave no kernel behind)
    if (cudaLaunchKernelEx(&cfg, coop ? expand_rows<true> : expand_rows<false>, p, t) != cudaSuccess) {
        cudaGetLastError();
        return SPB_OK;
    }
    SPB_CUDA_TRY(cudaStreamSynchronize(stream));
    *launched = true;
    const Outcome o = *static_cast<const Outcome*>(ctx->pinned);
    const dd res = o.total;
    out->value = std::ldexp(res.hi, p.exp_sum);
    out->value_lo = std::ldexp(res.lo, p.exp_sum);
    // every state carries a few roundings of 2^-104 per row, and no partial
    // sum exceeds the product of the rows' absolute sums; a sum that cancels
    // to zero has no relative error
    out->err_est = res.hi != 0.0 ? 4.0 * p.n * 0x1p-104 * p.abs_bound / std::fabs(res.hi) : HUGE_VAL;
    out->kernel_s = out->device_s = opt->skip_timing ? 0.0 : 1e-9 * (double)(o.end - o.begin);
    out->gray_steps = (uint64_t)p.n << (p.n - 1);
    out->launches = 1;
    out->active_rows = p.width;
    out->elapsed_s = wall_seconds() - t0;
    return out->status = SPB_OK;
}

}  // namespace frontier
}  // namespace spb
