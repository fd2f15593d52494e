// Grid-wide sums of a persistent kernel in the order of one kernel per step, bit for bit.
//
// A conjugate gradient iteration carries the rounding of its sums on to every later one: on long, badly
// conditioned grids (a Robin problem on 22 x 28 x 114 cells) two orders of addition end 6e-10 apart, or an
// iteration apart, which is more than a program that keeps its results may see change.  The order is therefore
// fixed by the system's size alone, as grid_reduce (rg_internal.cuh) has it in kernels of 256 threads:
//   a virtual thread adds its terms in turn, a warp by butterfly, a virtual block its 8 warps in turn, and
//   the last step adds blocks t, t + 256, ... per thread, then again warps by butterfly, and these in turn.
// Which CTA computes a virtual block is free.  Its sum is posted, every CTA counts itself in, waits for all,
// and adds all posts; all CTAs hold the same totals, and the exchange is the kernel's grid barrier: what any CTA
// wrote before it is visible to every CTA after it.
//
// Two sets of posts alternate: a CTA posts exchange g + 2 into the slots of g only after exchange g + 1, for
// which every CTA had to finish reading g.  The counter is zeroed before each launch, exchanges count from
// 1.  Waits are bounded: a CTA that gave up, or that sees the abort bit, returns false and posts no more.
//
// What bounds an exchange: the count's round trip, then the posts' (each CTA reads all of them, so their
// lines are hot: one post per virtual warp instead of per block took 2,600 instead of 900 cycles to read), and the
// chains of dependent FP64 additions (about 35 cycles each) that the order asks for.
#pragma once
#include "rg_gridmail.cuh"

namespace rg {

constexpr int kVirtualBlocks = kNumSMs * 8;  // grid_for's cap
constexpr int kOrderSlots = 1280;            // posts of a value
constexpr int kOrderVals = 4;                // most values of an exchange
constexpr size_t kOrderSet = (size_t)kOrderVals * kOrderSlots;
constexpr size_t kOrderBytes = 8 * (2 * kOrderSet + 16);
constexpr int kOrderRound = 16;              // virtual blocks that a CTA keeps the warps' sums of
static_assert(kVirtualBlocks <= kOrderSlots && kMailCtas <= kOrderSlots, "a post per virtual block");

// Sums over the nodes' pairs (2k, 2k + 1) as kernels over double2 form them: virtual thread g of `blocks` x 256
// takes pairs g, g + stride, ...; thread 0 also the last node of an odd count.  A CTA computes `per` virtual
// blocks, every grid's size from its own.
struct PairPlan {
    int blocks, stride, per;
};

inline PairPlan pair_plan(int64_t n, int grid)
{
    PairPlan p{};
    p.blocks = grid_for((n + 3) / 4, 256, 8);
    p.stride = p.blocks * 256;
    p.per = (p.blocks + grid - 1) / grid;
    return p;
}

// the warps' sums of a CTA's virtual blocks: of pairs, and of its one block of rows
struct OrderShared {
    double pairs[kOrderVals][kOrderRound][8], rows[8];
};

// A warp's sums of NV values by butterfly (warp_sum_split adds the same pairs): value j's in the lane where
// order_lane(lane) is j
template <int NV>
constexpr int order_lanes() { return NV <= 1 ? 32 : (NV <= 2 ? 16 : 8); }
template <int NV>
__device__ __forceinline__ int order_lane(int lane)
{
    constexpr int L = order_lanes<NV>();
    return lane % L == 0 && lane / L < NV ? lane / L : -1;
}
template <int NV>
__device__ __forceinline__ double order_warp_sum(const double (&v)[NV], int lane)
{
    constexpr int P = 32 / order_lanes<NV>();
    double a[P];
#pragma unroll
    for (int j = 0; j < P; ++j) a[j] = j < NV ? v[j] : 0.0;
    return warp_sum_split<P>(a, lane);
}

// v += a0 b0 + a1 b1, in the order kernels over double2 round it
__device__ __forceinline__ double add_pair(double v, double a0, double b0, double a1, double b1)
{
    return __dadd_rn(v, __fma_rn(a0, b0, __dmul_rn(a1, b1)));
}

// 8 warps' sums in turn
__device__ __forceinline__ double add_warps(const double* w)
{
    double t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = w[i];
    double s = t[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) s += t[i];
    return s;
}

__device__ __forceinline__ void order_post(unsigned long long* slot, double v)
{
    mail_store(slot, (unsigned long long)__double_as_longlong(v));
}

// Goes over the CTA's share of the pairs: load(k) returns what a pair needs, finish(k, loaded) adds to it what
// had to wait for the exchange before, use(k, loaded, v) adds its terms to v, last(i, v) those of the last node of
// an odd count.  The warps' sums go to `sh`, for ordered_sum to post to `set`.  Called by all
// threads of a block of W warps, the upper eight of which come first.  `pre`: what pair_ahead loaded.
template <class T>
struct PairAhead {
    T t[2];
};

template <int W>
__device__ __forceinline__ int pair_group() { return W / 8 - 1 - (int)(threadIdx.x >> 8); }

// the first two pairs' loads of a thread, ahead of pair_sums
template <int W, class T, class Load>
__device__ __forceinline__ void pair_ahead(const PairPlan& pp, int n, PairAhead<T>& pre, Load load)
{
    const int i = pair_group<W>(), vb = blockIdx.x + gridDim.x * i;
    if (i >= pp.per || vb >= pp.blocks) return;
    const int g = vb * 256 + (threadIdx.x & 255);
    if (g < n >> 1) pre.t[0] = load(g);
    if (g + pp.stride < n >> 1) pre.t[1] = load(g + pp.stride);
}

// posts the sums over pairs in `os`, of the CTA's virtual blocks base, base + 1, ... (by one warp)
__device__ __forceinline__ void post_pairs(const PairPlan& pp, const OrderShared& os, int base, int nv,
                                           unsigned long long* set, int lane)
{
    const int count = min(pp.per - base, kOrderRound);
    for (int t = lane; t < nv * count; t += 32) {
        const int j = t / count, i = t - j * count, vb = blockIdx.x + gridDim.x * (base + i);
        if (vb < pp.blocks) order_post(set + j * kOrderSlots + vb, add_warps(os.pairs[j][i]));
    }
}

// the first of the CTA's virtual blocks whose sums ordered_sum posts (0 on 74 SMs or more)
__device__ __forceinline__ int last_round(const PairPlan& pp) { return (pp.per - 1) / kOrderRound * kOrderRound; }

template <int NV, int W, class T, class Load, class Finish, class Use, class Last>
__device__ __forceinline__ void pair_sums(const PairPlan& pp, int n, OrderShared& sh, unsigned long long* set,
                                          const PairAhead<T>* pre, Load load, Finish finish, Use use, Last last)
{
    constexpr int kStep = W / 8;
    static_assert(W % 8 == 0 && NV <= kOrderVals && kOrderRound % (W / 8) == 0, "whole virtual blocks");
    const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) & 7;
    const int nv = n >> 1, val = order_lane<NV>(lane);
    bool loaded = pre != nullptr;
    auto load2 = [&](int k, T& a, T& b) {
        a = load(k);
        b = load(k + pp.stride < nv ? k + pp.stride : k);
    };
    for (int i = pair_group<W>(), base = 0; i < pp.per; i += kStep) {
        const int vb = blockIdx.x + gridDim.x * i;
        if (i - base >= kOrderRound) {  // (few SMs: more blocks than there is room for)
            __syncthreads();
            if (threadIdx.x < 32) post_pairs(pp, sh, base, NV, set, lane);
            __syncthreads();
            base += kOrderRound;
        }
        if (vb >= pp.blocks) continue;
        double v[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = 0.0;
        const int g = vb * 256 + (threadIdx.x & 255);
        for (int k = g; k < nv; k += 2 * pp.stride) {
            T a, b;
            if (loaded) {
                a = pre->t[0];
                b = pre->t[1];
            } else {
                load2(k, a, b);
            }
            finish(k, a);
            finish(k + pp.stride < nv ? k + pp.stride : k, b);
            loaded = false;
            use(k, a, v);
            if (k + pp.stride < nv) use(k + pp.stride, b, v);
        }
        if ((n & 1) && g == 0) last(n - 1, v);
        const double s = order_warp_sum<NV>(v, lane);
        if (val >= 0) sh.pairs[val][i - base][warp] = s;
    }
}

// The exchange: of the sum over rows, or (ROWS = false) of NP sums over pairs that pair_sums formed.  ROW_BLOCK: the CTA has one virtual block of rows, its warps' sums in sh.rows; else its warps posted their
// blocks.  Called by all threads of a block of at least 8 warps; the totals are valid in warp 0.  *bad (shared) set by any
// thread before the call makes the whole grid return false.
template <bool ROWS, bool ROW_BLOCK, int NP>
__device__ __forceinline__ bool ordered_sum(int rows, const PairPlan& pairs, double (&tot)[ROWS ? 1 : NP],
                                            const OrderShared& os, unsigned long long* set, unsigned long long* mail,
                                            unsigned gen, const int* bad, int polls, bool withhold)
{
    constexpr int NV = ROWS ? 1 : NP;
    static_assert(NV <= kOrderVals, "slots");
    const int blocks = ROWS ? rows : pairs.blocks;
    __shared__ double sh[8][NV];
    __shared__ int arrived;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (warp == 0) {
        if (!ROWS) post_pairs(pairs, os, last_round(pairs), NP, set, lane);
        if (ROWS && ROW_BLOCK && lane == 31) order_post(set + blockIdx.x, add_warps(os.rows));
        __syncwarp();
        unsigned* counter = reinterpret_cast<unsigned*>(mail + 2 * kOrderSet);
        if (lane == 0 && !withhold) {  // (withheld by the test of the timeout path only)
            if (*bad) asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(counter), "r"(kMailAbort) : "memory");
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        }
        const unsigned target = gen * gridDim.x;
        bool ok = true;
        for (int tries = 0;; ++tries) {
            const unsigned c = mail_count<true>(counter);
            if (c & kMailAbort || tries >= polls) {
                ok = false;
                break;
            }
            if (c >= target) break;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) arrived = ok ? 1 : 0;
    }
    __syncthreads();
    if (!arrived) return false;
    const int warps = min(8, (blocks + 31) >> 5);  // of virtual threads with posts
    if (warp < warps) {
        constexpr int K = (kVirtualBlocks + 255) / 256;
        double w[NV][K], a[NV];
#pragma unroll
        for (int j = 0; j < NV; ++j)
#pragma unroll
            for (int i = 0; i < K; ++i) {
                const int b = (int)threadIdx.x + 256 * i;
                w[j][i] = b < blocks
                              ? __longlong_as_double((long long)mail_load(set + j * kOrderSlots + b))
                              : 0.0;
            }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            a[j] = w[j][0];
#pragma unroll
            for (int i = 1; i < K; ++i) a[j] += w[j][i];
        }
        const double s = order_warp_sum<NV>(a, lane);
        const int val = order_lane<NV>(lane);
        if (val >= 0) sh[warp][val] = s;
    }
    __syncthreads();
    if (warp == 0) {
        double s = 0.0;
        if (lane < NV) {
            s = sh[0][lane];
            for (int w = 1; w < warps; ++w) s += sh[w][lane];
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) tot[j] = __shfl_sync(0xffffffffu, s, j);
    }
    return true;
}

}  // namespace rg
