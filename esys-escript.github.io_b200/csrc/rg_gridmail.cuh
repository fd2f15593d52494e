// Grid-wide sums inside a persistent kernel: every CTA posts its partial sums, counts itself in,
// waits until all CTAs of the exchange are in, reads all partial sums and adds them in the same
// fixed order.  All CTAs hold identical totals, and the exchange is the kernel's grid barrier.
//
// SYNC = true orders memory too: what any CTA wrote before the exchange is visible to every CTA
// after it (block barrier and release before the count, acquire and block barrier after the
// wait).  SYNC = false only exchanges the sums, for a phase whose inputs the same thread wrote
// itself: each double then travels as two 8-byte words, half of its bits beside the number of the
// exchange, so a word that was read with the number needs no fence; the count only tells when
// reading is worth while.  Measured on 148 CTAs (cycles): 3,700 with SYNC, 3,000 without; every
// CTA polling all CTAs' words instead of one counter 9,600 (the polls crowd out the posts), the
// last CTA to arrive publishing the totals 7,300, __threadfence() after the wait instead of
// ld.acquire polls 700 more.
//
// Two sets of slots alternate: a CTA posts exchange g + 2 into the slots of g only after exchange
// g + 1, for which every CTA had to finish reading g.  The mail is zeroed before each launch and
// exchanges count from 1.  Waits are bounded: a CTA that gave up, or that sees the abort bit of
// the counter, returns false and posts no more.
#pragma once
#include "rg_internal.cuh"

namespace rg {

constexpr int kMailCtas = 160;      // CTAs whose posts a warp reads at a time (5 per lane)
constexpr int kMailGrid = 2 * kMailCtas;  // most CTAs of a grid that exchanges with SYNC; else kMailCtas
constexpr int kMailVals = 8;        // most doubles of an exchange
constexpr size_t kMailSet = (size_t)2 * kMailVals * kMailCtas;  // 8-byte words of one set (kMailVals x kMailGrid with SYNC)
constexpr size_t kMailBytes = 8 * (2 * kMailSet + 16);
constexpr unsigned kMailAbort = 0x80000000u;

__device__ __forceinline__ void mail_store(unsigned long long* p, unsigned long long a)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}

__device__ __forceinline__ unsigned long long mail_load(const unsigned long long* p)
{
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return a;
}

template <bool ACQ>
__device__ __forceinline__ unsigned mail_count(const unsigned* p)
{
    unsigned a;
    if (ACQ)
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(p) : "memory");
    else
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(p) : "memory");
    return a;
}

// Sums P = 2^k values over a warp, each lane keeping half of its values at every step while there
// is more than one: lane l returns the total of value l / (32 / P).  For P = 4 that is 2 + 1 + 1 + 1
// + 1 shuffles instead of 5 per value.
template <int P>
__device__ __forceinline__ double warp_sum_split(double (&v)[P], int lane)
{
    int o = 16;
#pragma unroll
    for (int h = P / 2; h >= 1; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double send = up ? v[j] : v[j + h];
            v[j] = (up ? v[j + h] : v[j]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Adds v over the grid.  Called by all threads of a block of W warps; the totals are valid in
// every lane of warp 0 (other warps go on to the caller's __syncthreads at once).  *bad (shared)
// set by any thread of the block before the call makes the whole grid return false.
template <int NV, int W, bool SYNC>
__device__ __forceinline__ bool mail_sum(const double (&v)[NV], double (&tot)[NV], unsigned long long* mail,
                                         unsigned gen, const int* bad, int polls, bool withhold)
{
    constexpr int P = NV <= 1 ? 1 : (NV <= 2 ? 2 : (NV <= 4 ? 4 : 8));
    constexpr int L = 32 / P;           // lanes per value
    static_assert(NV <= kMailVals && W <= 32 && L >= 2, "mail slots");
    __shared__ double sh[P][W];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int val = lane / L, sub = lane % L;
    double a[P];
#pragma unroll
    for (int j = 0; j < P; ++j) a[j] = j < NV ? v[j] : 0.0;
    const double s1 = warp_sum_split<P>(a, lane);
    if (sub == 0) sh[val][warp] = s1;
    __syncthreads();
    if (warp != 0) return true;
    double s2 = 0.0;
#pragma unroll
    for (int w = 0; w < (W + L - 1) / L; ++w)
        if (sub + w * L < W) s2 += sh[val][sub + w * L];
#pragma unroll
    for (int o = L / 2; o >= 1; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    unsigned long long* set = mail + (size_t)(gen & 1u) * kMailSet;
    unsigned* counter = reinterpret_cast<unsigned*>(mail + 2 * kMailSet);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(s2);
    const unsigned long long tag = (unsigned long long)gen << 32;
    const int G = (int)gridDim.x;
    if (SYNC) {
        if (sub == 0 && val < NV) mail_store(set + val * kMailGrid + blockIdx.x, bits);
    } else if (sub < 2 && val < NV) {
        mail_store(set + (2 * val + sub) * kMailCtas + blockIdx.x, tag | (sub ? bits >> 32 : bits & 0xffffffffull));
    }
    __syncwarp();
    if (lane == 0 && !withhold) {  // (withheld by the test of the timeout path only)
        if (*bad) asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(counter), "r"(kMailAbort) : "memory");
        if (SYNC)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        else
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    }
    const unsigned target = gen * (unsigned)G;
    bool ok = true;
    int tries = 0;
    for (;; ++tries) {
        const unsigned c = mail_count<SYNC>(counter);
        if (c & kMailAbort || tries >= polls) {
            ok = false;
            break;
        }
        if (c >= target) break;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) return false;
    constexpr int K = kMailCtas / 32;
    double part[P];
#pragma unroll
    for (int j = 0; j < P; ++j) part[j] = 0.0;
    if (SYNC) {
        for (int first = 0; first < G; first += kMailCtas) {
            unsigned long long w[K][NV];
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    w[k][j] = first + lane + 32 * k < G ? mail_load(set + j * kMailGrid + first + lane + 32 * k) : 0ull;
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int k = 0; k < K; ++k) part[j] += __longlong_as_double((long long)w[k][j]);
        }
    } else {
        for (;; ++tries) {
            unsigned long long w[K][2 * NV];
            bool have = true;
#pragma unroll
            for (int k = 0; k < K; ++k)
#pragma unroll
                for (int j = 0; j < 2 * NV; ++j)
                    w[k][j] = lane + 32 * k < G ? mail_load(set + j * kMailCtas + lane + 32 * k) : tag;
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                part[j] = 0.0;
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    have = have && (unsigned)(w[k][2 * j] >> 32) == gen && (unsigned)(w[k][2 * j + 1] >> 32) == gen;
                    part[j] += __longlong_as_double((long long)((w[k][2 * j] & 0xffffffffull) | (w[k][2 * j + 1] << 32)));
                }
            }
            if (__all_sync(0xffffffffu, have)) break;
            if (tries >= polls) return false;
        }
    }
    const double s3 = warp_sum_split<P>(part, lane);
#pragma unroll
    for (int j = 0; j < NV; ++j) tot[j] = __shfl_sync(0xffffffffu, s3, j * L);
    return true;
}

}  // namespace rg
