// What the persistent FP64 PCG kernels share (rg_pcg64.cuh for scalar matrices, rg_system.cu for block
// ones): a CTA's copy of the iteration's scalars, paso's scalar steps (PCG.cpp:185-347), and division of
// node numbers by the grid's sizes.
#pragma once
#include <cstdint>

namespace rg {

// iteration status, as in the solvers' device scalars
enum { PCG_RUN = 0, PCG_CONV = 1, PCG_MAXIT = 3, PCG_BREAK = 4, PCG_TIMEOUT = 6 };

// Iterations of one launch of a persistent kernel that takes `iter_s` seconds for each: about 2 ms.  A launch holds
// every SM, so this is how long other streams of the program wait for their turn; at 20 ms a
// solve took 1 % less.
inline int launch_iters(double iter_s)
{
    const double k = 0.002 / iter_s;
    return k < 4.0 ? 4 : (k > 8192.0 ? 8192 : (int)k);
}

struct Pcg64State {  // (all CTAs compute the same values)
    double alpha, beta, g1, g2, tau, tau_next, rho, delta, norm, norm2;
    long long iter;
    int status, stop;
};

// After the product: t = {p.v, |rs|^2}.  With `pend` the iteration before is complete: its stopping tests;
// then alpha = tau / delta, breakdown on delta == 0.
__device__ __forceinline__ void paso_after_a(Pcg64State& sc, const double* t, bool pend, double tol, long long maxit)
{
    // (the square root and the division, some 500 cycles each, overlap)
    const double norm = sqrt(t[1]), tau = pend ? sc.tau_next : sc.tau, alpha = tau / t[0];
    if (pend) {
        sc.iter += 1;
        sc.norm = norm;
        if (sc.iter > maxit)
            sc.status = PCG_MAXIT;
        else if (fabs(sc.tau) <= 0.0)
            sc.status = PCG_BREAK;
        else if (sc.norm <= tol)
            sc.status = PCG_CONV;
        sc.tau = tau;
        if (sc.status != PCG_RUN) {
            sc.stop = 1;
            return;
        }
    }
    sc.delta = t[0];
    sc.alpha = alpha;
    if (fabs(t[0]) <= 0.0) {  // breakFlag
        sc.iter += 1;
        sc.status = PCG_BREAK;
        sc.stop = 1;
    }
}

// After the update: w = {z.r, d.d, d.rs} with d = r - rs: the smoothing weights and the next beta.
__device__ __forceinline__ void paso_after_b(Pcg64State& sc, const double* w)
{
    const double g = -w[2] / w[1], beta = w[0] / sc.tau;
    sc.g1 = fabs(w[1]) <= 0.0 ? 0.0 : g;
    sc.g2 = 1.0 - sc.g1;
    sc.tau_next = w[0];
    sc.beta = beta;
}

// k_pcg64's split of the two: the smoothing's |rs|^2 comes with phase B's sums, w = {z.r, d.d, d.rs, |rs|^2}.
// After the product: alpha = tau / delta; a breakdown waits for the tests of the iteration before.
__device__ __forceinline__ void paso_alpha(Pcg64State& sc, double delta, bool pend)
{
    sc.delta = delta;
    sc.alpha = (pend ? sc.tau_next : sc.tau) / delta;
    if (!pend && fabs(delta) <= 0.0) {
        sc.iter += 1;
        sc.status = PCG_BREAK;
        sc.stop = 1;
    }
}

// Called by thread 0.  (norm2: the square root, some 500 cycles, is taken only near the tolerance and at the end)
__device__ __forceinline__ void paso_next(Pcg64State& sc, const double* w, bool pend, double tol, long long maxit)
{
    const double tau = pend ? sc.tau_next : sc.tau;
    const double g = -w[2] / w[1], beta = w[0] / tau;
    if (pend) {
        sc.iter += 1;
        sc.norm2 = w[3];
        if (sc.iter > maxit)
            sc.status = PCG_MAXIT;
        else if (fabs(sc.tau) <= 0.0)
            sc.status = PCG_BREAK;
        else if (!(w[3] > 1.0000001 * (tol * tol)) && sqrt(w[3]) <= tol)
            sc.status = PCG_CONV;
        sc.tau = tau;
        if (sc.status == PCG_RUN && fabs(sc.delta) <= 0.0) {
            sc.iter += 1;
            sc.status = PCG_BREAK;
        }
        if (sc.status != PCG_RUN) {
            sc.stop = 1;
            return;
        }
    }
    sc.g1 = fabs(w[1]) <= 0.0 ? 0.0 : g;
    sc.g2 = 1.0 - sc.g1;
    sc.tau_next = w[0];
    sc.beta = beta;
}

// v / d = (v m) >> (31 + s) for v < 2^31
inline void fast_div(unsigned d, unsigned* m, int* s)
{
    int k = 0;
    while ((1ull << k) < d) ++k;
    *s = k;
    *m = (unsigned)((1ull << (31 + k)) / d + 1);
}

__device__ __forceinline__ unsigned fdiv(unsigned v, unsigned m, int s)
{
    return (unsigned)(((unsigned long long)v * m) >> (31 + s));
}

}  // namespace rg
