// FP64 PCG (paso's with residual smoothing, or textbook) as one persistent kernel over many
// iterations.  Included by rg_solver.cu inside namespace rg, after the solver's scalars.
//
// An iteration is two phases, each ended by one grid-wide sum (rg_gridmail.cuh):
//   A  (paso: of the iteration before, x2 += alpha p, rs and x smoothing, sum rs^2)  p = z + beta p,
//      v = A p, sum p.v -> alpha; textbook: x += alpha p of the iteration before
//   B  r -= alpha v, z = D^-1 r, sums -> beta (paso: gamma_1/2)
// (x2, and the textbook x, wait for the next phase A because the old p is read there anyway; the textbook
// x takes its last step when the launch ends.)
// p is double-buffered: in phase A every row forms the new p of its neighbours from their z and
// old p, so that no third phase (or pass over memory) is needed for the direction.
//
// The matrix is paso's CSR array itself.  On a ripley grid the columns of a row follow from its
// node (27 or 9 neighbours in id order, the missing ones left out), so idx is never read: 8
// bytes per entry instead of 12, without a band copy.  A warp owns tiles of 32 consecutive rows,
// whose entries are one contiguous run of val, bulk-copied (16-byte aligned, rounded outwards)
// into the warp's own ring of S stages; a lane then reads its row's entries from shared memory
// (rows start 27 or 9 doubles apart: odd, so no bank conflicts).  A warp whose tiles all fit
// its ring copies them once per launch.
//
// What bounds it: HBM at large sizes (216 B of matrix and about 15 vector accesses of 8 B per
// row and iteration), the two exchanges at small ones.  Measured per iteration against one
// kernel per step replayed from CUDA graphs: Brick 128^3 paso 130 against 215 us, Rectangle
// 200 x 200 paso 5.9 against 20 us, 403 x 297 textbook 6.4 against 15 us.
#pragma once

struct Pcg64Args {
    int n, nn0, nn1, nn2;
    int off[27];                  // column offset of band b
    unsigned m0, m1;              // row / d = (row * m) >> (31 + s) for d = nn0, nn0 nn1 (rows < 2^31)
    int s0, s1;
    const int32_t* ptr;
    const double* val;
    double *r, *q, *rs, *x, *x2, *z, *p0, *p1;
    const double* dinv;
    int ntiles, wpc;              // 32-row tiles; active warps per CTA
    int max_iters;                // iterations of this launch
    unsigned long long* mail;
};

template <int NB, int W, int S>
constexpr size_t pcg64_smem()
{
    return (size_t)W * S * (32 * NB * 8 + 16);
}

template <int NB, int W, int S, bool PASO>
__global__ void __launch_bounds__(W * 32, 1) k_pcg64(const __grid_constant__ Pcg64Args a, Scal* s)
{
    constexpr int kStageBytes = 32 * NB * 8 + 16;
    extern __shared__ __align__(128) unsigned char smem_pcg[];
    __shared__ __align__(8) uint64_t full[W][S];
    __shared__ Pcg64State sc;
    __shared__ int bad;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int G = (int)gridDim.x;
    const WaitCtl wc = g_wait_ctl;
    const int polls = wc.polls > 0 ? wc.polls : kDefaultPolls;
    if (s->done) return;
    if (threadIdx.x == 0) {
        bad = 0;
        sc.alpha = s->alpha;
        sc.beta = s->pend ? s->beta : 0.0;
        sc.g1 = s->gamma1;
        sc.g2 = s->gamma2;
        sc.tau = s->tau;
        sc.tau_next = s->tau_next;
        sc.rho = s->rho;
        sc.norm = s->norm;
        sc.iter = s->iter;
        sc.status = PCG_RUN;
        sc.stop = 0;
    }
    if (threadIdx.x < W * S) mbar_init(&full[threadIdx.x / S][threadIdx.x % S], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    const double tol = s->tol;
    const long long maxit = s->maxit;
    bool pend = s->pend != 0;
    int par = s->par;

    // this warp's tiles: chunk k of the grid is G * wpc consecutive tiles, wpc of them per CTA
    const int t0 = blockIdx.x * a.wpc + warp, tstep = G * a.wpc;
    const int mine = warp < a.wpc && t0 < a.ntiles ? (a.ntiles - 1 - t0) / tstep + 1 : 0;
    const bool resident = mine <= S;
    unsigned char* ring = smem_pcg + (size_t)warp * S * kStageBytes;
    int issued = 0, used = 0;     // tiles copied into / taken from the ring
    int nk = 0;                   // the warp's tile the next copy is for, and its entries' range
    int e0 = 0, e1 = 0;
    auto range = [&](int k) {
        const int row0 = (t0 + k * tstep) * 32;
        e0 = __ldg(a.ptr + row0);
        e1 = __ldg(a.ptr + min(row0 + 32, a.n));
    };
    auto issue = [&]() {          // lane 0: copy the next tile's entries into its stage
        const int st = issued % S;
        const int from = e0 & ~1, to = (e1 + 1) & ~1;
        mbar_expect_tx(&full[warp][st], (uint32_t)(to - from) * 8u);
        if (resident)
            bulk_g2s(ring + st * kStageBytes, a.val + from, (uint32_t)(to - from) * 8u, &full[warp][st]);
        else
            bulk_g2s_hint(ring + st * kStageBytes, a.val + from, (uint32_t)(to - from) * 8u, &full[warp][st],
                          evict_first_policy());
        ++issued;
        nk = nk + 1 == mine ? 0 : nk + 1;
        range(nk);
    };
    if (lane == 0 && mine > 0) {
        range(0);
        if (!wc.withhold)
            for (int k = 0; k < (resident ? mine : S); ++k) issue();
    }

    bool xpend = false;           // textbook: whether x has yet to take alpha p
    unsigned gen = 0;
    for (int left = a.max_iters; left > 0; --left) {
        // ---------------------------------------------------------------- phase A
        const double before = sc.alpha, beta = sc.beta, g1 = sc.g1, g2 = sc.g2;
        const double* pold = par ? a.p1 : a.p0;
        double* pnew = par ? a.p0 : a.p1;
        double v[2] = {0.0, 0.0};
        for (int k = 0; k < mine; ++k) {
            const int row0 = (t0 + k * tstep) * 32;
            const int row = row0 + lane;
            const bool in = row < a.n;
            double rs = 0.0, rr = 0.0, xx = 0.0, xx2 = 0.0;
            if (PASO && pend && in) {
                rs = a.rs[row];
                rr = a.r[row];
                xx = a.x[row];
                xx2 = a.x2[row];
            }
            if (!PASO && xpend && in) xx = a.x[row];
            const int kb = __ldg(a.ptr + (in ? row : row0));
            const int base = __shfl_sync(0xffffffffu, kb, 0);
            const unsigned plane = a.nn0 * a.nn1;
            const unsigned cz = NB == 27 ? fdiv(row, a.m1, a.s1) : 0u;
            const unsigned in_plane = row - cz * plane;
            const unsigned cy = fdiv(in_plane, a.m0, a.s0);
            const unsigned cx = in_plane - cy * a.nn0;
            const bool inner = in && cx > 0 && cx < (unsigned)a.nn0 - 1 && cy > 0 && cy < (unsigned)a.nn1 - 1 &&
                               (NB == 9 || (cz > 0 && cz < (unsigned)a.nn2 - 1));
            const int st = resident ? k : used % S;
            const uint32_t ph = resident ? 0u : (uint32_t)((used / S) & 1);
            const double* row_val =
                reinterpret_cast<const double*>(ring + st * kStageBytes) + (base & 1) + (kb - base);
            double acc = 0.0, pc = 0.0, po = 0.0;
            bool waited = false;
            if (__all_sync(0xffffffffu, inner)) {
#pragma unroll
                for (int g = 0; g < NB / 3; g += 3) {
                    double zz[9], pp[9];
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        zz[m] = a.z[row + a.off[3 * g + m]];
                        pp[m] = pold[row + a.off[3 * g + m]];
                    }
                    if (g == 0) waited = mbar_wait(&full[warp][st], ph, polls);
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const double pn = fma(beta, pp[m], zz[m]);
                        acc = fma(row_val[3 * g + m], pn, acc);
                        if (3 * g + m == NB / 2) {
                            pc = pn;
                            po = pp[m];
                        }
                    }
                }
            } else {
                // a tile with boundary rows (half of them at lines of 129 nodes): the same nine loads at a time,
                // a missing neighbour's from the row itself; its entry is left out.  ok9: which of the 3 x 3
                // neighbours (x, y) of a plane exist.  Loaded three at a time after the wait, solves took: 95 x
                // 97 x 96 paso 37.0 ms (now 32.3), textbook 41.8 (30.7); 128^3 100.7 (96.8) and 98.7 (94.5).
                const int rowc = in ? row : row0;
                const unsigned x3 = !in ? 0u : (cx > 0 ? 1u : 0u) | 2u | (cx + 1 < (unsigned)a.nn0 ? 4u : 0u);
                const unsigned ok9 = (cy > 0 ? x3 : 0u) | x3 << 3 | (cy + 1 < (unsigned)a.nn1 ? x3 << 6 : 0u);
                int e = 0;
#pragma unroll
                for (int g = 0; g < NB / 3; g += 3) {
                    const bool zv = NB == 9 || (g == 0 ? cz > 0 : (g == 6 ? cz + 1 < (unsigned)a.nn2 : true));
                    const unsigned okg = zv ? ok9 : 0u;
                    double zz[9], pp[9];
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const int j = okg >> m & 1u ? row + a.off[3 * g + m] : rowc;
                        zz[m] = a.z[j];
                        pp[m] = pold[j];
                    }
                    if (g == 0) waited = mbar_wait(&full[warp][st], ph, polls);
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const double pn = fma(beta, pp[m], zz[m]);
                        const bool ok = okg >> m & 1u;
                        if (ok) acc = fma(row_val[e], pn, acc);
                        e += ok ? 1 : 0;
                        if (3 * g + m == NB / 2) {
                            pc = pn;
                            po = pp[m];
                        }
                    }
                }
            }
            if (!__all_sync(0xffffffffu, waited)) {
                bad = 1;
                break;
            }
            if (!resident) {
                ++used;
                if (lane == 0) issue();
            }
            if (in) {
                pnew[row] = pc;
                a.q[row] = acc;
                v[0] += acc * pc;
                if (!PASO && xpend) a.x[row] = xx + before * po;
                if (PASO && pend) {
                    const double rn = g2 * rs + g1 * rr;
                    a.rs[row] = rn;
                    const double xn = xx2 + before * po;
                    a.x2[row] = xn;
                    a.x[row] = g2 * xx + g1 * xn;
                    v[1] += rn * rn;
                }
            }
        }
        // phase B walks the tiles backwards (the rows phase A touched last are the likeliest in L2),
        // two per step; a thread's rows are those it had in phase A, so all it reads but alpha is its
        // own work: the first pair is loaded before the exchange, whose wait covers the loads
        double fr[2], fq[2], frs[2], fd[2];
        int frow[2];
        auto fetch = [&](int k) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                frow[h] = (t0 + (k - h) * tstep) * 32 + lane;
                if (k - h < 0 || frow[h] >= a.n) frow[h] = -1;
                if (frow[h] >= 0) {
                    fr[h] = a.r[frow[h]];
                    fq[h] = a.q[frow[h]];
                    fd[h] = __ldg(a.dinv + frow[h]);
                    if (PASO) frs[h] = a.rs[frow[h]];
                }
            }
        };
        fetch(mine - 1);
        double t[2];
        ++gen;
        bool ok = mail_sum<2, W, false>(v, t, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                sc.status = PCG_TIMEOUT;
                sc.stop = 1;
            } else {
                if (PASO) {
                    paso_after_a(sc, t, pend, tol, maxit);
                } else {
                    sc.delta = t[0];
                    sc.alpha = sc.rho / t[0];
                    if (!(fabs(t[0]) > 0.0)) {
                        sc.iter += 1;
                        sc.status = PCG_BREAK;
                        sc.stop = 1;
                    }
                }
            }
        }
        __syncthreads();
        par ^= 1;
        xpend = false;
        if (sc.stop) break;

        // ---------------------------------------------------------------- phase B
        const double alpha = sc.alpha;
        double u[3] = {0.0, 0.0, 0.0};
        for (int k = mine - 1; k >= 0; k -= 2) {
            if (k < mine - 1) fetch(k);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (frow[h] >= 0) {
                    const double rn = fr[h] - alpha * fq[h];
                    a.r[frow[h]] = rn;
                    const double zn = rn * fd[h];
                    a.z[frow[h]] = zn;
                    u[0] += zn * rn;
                    if (PASO) {
                        const double d = rn - frs[h];
                        u[1] += d * d;
                        u[2] += d * frs[h];
                    } else {
                        u[1] += rn * rn;
                    }
                }
        }
        double w[3];
        ++gen;
        ok = mail_sum<3, W, true>(u, w, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                sc.status = PCG_TIMEOUT;
                sc.stop = 1;
            } else if (PASO) {
                paso_after_b(sc, w);
                if (left == 1) sc.stop = 1;
            } else {
                sc.iter += 1;
                sc.norm = sqrt(w[1]);
                sc.beta = w[0] / sc.rho;
                sc.rho = w[0];
                if (sc.norm <= tol)
                    sc.status = PCG_CONV;
                else if (sc.iter >= maxit)
                    sc.status = PCG_MAXIT;
                else if (!(fabs(w[0]) > 0.0))
                    sc.status = PCG_BREAK;
                if (sc.status != PCG_RUN || left == 1) sc.stop = 1;
            }
        }
        __syncthreads();
        pend = true;
        xpend = !PASO;
        if (sc.stop) break;
    }
    if (!PASO && xpend) {
        const double alpha = sc.alpha;
        const double* p = par ? a.p1 : a.p0;
        for (int k = 0; k < mine; ++k) {
            const int row = (t0 + k * tstep) * 32 + lane;
            if (row < a.n) a.x[row] = a.x[row] + alpha * p[row];
        }
    }
    // copies still in flight land (bounded) before the ring is given up
    if (lane == 0) {
        const int first = resident ? 0 : used;
        for (int k = first; k < issued; ++k)
            mbar_wait(&full[warp][k % S], (uint32_t)((k / S) & 1));
    }
    if (threadIdx.x == 0) {
        if (sc.status == PCG_TIMEOUT) {
            report_status(s, PCG_TIMEOUT);
        } else if (blockIdx.x == 0) {
            s->alpha = sc.alpha;
            s->beta = sc.beta;
            s->gamma1 = sc.g1;
            s->gamma2 = sc.g2;
            s->tau = sc.tau;
            s->tau_next = sc.tau_next;
            s->rho = sc.rho;
            s->delta = sc.delta;
            s->norm = sc.norm;
            s->iter = sc.iter;
            s->par = par;
            s->pend = pend ? 1 : 0;
            if (sc.status != PCG_RUN) report_status(s, sc.status);
        }
    }
}
