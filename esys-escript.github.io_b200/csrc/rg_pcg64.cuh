// FP64 PCG (paso's with residual smoothing, or textbook) as one persistent kernel over many
// iterations.  Included by rg_solver.cu inside namespace rg, after the solver's scalars.
//
// An iteration is two phases, each ended by one grid-wide sum (rg_ordersum.cuh):
//   A  p = z + beta p, v = A p, sum p.v -> alpha; of the iteration before: x += alpha p (textbook), or x2 +=
//      alpha p, rs and x smoothing (paso)
//   B  r -= alpha v, z = D^-1 r, sums -> beta (paso: gamma_1/2, and rs^2 of the iteration before, whose
//      stopping test therefore comes one phase B late: that phase changes nothing that is returned)
// (x2, and the textbook x, wait for the next phase A because the old p is read there anyway; the textbook
// x takes its last step when the launch ends.)
// p is double-buffered: in phase A every row forms the new p of its neighbours from their z and
// old p, so that no third phase (or pass over memory) is needed for the direction.
//
// All sums, and a row's products, are added in the order that a kernel per step adds them in (rounding that
// iterations amplify up to the solution's own error): a row's product like 8 lanes on the CSR entries (SEQ =
// false) or in band order (SEQ = true, RG_LAYOUT_BAND), p.v over rows by the virtual threads of that
// kernel, the other sums over pairs of rows.
//
// The matrix is paso's CSR array itself.  On a ripley grid the columns of a row follow from its
// node (27 or 9 neighbours in id order, the missing ones left out), so idx is never read: 8
// bytes per entry instead of 12, without a band copy.  Rows go in tiles of 32, one virtual block of the
// row sum (chain) being the tiles t, t + tstep, ...; a CTA owns `cpc` chains, whose tiles its warps w and
// w + 8 take in turn.  A tile's entries are one contiguous run of val, bulk-copied (16-byte aligned, rounded
// outwards) into the warp's own ring of S stages; a lane then reads its row's entries from shared memory
// (rows start 27 or 9 doubles apart: odd, so no bank conflicts).  A warp whose tiles all fit
// its ring copies them once per launch.  Phase B is shared out by pairs of rows instead, so the exchange after
// phase A orders memory as well.
//
// What bounds it: HBM at large sizes (216 B of matrix and about 16 vector accesses of 8 B per row and iteration),
// the two exchanges at small ones (some 4,500 of 7,000 cycles each, with the chains of dependent FP64 additions).
// Measured per iteration against a kernel per step replayed from CUDA graphs: paso on Rectangle 200 x 200 7.4
// against 20.2 us, Brick 21 x 17 x 14 9.0 against 13.2, 95 x 97 x 96 67 against 90, 128^3 158 against 210;
// textbook on 403 x 297 8.4 against 14.9.  (Added in an order of its own, with phase B on the tiles' rows and no
// memory order after phase A: 5.6, 6.3, 47, 134 and 6.5 us.)
#pragma once

struct Pcg64Args {
    int n, nn0, nn1, nn2;
    int off[27];                  // column offset of band b
    int step[4][27];              // of a row's e-th entry from its lowest neighbour, with 3 or 2 neighbours along x (bit
                                  // 0: 2) and y (bit 1: 2)
    unsigned m0, m1;              // row / d = (row * m) >> (31 + s) for d = nn0, nn0 nn1 (rows < 2^31)
    int s0, s1;
    const int32_t* ptr;
    const double* val;
    double *r, *q, *rs, *x, *x2, *z, *p0, *p1;
    const double* dinv;
    int ntiles;                   // 32-row tiles
    int tstep, chains, cpc;       // tiles from one to the next of a chain; chains, and chains per CTA
    int row_blocks;               // virtual blocks of the row sum
    PairPlan pairs;
    int max_iters;                // iterations of this launch
    unsigned long long* mail;
};

template <int NB, int W, int S>
constexpr size_t pcg64_smem()
{
    return (size_t)W * S * (32 * NB * 8 + 16);
}

// A chain's sum of p.v, from the sums v of its virtual threads.  SEQ: one of the 8 warps of a virtual block of 256
// rows; else a block of 8 warps of 4 rows each: rows 0 + 2 and 1 + 3, then these, then the warps in turn.
template <bool SEQ>
__device__ __forceinline__ double chain_sum(double v, int lane)
{
    if (SEQ) {
        const double a[1] = {v};
        return order_warp_sum<1>(a, lane);
    }
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    double w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = __shfl_sync(0xffffffffu, v, 4 * i);
#pragma unroll
    for (int i = 1; i < 8; ++i) w[0] += w[i];
    return w[0];
}

// a barrier of two warps
__device__ __forceinline__ void pair_barrier(int id) { asm volatile("barrier.sync %0, 64;" ::"r"(id) : "memory"); }

template <int NB, int W, int S, bool PASO, bool SEQ>
__global__ void __launch_bounds__(W * 32, 1) k_pcg64(const __grid_constant__ Pcg64Args a, Scal* s)
{
    static_assert(W == 16, "a chain's tiles go to warps w and w + 8");
    constexpr int kStageBytes = 32 * NB * 8 + 16;
    extern __shared__ __align__(128) unsigned char smem_pcg[];
    __shared__ __align__(8) uint64_t full[W][S];
    __shared__ Pcg64State sc;
    __shared__ int bad;
    __shared__ OrderShared os;
    __shared__ double2 hand[8][32];  // a row's A p and p, from warp w + 8 to w
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
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
        sc.norm2 = s->norm * s->norm;
        sc.iter = s->iter;
        sc.status = PCG_RUN;
        sc.stop = 0;
    }
    if (threadIdx.x < 8) os.rows[threadIdx.x] = 0.0;  // (the last CTA may have fewer chains)
    if (threadIdx.x < W * S) mbar_init(&full[threadIdx.x / S][threadIdx.x % S], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();
    const double tol = s->tol;
    const long long maxit = s->maxit;
    bool pend = s->pend != 0;
    int par = s->par;

    // this warp's tiles: of the CTA's chains warp & 7, + 8, ..., every second one
    const int c0 = blockIdx.x * a.cpc, nchains = min(a.cpc, a.chains - c0);
    const bool single = a.ntiles <= a.tstep;  // one tile per chain
    struct Cursor {
        int chain, tile;
    };
    auto seek = [&](Cursor& c) {
        while (c.chain < nchains && c.tile >= a.ntiles) {
            c.chain += 8;
            c.tile = c0 + c.chain + (warp >> 3) * a.tstep;
        }
    };
    auto first = [&]() {
        Cursor c{warp & 7, c0 + (warp & 7) + (warp >> 3) * a.tstep};
        seek(c);
        return c;
    };
    auto next = [&](Cursor& c) {
        c.tile += 2 * a.tstep;
        seek(c);
    };
    int mine = 0;
    for (Cursor c = first(); c.chain < nchains; next(c)) ++mine;
    const bool resident = mine <= S;
    unsigned char* ring = smem_pcg + (size_t)warp * S * kStageBytes;
    int issued = 0, used = 0;     // tiles copied into / taken from the ring
    Cursor nx = first();          // the tile the next copy is for, and its entries' range
    int e0 = 0, e1 = 0;
    auto range = [&]() {
        const int row0 = nx.tile * 32;
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
        next(nx);
        if (nx.chain >= nchains) nx = first();
        range();
    };
    if (lane == 0 && mine > 0) {
        range();
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
        ++gen;
        unsigned long long* set = a.mail + (size_t)(gen & 1u) * kOrderSet;
        // the products of a tile's rows, the warp's k-th; false: the wait for its entries gave up
        auto row_tile = [&](int tile, int k, double& av, double& pc) {
            const int row0 = tile * 32;
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
            constexpr int NA = SEQ ? 1 : 8;  // entry e goes to sum e % NA
            double acc[NA], po = 0.0;
#pragma unroll
            for (int j = 0; j < NA; ++j) acc[j] = 0.0;
            bool waited = false;
            if (__all_sync(0xffffffffu, inner)) {
#pragma unroll
                for (int g = 0; g < NB; g += 9) {
                    double zz[9], pp[9];
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        zz[m] = a.z[row + a.off[g + m]];
                        pp[m] = pold[row + a.off[g + m]];
                    }
                    if (g == 0) waited = mbar_wait(&full[warp][st], ph, polls);
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const double pn = fma(beta, pp[m], zz[m]);
                        acc[(g + m) % NA] = fma(row_val[g + m], pn, acc[(g + m) % NA]);
                        if (g + m == NB / 2) {
                            pc = pn;
                            po = pp[m];
                        }
                    }
                }
            } else if constexpr (SEQ) {
                // a tile with boundary rows (half of them at lines of 129 nodes): nine bands at a time like the
                // others, a missing neighbour's values from the row itself; its entry is left out.  ok9: which of the
                // 3 x 3 neighbours (x, y) of a plane exist
                const int rowc = in ? row : row0;
                const unsigned x3 = !in ? 0u : (cx > 0 ? 1u : 0u) | 2u | (cx + 1 < (unsigned)a.nn0 ? 4u : 0u);
                const unsigned ok9 = (cy > 0 ? x3 : 0u) | x3 << 3 | (cy + 1 < (unsigned)a.nn1 ? x3 << 6 : 0u);
                int e = 0;
#pragma unroll
                for (int g = 0; g < NB; g += 9) {
                    const bool zv = NB == 9 || (g == 0 ? cz > 0 : (g == 18 ? cz + 1 < (unsigned)a.nn2 : true));
                    const unsigned okg = zv ? ok9 : 0u;
                    double zz[9], pp[9];
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const int j = okg >> m & 1u ? row + a.off[g + m] : rowc;
                        zz[m] = a.z[j];
                        pp[m] = pold[j];
                    }
                    if (g == 0) waited = mbar_wait(&full[warp][st], ph, polls);
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const double pn = fma(beta, pp[m], zz[m]);
                        const bool ok = okg >> m & 1u;
                        if (ok) acc[0] = fma(row_val[e], pn, acc[0]);
                        e += ok ? 1 : 0;
                        if (g + m == NB / 2) {
                            pc = pn;
                            po = pp[m];
                        }
                    }
                }
            } else {
                // the same entry by entry, since an entry's number says which sum it goes to: its neighbour by a
                // table of steps
                const int rowc = in ? row : row0;
                const int lx = cx > 0, ly = cy > 0, lz = cz > 0;
                const int ax = 1 + lx + (cx + 1 < (unsigned)a.nn0), ay = 1 + ly + (cy + 1 < (unsigned)a.nn1);
                const int az = NB == 27 ? 1 + lz + (cz + 1 < (unsigned)a.nn2) : 1;
                const int count = in ? ax * ay * az : 0;
                const int ec = lx + ax * (ly + ay * lz);
                const int lowest = row - lx - a.nn0 * ly - (int)plane * lz;
#pragma unroll
                for (int g = 0; g < NB; g += 9) {
                    double zz[9], pp[9];
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const int s3 = ay == 3 ? a.step[0][g + m] : a.step[2][g + m];
                        const int s2 = ay == 3 ? a.step[1][g + m] : a.step[3][g + m];
                        const int j = g + m < count ? lowest + (ax == 3 ? s3 : s2) : rowc;
                        zz[m] = a.z[j];
                        pp[m] = pold[j];
                    }
                    if (g == 0) waited = mbar_wait(&full[warp][st], ph, polls);
#pragma unroll
                    for (int m = 0; m < 9; ++m) {
                        const int e = g + m;
                        const double pn = fma(beta, pp[m], zz[m]);
                        if (e < count) acc[e % NA] = fma(row_val[e], pn, acc[e % NA]);
                        if (e == ec) {
                            pc = pn;
                            po = pp[m];
                        }
                    }
                }
            }
            if (!__all_sync(0xffffffffu, waited)) return false;
            if (!resident) {
                ++used;
                __syncwarp();     // every lane has read the stage that the copy refills
                if (lane == 0) issue();
            }
            if constexpr (SEQ) {
                av = acc[0];
            } else {              // lanes 4, 2, 1 apart, as a butterfly over 8 lanes adds them
                av = ((acc[0] + acc[4]) + (acc[2] + acc[6])) + ((acc[1] + acc[5]) + (acc[3] + acc[7]));
            }
            if (in) {
                pnew[row] = pc;
                a.q[row] = av;
                if (!PASO && xpend) a.x[row] = fma(before, po, xx);
                if (PASO && pend) {
                    const double xn = fma(before, po, xx2);
                    a.x2[row] = xn;
                    a.x[row] = fma(g2, xx, g1 * xn);
                    a.rs[row] = fma(g2, rs, g1 * rr);
                }
            } else {
                av = pc = 0.0;
            }
            return true;
        };
        // a chain's tiles two at a time, by warps w and w + 8; w adds the terms of both in turn
        int k = 0;
        bool failed = false;
        for (int ch = warp & 7; ch < nchains && (warp < 8 || !single); ch += 8) {
            double v = 0.0;
            for (int t = c0 + ch; t < a.ntiles; t += 2 * a.tstep) {
                const int tile = warp < 8 ? t : t + a.tstep;
                double av = 0.0, pc = 0.0;
                if (tile < a.ntiles && !failed) failed = !row_tile(tile, k++, av, pc);
                if (single) {
                    v = fma(av, pc, v);
                } else if (warp < 8) {
                    v = fma(av, pc, v);
                    pair_barrier(1 + warp);
                    const double2 h = hand[warp][lane];
                    v = fma(h.x, h.y, v);
                    pair_barrier(1 + warp);
                } else {
                    hand[warp - 8][lane] = make_double2(av, pc);
                    pair_barrier(1 + warp - 8);
                    pair_barrier(1 + warp - 8);
                }
            }
            if (warp < 8) {
                const double sum = chain_sum<SEQ>(v, lane);
                if (lane == 0) {
                    if (SEQ)
                        os.rows[ch] = sum;
                    else
                        order_post(set + c0 + ch, sum);
                }
            }
        }
        if (failed) bad = 1;
        // phase B's first loads but A p and rs, which the exchange brings
        struct Update {
            double2 r, d, rs, q;
        };
        PairAhead<Update> ahead;
        auto load_update = [&](int h) {
            Update t;
            t.r = ld2(a.r, h);
            t.d = ld2(a.dinv, h);
            return t;
        };
        pair_ahead<W>(a.pairs, a.n, ahead, load_update);
        double t[1];
        bool ok = ordered_sum<true, SEQ, 0>(a.row_blocks, a.pairs, t, os, set, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                sc.status = PCG_TIMEOUT;
                sc.stop = 1;
            } else if (PASO) {
                paso_alpha(sc, t[0], pend);
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
        __syncthreads();
        par ^= 1;
        xpend = false;
        if (sc.stop) break;

        // ---------------------------------------------------------------- phase B
        const double alpha = sc.alpha;
        ++gen;
        set = a.mail + (size_t)(gen & 1u) * kOrderSet;
        constexpr int NX = PASO ? 4 : 2;
        // sums: paso z.r, d.d, d.rs with d = r - rs, and rs^2 of the smoothing; textbook z.r, r.r
        pair_sums<NX, W, Update>(
            a.pairs, a.n, os, set, &ahead, load_update,
            [&](int h, Update& t) {
                t.q = ld2(a.q, h);
                if (PASO) t.rs = ld2(a.rs, h);
            },
            [&](int h, const Update& t, double (&v)[NX]) {
                const double ra = fma(-alpha, t.q.x, t.r.x), rb = fma(-alpha, t.q.y, t.r.y);
                st2(a.r, h, make_double2(ra, rb));
                const double za = ra * t.d.x, zb = rb * t.d.y;
                st2(a.z, h, make_double2(za, zb));
                v[0] = add_pair(v[0], za, ra, zb, rb);
                if (PASO) {
                    const double da = ra - t.rs.x, db = rb - t.rs.y;
                    v[1] = add_pair(v[1], da, da, db, db);
                    v[2 % NX] = add_pair(v[2 % NX], da, t.rs.x, db, t.rs.y);
                    v[3 % NX] = add_pair(v[3 % NX], t.rs.x, t.rs.x, t.rs.y, t.rs.y);
                } else {
                    v[1] = add_pair(v[1], ra, ra, rb, rb);
                }
            },
            [&](int i, double (&v)[NX]) {
                const double rn = fma(-alpha, a.q[i], a.r[i]), zn = rn * a.dinv[i];
                a.r[i] = rn;
                a.z[i] = zn;
                v[0] = fma(zn, rn, v[0]);
                if (PASO) {
                    const double rs = a.rs[i], d = rn - rs;
                    v[1] = fma(d, d, v[1]);
                    v[2 % NX] = fma(d, rs, v[2 % NX]);
                    v[3 % NX] = fma(rs, rs, v[3 % NX]);
                } else {
                    v[1] = fma(rn, rn, v[1]);
                }
            });
        double w[NX];
        ok = ordered_sum<false, false, NX>(0, a.pairs, w, os, set, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                sc.status = PCG_TIMEOUT;
                sc.stop = 1;
            } else if (PASO) {
                paso_next(sc, w, pend, tol, maxit);
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
    if (!PASO && xpend) {         // this warp's rows: it wrote their p and x itself
        const double alpha = sc.alpha;
        const double* p = par ? a.p1 : a.p0;
        for (Cursor c = first(); c.chain < nchains; next(c)) {
            const int row = c.tile * 32 + lane;
            if (row < a.n) a.x[row] = fma(alpha, p[row], a.x[row]);
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
            s->norm = PASO ? sqrt(sc.norm2) : sc.norm;
            s->iter = sc.iter;
            s->par = par;
            s->pend = pend ? 1 : 0;
            if (sc.status != PCG_RUN) report_status(s, sc.status);
        }
    }
}
