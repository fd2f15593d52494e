// paso's FP64 PCG with the operator marched from the element coefficients (rg_march.cuh) instead of
// streamed from the CSR values: 8 bytes of kappa per row and iteration for 216 of matrix.  Included by
// rg_solver.cu inside namespace rg, after rg_pcg64.cuh.
//
// Used for matrices whose coefficient record describes the values (A = kappa I per element and a
// constraint), whose values no caller holds a pointer to, and that are large enough for the matrix's
// bytes to matter (kCoef64Rows).  The outer residual test reads the CSR values as ever.
//
// The balanced system B A B x~ = B b is iterated in the variables that need no balance vector at the
// neighbours: P = B p~ and Z = B z~ (A P is then B^-1 q~, and p~.q~ = P.A P), X = B x~, X2 = B x2~; r~ and
// rs~ stay balanced.  Rows of fixed nodes are identity rows with r~ = 0 (their first x~ is exact); Z is
// kept 0 there, so they drop out of the others' sums.
//
// Two phases and exchanges per iteration as in k_pcg64.  Phase B goes over the rows the block's own warps
// marched, so what it reads was written by this block.  Bound by HBM at 128^3 (19 vector accesses of 8 B
// per row): 84 against 158 us per iteration on the CSR values.
#pragma once

struct Pcg64CoefArgs {
    MarchGeom g;
    MarchTab<double> t;
    const double* khat;
    double *r, *q, *rs, *x, *x2, *z, *p0, *p1;
    const double *dinv, *bvm;     // bvm: the balance vector, negative at fixed nodes
    int max_iters;
    unsigned long long* mail;
};

// march_task's view of phase A
struct Pcg64CoefOp {
    struct Keep {
        double rs, r, x, x2, pold;
    };
    struct Side {
        double z, p;
    };
    struct Center {
        double z, p;
        Keep k;
    };
    const double *z, *pold;
    double *pnew, *q, *rs, *x, *x2;
    const double* r;
    double alpha, beta, g1, g2;   // alpha: of the iteration before
    bool pend;
    double v[2];                  // p.A p, |rs|^2
    __device__ __forceinline__ Side load(int row) const { return Side{load_ahead(z + row), load_ahead(pold + row)}; }
    __device__ __forceinline__ Center load_center(int row) const
    {
        Center c{load_ahead(z + row), load_ahead(pold + row), {0.0, 0.0, 0.0, 0.0, 0.0}};
        if (pend) c.k = Keep{load_ahead(rs + row), load_ahead(r + row), load_ahead(x + row), load_ahead(x2 + row), 0.0};
        return c;
    }
    __device__ __forceinline__ double value(const Side& s) const { return fma(beta, s.p, s.z); }
    __device__ __forceinline__ double value(const Center& c, Keep& k) const
    {
        k = c.k;
        k.pold = c.p;
        return fma(beta, c.p, c.z);
    }
    __device__ __forceinline__ void emit(int row, double p, const Keep& k, double au, double, bool fixed)
    {
        const double w = fixed ? p : au;
        pnew[row] = p;
        q[row] = w;
        v[0] += p * w;
        if (pend) {
            const double rn = g2 * k.rs + g1 * k.r;
            rs[row] = rn;
            const double xn = k.x2 + alpha * k.pold;
            x2[row] = xn;
            x[row] = g2 * k.x + g1 * xn;
            v[1] += rn * rn;
        }
    }
};

template <int DIM, int W>
__global__ void __launch_bounds__(W * 32, 1) k_pcg64_coef(const __grid_constant__ Pcg64CoefArgs a, Scal* s)
{
    __shared__ Pcg64State sc;
    __shared__ int bad;
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
        sc.norm = s->norm;
        sc.iter = s->iter;
        sc.status = PCG_RUN;
        sc.stop = 0;
    }
    __syncthreads();
    const double tol = s->tol;
    const long long maxit = s->maxit;
    bool pend = s->pend != 0;
    int par = s->par;
    unsigned gen = 0;
    const int blocks = a.g.per_slab * a.g.slabs;
    for (int left = a.max_iters; left > 0; --left) {
        // ---------------------------------------------------------------- phase A
        double* pnew = par ? a.p0 : a.p1;
        Pcg64CoefOp op{a.z, par ? a.p1 : a.p0, pnew, a.q, a.rs, a.x, a.x2, a.r,
                       sc.alpha, sc.beta, sc.g1, sc.g2, pend, {0.0, 0.0}};
        if (warp < a.g.wpc)
            for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
                const int slab = blk / a.g.per_slab, strip = (blk - slab * a.g.per_slab) * a.g.wpc + warp;
                if (strip < a.g.strips) march_task<DIM, 1, double, DiffRow<double>>(a.g, a.t, a.khat, strip, slab, lane, op);
            }
        double t[2];
        ++gen;
        bool ok = mail_sum<2, W, false>(op.v, t, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                sc.status = PCG_TIMEOUT;
                sc.stop = 1;
            } else {
                paso_after_a(sc, t, pend, tol, maxit);
            }
        }
        __syncthreads();
        par ^= 1;
        if (sc.stop) break;

        // ---------------------------------------------------------------- phase B
        const double alpha = sc.alpha;
        double u[3] = {0.0, 0.0, 0.0};
        for (int blk = blockIdx.x; blk < blocks; blk += gridDim.x) {
            // the block's strips are one run of nodes per plane of its slab
            const int slab = blk / a.g.per_slab, j0 = (blk - slab * a.g.per_slab) * a.g.wpc * kStrip;
            const int len = min(a.g.wpc * kStrip, a.g.J - j0);
            const int z0 = slab * a.g.tz, z1 = min(z0 + a.g.tz, a.g.NP);
            for (int z = z0 + warp; z < z1; z += W) {
                const int row0 = z * a.g.M + j0;
#pragma unroll 4
                for (int i = lane; i < len; i += 32) {
                    const int row = row0 + i;
                    const double b = __ldg(a.bvm + row), di = __ldg(a.dinv + row);
                    const double ri = a.r[row], qi = a.q[row], rsi = a.rs[row];
                    const bool fixed = b < 0.0;
                    const double rn = ri - alpha * (fixed ? 0.0 : b * qi);
                    a.r[row] = rn;
                    const double zn = di * rn;  // z~
                    a.z[row] = fixed ? 0.0 : b * zn;
                    u[0] += zn * rn;
                    const double d = rn - rsi;
                    u[1] += d * d;
                    u[2] += d * rsi;
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
            } else {
                paso_after_b(sc, w);
                if (left == 1) sc.stop = 1;
            }
        }
        __syncthreads();
        pend = true;
        if (sc.stop) break;
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
            s->delta = sc.delta;
            s->norm = sc.norm;
            s->iter = sc.iter;
            s->par = par;
            s->pend = pend ? 1 : 0;
            if (sc.status != PCG_RUN) report_status(s, sc.status);
        }
    }
}

// From k_paso_init's balanced z = p, x = x2 to the iteration's variables, and the signed balance vector.
__global__ void k_pcg64_coef_enter(int64_t n, const double* __restrict__ khat, const double* __restrict__ bv,
                                   double* __restrict__ bvm, double* __restrict__ z, double* __restrict__ p,
                                   double* __restrict__ x, double* __restrict__ x2)
{
    for (int64_t i = gtid(); i < n; i += gstride()) {
        const bool fixed = signbit(khat[i]);
        const double b = bv[i], zi = fixed ? 0.0 : b * z[i], xi = b * x[i];
        bvm[i] = fixed ? -b : b;
        z[i] = zi;
        p[i] = zi;
        x[i] = xi;
        x2[i] = xi;
    }
}

__global__ void k_pcg64_coef_leave(int64_t n, const double* __restrict__ bv, double* __restrict__ x)
{
    for (int64_t i = gtid(); i < n; i += gstride()) x[i] /= bv[i];
}
