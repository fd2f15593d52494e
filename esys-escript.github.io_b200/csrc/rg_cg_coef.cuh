// The FP32 PCG on the element-coefficient operator (RG_LAYOUT_COEF): the recurrence of k_f32_cg with
// A evaluated by marching strips (rg_march.cuh), many iterations in one persistent kernel.  Included by
// rg_solver.cu inside namespace rg, after cg_scalars.
//
// A is the unbalanced operator: the Jacobi-preconditioned iteration is the same for any symmetric
// diagonal scaling of the matrix, so the balancing is applied only where the FP64 refinement hands
// residuals and corrections over.  Rows of nodes fixed by the constraint are identity rows, solved
// exactly by the seed; their state stays zero, so their columns drop out of every other row without
// a mask.
//
// Per iteration a row's state {u, D^-1 A u, D^-1 s_prev, p_prev} (16 bytes) is read (again by its
// neighbours, from L1 or L2) and the new one written, with kappa (4); one grid-wide exchange of five sums
// ends it.  The correction d takes the steps of two iterations at a time (p of the one before is in the
// state): 8 bytes every second iteration, the same roundings in the same order; a step still to be taken
// when the iterations end (dpend) is taken where d is folded into the solution.
//
// What bounds it: loads from L2 and the exchange at 128^3 (issue slots 48 % active, DRAM 17 %;
// 68 MB of state, written and read alternately, and 17 MB of kappa and d in an L2 that keeps about 70 MB of
// such a pattern: a copy of 50 MB runs at 6.9 TB/s, one of 34 MB at 8.1), HBM at
// 256^3.  Measured per iteration (launches of ten) against one launch per iteration with a row's 27
// coefficients formed and multiplied by one thread: 27.3 against 46.3 us at 128^3, 180 against 269 us at
// 256^3, with the same bits.
#pragma once

struct CoefCgArgs {
    MarchGeom g;
    MarchTab<float> t;
    const float* khat;
    float4* v[2];
    float* d;
    int max_iters;
    unsigned long long* mail;
};

// march_task's view of an iteration: a node's state, and on the warp's own line the correction
struct CoefCgOp {
    struct Keep {
        float spn, pn, d;             // D^-1 s_i, p_i, the correction so far
    };
    struct Center {
        float4 s;
        float d;
    };
    using Side = float4;
    const float4* vin;
    float4* vout;
    float* d;
    float alpha, beta;
    float before;                     // the step length of the iteration before, when d has yet to take it
    bool step_d;                      // whether this iteration updates d
    double v[5];                      // r.u, u.w, u.s, p.w, p.s
    __device__ __forceinline__ Side load(int row) const { return load_ahead(vin + row); }
    __device__ __forceinline__ Center load_center(int row) const
    {
        return Center{load_ahead(vin + row), step_d ? load_ahead(d + row) : 0.f};
    }
    __device__ __forceinline__ float value(const Side& s) const { return next_u(s, alpha, beta); }
    __device__ __forceinline__ float value(const Center& c, Keep& k) const
    {
        const float4 s = c.s;
        k.d = fmaf(before, s.w, c.d);
        k.spn = fmaf(beta, s.z, s.y);
        k.pn = fmaf(beta, s.w, s.x);
        return fmaf(-alpha, k.spn, s.x);  // u_{i+1}, as next_u forms it
    }
    __device__ __forceinline__ void emit(int row, float un, const Keep& k, float au, float dg, bool fixed)
    {
        const float w = fixed ? 0.f : au;
        const float diag = fixed ? 1.f : dg;
        if (step_d) d[row] = fmaf(alpha, k.pn, k.d);
        vout[row] = make_float4(un, __fdividef(w, diag), k.spn, k.pn);
        const double du = un, dd = diag, dw = w, dp = k.pn, ds = (double)k.spn * dd;
        v[0] += dd * du * du;
        v[1] += du * dw;
        v[2] += du * ds;
        v[3] += dp * dw;
        v[4] += dp * ds;
    }
};

// and of a segment start: PASS 0 forms D^-1 A p, PASS 1 A u
template <int PASS>
struct CoefStartOp {
    using Side = float4;
    using Center = float4;
    using Keep = float4;
    const float4* vin;
    float4* vout;
    double v[6];
    __device__ __forceinline__ Side load(int row) const { return load_ahead(vin + row); }
    __device__ __forceinline__ Center load_center(int row) const { return load_ahead(vin + row); }
    __device__ __forceinline__ float value(const Side& s) const { return PASS == 0 ? s.w : s.x; }
    __device__ __forceinline__ float value(const Center& c, Keep& k) const
    {
        k = c;
        return PASS == 0 ? c.w : c.x;
    }
    __device__ __forceinline__ void emit(int row, float, const Keep& k, float au, float dg, bool fixed)
    {
        const float w = fixed ? 0.f : au;
        const float diag = fixed ? 1.f : dg;
        if (PASS == 0) {
            vout[row] = make_float4(k.x, 0.f, __fdividef(w, diag), k.w);
        } else {
            const float spn = vout[row].z;  // this thread's PASS 0
            vout[row] = make_float4(k.x, __fdividef(w, diag), spn, k.w);
            const double du = k.x, pn = k.w, dd = diag, ds = (double)spn * dd;
            v[0] += dd * du * du;
            v[2] += du * (double)w;
            v[3] += du * ds;
            v[4] += pn * (double)w;
            v[5] += pn * ds;
        }
    }
};

template <int DIM, int NR, int W>
__global__ void __launch_bounds__(W * 32, 1) k_f32_cg_coef(const __grid_constant__ CoefCgArgs a, Scal* s)
{
    __shared__ Scal sc;
    __shared__ int bad;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const WaitCtl wc = g_wait_ctl;
    const int polls = wc.polls > 0 ? wc.polls : kDefaultPolls;
    if (s->done) return;
    if (threadIdx.x == 0) {
        sc = *s;
        bad = 0;
    }
    __syncthreads();
    int par = (int)(sc.pk & 1);
    unsigned gen = 0;
    for (int it = 0; it < a.max_iters; ++it) {
        const bool step_d = sc.dpend_on != 0;
        CoefCgOp op{a.v[par], a.v[par ^ 1], a.d, (float)sc.alpha, (float)sc.beta, (float)sc.dpend, step_d, {}};
        if (warp < a.g.wpc)
            for (int blk = blockIdx.x; blk < a.g.per_slab * a.g.slabs; blk += gridDim.x) {
                const int slab = blk / a.g.per_slab, strip = (blk - slab * a.g.per_slab) * a.g.wpc + warp;
                if (strip < a.g.strips)
                    march_task<DIM, NR, float, BandRow<DIM>>(a.g, a.t, a.khat, strip, slab, lane, op);
            }
        double t[5];
        ++gen;
        const bool ok = mail_sum<5, W, true>(op.v, t, a.mail, gen, &bad, polls, wc.withhold != 0);
        if (threadIdx.x == 0) {
            if (!ok) {
                report_status(&sc, ST_TIMEOUT);
            } else {
                // the segment's stopping norm: r.u = r.D^-1 r, which paso's balancing leaves unchanged and
                // which is |B r|^2 when the balance vector is D^-1/2 (diagonally dominant rows)
                sc.dpend = step_d ? 0.0 : sc.alpha;
                sc.dpend_on = step_d ? 0 : 1;
                const double tt[6] = {t[0], t[0], t[1], t[2], t[3], t[4]};
                cg_scalars(&sc, tt, 0);
            }
        }
        __syncthreads();
        par ^= 1;
        if (sc.done) break;
    }
    if (threadIdx.x == 0) {
        if (sc.status == ST_TIMEOUT)
            report_status(s, ST_TIMEOUT);
        else if (blockIdx.x == 0)
            *s = sc;
    }
}

// Start of a segment (mode 1: fresh, 2: the direction is kept): u was just seeded from the FP64
// residual; A u and A p are formed afresh and the first step length set.  Two marches per strip.
template <int DIM>
__global__ void __launch_bounds__(128) k_f32_cg_coef_start(const __grid_constant__ CoefCgArgs a, ReduceBuf rb, Scal* s,
                                                           int mode)
{
    const int lane = threadIdx.x & 31;
    const int par = (int)(s->pk & 1);
    CoefStartOp<0> op0{a.v[par], a.v[par ^ 1], {}};
    CoefStartOp<1> op1{a.v[par], a.v[par ^ 1], {}};
    const int warps = (int)((gridDim.x * blockDim.x) >> 5);
    for (int task = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); task < a.g.strips * a.g.slabs; task += warps) {
        const int slab = task / a.g.strips, strip = task - slab * a.g.strips;
        march_task<DIM, 1, float, BandRow<DIM>>(a.g, a.t, a.khat, strip, slab, lane, op0);
        march_task<DIM, 1, float, BandRow<DIM>>(a.g, a.t, a.khat, strip, slab, lane, op1);
    }
    double tt[6];
    if (grid_reduce<6>(op1.v, rb, tt) && threadIdx.x == 0) {
        tt[1] = tt[0];
        cg_scalars(s, tt, mode);
    }
}
