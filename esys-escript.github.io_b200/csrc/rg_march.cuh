// The Q1 operator of A = kappa I per element applied on the fly, one warp marching a strip of
// nodes through the planes of the grid.  Included by rg_solver.cu inside namespace rg.
//
// A plane is NN0 x NN1 nodes in 3D (a line of NN0 in 2D), cut into groups of NR x-lines.  A lane owns
// one x of a group (NR nodes), the groups' positions are numbered in one run, and a warp owns 30
// consecutive ones (lanes 1 to 30; lanes 0 and 31 only carry the neighbours' values) and walks a slab of
// planes.  Runs wrap from one group to the next without a test: the elements that would join such
// nodes do not exist, and khat (node-indexed kappa of the element whose upper corner is the node) is 0
// there.  Two lines per lane share the loads, values and x-neighbours of the lines between them: 4 lines
// for 2 rows instead of 3 for one.
//
// Two ways to form a node's product:
//  DiffRow (FP64).  In a layer between two planes the elements beside a node column contribute
//     sum_e kappa_e (P_e(z) + Q_e(z+1) + w)  to the lower node,
//     sum_e kappa_e (P_e(z+1) + Q_e(z) - w)  to the upper,
//   where P_e and Q_e are the element's in-plane differences to the node's own value, weighted with
//   the Q1 table entries of nodes in the same plane and in different planes, and w = S_Q (u(z+1) -
//   u(z)), S_Q the sum of the latter (a row of the table sums to zero).  The table weights come after the
//   sums over the elements (differences in x times kappa summed over y, and so on), so a node costs 8
//   differences and about 34 multiply-adds instead of 27 coefficients formed and multiplied.
//  BandRow (FP32).  The 27 (9) coefficients T (sum of kappa), and the products added in band order, as a row of
//   the stored matrix: in FP32 another order ends a refinement elsewhere below the tolerance (1e-9 of the
//   solution), and this one is what every configuration and the segment start return bit for bit.  A
//   plane's values finish the node below (its upper nine), go into the node itself, and start the node above,
//   whose lower nine coefficients are the upper nine of this one: 27.3 us
//   per iteration at 128^3 and 180 at 256^3 against 26.8 and 178 by differences (which carry fewer terms).
//
// What is stored of the next plane's nodes, and kappa of the layer below it, is loaded into registers
// before the arithmetic of a layer.  Staged in shared memory instead (per-lane cp.async, three planes
// ahead) each line passes the L1 data pipe three times, and by bulk copies the copy engine sees nine
// small copies per plane and warp: both were slower (24.5 and 27.6 us per FP32 iteration at 128^3).
#pragma once

constexpr int kStrip = 30;            // run positions a warp owns
constexpr int kMarchAhead = 1;        // planes loaded ahead (by differences, 2 and 3 were slower: 26 and 27 against 22 us at 128^3)

struct MarchGeom {
    int M, NN0, NL, NP;               // nodes per plane, per line; lines per plane; planes
    int J;                            // run positions: groups of NR lines x NN0
    int strips, slabs, tz;            // strips of a plane; slabs of tz planes
    int wpc, per_slab;                // strips (warps) of a block, blocks of a slab: a block's strips lie side
                                      // by side in one slab and share their lines in L1
};

// Table entries T[x differs + 2 (y differs) + 4 (z differs)]; in 2D the marching axis is y.
template <typename T>
struct MarchTab {
    T t[8];
    T px, py, pxy;                    // DiffRow: same plane
    T qx, qy, qxy;                    // different planes
    T sq;                             // sum of the different-plane entries, the node's own column included
};

template <typename T>
MarchTab<T> march_table(const double (&t)[8])
{
    MarchTab<T> m{};
    for (int k = 0; k < 8; ++k) m.t[k] = (T)t[k];
    m.px = (T)t[1];
    m.py = (T)t[2];
    m.pxy = (T)t[3];
    m.qx = (T)t[5];
    m.qy = (T)t[6];
    m.qxy = (T)t[7];
    m.sq = (T)(t[4] + t[5] + t[6] + t[7]);
    return m;
}

// Loads that stay where they are written: ahead of the arithmetic that hides them (the compiler
// moves plain loads down to their uses to save registers).
__device__ __forceinline__ float4 load_ahead(const float4* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float load_ahead(const float* p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double load_ahead(const double* p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// kappa of a layer's elements beside a node: [a] along x, [b] along y
template <typename T>
struct Layer {
    T k[2][2];
};

template <typename T>
struct DiffRow {
    static constexpr bool kThree = true;  // 3D only
    // of the node below: its value, what it has got so far; what its plane adds to this node
    T u_lo = 0, acc = 0, up = 0;
    // the plane's values n[y][x] around the node, the layers below and above: emit(u, A u, diagonal) of the node below
    template <class Emit>
    __device__ __forceinline__ void step(const MarchTab<T>& t, const T (&n)[3][3], const Layer<T>& lb, const Layer<T>& la,
                                         Emit emit)
    {
        const T u = n[1][1];
        const T x0 = n[1][0] - u, x1 = n[1][2] - u, y0 = n[0][1] - u, y1 = n[2][1] - u;
        const T c00 = n[0][0] - u, c10 = n[0][2] - u, c01 = n[2][0] - u, c11 = n[2][2] - u;
        auto sums = [&](const Layer<T>& l, T& sx, T& sy, T& sxy, T& ks) {
            const T k00 = l.k[0][0], k10 = l.k[1][0], k01 = l.k[0][1], k11 = l.k[1][1];
            const T ky0 = k00 + k10, ky1 = k01 + k11;
            ks = ky0 + ky1;
            sx = fma(k10 + k11, x1, (k00 + k01) * x0);
            sy = fma(ky1, y1, ky0 * y0);
            sxy = fma(k11, c11, fma(k01, c01, fma(k10, c10, k00 * c00)));
        };
        T bx, by, bxy, ksb, ax, ay, axy, ksa;
        sums(lb, bx, by, bxy, ksb);
        sums(la, ax, ay, axy, ksa);
        const T qb = fma(t.qx, bx, fma(t.qy, by, t.qxy * bxy));
        const T qa = fma(t.qx, ax, fma(t.qy, ay, t.qxy * axy));
        const T p = fma(t.px, bx + ax, fma(t.py, by + ay, t.pxy * (bxy + axy)));
        const T w = t.sq * ((u - u_lo) * ksb);
        emit(u_lo, acc + (qb + w), T(0));
        acc = p + (up - w);
        up = qa;
        u_lo = u;
    }
    // the node of the last plane, which has no layer above
    template <class Emit>
    __device__ __forceinline__ void last(Emit emit) { emit(u_lo, acc, T(0)); }
};

template <int DIM>
struct BandRow {
    static constexpr int N = DIM == 3 ? 9 : 3;
    // of the node below: its value, its lower and middle products, its diagonal; this node's lower products
    float u_lo = 0.f, acc = 0.f, diag_lo = 0.f, lower = 0.f;
    // sums of kappa over the elements that a neighbour of band j of the plane shares with the node
    __device__ __forceinline__ static void sums(const Layer<float>& l, float (&s)[N])
    {
        float sx[3][2];
#pragma unroll
        for (int b = 0; b < (DIM == 3 ? 2 : 1); ++b) {
            sx[0][b] = l.k[0][b];
            sx[1][b] = l.k[0][b] + l.k[1][b];
            sx[2][b] = l.k[1][b];
        }
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            s[x] = sx[x][0];
            if (DIM == 3) {
                s[(3 + x) % N] = sx[x][0] + sx[x][1];
                s[(6 + x) % N] = sx[x][1];
                s[x] = sx[x][0];
            }
        }
    }
    template <class Emit>
    __device__ __forceinline__ void step(const MarchTab<float>& t, const float (&n)[3][3], const Layer<float>& lb,
                                         const Layer<float>& la, Emit emit)
    {
        float sb[N], sa[N];
        sums(lb, sb);
        sums(la, sa);
        float fin = acc, mid = lower, low = 0.f, diag = 0.f;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const int x = j % 3, y = DIM == 3 ? j / 3 : 1;
            const int cls = (x != 1) + (DIM == 3 ? 2 * (y != 1) : 0), other = cls + (DIM == 3 ? 4 : 2);
            const float v = n[y][x];
            fin = fmaf(t.t[other] * sb[j], v, fin);
            const float c = t.t[cls] * (sb[j] + sa[j]);
            mid = fmaf(c, v, mid);
            low = fmaf(t.t[other] * sa[j], v, low);
            if (j == N / 2) diag = c;
        }
        emit(u_lo, fin, diag_lo);
        acc = mid;
        lower = low;
        u_lo = n[1][1];
        diag_lo = diag;
    }
    template <class Emit>
    __device__ __forceinline__ void last(Emit emit) { emit(u_lo, acc, diag_lo); }
};

// One task: strip `strip` of slab `slab`.  op.load(row) / op.load_center(row) load what is stored of a
// node (Side / Center), op.value(side) and op.value(center, keep) form its value, keep being what emit
// needs of a node the warp owns.  emit(row, u, keep, au, diag, fixed) gets every owned node's value,
// (A u), the diagonal (BandRow) and whether the constraint fixes it (then au is meaningless).
template <int DIM, int NR, typename T, class Row, class Op>
__device__ __forceinline__ void march_task(const MarchGeom& g, const MarchTab<T>& t, const T* __restrict__ khat,
                                           int strip, int slab, int lane, Op& op)
{
    static_assert(DIM == 3 || NR == 1, "2D marches one line");
    constexpr int NKL = DIM == 3 ? NR + 1 : 1;                       // lines of kappa beside the lane's nodes
    const int z0 = slab * g.tz, z1 = min(z0 + g.tz, g.NP);
    const int j = strip * kStrip - 1 + lane;
    const int jj = min(max(j, 0), g.J - 1);
    const int group = jj / g.NN0;
    const int c = group * NR * g.NN0 + (jj - group * g.NN0);         // the lane's first node in the plane
    // past the run's end a lane stands in for the missing neighbour: kappa of a line's first node, 0
    const int ck = j < g.J ? c : group * NR * g.NN0;
    const bool own = lane >= 1 && lane <= kStrip && j < g.J;
    const int rows = own ? min(NR, g.NL - group * NR) : 0;
    int line[NR + 2];                                                // nodes of the lines, inside the plane
#pragma unroll
    for (int k = 0; k < NR + 2; ++k) line[k] = DIM == 3 ? min(max(c + (k - 1) * g.NN0, 0), g.M - 1) : c;
    const int pb = max(z0 - 1, 0), pe = min(z1, g.NP - 1);           // planes read
    struct Fetched {                  // a plane's stored nodes, and kappa (a = 0) of the layer above it
        typename Op::Center rc[NR];
        typename Op::Side rs[2];
        T k[NKL];
    };
    auto fetch_kappa = [&](int z, T (&k)[NKL]) {  // of the layer below plane z
#pragma unroll
        for (int l = 0; l < NKL; ++l) k[l] = load_ahead(khat + (z * g.M + ck + l * g.NN0));
    };
    auto fetch = [&](int z, Fetched& f) {
        const int o = z * g.M;
#pragma unroll
        for (int r = 0; r < NR; ++r) f.rc[r] = op.load_center(o + line[r + 1]);
        if (DIM == 3) {
            f.rs[0] = op.load(o + line[0]);
            f.rs[1] = op.load(o + line[NR + 1]);
        }
        fetch_kappa(z + 1, f.k);
    };
    // carried from plane to plane: kappa of the layer below, and of each node the row's sums, what emit needs
    // of it and whether it is fixed (the sign of kappa)
    T b0[NKL], b1[NKL];                   // of the elements at a = 0 / 1
    Row row[NR];
    typename Op::Keep keep[NR];
    bool fixed[NR], fixed_z[NR];
    Fetched f[kMarchAhead];
    T kb[NKL];
    fetch_kappa(pb, kb);
#pragma unroll
    for (int k = 0; k < kMarchAhead; ++k)
        if (pb + k <= pe) fetch(pb + k, f[k]);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        fixed[r] = false;
        fixed_z[r] = signbit(kb[r]);
    }
#pragma unroll
    for (int l = 0; l < NKL; ++l) {
        b0[l] = (T)fabs(kb[l]);
        b1[l] = __shfl_down_sync(0xffffffffu, b0[l], 1);
    }
    auto plane = [&](int z, Fetched& f) {
        T v[NR + 2];
        typename Op::Keep keep_z[NR];
        T a0[NKL], a1[NKL];
        bool fixed_a[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) v[r + 1] = op.value(f.rc[r], keep_z[r]);
        if (DIM == 3) {
            v[0] = op.value(f.rs[0]);
            v[NR + 1] = op.value(f.rs[1]);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) fixed_a[r] = signbit(f.k[r]);
#pragma unroll
        for (int l = 0; l < NKL; ++l) a0[l] = (T)fabs(f.k[l]);
        if (z + kMarchAhead <= pe) fetch(z + kMarchAhead, f);
        T vl[NR + 2], vh[NR + 2];
#pragma unroll
        for (int k = 0; k < NR + 2; ++k) {
            if (DIM == 2 && k != 1) continue;
            vl[k] = __shfl_up_sync(0xffffffffu, v[k], 1);
            vh[k] = __shfl_down_sync(0xffffffffu, v[k], 1);
        }
#pragma unroll
        for (int l = 0; l < NKL; ++l) a1[l] = __shfl_down_sync(0xffffffffu, a0[l], 1);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            T n[3][3];
            Layer<T> lb, la;
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                if (DIM == 2 && y != 1) continue;
                n[y][0] = vl[r + y];
                n[y][1] = v[r + y];
                n[y][2] = vh[r + y];
            }
#pragma unroll
            for (int y = 0; y < (DIM == 3 ? 2 : 1); ++y) {
                lb.k[0][y] = b0[r + y];
                lb.k[1][y] = b1[r + y];
                la.k[0][y] = a0[r + y];
                la.k[1][y] = a1[r + y];
            }
            row[r].step(t, n, lb, la, [&](T u, T au, T diag) {
                if (z > z0 && r < rows) op.emit((z - 1) * g.M + c + r * g.NN0, u, keep[r], au, diag, fixed[r]);
            });
            keep[r] = keep_z[r];
            fixed[r] = fixed_z[r];
            fixed_z[r] = fixed_a[r];
        }
#pragma unroll
        for (int l = 0; l < NKL; ++l) {
            b0[l] = a0[l];
            b1[l] = a1[l];
        }
    };
#pragma unroll 1
    for (int z = pb; z <= pe; z += kMarchAhead) {
#pragma unroll
        for (int k = 0; k < kMarchAhead; ++k)
            if (z + k <= pe) plane(z + k, f[k]);
    }
    if (z1 == g.NP)  // the last plane has no layer above
#pragma unroll
        for (int r = 0; r < NR; ++r)
            row[r].last([&](T u, T au, T diag) {
                if (r < rows) op.emit((z1 - 1) * g.M + c + r * g.NN0, u, keep[r], au, diag, fixed[r]);
            });
}

// Splits the grid for `ctas` blocks of at most `warps` warps: as many slabs as make the rounds of the
// blocks cheapest, counting a task's two halo planes.
inline MarchGeom march_geom(int dim, const int64_t nn[3], int lines, int ctas, int warps)
{
    MarchGeom g{};
    g.NN0 = (int)nn[0];
    g.NL = dim == 3 ? (int)nn[1] : 1;
    g.M = g.NN0 * g.NL;
    g.NP = (int)(dim == 3 ? nn[2] : nn[1]);
    g.J = (g.NL + lines - 1) / lines * g.NN0;
    g.strips = (g.J + kStrip - 1) / kStrip;
    double best = 1e300;
    for (int k = 1; k <= g.NP; ++k) {
        const int tz = (g.NP + k - 1) / k, slabs = (g.NP + tz - 1) / tz;
        // blocks of a slab: as few warps per block as still fit one round, at most `warps`
        int per_slab = (g.strips + warps - 1) / warps;
        if ((int64_t)per_slab * slabs <= ctas) per_slab = std::min(g.strips, ctas / slabs);
        const int wpc = (g.strips + per_slab - 1) / per_slab;
        per_slab = (g.strips + wpc - 1) / wpc;
        const int64_t rounds = ((int64_t)per_slab * slabs + ctas - 1) / ctas;
        const double cost = (double)rounds * (tz + 1.3) * (4 + wpc);
        if (cost < best * 0.999) {
            best = cost;
            g.slabs = slabs;
            g.tz = tz;
            g.wpc = wpc;
            g.per_slab = per_slab;
        }
    }
    return g;
}

inline int march_ctas(const MarchGeom& g, int ctas) { return std::min(ctas, g.per_slab * g.slabs); }
