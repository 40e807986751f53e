// Expansions at points as matrix products on the FP64 tensor cores: the body
// shared by the evaluation pass (lap_kernels.cu) and its Hessians (hess.cu).
//
// A harmonic sum over an expansion is, in real harmonics, a
// (points x harmonics) (harmonics x columns) product: one pair of columns (the
// real and imaginary parts) per quantity, the potential and the three gradient
// components or the six second derivatives, whose coefficient arrays the ladder
// identities give.  Each lane generates its A operands itself: in the MMA's
// layout lane l holds point l / 4 and harmonic l % 4 of a K step, and the K
// order is free, so lane l runs the recurrence of the orders m = 4 t + l % 4
// along the degree n, for t = 0, 1, ..., and no harmonic passes through shared
// memory.  A step (t, n) is two MMAs per column block, of the cosine and the
// sine parts; orders above the degree contribute zeros (a quarter of the steps).
// The columns, staged once per expansion and work item in shared memory, serve
// up to 128 points.
#pragma once
#include "dmma.cuh"
#include "lap_kernels.cuh"

namespace fmm {

constexpr int kEvalThreads = 128;   // threads and points of a work item
constexpr int kEvalGroup = 8;       // expansions of a work item
constexpr size_t kEmmSmemMax = 226 * 1024;

__device__ __forceinline__ int eval_nbx(const TreeView &tv, int b)
{
    return (tv.level[b] >= 2 ? 1 : 0) + tv.l3_start[b + 1] - tv.l3_start[b];
}

// Side of box b: the root side of its instance (forests) or of the tree, halved per level.
__device__ __forceinline__ double box_side(const TreeView &tv, int b)
{
    const double size = tv.binst ? tv.inst_geom[4 * tv.binst[b] + 3] : tv.size;
    return size / (double)(1L << tv.level[b]);
}

// Steps of degree <= nmax: for each t, the degrees 4 t .. nmax.
__host__ __device__ constexpr int emm_steps(int nmax)
{
    int s = 0;
    for (int t = 0; 4 * t <= nmax; t++) s += nmax - 4 * t + 1;
    return s;
}

// Doubles of shared memory for degrees up to nmax and nc column blocks of 8:
// columns, recurrence factors, diagonal factors and the step table.
__host__ __device__ constexpr size_t emm_smem(int nmax, int nc)
{
    const size_t s = emm_steps(nmax);
    return s * 8 * 8 * nc + s * 8 + nmax + 1 + (s + 1) / 2;
}

// What the steps of an order need beside the coefficients, on the device (made once
// per order): recurrence factors and degrees of the steps, diagonal factors, and
// the ladder factors of the columns, [step][q][2 signs of m][NF], for local
// expansions and for multipoles.
struct EmmTab {
    const double2 *ab;
    const double *cm;
    const int *step;
    const double *fac[2];   // multipole, local
};

struct EmmShared {
    double *B;      // [step][part][q][8 nc], columns rotated so that the half warp's rows meet different banks
    double2 *ab;    // [step][q]: recurrence factors of (n, m = 4 t + q)
    double *cm;     // [m]: factor of the diagonal R_{m-1}^{m-1} -> R_m^m
    int *step;      // degree and t of every step
    int nmax, nstep;
};

template <int NC>
__device__ __forceinline__ int emm_col(int step, int part, int q, int col)
{
    const int c = NC == 1 ? (col + 4 * (q >> 1)) & 7 : (col + 4 * q) & 15;
    return ((step * 2 + part) * 4 + q) * (8 * NC) + c;
}

// Recurrence factors of step i / 4, q = i % 4 at maximum degree nmax; returns n | t << 16.
__device__ __forceinline__ int emm_factors(int i, int nmax, double2 &ab)
{
    int s = i >> 2, t = 0;
    while (s >= nmax - 4 * t + 1) s -= nmax - 4 * t++ + 1;
    const int n = 4 * t + s, m = 4 * t + (i & 3);
    ab = make_double2(0, 0);
    if (n == m + 1) ab.x = sqrt(2.0 * m + 1);
    else if (n > m) {
        const double den = sqrt((double)(n - m) * (n + m));
        ab.x = (2.0 * n - 1) / den;
        ab.y = sqrt((double)(n + m - 1) * (n - m - 1)) / den;
    }
    return n | t << 16;
}

// Carves the shared memory and copies the tables.
template <int NC>
__device__ __forceinline__ EmmShared emm_init(double *sm, int nmax, const EmmTab &tab)
{
    EmmShared E;
    E.nmax = nmax;
    E.nstep = emm_steps(nmax);
    E.B = sm;
    E.ab = reinterpret_cast<double2 *>(sm + (size_t)E.nstep * 64 * NC);
    E.cm = reinterpret_cast<double *>(E.ab + E.nstep * 4);
    E.step = reinterpret_cast<int *>(E.cm + nmax + 1);
    for (int m = threadIdx.x; m <= nmax; m += blockDim.x) E.cm[m] = tab.cm[m];
    for (int i = threadIdx.x; i < E.nstep * 4; i += blockDim.x) E.ab[i] = tab.ab[i];
    for (int i = threadIdx.x; i < E.nstep; i += blockDim.x) E.step[i] = tab.step[i];
    return E;
}

// Stages the columns of one expansion.  quantity(i, sign, n, mu, v) writes the 4 NC
// coefficients of (n, mu) of every quantity (zero outside the quantity's degrees); i is the
// step and q, sign 1 for negative mu.

template <int NC, class Q>
__device__ __forceinline__ void emm_stage(const EmmShared &E, const Q &quantity)
{
    for (int i = threadIdx.x; i < E.nstep * 4; i += blockDim.x) {
        const int s = i >> 2, q = i & 3, n = E.step[s] & 0xffff, m = 4 * (E.step[s] >> 16) + q;
        double2 u[4 * NC], v[4 * NC];
#pragma unroll
        for (int k = 0; k < 4 * NC; k++) u[k] = v[k] = cmk(0, 0);
        if (m <= n) {
            quantity(i, 0, n, m, u);
            if (m) quantity(i, 1, n, -m, v);
        }
#pragma unroll
        for (int k = 0; k < 4 * NC; k++) {
            // u conj(h) + v h = (u + v) C + i (v - u) S; order 0 has no sine part
            const double2 c = cadd(u[k], v[k]), d = m ? csub(v[k], u[k]) : cmk(0, 0);
            *reinterpret_cast<double2 *>(E.B + emm_col<NC>(s, 0, q, 2 * k)) = c;
            *reinterpret_cast<double2 *>(E.B + emm_col<NC>(s, 1, q, 2 * k)) = cmk(-d.y, d.x);
        }
    }
}

// Harmonics of P points of this lane's row (l / 4) times the staged columns, degrees
// up to nmax <= E.nmax: r[i][c] is quantity 4 c + l % 4 at point i.
template <int NC, int P>
__device__ __forceinline__ void emm_points(const EmmShared &E, bool loc, int nmax, const double (&ux)[P],
                                           const double (&uy)[P], const double (&uz)[P], double2 (&r)[P][NC])
{
    const int lane = threadIdx.x & 31, q = lane & 3, col = lane >> 2;
    double zz[P], rr[P], vx[P], vy[P];
    double2 dg[P];
    double acc[P][NC][2][2];
#pragma unroll
    for (int i = 0; i < P; i++) {
        const double r2 = ux[i] * ux[i] + uy[i] * uy[i] + uz[i] * uz[i], ir2 = loc ? 1.0 : 1.0 / r2;
        zz[i] = loc ? uz[i] : uz[i] * ir2;
        rr[i] = loc ? r2 : ir2;
        vx[i] = -ux[i] * ir2;
        vy[i] = -uy[i] * ir2;
        dg[i] = cmk(loc ? 1.0 : sqrt(ir2), 0.0);
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int k = 0; k < 2; k++) acc[i][c][k][0] = acc[i][c][k][1] = 0;
    }
    auto diag = [&](int m) {
        const double f = m <= E.nmax ? E.cm[m] : 0.0;
#pragma unroll
        for (int i = 0; i < P; i++)
            dg[i] = cmk(f * (vx[i] * dg[i].x + vy[i] * dg[i].y), f * (vx[i] * dg[i].y - vy[i] * dg[i].x));
    };
    for (int m = 1; m <= 3; m++)
        if (m <= q) diag(m);
    int s0 = 0;
    for (int t = 0; 4 * t <= nmax; t++) {
        double2 h0[P], h1[P];
#pragma unroll
        for (int i = 0; i < P; i++) h0[i] = h1[i] = cmk(0, 0);
        const int len = nmax - 4 * t + 1;
        for (int k = 0; k < len; k++) {
            const double2 ab = E.ab[(s0 + k) * 4 + q];
            double b[NC][2];
#pragma unroll
            for (int c = 0; c < NC; c++) {
                b[c][0] = E.B[emm_col<NC>(s0 + k, 0, q, 8 * c + col)];
                b[c][1] = E.B[emm_col<NC>(s0 + k, 1, q, 8 * c + col)];
            }
#pragma unroll
            for (int i = 0; i < P; i++) {
                const double a = ab.x * zz[i], d = ab.y * rr[i];
                double2 h = cmk(fma(a, h0[i].x, -(d * h1[i].x)), fma(a, h0[i].y, -(d * h1[i].y)));
                if (k == q) h = dg[i];
                h1[i] = h0[i];
                h0[i] = h;
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    dmma(acc[i][c][0][0], acc[i][c][0][1], h.x, b[c][0]);
                    dmma(acc[i][c][1][0], acc[i][c][1][1], h.y, b[c][1]);
                }
            }
        }
        s0 += E.nmax - 4 * t + 1;
        if (4 * t + 4 <= nmax)
            for (int k = 1; k <= 4; k++) diag(4 * t + q + k);
    }
#pragma unroll
    for (int i = 0; i < P; i++)
#pragma unroll
        for (int c = 0; c < NC; c++)
            r[i][c] = cmk(acc[i][c][0][0] + acc[i][c][1][0], acc[i][c][0][1] + acc[i][c][1][1]);
}

// Where work item `item` lies: its leaf (position l), chunk of points and group.
__device__ __forceinline__ int emm_leaf(const int *off, int nleaves, int item)
{
    int lo = 0, hi = nleaves - 1;   // the last leaf with off[l] <= item
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= item) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// One work item: leaf, chunk of 128 points (32 per warp, as two pairs of 8-point
// rows) and group of up to 8 expansions.  order(d) is the degree of the harmonics of
// a local expansion (d = 0) or a multipole; scale(side, k) the factor of quantity k;
// quantity(loc, coef, i, sign, n, mu, v) the columns; store(e, k, value) takes the sum of
// quantity k at point e of the leaf.
template <int NC, class Deg, class Scale, class Quant, class Store>
__device__ __forceinline__ void emm_item(double *sm, int nmax, const EmmTab &tab, const TreeView &tv, int b, int grp, int e0, int ne,
                                         int ns, const double *sx, const double *sy, const double *sz,
                                         const double *tx, const double *ty, const double *tz, int K,
                                         const double2 *mpole, const double2 *local, const Deg &degree,
                                         const Scale &scale, const Quant &quantity, const Store &store)
{
    const EmmShared E = emm_init<NC>(sm, nmax, tab);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = lane & 3;
    const int s0 = tv.src0[b], t0 = tv.trg0[b], l3a = tv.l3_start[b];
    const bool has_local = tv.level[b] >= 2;
    const int nbx = eval_nbx(tv, b), ib1 = min(nbx, (grp + 1) * kEvalGroup);
    const int first = e0 + 32 * warp;
    double px[4], py[4], pz[4];
    double2 tot[4][NC];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int e = min(first + 8 * i + (lane >> 2), ne - 1);   // rows past the end repeat the last point
        const bool is_src = e < ns;
        const int j = is_src ? s0 + e : t0 + e - ns;
        px[i] = is_src ? sx[j] : tx[j];
        py[i] = is_src ? sy[j] : ty[j];
        pz[i] = is_src ? sz[j] : tz[j];
#pragma unroll
        for (int c = 0; c < NC; c++) tot[i][c] = cmk(0, 0);
    }
    for (int ib = grp * kEvalGroup; ib < ib1; ib++) {
        const bool loc = has_local && ib == 0;
        const int c = loc ? b : tv.l3_idx[l3a + ib - (has_local ? 1 : 0)];
        const double s = box_side(tv, c), is = 1.0 / s;
        const double2 *coef = (loc ? local : mpole) + (size_t)c * K;
        const double cx = tv.center[3L * c], cy = tv.center[3L * c + 1], cz = tv.center[3L * c + 2];
        __syncthreads();
        emm_stage<NC>(E, [&](int i, int sign, int n, int mu, double2 *v) { quantity(loc, coef, i, sign, n, mu, v); });
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (first + 16 * h >= ne) continue;
            double ux[2], uy[2], uz[2];
            double2 r[2][NC];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                ux[i] = (px[2 * h + i] - cx) * is;
                uy[i] = (py[2 * h + i] - cy) * is;
                uz[i] = (pz[2 * h + i] - cz) * is;
            }
            emm_points<NC, 2>(E, loc, degree(loc), ux, uy, uz, r);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int c2 = 0; c2 < NC; c2++)
                    tot[2 * h + i][c2] = cadd(tot[2 * h + i][c2], cscal(scale(is, 4 * c2 + q), r[i][c2]));
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int e = first + 8 * i + (lane >> 2);
        if (e >= ne) continue;
#pragma unroll
        for (int c = 0; c < NC; c++) store(e, 4 * c + q, tot[i][c]);
    }
}

}  // namespace fmm
