// Laplace FMM kernels, FP64 plain form, for sm_100a.
//
// Solid harmonics are generated by Cartesian recurrences (no trigonometric
// calls): with u = x - i y,
//   R_m^m = -u c_m R_{m-1}^{m-1},   R_{m+1}^m = sqrt(2m+1) z R_m^m,
//   R_n^m = a_nm z R_{n-1}^m - b_nm r^2 R_{n-2}^m,
// where R_n^m = r^n Y_n^m(cos theta) e^{-i m phi}, c_m = sqrt((2m-1)/(2m)),
// a_nm = (2n-1)/sqrt((n-m)(n+m)), b_nm = sqrt((n+m-1)(n-m-1)/((n-m)(n+m))).
// These are the recurrences of ylgndru (src/yrecursion.f:386-430) multiplied
// through by r^n.  The irregular harmonics I_n^m = Y_n^m e^{-i m phi}/r^(n+1)
// follow the same recurrences with z -> z/r^2, r^2 -> 1/r^2, u -> u/r^2.
// Gradients use the ladder identities
//   d/dz R_n^m = sqrt((n-m)(n+m)) R_{n-1}^m,
//   (d/dx + i d/dy) R_n^m = s(m) sqrt((n+m)(n+m-1)) R_{n-1}^{m-1},
//   (d/dx - i d/dy) R_n^m = t(m) sqrt((n-m)(n-m-1)) R_{n-1}^{m+1},
// with s(m) = -1 for m >= 1 else 1 and t(m) = -1 for m <= -1 else 1, and
// R_n^{-m} = conj(R_n^m); and for I_n^m
//   d/dz I_n^m = -sqrt((n+1-m)(n+1+m)) I_{n+1}^m,
//   (d/dx + i d/dy) I_n^m = s(m) sqrt((n-m+1)(n-m+2)) I_{n+1}^{m-1},
//   (d/dx - i d/dy) I_n^m = t(m) sqrt((n+m+1)(n+m+2)) I_{n+1}^{m+1}.
#include <algorithm>
#include <map>
#include <mutex>

#include "eval_mm.cuh"
#include "near.cuh"

namespace fmm {

constexpr int kTabP = 72;                         // largest order with tables
constexpr int kTabN = (kTabP + 2) * (kTabP + 3) / 2;

__constant__ double c_ra[kTabN];   // a_nm at tidx(n,m)
__constant__ double c_rb[kTabN];   // b_nm at tidx(n,m)
__constant__ double c_cm[kTabP + 2];  // c_m
__constant__ double c_sq[kTabP + 2];  // sqrt(2m+1)
// Recurrence factors (a_nm, b_nm) at tidx(n, m), with (sqrt(2m+1), 0) at n = m + 1, in global memory:
// copied to shared memory where every step of a column needs a pair.
__device__ double2 g_rab[kTabN];

void lap_init_constants(Status &st)
{
    static std::mutex mu;  // several host threads may make their first call at once
    std::lock_guard<std::mutex> lk(mu);
    static bool done = false;
    static double ra[kTabN], rb[kTabN], cm[kTabP + 2], sq[kTabP + 2];
    static double2 rab[kTabN];
    if (!done) {
        for (int n = 0; n <= kTabP + 1; n++)
            for (int m = 0; m <= n; m++) {
                double a = 0, b = 0;
                if (n >= m + 2) {
                    double den = sqrt((double)(n - m) * (n + m));
                    a = (2.0 * n - 1) / den;
                    b = sqrt((double)(n + m - 1) * (n - m - 1)) / den;
                }
                ra[tidx(n, m)] = a;
                rb[tidx(n, m)] = b;
            }
        cm[0] = 0;
        for (int m = 1; m <= kTabP + 1; m++) cm[m] = sqrt((2.0 * m - 1) / (2.0 * m));
        for (int m = 0; m <= kTabP + 1; m++) sq[m] = sqrt(2.0 * m + 1);
        for (int n = 0; n <= kTabP + 1; n++)
            for (int m = 0; m <= n; m++)
                rab[tidx(n, m)] = n == m + 1 ? make_double2(sq[m], 0) : make_double2(ra[tidx(n, m)], rb[tidx(n, m)]);
        done = true;
    }
    int dev = 0;
    cudaGetDevice(&dev);
    static bool uploaded[64] = {false};
    if (dev < 64 && uploaded[dev]) return;
    FMM_TRY(st, cudaMemcpyToSymbol(c_ra, ra, sizeof(ra)));
    FMM_TRY(st, cudaMemcpyToSymbol(c_rb, rb, sizeof(rb)));
    FMM_TRY(st, cudaMemcpyToSymbol(c_cm, cm, sizeof(cm)));
    FMM_TRY(st, cudaMemcpyToSymbol(c_sq, sq, sizeof(sq)));
    FMM_TRY(st, cudaMemcpyToSymbol(g_rab, rab, sizeof(rab)));
    if (st.ok() && dev < 64) uploaded[dev] = true;
}

// Regular solid harmonics R_n^m(u), 0 <= m <= n <= p, into out[tidx(n,m)].
__device__ __forceinline__ void regular_table(double x, double y, double z, int p, double2 *out, int stride)
{
    double r2 = x * x + y * y + z * z;
    double2 diag = cmk(1.0, 0.0);
    for (int m = 0; m <= p; m++) {
        if (m > 0) {
            // diag = -(x - i y) * c_m * diag
            double c = -c_cm[m];
            diag = cmk(c * (x * diag.x + y * diag.y), c * (x * diag.y - y * diag.x));
        }
        out[stride * tidx(m, m)] = diag;
        if (m < p) {
            double2 r1 = diag;
            double2 r0 = cscal(c_sq[m] * z, diag);
            out[stride * tidx(m + 1, m)] = r0;
            for (int n = m + 2; n <= p; n++) {
                double a = c_ra[tidx(n, m)] * z, b = c_rb[tidx(n, m)] * r2;
                double2 rn = cmk(a * r0.x - b * r1.x, a * r0.y - b * r1.y);
                out[stride * tidx(n, m)] = rn;
                r1 = r0;
                r0 = rn;
            }
        }
    }
}

// Irregular solid harmonics I_n^m(u), 0 <= m <= n <= p.
__device__ __forceinline__ void irregular_table(double x, double y, double z, int p, double2 *out, int stride)
{
    double r2 = x * x + y * y + z * z;
    double ir2 = 1.0 / r2;
    double zi = z * ir2;
    double2 diag = cmk(sqrt(ir2), 0.0);
    for (int m = 0; m <= p; m++) {
        if (m > 0) {
            double c = -c_cm[m] * ir2;
            diag = cmk(c * (x * diag.x + y * diag.y), c * (x * diag.y - y * diag.x));
        }
        out[stride * tidx(m, m)] = diag;
        if (m < p) {
            double2 r1 = diag;
            double2 r0 = cscal(c_sq[m] * zi, diag);
            out[stride * tidx(m + 1, m)] = r0;
            for (int n = m + 2; n <= p; n++) {
                double a = c_ra[tidx(n, m)] * zi, b = c_rb[tidx(n, m)] * ir2;
                double2 rn = cmk(a * r0.x - b * r1.x, a * r0.y - b * r1.y);
                out[stride * tidx(n, m)] = rn;
                r1 = r0;
                r0 = rn;
            }
        }
    }
}

// value of harmonic (n, m), any sign of m, from a triangular table (0 if |m|>n)
__device__ __forceinline__ double2 tab_get(const double2 *tab, int stride, int n, int m)
{
    if (n < 0 || m > n || -m > n) return cmk(0, 0);
    double2 v = tab[stride * tidx(n, m < 0 ? -m : m)];
    return m < 0 ? cconj(v) : v;
}

// ================================================================ P2P
// Near field of the childless boxes: evaluation points of a box (its sources,
// then its targets) against the sources of the box itself and of its list 1.
// Follows lfmm3dpart_direct_self/_targ (src/lfmm3dpart.f:1175-1385) with the
// pair formulas of lpotfld3d / lpotfld3d_dp (src/laprouts3d.f:1308, 1962).
//
// One warp per (leaf, run of 32 EMAX points), each lane with up to EMAX points;
// 32 sources at a time staged as records in the warp's shared memory.  Bound by
// the FP64 pipe: 35 operations a pair with charges and dipoles, 23 with charges
// (the products -d v are made once per source, the field is summed as
// r^-3 [(q + 3 d t) dx - d v], and 1/r takes five operations), against 49 and 29
// with a thread per point, the library's rsqrt and charge and dipole terms apart:
// 25.2 -> 19.5 ms at the 2M + 2M cube (6.25e9 pairs; 72% of the 17e12 FP64
// operations/s that a loop of independent multiply-adds reaches), 44.1 -> 34.6 ms
// at the 1M + 1M cube at order 26 (1.17e10 pairs).  Loading the next batch into
// registers during the current one, or four points per lane, cost more in
// resident warps than they saved (20.5, 23.9 ms).  All multiply-adds are written
// out, so that every instantiation rounds alike.
constexpr int kP2PThreads = 128;      // direct sums
constexpr int kNearWarps = 2;

// Source record: x, y, z, [q], [d, v, -d v (re), -d v (im)], padded to a stride
// whose 16-byte parts fall into different banks for consecutive sources.
template <bool CHG, bool DIP>
struct NearRec {
    static constexpr int kStride = DIP ? (CHG ? 18 : 14) : 6;
    static constexpr int kQ = 3, kD = CHG ? 5 : 3, kV = kD + 2, kN = kV + 3;
};

template <bool CHG, bool DIP, bool LIB>
__device__ __forceinline__ void near_pair(double dx, double dy, double dz, double qx, double qy, double ddx,
                                          double ddy, double vx, double vy, double vz, const double *nv, double *a,
                                          unsigned &odd)
{
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const double ri = rsqrt_near<LIB>(r2, odd);
    const double ri2 = ri * ri, ri3 = ri * ri2;
    if (!DIP) {
        a[0] = fma(qx, ri, a[0]);
        a[1] = fma(qy, ri, a[1]);
        const double bx = qx * ri3, by = qy * ri3;
        a[2] = fma(bx, dx, a[2]); a[3] = fma(by, dx, a[3]);
        a[4] = fma(bx, dy, a[4]); a[5] = fma(by, dy, a[5]);
        a[6] = fma(bx, dz, a[6]); a[7] = fma(by, dz, a[7]);
    } else {
        // pot = (q + d t) / r with t = (v.dx) / r^2;  fld = [(q + 3 d t) dx - d v] / r^3
        const double t = fma(dx, vx, fma(dy, vy, dz * vz)) * ri2;
        const double ax = CHG ? fma(ddx, t, qx) : ddx * t, ay = CHG ? fma(ddy, t, qy) : ddy * t;
        a[0] = fma(ax, ri, a[0]);
        a[1] = fma(ay, ri, a[1]);
        const double t2 = t + t;
        const double bx = fma(ddx, t2, ax), by = fma(ddy, t2, ay);
        a[2] = fma(ri3, fma(bx, dx, nv[0]), a[2]); a[3] = fma(ri3, fma(by, dx, nv[3]), a[3]);
        a[4] = fma(ri3, fma(bx, dy, nv[1]), a[4]); a[5] = fma(ri3, fma(by, dy, nv[4]), a[5]);
        a[6] = fma(ri3, fma(bx, dz, nv[2]), a[6]); a[7] = fma(ri3, fma(by, dz, nv[5]), a[7]);
    }
}

// cn staged sources at E points of a lane.  OWN: the sources are the points' own
// box; a point's own source (selfk) adds exact zeros (no strength, unit offset).
template <bool CHG, bool DIP, bool LIB, int E, bool OWN, int U>
__device__ __forceinline__ void near_batch(const double *rec, int cn, const double (&px)[E], const double (&py)[E],
                                           const double (&pz)[E], const int (&selfk)[E], double (&acc)[E][8],
                                           unsigned &odd)
{
    using R = NearRec<CHG, DIP>;
    constexpr int W = R::kStride;
#pragma unroll U
    for (int k = 0; k < cn; k++) {
        double r[W];
#pragma unroll
        for (int i = 0; i < W / 2; i++) {
            const double2 v = reinterpret_cast<const double2 *>(rec + k * W)[i];
            r[2 * i] = v.x;
            r[2 * i + 1] = v.y;
        }
#pragma unroll
        for (int e = 0; e < E; e++) {
            double dx = px[e] - r[0], dy = py[e] - r[1], dz = pz[e] - r[2];
            double qx = CHG ? r[R::kQ] : 0, qy = CHG ? r[R::kQ + 1] : 0;
            double ddx = DIP ? r[R::kD] : 0, ddy = DIP ? r[R::kD + 1] : 0;
            if (OWN) {
                const bool me = k == selfk[e];
                dx = me ? 1.0 : dx; dy = me ? 0.0 : dy; dz = me ? 0.0 : dz;
                qx = me ? 0.0 : qx; qy = me ? 0.0 : qy;
                ddx = me ? 0.0 : ddx; ddy = me ? 0.0 : ddy;
                double nv[6], v[3];
#pragma unroll
                for (int i = 0; i < 6; i++) nv[i] = DIP ? (me ? 0.0 : r[R::kN + i]) : 0;
#pragma unroll
                for (int i = 0; i < 3; i++) v[i] = DIP ? (me ? 0.0 : r[R::kV + i]) : 0;
                near_pair<CHG, DIP, LIB>(dx, dy, dz, qx, qy, ddx, ddy, v[0], v[1], v[2], nv, acc[e], odd);
            } else {
                near_pair<CHG, DIP, LIB>(dx, dy, dz, qx, qy, ddx, ddy, DIP ? r[R::kV] : 0, DIP ? r[R::kV + 1] : 0,
                                    DIP ? r[R::kV + 2] : 0, r + (DIP ? R::kN : 0), acc[e], odd);
            }
        }
    }
}

struct NearArgs {
    const int *leaves;
    int nleaves;
    TreeView tv;
    PointsSoA src;
    const double *tx, *ty, *tz;
    OutSoA outs, outt;
    int do_src, do_trg, want_fs, want_ft, want_ps, want_pt;
};

// Points e0 + lane, + 32, ... of leaf b (E per lane).  Returns whether a pair of
// this warp needs the library's rsqrt; nothing is written then (LIB: never).
template <bool CHG, bool DIP, bool LIB, int E, int U>
__device__ __forceinline__ bool near_points(const NearArgs &A, int b, int e0, int ne, int ns, double *rec)
{
    using R = NearRec<CHG, DIP>;
    constexpr int W = R::kStride;
    const int lane = threadIdx.x & 31;
    const int s0 = A.tv.src0[b], t0 = A.tv.trg0[b];
    double px[E], py[E], pz[E], acc[E][8];
    int self[E];
    unsigned odd = 0;
#pragma unroll
    for (int k = 0; k < E; k++) {
        // (lanes past the end repeat the last point; nothing of theirs is written)
        self[k] = -1;
        const int ee = min(e0 + lane + 32 * k, ne - 1);
        if (ee < ns) { const int i = s0 + ee; px[k] = A.src.x[i]; py[k] = A.src.y[i]; pz[k] = A.src.z[i]; self[k] = ee; }
        else { const int i = t0 + ee - ns; px[k] = A.tx[i]; py[k] = A.ty[i]; pz[k] = A.tz[i]; }
#pragma unroll
        for (int i = 0; i < 8; i++) acc[k][i] = 0;
    }
    const int l1a = A.tv.l1_start[b], nl = 1 + A.tv.l1_start[b + 1] - l1a;
    for (int j = 0; j < nl; j++) {
        const int jb = j == 0 ? b : A.tv.l1_idx[l1a + j - 1];
        const int js0 = A.tv.src0[jb], jn = A.tv.nsrc[jb];
        for (int c0 = 0; c0 < jn; c0 += 32) {
            const int cn = min(32, jn - c0);
            __syncwarp();
            if (lane < cn) {
                const int i = js0 + c0 + lane;
                double r[W] = {};
                r[0] = A.src.x[i]; r[1] = A.src.y[i]; r[2] = A.src.z[i];
                if (CHG) { const double2 q = A.src.q[i]; r[R::kQ] = q.x; r[R::kQ + 1] = q.y; }
                if (DIP) {
                    const double2 d = A.src.dq[i];
                    const double v[3] = {A.src.vx[i], A.src.vy[i], A.src.vz[i]};
                    r[R::kD] = d.x; r[R::kD + 1] = d.y;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        r[R::kV + c] = v[c];
                        r[R::kN + c] = -d.x * v[c];
                        r[R::kN + 3 + c] = -d.y * v[c];
                    }
                }
#pragma unroll
                for (int c = 0; c < W / 2; c++)
                    reinterpret_cast<double2 *>(rec + lane * W)[c] = make_double2(r[2 * c], r[2 * c + 1]);
            }
            __syncwarp();
            int selfk[E];
            if (j == 0 && e0 < ns) {
#pragma unroll
                for (int k = 0; k < E; k++) selfk[k] = self[k] < 0 ? -1 : self[k] - c0;
                near_batch<CHG, DIP, LIB, E, true, 1>(rec, cn, px, py, pz, selfk, acc, odd);
            } else {
                near_batch<CHG, DIP, LIB, E, false, U>(rec, cn, px, py, pz, selfk, acc, odd);
            }
        }
    }
    if (!LIB && __any_sync(0xffffffffu, odd > kRsqrtSpan)) return true;
#pragma unroll
    for (int k = 0; k < E; k++) {
        const int e = e0 + lane + 32 * k;
        if (e >= ne) continue;
        const bool is_src = e < ns;
        const int i = is_src ? s0 + e : t0 + e - ns;
        const OutSoA o = is_src ? A.outs : A.outt;
        if (is_src ? A.want_ps : A.want_pt) o.pot[i] = cadd(o.pot[i], cmk(acc[k][0], acc[k][1]));
        if (is_src ? A.want_fs : A.want_ft) {
            o.fx[i] = cadd(o.fx[i], cmk(acc[k][2], acc[k][3]));
            o.fy[i] = cadd(o.fy[i], cmk(acc[k][4], acc[k][5]));
            o.fz[i] = cadd(o.fz[i], cmk(acc[k][6], acc[k][7]));
        }
    }
    return false;
}

template <bool CHG, bool DIP, int E, int U>
__device__ __forceinline__ void near_run(const NearArgs &A, int b, int e0, int ne, int ns, double *rec)
{
    if (near_points<CHG, DIP, false, E, U>(A, b, e0, ne, ns, rec))
        near_points<CHG, DIP, true, E, 1>(A, b, e0, ne, ns, rec);
}

template <bool CHG, bool DIP, int EMAX, int U, int CT>
__global__ void __launch_bounds__(32 * kNearWarps, CT) k_p2p(NearArgs A)
{
    __shared__ __align__(16) double rec[kNearWarps][32 * NearRec<CHG, DIP>::kStride];
    const int warp = threadIdx.x >> 5, li = blockIdx.x * kNearWarps + warp;
    if (li >= A.nleaves) return;
    const int b = A.leaves[li];
    const int ns = A.do_src ? A.tv.nsrc[b] : 0, ne = ns + (A.do_trg ? A.tv.ntrg[b] : 0);
    // runs blockIdx.y, + gridDim.y, ... of the leaf's points (a large leaf of an
    // adaptive tree would otherwise hold the pass's tail alone)
    for (int e0 = blockIdx.y * 32 * EMAX; e0 < ne; e0 += gridDim.y * 32 * EMAX) {
        if (EMAX == 2 && ne - e0 > 32) near_run<CHG, DIP, EMAX, U>(A, b, e0, ne, ns, rec[warp]);
        else near_run<CHG, DIP, 1, U>(A, b, e0, ne, ns, rec[warp]);
    }
}

template <bool CHG, bool DIP>
static void launch_p2p_t(const NearArgs &A, cudaStream_t s, Status &st)
{
    const int ctas = div_up(A.nleaves, kNearWarps);
    // Two points per lane share the staging and the record reads, one gives twice the
    // warps: 2M + 2M cube (32,768 leaves) 19.5 against 20.1 ms, 1M + 1M cube (4,096)
    // 34.6 / 34.9; 100k sphere (1,489) 0.41 / 0.38, 64 leaves 0.13 / 0.08 ms.  The
    // line is the 16 warps a multiprocessor holds, on all of them.
    if (A.nleaves >= 16 * device_sms())
        k_p2p<CHG, DIP, 2, 1, 8><<<dim3(ctas, 4), 32 * kNearWarps, 0, s>>>(A);
    else
        k_p2p<CHG, DIP, 1, 2, 1><<<dim3(ctas, 8), 32 * kNearWarps, 0, s>>>(A);
    FMM_COUNT_LAUNCH();
}

void launch_p2p(const int *leaves, int nleaves, const TreeView &tv, const PointsSoA &src, const double *tx,
                const double *ty, const double *tz, OutSoA outs, OutSoA outt, int ifcharge, int ifdipole,
                int ifpot, int iffld, int ifpottarg, int iffldtarg, cudaStream_t s, Status &st)
{
    if (nleaves == 0 || !st.ok()) return;
    const bool c = ifcharge == 1, d = ifdipole == 1;
    if (!c && !d) return;
    NearArgs A;
    A.leaves = leaves; A.nleaves = nleaves; A.tv = tv; A.src = src; A.tx = tx; A.ty = ty; A.tz = tz;
    A.outs = outs; A.outt = outt;
    A.do_src = ifpot == 1 || iffld == 1; A.do_trg = ifpottarg == 1 || iffldtarg == 1;
    A.want_fs = iffld == 1; A.want_ft = iffldtarg == 1; A.want_ps = ifpot == 1; A.want_pt = ifpottarg == 1;
    if (c && d) launch_p2p_t<true, true>(A, s, st);
    else if (c) launch_p2p_t<true, false>(A, s, st);
    else launch_p2p_t<false, true>(A, s, st);
    FMM_LAUNCH_CHECK(st);
}

// ================================================================ direct sum
// O(N^2) sum of l3dpartdirect (src/lfmm3dpart.f:1391-1523): one evaluation
// point per thread, sources staged through shared memory.
template <bool CHG, bool DIP>
__global__ void __launch_bounds__(kP2PThreads) k_direct(int nsrc, const double *sx_, const double *sy_,
                                                         const double *sz_, const double2 *q_, const double2 *dq_,
                                                         const double *vx_, const double *vy_, const double *vz_,
                                                         int neval, const double *ex_, const double *ey_,
                                                         const double *ez_, const int *skip, int self, OutSoA out,
                                                         int chunk)
{
    __shared__ double sx[kP2PThreads], sy[kP2PThreads], sz[kP2PThreads];
    __shared__ double2 sq[kP2PThreads], sd[kP2PThreads];
    __shared__ double svx[kP2PThreads], svy[kP2PThreads], svz[kP2PThreads];
    int e = blockIdx.x * kP2PThreads + threadIdx.x;
    bool act = e < neval;
    double ex = act ? ex_[e] : 0, ey = act ? ey_[e] : 0, ez = act ? ez_[e] : 0;
    double pr = 0, pi = 0, fxr = 0, fxi = 0, fyr = 0, fyi = 0, fzr = 0, fzi = 0;
    const int cb = blockIdx.y * chunk, ce = min(nsrc, cb + chunk);
    for (int c0 = cb; c0 < ce; c0 += kP2PThreads) {
        int cn = min(kP2PThreads, ce - c0);
        __syncthreads();
        if (threadIdx.x < cn) {
            int i = c0 + threadIdx.x;
            sx[threadIdx.x] = sx_[i]; sy[threadIdx.x] = sy_[i]; sz[threadIdx.x] = sz_[i];
            if (CHG) sq[threadIdx.x] = q_[i];
            if (DIP) { sd[threadIdx.x] = dq_[i]; svx[threadIdx.x] = vx_[i]; svy[threadIdx.x] = vy_[i]; svz[threadIdx.x] = vz_[i]; }
        }
        __syncthreads();
        int selfk = (act && skip) ? skip[e] - c0 : (self ? e - c0 : -1);
        for (int k = 0; k < cn; k++) {
            if (k == selfk) continue;
            double dx = ex - sx[k], dy = ey - sy[k], dz = ez - sz[k];
            double r2 = dx * dx + dy * dy + dz * dz;
            double ri = rsqrt(r2), ri2 = ri * ri, ri3 = ri * ri2;
            if (CHG) {
                double2 q = sq[k];
                pr = fma(q.x, ri, pr); pi = fma(q.y, ri, pi);
                double qx = q.x * ri3, qy = q.y * ri3;
                fxr = fma(qx, dx, fxr); fxi = fma(qy, dx, fxi);
                fyr = fma(qx, dy, fyr); fyi = fma(qy, dy, fyi);
                fzr = fma(qx, dz, fzr); fzi = fma(qy, dz, fzi);
            }
            if (DIP) {
                double2 d = sd[k];
                double dot = dx * svx[k] + dy * svy[k] + dz * svz[k];
                double a = dot * ri3;
                pr = fma(d.x, a, pr); pi = fma(d.y, a, pi);
                double rt = 3.0 * dot * ri3 * ri2;
                double gx = rt * dx - ri3 * svx[k], gy = rt * dy - ri3 * svy[k], gz = rt * dz - ri3 * svz[k];
                fxr = fma(d.x, gx, fxr); fxi = fma(d.y, gx, fxi);
                fyr = fma(d.x, gy, fyr); fyi = fma(d.y, gy, fyi);
                fzr = fma(d.x, gz, fzr); fzi = fma(d.y, gz, fzi);
            }
        }
    }
    if (act) {
        long o = (long)blockIdx.y * neval + e;
        if (out.pot) out.pot[o] = cmk(pr, pi);
        if (out.fx) { out.fx[o] = cmk(fxr, fxi); out.fy[o] = cmk(fyr, fyi); out.fz[o] = cmk(fzr, fzi); }
    }
}

void launch_direct(int nsrc, const double *sx, const double *sy, const double *sz, const double2 *q,
                   const double2 *dq, const double *vx, const double *vy, const double *vz, int ifcharge,
                   int ifdipole, int neval, const double *ex, const double *ey, const double *ez, const int *skip, int self,
                   OutSoA out, cudaStream_t s, Status &st)
{
    if (neval == 0 || !st.ok()) return;
    int g = div_up(neval, kP2PThreads);
    bool c = ifcharge == 1, d = ifdipole == 1;
    if (c && d) { k_direct<true, true><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, self, out, nsrc); FMM_COUNT_LAUNCH(); }
    else if (c) { k_direct<true, false><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, self, out, nsrc); FMM_COUNT_LAUNCH(); }
    else if (d) { k_direct<false, true><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, self, out, nsrc); FMM_COUNT_LAUNCH(); }
    else { k_direct<false, false><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, self, out, nsrc); FMM_COUNT_LAUNCH(); }
    FMM_LAUNCH_CHECK(st);
}

// Direct sum for few evaluation points: the sources are split into chunks
// over gridDim.y, each chunk writes its partial sums, and k_direct_reduce adds
// the chunks in a fixed order (deterministic).  partial holds 4 x nchunk x neval.
__global__ void k_direct_reduce(int neval, int nchunk, OutSoA part, OutSoA out)
{
    int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= neval) return;
    double2 p = cmk(0, 0), a = cmk(0, 0), b = cmk(0, 0), c = cmk(0, 0);
    for (int k = 0; k < nchunk; k++) {
        long o = (long)k * neval + e;
        p = cadd(p, part.pot[o]); a = cadd(a, part.fx[o]); b = cadd(b, part.fy[o]); c = cadd(c, part.fz[o]);
    }
    out.pot[e] = p; out.fx[e] = a; out.fy[e] = b; out.fz[e] = c;
}

void launch_direct_split(int nsrc, const double *sx, const double *sy, const double *sz, const double2 *q,
                         const double2 *dq, const double *vx, const double *vy, const double *vz, int ifcharge,
                         int ifdipole, int neval, const double *ex, const double *ey, const double *ez,
                         const int *skip, OutSoA out, cudaStream_t s, Status &st)
{
    if (neval == 0 || !st.ok()) return;
    int gx = div_up(neval, kP2PThreads);
    int nchunk = std::max(1, std::min(div_up(4 * device_sms(), gx), div_up(nsrc, 4096)));
    int chunk = div_up(nsrc, nchunk);
    nchunk = div_up(nsrc, chunk);
    DBuf<double2> part;
    if (!part.alloc((size_t)4 * nchunk * neval, s, st)) return;
    OutSoA P;
    P.pot = part.p; P.fx = part.p + (size_t)nchunk * neval; P.fy = P.fx + (size_t)nchunk * neval;
    P.fz = P.fy + (size_t)nchunk * neval;
    dim3 g(gx, nchunk);
    bool c = ifcharge == 1, d = ifdipole == 1;
    if (c && d) { k_direct<true, true><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, 0, P, chunk); FMM_COUNT_LAUNCH(); }
    else if (c) { k_direct<true, false><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, 0, P, chunk); FMM_COUNT_LAUNCH(); }
    else if (d) { k_direct<false, true><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, 0, P, chunk); FMM_COUNT_LAUNCH(); }
    else { k_direct<false, false><<<g, kP2PThreads, 0, s>>>(nsrc, sx, sy, sz, q, dq, vx, vy, vz, neval, ex, ey, ez, skip, 0, P, chunk); FMM_COUNT_LAUNCH(); }
    k_direct_reduce<<<div_up(neval, 256), 256, 0, s>>>(neval, nchunk, P, out); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
}

// ================================================================ P2M / P2L
// Expansion formation for one box per CTA.  The sources (the box's own for
// P2M, those of all its list-4 boxes for P2L, concatenated) are processed in
// chunks of C points.  Table phase: the 128 threads split the chunk as
// (point, column group) and write the harmonic table in shared memory with
// a row stride of C + 1 entries, so the rows read together in the next
// phase fall into distinct banks.  Accumulation phase: one thread per
// (degree n, order |m|) pair accumulates both coefficients (n, m) and
// (n, -m) from one table read.
// P2M follows l3dformmp_trunc0 / l3dformmp0_dp_trunc (src/laprouts3d.f:3348,
// 3970); P2L (list 4) follows l3dformta_trunc0 / l3dformta0_dp_trunc
// (src/laprouts3d.f:3689, 4355).
constexpr int kFormThreads = 128;
constexpr int kFormWin = 256;  // source boxes per prefix window

// Directional-derivative weights of the harmonic (n, m) (signed m): the
// derivative along v of R_n^m (P2M) or I_n^m (P2L) is
// vz cz h(nn, m) + (vx - i vy)/2 cp h(nn, m-1) + (vx + i vy)/2 cm h(nn, m+1).
template <bool IRREG>
__device__ __forceinline__ void dip_weights(int n, int m, double &cz, double &cp, double &cm)
{
    if (!IRREG) {
        cz = sqrt((double)(n - m) * (n + m));
        cp = (m >= 1 ? -1.0 : 1.0) * sqrt((double)(n + m) * (n + m - 1));
        cm = (m <= -1 ? -1.0 : 1.0) * sqrt((double)(n - m) * (n - m - 1));
    } else {
        cz = -sqrt((double)(n + 1 - m) * (n + 1 + m));
        cp = (m >= 1 ? -1.0 : 1.0) * sqrt((double)(n - m + 1) * (n - m + 2));
        cm = (m <= -1 ? -1.0 : 1.0) * sqrt((double)(n + m + 1) * (n + m + 2));
    }
}

// Column m (degrees m..pt) of the regular or irregular harmonic table.
template <bool IRREG>
__device__ __forceinline__ void table_column(double x, double y, double z, int pt, int m, double2 diag,
                                             double2 *out, int S)
{
    const double r2 = x * x + y * y + z * z;
    const double ir2 = IRREG ? 1.0 / r2 : 0.0, zz = IRREG ? z * ir2 : z, rr = IRREG ? ir2 : r2;
    out[S * tidx(m, m)] = diag;
    if (m < pt) {
        double2 r1 = diag;
        double2 r0 = cscal(c_sq[m] * zz, diag);
        out[S * tidx(m + 1, m)] = r0;
        for (int n = m + 2; n <= pt; n++) {
            double a = c_ra[tidx(n, m)] * zz, bb = c_rb[tidx(n, m)] * rr;
            double2 rn = cmk(a * r0.x - bb * r1.x, a * r0.y - bb * r1.y);
            out[S * tidx(n, m)] = rn;
            r1 = r0;
            r0 = rn;
        }
    }
}

template <bool IRREG, int NPK>
__global__ void __launch_bounds__(kFormThreads) k_form(const int *boxes, const int *l4s, const int *l4i,
                                                       TreeView tv, PointsSoA src, int ifcharge, int ifdipole,
                                                       int p, int C, double2 *coef)
{
    extern __shared__ double2 smem[];
    const int pt = IRREG ? p + 1 : p;         // table degree (one more for dipole gradients of I)
    const int ntab = (pt + 1) * (pt + 2) / 2;
    const int S = C + 1;
    double2 *tab = smem;                       // [ntab][S] (point fastest)
    double2 *qs = tab + (size_t)ntab * S;      // [C] charges
    double2 *dA = qs + C;                      // [C] d vz           (dipole strength d, direction v)
    double2 *dM = dA + C;                      // [C] d (vx - i vy) / 2
    double2 *dP = dM + C;                      // [C] d (vx + i vy) / 2
    int *pre = (int *)(dP + C);                // [kFormWin + 1]
    const int b = boxes[blockIdx.x];
    const int nsb = IRREG ? l4s[b + 1] - l4s[b] : 1;
    if (IRREG && nsb == 0) return;
    const double s = box_side(tv, b), is = 1.0 / s;
    const double cx = tv.center[3L * b], cy = tv.center[3L * b + 1], cz = tv.center[3L * b + 2];
    const int npair = (p + 1) * (p + 2) / 2;
    const int G = kFormThreads / C, j = threadIdx.x % C, g = threadIdx.x / C;
    int pn[NPK], pm[NPK];
    double2 ap[NPK], am[NPK];
#pragma unroll
    for (int k = 0; k < NPK; k++) {
        int u = threadIdx.x + k * kFormThreads, n = 0;
        while ((n + 1) * (n + 2) / 2 <= u) n++;
        pn[k] = n;
        pm[k] = u - n * (n + 1) / 2;
        ap[k] = cmk(0, 0);
        am[k] = cmk(0, 0);
    }
    for (int w0 = 0; w0 < nsb; w0 += kFormWin) {
        const int nw = min(kFormWin, nsb - w0);
        __syncthreads();
        if (threadIdx.x < 32) {
            int run = 0;
            if (threadIdx.x == 0) pre[0] = 0;
            for (int g0 = 0; g0 < nw; g0 += 32) {
                int k = g0 + threadIdx.x, c = 0;
                if (k < nw) c = tv.nsrc[IRREG ? l4i[l4s[b] + w0 + k] : b];
                int v = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    int t = __shfl_up_sync(0xffffffffu, v, o);
                    if (threadIdx.x >= o) v += t;
                }
                if (k < nw) pre[k + 1] = run + v;
                run += __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        const int total = pre[nw];
        for (int c0 = 0; c0 < total; c0 += C) {
            const int cn = min(C, total - c0);
            __syncthreads();
            if (j < cn) {
                // the source of concatenated position c0 + j: last window box with pre[k] <= pos
                const int pos = c0 + j;
                int lo = 0, hi = nw - 1;
                while (lo < hi) {
                    int mid = (lo + hi + 1) >> 1;
                    if (pre[mid] <= pos) lo = mid;
                    else hi = mid - 1;
                }
                const int jb = IRREG ? l4i[l4s[b] + w0 + lo] : b;
                const int i = tv.src0[jb] + pos - pre[lo];
                const double ux = (src.x[i] - cx) * is, uy = (src.y[i] - cy) * is, uz = (src.z[i] - cz) * is;
                if (g == 0) {
                    qs[j] = ifcharge == 1 ? src.q[i] : cmk(0, 0);
                    if (ifdipole == 1) {
                        const double2 dq = cscal(is, src.dq[i]);
                        const double vx = src.vx[i], vy = src.vy[i], vz = src.vz[i];
                        dA[j] = cscal(vz, dq);
                        dM[j] = cscal(0.5, cmul(dq, cmk(vx, -vy)));
                        dP[j] = cscal(0.5, cmul(dq, cmk(vx, vy)));
                    }
                }
                const double ir2 = IRREG ? 1.0 / (ux * ux + uy * uy + uz * uz) : 1.0;
                double2 diag = cmk(IRREG ? sqrt(ir2) : 1.0, 0.0);
                for (int m = 0; m <= pt; m++) {
                    if (m > 0) {
                        double cc = -c_cm[m] * ir2;
                        diag = cmk(cc * (ux * diag.x + uy * diag.y), cc * (ux * diag.y - uy * diag.x));
                    }
                    if (m % G == g) table_column<IRREG>(ux, uy, uz, pt, m, diag, tab + j, S);
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NPK; k++) {
                const int n = pn[k], mm = pm[k];
                if (n > p) continue;
                double2 a1 = ap[k], a2 = am[k];
                if (ifcharge == 1) {
                    // four real sums give both coefficients: q h = (c0 - c1, c2 + c3),
                    // q conj(h) = (c0 + c1, c3 - c2)
                    const double2 *tp = tab + (size_t)S * tidx(n, mm);
                    double c0 = 0, c1 = 0, c2 = 0, c3 = 0;
#pragma unroll 4
                    for (int jj = 0; jj < cn; jj++) {
                        const double2 t = tp[jj], q = qs[jj];
                        c0 = fma(q.x, t.x, c0);
                        c1 = fma(q.y, t.y, c1);
                        c2 = fma(q.x, t.y, c2);
                        c3 = fma(q.y, t.x, c3);
                    }
                    a1 = cadd(a1, cmk(c0 - c1, c2 + c3));
                    a2 = cadd(a2, cmk(c0 + c1, c3 - c2));
                }
                if (ifdipole == 1) {
                    const int nn = IRREG ? n + 1 : n - 1;
                    double zp, pp, mp, zm, pm_, mm_;
                    dip_weights<IRREG>(n, mm, zp, pp, mp);
                    dip_weights<IRREG>(n, -mm, zm, pm_, mm_);
                    // table entries of degree nn at orders mm - 1, mm, mm + 1 (0 outside the table)
                    const bool okn = nn >= 0;
                    const bool o0 = okn && mm <= nn, o1 = okn && mm + 1 <= nn, om = okn && mm >= 1 && mm - 1 <= nn;
                    const double2 *r0 = tab + (size_t)S * (o0 ? tidx(nn, mm) : 0);
                    const double2 *r1 = tab + (size_t)S * (o1 ? tidx(nn, mm + 1) : 0);
                    const double2 *rm = tab + (size_t)S * (om ? tidx(nn, mm - 1) : 0);
                    // the weights depend on (n, mm) only, so the chunk's sums over the
                    // sources are formed per harmonic and weighted once:
                    //   order +mm: zp sum A h(nn, mm) + pp sum M h(nn, mm - 1) + mp sum P h(nn, mm + 1)
                    //   order -mm: zm sum A h(nn, -mm) + pm sum M h(nn, -mm - 1) + mm sum P h(nn, -mm + 1)
                    double2 s0 = cmk(0, 0), s1 = s0, s2 = s0, s3 = s0, s4 = s0, s5 = s0;
                    for (int jj = 0; jj < cn; jj++) {
                        const double2 E0 = o0 ? r0[jj] : cmk(0, 0), E1 = o1 ? r1[jj] : cmk(0, 0);
                        const double2 Em = om ? rm[jj] : cmk(0, 0);
                        const double2 A = dA[jj], M = dM[jj], P = dP[jj];
                        const double2 hpp = mm >= 1 ? Em : cconj(E1);
                        cfma(s0, A, E0);
                        cfma(s1, M, hpp);
                        cfma(s2, P, E1);
                        if (mm > 0) {
                            const double2 hmm = mm >= 2 ? cconj(Em) : Em;
                            cfma(s3, A, cconj(E0));
                            cfma(s4, M, cconj(E1));
                            cfma(s5, P, hmm);
                        }
                    }
                    a1 = cadd(a1, cadd(cadd(cscal(zp, s0), cscal(pp, s1)), cscal(mp, s2)));
                    if (mm > 0) a2 = cadd(a2, cadd(cadd(cscal(zm, s3), cscal(pm_, s4)), cscal(mm_, s5)));
                }
                ap[k] = a1;
                am[k] = a2;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NPK; k++) {
        const int n = pn[k], mm = pm[k];
        if (n > p) continue;
        double2 *out = coef + (size_t)b * (p + 1) * (p + 1);
        const int ep = eidx(n, mm), em = eidx(n, -mm);
        if (IRREG) {
            out[ep] = cadd(out[ep], ap[k]);
            if (mm > 0) out[em] = cadd(out[em], am[k]);
        } else {
            out[ep] = ap[k];
            if (mm > 0) out[em] = am[k];
        }
    }
}

static int form_chunk(int pt)
{
    const size_t ntab = (size_t)(pt + 1) * (pt + 2) / 2;
    for (int c = 32; c >= 1; c >>= 1) {
        size_t need = ntab * (c + 1) * 16 + (size_t)c * 64 + (kFormWin + 1) * 4;
        if (need <= (c == 32 ? 100u * 1024 : 200u * 1024)) return c;
    }
    return 1;
}

static size_t form_smem(int pt, int C)
{
    const size_t ntab = (size_t)(pt + 1) * (pt + 2) / 2;
    return ntab * (C + 1) * 16 + (size_t)C * 64 + (kFormWin + 1) * 4;
}

template <bool IRREG, int NPK>
static void launch_form_t(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge,
                          int ifdipole, int p, double2 *coef, cudaStream_t s, Status &st)
{
    const int pt = IRREG ? p + 1 : p;
    const int C = form_chunk(pt);
    const size_t sm = form_smem(pt, C);
    FMM_TRY(st, smem_allow(k_form<IRREG, NPK>, (int)sm));
    k_form<IRREG, NPK><<<nboxes, kFormThreads, sm, s>>>(boxes, IRREG ? tv.l4_start : nullptr,
                                                        IRREG ? tv.l4_idx : nullptr, tv, src, ifcharge, ifdipole,
                                                        p, C, coef); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
}

// ---------------------------------------------------------------- dipoles: in matrix products
// With dipoles every harmonic h = C + iS meets four complex weights of a source:
// q, d vz, d vx and d vy (the ladder identities turn the derivative along v into
// harmonics of degree n +- 1 with weights of the degree and order alone, applied
// once to the sums).  The sums of all real harmonics with the 8 real weights are
// one (harmonics x sources) (sources x 8) product, an exact fit for the 8 columns
// of the FP64 MMA.  Per chunk of C sources the CTA writes the table of real
// harmonics in shared memory (row n^2, then n^2 + 2m - 1 and n^2 + 2m for the
// cosine and sine parts of (n, m); row stride = 4 mod 16 doubles, so the 4 x 4
// lanes of a half warp reading a fragment meet different banks), then each warp
// multiplies its 8-row blocks, whose sums stay in its accumulators.  Bound by the
// FP64 pipe: about 0.9 k operations for the table and 2 k in MMAs a source at order
// 14, against 4.6 k with one thread per (n, m).
template <int C>
constexpr int kFmmLd = C + 4;
constexpr int kFmmLdw = 12;   // row stride of the weights, = 12 mod 16

template <bool IRREG, int NW, int C, int TPW, int CTAS>
__global__ void __launch_bounds__(32 * NW, CTAS) k_form_mm(const int *boxes, const int *l4s, const int *l4i, TreeView tv,
                                                        PointsSoA src, int ifcharge, int p, double2 *coef)
{
    constexpr int S = kFmmLd<C>, NT = 32 * NW, G = NT / C;
    extern __shared__ double fsm[];
    const int pt = IRREG ? p + 1 : p;                 // table degree
    const int rows = (pt + 1) * (pt + 1), ntile = (rows + 7) / 8, ntri = (pt + 1) * (pt + 2) / 2;
    double *tab = fsm;                                // [8 ntile][S]
    double2 *ab = reinterpret_cast<double2 *>(tab + (size_t)8 * ntile * S);   // recurrence factors
    double *wt = reinterpret_cast<double *>(ab + ntri);                       // [C][kFmmLdw]
    int *pre = (int *)(wt + C * kFmmLdw);             // [kFormWin + 1]
    const int b = boxes[blockIdx.x];
    const int nsb = IRREG ? l4s[b + 1] - l4s[b] : 1;
    if (IRREG && nsb == 0) return;
    if (!IRREG && tv.nsrc[b] == 0) return;            // the coefficients are zero already
    const double s = box_side(tv, b), is = 1.0 / s;
    const double cx = tv.center[3L * b], cy = tv.center[3L * b + 1], cz = tv.center[3L * b + 2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j = tid % C, g = tid / C;
    double acc[TPW][2];
#pragma unroll
    for (int i = 0; i < TPW; i++) acc[i][0] = acc[i][1] = 0;
    for (int i = rows * S + tid; i < 8 * ntile * S; i += NT) tab[i] = 0;
    for (int i = tid; i < ntri; i += NT) ab[i] = g_rab[i];
    for (int w0 = 0; w0 < nsb; w0 += kFormWin) {
        const int nw = min(kFormWin, nsb - w0);
        __syncthreads();
        if (tid < 32) {
            int run = 0;
            if (tid == 0) pre[0] = 0;
            for (int g0 = 0; g0 < nw; g0 += 32) {
                const int k = g0 + tid;
                int v = k < nw ? tv.nsrc[IRREG ? l4i[l4s[b] + w0 + k] : b] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, v, o);
                    if (tid >= o) v += t;
                }
                if (k < nw) pre[k + 1] = run + v;
                run += __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        const int total = pre[nw];
        // the chunk's source of this thread: of concatenated position c0 + j, in the last window
        // box with pre[k] <= pos (positions that fill the last K step repeat the last
        // source, without weight); the next chunk's is read while this one is multiplied
        double sx = 0, sy = 0, sz = 0, v[3] = {0, 0, 0};
        double2 q = cmk(0, 0), d = cmk(0, 0);
        auto fetch = [&](int c0) {
            const int cn = min(C, total - c0);
            if (cn <= 0 || j >= ((cn + 3) & ~3)) return;
            const int pos = c0 + min(j, cn - 1);
            int lo = 0, hi = nw - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (pre[mid] <= pos) lo = mid;
                else hi = mid - 1;
            }
            const int jb = IRREG ? l4i[l4s[b] + w0 + lo] : b;
            const int i = tv.src0[jb] + pos - pre[lo];
            sx = src.x[i]; sy = src.y[i]; sz = src.z[i];
            if (g == 0) {
                q = ifcharge == 1 ? src.q[i] : cmk(0, 0);
                d = src.dq[i];
                v[0] = src.vz[i]; v[1] = src.vx[i]; v[2] = src.vy[i];
            }
        };
        fetch(0);
        for (int c0 = 0; c0 < total; c0 += C) {
            const int cn = min(C, total - c0);
            __syncthreads();
            if (j < ((cn + 3) & ~3)) {
                const double ux = (sx - cx) * is, uy = (sy - cy) * is, uz = (sz - cz) * is;
                if (g == 0) {
                    double *w = wt + j * kFmmLdw;
                    const bool in = j < cn;
                    w[0] = in ? q.x : 0; w[1] = in ? q.y : 0;
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        w[2 + 2 * k] = in ? is * d.x * v[k] : 0;
                        w[3 + 2 * k] = in ? is * d.y * v[k] : 0;
                    }
                }
                const double r2 = ux * ux + uy * uy + uz * uz;
                const double ir2 = IRREG ? 1.0 / r2 : 1.0;
                const double zz = IRREG ? uz * ir2 : uz, rr = IRREG ? ir2 : r2;
                double2 diag = cmk(IRREG ? sqrt(ir2) : 1.0, 0.0);
                for (int m = 0; m <= pt; m++) {
                    if (m > 0) {
                        const double cc = -c_cm[m] * ir2;
                        diag = cmk(cc * (ux * diag.x + uy * diag.y), cc * (ux * diag.y - uy * diag.x));
                    }
                    // (columns dealt back and forth: a long one and a short one for each thread)
                    if ((m / G & 1 ? G - 1 - m % G : m % G) != g) continue;
                    double2 h0 = diag, h1 = cmk(0, 0);
                    double *t = tab + (size_t)(m ? m * m + 2 * m - 1 : 0) * S + j;
                    t[0] = h0.x;
                    if (m) t[S] = h0.y;
                    int at = tidx(m, m);
#pragma unroll 2
                    for (int n = m + 1; n <= pt; n++) {
                        at += n;                      // tidx(n, m)
                        t += (2 * n - 1) * S;         // row n^2 + ...
                        const double2 f = ab[at];
                        const double a = f.x * zz, bb = f.y * rr;
                        const double2 h = cmk(a * h0.x - bb * h1.x, a * h0.y - bb * h1.y);
                        h1 = h0;
                        h0 = h;
                        t[0] = h.x;
                        if (m) t[S] = h.y;
                    }
                }
            }
            __syncthreads();
            fetch(c0 + C);
            double bf[C / 4];
#pragma unroll
            for (int ks = 0; ks < C / 4; ks++) bf[ks] = 4 * ks < cn ? wt[(4 * ks + (lane & 3)) * kFmmLdw + (lane >> 2)] : 0;
#pragma unroll
            for (int i = 0; i < TPW; i++) {
                const int t = warp + NW * i;
                if (t >= ntile) continue;
                const double *ta = tab + (size_t)(8 * t + (lane >> 2)) * S + (lane & 3);
#pragma unroll
                for (int ks = 0; ks < C / 4; ks++)
                    if (4 * ks < cn) dmma(acc[i][0], acc[i][1], ta[4 * ks], bf[ks]);
            }
        }
    }
    // sums of row r with weight k (0: q, 1: d vz, 2: d vx, 3: d vy)
    __syncthreads();
    double2 *sum = reinterpret_cast<double2 *>(fsm);
#pragma unroll
    for (int i = 0; i < TPW; i++) {
        const int t = warp + NW * i;
        if (t < ntile) sum[(8 * t + (lane >> 2)) * 4 + (lane & 3)] = cmk(acc[i][0], acc[i][1]);
    }
    __syncthreads();
    // cosine and sine sums of (n, m) with weight k; the sums of M = d (vx - i vy) / 2 and
    // P = d (vx + i vy) / 2 follow from those of d vx and d vy
    auto cs = [&](int n, int m, int k, double2 &c, double2 &sn) {
        c = cmk(0, 0);
        sn = cmk(0, 0);
        if (n < 0 || m > n || m < 0) return;
        c = sum[(m ? n * n + 2 * m - 1 : n * n) * 4 + k];
        if (m) sn = sum[(n * n + 2 * m) * 4 + k];
    };
    auto weighted = [&](int n, int m, int k, bool conj) {   // k: 1 A, 2 M, 3 P; sum of the weight times h or conj(h)
        double2 c, sn;
        if (k == 1) cs(n, m, 1, c, sn);
        else {
            double2 xc, xs, yc, ys;
            cs(n, m, 2, xc, xs);
            cs(n, m, 3, yc, ys);
            const double f = k == 2 ? 0.5 : -0.5;   // M: (x - i y) / 2, P: (x + i y) / 2
            c = cmk(0.5 * xc.x + f * yc.y, 0.5 * xc.y - f * yc.x);
            sn = cmk(0.5 * xs.x + f * ys.y, 0.5 * xs.y - f * ys.x);
        }
        return conj ? cmk(c.x + sn.y, c.y - sn.x) : cmk(c.x - sn.y, c.y + sn.x);
    };
    const int npair = (p + 1) * (p + 2) / 2;
    double2 *out = coef + (size_t)b * (p + 1) * (p + 1);
    for (int u = tid; u < npair; u += NT) {
        int n = (int)((sqrtf(8.0f * u + 1.0f) - 1.0f) * 0.5f);
        while (n * (n + 1) / 2 > u) n--;
        while ((n + 1) * (n + 2) / 2 <= u) n++;
        const int mm = u - n * (n + 1) / 2;
        double2 a1, a2;
        {
            double2 c, sn;
            cs(n, mm, 0, c, sn);
            a1 = cmk(c.x - sn.y, c.y + sn.x);
            a2 = cmk(c.x + sn.y, c.y - sn.x);
        }
        const int nn = IRREG ? n + 1 : n - 1;
        double z, pp, mp;
        dip_weights<IRREG>(n, mm, z, pp, mp);
        a1 = cadd(a1, cadd(cadd(cscal(z, weighted(nn, mm, 1, false)),
                                cscal(pp, mm >= 1 ? weighted(nn, mm - 1, 2, false) : weighted(nn, 1, 2, true))),
                           cscal(mp, weighted(nn, mm + 1, 3, false))));
        if (mm > 0) {
            dip_weights<IRREG>(n, -mm, z, pp, mp);
            a2 = cadd(a2, cadd(cadd(cscal(z, weighted(nn, mm, 1, true)), cscal(pp, weighted(nn, mm + 1, 2, true))),
                               cscal(mp, weighted(nn, mm - 1, 3, mm >= 2))));
        }
        const int ep = eidx(n, mm), em = eidx(n, -mm);
        if (IRREG) {
            out[ep] = cadd(out[ep], a1);
            if (mm > 0) out[em] = cadd(out[em], a2);
        } else {
            out[ep] = a1;
            if (mm > 0) out[em] = a2;
        }
    }
}

template <bool IRREG, int NW, int C, int TPW, int CTAS>
static void launch_form_mm(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge, int p,
                           double2 *coef, cudaStream_t s, Status &st)
{
    const int pt = IRREG ? p + 1 : p, ntile = ((pt + 1) * (pt + 1) + 7) / 8;
    const size_t sm = sizeof(double) * ((size_t)8 * ntile * kFmmLd<C> + (pt + 1) * (pt + 2) + C * kFmmLdw) + sizeof(int) * (kFormWin + 1);
    FMM_TRY(st, smem_allow(k_form_mm<IRREG, NW, C, TPW, CTAS>, sm));
    k_form_mm<IRREG, NW, C, TPW, CTAS><<<nboxes, 32 * NW, sm, s>>>(boxes, IRREG ? tv.l4_start : nullptr,
                                                             IRREG ? tv.l4_idx : nullptr, tv, src, ifcharge, p,
                                                             coef); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
}

// Dipoles up to order 28 (table degree 29: 113 blocks of 8 harmonics).  32 sources a
// chunk while three CTAs fit an SM, then 16 with twice the warps.
template <bool IRREG>
static bool form_mm(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge, int p,
                    double2 *coef, cudaStream_t s, Status &st)
{
    const int pt = IRREG ? p + 1 : p, ntile = ((pt + 1) * (pt + 1) + 7) / 8;
    if (pt > 29) return false;
    if (ntile <= 16) launch_form_mm<IRREG, 4, 32, 4, 4>(boxes, nboxes, tv, src, ifcharge, p, coef, s, st);
    else if (ntile <= 32) launch_form_mm<IRREG, 8, 32, 4, 2>(boxes, nboxes, tv, src, ifcharge, p, coef, s, st);
    else launch_form_mm<IRREG, 16, 16, 8, 1>(boxes, nboxes, tv, src, ifcharge, p, coef, s, st);
    return true;
}

template <bool IRREG>
static void launch_form(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge,
                        int ifdipole, int p, double2 *coef, cudaStream_t s, Status &st)
{
    if (nboxes == 0 || !st.ok()) return;
    if (ifdipole == 1 && form_mm<IRREG>(boxes, nboxes, tv, src, ifcharge, p, coef, s, st)) return;
    const int npair = (p + 1) * (p + 2) / 2;
    if (npair <= kFormThreads) launch_form_t<IRREG, 1>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, coef, s, st);
    else if (npair <= 2 * kFormThreads) launch_form_t<IRREG, 2>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, coef, s, st);
    else if (npair <= 4 * kFormThreads) launch_form_t<IRREG, 4>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, coef, s, st);
    else if (npair <= 8 * kFormThreads) launch_form_t<IRREG, 8>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, coef, s, st);
    else launch_form_t<IRREG, ((kTabP + 1) * (kTabP + 2) / 2 + kFormThreads - 1) / kFormThreads>(
        boxes, nboxes, tv, src, ifcharge, ifdipole, p, coef, s, st);
}

void launch_p2m(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge,
                int ifdipole, int p, double2 *mpole, cudaStream_t s, Status &st)
{
    launch_form<false>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, mpole, s, st);
}

void launch_p2l(const int *boxes, int nboxes, const TreeView &tv, const PointsSoA &src, int ifcharge,
                int ifdipole, int p, double2 *local, cudaStream_t s, Status &st)
{
    launch_form<true>(boxes, nboxes, tv, src, ifcharge, ifdipole, p, local, s, st);
}

// ================================================================ L2P + M2P
// Far field at the evaluation points of one childless box per CTA: its
// local expansion (levels >= 2; l3dtaeval_trunc0, src/laprouts3d.f:2941)
// plus the multipoles of its list-3 boxes (l3dmpeval_trunc0,
// src/laprouts3d.f:2606).  The potential and the three gradient components
// are four dot products of coefficient arrays (in shared memory) with the
// harmonics of the point, generated on the fly.  Adds to the outputs (the
// near field is summed into them first, concurrently with the far field).
// MASK selects the sums that a call feeds: bit 0 the potential (A), bit 1 the
// z-gradient (Gz), bit 2 the two transverse gradients (Gp, Gm).
template <int MASK>
__device__ __forceinline__ void dot4_acc(double2 h, int n, int m, const double2 *A, const double2 *Gz,
                                         const double2 *Gp, const double2 *Gm, int ng_lo, int ng_hi, double2 &phi,
                                         double2 &dz, double2 &dp, double2 &dm)
{
    // contributions of R or I (n, +-m) with coefficient arrays indexed by
    // the conjugate partner: value(n,-m) pairs with coefficient (n, m)
    double2 hc = cconj(h);
    int ip = eidx(n, m), im = eidx(n, -m);
    if ((MASK & 1) && A) {
        cfma(phi, A[ip], hc);
        if (m > 0) cfma(phi, A[im], h);
    }
    if ((MASK & 6) && n >= ng_lo && n <= ng_hi) {
        int o = ng_lo == 1 ? -1 : 0;  // gradient arrays start at degree 1 for multipoles
        int gp = eidx(n, m) + (o ? -1 : 0), gm = eidx(n, -m) + (o ? -1 : 0);
        if (MASK & 2) cfma(dz, Gz[gp], hc);
        if (MASK & 4) {
            cfma(dp, Gp[gp], hc);
            cfma(dm, Gm[gp], hc);
        }
        if (m > 0) {
            if (MASK & 2) cfma(dz, Gz[gm], h);
            if (MASK & 4) {
                cfma(dp, Gp[gm], h);
                cfma(dm, Gm[gm], h);
            }
        }
    }
}

// Gradient coefficient arrays of a local expansion (degrees 0..p-1, index
// eidx(k, mu)) or of a multipole (degrees 1..p+1, index eidx(k, mu) - 1),
// from its coefficients C (shared or global memory).  WHICH bit 1: Gz,
// bit 2: Gp and Gm.
template <int WHICH>
__device__ __forceinline__ void stage_grad(bool loc, int p, const double2 *C, double2 *Gz, double2 *Gp, double2 *Gm)
{
    const int K1 = (p + 2) * (p + 2);
    if (loc) {
        for (int i = threadIdx.x; i < p * p; i += kEvalThreads) {
            int k = (int)sqrtf((float)i);
            while (k * k > i) k--;
            while ((k + 1) * (k + 1) <= i) k++;
            int mu = i - k * k - k;
            if (WHICH & 2) Gz[i] = cscal(sqrt((double)(k + 1 + mu) * (k + 1 - mu)), C[eidx(k + 1, mu)]);
            if (WHICH & 4) {
                Gp[i] = cscal((mu <= 0 ? -1.0 : 1.0) * sqrt((double)(k + 2 - mu) * (k + 1 - mu)), C[eidx(k + 1, mu - 1)]);
                Gm[i] = cscal((mu >= 0 ? -1.0 : 1.0) * sqrt((double)(k + 2 + mu) * (k + 1 + mu)), C[eidx(k + 1, mu + 1)]);
            }
        }
    } else {
        for (int i = 1 + threadIdx.x; i < K1; i += kEvalThreads) {
            int k = (int)sqrtf((float)i);
            while (k * k > i) k--;
            while ((k + 1) * (k + 1) <= i) k++;
            int mu = i - k * k - k;
            if (WHICH & 2) {
                double2 mz = (abs(mu) <= k - 1) ? C[eidx(k - 1, mu)] : cmk(0, 0);
                Gz[i - 1] = cscal(-sqrt((double)(k + mu) * (k - mu)), mz);
            }
            if (WHICH & 4) {
                double2 mp = (abs(mu - 1) <= k - 1) ? C[eidx(k - 1, mu - 1)] : cmk(0, 0);
                double2 mm = (abs(mu + 1) <= k - 1) ? C[eidx(k - 1, mu + 1)] : cmk(0, 0);
                Gp[i - 1] = cscal((mu <= 0 ? -1.0 : 1.0) * sqrt((double)(k + mu - 1) * (k + mu)), mp);
                Gm[i - 1] = cscal((mu >= 0 ? -1.0 : 1.0) * sqrt((double)(k - mu - 1) * (k - mu)), mm);
            }
        }
    }
}

// Harmonics of one point in box units (u), generated by the three-term
// recurrences, dotted with the staged arrays selected by MASK.
template <int MASK>
__device__ __forceinline__ void eval_point(bool loc, int p, double ux, double uy, double uz, const double2 *A,
                                           const double2 *Gz, const double2 *Gp, const double2 *Gm, double2 &phi,
                                           double2 &dz, double2 &dp, double2 &dm)
{
    const double r2 = ux * ux + uy * uy + uz * uz;
    if (loc) {
        double2 diag = cmk(1.0, 0.0);
        for (int m = 0; m <= p; m++) {
            if (m > 0) {
                double cc = -c_cm[m];
                diag = cmk(cc * (ux * diag.x + uy * diag.y), cc * (ux * diag.y - uy * diag.x));
            }
            double2 r1 = cmk(0, 0), r0 = diag;
            for (int n = m; n <= p; n++) {
                double2 h;
                if (n == m) h = diag;
                else if (n == m + 1) h = cscal(c_sq[m] * uz, diag);
                else {
                    double a = c_ra[tidx(n, m)] * uz, bb = c_rb[tidx(n, m)] * r2;
                    h = cmk(a * r0.x - bb * r1.x, a * r0.y - bb * r1.y);
                }
                if (n > m) { r1 = r0; r0 = h; }
                dot4_acc<MASK>(h, n, m, A, Gz, Gp, Gm, 0, p - 1, phi, dz, dp, dm);
            }
        }
    } else {
        const double ir2 = 1.0 / r2, zi = uz * ir2;
        double2 diag = cmk(sqrt(ir2), 0.0);
        for (int m = 0; m <= p + 1; m++) {
            if (m > 0) {
                double cc = -c_cm[m] * ir2;
                diag = cmk(cc * (ux * diag.x + uy * diag.y), cc * (ux * diag.y - uy * diag.x));
            }
            double2 r1 = cmk(0, 0), r0 = diag;
            for (int n = m; n <= p + 1; n++) {
                double2 h;
                if (n == m) h = diag;
                else if (n == m + 1) h = cscal(c_sq[m] * zi, diag);
                else {
                    double a = c_ra[tidx(n, m)] * zi, bb = c_rb[tidx(n, m)] * ir2;
                    h = cmk(a * r0.x - bb * r1.x, a * r0.y - bb * r1.y);
                }
                if (n > m) { r1 = r0; r0 = h; }
                dot4_acc<MASK>(h, n, m, n <= p ? A : nullptr, Gz, Gp, Gm, 1, p + 1, phi, dz, dp, dm);
            }
        }
    }
}

// The evaluation pass is cut into work items of one leaf, one chunk of
// kEvalThreads of its points and one group of at most kEvalGroup of its source
// expansions (the leaf's local expansion first, then its list-3 multipoles),
// one CTA each: list 3 is very uneven on adaptive trees (on a sphere surface
// most leaves have none and a few have dozens).  Leaves with one group add
// their sums to the outputs directly, exactly as one pass over the leaf; the
// groups of the other leaves write their sums to scratch slots, which
// k_eval_add adds to the outputs in group order.  The item offsets (off) and
// the scratch offsets (soff) come from k_eval_count and two scans, made with
// the tree.
//
// k_eval_mm serves the orders whose columns fit shared memory (p <= 52).  k_eval, above
// them: the potential and z-gradient first, then the transverse gradients, each
// point's harmonics generated once per phase, one point per thread.
__global__ void k_eval_count(const int *leaves, int nleaves, TreeView tv, int do_src, int do_trg, int *cnt,
                             int *scnt)
{
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nleaves) return;
    const int b = leaves[l];
    const int ne = (do_src ? tv.nsrc[b] : 0) + (do_trg ? tv.ntrg[b] : 0), nbx = eval_nbx(tv, b);
    const int items = (ne > 0 && nbx > 0)
                          ? ((ne + kEvalThreads - 1) / kEvalThreads) * ((nbx + kEvalGroup - 1) / kEvalGroup)
                          : 0;
    cnt[l] = items;
    scnt[l] = nbx > kEvalGroup ? items : 0;
}

// Factors of the gradient arrays at (k, mu): d/dz, D+ and D- of an order-p
// expansion take its coefficients (k', mu), (k', mu - 1) and (k', mu + 1), k' = k + 1
// for a local expansion and k - 1 for a multipole, times these (0: no such coefficient).
__device__ void grad_factors(bool loc, int p, int k, int mu, double *f)
{
    f[0] = f[1] = f[2] = 0;
    if (loc) {
        if (k >= p) return;
        f[0] = sqrt((double)(k + 1 + mu) * (k + 1 - mu));
        f[1] = (mu <= 0 ? -1.0 : 1.0) * sqrt((double)(k + 2 - mu) * (k + 1 - mu));
        f[2] = (mu >= 0 ? -1.0 : 1.0) * sqrt((double)(k + 2 + mu) * (k + 1 + mu));
    } else {
        if (k < 1) return;
        if (abs(mu) <= k - 1) f[0] = -sqrt((double)(k + mu) * (k - mu));
        if (abs(mu - 1) <= k - 1) f[1] = (mu <= 0 ? -1.0 : 1.0) * sqrt((double)(k + mu - 1) * (k + mu));
        if (abs(mu + 1) <= k - 1) f[2] = (mu >= 0 ? -1.0 : 1.0) * sqrt((double)(k - mu - 1) * (k - mu));
    }
}

__global__ void k_emm_tables(int p, int nstep, double2 *ab, double *cm, int *step, double *fm, double *fl)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, nmax = p + 1;
    if (i <= nmax) cm[i] = i ? sqrt((2.0 * i - 1) / (2.0 * i)) : 0.0;
    if (i >= nstep * 4) return;
    double2 f;
    const int st = emm_factors(i, nmax, f), n = st & 0xffff, m = 4 * (st >> 16) + (i & 3);
    ab[i] = f;
    if ((i & 3) == 0) step[i >> 2] = st;
    for (int sg = 0; sg < 2; sg++) {
        double z[6] = {0, 0, 0, 0, 0, 0};
        if (m <= n) {
            grad_factors(false, p, n, sg ? -m : m, z);
            grad_factors(true, p, n, sg ? -m : m, z + 3);
        }
        for (int c = 0; c < 3; c++) {
            fm[(2 * i + sg) * 3 + c] = z[c];
            fl[(2 * i + sg) * 3 + c] = z[3 + c];
        }
    }
}

static_assert(sizeof(double) * emm_smem(52 + 1, 1) <= kEmmSmemMax && sizeof(double) * emm_smem(53 + 1, 1) > kEmmSmemMax,
              "largest order of k_eval_mm");

void build_emm_tables(int p, EmmTables &E, cudaStream_t s, Status &st)
{
    if (sizeof(double) * emm_smem(p + 1, 1) > kEmmSmemMax) return;
    const int ns = emm_steps(p + 1);
    if (!E.ab.alloc(4 * ns, s, st) || !E.cm.alloc(p + 2, s, st) || !E.step.alloc(ns, s, st) ||
        !E.fac[0].alloc(24 * ns, s, st) || !E.fac[1].alloc(24 * ns, s, st))
        return;
    k_emm_tables<<<div_up(4 * ns + p + 2, 128), 128, 0, s>>>(p, ns, E.ab.p, E.cm.p, E.step.p, E.fac[0].p, E.fac[1].p);
    FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
    E.ab.s = E.cm.s = E.step.s = E.fac[0].s = E.fac[1].s = nullptr;   // kept for the life of the process
    E.ready = st.ok();
}

// Potential and field of a work item in matrix products (eval_mm.cuh): the 8
// columns are the potential and the three gradient components, real and
// imaginary.
__global__ void __launch_bounds__(kEvalThreads) k_eval_mm(const int *leaves, int nleaves, const int *off,
                                                          const int *soff, TreeView tv, const double *sx,
                                                          const double *sy, const double *sz, const double *tx,
                                                          const double *ty, const double *tz, int p,
                                                          const double2 *mpole, const double2 *local, OutSoA outs,
                                                          OutSoA outt, int do_src, int do_trg, double *part,
                                                          EmmTab tab)
{
    extern __shared__ double emm_sm[];
    const int l = emm_leaf(off, nleaves, blockIdx.x), b = leaves[l];
    const int ns = do_src ? tv.nsrc[b] : 0, ne = ns + (do_trg ? tv.ntrg[b] : 0);
    const int ngr = (eval_nbx(tv, b) + kEvalGroup - 1) / kEvalGroup;
    const int local_item = blockIdx.x - off[l], ck = local_item / ngr, grp = local_item - ck * ngr;
    const int s0 = tv.src0[b], t0 = tv.trg0[b];
    emm_item<1>(
        emm_sm, p + 1, tab, tv, b, grp, ck * kEvalThreads, ne, ns, sx, sy, sz, tx, ty, tz, (p + 1) * (p + 1), mpole, local,
        [&](bool loc) { return loc ? p : p + 1; },
        [](double is, int k) { return k ? is * is : is; },
        [&](bool loc, const double2 *C, int i, int sign, int n, int mu, double2 *v) {
            if (n <= p) v[0] = C[eidx(n, mu)];
            const double *f = tab.fac[loc] + (2 * i + sign) * 3;
            const double f0 = __ldg(f), f1 = __ldg(f + 1), f2 = __ldg(f + 2);
            const double2 *c = C + (loc ? eidx(n + 1, mu) : eidx(n - 1, mu));
            const double2 z = f0 != 0 ? cscal(f0, c[0]) : cmk(0, 0), dp = f1 != 0 ? cscal(f1, c[-1]) : cmk(0, 0),
                          dm = f2 != 0 ? cscal(f2, c[1]) : cmk(0, 0);
            const double2 d = csub(dp, dm);
            v[1] = cscal(0.5, cadd(dp, dm));             // d/dx = (D+ + D-) / 2
            v[2] = cmk(0.5 * d.y, -0.5 * d.x);           // d/dy = (D+ - D-) / 2i
            v[3] = z;
        },
        [&](int e, int k, double2 v) {
            if (k) v = cmk(-v.x, -v.y);                  // the field is minus the gradient
            if (ngr > 1) {
                double *o = part + ((size_t)(soff[l] + local_item) * 8 + 2 * k) * kEvalThreads + e - ck * kEvalThreads;
                o[0] = v.x;
                o[kEvalThreads] = v.y;
                return;
            }
            const OutSoA &o = e < ns ? outs : outt;
            double2 *a = k == 0 ? o.pot : k == 1 ? o.fx : k == 2 ? o.fy : o.fz;
            const int i = e < ns ? s0 + e : t0 + e - ns;
            if (a) a[i] = cadd(a[i], v);
        });
}

__global__ void __launch_bounds__(kEvalThreads) k_eval(const int *leaves, int nleaves, const int *off,
                                                       const int *soff, TreeView tv, const double *sx,
                                                       const double *sy, const double *sz, const double *tx,
                                                       const double *ty, const double *tz, int p,
                                                       const double2 *mpole, const double2 *local, OutSoA outs,
                                                       OutSoA outt, int do_src, int do_trg, double *part)
{
    extern __shared__ double2 sm[];
    const int K = (p + 1) * (p + 1), K1 = (p + 2) * (p + 2);
    double2 *b0 = sm, *b1 = sm + K1;
    const int item = blockIdx.x, l = emm_leaf(off, nleaves, item);
    const int b = leaves[l];
    const int lev = tv.level[b];
    const int s0 = tv.src0[b], ns = do_src ? tv.nsrc[b] : 0;
    const int t0 = tv.trg0[b], nt = do_trg ? tv.ntrg[b] : 0;
    const int ne = ns + nt;
    const int l3a = tv.l3_start[b];
    const bool has_local = lev >= 2;
    const int nbx = eval_nbx(tv, b), ngr = (nbx + kEvalGroup - 1) / kEvalGroup;
    const int local_item = item - off[l], ck = local_item / ngr, grp = local_item - ck * ngr;
    const int e = ck * kEvalThreads + threadIdx.x;
    const bool act = e < ne;
    const bool is_src = e < ns;
    double px = 0, py = 0, pz = 0;
    if (act) {
        if (is_src) { px = sx[s0 + e]; py = sy[s0 + e]; pz = sz[s0 + e]; }
        else { px = tx[t0 + e - ns]; py = ty[t0 + e - ns]; pz = tz[t0 + e - ns]; }
    }
    double2 pot = cmk(0, 0), gx = cmk(0, 0), gy = cmk(0, 0), gzz = cmk(0, 0);
    const int ib1 = min(nbx, (grp + 1) * kEvalGroup);
    for (int ib = grp * kEvalGroup; ib < ib1; ib++) {
        const bool loc = has_local && ib == 0;
        const int c = loc ? b : tv.l3_idx[l3a + ib - (has_local ? 1 : 0)];
        const double s = box_side(tv, c), is = 1.0 / s;
        const double2 *coef = loc ? local + (size_t)c * K : mpole + (size_t)c * K;
        const double ux = (px - tv.center[3L * c]) * is, uy = (py - tv.center[3L * c + 1]) * is,
                     uz = (pz - tv.center[3L * c + 2]) * is;
        double2 phi = cmk(0, 0), dz = cmk(0, 0), dp = cmk(0, 0), dm = cmk(0, 0);
        for (int ph = 0; ph < 2; ph++) {
            __syncthreads();
            if (ph == 0) {
                for (int i = threadIdx.x; i < K; i += kEvalThreads) b0[i] = coef[i];
                stage_grad<2>(loc, p, coef, b1, nullptr, nullptr);
            } else {
                stage_grad<4>(loc, p, coef, nullptr, b0, b1);
            }
            __syncthreads();
            if (!act) continue;
            if (ph == 0) eval_point<3>(loc, p, ux, uy, uz, b0, b1, nullptr, nullptr, phi, dz, dp, dm);
            else eval_point<4>(loc, p, ux, uy, uz, nullptr, nullptr, b0, b1, phi, dz, dp, dm);
        }
        if (!act) continue;
        // phi and gradient in box units -> physical units
        double is2 = is * is;
        pot = cadd(pot, cscal(is, phi));
        // d/dx = (D+ + D-)/2, d/dy = (D+ - D-)/(2i)
        double2 ddx = cscal(0.5, cadd(dp, dm));
        double2 dd = csub(dp, dm);
        double2 ddy = cmk(0.5 * dd.y, -0.5 * dd.x);
        gx = cadd(gx, cscal(is2, ddx));
        gy = cadd(gy, cscal(is2, ddy));
        gzz = cadd(gzz, cscal(is2, dz));
    }
    if (!act) return;
    if (ngr > 1) {
        // this group's sums: pot, then -grad (x, y, z)
        double *o = part + (size_t)(soff[l] + local_item) * 8 * kEvalThreads + threadIdx.x;
        o[0] = pot.x; o[kEvalThreads] = pot.y;
        o[2 * kEvalThreads] = -gx.x; o[3 * kEvalThreads] = -gx.y;
        o[4 * kEvalThreads] = -gy.x; o[5 * kEvalThreads] = -gy.y;
        o[6 * kEvalThreads] = -gzz.x; o[7 * kEvalThreads] = -gzz.y;
        return;
    }
    if (is_src) {
        int i = s0 + e;
        if (outs.pot) outs.pot[i] = cadd(outs.pot[i], pot);
        if (outs.fx) { outs.fx[i] = csub(outs.fx[i], gx); outs.fy[i] = csub(outs.fy[i], gy); outs.fz[i] = csub(outs.fz[i], gzz); }
    } else {
        int i = t0 + e - ns;
        if (outt.pot) outt.pot[i] = cadd(outt.pot[i], pot);
        if (outt.fx) { outt.fx[i] = csub(outt.fx[i], gx); outt.fy[i] = csub(outt.fy[i], gy); outt.fz[i] = csub(outt.fz[i], gzz); }
    }
}

// Adds the groups' sums of the leaves with more than one group, group by group.
__global__ void __launch_bounds__(kEvalThreads) k_eval_add(const int *leaves, const int *soff, TreeView tv,
                                                           OutSoA outs, OutSoA outt, int do_src, int do_trg,
                                                           const double *part)
{
    const int l = blockIdx.x, b = leaves[l];
    const int nbx = eval_nbx(tv, b);
    if (nbx <= kEvalGroup) return;
    const int s0 = tv.src0[b], ns = do_src ? tv.nsrc[b] : 0;
    const int t0 = tv.trg0[b], nt = do_trg ? tv.ntrg[b] : 0;
    const int ne = ns + nt, ngr = (nbx + kEvalGroup - 1) / kEvalGroup, nch = (ne + kEvalThreads - 1) / kEvalThreads;
    for (int ck = blockIdx.y; ck < nch; ck += gridDim.y) {
        const int e = ck * kEvalThreads + threadIdx.x;
        if (e >= ne) continue;
        const bool is_src = e < ns;
        const int i = is_src ? s0 + e : t0 + e - ns;
        double2 *po = is_src ? outs.pot : outt.pot;
        double2 *ox = is_src ? outs.fx : outt.fx, *oy = is_src ? outs.fy : outt.fy, *oz = is_src ? outs.fz : outt.fz;
        double2 vp = po ? po[i] : cmk(0, 0), vx = ox ? ox[i] : cmk(0, 0), vy = ox ? oy[i] : cmk(0, 0),
                vz = ox ? oz[i] : cmk(0, 0);
        for (int g = 0; g < ngr; g++) {
            const double *q = part + (size_t)(soff[l] + ck * ngr + g) * 8 * kEvalThreads + threadIdx.x;
            vp = cadd(vp, cmk(q[0], q[kEvalThreads]));
            vx = cadd(vx, cmk(q[2 * kEvalThreads], q[3 * kEvalThreads]));
            vy = cadd(vy, cmk(q[4 * kEvalThreads], q[5 * kEvalThreads]));
            vz = cadd(vz, cmk(q[6 * kEvalThreads], q[7 * kEvalThreads]));
        }
        if (po) po[i] = vp;
        if (ox) {
            ox[i] = vx;
            oy[i] = vy;
            oz[i] = vz;
        }
    }
}

int eval_items_prepare(const int *leaves, int nleaves, const TreeView &tv, int do_src, int do_trg, int hess,
                       EvalItems &E, cudaStream_t s, Status &st)
{
    E.nitems = E.nscratch = 0;
    if (nleaves == 0 || !st.ok()) return 0;
    DBuf<int> cnt, scnt;
    if (!cnt.alloc(nleaves, s, st) || !scnt.alloc(nleaves, s, st) || !E.off.alloc(nleaves, s, st) ||
        !E.soff.alloc(nleaves, s, st))
        return 0;
    k_eval_count<<<div_up(nleaves, 256), 256, 0, s>>>(leaves, nleaves, tv, do_src, do_trg, cnt.p, scnt.p);
    FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
    DBuf<int> tot;
    int h[2] = {0, 0};
    if (!tot.alloc(2, s, st)) return 0;
    const ScanJob jobs[2] = {{cnt.p, E.off.p, nleaves, nullptr}, {scnt.p, E.soff.p, nleaves, nullptr}};
    scan_exclusive_multi(jobs, 2, tot.p, s, st);
    FMM_TRY(st, cudaMemcpyAsync(h, tot.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    FMM_TRY(st, cudaStreamSynchronize(s));
    if (!st.ok()) return 0;
    E.nitems = h[0];
    E.nscratch = h[1];
    if (E.nscratch > 0) E.part.alloc((size_t)E.nscratch * 8 * kEvalThreads, s, st);
    if (E.nscratch > 0 && hess) E.hpart.alloc((size_t)E.nscratch * 12 * kEvalThreads, s, st);
    return E.nitems;
}

void launch_eval(const int *leaves, int nleaves, const EvalItems &E, const EmmTables &tab, const TreeView &tv, const double *sx,
                 const double *sy, const double *sz, const double *tx, const double *ty, const double *tz, int p,
                 const double2 *mpole, const double2 *local, OutSoA outs, OutSoA outt, int do_src, int do_trg,
                 cudaStream_t s, Status &st)
{
    if (nleaves == 0 || E.nitems == 0 || !st.ok()) return;
    if (tab.ready) {
        const size_t mm = sizeof(double) * emm_smem(p + 1, 1);
        const EmmTab t = {tab.ab.p, tab.cm.p, tab.step.p, {tab.fac[0].p, tab.fac[1].p}};
        FMM_TRY(st, smem_allow(k_eval_mm, mm));
        k_eval_mm<<<E.nitems, kEvalThreads, mm, s>>>(leaves, nleaves, E.off.p, E.soff.p, tv, sx, sy, sz, tx, ty, tz, p,
                                                     mpole, local, outs, outt, do_src, do_trg, E.part.p, t);
    } else {
        const size_t arr = (size_t)(p + 2) * (p + 2) * sizeof(double2);
        FMM_TRY(st, smem_allow(k_eval, 2 * arr));
        k_eval<<<E.nitems, kEvalThreads, 2 * arr, s>>>(leaves, nleaves, E.off.p, E.soff.p, tv, sx, sy, sz, tx, ty, tz,
                                                       p, mpole, local, outs, outt, do_src, do_trg, E.part.p);
    }
    FMM_COUNT_LAUNCH();
    if (E.nscratch > 0) {
        k_eval_add<<<dim3(nleaves, 2), kEvalThreads, 0, s>>>(leaves, E.soff.p, tv, outs, outt, do_src, do_trg,
                                                             E.part.p);
        FMM_COUNT_LAUNCH();
    }
    FMM_LAUNCH_CHECK(st);
}

// ================================================================ rotations
// Rotation matrices about the y axis, one per class (theta), in the basis
// S_n^m = Y_n^|m| e^{i m phi}: D^n[m][m'] = (2n+1)/(4 pi) *
// Integral S_n^m(R_y(theta) w) conj(S_n^m'(w)) dw, evaluated exactly with a
// product rule of (p+1) Gauss-Legendre nodes in cos(theta) times 2p+1
// equispaced azimuths (exact for the degree-2p integrands).  Storage per
// class: degree n at offset n(4n^2-1)/3, (2n+1)x(2n+1) row-major [m+n][m'+n].
// The reference builds the same matrices by the recursion of
// rotviarecur3p_init (src/rotviarecur3.f:717-869).
// Recurrence tables of regular_table for the rotation builder, in global
// memory and long enough for the Helmholtz orders (the __constant__ copies
// above serve the Laplace kernels up to kTabP).
constexpr int kRotTabN = (kRotTabP + 2) * (kRotTabP + 3) / 2;
__device__ double g_rot_ra[kRotTabN], g_rot_rb[kRotTabN], g_rot_cm[kRotTabP + 2], g_rot_sq[kRotTabP + 2];

static void rot_tables_init(Status &st)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    static std::vector<double> ra, rb, cm, sq;
    if (ra.empty()) {
        ra.assign(kRotTabN, 0.0);
        rb.assign(kRotTabN, 0.0);
        cm.assign(kRotTabP + 2, 0.0);
        sq.assign(kRotTabP + 2, 0.0);
        for (int n = 0; n <= kRotTabP + 1; n++)
            for (int m = 0; m <= n; m++) {
                if (n >= m + 2) {
                    double den = sqrt((double)(n - m) * (n + m));
                    ra[tidx(n, m)] = (2.0 * n - 1) / den;
                    rb[tidx(n, m)] = sqrt((double)(n + m - 1) * (n - m - 1)) / den;
                }
            }
        for (int m = 1; m <= kRotTabP + 1; m++) cm[m] = sqrt((2.0 * m - 1) / (2.0 * m));
        for (int m = 0; m <= kRotTabP + 1; m++) sq[m] = sqrt(2.0 * m + 1);
    }
    int dev = 0;
    cudaGetDevice(&dev);
    static bool uploaded[64] = {false};
    if (dev < 64 && uploaded[dev]) return;
    FMM_TRY(st, cudaMemcpyToSymbol(g_rot_ra, ra.data(), sizeof(double) * ra.size()));
    FMM_TRY(st, cudaMemcpyToSymbol(g_rot_rb, rb.data(), sizeof(double) * rb.size()));
    FMM_TRY(st, cudaMemcpyToSymbol(g_rot_cm, cm.data(), sizeof(double) * cm.size()));
    FMM_TRY(st, cudaMemcpyToSymbol(g_rot_sq, sq.data(), sizeof(double) * sq.size()));
    if (st.ok() && dev < 64) uploaded[dev] = true;
}

// regular_table with the global tables (orders up to kRotTabP)
__device__ void regular_table_rot(double x, double y, double z, int p, double2 *out)
{
    double r2 = x * x + y * y + z * z;
    double2 diag = cmk(1.0, 0.0);
    for (int m = 0; m <= p; m++) {
        if (m > 0) {
            double c = -g_rot_cm[m];
            diag = cmk(c * (x * diag.x + y * diag.y), c * (x * diag.y - y * diag.x));
        }
        out[tidx(m, m)] = diag;
        if (m < p) {
            double2 r1 = diag;
            double2 r0 = cscal(g_rot_sq[m] * z, diag);
            out[tidx(m + 1, m)] = r0;
            for (int n = m + 2; n <= p; n++) {
                double a = g_rot_ra[tidx(n, m)] * z, b = g_rot_rb[tidx(n, m)] * r2;
                double2 rn = cmk(a * r0.x - b * r1.x, a * r0.y - b * r1.y);
                out[tidx(n, m)] = rn;
                r1 = r0;
                r0 = rn;
            }
        }
    }
}

__global__ void k_rot_nodes(int p, int nq, const double *gl_x, const double *cs, int cls0, double2 *Sr, double2 *S0)
{
    const int cls = cls0 + blockIdx.y;
    // one thread per quadrature node: harmonics at the node and at the rotated node
    int nphi = 2 * p + 1;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq * nphi) return;
    int a = i / nphi, bphi = i % nphi;
    double mu = gl_x[a], st_ = sqrt(fmax(0.0, 1 - mu * mu));
    double ph = 2.0 * M_PI * bphi / nphi;
    double sp, cp;
    sincos(ph, &sp, &cp);
    double wx = st_ * cp, wy = st_ * sp, wz = mu;
    double ct = cs[2 * cls], stt = cs[2 * cls + 1];
    double rx = wx * ct + wz * stt, ry = wy, rz = -wx * stt + wz * ct;
    int ntab = (p + 1) * (p + 2) / 2;
    regular_table_rot(rx, ry, rz, p, Sr + ((size_t)blockIdx.y * nq * nphi + i) * ntab);
    if (S0 && blockIdx.y == 0) regular_table_rot(wx, wy, wz, p, S0 + (size_t)i * ntab);
}

__global__ void k_rot_reduce(int p, int nq, const double *gl_w, const double2 *Sr, const double2 *S0, double *rot)
{
    // one thread per (n, m, m') of this class
    size_t tot = rot_class_size(p);
    size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (e >= tot) return;
    int n = 0;
    while ((size_t)(n + 1) * (4 * (n + 1) * (n + 1) - 1) / 3 <= e) n++;
    size_t off = (size_t)n * (4 * n * n - 1) / 3;
    int w = 2 * n + 1;
    int r = (int)((e - off) / w), c = (int)((e - off) % w);
    int m = r - n, mp = c - n;
    int nphi = 2 * p + 1, ntab = (p + 1) * (p + 2) / 2;
    Sr += (size_t)blockIdx.y * nq * nphi * ntab;
    rot += tot * blockIdx.y;
    double acc = 0;
    int tm = tidx(n, m < 0 ? -m : m), tmp = tidx(n, mp < 0 ? -mp : mp);
    for (int i = 0; i < nq * nphi; i++) {
        // S_n^m(v) = conj(R_n^m(v)) for m >= 0, R_n^|m|(v) for m < 0 (unit v)
        double2 a = Sr[(size_t)i * ntab + tm];
        if (m >= 0) a = cconj(a);
        double2 bb = S0[(size_t)i * ntab + tmp];
        if (mp >= 0) bb = cconj(bb);
        // Re(a * conj(bb))
        acc += gl_w[i / nphi] * (a.x * bb.x + a.y * bb.y);
    }
    rot[e] = acc * (2.0 * M_PI / nphi) * (2 * n + 1) / (4.0 * M_PI);
}

// n-point Gauss-Legendre rule; each n is computed once per process (the
// Helmholtz driver asks for the same few rules for every operator block of
// every call)
void gauss_legendre(int n, std::vector<double> &x, std::vector<double> &w)
{
    static std::mutex mu;
    static std::map<int, std::pair<std::vector<double>, std::vector<double>>> memo;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = memo.find(n);
        if (it != memo.end()) {
            x = it->second.first;
            w = it->second.second;
            return;
        }
    }
    x.resize(n);
    w.resize(n);
    for (int i = 0; i < n; i++) {
        double z = cos(M_PI * (i + 0.75) / (n + 0.5)), pp = 0;
        for (int it = 0; it < 100; it++) {
            double p1 = 1, p2 = 0;
            for (int j = 1; j <= n; j++) {
                double p3 = p2;
                p2 = p1;
                p1 = ((2.0 * j - 1) * z * p2 - (j - 1.0) * p3) / j;
            }
            pp = n * (z * p1 - p2) / (z * z - 1);
            double z1 = z;
            z = z1 - p1 / pp;
            if (fabs(z - z1) < 1e-16) break;
        }
        x[i] = z;
        w[i] = 2 / ((1 - z * z) * pp * pp);
    }
    std::lock_guard<std::mutex> lk(mu);
    memo.emplace(n, std::make_pair(x, w));
}

void build_rotations(int p, int ncls, const double *d_cs, double *d_rot, cudaStream_t s, Status &st)
{
    if (!st.ok()) return;
    if (p > kRotTabP) {
        st.err = cudaErrorInvalidValue;
        st.where = "rotation order above the recurrence tables";
        return;
    }
    rot_tables_init(st);     // regular_table_rot reads the recurrence tables
    std::vector<double> gx, gw;
    gauss_legendre(p + 1, gx, gw);
    int nq = p + 1, nphi = 2 * p + 1, nodes = nq * nphi, ntab = (p + 1) * (p + 2) / 2;
    DBuf<double> dx, dw;
    DBuf<double2> Sr, S0;
    dx.alloc(nq, s, st);
    dw.alloc(nq, s, st);
    // as many classes per launch as 256 MB of node tables hold
    const int per = (int)std::max<size_t>(1, std::min<size_t>(ncls, (256u << 20) / ((size_t)nodes * ntab * 16)));
    Sr.alloc((size_t)nodes * ntab * per, s, st);
    S0.alloc((size_t)nodes * ntab, s, st);
    if (!st.ok()) return;
    FMM_TRY(st, cudaMemcpyAsync(dx.p, gx.data(), sizeof(double) * nq, cudaMemcpyHostToDevice, s));
    FMM_TRY(st, cudaMemcpyAsync(dw.p, gw.data(), sizeof(double) * nq, cudaMemcpyHostToDevice, s));
    size_t csz = rot_class_size(p);
    for (int c = 0; c < ncls; c += per) {
        const int k = std::min(per, ncls - c);
        k_rot_nodes<<<dim3(div_up(nodes, 128), k), 128, 0, s>>>(p, nq, dx.p, d_cs, c, Sr.p, c == 0 ? S0.p : nullptr);
        FMM_COUNT_LAUNCH();
        k_rot_reduce<<<dim3(div_up((long)csz, 128), k), 128, 0, s>>>(p, nq, dw.p, Sr.p, S0.p, d_rot + csz * c);
        FMM_COUNT_LAUNCH();
    }
    FMM_LAUNCH_CHECK(st);
    FMM_TRY(st, cudaStreamSynchronize(s));  // the host vectors above must outlive the copies
}

// ================================================================ translations
// Rotate-shift-rotate translation of FMMLIB3D's l3dmpmpquad0 (M2M),
// l3dmplocquad2_trunc0 (M2L) and l3dloclocquad0 (L2L)
// (src/l3dtrans.f:223, 1260, 1676), batched: a CTA owns a tile of up to KT
// target boxes that share a level and an octant, hence the same list of
// source slots; for each slot it gathers the KT source expansions, applies
// e^{i m phi}, the rotation D(theta), the z-shift of the kind, D(theta)^T
// and e^{-i m phi}, and accumulates into the targets in shared memory.
// The z-shift coefficients, in units of the box side, are
//   M2M: (-rt)^l sqrt(C(j-k,l) C(j+k,l)) / 2^j          (l3dmpmpzshift :351)
//   M2L: (-1)^(j+k) sqrt(C(l+j,l-k) C(l+j,l+k)) / rt^(l+j+1)
//                                              (l3dmploczshiftstab_fast :1439)
//   L2L: rt^l sqrt(C(j+l+k,l) C(j+l-k,l)) / 2^(j+l+1)    (l3dlocloczshift :1798)
constexpr int kTransThreads = 256;

__device__ __forceinline__ int src_of(int kind, const TreeView &tv, int t, const Slot &sl)
{
    if (kind == 0) return tv.child[8L * t + sl.oct];
    if (kind == 2) return tv.parent[t];
    int P = tv.parent[t];
    if (P < 0) return -1;
    int C = tv.coll[27L * P + sl.coll];
    if (C < 0) return -1;
    return tv.child[8L * C + sl.oct];
}

template <int KIND, int KT, int RPT>
__global__ void __launch_bounds__(kTransThreads) k_translate(const Tile *tiles, const int *grouped,
                                                             const Slot *slots, TreeView tv, int p,
                                                             const double *rot, const double *dc, int lddc,
                                                             const double2 *in, double2 *out, int prune)
{
    // RPT > 0: the running sums live in registers, RPT coefficient rows per
    // thread (row = thread + 256 j), which leaves shared memory for more
    // targets per tile; RPT == 0: in shared memory.
    extern __shared__ double2 sm[];
    const int NC = (p + 1) * (p + 1);
    double2 *acc = sm;
    double2 *bA = acc + (RPT > 0 ? 0 : (size_t)KT * NC);
    double2 *bB = bA + (size_t)KT * NC;
    double2 *eph = bB + (size_t)KT * NC;  // e^{i m phi}, m = 0..p
    double2 racc[RPT > 0 ? RPT : 1][KT];
#pragma unroll
    for (int j = 0; j < (RPT > 0 ? RPT : 1); j++)
#pragma unroll
        for (int k = 0; k < KT; k++) racc[j][k] = cmk(0, 0);
    double *pw = (double *)(eph + (p + 1));  // powers, 0..2p+2
    __shared__ int tg[8], sv[8];
    __shared__ int anyv;
    const Tile tile = tiles[blockIdx.x];
    if (threadIdx.x < 8) {
        int t = threadIdx.x < tile.count ? grouped[tile.first + threadIdx.x] : -1;
        if (t >= 0 && KIND == 0 && tv.nchild[t] == 0) t = -1;  // M2M only into boxes with children
        tg[threadIdx.x] = t;
    }
    if (RPT == 0)
        for (int i = threadIdx.x; i < KT * NC; i += kTransThreads) acc[i] = cmk(0, 0);
    const size_t csz = rot_class_size(p);
    for (int si = 0; si < tile.nslot; si++) {
        const Slot sl = slots[tile.slot0 + si];
        __syncthreads();
        if (threadIdx.x == 0) anyv = 0;
        __syncthreads();
        if (threadIdx.x < KT) {
            int t = tg[threadIdx.x];
            int sb = -1;
            if (t >= 0) {
                sb = src_of(KIND, tv, t, sl);
                if (sb >= 0 && KIND != 2 && tv.nsrc[sb] == 0) sb = -1;
                if (KIND == 1 && prune && tv.ntrg[t] == 0) sb = -1;
            }
            sv[threadIdx.x] = sb;
            if (sb >= 0) atomicOr(&anyv, 1);
        }
        if (threadIdx.x == 32) {
            double2 e1 = cmk(sl.ex, sl.ey), e = cmk(1, 0);
            for (int m = 0; m <= p; m++) { eph[m] = e; e = cmul(e, e1); }
            double r = sl.rt, x = 1;
            if (KIND == 1) {
                double ir = 1.0 / r;
                x = ir;
                for (int l = 0; l <= 2 * p + 2; l++) { pw[l] = x; x *= ir; }  // pw[l] = rt^-(l+1)
            } else {
                for (int l = 0; l <= 2 * p + 2; l++) { pw[l] = x; x *= r; }   // pw[l] = rt^l
            }
        }
        __syncthreads();
        if (!anyv) continue;
        const int pin = KIND == 1 ? sl.pt : p;   // source degrees used
        const int pout = KIND == 1 ? sl.pt : p;  // target degrees produced
        const int Rin = (pin + 1) * (pin + 1), Rout = (pout + 1) * (pout + 1);
        // phase 1: gather, times e^{i m phi}
        for (int i = threadIdx.x; i < KT * Rin; i += kTransThreads) {
            int k = i / Rin, e = i % Rin;
            int sb = sv[k];
            double2 v = cmk(0, 0);
            if (sb >= 0) {
                int n = (int)sqrtf((float)e);
                while (n * n > e) n--;
                while ((n + 1) * (n + 1) <= e) n++;
                int m = e - n * n - n;
                double2 ph = m >= 0 ? eph[m] : cconj(eph[-m]);
                v = cmul(in[(size_t)sb * NC + e], ph);
            }
            bA[(size_t)k * NC + e] = v;
        }
        __syncthreads();
        const double *R = rot + csz * sl.cls;
        // phase 2: bB[n][m'] = sum_m bA[n][m] D[m][m']
        for (int row = threadIdx.x; row < Rin; row += kTransThreads) {
            int n = (int)sqrtf((float)row);
            while (n * n > row) n--;
            while ((n + 1) * (n + 1) <= row) n++;
            int mp = row - n * n - n;
            const double *Dn = R + (size_t)n * (4 * n * n - 1) / 3;
            int w = 2 * n + 1;
            double2 a[KT];
            _Pragma("unroll") for (int k = 0; k < KT; k++) a[k] = cmk(0, 0);
            for (int m = -n; m <= n; m++) {
                double d = Dn[(m + n) * w + (mp + n)];
                _Pragma("unroll") for (int k = 0; k < KT; k++) crfma(a[k], d, bA[(size_t)k * NC + eidx(n, m)]);
            }
            _Pragma("unroll") for (int k = 0; k < KT; k++) bB[(size_t)k * NC + row] = a[k];
        }
        __syncthreads();
        // phase 3: z-shift, bA[j][kk] from bB[.][kk]
        for (int row = threadIdx.x; row < Rout; row += kTransThreads) {
            int j = (int)sqrtf((float)row);
            while (j * j > row) j--;
            while ((j + 1) * (j + 1) <= row) j++;
            int kk = row - j * j - j, ak = kk < 0 ? -kk : kk;
            double2 a[KT];
            _Pragma("unroll") for (int k = 0; k < KT; k++) a[k] = cmk(0, 0);
            if (KIND == 1) {
                double sg = ((j + ak) & 1) ? -1.0 : 1.0;
                for (int l = ak; l <= pin; l++) {
                    double c = sg * pw[l + j] * dc[(l + j) * lddc + (l - kk)] * dc[(l + j) * lddc + (l + kk)];
                    _Pragma("unroll") for (int k = 0; k < KT; k++) crfma(a[k], c, bB[(size_t)k * NC + eidx(l, kk)]);
                }
            } else if (KIND == 0) {
                double sc = ldexp(1.0, -j);
                for (int l = 0; l <= j - ak; l++) {
                    double c = ((l & 1) ? -sc : sc) * pw[l] * dc[(j - kk) * lddc + l] * dc[(j + kk) * lddc + l];
                    _Pragma("unroll") for (int k = 0; k < KT; k++) crfma(a[k], c, bB[(size_t)k * NC + eidx(j - l, kk)]);
                }
            } else {
                for (int l = 0; l <= p - j; l++) {
                    int ll = j + l;
                    double c = ldexp(1.0, -(ll + 1)) * pw[l] * dc[(ll + kk) * lddc + l] * dc[(ll - kk) * lddc + l];
                    _Pragma("unroll") for (int k = 0; k < KT; k++) crfma(a[k], c, bB[(size_t)k * NC + eidx(ll, kk)]);
                }
            }
            _Pragma("unroll") for (int k = 0; k < KT; k++) bA[(size_t)k * NC + row] = a[k];
        }
        __syncthreads();
        // phase 4 + 5: back rotation, times e^{-i m phi}, accumulate
        auto back = [&](int row, double2 *a) {
            int n = (int)sqrtf((float)row);
            while (n * n > row) n--;
            while ((n + 1) * (n + 1) <= row) n++;
            int m = row - n * n - n;
            const double *Dn = R + (size_t)n * (4 * n * n - 1) / 3 + (size_t)(m + n) * (2 * n + 1);
            _Pragma("unroll") for (int k = 0; k < KT; k++) a[k] = cmk(0, 0);
            for (int mp = -n; mp <= n; mp++) {
                double d = Dn[mp + n];
                _Pragma("unroll") for (int k = 0; k < KT; k++) crfma(a[k], d, bA[(size_t)k * NC + eidx(n, mp)]);
            }
            double2 ph = m >= 0 ? cconj(eph[m]) : eph[-m];
            _Pragma("unroll") for (int k = 0; k < KT; k++) a[k] = cmul(a[k], ph);
        };
        if (RPT > 0) {
#pragma unroll
            for (int j = 0; j < (RPT > 0 ? RPT : 1); j++) {
                const int row = threadIdx.x + kTransThreads * j;
                if (row < Rout) {
                    double2 a[KT];
                    back(row, a);
                    _Pragma("unroll") for (int k = 0; k < KT; k++)
                        if (sv[k] >= 0) racc[j][k] = cadd(racc[j][k], a[k]);
                }
            }
        } else {
            for (int row = threadIdx.x; row < Rout; row += kTransThreads) {
                double2 a[KT];
                back(row, a);
                _Pragma("unroll") for (int k = 0; k < KT; k++)
                    if (sv[k] >= 0) acc[(size_t)k * NC + row] = cadd(acc[(size_t)k * NC + row], a[k]);
            }
        }
    }
    __syncthreads();
    if (RPT > 0) {
#pragma unroll
        for (int j = 0; j < (RPT > 0 ? RPT : 1); j++) {
            const int e = threadIdx.x + kTransThreads * j;
            if (e >= NC) continue;
            _Pragma("unroll") for (int k = 0; k < KT; k++) {
                const int t = tg[k];
                if (t < 0) continue;
                double2 *o = out + (size_t)t * NC + e;
                if (KIND == 0) *o = racc[j][k];
                else *o = cadd(*o, racc[j][k]);
            }
        }
        return;
    }
    for (int i = threadIdx.x; i < KT * NC; i += kTransThreads) {
        int k = i / NC, e = i % NC;
        int t = tg[k];
        if (t < 0) continue;
        double2 *o = out + (size_t)t * NC + e;
        if (KIND == 0) *o = acc[i];
        else *o = cadd(*o, acc[i]);
    }
}

template <int KIND>
static void launch_translate_kind(const Tile *tiles, int ntiles, const int *grouped, const Slot *slots,
                                  const TreeView &tv, int p, const double *rot, const double *dc, int lddc,
                                  const double2 *in, double2 *out, int prune, int kt, size_t sm, cudaStream_t s,
                                  Status &st)
{
#define FMM_TR(KTV, RP)                                                                                       \
    do {                                                                                                      \
        FMM_TRY(st, smem_allow(k_translate<KIND, KTV, RP>, \
                                         (int)sm));                                                           \
        k_translate<KIND, KTV, RP><<<ntiles, kTransThreads, sm, s>>>(tiles, grouped, slots, tv, p, rot, dc, lddc, \
                                                                     in, out, prune); FMM_COUNT_LAUNCH();     \
    } while (0)
    if (KIND == 1 && kt == 8 && (p + 1) * (p + 1) <= 3 * kTransThreads) FMM_TR(8, 3);
    else if (kt == 8) FMM_TR(8, 0);
    else if (kt == 4) FMM_TR(4, 0);
    else if (kt == 2) FMM_TR(2, 0);
    else FMM_TR(1, 0);
#undef FMM_TR
}

void launch_translate(int kind, const Tile *tiles, int ntiles, const int *grouped, const Slot *slots,
                      const TreeView &tv, int p, const double *rot, const double *dc, int lddc,
                      const double2 *in, double2 *out, int prune, int kt, cudaStream_t s, Status &st)
{
    if (ntiles == 0 || !st.ok()) return;
    int NC = (p + 1) * (p + 1);
    // running sums in registers for M2L tiles of 8 targets at orders with at most 3 rows per thread
    const int nbuf = (kind == 1 && kt == 8 && NC <= 3 * kTransThreads) ? 2 : 3;
    size_t sm = (size_t)nbuf * kt * NC * sizeof(double2) + (p + 1) * sizeof(double2) + (2 * p + 4) * sizeof(double);
    if (kind == 0) launch_translate_kind<0>(tiles, ntiles, grouped, slots, tv, p, rot, dc, lddc, in, out, prune, kt, sm, s, st);
    else if (kind == 1) launch_translate_kind<1>(tiles, ntiles, grouped, slots, tv, p, rot, dc, lddc, in, out, prune, kt, sm, s, st);
    else launch_translate_kind<2>(tiles, ntiles, grouped, slots, tv, p, rot, dc, lddc, in, out, prune, kt, sm, s, st);
    FMM_LAUNCH_CHECK(st);
}

}  // namespace fmm
