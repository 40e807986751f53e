// Device octree build and interaction lists (see tree.cuh).
#include <algorithm>

#include "tree.cuh"

namespace fmm {

namespace {

// ---------------------------------------------------------------- bounding cube
// d3tallbem (src/d3tstrcr.f:1357-1395): min/max over sources and targets,
// size = largest extent, center = midpoints.
__global__ void k_bbox_partial(const double *src, int n, const double *trg, int m, double *part)
{
    double mn[3] = {1e308, 1e308, 1e308}, mx[3] = {-1e308, -1e308, -1e308};
    long tot = (long)n + m;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < tot; i += (long)gridDim.x * blockDim.x) {
        const double *p = i < n ? src + 3 * i : trg + 3 * (i - n);
        for (int d = 0; d < 3; d++) {
            double v = p[d];
            mn[d] = fmin(mn[d], v);
            mx[d] = fmax(mx[d], v);
        }
    }
    for (int d = 0; d < 3; d++) {
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fmin(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmax(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    }
    __shared__ double s[32][6];
    int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int d = 0; d < 3; d++) { s[w][d] = mn[d]; s[w][3 + d] = mx[d]; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int ww = 1; ww < (int)(blockDim.x >> 5); ww++)
            for (int d = 0; d < 3; d++) {
                s[0][d] = fmin(s[0][d], s[ww][d]);
                s[0][3 + d] = fmax(s[0][3 + d], s[ww][3 + d]);
            }
        for (int d = 0; d < 6; d++) part[6 * blockIdx.x + d] = s[0][d];
    }
}

// Reduces the per-block partials with one CTA (min / max are exact in any order).
__global__ void k_bbox_final(const double *part, int nb, double *geom /* c0x c0y c0z size */)
{
    double mn[3] = {1e308, 1e308, 1e308}, mx[3] = {-1e308, -1e308, -1e308};
    for (int b = threadIdx.x; b < nb; b += blockDim.x)
        for (int d = 0; d < 3; d++) {
            mn[d] = fmin(mn[d], part[6 * b + d]);
            mx[d] = fmax(mx[d], part[6 * b + 3 + d]);
        }
    for (int d = 0; d < 3; d++)
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fmin(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmax(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    __shared__ double sh[32][6];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int d = 0; d < 3; d++) { sh[w][d] = mn[d]; sh[w][3 + d] = mx[d]; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int ww = 1; ww < (int)(blockDim.x >> 5); ww++)
        for (int d = 0; d < 3; d++) {
            sh[0][d] = fmin(sh[0][d], sh[ww][d]);
            sh[0][3 + d] = fmax(sh[0][3 + d], sh[ww][3 + d]);
        }
    for (int d = 0; d < 3; d++) { mn[d] = sh[0][d]; mx[d] = sh[0][3 + d]; }
    double size = __dsub_rn(mx[0], mn[0]);
    double sy = __dsub_rn(mx[1], mn[1]), sz = __dsub_rn(mx[2], mn[2]);
    if (sy > size) size = sy;
    if (sz > size) size = sz;
    for (int d = 0; d < 3; d++) geom[d] = __dadd_rn(mn[d], mx[d]) / 2;
    geom[3] = size;
}

// Bounding cube of every instance of a forest: CTA per instance over its
// source range [so[i], so[i+1]) and target range [to[i], to[i+1]).
__global__ void k_bbox_inst(const double *src, const int *so, const double *trg, const int *to, double *geom)
{
    const int inst = blockIdx.x;
    double mn[3] = {1e308, 1e308, 1e308}, mx[3] = {-1e308, -1e308, -1e308};
    const long a = so[inst], ns = so[inst + 1] - a, b = to[inst], nt = to[inst + 1] - b;
    for (long i = threadIdx.x; i < ns + nt; i += blockDim.x) {
        const double *p = i < ns ? src + 3 * (a + i) : trg + 3 * (b + i - ns);
        for (int d = 0; d < 3; d++) {
            mn[d] = fmin(mn[d], p[d]);
            mx[d] = fmax(mx[d], p[d]);
        }
    }
    for (int d = 0; d < 3; d++)
        for (int o = 16; o > 0; o >>= 1) {
            mn[d] = fmin(mn[d], __shfl_xor_sync(0xffffffffu, mn[d], o));
            mx[d] = fmax(mx[d], __shfl_xor_sync(0xffffffffu, mx[d], o));
        }
    __shared__ double sh[32][6];
    int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int d = 0; d < 3; d++) { sh[w][d] = mn[d]; sh[w][3 + d] = mx[d]; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int ww = 1; ww < (int)(blockDim.x >> 5); ww++)
            for (int d = 0; d < 3; d++) {
                sh[0][d] = fmin(sh[0][d], sh[ww][d]);
                sh[0][3 + d] = fmax(sh[0][3 + d], sh[ww][3 + d]);
            }
        double size = __dsub_rn(sh[0][3], sh[0][0]);
        double sy = __dsub_rn(sh[0][4], sh[0][1]), sz = __dsub_rn(sh[0][5], sh[0][2]);
        if (sy > size) size = sy;
        if (sz > size) size = sz;
        for (int d = 0; d < 3; d++) geom[4 * inst + d] = __dadd_rn(sh[0][d], sh[0][3 + d]) / 2;
        geom[4 * inst + 3] = size;
    }
}

// instance id of every point of the concatenated arrays
__global__ void k_point_inst(const int *off, int *pinst)
{
    for (int i = off[blockIdx.x] + threadIdx.x; i < off[blockIdx.x + 1]; i += blockDim.x) pinst[i] = blockIdx.x;
}

// ---------------------------------------------------------------- keys
// Path key of a point: for every level the octant (z,y,x bits) it falls in,
// decided exactly as d3tsepa0 does (upper half iff coordinate > center) with
// the center computed as in d3tcentf (src/d3tstrcr.f:1671-1700):
// x0 + (i-1)*side + side/2, evaluated without contraction.
__global__ void k_keys(const double *pts, int n, const double *geom_all, const int *pinst, uint64_t *keys, int *idx)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *geom = geom_all + (pinst ? 4 * pinst[i] : 0);
    double size = geom[3];
    double h = size / 2;
    double x0[3] = {__dsub_rn(geom[0], h), __dsub_rn(geom[1], h), __dsub_rn(geom[2], h)};
    double p[3] = {pts[3L * i], pts[3L * i + 1], pts[3L * i + 2]};
    int c[3] = {0, 0, 0};
    uint64_t key = 0;
    for (int l = 0; l < kMaxLevel; l++) {
        // size / 2^l and side / 2 by exact power-of-two scaling (bitwise the same values)
        double side = ldexp(size, -l);
        double side2 = ldexp(side, -1);
        int oct = 0;
        for (int d = 0; d < 3; d++) {
            double ce = __dadd_rn(__dadd_rn(x0[d], __dmul_rn((double)c[d], side)), side2);
            int bit = p[d] > ce;
            c[d] = 2 * c[d] + bit;
            oct |= bit << d;
        }
        key = (key << 3) | (uint64_t)oct;
    }
    keys[i] = key;
    idx[i] = i;
}

__device__ __forceinline__ int key_digit(uint64_t key, int child_level)
{
    return (int)((key >> (3 * (kMaxLevel - child_level))) & 7);
}

// first index in [lo, hi) whose digit at child_level is >= d
__device__ int lower_digit(const uint64_t *keys, int lo, int hi, int child_level, int d)
{
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (key_digit(keys[mid], child_level) < d) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Boxes of every level on the device: first box and count, so that several
// levels can be built before the host reads the counts back.
struct LevelTable {
    int start[kMaxLevel + 2], count[kMaxLevel + 2];
    int total;   // children of the current level
    int over;    // level whose boxes did not fit the arrays (0: none)
    int want;    // and their number
    double geom[4];   // bounding cube of the (first) tree
};

// Split decision and child ranges for the boxes of one level
// (d3tallbem, src/d3tstrcr.f:1458-1578).  Sixteen threads per box: the
// fourteen digit boundaries (7 source, 7 target) are independent binary
// searches over the box's sorted range, done in parallel.
constexpr int kSplitLanes = 16;

__global__ void k_split(const LevelTable *L, int level, int nbox, TreeOptions opt, const int *src0, const int *nsrc,
                        const int *trg0, const int *ntrg, const uint64_t *ksrc, const uint64_t *ktrg, int *nkids,
                        int *cs0, int *cns, int *ct0, int *cnt)
{
    __shared__ int bound[128 / kSplitLanes][16];
    const int b0 = L->start[level], nb = L->count[level];
    const int g = threadIdx.x / kSplitLanes, j = threadIdx.x % kSplitLanes;
    const int t = blockIdx.x * (blockDim.x / kSplitLanes) + g;
    const bool live = t < nb;
    int s0 = 0, ns = 0, q0 = 0, nq = 0;
    bool split = false;
    if (live) {
        const int b = b0 + t;
        s0 = src0[b]; ns = nsrc[b]; q0 = trg0[b]; nq = ntrg[b];
        split = level < opt.maxlevel && (ns > nbox || nq > nbox || level < opt.minlevel);
        const int cl = level + 1;
        if (split && j >= 1 && j <= 7) bound[g][j] = lower_digit(ksrc, s0, s0 + ns, cl, j);
        if (split && j >= 9 && j <= 15) bound[g][j] = lower_digit(ktrg, q0, q0 + nq, cl, j - 8);
    }
    __syncthreads();
    if (!live || j != 0) return;
    int k = 0;
    if (split) {
        int sb[9], tb[9];
        sb[0] = s0; sb[8] = s0 + ns;
        tb[0] = q0; tb[8] = q0 + nq;
        for (int d = 1; d < 8; d++) {
            sb[d] = bound[g][d];
            tb[d] = bound[g][8 + d];
        }
        for (int d = 0; d < 8; d++) {
            cs0[8 * t + d] = sb[d];
            cns[8 * t + d] = sb[d + 1] - sb[d];
            ct0[8 * t + d] = tb[d];
            cnt[8 * t + d] = tb[d + 1] - tb[d];
            k += opt.ifempty == 1 || (sb[d + 1] > sb[d]) || (tb[d + 1] > tb[d]);
        }
    }
    nkids[t] = k;
}

__global__ void k_make_children(LevelTable *L, int level, int cap, int keep_empty, const int *kbase,
                                const int *nkids, const int *cs0, const int *cns, const int *ct0, const int *cnt,
                                const double *geom_all, int *ijk, int *lev, int *par, int *oct, int *nch,
                                int *child, int *src0, int *nsrc, int *trg0, int *ntrg, double *center, int *binst)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int b0 = L->start[level], nb = L->count[level], next0 = b0 + nb;
    const int total = nb > 0 ? L->total : 0;
    const bool fits = total <= cap - next0;
    if (t == 0) {
        L->start[level + 1] = next0;
        L->count[level + 1] = fits ? total : 0;
        if (!fits) {
            L->over = level + 1;
            L->want = total;
        }
    }
    if (t >= nb || !fits) return;
    int b = b0 + t;
    int id = next0 + kbase[t];
    nch[b] = nkids[t];
    if (nkids[t] == 0) return;
    const int inst = binst[b];
    const double *geom = geom_all + 4 * inst;
    double size = geom[3], h = size / 2;
    double side = size / (double)(1 << (level + 1)), side2 = side / 2;
    for (int d = 0; d < 8; d++) {
        int ns = cns[8 * t + d], nq = cnt[8 * t + d];
        if (ns == 0 && nq == 0 && !keep_empty) continue;
        int c[3] = {2 * ijk[3 * b] + (d & 1), 2 * ijk[3 * b + 1] + ((d >> 1) & 1), 2 * ijk[3 * b + 2] + ((d >> 2) & 1)};
        for (int e = 0; e < 3; e++) {
            ijk[3L * id + e] = c[e];
            // d3tcentc, src/d3tstrcr.f:1589-1669
            double x00 = __dsub_rn(geom[e], h);
            center[3L * id + e] = __dadd_rn(__dadd_rn(x00, __dmul_rn((double)c[e], side)), side2);
        }
        lev[id] = level + 1;
        binst[id] = inst;
        par[id] = b;
        oct[id] = d;
        nch[id] = 0;
        for (int e = 0; e < 8; e++) child[8L * id + e] = -1;
        src0[id] = cs0[8 * t + d];
        nsrc[id] = ns;
        trg0[id] = ct0[8 * t + d];
        ntrg[id] = nq;
        child[8L * b + d] = id;
        id++;
    }
}

// Root box of every instance (box id = instance id).
__global__ void k_root(int ninst, const int *so, const int *to, int n, int m, LevelTable *L, const double *geom, int *ijk, int *lev, int *par,
                       int *oct, int *nch, int *child, int *src0, int *nsrc, int *trg0, int *ntrg, double *center,
                       int *binst)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r == 0) {
        L->start[0] = 0;
        L->count[0] = ninst;
        L->over = L->want = 0;
        for (int e = 0; e < 4; e++) L->geom[e] = geom[e];
    }
    if (r >= ninst) return;
    for (int e = 0; e < 3; e++) { ijk[3 * r + e] = 0; center[3 * r + e] = geom[4 * r + e]; }
    lev[r] = 0; par[r] = -1; oct[r] = 0; nch[r] = 0; binst[r] = r;
    for (int e = 0; e < 8; e++) child[8 * r + e] = -1;
    // (one tree: the whole arrays)
    src0[r] = so ? so[r] : 0; nsrc[r] = so ? so[r + 1] - so[r] : n;
    trg0[r] = to ? to[r] : 0; ntrg[r] = to ? to[r + 1] - to[r] : m;
}

// ---------------------------------------------------------------- colleagues (list 5 plus self)
// One thread per (box, slot): the neighbour at offset d of a box with octant bits
// o lies in the parent's colleague at floor((o + d) / 2), child (o + d) mod 2.
__global__ void k_colleagues(int b0, int nb, const int *oct, const int *par, const int *child, int *coll)
{
    const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (t >= 27L * nb) return;
    const int b = b0 + (int)(t / 27), s = (int)(t % 27), P = par[b];
    int out = -1;
    if (P < 0) {
        out = s == 13 ? b : -1;
    } else {
        const int o = oct[b], d[3] = {s / 9 - 1, (s / 3) % 3 - 1, s % 3 - 1};
        int slot = 0, ch = 0;
        for (int e = 0; e < 3; e++) {
            const int pos = (o >> e & 1) + d[e];
            slot = slot * 3 + (pos >> 1) + 1;
            ch |= (pos & 1) << e;
        }
        const int C = coll[27L * P + slot];
        if (C >= 0) out = child[8L * C + ch];
    }
    coll[27L * b + s] = out;
}

// Closed boxes on (possibly different) levels intersect or touch: the
// integer form of d3tifint (src/d3tstrcr.f:1075-1172).
__device__ __forceinline__ bool touch(const int *ijk, const int *lev, int a, int b)
{
    int la = lev[a], lb = lev[b];
    if (la > lb) { int t = a; a = b; b = t; t = la; la = lb; lb = t; }
    long sc = 1L << (lb - la);
    for (int e = 0; e < 3; e++) {
        long ia = ijk[3L * a + e], ib = ijk[3L * b + e];
        if (ia * sc > ib + 1 || ib > (ia + 1) * sc) return false;
    }
    return true;
}

// Lists 1 and 3 of a childless non-root box b (d3tlsts/d3tlst31,
// src/d3tstrcr.f:827-851 and :912-1069).  List 1 = childless boxes that
// touch b (any level); list 3 = boxes on finer levels that do not touch b
// but whose parents do.  One warp per box: lane s walks the boxes below
// colleague s, then the lanes take the ancestors' colleagues (childless boxes on
// coarser levels are colleagues of an ancestor); entries in the order of the
// slots.  FILL 0 counts (n1, n3 and the leaf flag of every box, zeros in the
// entry past the end), 1 writes and counts the dual of list 3, list 4.
template <int FILL>
__device__ __forceinline__ void walk_below(int b, int C, const int *ijk, const int *lev, const int *nch,
                                           const int *child, int &c1, int &c3, int *i1, int *i3, int *n4)
{
    if (nch[C] == 0) {
        if (FILL) i1[c1] = C;
        c1++;
        return;
    }
    int stk[8 * kMaxLevel + 8], top = 0;
    for (int d = 7; d >= 0; d--)
        if (child[8L * C + d] >= 0) stk[top++] = child[8L * C + d];
    while (top) {
        const int x = stk[--top];
        if (!touch(ijk, lev, b, x)) {
            if (FILL) {
                i3[c3] = x;
                atomicAdd(&n4[x], 1);
            }
            c3++;
        } else if (nch[x] == 0) {
            if (FILL) i1[c1] = x;
            c1++;
        } else {
            for (int d = 7; d >= 0; d--)
                if (child[8L * x + d] >= 0) stk[top++] = child[8L * x + d];
        }
    }
}

template <int FILL>
__global__ void __launch_bounds__(128) k_lists13(int nboxes, const int *ijk, const int *lev, const int *par,
                                                 const int *nch, const int *child, const int *coll, int *n1, int *n3,
                                                 int *flag, const int *s1, int *i1, const int *s3, int *i3, int *n4)
{
    const int b = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (b > nboxes) return;
    if (b == nboxes || nch[b] != 0) {
        if (!FILL && lane == 0) {
            n1[b] = n3[b] = 0;
            if (b < nboxes) flag[b] = 0;
        }
        return;
    }
    const int C = lane < 27 && lane != 13 ? coll[27L * b + lane] : -1;
    int c1 = 0, c3 = 0;
    if (C >= 0) walk_below<0>(b, C, ijk, lev, nch, child, c1, c3, nullptr, nullptr, nullptr);
    int p1 = c1, p3 = c3;   // inclusive sums over the lanes
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, p1, o), v = __shfl_up_sync(0xffffffffu, p3, o);
        if (lane >= o) { p1 += u; p3 += v; }
    }
    int t1 = __shfl_sync(0xffffffffu, p1, 31);
    const int t3 = __shfl_sync(0xffffffffu, p3, 31);
    if (FILL && C >= 0) {
        int k1 = 0, k3 = 0;
        walk_below<1>(b, C, ijk, lev, nch, child, k1, k3, i1 + s1[b] + p1 - c1, i3 + s3[b] + p3 - c3, n4);
    }
    for (int A = par[b]; A >= 0 && lev[A] >= 1; A = par[A]) {
        const int D = lane < 27 && lane != 13 ? coll[27L * A + lane] : -1;
        const bool in = D >= 0 && nch[D] == 0 && touch(ijk, lev, b, D);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (FILL && in) i1[s1[b] + t1 + __popc(m & ((1u << lane) - 1))] = D;
        t1 += __popc(m);
    }
    if (!FILL && lane == 0) {
        n1[b] = t1;
        n3[b] = t3;
        flag[b] = 1;
    }
}

__global__ void k_list4_fill(const int *leaves, int nleaves, const int *s3, const int *i3, int *cursor, int *i4)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nleaves) return;
    int b = leaves[t];
    for (int k = s3[b]; k < s3[b + 1]; k++) i4[atomicAdd(&cursor[i3[k]], 1)] = b;
}

// deterministic order inside each list-4 row
__global__ void k_sort_rows(int nb, const int *st, int *idx)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    int lo = st[b], hi = st[b + 1];
    for (int i = lo + 1; i < hi; i++) {
        int v = idx[i], j = i - 1;
        while (j >= lo && idx[j] > v) { idx[j + 1] = idx[j]; j--; }
        idx[j + 1] = v;
    }
}

__global__ void k_compact(int nb, const int *flag, const int *pos, int *out)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b < nb && flag[b]) out[pos[b]] = b;
}

__global__ void k_group_keys(int nb, const int *lev, const int *oct, uint64_t *keys, int *vals)
{
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    keys[b] = (uint64_t)(lev[b] * 8 + oct[b]);
    vals[b] = b;
}

__global__ void k_group_bounds(int nb, const uint64_t *keys, int ngroups, int *gstart)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > nb) return;
    int g0 = i == 0 ? 0 : (int)keys[i - 1] + 1;
    int g1 = i == nb ? ngroups : (int)keys[i];
    for (int g = g0; g <= g1 && g <= ngroups; g++) gstart[g] = i;
}

template <typename T>
bool grow(DBuf<T> &b, size_t need, size_t copy, cudaStream_t s, Status &st)
{
    if (b.n >= need) return true;
    DBuf<T> nb;
    if (!nb.alloc(need, s, st)) return false;
    if (copy) FMM_TRY(st, cudaMemcpyAsync(nb.p, b.p, sizeof(T) * copy, cudaMemcpyDeviceToDevice, s));
    std::swap(b.p, nb.p);
    std::swap(b.n, nb.n);
    std::swap(b.s, nb.s);
    return st.ok();
}

// Levels whose key bits the first sort covers (3 (21 - 13) = 24 bits left out).
constexpr int kSortedLevel = 13;

// Stable reorder of (key, perm) into instance-major order: sort by the
// instance of each point (gathered through perm), carrying the position,
// then gather keys and perm by the resulting order.
__global__ void k_gather_inst(int n, const int *perm, const int *pinst, uint64_t *ikey, int *pos)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ikey[i] = (uint64_t)pinst[perm[i]];
    pos[i] = i;
}

__global__ void k_apply_pos(int n, const int *pos, const uint64_t *kin, const int *pin, uint64_t *kout, int *pout)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    kout[i] = kin[pos[i]];
    pout[i] = pin[pos[i]];
}

void instance_major(DBuf<uint64_t> &keys, DBuf<int> &perm, const DBuf<int> &pinst, int n, int ibits,
                    cudaStream_t s, Status &st)
{
    if (n == 0 || !st.ok()) return;
    DBuf<uint64_t> ik, k2;
    DBuf<int> pos, p2;
    if (!ik.alloc(n, s, st) || !pos.alloc(n, s, st) || !k2.alloc(n, s, st) || !p2.alloc(n, s, st)) return;
    k_gather_inst<<<div_up(n, 256), 256, 0, s>>>(n, perm.p, pinst.p, ik.p, pos.p); FMM_COUNT_LAUNCH();
    radix_sort_pair(ik, pos, n, nullptr, nullptr, 0, 0, ibits, s, st);
    k_apply_pos<<<div_up(n, 256), 256, 0, s>>>(n, pos.p, keys.p, perm.p, k2.p, p2.p); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
    std::swap(keys.p, k2.p);
    std::swap(keys.n, k2.n);
    std::swap(perm.p, p2.p);
    std::swap(perm.n, p2.n);
}

}  // namespace

void build_tree(Tree &T, const double *d_src, int n, const double *d_trg, int m, int nbox, cudaStream_t s,
                Status &st, const TreeOptions &opt)
{
    std::vector<int> so = {0, n}, to = {0, m};
    build_forest(T, d_src, so, d_trg, to, nbox, s, st, opt);
}

void build_forest(Tree &T, const double *d_src, const std::vector<int> &so, const double *d_trg,
                  const std::vector<int> &to, int nbox, cudaStream_t s, Status &st, const TreeOptions &opt_in)
{
    TreeOptions opt = opt_in;
    opt.ifempty = opt.ifempty == 1;
    opt.minlevel = std::max(0, std::min(opt.minlevel, kMaxLevel));
    opt.maxlevel = std::max(0, std::min(opt.maxlevel, kMaxLevel));
    T.nbox = nbox;
    const int ninst = (int)so.size() - 1;
    const int n = so[ninst], m = to[ninst];
    T.n = n;
    T.m = m;
    T.ninst = ninst;
    // bounding cube of every instance
    DBuf<double> part, &geom = T.inst_geom;
    DBuf<int> dso, dto, pis, pit;
    geom.alloc(4L * ninst, s, st);
    if (!st.ok()) return;
    if (ninst == 1) {
        int nbb = std::max(1, std::min(1184, div_up((long)n + m, 256)));
        part.alloc(6 * nbb, s, st);
        if (!st.ok()) return;
        k_bbox_partial<<<nbb, 256, 0, s>>>(d_src, n, d_trg, m, part.p); FMM_COUNT_LAUNCH();
        k_bbox_final<<<1, 256, 0, s>>>(part.p, nbb, geom.p); FMM_COUNT_LAUNCH();
    } else {
        if (!dso.alloc(ninst + 1, s, st) || !dto.alloc(ninst + 1, s, st) || !pis.alloc(std::max(n, 1), s, st) ||
            !pit.alloc(std::max(m, 1), s, st))
            return;
        FMM_TRY(st, cudaMemcpyAsync(dso.p, so.data(), sizeof(int) * (ninst + 1), cudaMemcpyHostToDevice, s));
        FMM_TRY(st, cudaMemcpyAsync(dto.p, to.data(), sizeof(int) * (ninst + 1), cudaMemcpyHostToDevice, s));
        k_bbox_inst<<<ninst, 256, 0, s>>>(d_src, dso.p, d_trg, dto.p, geom.p); FMM_COUNT_LAUNCH();
        k_point_inst<<<ninst, 256, 0, s>>>(dso.p, pis.p); FMM_COUNT_LAUNCH();
        k_point_inst<<<ninst, 256, 0, s>>>(dto.p, pit.p); FMM_COUNT_LAUNCH();
    }
    // keys and sort: by path key, then (forests) stably by instance
    DBuf<uint64_t> ks, kt;
    ks.alloc(std::max(n, 1), s, st);
    kt.alloc(std::max(m, 1), s, st);
    T.perm_src.alloc(std::max(n, 1), s, st);
    T.perm_trg.alloc(std::max(m, 1), s, st);
    if (!st.ok()) return;
    if (n) { k_keys<<<div_up(n, 256), 256, 0, s>>>(d_src, n, geom.p, ninst > 1 ? pis.p : nullptr, ks.p, T.perm_src.p); FMM_COUNT_LAUNCH(); }
    if (m) { k_keys<<<div_up(m, 256), 256, 0, s>>>(d_trg, m, geom.p, ninst > 1 ? pit.p : nullptr, kt.p, T.perm_trg.p); FMM_COUNT_LAUNCH(); }
    FMM_LAUNCH_CHECK(st);
    // The bits of the first kSortedLevel levels only: five passes instead of eight (a
    // deeper tree sorts again by all bits before it splits below that level).
    auto sort_keys = [&](int low) {
        radix_sort_pair(ks, T.perm_src, n, &kt, &T.perm_trg, m, low, 3 * kMaxLevel, s, st);
        if (ninst > 1) {
            int ibits = 8;
            while ((1L << ibits) < ninst) ibits += 8;
            instance_major(ks, T.perm_src, pis, n, ibits, s, st);
            instance_major(kt, T.perm_trg, pit, m, ibits, s, st);
        }
    };
    sort_keys(3 * (kMaxLevel - kSortedLevel));
    // boxes
    int cap = std::max(1024, 2 * (int)(((long)n + m) / std::max(nbox, 1)) + 64 + 2 * ninst);
    auto ensure = [&](int need, int used) {
        if (need <= T.cap) return st.ok();
        int nc = std::max(need, 2 * T.cap);
        grow(T.ijk, 3L * nc, 3L * used, s, st);
        grow(T.level, nc, used, s, st);
        grow(T.parent, nc, used, s, st);
        grow(T.octant, nc, used, s, st);
        grow(T.nchild, nc, used, s, st);
        grow(T.child, 8L * nc, 8L * used, s, st);
        grow(T.src0, nc, used, s, st);
        grow(T.nsrc, nc, used, s, st);
        grow(T.trg0, nc, used, s, st);
        grow(T.ntrg, nc, used, s, st);
        grow(T.center, 3L * nc, 3L * used, s, st);
        grow(T.binst, nc, used, s, st);
        T.cap = nc;
        return st.ok();
    };
    T.cap = 0;
    if (!ensure(cap, 0)) return;
    DBuf<LevelTable> dlev;
    DBuf<int> rso, rto;
    if (!dlev.alloc(1, s, st)) return;
    if (ninst > 1) {
        if (!rso.alloc(ninst + 1, s, st) || !rto.alloc(ninst + 1, s, st)) return;
        // root ranges in sorted order: instances are contiguous and in order
        FMM_TRY(st, cudaMemcpyAsync(rso.p, so.data(), sizeof(int) * (ninst + 1), cudaMemcpyHostToDevice, s));
        FMM_TRY(st, cudaMemcpyAsync(rto.p, to.data(), sizeof(int) * (ninst + 1), cudaMemcpyHostToDevice, s));
    }
    k_root<<<div_up(ninst, 128), 128, 0, s>>>(ninst, rso.p, rto.p, n, m, dlev.p, geom.p, T.ijk.p, T.level.p, T.parent.p,
                                              T.octant.p, T.nchild.p, T.child.p, T.src0.p, T.nsrc.p, T.trg0.p,
                                              T.ntrg.p, T.center.p, T.binst.p); FMM_COUNT_LAUNCH();
    if (ninst > 1) FMM_TRY(st, cudaStreamSynchronize(s));  // the host range vectors are read by the copies above
    T.lev_start.assign(1, 0);
    T.lev_count.assign(1, ninst);
    int nboxes = ninst;
    DBuf<int> nk, kb, cs0, cns, ct0, cnt;
    size_t ncap = 0;
    auto scratch = [&](size_t need) {
        if (need <= ncap) return true;
        ncap = need;
        return nk.alloc(need, s, st) && kb.alloc(need, s, st) && cs0.alloc(8 * need, s, st) && cns.alloc(8 * need, s, st) &&
               ct0.alloc(8 * need, s, st) && cnt.alloc(8 * need, s, st);
    };
    // Several levels are built between two reads of their counts: as many as a uniform
    // volume of points needs and one more, then two at a time (a read costs about
    // as much as the kernels of two small levels).  With arrays too long for the one-CTA scan the
    // exact count of each level is read.
    int ahead = 2;
    for (double c = (double)std::max(n, m) / std::max(nbox, 1) / ninst; c > 1; c /= 8) ahead++;
    bool sorted_all = false;
    LevelTable hl;
    for (int level = 0; level < kMaxLevel;) {
        const bool blind = T.cap <= 65536;
        int last = std::min(level + (blind ? ahead : 1), kMaxLevel);
        if (!sorted_all && last > kSortedLevel) {
            if (level >= kSortedLevel) {
                sort_keys(0);
                sorted_all = true;
            } else {
                last = kSortedLevel;
            }
        }
        for (int q = level; q < last; q++) {
            long bound = T.lev_count[level];
            for (int k = level; k < q && bound < T.cap; k++) bound *= 8;
            bound = std::min(bound, (long)T.cap);
            if (!scratch(blind ? T.cap : bound)) return;
            k_split<<<div_up(bound, 128 / kSplitLanes), 128, 0, s>>>(dlev.p, q, nbox, opt, T.src0.p, T.nsrc.p, T.trg0.p,
                                                                   T.ntrg.p, ks.p, kt.p, nk.p, cs0.p, cns.p, ct0.p,
                                                                   cnt.p); FMM_COUNT_LAUNCH();
            FMM_LAUNCH_CHECK(st);
            const ScanJob job = {nk.p, kb.p, (int)bound, blind ? &dlev.p->count[q] : nullptr};
            scan_exclusive_multi(&job, 1, &dlev.p->total, s, st);
            k_make_children<<<div_up(bound, 128), 128, 0, s>>>(dlev.p, q, T.cap, opt.ifempty, kb.p, nk.p, cs0.p, cns.p,
                                                              ct0.p, cnt.p, geom.p, T.ijk.p, T.level.p, T.parent.p,
                                                              T.octant.p, T.nchild.p, T.child.p, T.src0.p, T.nsrc.p,
                                                              T.trg0.p, T.ntrg.p, T.center.p, T.binst.p);
            FMM_COUNT_LAUNCH();
            FMM_LAUNCH_CHECK(st);
        }
        FMM_TRY(st, cudaMemcpyAsync(&hl, dlev.p, sizeof(hl), cudaMemcpyDeviceToHost, s));
        FMM_TRY(st, cudaStreamSynchronize(s));
        if (!st.ok()) return;
        bool done = false;
        for (int q = level; q < last; q++) {
            if (hl.over == q + 1) {
                // the arrays were too short: grow them and build this level again
                if (!ensure(nboxes + hl.want, nboxes)) return;
                FMM_TRY(st, cudaMemsetAsync(&dlev.p->over, 0, sizeof(int), s));
                last = q;
                break;
            }
            if (hl.count[q + 1] == 0) { done = true; break; }
            T.lev_start.push_back(nboxes);
            T.lev_count.push_back(hl.count[q + 1]);
            nboxes += hl.count[q + 1];
        }
        if (done) break;
        level = last;
        ahead = 2;
    }
    T.nboxes = nboxes;
    T.nlev = (int)T.lev_start.size() - 1;
    T.capped = 0;
    if (opt_in.maxlevel > kMaxLevel && T.nlev == kMaxLevel && st.ok()) {
        const int b0 = T.lev_start[kMaxLevel], nb = T.lev_count[kMaxLevel];
        std::vector<int> hs(nb), ht(nb);
        FMM_TRY(st, cudaMemcpyAsync(hs.data(), T.nsrc.p + b0, sizeof(int) * nb, cudaMemcpyDeviceToHost, s));
        FMM_TRY(st, cudaMemcpyAsync(ht.data(), T.ntrg.p + b0, sizeof(int) * nb, cudaMemcpyDeviceToHost, s));
        FMM_TRY(st, cudaStreamSynchronize(s));
        for (int i = 0; i < nb && st.ok(); i++) T.capped += (hs[i] > nbox || ht[i] > nbox) ? 1 : 0;
    }
    for (int d = 0; d < 3; d++) T.center0[d] = hl.geom[d];
    T.size = hl.geom[3];

    // colleagues, level by level
    T.coll.alloc(27L * nboxes, s, st);
    if (!st.ok()) return;
    for (int l = 0; l <= T.nlev; l++) {
        k_colleagues<<<div_up(27L * T.lev_count[l], 256), 256, 0, s>>>(T.lev_start[l], T.lev_count[l], T.octant.p,
                                                                      T.parent.p, T.child.p, T.coll.p);
        FMM_COUNT_LAUNCH();
    }
    FMM_LAUNCH_CHECK(st);

    // leaves and lists 1 and 3 (count, scan, fill), list 4 as the dual of list 3
    DBuf<int> flag, pos, n1, n3, n4, cur, tot;
    flag.alloc(nboxes, s, st);
    pos.alloc(nboxes, s, st);
    n1.alloc(nboxes + 1, s, st);
    n3.alloc(nboxes + 1, s, st);
    n4.alloc(nboxes + 1, s, st);
    cur.alloc(nboxes + 1, s, st);
    tot.alloc(3, s, st);
    T.l1_start.alloc(nboxes + 1, s, st);
    T.l3_start.alloc(nboxes + 1, s, st);
    T.l4_start.alloc(nboxes + 1, s, st);
    if (!st.ok()) return;
    n4.zero(st);
    k_lists13<0><<<div_up(nboxes + 1, 4), 128, 0, s>>>(nboxes, T.ijk.p, T.level.p, T.parent.p, T.nchild.p, T.child.p,
                                                      T.coll.p, n1.p, n3.p, flag.p, nullptr, nullptr, nullptr, nullptr,
                                                      nullptr); FMM_COUNT_LAUNCH();
    const ScanJob jobs[3] = {{flag.p, pos.p, nboxes, nullptr},
                             {n1.p, T.l1_start.p, nboxes + 1, nullptr},
                             {n3.p, T.l3_start.p, nboxes + 1, nullptr}};
    scan_exclusive_multi(jobs, 3, tot.p, s, st);
    int h[3] = {0, 0, 0};   // leaves, entries of lists 1 and 3
    FMM_TRY(st, cudaMemcpyAsync(h, tot.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    FMM_TRY(st, cudaStreamSynchronize(s));
    const int nleaves = T.nleaves = h[0];
    T.leaves.alloc(std::max(nleaves, 1), s, st);
    T.l1_idx.alloc(std::max(h[1], 1), s, st);
    T.l3_idx.alloc(std::max(h[2], 1), s, st);
    T.l4_idx.alloc(std::max(h[2], 1), s, st);
    if (!st.ok()) return;
    k_compact<<<div_up(nboxes, 256), 256, 0, s>>>(nboxes, flag.p, pos.p, T.leaves.p); FMM_COUNT_LAUNCH();
    k_lists13<1><<<div_up(nboxes + 1, 4), 128, 0, s>>>(nboxes, T.ijk.p, T.level.p, T.parent.p, T.nchild.p, T.child.p,
                                                      T.coll.p, nullptr, nullptr, nullptr, T.l1_start.p, T.l1_idx.p,
                                                      T.l3_start.p, T.l3_idx.p, n4.p); FMM_COUNT_LAUNCH();
    const ScanJob jobs4[2] = {{n4.p, T.l4_start.p, nboxes + 1, nullptr}, {n4.p, cur.p, nboxes + 1, nullptr}};
    scan_exclusive_multi(jobs4, 2, nullptr, s, st);
    if (h[2] > 0) {
        k_list4_fill<<<div_up(nleaves, 128), 128, 0, s>>>(T.leaves.p, nleaves, T.l3_start.p, T.l3_idx.p, cur.p,
                                                          T.l4_idx.p); FMM_COUNT_LAUNCH();
        k_sort_rows<<<div_up(nboxes, 128), 128, 0, s>>>(nboxes, T.l4_start.p, T.l4_idx.p); FMM_COUNT_LAUNCH();
    }
    FMM_LAUNCH_CHECK(st);

    // boxes grouped by (level, octant)
    int ngroups = (T.nlev + 1) * 8;
    DBuf<uint64_t> gk;
    DBuf<int> gs;
    gk.alloc(nboxes, s, st);
    T.grouped.alloc(nboxes, s, st);
    gs.alloc(ngroups + 1, s, st);
    if (!st.ok()) return;
    k_group_keys<<<div_up(nboxes, 256), 256, 0, s>>>(nboxes, T.level.p, T.octant.p, gk.p, T.grouped.p); FMM_COUNT_LAUNCH();
    int gbits = 8;
    while ((1 << gbits) < ngroups + 1) gbits += 8;
    radix_sort_pair(gk, T.grouped, nboxes, nullptr, nullptr, 0, 0, gbits, s, st);
    if (!st.ok()) return;
    k_group_bounds<<<div_up(nboxes + 1, 256), 256, 0, s>>>(nboxes, gk.p, ngroups, gs.p); FMM_COUNT_LAUNCH();
    T.group_start.assign(ngroups + 1, 0);
    FMM_TRY(st, cudaMemcpyAsync(T.group_start.data(), gs.p, sizeof(int) * (ngroups + 1), cudaMemcpyDeviceToHost, s));
    FMM_TRY(st, cudaStreamSynchronize(s));
}

}  // namespace fmm
