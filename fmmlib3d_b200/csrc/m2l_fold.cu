// M2L by dense operators folded over the reflections of the list-2 offsets.
//
// The translation of a list-2 offset D (l3dmplocquad2_trunc0,
// src/l3dtrans.f:1260-1387, truncated to nterms_trunc = pt) is a linear map
// T_D of the source coefficients.  Two symmetries make it cheap:
//   - in the real basis A = (M_n^m + M_n^{-m}) / 2 (cosine part) and
//     B = (M_n^m - M_n^{-m}) / 2i (sine part) T_D is a real matrix, and the
//     real and imaginary parts of the strengths are two right-hand sides;
//   - every real harmonic is even or odd under x -> -x, y -> -y and z -> -z.
//     With the coefficients in 8 parity classes, a reflection g of D only
//     changes signs, T_{gD}[a][b] = chi_a(g) chi_b(g) T_D[a][b], so the sources
//     of a target at all reflections of D are added first,
//       X[c][b] = sum_g chi_c(g) M_{gD}[b],
//     and L[a] += sum_b T_D[a][b] X[a ^ b][b] once for all of them.
// The 189 offsets of a target fall into 56 classes |D|; a zero component of D
// leaves only the blocks with equal parity on that axis.  At order 14
// that is 0.57 M multiply-adds per target against 7.95 M for one complex
// operator per offset; at order 26 6.8 M against 7.6 M of rotate-shift-
// rotate, all of them in matrix products.
//
// k_m2l_fold: a CTA owns 16 consecutive target boxes (32 columns: 16 targets x
// 2 right-hand sides; 8 at order 26) and all their coefficients; warp w < 8 owns the rows of
// parity class w in DMMA accumulators.  Per
// batch other warps stage X (32 rows per parity class, 74 KB, two buffers) and bring
// the batch's operator fragments into L1; each
// warp multiplies its fragments, in the lane order of the MMA and each used for
// all 32 columns, with its rows.  Offset classes
// that no target of the tile has a source in are skipped.
// The sums of a target are formed in 8 fixed groups of batches, added in
// order; a small problem, or one above order 15, runs one CTA per (tile, group) and
// adds the groups afterwards, with the same result bit for bit.
//
// Bound: latency of the fragments and source rows in L2 (DMMA pipe 30% busy, long
// scoreboard half of the stalls).  M2L pass, one B200, against the dense product per
// offset that it replaced (orders <= 16) and rotate-shift-rotate (order 26):
//   cube 2M + 2M, order 14   33.2 -> 6.0 ms     10k sphere, order 14    1.8 -> 0.07 ms
//   100k sphere, order 14    2.6 -> 0.29 ms     cube 1M + 1M, order 26  11.5 -> 4.5 ms
//   328k triangles, order 14 39.6 -> 8.3 ms
// On the way: staging and products by the same 16 warps in turn 9.2 ms at the 2M cube;
// staging by warps of their own 8.15; the next batch's fragments to L1 ahead of use 6.0.
// (Fragments fetched into registers ahead: spills, 10.9 ms; raw rows by cp.async: 10.1.)
#include <algorithm>

#include "dmma.cuh"
#include "m2l_fold.cuh"

namespace fmm {

constexpr int kFoldCap = 32;                    // operand rows per parity class and batch
// Row stride of the operands of NT targets: = 4 mod 16 doubles, so that the 4 x 4
// lanes of a half warp reading a fragment meet different banks.
template <int NT>
constexpr int kFoldLd = 2 * NT + 4;
// Fewer tiles than two for each multiprocessor: one CTA per group.  M2L at 148, one
// CTA per tile against one per (tile, group): 4 tiles 0.35 / 0.062 ms, 111 tiles 0.36 /
// 0.29, 292 tiles 0.78 / 0.80, 1,390 tiles 3.42 / 3.58, 2,330 tiles 6.0 / 6.5.
// Tiles of 8 targets (above order 15, one CTA per multiprocessor) always run per group: eight
// times the CTAs even out the tiles at a domain's faces.  Order 26: 585 tiles 4.83 /
// 4.53, 4,681 tiles 38.9 / 35.7, with the groups' sums held to 256 MB at a time.
static bool fold_split(const FoldPlan &F, int count)
{
    return F.tile == 8 || div_up(count, F.tile) < 2 * device_sms();
}

// ---------------------------------------------------------------- operators
struct FoldBlock {
    long long off;
    int k4, rb, off_id, alpha, beta, na, nb, k0;
};

// T_D[(j, m)][(n, mc)] = e^{i (mc - m) phi} sum_k D^j[m][k] Z(j, k, n) D^n[mc][k],
// Z(j, k, n) = (-1)^(j+k) sqrt(C(n+j, n-k) C(n+j, n+k)) / rt^(n+j+1).
__device__ double2 fold_entry(const FoldOffset &o, const double *Rm, const double *dc, int lddc, int j, int m, int n,
                              int mc)
{
    const double *Dn = Rm + (size_t)n * (4 * n * n - 1) / 3 + (size_t)(mc + n) * (2 * n + 1);
    const double *Dj = Rm + (size_t)j * (4 * j * j - 1) / 3 + (size_t)(m + j) * (2 * j + 1);
    const double ir = 1.0 / o.rt;
    double pw = 1;
    for (int i = 0; i < n + j + 1; i++) pw *= ir;
    const int kmax = j < n ? j : n;
    double s = 0;
    for (int k = -kmax; k <= kmax; k++) {
        const double z = (((j + k) & 1) ? -1.0 : 1.0) * pw * dc[(n + j) * lddc + (n - k)] * dc[(n + j) * lddc + (n + k)];
        s += Dj[k + j] * z * Dn[k + n];
    }
    const int d = mc - m;
    double2 e = cmk(1, 0);
    for (int i = 0; i < (d < 0 ? -d : d); i++) e = cmul(e, cmk(o.ex, o.ey));
    if (d < 0) e = cconj(e);
    return cscal(s, e);
}

// One thread per fragment entry: blocks (offset class, row class, column
// class) as K steps x row blocks x 32 lanes.
__global__ void k_fold_ops(const FoldBlock *blocks, const FoldOffset *offs, const int4 *kmap, const int *base, int p,
                           const double *rot, const double *dc, int lddc, double *A)
{
    const FoldBlock B = blocks[blockIdx.x];
    const FoldOffset o = offs[B.off_id];
    const double *Rm = rot + rot_class_size(p) * o.cls;
    for (int e = threadIdx.x; e < B.k4 * B.rb * 32; e += blockDim.x) {
        const int lane = e & 31, rb = (e >> 5) % B.rb, ks = (e >> 5) / B.rb;
        const int row = rb * 8 + (lane >> 2), col = B.k0 + ks * 4 + (lane & 3);
        double v = 0;
        if (row < B.na && col < B.nb) {
            const int4 r = kmap[base[B.alpha] + row], c = kmap[base[B.beta] + col];
            int j = 0, n = 0;
            while ((j + 1) * (j + 1) <= r.x) j++;
            while ((n + 1) * (n + 1) <= c.x) n++;
            const int m = r.x - j * j - j, mc = c.x - n * n - n;
            const double2 t1 = fold_entry(o, Rm, dc, lddc, j, m, n, mc);
            const double2 t2 = mc > 0 ? fold_entry(o, Rm, dc, lddc, j, m, n, -mc) : cmk(0, 0);
            // the reality of the map, T[-m][-mc] = conj T[m][mc], gives the four parts
            if (!r.z) v = c.z ? t2.y - t1.y : t1.x + t2.x;
            else v = c.z ? t1.x - t2.x : t1.y + t2.y;
        }
        A[B.off + e] = v;
    }
}

bool fold_build(FoldPlan &F, int p, const FoldOffset *off, const double *rot, const double *dc, int lddc,
                cudaStream_t s, Status &st)
{
    F.p = p;
    F.K = (p + 1) * (p + 1);
    // parity classes: bit 0 odd in x, bit 1 odd in y (sine parts), bit 2 odd in z; by degree inside a class
    std::vector<int4> kmap, rmap;
    std::vector<int> base(16);
    std::vector<std::vector<int>> cnt(8, std::vector<int>(p + 1, 0));   // coefficients of degree <= n
    std::vector<int> kc((size_t)(p + 1) * (p + 1), -1), ksn((size_t)(p + 1) * (p + 1), -1);
    for (int c = 0; c < 8; c++) {
        base[c] = (int)kmap.size();
        for (int n = 0; n <= p; n++) {
            const int sine = (c >> 1) & 1;
            for (int m = sine; m <= n; m++) {
                if (((m + sine) & 1) != (c & 1) || ((n + m) & 1) != (c >> 2)) continue;
                (sine ? ksn : kc)[n * (p + 1) + m] = (int)kmap.size();
                kmap.push_back(make_int4(eidx(n, m), eidx(n, -m), sine, m));
            }
            cnt[c][n] = (int)kmap.size() - base[c];
        }
        base[8 + c] = cnt[c][p];
        F.rows = std::max(F.rows, div_up(cnt[c][p], 8));
    }
    for (int n = 0; n <= p; n++)
        for (int m = 0; m <= n; m++)
            rmap.push_back(make_int4(eidx(n, m), eidx(n, -m), kc[n * (p + 1) + m], m ? ksn[n * (p + 1) + m] : -1));

    // Segments (offset class, round of column classes, K range) packed into batches.  The
    // segments of one offset class in a batch are a run: their operand rows follow each other in
    // every parity class's slot, and so do the K steps of its operator fragments, so
    // that a warp multiplies a run in one loop.
    F.tile = F.rows <= 5 ? 16 : 8;
    std::vector<FoldBlock> blocks;
    std::vector<int4> cls;
    std::vector<FoldTask> tasks;
    std::vector<FoldBatch> batches;
    std::vector<int2> runs;
    std::vector<double> cost;
    long long tot = 0;
    int fill = 0;
    struct Seg { int rb, k0, depth; };
    std::vector<Seg> open_;
    int open_cls = -1, open_row = 0;
    auto close_run = [&]() {
        if (open_.empty()) return;
        const FoldOffset &o = off[open_cls];
        const int z = 7 ^ cls[open_cls].w;
        int depth = 0;
        double most = 0;
        for (const Seg &g : open_) depth += g.depth;
        for (int al = 0; al < 8; al++) {
            const int na = cnt[al][o.pt], rb = div_up(na, 8);
            runs.push_back(na ? make_int2((int)(tot / 32), depth / 4 | rb << 4 | open_row << 8 | open_cls << 16)
                              : make_int2(0, open_cls << 16));
            if (!na) continue;
            for (const Seg &g : open_) {
                const int be = (al & z) | g.rb;
                FoldBlock b;
                b.off = tot; b.k4 = g.depth / 4; b.rb = rb; b.off_id = open_cls; b.alpha = al; b.beta = be; b.na = na;
                b.nb = cnt[be][o.pt]; b.k0 = g.k0;
                blocks.push_back(b);
                tot += (long long)b.k4 * b.rb * 32;
            }
            most = std::max(most, depth / 4.0 * rb);
        }
        batches.back().nrun++;
        batches.back().classes |= 1ull << open_cls;
        cost.back() += most;
        open_.clear();
        batches.back().na = (int)(tot / 32) - batches.back().a0;
    };
    for (int q = 0; q < kFoldClasses; q++) {
        const FoldOffset &o = off[q];
        const int z = (o.a == 0) | (o.b == 0) << 1 | (o.c == 0) << 2, free_ = 7 ^ z;
        cls.push_back(make_int4(o.a, o.b, o.c, free_));
        int axis[3], bits = 0;
        for (int i = 0; i < 3; i++)
            if (free_ >> i & 1) axis[bits++] = i;
        int most = 0;
        for (int c = 0; c < 8; c++) most = std::max(most, cnt[c][o.pt]);
        // (kFoldCap rows of at most four column classes a round: at most kFoldMaxTask tasks)
        open_cls = q;
        for (int r = 0; r < 1 << bits; r++)
            for (int k0 = 0; k0 < most; k0 += kFoldCap) {
                int rb = 0;   // the round's column classes: these bits on the free axes, any on the others
                for (int i = 0; i < bits; i++) rb |= (r >> i & 1) << axis[i];
                int depth = 0, ntask = 0;
                for (int be = 0; be < 8; be++) {
                    const int nb = (be & free_) == rb ? std::min(cnt[be][o.pt] - k0, kFoldCap) : 0;
                    if (nb <= 0) continue;
                    depth = std::max(depth, 4 * div_up(nb, 4));
                    ntask += div_up(nb, 4);
                }
                if (depth == 0) continue;
                if (batches.empty() || fill + depth > kFoldCap || batches.back().ntask + ntask > kFoldMaxTask ||
                    (open_.empty() && batches.back().nrun == kFoldMaxRun)) {
                    close_run();
                    batches.push_back({(int)tasks.size(), 0, (int)runs.size() / 8, 0, 0, (int)(tot / 32), 0});
                    cost.push_back(8.0);   // latency of a batch, in K steps of one row block
                    fill = 0;
                }
                if (open_.empty()) open_row = fill;
                open_.push_back({rb, k0, depth});
                // staging tasks: the round's column classes, 4 coefficients each, zeros up to the depth
                for (int be = 0; be < 8; be++) {
                    if ((be & free_) != rb) continue;
                    const int nb = std::max(0, std::min(cnt[be][o.pt] - k0, kFoldCap));
                    for (int k = 0; k < nb; k += 4) {
                        FoldTask t = {};
                        t.src0 = (unsigned short)(base[be] + k0 + k);
                        t.cls = (unsigned char)q;
                        t.n_beta_free = (unsigned char)((std::min(4, nb - k) - 1) | be << 2 | free_ << 5);
                        t.row = (unsigned short)(fill + k);
                        tasks.push_back(t);
                    }
                }
                batches.back().ntask = (int)tasks.size() - batches.back().task0;
                fill += depth;
            }
        close_run();
    }
    F.nbatch = (int)batches.size();
    double all = 0, run = 0;
    for (double c : cost) all += c;
    std::vector<int> group;
    for (int b = 0; b < F.nbatch; b++) {
        while (group.size() < kFoldGroups && run >= all * group.size() / kFoldGroups) group.push_back(b);
        run += cost[b];
    }
    group.resize(kFoldGroups + 1, F.nbatch);

    DBuf<FoldBlock> dblocks;
    DBuf<FoldOffset> doffs;
    auto put = [&](auto &d, const auto &h) {
        if (d.alloc(std::max<size_t>(h.size(), 1), s, st) && !h.empty())
            FMM_TRY(st, cudaMemcpyAsync(d.p, h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice, s));
    };
    std::vector<FoldOffset> offs(off, off + kFoldClasses);
    put(F.kmap, kmap); put(F.rmap, rmap); put(F.base, base); put(F.group, group); put(F.cls, cls); put(F.tasks, tasks);
    put(F.batches, batches); put(F.runs, runs); put(dblocks, blocks); put(doffs, offs);
    F.A.alloc(tot, s, st);
    if (!st.ok()) return false;
    k_fold_ops<<<(unsigned)blocks.size(), 128, 0, s>>>(dblocks.p, doffs.p, F.kmap.p, F.base.p, p, rot, dc, lddc,
                                                       F.A.p); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
    FMM_TRY(st, cudaStreamSynchronize(s));
    F.kmap.s = F.rmap.s = F.base.s = F.group.s = F.cls.s = F.tasks.s = F.batches.s = F.runs.s = F.A.s = nullptr;
    return st.ok();
}

// ---------------------------------------------------------------- complex <-> real basis
__global__ void k_fold_real(long long n, int K, const int4 *kmap, const double2 *in, double2 *mr)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long b = i / K;
    const int4 k = kmap[i - b * K];
    const double2 u = in[b * K + k.x], v = in[b * K + k.y];
    // A = (u + v) / 2, B = (u - v) / 2i
    mr[i] = k.z ? cmk(0.5 * (u.y - v.y), 0.5 * (v.x - u.x)) : cmk(0.5 * (u.x + v.x), 0.5 * (u.y + v.y));
}

// Adds the slots' sums in order and, as complex coefficients, to the local expansions.
__global__ void k_fold_add(long long n, int nr, int K, int slots, const int4 *rmap, const double2 *lr, double2 *out)
{
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n * nr) return;
    const long long b = i / nr;
    const int4 r = rmap[i - b * nr];
    double2 a = lr[b * K + r.z], c = r.w >= 0 ? lr[b * K + r.w] : cmk(0, 0);
    for (int s = 1; s < slots; s++) {
        const double2 *l = lr + ((long long)s * n + b) * K;
        a = cadd(a, l[r.z]);
        if (r.w >= 0) c = cadd(c, l[r.w]);
    }
    double2 *o = out + b * K;
    if (r.w < 0) {
        o[r.x] = cadd(o[r.x], a);
        return;
    }
    o[r.x] = cadd(o[r.x], cmk(a.x - c.y, a.y + c.x));
    o[r.y] = cadd(o[r.y], cmk(a.x + c.y, a.y - c.x));
}

// ---------------------------------------------------------------- the products
struct FoldView {
    const int *base;
    const int4 *cls;
    const FoldTask *tasks;
    const FoldBatch *batches;
    const int2 *runs;
    const double *A;
    const int *group;
    int K;
};

__device__ __forceinline__ FoldTask fold_task(int x, int y)
{
    FoldTask t;
    t.src0 = (unsigned short)(x & 0xffff);
    t.cls = (unsigned char)(x >> 16 & 0xff);
    t.n_beta_free = (unsigned char)((unsigned)x >> 24);
    t.row = (unsigned short)(y & 0xffff);
    return t;
}

// Staging of one task for the 8 targets of this lane group, BITS reflections: the
// sources' coefficients, then their sums with the signs of every character into X.
template <int BITS, int NT>
__device__ __forceinline__ void fold_load(const FoldTask &t, const unsigned *idx, int tl, int kk, const double2 *mr,
                                          double2 (&v)[8])
{
    const unsigned at = t.src0 + kk, none = kk < (t.n_beta_free & 3) + 1 ? 0 : ~0u;
    const unsigned *id = idx + t.cls * 8 * NT + tl;
#pragma unroll
    for (int g = 0; g < 1 << BITS; g++) {
        const unsigned b = id[g * NT] | none;
        v[g] = b != ~0u ? __ldg(mr + (b + at)) : cmk(0, 0);
    }
}

template <int BITS, int NT>
__device__ __forceinline__ void fold_store(const FoldTask &t, int tl, int kk, double2 (&v)[8], double *X)
{
    constexpr int NS = 1 << BITS;
    const int beta = t.n_beta_free >> 2 & 7, fr = t.n_beta_free >> 5;
    const int lo = fr & -fr, hi = fr ^ lo;   // the axes of bits 0 and 1 (one or two reflections)
#pragma unroll
    for (int h = 1; h < NS; h <<= 1)
#pragma unroll
        for (int g = 0; g < NS; g++)
            if (!(g & h)) {
                const double2 a = v[g], b = v[g | h];
                v[g] = cadd(a, b);
                v[g | h] = csub(a, b);
            }
    double *x = X + (t.row + kk) * kFoldLd<NT> + 2 * tl;
#pragma unroll
    for (int c = 0; c < NS; c++) {
        const int sp = BITS == 3 ? c : (c & 1 ? lo : 0) | (c & 2 ? hi : 0);
        *reinterpret_cast<double2 *>(x + (beta ^ sp) * (kFoldCap * kFoldLd<NT>)) = v[c];
    }
}

template <int NT>
__device__ __forceinline__ void fold_load_n(int bits, const FoldTask &t, const unsigned *idx, int tl, int kk,
                                            const double2 *mr, double2 (&v)[8])
{
    if (bits == 3) fold_load<3, NT>(t, idx, tl, kk, mr, v);
    else if (bits == 2) fold_load<2, NT>(t, idx, tl, kk, mr, v);
    else fold_load<1, NT>(t, idx, tl, kk, mr, v);
}

template <int NT>
__device__ __forceinline__ void fold_store_n(int bits, const FoldTask &t, int tl, int kk, double2 (&v)[8], double *X)
{
    if (bits == 3) fold_store<3, NT>(t, tl, kk, v, X);
    else if (bits == 2) fold_store<2, NT>(t, tl, kk, v, X);
    else fold_store<1, NT>(t, tl, kk, v, X);
}

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// One K step: R row blocks x NT / 4 column blocks.
template <int R, int RT, int NT>
__device__ __forceinline__ void fold_step(double (&acc)[RT][NT / 4][2], const double *A, const double *X)
{
    double a[R], b[NT / 4];
#pragma unroll
    for (int r = 0; r < R; r++) a[r] = __ldg(A + 32 * r);
#pragma unroll
    for (int c = 0; c < NT / 4; c++) b[c] = X[8 * c];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int c = 0; c < NT / 4; c++) dmma(acc[r][c][0], acc[r][c][1], a[r], b[c]);
}

// R row blocks over k4 K steps (the fragments are in L1 by then).  Few row blocks: the
// fragments of the next U steps are loaded while U steps are multiplied.
template <int R, int RT, int NT>
__device__ __forceinline__ void fold_mma(double (&acc)[RT][NT / 4][2], const double *A, int k4, const double *X)
{
    if constexpr (R > 3) {
        for (int k = 0; k < k4; k++) {
            fold_step<R, RT, NT>(acc, A, X);
            A += 32 * R;
            X += 4 * kFoldLd<NT>;
        }
    } else {
        constexpr int U = R == 1 ? 3 : 1;
        double cur[U][R], nxt[U][R];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int r = 0; r < R; r++) cur[u][r] = u < k4 ? __ldg(A + 32 * (u * R + r)) : 0;
        for (int k0 = 0; k0 < k4; k0 += U) {
            A += 32 * U * R;
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = 0; r < R; r++) nxt[u][r] = k0 + U + u < k4 ? __ldg(A + 32 * (u * R + r)) : 0;
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (k0 + u >= k4) break;
                double b[NT / 4];
#pragma unroll
                for (int c = 0; c < NT / 4; c++) b[c] = X[8 * c];
                X += 4 * kFoldLd<NT>;
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int c = 0; c < NT / 4; c++) dmma(acc[r][c][0], acc[r][c][1], cur[u][r], b[c]);
            }
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int r = 0; r < R; r++) cur[u][r] = nxt[u][r];
        }
    }
}

template <int R, int RT, int NT>
__device__ __forceinline__ void fold_mma_n(int n, double (&acc)[RT][NT / 4][2], const double *A, int k4, const double *X)
{
    if constexpr (R > 0) {
        if (n == R) fold_mma<R, RT, NT>(acc, A, k4, X);
        else fold_mma_n<R - 1, RT, NT>(n, acc, A, k4, X);
    }
}

// Warps 0 .. 7 multiply, one parity class each (up to RT row blocks); the SW warps after
// them stage the next batch into the other of two buffers meanwhile, two tasks' loads
// in flight each.  Named barriers 1, 2 (a buffer is full) and 3, 4 (free again): both
// sides walk the same list of batches, so every arrival meets one wait.
// Descriptors are read a batch ahead, one per lane, and handed round by shuffles: read
// where they are used, each costs a trip to L2 per warp.
template <int RT, int NT, int SW>
__global__ void __launch_bounds__(256 + 32 * SW, 1) k_m2l_fold(FoldView f, TreeView tv, int first, int count,
                                                            const double2 *mr, double2 *lr, int slots, int prune)
{
    constexpr int NTHR = 256 + 32 * SW, H = NT / 8, XBUF = 8 * kFoldCap * kFoldLd<NT>;
    extern __shared__ double fold_sm[];
    double *X = fold_sm;                                         // two buffers [8][kFoldCap][kFoldLd]
    unsigned *idx = reinterpret_cast<unsigned *>(X + 2 * XBUF);  // first coefficient of the source
                                                                 // boxes [class][reflection][target]
    int4 *order = reinterpret_cast<int4 *>(idx + kFoldClasses * 8 * NT);   // batches with sources: number, first task,
                                                                           // first run, tasks and runs; fragments
    __shared__ int gend[kFoldGroups];
    __shared__ unsigned present[2];
    __shared__ int norder;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t0 = blockIdx.x * NT;
    if (tid < 2) present[tid] = 0;
    if (tid < kFoldGroups) gend[tid] = f.group[tid + 1];
    // rows that a class does not fill meet zeros of the operator: they have to be finite
    for (int i = tid; i < 2 * XBUF; i += NTHR) X[i] = 0;
    __syncthreads();
    {
        // tid % NT is the target throughout
        static_assert(NTHR % NT == 0, "");
        const int t = tid & (NT - 1);
        const int b = t0 + t < count ? first + t0 + t : -1;
        const bool use = b >= 0 && !(prune && tv.ntrg[b] == 0);
        const int o = use ? tv.octant[b] : 0, P = use ? tv.parent[b] : -1;
        for (int e = tid / NT; e < kFoldClasses * 8; e += NTHR / NT) {
            const int q = e >> 3, j = e & 7;
            const int4 c = f.cls[q];
            int src = -1;
            if (P >= 0 && j < 1 << __popc(c.w)) {
                // reflection bits of the nonzero axes, then the source's position
                // in the parent's grid of children
                int d[3] = {c.x, c.y, c.z}, k = 0, cp = 0, oct = 0;
                bool in = true;
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    if (c.w >> i & 1) {
                        if (j >> k & 1) d[i] = -d[i];
                        k++;
                    }
                    const int pos = (o >> i & 1) + d[i], pp = pos >> 1;
                    in &= pp >= -1 && pp <= 1;
                    cp = cp * 3 + pp + 1;
                    oct |= (pos & 1) << i;
                }
                const int C = in ? tv.coll[27L * P + cp] : -1;
                src = C >= 0 ? tv.child[8L * C + oct] : -1;
                if (src >= 0 && tv.nsrc[src] == 0) src = -1;
            }
            idx[e * NT + t] = src >= 0 ? (unsigned)src * (unsigned)f.K : ~0u;
            if (src >= 0) atomicOr(&present[q >> 5], 1u << (q & 31));
        }
    }
    __syncthreads();
    const unsigned long long have = present[0] | (unsigned long long)present[1] << 32;
    const int g0 = slots > 1 ? blockIdx.y : 0, g1 = slots > 1 ? g0 + 1 : kFoldGroups;
    const int bbeg = f.group[g0], bend = f.group[g1];
    if (warp == 0) {
        int n = 0;
        for (int b0 = bbeg; b0 < bend; b0 += 32) {
            FoldBatch B = {};
            if (b0 + lane < bend) B = f.batches[b0 + lane];
            const bool need = B.classes & have;
            const unsigned m = __ballot_sync(0xffffffffu, need);
            if (need)
            {
                int4 *o = order + 2 * (n + __popc(m & ((1u << lane) - 1)));
                o[0] = make_int4(b0 + lane, B.task0, B.run0, B.ntask | B.nrun << 16);
                o[1] = make_int4(B.a0, B.na, 0, 0);
            }
            n += __popc(m);
        }
        if (lane == 0) norder = n;
    }
    __syncthreads();
    const int N = norder;
    if (warp >= 8) {
        // ---- staging
        const int w = warp - 8, kk = lane >> 3;
        int ntask = 0;
        int2 task = make_int2(0, 0);
        auto fetch = [&](int n) {
            if (n >= N) return;
            const int4 B = order[2 * n];
            ntask = B.w & 0xffff;
            if (lane < ntask) task = reinterpret_cast<const int2 *>(f.tasks + B.y)[lane];
        };
        fetch(0);
        for (int n = 0; n < N; n++) {
            const int2 cur = task;
            const int units = H * ntask;
            fetch(n + 1);
            {
                // this batch's fragments into L1
                const int4 B = order[2 * n + 1];
                const char *a = reinterpret_cast<const char *>(f.A + (size_t)B.x * 32);
                for (int i = w * 32 + lane; i < 2 * B.y; i += 32 * SW)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(a + 128 * i));
            }
            if (n >= 2) bar_sync(3 + (n & 1), NTHR);
            double *x = X + (n & 1) * XBUF;
            for (int u = w; u < units; u += 2 * SW) {
                const int u1 = u + SW;
                const FoldTask a = fold_task(__shfl_sync(0xffffffffu, cur.x, u / H), __shfl_sync(0xffffffffu, cur.y, u / H));
                const FoldTask b = fold_task(__shfl_sync(0xffffffffu, cur.x, u1 / H & 31),
                                             __shfl_sync(0xffffffffu, cur.y, u1 / H & 31));
                const bool ua = have >> a.cls & 1, ub = u1 < units && (have >> b.cls & 1);
                const int ta = u % H * 8 + (lane & 7), tb = u1 % H * 8 + (lane & 7);
                const int ba = __popc(a.n_beta_free >> 5), bb = __popc(b.n_beta_free >> 5);
                double2 va[8], vb[8];
                if (ua) fold_load_n<NT>(ba, a, idx, ta, kk, mr, va);
                if (ub) fold_load_n<NT>(bb, b, idx, tb, kk, mr, vb);
                if (ua) fold_store_n<NT>(ba, a, ta, kk, va, x);
                if (ub) fold_store_n<NT>(bb, b, tb, kk, vb, x);
            }
            bar_arrive(1 + (n & 1), NTHR);
        }
        return;
    }
    // ---- products
    const int al = warp;
    double acc[RT][NT / 4][2];
    auto clear = [&]() {
#pragma unroll
        for (int r = 0; r < RT; r++)
#pragma unroll
            for (int c = 0; c < NT / 4; c++) acc[r][c][0] = acc[r][c][1] = 0;
    };
    // a group's sums: lane l holds both right-hand sides of target 4 c + l % 4, row 8 r + l / 4
    auto flush = [&](int g, bool any) {
        if (!any && slots == 1 && g > 0) return;
        const int na = f.base[8 + al];
#pragma unroll
        for (int r = 0; r < RT; r++) {
            const int row = r * 8 + (lane >> 2);
#pragma unroll
            for (int c = 0; c < NT / 4; c++) {
                const int t = t0 + 4 * c + (lane & 3);
                if (row >= na || t >= count) continue;
                double2 *o = lr + ((size_t)(slots > 1 ? g : 0) * count + t) * f.K + f.base[al] + row;
                const double2 v = cmk(acc[r][c][0], acc[r][c][1]);
                *o = slots > 1 || g == 0 ? v : cadd(*o, v);
            }
        }
        clear();
    };
    int nrun = 0;
    int2 run = make_int2(0, 0);
    auto fetch = [&](int n) {
        if (n >= N) return;
        const int4 B = order[2 * n];
        nrun = B.w >> 16;
        if (lane < nrun) run = f.runs[(B.z + lane) * 8 + al];
    };
    clear();
    int g = g0;
    bool any = false;
    fetch(0);
    for (int n = 0; n < N; n++) {
        while (order[2 * n].x >= gend[g]) {
            flush(g++, any);
            any = false;
        }
        any = true;
        const int2 ru = run;
        const int nr = nrun;
        fetch(n + 1);
        bar_sync(1 + (n & 1), NTHR);
        const double *x = X + (n & 1) * XBUF + (al * kFoldCap + (lane & 3)) * kFoldLd<NT> + (lane >> 2);
        for (int i = 0; i < nr; i++) {
            const int a = __shfl_sync(0xffffffffu, ru.x, i), w = __shfl_sync(0xffffffffu, ru.y, i);
            if (!(have >> (w >> 16) & 1)) continue;
            const int k4 = w & 15, rb = w >> 4 & 15, row = w >> 8 & 255;
            if (rb == 0) continue;
            fold_mma_n<RT, RT, NT>(rb, acc, f.A + (size_t)a * 32 + lane, k4, x + row * kFoldLd<NT>);
        }
        if (n + 2 < N) bar_arrive(3 + (n & 1), NTHR);
    }
    for (; g < g1; g++) {
        flush(g, any);
        any = false;
    }
}

bool fold_prepare(const FoldPlan &F, FoldWork &W, int nboxes, int count, cudaStream_t s, Status &st)
{
    if (count <= 0) return true;
    W.slots = fold_split(F, count) ? kFoldGroups : 1;
    // at most 256 MB of sums at a time
    const long long most = std::max<long long>((1LL << 28) / (16LL * F.K * W.slots) / F.tile, 1) * F.tile;
    W.chunk = (int)std::min<long long>(count, most);
    return W.mr.alloc((size_t)nboxes * F.K, s, st) && W.lr.alloc((size_t)W.chunk * F.K * W.slots, s, st);
}

template <int RT, int NT, int SW>
static void launch_fold_t(const FoldPlan &F, const FoldView &f, const FoldWork &W, const TreeView &tv, int first,
                          int count, double2 *out, int prune, cudaStream_t s, Status &st)
{
    const size_t sm = sizeof(double) * 2 * 8 * kFoldCap * kFoldLd<NT> + sizeof(int) * kFoldClasses * 8 * NT +
                      2 * sizeof(int4) * F.nbatch;
    FMM_TRY(st, smem_allow(k_m2l_fold<RT, NT, SW>, sm));
    const int nr = (F.p + 1) * (F.p + 2) / 2;
    for (int c0 = 0; c0 < count && st.ok(); c0 += W.chunk) {
        const int n = std::min(W.chunk, count - c0);
        k_m2l_fold<RT, NT, SW><<<dim3(div_up(n, NT), W.slots), 256 + 32 * SW, sm, s>>>(
            f, tv, first + c0, n, W.mr.p, W.lr.p, W.slots, prune); FMM_COUNT_LAUNCH();
        k_fold_add<<<div_up((long)n * nr, 256), 256, 0, s>>>(n, nr, F.K, W.slots, F.rmap.p, W.lr.p,
                                                             out + (size_t)(first + c0) * F.K); FMM_COUNT_LAUNCH();
        FMM_LAUNCH_CHECK(st);
    }
}

void launch_m2l_fold(const FoldPlan &F, const FoldWork &W, const TreeView &tv, int nboxes, int first, int count,
                     const double2 *in, double2 *out, int prune, cudaStream_t s, Status &st)
{
    if (!st.ok() || count <= 0) return;
    const long long n = (long long)nboxes * F.K;
    k_fold_real<<<div_up(n, 256), 256, 0, s>>>(n, F.K, F.kmap.p, in, W.mr.p); FMM_COUNT_LAUNCH();
    FoldView f;
    f.base = F.base.p; f.cls = F.cls.p; f.tasks = F.tasks.p; f.batches = F.batches.p; f.runs = F.runs.p;
    f.A = F.A.p; f.group = F.group.p; f.K = F.K;
    // row blocks of the largest parity class: orders <= 5, <= 9, <= 15, above (up to 14 at kFoldMaxP)
    if (F.rows <= 1) launch_fold_t<1, 16, 8>(F, f, W, tv, first, count, out, prune, s, st);
    else if (F.rows <= 2) launch_fold_t<2, 16, 8>(F, f, W, tv, first, count, out, prune, s, st);
    else if (F.rows <= 5) launch_fold_t<5, 16, 8>(F, f, W, tv, first, count, out, prune, s, st);
    else launch_fold_t<14, 8, 4>(F, f, W, tv, first, count, out, prune, s, st);
}

}  // namespace fmm
