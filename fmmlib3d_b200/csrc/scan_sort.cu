// Device-wide exclusive scan and a stable LSD radix sort (64-bit keys,
// 32-bit payload) used by the octree build.  Written for sm_100a: 256-thread
// CTAs, warp shuffles for intra-warp prefix, one read + one write per pass.
#include "fmm_common.cuh"

namespace fmm {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;  // items per thread per tile
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ int warp_incl_scan(int v)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ int block_excl_scan(int v, int &excl)
{
    __shared__ int wsum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int inc = warp_incl_scan(v);
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
        int t = lane < kScanThreads / 32 ? wsum[lane] : 0;
        int ti = warp_incl_scan(t);
        if (lane < kScanThreads / 32) wsum[lane] = ti - t;
    }
    __syncthreads();
    excl = inc - v + wsum[w];
    __shared__ int tot;
    if (threadIdx.x == kScanThreads - 1) tot = excl + v;
    __syncthreads();
    int total = tot;
    __syncthreads();
    return total;
}

__global__ void k_tile_sums(const int *in, int n, int *tile_sum)
{
    long base = (long)blockIdx.x * kScanTile;
    int s = 0;
    for (int i = 0; i < kScanItems; i++) {
        long j = base + (long)i * kScanThreads + threadIdx.x;
        if (j < n) s += in[j];
    }
    int ex;
    int tot = block_excl_scan(s, ex);
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

// Single-CTA exclusive scan of the tile sums (ntiles small).
__global__ void k_scan_tiles(int *tile_sum, int ntiles, int *total)
{
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < ntiles; b += kScanThreads) {
        int j = b + threadIdx.x;
        int v = j < ntiles ? tile_sum[j] : 0;
        int ex;
        int tot = block_excl_scan(v, ex);
        if (j < ntiles) tile_sum[j] = ex + carry;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void k_scan_apply(const int *in, int *out, int n, const int *tile_off)
{
    long base = (long)blockIdx.x * kScanTile + (long)threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
    for (int i = 0; i < kScanItems; i++) {
        long j = base + i;
        v[i] = j < n ? in[j] : 0;
        s += v[i];
    }
    int ex;
    block_excl_scan(s, ex);
    int run = ex + tile_off[blockIdx.x];
    for (int i = 0; i < kScanItems; i++) {
        long j = base + i;
        if (j < n) out[j] = run;
        run += v[i];
    }
}

// Whole exclusive scans by one CTA each (blockIdx.x picks the array), 8192
// values a step, for arrays where one launch is worth more than many CTAs.
constexpr int kSmallThreads = 1024, kSmallScan = 65536;
__global__ void __launch_bounds__(kSmallThreads) k_scan_small(ScanJobs J, int *totals)
{
    __shared__ int wsum[33];
    const int *in = J.job[blockIdx.x].in;
    int *out = J.job[blockIdx.x].out;
    const int n = J.job[blockIdx.x].n_dev ? *J.job[blockIdx.x].n_dev : J.job[blockIdx.x].n;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < n; base += kSmallThreads * kScanItems) {
        const int j0 = base + threadIdx.x * kScanItems;
        int v[kScanItems], sum = 0;
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            v[i] = j0 + i < n ? in[j0 + i] : 0;
            sum += v[i];
        }
        const int inc = warp_incl_scan(sum);
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        if (w == 0) {
            const int t = wsum[lane], ti = warp_incl_scan(t);
            wsum[lane] = ti - t;
            if (lane == 31) wsum[32] = ti;
        }
        __syncthreads();
        int run = carry + wsum[w] + inc - sum;
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
            if (j0 + i < n) out[j0 + i] = run;
            run += v[i];
        }
        carry += wsum[32];
        __syncthreads();
    }
    if (threadIdx.x == 0 && totals) totals[blockIdx.x] = carry;
}

}  // namespace

static void scan_large(const int *d_in, int *d_out, int n, int *d_total, cudaStream_t s, Status &st)
{
    const int ntiles = div_up(n, kScanTile);
    DBuf<int> tiles;
    if (!tiles.alloc(ntiles, s, st)) return;
    k_tile_sums<<<ntiles, kScanThreads, 0, s>>>(d_in, n, tiles.p); FMM_COUNT_LAUNCH();
    k_scan_tiles<<<1, kScanThreads, 0, s>>>(tiles.p, ntiles, d_total); FMM_COUNT_LAUNCH();
    k_scan_apply<<<ntiles, kScanThreads, 0, s>>>(d_in, d_out, n, tiles.p); FMM_COUNT_LAUNCH();
    FMM_LAUNCH_CHECK(st);
}

void scan_exclusive_multi(const ScanJob *jobs, int njobs, int *d_totals, cudaStream_t s, Status &st)
{
    if (!st.ok() || njobs <= 0) return;
    bool small = true;
    for (int i = 0; i < njobs; i++) small &= jobs[i].n <= kSmallScan || jobs[i].n_dev;
    if (small) {
        ScanJobs J;
        for (int i = 0; i < njobs; i++) J.job[i] = jobs[i];
        k_scan_small<<<njobs, kSmallThreads, 0, s>>>(J, d_totals); FMM_COUNT_LAUNCH();
        FMM_LAUNCH_CHECK(st);
        return;
    }
    for (int i = 0; i < njobs; i++) {
        if (jobs[i].n > 0) scan_large(jobs[i].in, jobs[i].out, jobs[i].n, d_totals ? d_totals + i : nullptr, s, st);
        else if (d_totals) FMM_TRY(st, cudaMemsetAsync(d_totals + i, 0, sizeof(int), s));
    }
}

void scan_exclusive_int(const int *d_in, int *d_out, int n, cudaStream_t s, Status &st, int *h_total)
{
    if (n <= 0) {
        if (h_total) *h_total = 0;
        return;
    }
    DBuf<int> tot;
    if (!tot.alloc(1, s, st)) return;
    ScanJob j{d_in, d_out, n, nullptr};
    scan_exclusive_multi(&j, 1, tot.p, s, st);
    if (h_total) {
        FMM_TRY(st, cudaMemcpyAsync(h_total, tot.p, sizeof(int), cudaMemcpyDeviceToHost, s));
        FMM_TRY(st, cudaStreamSynchronize(s));
    }
}

// ---------------------------------------------------------------- radix sort
namespace {

constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096 items per tile

// Up to two independent arrays are sorted by the same launches (blockIdx.y).
struct SortSide {
    const uint64_t *kin;
    const int *vin;
    uint64_t *kout;
    int *vout;
    int *hist;    // [kRadix][ntiles], then the digit totals [kRadix]
    int n, ntiles;
};
struct SortPass {
    SortSide side[2];
};

// Per-tile digit histogram, written digit-major: hist[digit * ntiles + tile].
__global__ void k_radix_hist(SortPass P, int shift)
{
    const SortSide &A = P.side[blockIdx.y];
    if ((int)blockIdx.x >= A.ntiles) return;
    __shared__ int h[kRadix];
    for (int i = threadIdx.x; i < kRadix; i += kSortThreads) h[i] = 0;
    __syncthreads();
    long base = (long)blockIdx.x * kSortTile;
    for (int i = 0; i < kSortItems; i++) {
        long j = base + (long)i * kSortThreads + threadIdx.x;
        if (j < A.n) atomicAdd(&h[(A.kin[j] >> shift) & (kRadix - 1)], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRadix; i += kSortThreads) A.hist[(long)i * A.ntiles + blockIdx.x] = h[i];
}

// Exclusive scan of one digit's tile counts, and the digit's total.
__global__ void __launch_bounds__(kScanThreads) k_radix_digits(SortPass P)
{
    const SortSide &A = P.side[blockIdx.y];
    int *h = A.hist + (long)blockIdx.x * A.ntiles;
    int carry = 0;
    for (int b = 0; b < A.ntiles; b += kScanThreads) {
        const int j = b + threadIdx.x, v = j < A.ntiles ? h[j] : 0;
        int ex;
        const int tot = block_excl_scan(v, ex);
        if (j < A.ntiles) h[j] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) A.hist[(long)kRadix * A.ntiles + blockIdx.x] = carry;
}

// Stable scatter.  Items of a tile are taken in tile order (item r of the
// tile is at base + r); the tile is processed in rounds of kSortThreads
// consecutive items, each warp ranks its 32 items with __match_any_sync and
// warps are ordered through a per-round shared prefix.
__global__ void k_radix_scatter(SortPass P, int shift)
{
    const SortSide &A = P.side[blockIdx.y];
    if ((int)blockIdx.x >= A.ntiles) return;
    __shared__ int base_d[kRadix];       // running output position per digit
    __shared__ int wcnt[kSortThreads / 32][kRadix];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    {
        static_assert(kRadix == kSortThreads && kSortThreads == kScanThreads, "one digit per thread");
        int ex;
        block_excl_scan(A.hist[(long)kRadix * A.ntiles + threadIdx.x], ex);
        base_d[threadIdx.x] = ex + A.hist[(long)threadIdx.x * A.ntiles + blockIdx.x];
    }
    long tbase = (long)blockIdx.x * kSortTile;
    const int rounds = (int)min((long)kSortItems, (A.n - tbase + kSortThreads - 1) / kSortThreads);
    for (int r = 0; r < rounds; r++) {
        for (int i = threadIdx.x; i < (kSortThreads / 32) * kRadix; i += kSortThreads) (&wcnt[0][0])[i] = 0;
        __syncthreads();
        long j = tbase + (long)r * kSortThreads + threadIdx.x;
        bool valid = j < A.n;
        uint64_t k = valid ? A.kin[j] : 0;
        int v = valid ? A.vin[j] : 0;
        int d = valid ? (int)((k >> shift) & (kRadix - 1)) : -1;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int rank_in_warp = __popc(peers & ((1u << lane) - 1));
        int leader = __ffs(peers) - 1;
        if (valid && lane == leader) wcnt[w][d] = __popc(peers);
        __syncthreads();
        // exclusive prefix over warps for this digit
        int pre = 0;
        if (valid) {
            for (int ww = 0; ww < w; ww++) pre += wcnt[ww][d];
            int pos = base_d[d] + pre + rank_in_warp;
            A.kout[pos] = k;
            A.vout[pos] = v;
        }
        __syncthreads();
        // advance digit bases by this digit pass's totals
        for (int dd = threadIdx.x; dd < kRadix; dd += kSortThreads) {
            int t = 0;
            for (int ww = 0; ww < kSortThreads / 32; ww++) t += wcnt[ww][dd];
            base_d[dd] += t;
        }
        __syncthreads();
    }
}

}  // namespace

void radix_sort_pair(DBuf<uint64_t> &k1, DBuf<int> &v1, int n1, DBuf<uint64_t> *k2, DBuf<int> *v2, int n2, int low,
                     int bits, cudaStream_t s, Status &st)
{
    DBuf<uint64_t> kb[2];
    DBuf<int> vb[2], hist[2];
    DBuf<uint64_t> *k[2] = {&k1, k2};
    DBuf<int> *v[2] = {&v1, v2};
    const int n[2] = {n1, k2 ? n2 : 0};
    const int sides = k2 ? 2 : 1;
    int most = 0;
    for (int i = 0; i < sides; i++) {
        const int nt = div_up(std::max(n[i], 0), kSortTile);
        most = std::max(most, nt);
        if (nt == 0) continue;
        if (!kb[i].alloc(k[i]->n, s, st) || !vb[i].alloc(v[i]->n, s, st) || !hist[i].alloc((size_t)kRadix * (nt + 1), s, st))
            return;
    }
    if (most == 0) return;
    for (int shift = low; shift < bits; shift += kRadixBits) {
        SortPass P = {};
        for (int i = 0; i < sides; i++)
            P.side[i] = {k[i]->p, v[i]->p, kb[i].p, vb[i].p, hist[i].p, n[i], div_up(std::max(n[i], 0), kSortTile)};
        k_radix_hist<<<dim3(most, sides), kSortThreads, 0, s>>>(P, shift); FMM_COUNT_LAUNCH();
        // (an empty side has no tiles and no histogram)
        const int first = P.side[0].ntiles ? 0 : 1;
        if (first) P.side[0] = P.side[1];
        const int live = first ? 1 : (sides == 2 && P.side[1].ntiles ? 2 : 1);
        k_radix_digits<<<dim3(kRadix, live), kScanThreads, 0, s>>>(P); FMM_COUNT_LAUNCH();
        k_radix_scatter<<<dim3(most, live), kSortThreads, 0, s>>>(P, shift); FMM_COUNT_LAUNCH();
        FMM_LAUNCH_CHECK(st);
        if (!st.ok()) return;
        for (int i = 0; i < sides; i++)
            if (n[i] > 0) {
                std::swap(k[i]->p, kb[i].p);
                std::swap(v[i]->p, vb[i].p);
            }
    }
}

}  // namespace fmm
