// M2L by dense operators folded over the reflections of the list-2 offsets
// (see m2l_fold.cu).
#pragma once
#include "lap_kernels.cuh"

namespace fmm {

constexpr int kFoldMaxP = 26;      // largest expansion order served
constexpr int kFoldClasses = 56;   // |offset| triples of list 2
constexpr int kFoldGroups = 8;     // partial sums of one target

// One |offset| = (a, b, c): truncation and the direction's rotation class,
// azimuth and distance for D = (a, b, c) (source minus target).
struct FoldOffset {
    int a, b, c, pt, cls;
    double ex, ey, rt;
};

// Staging of 4 consecutive coefficients of one parity class: source
// coefficients from `src0` on, `n` of them valid, combined over the reflections
// of offset class `cls` (coordinate axes `free`, a bit each) into the operand rows from
// `row` on of the parity classes beta ^ (j spread over the axes).
struct __align__(8) FoldTask {
    unsigned short src0;
    unsigned char cls, n_beta_free;   // n - 1 (2 bits), beta (3 bits), free (3 bits)
    unsigned short row, pad;
};

// A batch: the tasks and runs (offset classes) that share one filling of shared memory.
struct FoldBatch {
    int task0, ntask, run0, nrun;
    unsigned long long classes;   // offset classes of its runs
    int a0, na;                   // its operator fragments (32 doubles each)
};
constexpr int kFoldMaxTask = 32, kFoldMaxRun = 16;   // of a batch (a task and a run per lane)

struct FoldPlan {
    int p = 0, K = 0, nbatch = 0;
    int rows = 0;             // 8-row blocks of the largest parity class
    int tile = 16;            // targets per CTA
    DBuf<int4> kmap;          // real coefficient -> (n, m), (n, -m), 1 for the sine part
    DBuf<int4> rmap;          // (n, m >= 0) -> (n, m), (n, -m), cosine and sine coefficients
    DBuf<int> base;           // first coefficient and count of every parity class
    DBuf<int> group;          // first batch of each group of partial sums
    DBuf<int4> cls;           // offset classes: a, b, c, reflection bits
    DBuf<FoldTask> tasks;
    DBuf<FoldBatch> batches;
    DBuf<int2> runs;          // (run, parity class): operator fragment; K steps, row blocks, first operand row, class
    DBuf<double> A;           // operator fragments
};

// Builds the plan of order p from the 56 offsets (any order) and the rotation
// matrices; buffers are detached from the stream.
bool fold_build(FoldPlan &F, int p, const FoldOffset *off, const double *rot, const double *dc, int lddc,
                cudaStream_t s, Status &st);

// Workspace of one geometry and the launch for the targets first ..
// first + count - 1 (boxes of level >= 2).
struct FoldWork {
    DBuf<double2> mr, lr;
    int slots = 1, chunk = 0;
};
bool fold_prepare(const FoldPlan &F, FoldWork &W, int nboxes, int count, cudaStream_t s, Status &st);
void launch_m2l_fold(const FoldPlan &F, const FoldWork &W, const TreeView &tv, int nboxes, int first, int count,
                     const double2 *in, double2 *out, int prune, cudaStream_t s, Status &st);

}  // namespace fmm
