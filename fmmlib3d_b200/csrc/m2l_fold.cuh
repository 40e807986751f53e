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
// coefficients from `src0` on, `n` of them valid, combined over the
// 2^bits reflections of offset class `cls` into the operand rows `row[j]` of
// parity classes beta ^ spread(j).
struct __align__(16) FoldTask {
    int src0;
    unsigned char cls, n, bits, beta;
    unsigned char axis[4];    // axis[i]: coordinate axis of reflection bit i
    unsigned char row[8];
    int pad[3];
};

// A batch: the segments whose operands share one filling of shared memory.
struct FoldBatch {
    int task0, ntask, seg0, nseg;
};

struct FoldPlan {
    int p = 0, K = 0, nbatch = 0, rows = 0;   // rows: 8-row blocks of the largest parity class
    DBuf<int4> kmap;          // real coefficient -> (n, m), (n, -m), 1 for the sine part
    DBuf<int4> rmap;          // (n, m >= 0) -> (n, m), (n, -m), cosine and sine coefficients
    DBuf<int> base;           // first coefficient and count of every parity class
    DBuf<int> group;          // first batch of each group of partial sums
    DBuf<int4> cls;           // offset classes: a, b, c, reflection bits
    DBuf<FoldTask> tasks;
    DBuf<FoldBatch> batches;
    DBuf<int> seg_cls;
    DBuf<int4> wseg;          // (segment, parity class): operator fragment, K steps, row blocks, operand row
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
    int slots = 1, chunk = 0, tile = 16;   // tile: targets per CTA
};
bool fold_prepare(const FoldPlan &F, FoldWork &W, int nboxes, int count, cudaStream_t s, Status &st);
void launch_m2l_fold(const FoldPlan &F, const FoldWork &W, const TreeView &tv, int nboxes, int first, int count,
                     const double2 *in, double2 *out, int prune, cudaStream_t s, Status &st);

}  // namespace fmm
