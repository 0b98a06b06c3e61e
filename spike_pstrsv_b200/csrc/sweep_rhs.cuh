// Back substitution of many right-hand sides on 16-row records (sweep_rhs.cu).
#pragma once

#include "spk_internal.cuh"

namespace spk {

struct RhsSweep {
    const void *tasks;  // ChainTask, or SegTask (seg)
    int ntasks, seg;
    const int2 *hdr;    // per 16-row tile: record offset in 16-byte units, bytes
    const unsigned char *rec;
    long long nrec;     // bytes of records (bounds of the checked build)
    int n, nk;          // rows; right-hand sides of this pass
    const double *B;    // caller order, column-major
    long long ldb;
    void *X;            // result, column-major: FP64, or the work columns' type (out_work)
    long long ldx;
    int out_work;
    int acc;            // X += x (FP64 result)
    const void *pre;    // x of the rows from a task's top up: work columns, U order, leading dimension n (null: zero)
    int rev_b, rev_x;   // 1: element of row r at n - 1 - r
    int win, mirror;    // ring rows, and how many of its first are mirrored behind its end (multiples of 16)
    int reach;
    int shape;          // how the columns are dealt to lanes and warps
    int ns, stage;      // records staged per task, bytes of a stage (record, then 16 x columns of b)
    const int *ia, *ja; // U, for a task that ends inside a tile (seg)
    const double *a;
    const int2 *copies; // row ranges to copy from pre to X (seg)
    int ncopies;
    int *err;
    int fail_entry;
};

// The records' shape from the histogram of the rows' outside columns (0 .. most).
void rhs_sweep_choose(spk_system *s, const int *hist, int most);
// The records in FP64 or FP32, made on the first call that needs them; rs_ok[fp32] stays 0
// where they cannot be used.
int rhs_sweep_prepare(spk_system *s, int fp32);
void rhs_sweep_release(spk_system *s);
// Whether nk right-hand sides fit (the window of wide rows may not).
bool rhs_sweep_fits(const spk_system *s, int fp32, int nk);
RhsSweep rhs_sweep_args(const spk_system *s, int fp32, int nk);
int rhs_sweep_launch(const spk_system *s, const RhsSweep &A, int fp32, cudaStream_t st);
// Shared memory and kernel class of a launch; launches of one class may be joined.
int rhs_sweep_class(const spk_system *s, int fp32, int nk);
size_t rhs_sweep_smem(const spk_system *s, int fp32, int nk);
int rhs_sweep_launch_multi(const RhsSweep *tab, const int2 *work, int nwork, int cls, int fp32, size_t smem,
                           cudaStream_t st);

}  // namespace spk
