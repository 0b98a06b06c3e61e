// One-right-hand-side back substitution on 16-row records (sweep.cu), shared by
// the chain solve, the partition solve and the many-system groups.
#pragma once

#include "spk_internal.cuh"

namespace spk {

struct SweepArgs {
    const void *tasks;  // ChainTask, or SegTask (seg)
    int ntasks;
    int seg;            // tasks are SegTask
    const int2 *hdr;    // per 16-row tile: record offset in 16-byte units, bytes
    const unsigned char *rec;
    long long nrec;     // bytes of records (bounds of the checked build)
    int n;
    const double *b;    // right-hand side, caller order
    double *x;          // result
    const double *pre;  // x of the rows from a task's top up (null: zero)
    int rev_b, rev_x, rev_pre;  // 1: element of row r at n - 1 - r
    int win;            // window rows (a power of two >= reach + 16)
    int reach;
    int ns;             // records staged per task
    int stage;          // bytes of a stage
    const int *ia, *ja; // U, for a task that ends inside a tile (seg)
    const double *a;
    const int2 *copies; // row ranges to copy from pre to x (seg)
    int ncopies;
    int *err;
    int fail_entry;
};

int sweep_prepare(spk_system *s);
int sweep_copies(spk_system *s, const std::vector<SegTask> &t2);
// Arguments that depend on the system alone.
SweepArgs sweep_args(const spk_system *s);
size_t sweep_smem(const spk_system *s);
int sweep_occupancy(const spk_system *s, int *occ);
// One launch over A.ntasks tasks (and A.ncopies copies).  dependent: starts while the
// launch before it on the stream still runs (it waits for it before reading x or pre).
int sweep_launch(const spk_system *s, const SweepArgs &A, bool dependent, cudaStream_t st);
// Many systems of equal sw_slots and sw_wide: block b runs task work[b].y of tab[work[b].x]
// (a task number from ntasks up is a copy).  smem: the largest sweep_smem of the systems.
int sweep_launch_multi(const SweepArgs *tab, const int2 *work, int nwork, int slots, bool wide, size_t smem, cudaStream_t st);

}  // namespace spk
