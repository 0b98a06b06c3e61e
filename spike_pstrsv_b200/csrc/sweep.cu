// One-right-hand-side back substitution on 16-row records.
//
// A task walks rows [lo, hi) of U bottom-up, tile by tile.  What bounds it is the latency
// of a tile, not bandwidth: with the off-diagonals applied row by row, a 32-row tile is
// a chain of 32 dependent broadcasts and multiply-adds (eight steps of four), 1.4 us a
// tile for 16 off-diagonals a row.  So the inverse of each tile's unit triangle is computed
// once, at preprocessing, and a tile is two short products:
//
//   r = b / a_ii - sum over the columns outside the tile     (gathered from a window)
//   x = W r,  W = (I + N)^-1 of the tile's row-scaled triangle (120 values)
//
// 16 rows: a product with W costs 7.5 values a row and four multiply-adds a lane; 32
// rows would double the bytes of W, 8 rows would double the dependent steps per row.
//
// One warp alone on its scheduler takes about five cycles an instruction, so the rest of
// the design counts instructions and branches on the solving warp's path:
// * Rows g and 15 - g share the four lanes 4g .. 4g + 3.  Each row's outside columns are
//   dealt to its two lanes, S of them a lane, S a template parameter (the one that costs
//   the fewest slots over the system; a tile with a longer row has extra slots, taken
//   off the common path).  Row g has 15 - g values in W and row 15 - g has g, so the
//   four lanes share 15 whatever g; only the last two of a lane's four values can belong to
//   either row.
// * A second warp issues the copies: a tile's record (W, 1 / diagonal, slot values and
//   offsets) is contiguous and comes by one bulk copy, up to ns records ahead; b by 8-byte
//   asynchronous copies on the same barrier.
// * The solving warp loads the next record into registers while the gathers of the
//   current tile are in flight.
// * Solved rows stay in a window in shared memory that covers every column a row reaches,
//   held twice, end to end, so that a column's address is one addition.  Rows from the
//   task's top up come from `pre` (or are zero).
// * An unused slot repeats its row's first column with value 0.  A row without any must not read
//   one that it does not depend on (it may hold an infinity or a NaN, or, in `pre`, be one that
//   phase 1 never writes): by a bit of the record its slots read a zero beside the window.  The
//   choice is made on the address, a tile ahead: it costs nothing there (128 x 128 Poisson factor
//   160 us, 176 us where the sum was dropped instead, on the way from one tile to the next).
//
// Measured (one solve, the row-by-row kernels -> this one): banded rows with 16 off-diagonals,
// 4,194,304 rows: lower 234 -> 201 to 212 us (191 back to back; 6 tasks an SM, 233 bytes a row:
// bound by HBM), its transpose 573 -> 250 us; 262,147 rows, transpose, in the same two phases: 264
// -> 80 us (0.40 us a tile of 16 rows: its latency), in the one launch that plain solves take 50 us
// (chain.cu); 128 x 128 Poisson factor in 4 partitions: 298 -> 160 us (0.28 us a tile).
// Staged records (two phases): 2 / 3 / 4 / 6 a task take 180 / 99 / 80 / 80 us at 262,147 rows and
// 3 / 4 / 5 / 6 take 233 / 211 / 208 / 194 us at full size.
//
// W is used only where its rows' absolute sums stay at most kGrowth: the error of the product
// grows with them (c u |W||T||W||r| against c u |W||T||x| of the substitution).  Over 40,000 random
// triangles of 16 rows, against 80 bits, the product's mean error is 0.5 to 0.65 of the
// substitution's for sums up to 4, 0.77 to 5.7, 0.98 to 8, 1.24 to 11 and 1.45 to 16, and its largest
// one passes the substitution's from about 5 on: the limit is 4 (it was 16).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>

#include "checks.cuh"
#include "records.cuh"
#include "sweep.cuh"
#include "sweep_rhs.cuh"

namespace spk {

namespace {

constexpr int kThreads = 64;        // a solving and a copying warp
constexpr int kMaxSlots = 64;       // slots per lane
constexpr int kMaxWindow = 8192;    // rows
constexpr double kGrowth = 4.0;     // largest absolute row sum of W
constexpr int kCopyRows = 1024;     // rows per copy block
constexpr int kMaxStages = 9;

constexpr int kSlots[] = {2, 4, 6, 8, 10, 12, 16, 20};  // slots per lane on the common path

__device__ __forceinline__ double lds(unsigned a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

// Shared memory of a task: full and empty barriers of the stages, a zero, the window, the stages.
struct Smem {
    unsigned full, empty, zero, win, stage0;
    __device__ explicit Smem(unsigned base, int win_rows)
        : full(base), empty(base + 8 * kMaxStages), zero(base + 16 * kMaxStages), win(base + 256), stage0(base + 256 + 16 * win_rows) {}
};

// The copying warp: tiles of rows [lo, hi), top first.
__device__ __forceinline__ bool copy_tiles(const SweepArgs &A, const Smem &M, Ring &R, int lo, int hi, int lane) {
    const int jt = (hi - 1) >> 4, jb = lo >> 4;
    int2 h = make_int2(0, 0);
    for (int j = jt; j >= jb; j--) {
        const int k = (jt - j) & 31;
        if (k == 0) h = j - lane >= jb ? __ldg(A.hdr + CK(j - lane, (A.n + 15) >> 4, 60)) : make_int2(0, 0);
        const unsigned at = __shfl_sync(kFull, h.x, k);
        const unsigned bytes = CKU(__shfl_sync(kFull, h.y, k), A.stage - 127, 61);
        const unsigned bar = M.full + 8 * R.slot, dst = M.stage0 + R.slot * A.stage;
        if (!try_wait(M.empty + 8 * R.slot, R.parity ^ 1) && !slow_wait(M.empty + 8 * R.slot, R.parity ^ 1)) return false;
        if (lane == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                         "l"(A.rec + CK((unsigned long long)at * 16, A.nrec - bytes + 1, 62)), "r"(bytes), "r"(bar)
                         : "memory");
        }
        const int r = 16 * j + lane;
        if (lane < 16 && r >= lo && r < hi) {
            const double *src = A.b + CK(A.rev_b ? A.n - 1 - r : r, A.n, 63);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + A.stage - 128 + 8 * lane), "l"(src) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
        R.next(A.ns);
    }
    return true;
}

__device__ __forceinline__ void lds2(unsigned a, double &x, double &y) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a));
}
__device__ __forceinline__ unsigned ldsu(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// One lane's part of a record, in registers.
template <int S, bool WIDE>
struct Record {
    static constexpr int kWords = WIDE ? S / 2 : (S + 3) / 4;
    unsigned o[kWords], extra;
    double v[S], w[4], b, rd;
    __device__ __forceinline__ void load(unsigned st, unsigned lane, unsigned myrow, unsigned boff) {
        extra = ldsu(st + kExtra);  // first: the tile's addresses wait for it
#pragma unroll
        for (int h = 0; h < kWords; h++) o[h] = ldsu(st + kHead + 256 * S + 128 * h + 4 * lane);
#pragma unroll
        for (int h = 0; h < S / 2; h++) lds2(st + kHead + 512 * h + 16 * lane, v[2 * h], v[2 * h + 1]);
        b = lds(st + boff + 8 * myrow);
        rd = lds(st + kDiag + 8 * myrow);
#pragma unroll
        for (int h = 0; h < 2; h++) lds2(st + 512 * h + 16 * lane, w[2 * h], w[2 * h + 1]);
    }
    __device__ __forceinline__ unsigned off(int u) const {
        return WIDE ? (u & 1 ? o[u / 2] >> 16 : o[u / 2] & 0xffffu) : (o[u / 4] >> (8 * (u & 3))) & 0xffu;
    }
};

// The extra slots of a tile.
template <bool WIDE>
__device__ __noinline__ double extra_slots(unsigned at, int E, unsigned gather, int lane) {
    double s = 0.0;
    for (int u = 0; u < E; u++) {
        const unsigned w = ldsu(at + 256 * E + 128 * (WIDE ? u / 2 : u / 4) + 4 * lane);
        const unsigned o = WIDE ? (w >> (16 * (u & 1))) & 0xffffu : (w >> (8 * (u & 3))) & 0xffu;
        s = fma(lds(at + 512 * (u / 2) + 16 * lane + 8 * (u & 1)), lds(gather + 8 * o), s);
    }
    return s;
}

// A tile that the task's top cuts: its rows from hi up are known (in the window) and have
// r = 0, which leaves W the inverse of the rows below (a triangle's leading block); what
// those rows read of them is subtracted here.
__device__ __noinline__ double cut(const int *ia, const int *ja, const double *a, int row, int hi, double r, unsigned win,
                                   unsigned maskb) {
    const int e0 = ia[row], e1 = ia[row + 1], top = (row | 15) + 1;
    double s = 0.0;
    for (int e = e0 + 1; e < e1 && ja[e] < top; e++)
        if (ja[e] >= hi) s = fma(a[e], lds(win + ((8u * (unsigned)ja[e]) & maskb)), s);
    return r - s / a[e0];
}

// The solving warp: rows [lo, hi) bottom-up, storing rows [st_lo, st_hi) of them; the window
// holds x of rows [hi, hi + reach).  False after a barrier wait that gave up.
template <int S, bool WIDE>
struct Solver {
    const SweepArgs &A;
    const Smem &M;
    Ring &R;
    const int lane, hi;
    bool second;
    int g, myrow;
    int src[4];         // lanes that hold r of this lane's columns in W
    bool isa2, isa3;    // whether its last two values belong to row g
    unsigned maskb, winb, boff;
    unsigned outbit;    // of the record's word: the row has a column outside its tile
    unsigned pos;       // 8 * (first row of the tile above, modulo the window)
    unsigned from;      // what the distances of the tile's outside columns count from
    int row, st_lo, st_hi;
    double *xp;
    int step;

    __device__ __forceinline__ Solver(const SweepArgs &A_, const Smem &M_, Ring &R_, int lane_, int lo, int hi_, int slo, int shi)
        : A(A_), M(M_), R(R_), lane(lane_), hi(hi_) {
        second = lane & 2;
        g = lane >> 2;
        myrow = second ? 15 - g : g;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int e = (lane & 3) + 4 * u;
            const bool isa = e < 15 - g;  // always for the first two
            const int col = isa ? g + 1 + e : min(e + 1, 15);
            src[u] = col < 8 ? 4 * col : 4 * (15 - col) + 2;
            if (u == 2) isa2 = isa;
            if (u == 3) isa3 = isa;
        }
        maskb = 8u * (unsigned)(A.win - 1);
        winb = 8u * (unsigned)A.win;
        boff = A.stage - 128;
        outbit = 0x10000u << myrow;
        const int jt = (hi - 1) >> 4;
        pos = (8u * (unsigned)(16 * jt + 16)) & maskb;
        row = 16 * jt + myrow;
        st_lo = (lane & 1) ? 2147483647 : max(slo, lo);  // one of a row's two lanes stores it
        st_hi = min(shi, hi);
        xp = A.x + (A.rev_x ? (long long)A.n - 1 - row : (long long)row);
        step = A.rev_x ? 16 : -16;
    }

    __device__ __forceinline__ unsigned base(const Record<S, WIDE> &C) const { return C.extra & outbit ? M.win + pos : M.zero; }

    // One tile: its record in C; the next one (if any) goes to N meanwhile.
    template <bool TOP>
    __device__ __forceinline__ bool tile(const Record<S, WIDE> &C, Record<S, WIDE> &N, bool more) {
        const unsigned gather = from, release = M.empty + 8 * R.slot, old = M.stage0 + R.slot * A.stage;
        double x[S];
#pragma unroll
        for (int u = 0; u < S; u++) x[u] = lds(gather + 8 * CKU(C.off(u), max(A.reach, 1), 64));
        R.next(A.ns);
        if (more) {
            const unsigned bar = M.full + 8 * R.slot;
            if (!try_wait(bar, R.parity) && !slow_wait(bar, R.parity)) return false;
            N.load(M.stage0 + R.slot * A.stage, lane, myrow, boff);
        }
        double own[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < S; u++) own[u & 1] = fma(C.v[u], x[u], own[u & 1]);
        double r = own[0] + own[1];
        if (C.extra & 0xffffu) r += extra_slots<WIDE>(old + kHead + slot_bytes(S, WIDE), C.extra & 0xffffu, gather, lane);
        r = fma(C.b, C.rd, -(r + __shfl_xor_sync(kFull, r, 1)));
        if (TOP && (row | 15) >= hi) {  // the task's top cuts the tile
            if (row >= hi) r = 0.0;
            else if (hi < A.n && A.pre) r = cut(A.ia, A.ja, A.a, row, hi, r, M.win, maskb);
            __syncwarp();
        }
        pos = (pos - 128) & maskb;
        from = base(N);  // here: N has arrived, and r is on its way
        const double r0 = __shfl_sync(kFull, r, src[0]), r1 = __shfl_sync(kFull, r, src[1]);
        const double r2 = __shfl_sync(kFull, r, src[2]), r3 = __shfl_sync(kFull, r, src[3]);
        double p0 = C.w[0] * r0, p1 = C.w[1] * r1;
        p0 = fma(C.w[2], isa2 ? r2 : 0.0, p0);
        p1 = fma(C.w[3], isa3 ? r3 : 0.0, p1);
        const double qa = fma(C.w[3], isa3 ? 0.0 : r3, C.w[2] * (isa2 ? 0.0 : r2)), pa = p0 + p1;
        // both rows' sums over the four lanes
        double t = (second ? qa : pa) + __shfl_xor_sync(kFull, second ? pa : qa, 2);
        t += __shfl_xor_sync(kFull, t, 1);
        const double xv = r + t;  // one rounding at the size of x, as in the substitution
        const unsigned at = M.win + pos + 8 * myrow;
        if (!TOP || row < hi) {
            asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(xv) : "memory");
            asm volatile("st.shared.f64 [%0], %1;" ::"r"(at + winb), "d"(xv) : "memory");
        }
        if (row >= st_lo && row < st_hi) *CKP(xp, A.x, A.n, 65) = xv;
        __syncwarp();  // the window rows; every lane is done with the stage
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(release) : "memory");
        row -= 16;
        xp += step;
        return true;
    }

    __device__ __forceinline__ bool run(int tiles) {
        Record<S, WIDE> P, Q;
        Q.extra = 0;
        const unsigned bar = M.full + 8 * R.slot;
        if (!try_wait(bar, R.parity) && !slow_wait(bar, R.parity)) return false;
        P.load(M.stage0 + R.slot * A.stage, lane, myrow, boff);
        from = base(P);
        if (!tile<true>(P, Q, tiles > 1)) return false;
        for (int k = 1; k < tiles; k += 2) {
            if (!tile<false>(Q, P, k + 1 < tiles)) return false;
            if (k + 1 < tiles && !tile<false>(P, Q, k + 2 < tiles)) return false;
        }
        return true;
    }
};

template <int S, bool WIDE>
__device__ __forceinline__ bool solve_tiles(const SweepArgs &A, const Smem &M, Ring &R, int lo, int hi, int st_lo, int st_hi,
                                            int lane) {
    Solver<S, WIDE> V(A, M, R, lane, lo, hi, st_lo, st_hi);
    return V.run(((hi - 1) >> 4) - (lo >> 4) + 1);
}

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <int S, bool WIDE>
__device__ __forceinline__ void sweep_task(const SweepArgs &A, int task) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    if (A.fail_entry) {
        if (threadIdx.x == 0) atomicExch(A.err, 1);
        return;
    }
    if (task >= A.ntasks) {  // rows that keep the phase-1 values
        grid_wait();
        const int2 c = A.copies[task - A.ntasks];
        for (int r0 = c.x; r0 < c.y; r0 += kThreads * 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int r = r0 + kThreads * u + (int)threadIdx.x;
                v[u] = r < c.y ? A.pre[CK(A.rev_pre ? A.n - 1 - r : r, A.n, 66)] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int r = r0 + kThreads * u + (int)threadIdx.x;
                if (r < c.y) A.x[CK(A.rev_x ? A.n - 1 - r : r, A.n, 67)] = v[u];
            }
        }
        return;
    }
    const Smem M(su32(smem), A.win);
    if (threadIdx.x == 0) {
        for (int k = 0; k < A.ns; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(M.full + 8 * k), "r"(33u) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(M.empty + 8 * k), "r"(1u) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("st.shared.f64 [%0], %1;" ::"r"(M.zero), "d"(0.0) : "memory");
    }
    __syncthreads();
    int lo, hi, st_lo, st_hi, skip_lo = 0, skip_hi = 0;
    if (A.seg) {
        const SegTask t = ((const SegTask *)A.tasks)[task];
        lo = t.lo, hi = t.hi, skip_lo = t.skip_lo, skip_hi = t.skip_hi, st_lo = 0, st_hi = A.n;
    } else {
        const ChainTask t = ((const ChainTask *)A.tasks)[task];
        lo = t.lo, hi = t.hi, st_lo = t.st_lo, st_hi = t.st_hi;
    }
    const bool two = skip_hi > skip_lo;
    const int lo1 = two ? skip_hi : lo;  // first range [lo1, hi), second [lo, skip_lo)
    const bool first = lo1 < hi, then = two && lo < skip_lo;
    Ring R;
    if (threadIdx.x >= 32) {  // records and b do not depend on the launch before
        bool ok = true;
        if (first) ok = copy_tiles(A, M, R, lo1, hi, lane);
        if (then && ok) ok = copy_tiles(A, M, R, lo, skip_lo, lane);
        // no copy may land after the block is gone: the stages still in flight (a stage not filled
        // yet is asked for the parity before its first, which a new barrier has)
        for (int k = 0; k < A.ns; k++) {
            if (R.slot == 0) R.parity ^= 1;
            R.slot = R.slot == 0 ? A.ns - 1 : R.slot - 1;
            slow_wait(M.full + 8 * R.slot, R.parity);
        }
        return;
    }
    // x of rows [r0, r0 + count) into the window (zero past the matrix or without pre)
    const unsigned maskb = 8u * (unsigned)(A.win - 1);
    auto load_window = [&](int r0, int count) {
        for (int k = lane; k < count; k += 32) {
            const int r = r0 + k;
            const double v = A.pre && r < A.n ? A.pre[CK(A.rev_pre ? A.n - 1 - r : r, A.n, 68)] : 0.0;
            const unsigned at = M.win + ((8u * (unsigned)r) & maskb);
            asm volatile("st.shared.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
            asm volatile("st.shared.f64 [%0], %1;" ::"r"(at + 8 * A.win), "d"(v) : "memory");
        }
        __syncwarp();
    };
    grid_wait();
    grid_release();
    load_window(hi, A.reach);
    bool ok = true;
    if (first) ok = solve_tiles<S, WIDE>(A, M, R, lo1, hi, st_lo, st_hi, lane);
    if (two && ok) {
        load_window(skip_lo, min(skip_hi - skip_lo, A.reach));
        if (then) ok = solve_tiles<S, WIDE>(A, M, R, lo, skip_lo, st_lo, st_hi, lane);
    }
    if (!ok && lane == 0) atomicExch(A.err, 1);
}

template <int S, bool WIDE>
__global__ void __launch_bounds__(kThreads) k_sweep(const SweepArgs *__restrict__ tab, const int2 *__restrict__ work,
                                                    SweepArgs one) {
    if (tab) {
        const int2 w = work[blockIdx.x];
        const SweepArgs A = tab[w.x];
        sweep_task<S, WIDE>(A, w.y);
    } else {
        sweep_task<S, WIDE>(one, blockIdx.x);
    }
}

// ---- records ------------------------------------------------------------------------

// First entry of row r whose column is at or past `col` (columns are sorted, the diagonal first).
__device__ __forceinline__ int first_from(const int *__restrict__ ja, int b, int e, int col) {
    while (b < e) {
        const int m = (b + e) >> 1;
        if (ja[m] < col) b = m + 1;
        else e = m;
    }
    return b;
}

// Per tile: slots per lane that its longest row needs (two lanes a row; even); the matrix's
// reach, and a histogram of the rows' outside columns.  A half warp per tile.
__global__ void k_sweep_count(int n, int ntiles, const int *__restrict__ ia, const int *__restrict__ ja,
                              int *__restrict__ slots, int *__restrict__ reach, int *__restrict__ hist) {
    __shared__ int sh[2 * kMaxSlots + 1];
    for (int i = threadIdx.x; i <= 2 * kMaxSlots; i += blockDim.x) sh[i] = 0;
    __syncthreads();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = r >> 4;
    int out = 0, d = 0;
    if (r < n) {
        const int b = ia[r], e = ia[r + 1];
        out = e - first_from(ja, b, e, 16 * j + 16);
        d = ja[e - 1] - r;
        atomicAdd(&sh[min(out, 2 * kMaxSlots)], 1);
    }
#pragma unroll
    for (int o = 8; o; o >>= 1) out = max(out, __shfl_xor_sync(kFull, out, o, 16));
#pragma unroll
    for (int o = 16; o; o >>= 1) d = max(d, __shfl_xor_sync(kFull, d, o));
    if ((r & 15) == 0 && j < ntiles) slots[j] = ((out + 1) / 2 + 1) & ~1;
    if ((threadIdx.x & 31) == 0) atomicMax(reach, d);
    __syncthreads();
    for (int i = threadIdx.x; i <= 2 * kMaxSlots; i += blockDim.x)
        if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// The records, a warp per tile.
template <bool WIDE>
__global__ void __launch_bounds__(128) k_sweep_fill(int n, int ntiles, const int *__restrict__ ia,
                                                    const int *__restrict__ ja, const double *__restrict__ a, int S0,
                                                    const int2 *__restrict__ hdr, unsigned char *__restrict__ rec,
                                                    unsigned long long *__restrict__ growth) {
    __shared__ double sm[4][2][16][17];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, j = blockIdx.x * 4 + wp;
    if (j >= ntiles) return;
    double (*t)[17] = sm[wp][0], (*W)[17] = sm[wp][1];
    const int row0 = 16 * j, E = (hdr[j].y - kHead - slot_bytes(S0, WIDE)) / slot_bytes(4, WIDE) * 4;
    unsigned char *R = rec + (unsigned long long)(unsigned)hdr[j].x * 16;
    for (int e = lane; e < 256; e += 32) t[e >> 4][e & 15] = W[e >> 4][e & 15] = 0.0;
    __syncwarp();
    int b = 0, f = 0, e = 0;  // this lane's row (i = lane & 15): diagonal, first outside entry, end
    double rd = 0.0;
    const int i = lane & 15, row = row0 + i;
    if (row < n) {
        b = ia[row], e = ia[row + 1];
        f = first_from(ja, b, e, row0 + 16);
        rd = 1.0 / a[b];
    }
    if (lane < 16) {
        ((double *)(R + kDiag))[i] = rd;
        for (int q = b + 1; q < f; q++) t[i][ja[q] - row0] = a[q] * rd;
    }
    __syncwarp();
    // column i of W: W(p, i) = -(t(p, i) + sum over p < k < i of t(p, k) W(k, i))
    if (lane < 16)
        for (int p = i - 1; p >= 0; p--) {
            double s = t[p][i];
            for (int k = p + 1; k < i; k++) s = fma(t[p][k], W[k][i], s);
            W[p][i] = -s;
        }
    __syncwarp();
    double sum = 1.0;
    if (lane < 16)
        for (int k = i + 1; k < 16; k++) sum += fabs(W[i][k]);
    if (!(sum <= kGrowth)) sum = 1e300;  // a NaN too
#pragma unroll
    for (int o = 16; o; o >>= 1) sum = fmax(sum, __shfl_xor_sync(kFull, sum, o));
    if (lane == 0) atomicMax(growth, __double_as_longlong(sum));
    const int g = lane >> 2;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int q = (lane & 3) + 4 * u;
        const double v = q < 15 - g ? W[g][g + 1 + q] : (q < 15 ? W[15 - g][q + 1] : 0.0);
        ((double *)R)[((u >> 1) * 32 + lane) * 2 + (u & 1)] = v;
    }
    const unsigned out = __ballot_sync(kFull, lane < 16 && e > f);
    if (lane == 0) *(int4 *)(R + kExtra) = make_int4((int)((unsigned)E | out << 16), 0, 0, 0);
    // slot u of a lane: entry 2 u + (lane & 1) of its row's outside columns; an unused one repeats
    // the first (distance 0 where there is none: the zero)
    const int mine = (lane & 2) ? 15 - g : g;
    const int f0 = __shfl_sync(kFull, f, mine), n0 = __shfl_sync(kFull, e, mine) - f0;
    const double r0 = __shfl_sync(kFull, rd, mine);
    auto put = [&](unsigned char *at, int count, int from) {
        const int words = WIDE ? count : 4 * ((count + 3) / 4);
        for (int u = 0; u < words; u++) {
            const int q = 2 * (from + u) + (lane & 1);
            const bool used = u < count && q < n0;
            const double v = used ? a[f0 + q] * r0 : 0.0;
            const int o = used ? ja[f0 + q] - row0 - 16 : (n0 > 0 ? ja[f0] - row0 - 16 : 0);
            if (u < count) ((double *)at)[((u >> 1) * 32 + lane) * 2 + (u & 1)] = v;
            if (WIDE) ((unsigned short *)(at + 256 * count))[((u >> 1) * 32 + lane) * 2 + (u & 1)] = (unsigned short)o;
            else (at + 256 * count)[((u >> 2) * 32 + lane) * 4 + (u & 3)] = (unsigned char)o;
        }
    };
    put(R + kHead, S0, 0);
    if (E) put(R + kHead + slot_bytes(S0, WIDE), E, S0);
}

}  // namespace

// The records of U; sw_ok = 0 (the row-by-row kernels run) when a row reaches past the
// window, a row has more than 2 kMaxSlots of them, or W grows past kGrowth.
int sweep_prepare(spk_system *s) {
    rhs_sweep_release(s);
    s->sw_ok = 0;
    // the records of a system preprocessed again take the memory of the last ones (4.7 MB: 0.35 ms
    // to give back and get): no solve reads them any more, the steps before have waited for the device
    struct Unused {
        spk_system *s;
        ~Unused() {
            if (s->sw_ok) return;
            s->sw_rec.release();
            s->sw_hdr.release();
        }
    } unused{s};
    const char *no = getenv("SPK_DISABLE_SWEEP");  // test hook: the row-by-row kernels
    if (no && no[0] == '1') return SPK_OK;
    const int n = s->n, nt = (n + 15) / 16;
    cudaStream_t st = s->stream;
    constexpr int kTail = 1 + 2 * kMaxSlots + 1;  // after the tiles: the reach, the histogram
    std::vector<int> hs(nt + kTail);
    std::vector<int2> hd(nt);
    {
        DBuf<int> d(st);
        SPK_TRY(d.alloc(nt + kTail));
        SPK_CUDA(cudaMemsetAsync(d.p + nt, 0, sizeof(int) * kTail, st));
        k_sweep_count<<<(nt * 16 + 255) / 256, 256, 0, st>>>(n, nt, s->uia.p, s->uja.p, d.p, d.p + nt, d.p + nt + 1);
        SPK_CUDA(cudaGetLastError());
        SPK_CUDA(cudaMemcpyAsync(hs.data(), d.p, sizeof(int) * (nt + kTail), cudaMemcpyDeviceToHost, st));
        SPK_CUDA(cudaStreamSynchronize(st));
    }
    const int reach = hs[nt];
    const bool wide = reach > 128;
    long long hist[kMaxSlots + 1] = {};
    int smax = 0;
    for (int j = 0; j < nt; j++) {
        if (hs[j] > kMaxSlots) return SPK_OK;
        hist[hs[j]]++;
        smax = std::max(smax, hs[j]);
    }
    if (reach + 16 > kMaxWindow) return SPK_OK;
    // slots on the common path: the fewest over all tiles, an extra slot counted twice (it
    // comes through a loop) and a tile that has any as ten more
    int S0 = 0;
    double best = 0;
    for (int c : kSlots) {
        double cost = 0;
        for (int k = 0; k <= smax; k++) cost += hist[k] * (c + (k > c ? 2.0 * ((k - c + 3) & ~3) + 10.0 : 0.0));
        if (!S0 || cost < best) S0 = c, best = cost;
    }
    long long at = 0;
    int most = 0;
    for (int j = 0; j < nt; j++) {
        const int E = hs[j] > S0 ? (hs[j] - S0 + 3) & ~3 : 0;
        const int bytes = kHead + slot_bytes(S0, wide) + (E ? slot_bytes(E, wide) : 0);
        hd[j] = make_int2((int)(unsigned)at, bytes);
        most = std::max(most, bytes);
        at += bytes / 16;
    }
    if (at >= (1ll << 32)) return SPK_OK;
    SPK_TRY(s->sw_hdr.reserve(nt));
    SPK_CUDA(cudaMemcpyAsync(s->sw_hdr.p, hd.data(), sizeof(int2) * nt, cudaMemcpyHostToDevice, st));
    SPK_TRY(s->sw_rec.reserve((size_t)at * 16));
    s->sw_bytes = at * 16;
    DBuf<unsigned long long> g(st);
    SPK_TRY(g.alloc(1));
    SPK_CUDA(cudaMemsetAsync(g.p, 0, sizeof(unsigned long long), st));
    if (wide)
        k_sweep_fill<true><<<(nt + 3) / 4, 128, 0, st>>>(n, nt, s->uia.p, s->uja.p, s->ua.p, S0, s->sw_hdr.p, s->sw_rec.p, g.p);
    else
        k_sweep_fill<false><<<(nt + 3) / 4, 128, 0, st>>>(n, nt, s->uia.p, s->uja.p, s->ua.p, S0, s->sw_hdr.p, s->sw_rec.p, g.p);
    SPK_CUDA(cudaGetLastError());
    unsigned long long h = 0;
    SPK_CUDA(cudaMemcpyAsync(&h, g.p, sizeof(h), cudaMemcpyDeviceToHost, st));
    SPK_CUDA(cudaStreamSynchronize(st));
    double growth;
    memcpy(&growth, &h, sizeof(growth));
    if (!(growth <= kGrowth)) return SPK_OK;
    int win = 32;
    while (win < reach + 16) win <<= 1;
    s->sw_win = win;
    s->sw_reach = reach;
    s->sw_wide = wide;
    s->sw_slots = S0;
    s->sw_stage = most + 128;
    s->sw_ok = 1;
    rhs_sweep_choose(s, hs.data() + nt + 1, 2 * kMaxSlots);
    return SPK_OK;
}

long long sweep_device_check() { return first_failed_check(); }

SweepArgs sweep_args(const spk_system *s) {
    SweepArgs A{};
    A.hdr = s->sw_hdr.p;
    A.rec = s->sw_rec.p;
    A.nrec = s->sw_bytes;
    A.n = s->n;
    A.win = s->sw_win;
    A.reach = s->sw_reach;
    A.ns = 3 * s->ch_stages;
    A.stage = s->sw_stage;
    // fewer stages where the window leaves no room for them
    while (A.ns > 2 && 256 + 16ll * A.win + (long long)A.ns * A.stage > 227 * 1024) A.ns--;
    A.ia = s->uia.p;
    A.ja = s->uja.p;
    A.a = s->ua.p;
    A.err = s->d_err.p;
    A.fail_entry = s->dbg_fail_waits > 0;
    return A;
}

size_t sweep_smem(const spk_system *s) {
    const SweepArgs A = sweep_args(s);
    return 256 + 16 * (size_t)A.win + (size_t)A.ns * A.stage;
}

namespace {
template <int S>
int launch_s(bool wide, const SweepArgs *tab, const int2 *work, const SweepArgs &one, int blocks, size_t smem,
             bool dependent, cudaStream_t st, int *occ) {
    auto go = [&](auto kern) -> int {
        SPK_TRY(allow_smem(kern));
        if (occ) {
            SPK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kern, kThreads, smem));
            return SPK_OK;
        }
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = dependent ? 1 : 0;
        SPK_CUDA(cudaLaunchKernelEx(&cfg, kern, tab, work, one));
        return SPK_OK;
    };
    return wide ? go(k_sweep<S, true>) : go(k_sweep<S, false>);
}

int launch_any(int slots, bool wide, const SweepArgs *tab, const int2 *work, const SweepArgs &one, int blocks, size_t smem,
               bool dependent, cudaStream_t st, int *occ = nullptr) {  // occ: query instead of launch
    switch (slots) {
        case 2: return launch_s<2>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 4: return launch_s<4>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 6: return launch_s<6>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 8: return launch_s<8>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 10: return launch_s<10>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 12: return launch_s<12>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        case 16: return launch_s<16>(wide, tab, work, one, blocks, smem, dependent, st, occ);
        default: return launch_s<20>(wide, tab, work, one, blocks, smem, dependent, st, occ);
    }
}
}  // namespace

// Tasks of s an SM holds at once.
int sweep_occupancy(const spk_system *s, int *occ) {
    return launch_any(s->sw_slots, s->sw_wide, nullptr, nullptr, SweepArgs{}, 0, sweep_smem(s), false, nullptr, occ);
}

int sweep_launch(const spk_system *s, const SweepArgs &A, bool dependent, cudaStream_t st) {
    const int blocks = A.ntasks + A.ncopies;
    if (blocks <= 0) return SPK_OK;
    return launch_any(s->sw_slots, s->sw_wide, nullptr, nullptr, A, blocks, sweep_smem(s), dependent, st);
}

int sweep_launch_multi(const SweepArgs *tab, const int2 *work, int nwork, int slots, bool wide, size_t smem, cudaStream_t st) {
    if (nwork <= 0) return SPK_OK;
    return launch_any(slots, wide, tab, work, SweepArgs{}, nwork, smem, false, st);
}

// The row ranges of phase 3+4 that keep their phase-1 values, in blocks of kCopyRows.
int sweep_copies(spk_system *s, const std::vector<SegTask> &t2) {
    std::vector<int2> c;
    auto add = [&](int lo, int hi) {
        for (; lo < hi; lo += kCopyRows) c.push_back(make_int2(lo, std::min(hi, lo + kCopyRows)));
    };
    for (const SegTask &t : t2) {
        add(t.hi, t.tail);
        add(t.skip_lo, t.skip_hi);
    }
    s->ncopies = (int)c.size();
    SPK_TRY(s->d_copies.alloc(c.size()));
    if (!c.empty())
        SPK_CUDA(cudaMemcpy(s->d_copies.p, c.data(), sizeof(int2) * c.size(), cudaMemcpyHostToDevice));
    return SPK_OK;
}

}  // namespace spk
