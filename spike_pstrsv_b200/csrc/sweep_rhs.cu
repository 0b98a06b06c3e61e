// Back substitution of up to 32 right-hand sides on 16-row records.
//
// The same tiles as the one-right-hand-side kernel (sweep.cu): r = b / a_ii - sum over the
// columns outside the tile, x = W r.  Here a lane owns right-hand sides, so nothing is
// reduced across lanes, and a coefficient is one broadcast read that serves a group of
// lanes.  What bounds it with many tasks in flight is the shared-memory pipe, 128 bytes a
// cycle into registers whether lanes read one address or many: a broadcast FP64
// coefficient costs as much as a window row of 32 right-hand sides.  So a lane takes R
// right-hand sides (a 16-byte read in FP64 at R = 2), and a coefficient serves R products.
//
// Lanes.  A warp's 32 lanes are four groups of eight; group q takes rows 4 k + q of the
// tile, so that four rows advance together and a tile takes four steps.  17 to 32
// right-hand sides run as two warps of 16 (R = 2), 9 to 16 as one, fewer as one of R = 1.
//
// Record.  W by quads of rows (rows 4 i .. 4 i + 3 hold columns from 4 i on, the unit
// diagonal included), 1 / diagonal in FP64, 4 C outside coefficients a row (C a template parameter,
// chosen like the slots of sweep.cu), their columns as row distances from the tile above, and a
// list of what the longer rows have more.
//
// A further warp copies: records by one bulk copy each, the tile's right-hand sides by
// 8-byte asynchronous copies into a padded [right-hand side][row] block, and solved
// tiles out of the window, 16 rows of a column at a time (128-byte runs), when it takes back
// their stage.  The window is a ring of rows padded by one element; its first reach + 16
// rows are mirrored behind its end, so that a column's address is one multiply-add.
// Measured against the kernel of chain.cu (FP64, before -> after): 4,194,304 banded rows, 32
// right-hand sides 1,657 -> 1,445 us (shared-memory pipe), 16: 1,010 -> 890 us; 300,007 rows, band
// of 96, 21 right-hand sides in FP32 1,185 -> 215 us.  A tile with 4 right-hand sides takes
// 1.15 us, with 32 1.3 us (2.1 with two tasks an SM): loads issued row by row in program
// order took 1.7 and 1.8, generic pointers and R = 1 with two groups of lanes 3.3 and 2.9.
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <set>
#include <type_traits>
#include <vector>

#include <cub/cub.cuh>

#include "checks.cuh"
#include "records.cuh"
#include "sweep.cuh"
#include "sweep_rhs.cuh"

namespace spk {

namespace {

constexpr int kMaxStages = 4;
constexpr size_t kMaxSmem = 220 * 1024;
constexpr int kGroups[] = {1, 2, 3, 4, 5, 6};  // C: groups of four outside coefficients a row

__host__ __device__ constexpr int w_rows(int i) { return 16 - 4 * (i / 4); }                 // values of row i in W
__host__ __device__ constexpr int w_at(int i) { return (i / 4) * (64 - 8 * (i / 4 - 1)) + (i & 3) * w_rows(i); }  // its first
static_assert(w_at(4) == 64 && w_at(8) == 112 && w_at(12) == 144 && w_at(15) + w_rows(15) == 160, "quads of W");

template <typename T>
__host__ __device__ constexpr int head_bytes() { return 160 * (int)sizeof(T) + 128; }  // W, 1 / diagonal (FP64)
template <typename T>
__host__ __device__ constexpr int base_bytes(int C) { return head_bytes<T>() + 64 * C * ((int)sizeof(T) + 4) + 16; }
// base: W, 1 / diagonal, values [16][4 C], distances [16][4 C], 16 bytes with the number of extras
// and the rows that have a column outside the tile (a bit each; the others read a zero row beside
// the window, not one they do not depend on); then the extras, 16 bytes each: row, distance, value (FP64)

__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) { return try_wait(bar, parity) || slow_wait(bar, parity); }

// N consecutive values in shared memory (32-bit addresses), in the widest pieces that the
// caller's alignment allows.  volatile: the loads stay in the order written below.
__device__ __forceinline__ void lds2(unsigned a, double &x, double &y) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a) : "memory");
}
__device__ __forceinline__ void lds4(unsigned a, float *v) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ int4 ldsi4(unsigned a) {
    int4 v;
    asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double lds1(unsigned a, double) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float lds1(unsigned a, float) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
template <int N>
__device__ __forceinline__ void lds(unsigned a, double (&v)[N]) {
    if constexpr (N == 1) v[0] = lds1(a, 0.0);
    else
#pragma unroll
        for (int i = 0; i < N / 2; i++) lds2(a + 16 * i, v[2 * i], v[2 * i + 1]);
}
template <int N>
__device__ __forceinline__ void lds(unsigned a, float (&v)[N]) {
    if constexpr (N == 1) v[0] = lds1(a, 0.0f);
    else if constexpr (N == 2) asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "r"(a) : "memory");
    else
#pragma unroll
        for (int i = 0; i < N / 4; i++) lds4(a + 16 * i, v + 4 * i);
}
template <int N>
__device__ __forceinline__ void sts(unsigned a, const double (&v)[N]) {
    if constexpr (N == 1) asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v[0]) : "memory");
    else asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[0]), "d"(v[1]) : "memory");
}
template <int N>
__device__ __forceinline__ void sts(unsigned a, const float (&v)[N]) {
    if constexpr (N == 1) asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v[0]) : "memory");
    else asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v[0]), "f"(v[1]) : "memory");
}

// Shared memory of a task: barriers, r of the tile, a zero row, the window (win + mirror rows), the stages.
// COLS columns padded to keep rows aligned for reads of R columns.
template <typename T, int COLS, int R>
struct Smem {
    static constexpr int LD = COLS + (R * (int)sizeof(T) >= 16 ? 16 / (int)sizeof(T) : R);
    unsigned full, empty;
    T *r, *zero, *win;
    unsigned char *stage;
    __device__ Smem(unsigned char *base, int rows)
        : full(su32(base)), empty(su32(base) + 8 * kMaxStages), r((T *)(base + 128)), zero(r + 16 * LD), win(zero + LD),
          stage((unsigned char *)(((size_t)(win + (size_t)rows * LD) + 127) & ~(size_t)127)) {}
};
template <typename T>
size_t smem_bytes(int cols, int per_lane, int rows, int ns, int stage) {
    const int ld = cols + (per_lane * (int)sizeof(T) >= 16 ? 16 / (int)sizeof(T) : per_lane);
    return 128 + (size_t)(17 + rows) * ld * sizeof(T) + 128 + (size_t)ns * stage;
}

// One task's walk over rows [lo, hi), as every warp of the block sees it.
struct Range {
    int lo, hi, jt, jb;
    __device__ Range(int lo_, int hi_) : lo(lo_), hi(hi_), jt((hi_ - 1) >> 4), jb(lo_ >> 4) {}
};

// Solved rows [r0, r0 + 16) of tile j, ring rows from `pos` on, out of the window: the lanes
// take 16 rows of two columns at a time.
template <typename T, int COLS, int R>
__device__ __forceinline__ void store_tile(const RhsSweep &A, const Smem<T, COLS, R> &M, int j, int pos, int lo, int hi, int lane) {
    const int i = lane & 15, row = 16 * j + i;
    if (row < lo || row >= hi) return;
    const long long o = CK(A.rev_x ? (long long)A.n - 1 - row : row, A.n, 84);
    const T *w = M.win + (pos + i) * M.LD;
    if (A.out_work) {
        T *x = (T *)A.X + o;
#pragma unroll 4
        for (int k = lane >> 4; k < A.nk; k += 2) x[k * A.ldx] = w[k];
    } else if (A.acc) {
        double *x = (double *)A.X + o;
        double old[COLS / 2];
#pragma unroll
        for (int u = 0; u < COLS / 2; u++) {
            const int k = 2 * u + (lane >> 4);
            if (k < A.nk) old[u] = x[k * A.ldx];
        }
#pragma unroll
        for (int u = 0; u < COLS / 2; u++) {
            const int k = 2 * u + (lane >> 4);
            if (k < A.nk) x[k * A.ldx] = old[u] + (double)w[k];
        }
    } else {
        double *x = (double *)A.X + o;
#pragma unroll 4
        for (int k = lane >> 4; k < A.nk; k += 2) x[k * A.ldx] = (double)w[k];
    }
}

// The copying warp over one range: each tile's record and right-hand sides into the ring of
// stages; before a stage is used again, the tile it held out of the window (the last
// ones at the end).  pos: ring row of tile jt.  False after a wait that gave up.
template <typename T, int COLS, int PER>
__device__ bool copy_range(const RhsSweep &A, const Smem<T, COLS, PER> &M, Ring &R, const Range &g, int pos, int st_lo, int st_hi,
                           int lane) {
    const int tiles = g.jt - g.jb + 1, slo = max(g.lo, st_lo), shi = min(g.hi, st_hi);
    int2 h = make_int2(0, 0);
    Ring S = R;  // the next tile to store
    auto solved = [&]() { return bar_wait(M.empty + 8 * S.slot, S.parity); };
    auto store_next = [&](int t) {
        S.next(A.ns);
        store_tile<T, COLS, PER>(A, M, g.jt - t, pos, slo, shi, lane);
        pos = pos == 0 ? A.win - 16 : pos - 16;
    };
    for (int t = 0; t < tiles; t++) {
        // the stage's last use: this range's, or the range's before (stored already)
        if (!(t >= A.ns ? solved() : bar_wait(M.empty + 8 * R.slot, R.parity ^ 1))) return false;
        const int j = g.jt - t, k = t & 31;
        if (k == 0) h = j - lane >= g.jb ? __ldg(A.hdr + CK(j - lane, (A.n + 15) >> 4, 80)) : make_int2(0, 0);
        const unsigned at = __shfl_sync(kFull, h.x, k), bytes = CKU(__shfl_sync(kFull, h.y, k), A.stage - COLS * 17 * 8 + 1, 81);
        const unsigned bar = M.full + 8 * R.slot;
        unsigned char *dst = M.stage + (size_t)R.slot * A.stage;
        if (lane == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             su32(dst)),
                         "l"(A.rec + CK((unsigned long long)at * 16, A.nrec - bytes + 1, 82)), "r"(bytes), "r"(bar)
                         : "memory");
        }
        const int i = lane & 15, row = 16 * j + i;
        if (row >= g.lo && row < g.hi) {
            const double *src = A.B + CK(A.rev_b ? (long long)A.n - 1 - row : (long long)row, A.n, 83);
            const unsigned b = su32(dst + A.stage - COLS * 17 * 8) + 8 * i;
#pragma unroll 4
            for (int c = lane >> 4; c < A.nk; c += 2)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(b + c * 17 * 8), "l"(src + c * A.ldb) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
        R.next(A.ns);
        if (t >= A.ns) store_next(t - A.ns);  // after the copies: they are on the next tiles' path
    }
    for (int t = max(0, tiles - A.ns); t < tiles; t++) {
        if (!solved()) return false;
        store_next(t);
    }
    return true;
}

// What the rows of a cut tile read of its rows from hi up.
template <typename T>
__device__ __noinline__ double cut_sum(const int *ia, const int *ja, const double *a, const T *win, int ld, int pos, int row,
                                       int hi) {
    const int e0 = ia[row], e1 = ia[row + 1], top = (row | 15) + 1;
    double s = 0.0;
    for (int e = e0 + 1; e < e1 && ja[e] < top; e++)
        if (ja[e] >= hi) s = fma(a[e], (double)win[(pos + (ja[e] & 15)) * ld], s);
    return s / a[e0];
}

// A solving warp over one range; w: which of the task's solving warps.  The loads are
// written in the order they should issue: a row's gathers before the next row's column
// distances and its own coefficients, all before its products; all of r's readers before
// the products with W.
template <typename T, int R, int NW, int C>
__device__ bool solve_range(const RhsSweep &A, const Smem<T, NW * 8 * R, R> &M, Ring &ring, const Range &g, int &pos, int w,
                            int lane) {
    constexpr int COLS = NW * 8 * R, B = (int)sizeof(T), LD = Smem<T, COLS, R>::LD * B;
    const int q = lane >> 3, col = (w * 8 + (lane & 7)) * R;
    const unsigned wcol = su32(M.win) + col * B, rcol = su32(M.r) + col * B, st0 = su32(M.stage);
    const unsigned boff = A.stage - COLS * 17 * 8 + col * 17 * 8 + 8 * q;
    bool ready = false;
    for (int j = g.jt; j >= g.jb; j--) {
        const unsigned st = st0 + ring.slot * A.stage, release = M.empty + 8 * ring.slot;
        if (!ready && !bar_wait(M.full + 8 * ring.slot, ring.parity)) return false;
        ring.next(A.ns);
        const unsigned rd = st + 160 * B, val = st + head_bytes<T>(), off = val + 64 * C * B;
        const int above = pos + 16 == A.win ? 0 : pos + 16;  // ring row of the tile above
        const unsigned gat = wcol + above * LD, zero = rcol + 16 * LD;
        const bool top = 16 * j + 16 > g.hi, bottom = 16 * j < g.lo;
        T r[4][R];
        int4 o[C];
#pragma unroll
        for (int e = 0; e < C; e++) o[e] = ldsi4(off + 16 * (C * q + e));
        int ne, has;
        asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(ne), "=r"(has) : "r"(st + base_bytes<T>(C) - 16) : "memory");
        has >>= q;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            T x[4 * C][R], v[4 * C];
            const unsigned from = has >> 4 * k & 1 ? gat : zero;  // distances of a row without any are 0
#pragma unroll
            for (int e = 0; e < C; e++) {
                lds(from + CKU(o[e].x, max(A.reach, 1), 85) * LD, x[4 * e]);
                lds(from + CKU(o[e].y, max(A.reach, 1), 85) * LD, x[4 * e + 1]);
                lds(from + CKU(o[e].z, max(A.reach, 1), 85) * LD, x[4 * e + 2]);
                lds(from + CKU(o[e].w, max(A.reach, 1), 85) * LD, x[4 * e + 3]);
            }
            lds(val + 4 * C * B * (4 * k + q), v);
            if (k < 3)
#pragma unroll
                for (int e = 0; e < C; e++) o[e] = ldsi4(off + 16 * (C * (4 * k + 4 + q) + e));
            const double d = lds1(rd + 8 * (4 * k + q), 0.0);
            double b[R];
#pragma unroll
            for (int u = 0; u < R; u++) {
                b[u] = lds1(st + boff + 17 * 8 * u + 32 * k, 0.0);
                // a right-hand side past FP32's range overflows in FP32, as the values would
                if (sizeof(T) == 4) b[u] = fabs(b[u]) <= 3.4028234663852886e38 ? b[u] : b[u] * 1e308;
            }
            T s[2][R];
#pragma unroll
            for (int u = 0; u < R; u++) s[0][u] = s[1][u] = T(0);
#pragma unroll
            for (int e = 0; e < 4 * C; e++)
#pragma unroll
                for (int u = 0; u < R; u++) s[e & 1][u] = fma(v[e], x[e][u], s[e & 1][u]);
#pragma unroll
            for (int u = 0; u < R; u++) r[k][u] = (T)fma(b[u], d, -(double)(s[0][u] + s[1][u]));  // FP32: one rounding
        }
        if (top || bottom) {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int row = 16 * j + 4 * k + q;
#pragma unroll
                for (int u = 0; u < R; u++) {
                    // above the task's top the rows are known, below its last no right-hand side was copied
                    if (row >= g.hi || row < g.lo) r[k][u] = T(0);
                    else if (top && g.hi < A.n && A.pre)
                        r[k][u] -= (T)cut_sum<T>(A.ia, A.ja, A.a, M.win + col + u, LD / B, pos, row, g.hi);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) sts(rcol + (4 * k + q) * LD, r[k]);
        if (ne) {
            __syncwarp();
            const unsigned ex = st + base_bytes<T>(C);
            for (int e = 0; e < ne; e++) {
                const int4 at = ldsi4(ex + 16 * e);
                if ((at.x & 3) == q && !(top && 16 * j + at.x >= g.hi) && !(bottom && 16 * j + at.x < g.lo)) {
                    T x[R], y[R];
                    lds(gat + CKU(at.y, max(A.reach, 1), 86) * LD, x);
                    lds(rcol + CKU(at.x, 16, 87) * LD, y);
                    const T v = (T)__hiloint2double(at.w, at.z);
#pragma unroll
                    for (int u = 0; u < R; u++) y[u] = fma(-v, x[u], y[u]);
                    sts(rcol + at.x * LD, y);
                }
            }
        }
        __syncwarp();
        T rr[16][R], wv[10][4];
#pragma unroll
        for (int c = 15; c >= 0; c--) lds(rcol + c * LD, rr[c]);
#pragma unroll
        for (int k = 0, m = 0; k < 4; k++)
#pragma unroll
            for (int c = 12; c >= 4 * k; c -= 4, m++) lds(st + B * (w_at(4 * k) + q * w_rows(4 * k) + c - 4 * k), wv[m]);
        ready = j > g.jb && try_wait(M.full + 8 * ring.slot, ring.parity);
#pragma unroll
        for (int k = 0, m = 0; k < 4; k++) {
#pragma unroll
            for (int u = 0; u < R; u++) r[k][u] = T(0);
#pragma unroll
            for (int c = 12; c >= 4 * k; c -= 4, m++)  // the diagonal last but for zeros
#pragma unroll
                for (int f = 3; f >= 0; f--)
#pragma unroll
                    for (int u = 0; u < R; u++) r[k][u] = fma(wv[m][f], rr[c + f][u], r[k][u]);
        }
        const unsigned out = wcol + (pos + q) * LD, twin = out + A.win * LD;
        const bool twice = pos < A.mirror;
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (!top || 16 * j + 4 * k + q < g.hi) sts(out + 4 * k * LD, r[k]);
        if (twice)
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (!top || 16 * j + 4 * k + q < g.hi) sts(twin + 4 * k * LD, r[k]);
        __syncwarp();  // the window rows; every lane is done with the stage and with r
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(release) : "memory");
        pos = pos == 0 ? A.win - 16 : pos - 16;
    }
    return true;
}

template <typename T, int PER, int NW, int C>
__device__ __forceinline__ void rhs_task(const RhsSweep &A, int task) {
    constexpr int COLS = NW * 8 * PER, LD = Smem<T, COLS, PER>::LD;
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (A.fail_entry) {
        if (threadIdx.x == 0) atomicExch(A.err, 1);
        return;
    }
    if (task >= A.ntasks) {  // rows that keep the phase-1 values
        const int2 c = A.copies[task - A.ntasks];
        const T *pre = (const T *)A.pre;
        for (int k = 0; k < A.nk; k++)
            for (int r = c.x + (int)threadIdx.x; r < c.y; r += blockDim.x) {
                double *x = (double *)A.X + k * A.ldx + CK(A.rev_x ? A.n - 1 - r : r, A.n, 88);
                const double v = (double)pre[(long long)k * A.n + r];
                *x = A.acc ? *x + v : v;
            }
        return;
    }
    const Smem<T, COLS, PER> M(smem, A.win + A.mirror);
    if (threadIdx.x == 0) {
        for (int k = 0; k < A.ns; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(M.full + 8 * k), "r"(33u) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(M.empty + 8 * k), "r"((unsigned)NW) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
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
    Ring R;
    bool ok = true;
    // row r has ring row r modulo win
    auto load_window = [&](int r0, int count) {
        const T *pre = (const T *)A.pre;
        const int p0 = r0 % A.win;
        for (int e = threadIdx.x; e < count * COLS; e += NW * 32) {
            const int k = e / count, i = e - k * count, r = r0 + i, p = p0 + i >= A.win ? p0 + i - A.win : p0 + i;
            const T v = pre && r < A.n && k < A.nk ? pre[(long long)k * A.n + r] : T(0);
            M.win[CK(p, A.win, 89) * LD + k] = v;
            if (p < A.mirror) M.win[(p + A.win) * LD + k] = v;
        }
    };
    if (threadIdx.x < COLS) M.zero[threadIdx.x] = T(0);
    for (int part = 0; part < (two ? 2 : 1); part++) {
        const Range g = part ? Range(lo, skip_lo) : Range(lo1, hi);
        // the second range reads the rows between, and above them those of the first
        if (warp < NW) load_window(g.hi, part ? min(skip_hi - skip_lo, A.reach) : A.reach);
        __syncthreads();
        if (g.lo < g.hi) {
            int pos = (int)((16ll * g.jt) % A.win);
            if (warp < NW) ok = solve_range<T, PER, NW, C>(A, M, R, g, pos, warp, lane);
            else ok = copy_range<T, COLS, PER>(A, M, R, g, pos, st_lo, st_hi, lane);
        }
        if (!__syncthreads_and(ok)) break;
    }
    if (!ok) {
        if (warp == NW)  // no copy may land after the block is gone
            for (int k = 0; k < A.ns; k++) {
                if (R.slot == 0) R.parity ^= 1;
                R.slot = R.slot == 0 ? A.ns - 1 : R.slot - 1;
                slow_wait(M.full + 8 * R.slot, R.parity);
            }
        if (lane == 0) atomicExch(A.err, 1);
    }
}

template <typename T, int PER, int NW, int C>
__global__ void __launch_bounds__(32 * (NW + 1)) k_sweep_rhs(const RhsSweep *__restrict__ tab, const int2 *__restrict__ work,
                                                             RhsSweep one) {
    if (tab) {
        const int2 w = work[blockIdx.x];
        const RhsSweep A = tab[w.x];
        rhs_task<T, PER, NW, C>(A, w.y);
    } else {
        rhs_task<T, PER, NW, C>(one, blockIdx.x);
    }
}

// ---- records ------------------------------------------------------------------------

// A lane's slots in the one-right-hand-side record: slot u of S (then of the E extra).
template <bool WIDE>
__device__ __forceinline__ void sw_slot(const unsigned char *R, int S, int E, int u, int lane, double &v, int &o) {
    const unsigned char *at = R + kHead;
    int count = S;
    if (u >= S) {
        at += slot_bytes(S, WIDE);
        count = E;
        u -= S;
    }
    v = ((const double *)at)[((u >> 1) * 32 + lane) * 2 + (u & 1)];
    at += 256 * count;
    o = WIDE ? ((const unsigned short *)at)[((u >> 1) * 32 + lane) * 2 + (u & 1)] : at[((u >> 2) * 32 + lane) * 4 + (u & 3)];
}

__device__ __forceinline__ int extra_slots(const unsigned char *R) { return *(const int *)(R + kExtra) & 0xffff; }

__device__ __forceinline__ int lane_row(int lane) { return (lane & 2) ? 15 - (lane >> 2) : lane >> 2; }

// Outside coefficients of this lane's row up to the last nonzero one.
template <bool WIDE>
__device__ __forceinline__ int row_count(const unsigned char *R, int S, int E, int lane) {
    int c = 0;
    for (int u = 0; u < S + E; u++) {
        double v;
        int o;
        sw_slot<WIDE>(R, S, E, u, lane, v, o);
        if (v != 0.0) c = 2 * u + (lane & 1) + 1;
    }
    return max(c, __shfl_xor_sync(kFull, c, 1));
}

// Records with extras: the size of each in units of 16 bytes, and the largest.  A warp per tile.
template <bool WIDE>
__global__ void k_rhs_sizes(int nt, const int2 *__restrict__ sw_hdr, const unsigned char *__restrict__ sw_rec, int S, int C,
                            int base, unsigned *__restrict__ size, unsigned *__restrict__ most) {
    const int lane = threadIdx.x & 31, j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= nt) return;
    const unsigned char *R = sw_rec + (unsigned long long)(unsigned)sw_hdr[j].x * 16;
    int e = max(0, row_count<WIDE>(R, S, extra_slots(R), lane) - 4 * C);
    e = (lane & 1) ? 0 : e;
#pragma unroll
    for (int o = 16; o; o >>= 1) e += __shfl_xor_sync(kFull, e, o);
    if (lane == 0) {
        size[j] = base / 16 + e;
        atomicMax(most, base / 16 + e);
    }
}

__global__ void k_rhs_headers(int nt, const unsigned *__restrict__ size, const unsigned *__restrict__ at, int2 *__restrict__ hdr) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nt) hdr[j] = make_int2((int)at[j], (int)(16 * size[j]));
}

template <typename T, bool WIDE>
__global__ void k_rhs_fill(int nt, const int2 *__restrict__ sw_hdr, const unsigned char *__restrict__ sw_rec, int S,
                           int C, int extras, int2 *__restrict__ hdr, unsigned char *__restrict__ rec) {
    const int lane = threadIdx.x & 31, j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (j >= nt) return;
    const unsigned char *R = sw_rec + (unsigned long long)(unsigned)sw_hdr[j].x * 16;
    if (!extras && lane == 0) hdr[j] = make_int2((int)((unsigned)j * (base_bytes<T>(C) / 16)), base_bytes<T>(C));
    unsigned char *D = rec + (extras ? (unsigned long long)(unsigned)hdr[j].x : (unsigned long long)j * (base_bytes<T>(C) / 16)) * 16;
    const int E = extra_slots(R);
    T *W = (T *)D, *val = (T *)(D + head_bytes<T>());
    int *off = (int *)(val + 64 * C);
    const double *Wf = (const double *)R;
#pragma unroll
    for (int e0 = 0; e0 < 160; e0 += 32) {
        const int at = e0 + lane, k = at < 64 ? 0 : at < 112 ? 1 : at < 144 ? 2 : 3, in = at - w_at(4 * k);
        const int i = 4 * k + in / w_rows(4 * k), c = 4 * k + in % w_rows(4 * k);
        double v = c == i ? 1.0 : 0.0;
        if (c > i) {
            const int g = i < 8 ? i : 15 - i, e = i < 8 ? c - i - 1 : c - 1, u = e >> 2, l = 4 * g + (e & 3);
            v = Wf[((u >> 1) * 32 + l) * 2 + (u & 1)];
        }
        W[at] = (T)v;
    }
    if (lane < 16) ((double *)(W + 160))[lane] = ((const double *)(R + kDiag))[lane];
    // extras of the rows before each: rows in order
    const int mine = lane & 15, held = row_count<WIDE>(R, S, E, lane);
    const int c = __shfl_sync(kFull, held, mine < 8 ? 4 * mine : 4 * (15 - mine) + 2), ex = max(0, c - 4 * C);
    int before = lane < 16 ? ex : 0;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const int t = __shfl_up_sync(kFull, before, o);
        if (lane >= o) before += t;
    }
    const int total = __shfl_sync(kFull, before, 15);
    before -= ex;
    const int row = lane_row(lane), rc = __shfl_sync(kFull, c, row), rb = __shfl_sync(kFull, before, row);
    const unsigned out = __ballot_sync(kFull, lane < 16 && c > 0);
    if (lane == 0) *(int4 *)(D + base_bytes<T>(C) - 16) = make_int4(total, (int)out, 0, 0);
    for (int at = lane; at < 64 * C; at += 32) {  // in the order of the record; unused places repeat the row's first column
        const int i = at / (4 * C), q = at - 4 * C * i, ci = __shfl_sync(kFull, c, i);
        const int l0 = i < 8 ? 4 * i : 4 * (15 - i) + 2;  // the first lane of row i
        double v = 0.0;
        int o = 0;
        if (q < ci) sw_slot<WIDE>(R, S, E, q >> 1, l0 + (q & 1), v, o);
        else if (ci) {
            sw_slot<WIDE>(R, S, E, 0, l0, v, o);
            v = 0.0;
        }
        val[at] = (T)v;
        off[at] = o;
    }
    unsigned char *X = D + base_bytes<T>(C);
    for (int q = 4 * C + (lane & 1); q < rc; q += 2) {
        double v;
        int o;
        sw_slot<WIDE>(R, S, E, q >> 1, lane, v, o);
        unsigned char *at = X + 16ll * (rb + q - 4 * C);
        *(int2 *)at = make_int2(row, o);
        *(double *)(at + 8) = v;
    }
}

// ---- host ---------------------------------------------------------------------------

struct Launch {
    const RhsSweep *tab;
    const int2 *work;
    RhsSweep one;
    int blocks;
    size_t smem;
    cudaStream_t st;
};

template <typename T, int PER, int NW, int C>
int launch_one(const Launch &L) {
    auto kern = k_sweep_rhs<T, PER, NW, C>;
    SPK_TRY(allow_smem(kern));
    kern<<<L.blocks, 32 * (NW + 1), L.smem, L.st>>>(L.tab, L.work, L.one);
    SPK_CUDA(cudaGetLastError());
    return SPK_OK;
}

template <typename T, int PER, int NW>
int launch_c(int C, const Launch &L) {
    switch (C) {
        case 1: return launch_one<T, PER, NW, 1>(L);
        case 2: return launch_one<T, PER, NW, 2>(L);
        case 3: return launch_one<T, PER, NW, 3>(L);
        case 4: return launch_one<T, PER, NW, 4>(L);
        case 5: return launch_one<T, PER, NW, 5>(L);
        default: return launch_one<T, PER, NW, 6>(L);
    }
}

// Classes: shape (how the columns of a task are dealt) times C.
struct Shape {
    int cols, per, warps;
};
constexpr Shape kShapes[] = {{32, 2, 2}, {16, 2, 1}, {8, 1, 1}};
int shape_of(int nk) { return nk > 16 ? 0 : (nk > 8 ? 1 : 2); }

int launch_class(int cls, int fp32, const Launch &L) {
    const int C = cls % 16;
    switch (cls / 16 + (fp32 ? 3 : 0)) {
        case 0: return launch_c<double, 2, 2>(C, L);
        case 1: return launch_c<double, 2, 1>(C, L);
        case 2: return launch_c<double, 1, 1>(C, L);
        case 3: return launch_c<float, 2, 2>(C, L);
        case 4: return launch_c<float, 2, 1>(C, L);
        default: return launch_c<float, 1, 1>(C, L);
    }
}

int ring_rows(const spk_system *s, int ns) { return (std::max(s->sw_reach + 32, 16 * ns + 16) + 15) & ~15; }

}  // namespace

void rhs_sweep_release(spk_system *s) {
    for (int f = 0; f < 2; f++) {
        s->rs_ok[f] = 0;
        s->rs_rec[f].release();
        s->rs_hdr[f].release();
    }
}

// Groups of four on the common path: the fewest coefficients read, an extra one counted sixty
// times (a dependent chain of its own with one group of lanes at work: about 150 cycles).
void rhs_sweep_choose(spk_system *s, const int *hist, int most) {
    double best = 0;
    s->rs_groups = 0;
    for (int c : kGroups) {
        double cost = 0;
        long long extras = 0;
        for (int k = 0; k <= most; k++) {
            cost += hist[k] * (4.0 * c + 60.0 * std::max(0, k - 4 * c));
            extras += (long long)hist[k] * std::max(0, k - 4 * c);
        }
        if (!s->rs_groups || cost < best) s->rs_groups = c, s->rs_extras = extras, best = cost;
    }
}

int rhs_sweep_prepare(spk_system *s, int fp32) {
    if (s->rs_ok[fp32] || !s->sw_ok) return SPK_OK;
    SPK_TRY(debug_no_memory(s));
    const int nt = (s->n + 15) / 16, S = s->sw_slots, C = s->rs_groups, blocks = (nt + 3) / 4;
    const int base = fp32 ? base_bytes<float>(C) : base_bytes<double>(C);
    cudaStream_t st = s->stream;
    if ((long long)nt * (base / 16) + s->rs_extras >= (1ll << 32)) return SPK_OK;  // offsets are 32-bit, in 16 bytes
    SPK_TRY(s->rs_hdr[fp32].alloc(nt));
    unsigned all = (unsigned)nt * (base / 16), most = base / 16;
    if (s->rs_extras) {
        // sizes, offsets (a last element each: the largest size, the sum) and the scan's space
        size_t scan = 0;
        SPK_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan, (unsigned *)nullptr, (unsigned *)nullptr, nt + 1, st));
        DBuf<unsigned char> scratch(st);
        const size_t words = ((size_t)nt + 2 + 63) / 64 * 64;
        SPK_TRY(scratch.alloc(8 * words + scan));
        unsigned *const size = (unsigned *)scratch.p, *const first = size + words;
        SPK_CUDA(cudaMemsetAsync(size + nt, 0, 2 * sizeof(unsigned), st));
        if (s->sw_wide) k_rhs_sizes<true><<<blocks, 128, 0, st>>>(nt, s->sw_hdr.p, s->sw_rec.p, S, C, base, size, size + nt + 1);
        else k_rhs_sizes<false><<<blocks, 128, 0, st>>>(nt, s->sw_hdr.p, s->sw_rec.p, S, C, base, size, size + nt + 1);
        SPK_CUDA(cudaGetLastError());
        SPK_CUDA(cub::DeviceScan::ExclusiveSum(scratch.p + 8 * words, scan, size, first, nt + 1, st));
        k_rhs_headers<<<(nt + 255) / 256, 256, 0, st>>>(nt, size, first, s->rs_hdr[fp32].p);
        SPK_CUDA(cudaGetLastError());
        SPK_CUDA(cudaMemcpyAsync(&all, first + nt, sizeof(all), cudaMemcpyDeviceToHost, st));
        SPK_CUDA(cudaMemcpyAsync(&most, size + nt + 1, sizeof(most), cudaMemcpyDeviceToHost, st));
        SPK_CUDA(cudaStreamSynchronize(st));
    }
    SPK_TRY(s->rs_rec[fp32].alloc((size_t)all * 16));
    auto fill = [&](auto kern) {
        kern<<<blocks, 128, 0, st>>>(nt, s->sw_hdr.p, s->sw_rec.p, S, C, s->rs_extras > 0, s->rs_hdr[fp32].p, s->rs_rec[fp32].p);
    };
    if (fp32) s->sw_wide ? fill(k_rhs_fill<float, true>) : fill(k_rhs_fill<float, false>);
    else s->sw_wide ? fill(k_rhs_fill<double, true>) : fill(k_rhs_fill<double, false>);
    SPK_CUDA(cudaGetLastError());
    SPK_CUDA(cudaStreamSynchronize(st));
    s->rs_bytes[fp32] = 16 * (int)most;
    s->rs_ok[fp32] = 1;
    return SPK_OK;
}

long long rhs_sweep_device_check() { return first_failed_check(); }

RhsSweep rhs_sweep_args(const spk_system *s, int fp32, int nk) {
    RhsSweep A{};
    A.hdr = s->rs_hdr[fp32].p;
    A.rec = s->rs_rec[fp32].p;
    A.nrec = (long long)s->rs_rec[fp32].n;
    A.n = s->n;
    A.nk = nk;
    A.reach = s->sw_reach;
    A.shape = shape_of(nk);
    A.stage = ((s->rs_bytes[fp32] + 127) & ~127) + kShapes[A.shape].cols * 17 * 8;
    A.ns = 4;
    A.win = ring_rows(s, A.ns);
    A.mirror = (A.reach + 31) & ~15;
    A.ia = s->uia.p;
    A.ja = s->uja.p;
    A.a = s->ua.p;
    A.err = s->d_err.p;
    A.fail_entry = s->dbg_fail_waits > 0;
    return A;
}

size_t rhs_sweep_smem(const spk_system *s, int fp32, int nk) {
    const RhsSweep A = rhs_sweep_args(s, fp32, nk);
    const Shape &h = kShapes[A.shape];
    const int rows = A.win + A.mirror;
    return fp32 ? smem_bytes<float>(h.cols, h.per, rows, A.ns, A.stage)
                : smem_bytes<double>(h.cols, h.per, rows, A.ns, A.stage);
}

bool rhs_sweep_fits(const spk_system *s, int fp32, int nk) {
    return s->rs_ok[fp32] && rhs_sweep_smem(s, fp32, nk) <= kMaxSmem;
}

int rhs_sweep_class(const spk_system *s, int fp32, int nk) {
    return 16 * rhs_sweep_args(s, fp32, nk).shape + s->rs_groups;
}

int rhs_sweep_launch(const spk_system *s, const RhsSweep &A, int fp32, cudaStream_t st) {
    Launch L{};
    L.one = A;
    L.blocks = A.ntasks + A.ncopies;
    if (L.blocks <= 0) return SPK_OK;
    L.smem = rhs_sweep_smem(s, fp32, A.nk);
    L.st = st;
    return launch_class(rhs_sweep_class(s, fp32, A.nk), fp32, L);
}

int rhs_sweep_launch_multi(const RhsSweep *tab, const int2 *work, int nwork, int cls, int fp32, size_t smem,
                           cudaStream_t st) {
    if (nwork <= 0) return SPK_OK;
    Launch L{};
    L.tab = tab;
    L.work = work;
    L.blocks = nwork;
    L.smem = smem;
    L.st = st;
    return launch_class(cls, fp32, L);
}

}  // namespace spk
