// R = B - A X in FP64 for 2 to 32 right-hand sides, with the norms of a scaled residual.
//
// A block takes 128 rows (U order) and copies what they read, the matrix's slots and 128 +
// reach rows of X ([row][column], padded), into shared memory at once, so that the memory's
// latency is met once a block and a few blocks an SM keep it busy.  A lane owns COLS / 8
// columns, in pairs that a quarter warp reads as 128 contiguous bytes, and a quarter warp a
// row: a coefficient read once serves all columns of its row.  32 rows at a time go back
// through shared memory so that B and R move 32 rows of a column together.
// What bounds it is the shared-memory pipe (a row of X per coefficient).  The kernel it
// replaces walked 32 tiles in series in two blocks an SM: 300,007 rows, 21 columns, band of
// 96: 266 -> 96 us (global loads in the slot loop: 193 us).
#include <algorithm>
#include <mutex>
#include <set>

#include "checks.cuh"
#include "spk_internal.cuh"

namespace spk {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kRows = 128, kThreads = 256;

// max(m, v) that does not lose a NaN
__device__ __forceinline__ double nanmax(double m, double v) { return (v > m || v != v) ? v : m; }

struct ResArgs {
    int n, nk, rows, slots;  // rows of X and slots in shared memory
    const int *ptr;
    const double *ev;
    const int *ec;
    const double *diag;
    const double *X;
    long long ldx;
    const double *B;
    long long ldb;
    double *R;
    long long ldr;
    int rev;
    unsigned long long *norms;  // max |R|, |X|, |B| per column, or null
    long long nell;             // matrix slots (bounds of the checked build)
};

__device__ __forceinline__ void cpa(unsigned dst, const void *src, int bytes) {
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

template <int COLS>
__global__ void __launch_bounds__(kThreads) k_residual_block(ResArgs A) {
    constexpr int P = COLS / 8, LD = COLS + (P >= 2 ? 2 : 1), W = kThreads / 32, CW = (COLS + W - 1) / W;
    extern __shared__ __align__(16) double xs[];  // [rows][LD], [32][LD], slot values, slot columns
    double *const os = xs + (size_t)A.rows * LD, *const vs = os + 32 * LD;
    int *const cs = (int *)(vs + A.slots);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r0 = blockIdx.x * kRows;
    const int nt = (A.n + 31) >> 5, j0 = r0 >> 5, p0 = __ldg(A.ptr + j0), p1 = __ldg(A.ptr + min(j0 + kRows / 32, nt));
    auto in_rows = [&](int c) { return (long long)r0 + CK(c - r0, A.rows, 123); };  // a column, among the rows of X copied
    auto at = [&](int r) { return A.rev ? (long long)A.n - 1 - r : (long long)r; };
    const unsigned xa = (unsigned)__cvta_generic_to_shared(xs), va = (unsigned)__cvta_generic_to_shared(vs),
                   ca = (unsigned)__cvta_generic_to_shared(cs);
    for (int e = 4 * threadIdx.x; e < p1 - p0; e += 4 * kThreads) {  // tiles hold multiples of 32 slots
        const int at = (int)CK(e, A.slots - 3, 120), from = (int)CK(p0 + e, A.nell - 3, 121);
        cpa(va + 8 * at, A.ev + from, 16);
        cpa(va + 8 * at + 16, A.ev + from + 2, 16);
        cpa(ca + 4 * at, A.ec + from, 16);
    }
    for (int c = warp; c < A.nk; c += W) {
        const double *x = A.X + c * A.ldx;
        for (int i = lane; i < A.rows; i += 32)
            if (r0 + i < A.n) cpa(xa + 8 * (i * LD + c), x + CK(at(r0 + i), A.n, 122), 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int q = lane >> 3, col = (lane & 7) * (P >= 2 ? 2 : 1);  // columns col, col + 1, col + 16, col + 17
    double mr[CW], mx[CW], mb[CW];
#pragma unroll
    for (int u = 0; u < CW; u++) mr[u] = mx[u] = mb[u] = 0.0;
    auto row_of = [&](const double *y, double (&v)[P]) {
        if constexpr (P == 1) {
            v[0] = y[0];
        } else {
#pragma unroll
            for (int u = 0; u < P; u += 2) {
                const double2 t = *(const double2 *)(y + 8 * u);
                v[u] = t.x, v[u + 1] = t.y;
            }
        }
    };
    for (int t = 0; t < kRows / 32 && r0 + 32 * t < A.n; t++) {
        const int i = 4 * warp + q, r = r0 + 32 * t + i;  // this group's row
        const int rr = r0 + 32 * t + lane;                // later a lane is a row
        const long long o = at(rr);
        double b[CW];
#pragma unroll
        for (int u = 0; u < CW; u++) b[u] = rr < A.n && warp + W * u < A.nk ? A.B[(warp + W * u) * A.ldb + o] : 0.0;
        if (r < A.n) {
            const int j = r >> 5, s0 = __ldg(A.ptr + j), w = (__ldg(A.ptr + j + 1) - s0) >> 5;
            const double *ev = vs + (s0 - p0) + i, *x0 = xs + col - (long long)r0 * LD;
            const int *ec = cs + (s0 - p0) + i;
            double a0[P], a1[P], y0[P], y1[P];
#pragma unroll
            for (int u = 0; u < P; u++) a0[u] = a1[u] = 0.0;
            int k = 0;
#pragma unroll 4
            for (; k + 2 <= w; k += 2) {
                const double v0 = ev[32 * k], v1 = ev[32 * k + 32];
                row_of(x0 + in_rows(ec[32 * k]) * LD, y0);
                row_of(x0 + in_rows(ec[32 * k + 32]) * LD, y1);
#pragma unroll
                for (int u = 0; u < P; u++) {
                    a0[u] = fma(v0, y0[u], a0[u]);
                    a1[u] = fma(v1, y1[u], a1[u]);
                }
            }
            if (k < w) {
                const double v = ev[32 * k];
                row_of(x0 + in_rows(ec[32 * k]) * LD, y0);
#pragma unroll
                for (int u = 0; u < P; u++) a0[u] = fma(v, y0[u], a0[u]);
            }
            const double d = A.diag[r];
            row_of(x0 + (long long)r * LD, y0);
#pragma unroll
            for (int u = 0; u < P; u++)
                os[i * LD + col + (P == 1 ? 0 : 16 * (u / 2) + (u & 1))] = fma(d, y0[u], a0[u] + a1[u]);
        }
        __syncthreads();
        if (rr < A.n) {
#pragma unroll
            for (int u = 0; u < CW; u++) {
                const int c = warp + W * u;
                if (c < A.nk) {
                    const double res = b[u] - os[lane * LD + c];
                    A.R[c * A.ldr + CK(o, A.n, 124)] = res;
                    mr[u] = nanmax(mr[u], fabs(res));
                    mx[u] = nanmax(mx[u], fabs(xs[(32 * t + lane) * LD + c]));
                    mb[u] = nanmax(mb[u], fabs(b[u]));
                }
            }
        }
        __syncthreads();
    }
    if (!A.norms) return;
#pragma unroll
    for (int u = 0; u < CW; u++) {
        const int c = warp + W * u;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            mr[u] = nanmax(mr[u], __shfl_xor_sync(kFull, mr[u], o));
            mx[u] = nanmax(mx[u], __shfl_xor_sync(kFull, mx[u], o));
            mb[u] = nanmax(mb[u], __shfl_xor_sync(kFull, mb[u], o));
        }
        if (lane == 0 && c < A.nk) {
            atomicMax(&A.norms[3 * c + 0], __double_as_longlong(mr[u]));
            atomicMax(&A.norms[3 * c + 1], __double_as_longlong(mx[u]));
            atomicMax(&A.norms[3 * c + 2], __double_as_longlong(mb[u]));
        }
    }
}

template <int COLS>
size_t smem_of(int rows, int slots) {
    return (size_t)(rows + 32) * (COLS + (COLS >= 16 ? 2 : 1)) * sizeof(double) + 12 * (size_t)slots;
}

// Rows of X that 128 rows read; even, so that the slots behind them stay 16-byte aligned at an odd
// row length.
int rows_of(const spk_system *s) { return (std::max(kRows, kRows - 32 + s->ell_reach + 1) + 1) & ~1; }

template <int COLS>
int go(const ResArgs &A, cudaStream_t st) {
    static std::mutex mu;
    static std::set<int> done;
    int dev = 0;
    SPK_CUDA(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> g(mu);
        if (!done.count(dev)) {
            SPK_CUDA(cudaFuncSetAttribute(k_residual_block<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
            done.insert(dev);
        }
    }
    k_residual_block<COLS><<<(A.n + kRows - 1) / kRows, kThreads, smem_of<COLS>(A.rows, A.slots), st>>>(A);
    SPK_CUDA(cudaGetLastError());
    return SPK_OK;
}

}  // namespace

// Whether K columns of a matrix whose columns lie at most ell_reach rows past their tile's first
// row fit (two blocks an SM).
bool residual_fits(const spk_system *s, int K) {
    const int rows = rows_of(s);
    return K >= 2 && K <= 32 && s->ell_reach >= 0 &&
           (K > 16 ? smem_of<32>(rows, s->ell_chunk) : K > 8 ? smem_of<16>(rows, s->ell_chunk) : smem_of<8>(rows, s->ell_chunk)) <=
               112 * 1024;
}

long long residual_device_check() { return first_failed_check(); }

// R = B - A X (residual_fits); norms: 3 per column, zeroed before, or null.
int residual_launch(const spk_system *s, int K, const double *X, long long ldx, const double *B, long long ldb, double *R,
                    long long ldr, unsigned long long *norms, cudaStream_t st) {
    const ResArgs A{s->n, K, rows_of(s), s->ell_chunk, s->ell_ptr.p, s->ell_val.p, s->ell_col.p,
                    s->diag.p, X, ldx, B, ldb, R, ldr, s->uplo == 'L', norms,
                    (long long)s->ell_val.n};
    return K > 16 ? go<32>(A, st) : K > 8 ? go<16>(A, st) : go<8>(A, st);
}

}  // namespace spk
