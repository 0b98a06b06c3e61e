// The reduced system of the partition solve: produceReducedY + __usol2 + updateX
// (src/spike_pstrsv_ops.c:1152-1177, 1247-1262) on the kept reduced rows.
//
// A level is one partition's dependents; its rows read unknowns of later
// partitions only, so the levels run one after another, in descending partition
// order.  Rows whose spike is negligible are not kept: they hold y, the phase-1
// value, and no arithmetic touches them.  All arithmetic is FP64; FP32 work
// columns are rounded once, when an unknown is stored back.
#include <algorithm>
#include <array>
#include <cstdlib>
#include <map>
#include <mutex>

#include "checks.cuh"
#include "reduced.cuh"

namespace spk {

namespace {

inline int blocks_for(long long n, int bs = 256) { return (int)((n + bs - 1) / bs); }

template <typename T>
int upload(DBuf<T> &d, const std::vector<T> &h) {
    SPK_TRY(d.alloc(h.size()));
    if (h.empty()) return SPK_OK;
    if (d.on_stream) SPK_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, d.ord));
    else SPK_CUDA(cudaMemcpy(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice));
    return SPK_OK;
}

// ---- one CTA per system, on the CSR copy --------------------------------------------
//
// Only for systems whose levels span more unknowns than a cluster's shared
// memory holds (below).  FP32 work columns are gathered into the FP64 scratch
// `red` ([K][nred]) and rounded once, on the way back.
template <int K>
constexpr int red_threads() { return K >= 16 ? 512 : 1024; }  // K >= 16: registers for the K sums

struct RedArgs {
    const int *rows, *lvl_off;
    int nlvl;
    const int *mapRedX, *IT, *JT;
    const double *Tv;
    void *xbuf;  // T
    int n;
    double *red;  // FP64 reduced unknowns of FP32 work columns, or null
    int nred;
};

template <int K, typename T>
__global__ void __launch_bounds__(red_threads<K>()) k_reduced_csr(const RedArgs *__restrict__ tab, RedArgs one) {
    const RedArgs A = tab ? tab[blockIdx.x] : one;
    T *xbuf = (T *)A.xbuf;
    double *red = A.red;
    const long long n = A.n, nred = A.nred;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (red) {
        for (long long e = threadIdx.x; e < K * nred; e += blockDim.x)
            red[e] = (double)xbuf[(e / nred) * n + A.mapRedX[e % nred]];
        __syncthreads();
    }
    for (int li = 0; li < A.nlvl; li++) {
        for (int q = A.lvl_off[li] + warp; q < A.lvl_off[li + 1]; q += nwarps) {
            const int kr = A.rows[q];
            double sum[K];
#pragma unroll
            for (int k = 0; k < K; k++) sum[k] = 0.0;
            for (int j = A.IT[kr] + lane; j < A.IT[kr + 1]; j += 32) {
                const long long c = red ? A.JT[j] : A.mapRedX[A.JT[j]];
#pragma unroll
                for (int k = 0; k < K; k++)
                    sum[k] = fma(A.Tv[j], red ? red[k * nred + c] : (double)xbuf[k * n + c], sum[k]);
            }
#pragma unroll
            for (int k = 0; k < K; k++) {
#pragma unroll
                for (int o = 16; o; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
            }
            if (lane == 0) {
                const long long r = A.mapRedX[kr];
#pragma unroll
                for (int k = 0; k < K; k++) {
                    if (red) red[k * nred + kr] -= sum[k];
                    else xbuf[k * n + r] = (T)((double)xbuf[k * n + r] - sum[k]);
                }
            }
        }
        __syncthreads();
    }
    if (red)
        for (long long e = threadIdx.x; e < K * nred; e += blockDim.x)
            xbuf[(e / nred) * n + A.mapRedX[e % nred]] = (T)red[e];
}

// ---- a cluster of CTAs per system and column block ----------------------------------
//
// The levels are a serial chain, so what bounds the solve is the latency of a
// level: one CTA alone took 5 to 20 us a level, most of it waiting for
// coefficients that a single SM cannot pull in faster.  Here a cluster of C CTAs
// takes each level.  A warp computes one or two rows as dot products against a
// ring of unknowns that every CTA keeps whole in its own shared memory, then
// stores the new unknowns into all C rings (distributed shared memory) and into the
// work vector; one hardware cluster barrier ends the level.  Whatever no unknown
// enters is loaded across the barrier before: the next level's row headers and
// first coefficients, the U rows of the unknowns that enter the ring with the
// level after it.
//
// Coefficients are dense ([row][column] over the level's column range) when that
// at most doubles the nonzeros of the kept rows: no column indices, and with four or more columns a
// warp takes two rows, which halves the shared-memory reads of the unknowns (the
// bound at eight columns).  A row whose sum is not finite is summed once more over its nonzeros,
// so that an unknown reaches the rows that read it and no others.  Otherwise they stay in CSR order.
//
// Measured (one right-hand side, this kernel alone against one CTA on the CSR
// copy; the look at every row's sum has since added 1 to 2 %): banded rows, 524,288 rows in 128 partitions, 126 levels of 61 rows: 690 ->
// 218 us (1.7 us a level: the barrier's release waits 0.4 us for the remote stores, the rest
// is one row's dependent steps; loading all of it two levels ahead changed nothing);
// band of 200, 100,003 rows in 48 partitions, 46 levels of 176 rows: 958 -> 90 us (170 with
// 8 warps a CTA, where some take two rows); a 32^3 IC(0)-like factor in 8 partitions (CSR,
// levels of 1,024 rows): 925 -> 105 us (183).  32 systems of 1,024 to 131,072 rows, 364
// columns: 20.3 -> 1.24 ms over the launches.
template <int K>
__host__ __device__ constexpr int ring_stride() { return K <= 2 ? K : K + 2; }  // doubles per unknown: 16-byte reads, no bank conflicts
constexpr int kRingWarps = 8;  // per CTA; 16 with one or two columns and more rows a level than 16 CTAs have warps
constexpr size_t kRingBytes = 208 * 1024;

struct RedLevel {  // rows rr[q0, q0 + nr); columns [c0, c0 + w); unknowns [f0, f1) enter with it; dense block at D + d
    int q0, nr, c0, w, f0, f1;
    long long d;
};

struct RingArgs {
    const RedLevel *lv;
    int nlvl;
    const int4 *rr;      // kept rows: reduced unknown, U row, first and last + 1 CSR entry
    const int *mapRedX;  // U row of a reduced unknown
    const double *D;     // dense blocks, or the CSR values
    const int *JT;       // CSR columns
    void *xbuf;          // T, U order, leading dimension n
    int n, nred, mask;   // mask: ring slots - 1
    int nkept;           // kept rows, coefficients, CSR entries (bounds of the checked build)
    long long nd, nnz;
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void dsmem_store(unsigned local, unsigned cta, double v) {
    unsigned remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(cta));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
}

template <int K, typename T, bool CSR, int TH>
__global__ void __launch_bounds__(TH, TH == 256 ? 2 : 1) k_reduced_ring(const RingArgs *__restrict__ tab, RingArgs one) {
    constexpr int KS = ring_stride<K>(), RB = !CSR && K >= 4 ? 2 : 1;
    constexpr int LK = K == 8 ? 3 : (K == 4 ? 2 : (K == 2 ? 1 : 0));
    constexpr int PF = RB == 2 ? 4 : 8;                  // columns / 32 whose coefficients are loaded ahead
    constexpr int FU = K >= 4 ? 1 : (K == 2 ? 2 : 4);    // entering unknowns a thread holds
    extern __shared__ __align__(16) double ring[];
    const unsigned C = cluster_size(), rank = cluster_rank();
    const RingArgs A = tab ? tab[blockIdx.x / C] : one;
    const int tid = threadIdx.x, lane = tid & 31;
    const int gw = ((int)rank * (TH / 32) + (tid >> 5)) * RB, nw = (int)C * (TH / 32) * RB;
    T *xb = (T *)A.xbuf + (long long)blockIdx.y * K * A.n;
    auto fill = [&](int lo, int hi) {
        for (int id = lo + tid; id < hi; id += TH) {
            const T *x = xb + CK(A.mapRedX[CK(id, A.nred, 100)], A.n, 101);
#pragma unroll
            for (int k = 0; k < K; k++) ring[(id & A.mask) * KS + k] = (double)x[(long long)k * A.n];
        }
    };
    auto level = [&](int li) { return A.lv[min(li, A.nlvl - 1)]; };
    // what the first rows of level M need, and the U rows of the unknowns entering with level E
    int4 rr[RB];
    double pf[RB][PF];
    int pc[CSR ? PF : 1], fid[FU];
    auto ahead = [&](const RedLevel &M, const RedLevel &E) {
#pragma unroll
        for (int b = 0; b < RB; b++) {
            const int q = min(gw + b, M.nr - 1);
            rr[b] = A.rr[CK(M.q0 + q, A.nkept, 102)];
            if constexpr (!CSR) {
#pragma unroll
                for (int u = 0; u < PF; u++)
                    pf[b][u] = lane + 32 * u < M.w ? A.D[CK(M.d + (long long)q * M.w + lane + 32 * u, A.nd, 103)] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < FU; u++) {
            const int id = E.f0 + tid + TH * u;
            fid[u] = id < E.f1 ? (int)CK(A.mapRedX[CK(id, A.nred, 104)], A.n, 105) : -1;
        }
        if constexpr (CSR) {
#pragma unroll
            for (int u = 0; u < PF; u++) {
                const int j = rr[0].z + lane + 32 * u;
                pf[0][u] = j < rr[0].w ? A.D[CK(j, A.nd, 106)] : 0.0;
                pc[u] = j < rr[0].w ? A.JT[CK(j, A.nnz, 107)] : 0;
            }
        }
    };
    RedLevel L = level(0), N = level(1), NN = level(2);
    fill(L.f0, min(A.nred, L.f0 + A.mask + 1));
    ahead(L, N);
    cluster_arrive();  // every CTA of the cluster has started and filled its ring
    cluster_wait();
    for (int li = 0; li < A.nlvl; li++) {
        const bool more = li + 1 < A.nlvl;
        double fv[FU][K];  // the unknowns that enter with the next level
#pragma unroll
        for (int u = 0; u < FU; u++)
#pragma unroll
            for (int k = 0; k < K; k++) fv[u][k] = more && fid[u] >= 0 ? (double)xb[(long long)k * A.n + fid[u]] : 0.0;
        for (int q = gw; q < L.nr; q += nw) {
            double acc[RB][K];
#pragma unroll
            for (int b = 0; b < RB; b++) {
#pragma unroll
                for (int k = 0; k < K; k++) acc[b][k] = 0.0;
            }
            auto step = [&](int c, const double (&v)[RB]) {
                const double *x = ring + (c & A.mask) * KS;
                if constexpr (K == 1) {
#pragma unroll
                    for (int b = 0; b < RB; b++) acc[b][0] = fma(v[b], x[0], acc[b][0]);
                } else {
#pragma unroll
                    for (int k = 0; k < K; k += 2) {
                        const double2 xv = *reinterpret_cast<const double2 *>(x + k);
#pragma unroll
                        for (int b = 0; b < RB; b++) {
                            acc[b][k] = fma(v[b], xv.x, acc[b][k]);
                            acc[b][k + 1] = fma(v[b], xv.y, acc[b][k + 1]);
                        }
                    }
                }
            };
            const bool first = q == gw;
            if (!first) {
#pragma unroll
                for (int b = 0; b < RB; b++) rr[b] = A.rr[CK(L.q0 + min(q + b, L.nr - 1), A.nkept, 108)];
            }
            if constexpr (CSR) {
                int j = rr[0].z + lane;
                const int je = rr[0].w;
                if (first) {
#pragma unroll
                    for (int u = 0; u < PF; u++, j += 32) {
                        const double v[RB] = {pf[0][u]};
                        if (j < je) step(pc[u], v);
                    }
                }
                for (; j + 96 < je; j += 128) {  // four entries a lane in flight
                    double v[4];
                    int c[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) v[u] = A.D[CK(j + 32 * u, A.nd, 109)], c[u] = A.JT[CK(j + 32 * u, A.nnz, 110)];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const double w[RB] = {v[u]};
                        step(c[u], w);
                    }
                }
                for (; j < je; j += 32) {
                    const double v[RB] = {A.D[CK(j, A.nd, 111)]};
                    step(A.JT[CK(j, A.nnz, 112)], v);
                }
            } else {
                const double *d[RB];
#pragma unroll
                for (int b = 0; b < RB; b++) d[b] = A.D + CK(L.d + (long long)min(q + b, L.nr - 1) * L.w, A.nd - L.w + 1, 113);
                int c = lane;
                if (first) {
#pragma unroll
                    for (int u = 0; u < PF; u++, c += 32) {
                        double v[RB];
#pragma unroll
                        for (int b = 0; b < RB; b++) v[b] = pf[b][u];
                        if (c < L.w) step(L.c0 + c, v);
                    }
                }
                for (; c + 96 < L.w; c += 128) {
                    double v[4][RB];
#pragma unroll
                    for (int u = 0; u < 4; u++)
#pragma unroll
                        for (int b = 0; b < RB; b++) v[u][b] = d[b][c + 32 * u];
#pragma unroll
                    for (int u = 0; u < 4; u++) step(L.c0 + c + 32 * u, v[u]);
                }
                for (; c < L.w; c += 32) {
                    double v[RB];
#pragma unroll
                    for (int b = 0; b < RB; b++) v[b] = d[b][c];
                    step(L.c0 + c, v);
                }
            }
            // sums over the lanes: halves of the columns are exchanged while there are
            // several, so lane l ends with column l >> (5 - LK)
            auto lane_sums = [&]() {
#pragma unroll
                for (int b = 0; b < RB; b++) {
#pragma unroll
                    for (int s = 0; s < LK; s++) {
                        const int h = K >> (s + 1), o = 16 >> s;
#pragma unroll
                        for (int i = 0; i < h; i++) {
                            const bool up = lane & o;
                            const double give = up ? acc[b][i] : acc[b][i + h], keep = up ? acc[b][i + h] : acc[b][i];
                            acc[b][i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                        }
                    }
#pragma unroll
                    for (int o = 16 >> LK; o; o >>= 1) acc[b][0] += __shfl_xor_sync(0xffffffffu, acc[b][0], o);
                }
            };
            lane_sums();
            if constexpr (!CSR) {
                bool odd = false;  // an infinity or a NaN, which a coefficient 0 may have let in: once more without those
#pragma unroll
                for (int b = 0; b < RB; b++) odd |= !(fabs(acc[b][0]) <= 1.7976931348623157e308);
                if (__any_sync(0xffffffffu, odd)) {
#pragma unroll
                    for (int b = 0; b < RB; b++) {
#pragma unroll
                        for (int k = 0; k < K; k++) acc[b][k] = 0.0;
                        const double *d = A.D + L.d + (long long)min(q + b, L.nr - 1) * L.w;
#pragma unroll 1
                        for (int c = lane; c < L.w; c += 32) {
                            const double v = d[c], *x = ring + ((L.c0 + c) & A.mask) * KS;
                            if (v != 0.0)
#pragma unroll
                                for (int k = 0; k < K; k++) acc[b][k] = fma(v, x[k], acc[b][k]);
                        }
                        __syncwarp();
                    }
                    lane_sums();
                }
            }
            const int k = lane >> (5 - LK), sub = lane & ((32 >> LK) - 1);
#pragma unroll
            for (int b = 0; b < RB; b++) {
                if (q + b < L.nr) {
                    double *slot = ring + (rr[b].x & A.mask) * KS + k;
                    const double x = *slot - acc[b][0];
                    if (sub == 0) xb[(long long)k * A.n + CK(rr[b].y, A.n, 114)] = (T)x;
                    __syncwarp();  // every lane has read the old value
                    for (unsigned j = sub; j < C; j += 32 >> LK)
                        dsmem_store((unsigned)__cvta_generic_to_shared(slot), j, x);
                }
            }
        }
        if (more) {
#pragma unroll
            for (int u = 0; u < FU; u++) {
                if (fid[u] >= 0) {
                    const int id = N.f0 + tid + TH * u;
#pragma unroll
                    for (int k = 0; k < K; k++) ring[(id & A.mask) * KS + k] = fv[u][k];
                }
            }
            fill(N.f0 + TH * FU, N.f1);
        }
        cluster_arrive();
        L = N;
        N = NN;
        NN = level(li + 3);
        if (more) ahead(L, N);
        cluster_wait();
    }
}

// First and last column of each level (columns are sorted in a row), and the nonzeros of all.
__global__ void k_red_span(int nkept, const int4 *__restrict__ rr, const int *__restrict__ level,
                           const int *__restrict__ JT, int *__restrict__ cmin, int *__restrict__ cmax, int *__restrict__ nnz) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nkept) return;
    atomicAdd(nnz, rr[q].w - rr[q].z);
    atomicMin(&cmin[level[q]], JT[rr[q].z]);
    atomicMax(&cmax[level[q]], JT[rr[q].w - 1]);
}

__global__ void k_red_rows(int nkept, const int *__restrict__ rows, const int *__restrict__ mapRedX,
                           const int *__restrict__ IT, int4 *__restrict__ rr) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nkept) return;
    const int k = rows[q];
    rr[q] = make_int4(k, mapRedX[k], IT[k], IT[k + 1]);
}

// The dense blocks from the CSR rows (one warp per kept row, blocks zeroed before).
__global__ void k_red_dense(int nkept, const int4 *__restrict__ rr, const int *__restrict__ level,
                            const int *__restrict__ JT, const double *__restrict__ Tv,
                            const RedLevel *__restrict__ lv, double *__restrict__ D) {
    const int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= nkept) return;
    const RedLevel L = lv[level[q]];
    double *d = D + L.d + (long long)(q - L.q0) * L.w - L.c0;
    for (int j = rr[q].z + (threadIdx.x & 31); j < rr[q].w; j += 32) d[JT[j]] = Tv[j];
}

// ---- host ---------------------------------------------------------------------------

// Ring slots (a power of two) for column blocks of K, or 0 when they do not fit
// shared memory.
template <int K>
int ring_slots(int need) {
    int r = 64;
    while (r < need) r <<= 1;
    return (size_t)r * ring_stride<K>() * sizeof(double) <= kRingBytes ? r : 0;
}

int ring_slots(int K, int need) {
    return K == 8 ? ring_slots<8>(need) : K == 4 ? ring_slots<4>(need) : K == 2 ? ring_slots<2>(need) : ring_slots<1>(need);
}

// The widest column block (8, 4, 2, 1) that ncols fill and shared memory holds.
int ring_cols(int need, int ncols) {
    for (int k = 8; k > 1; k >>= 1)
        if (ncols >= k && ring_slots(k, need)) return k;
    return 1;
}

RingArgs ring_args(const spk_system *s, void *work, int slots) {
    const bool dense = s->red_full;
    return RingArgs{(const RedLevel *)s->d_red_lv.p, s->nlvl, s->d_red_rr.p, s->mapRedX.p,
                    dense ? s->red_dense.p : s->T.p, s->JT.p, work, s->n, s->nRed, slots - 1, s->nkept,
                    (long long)(dense ? s->red_dense.n : s->T.n), (long long)s->JT.n};
}

struct RingLaunch {
    const RingArgs *tab;
    RingArgs one;
    int nsys, nblk, slots, ctas, warps;
    cudaStream_t st;
    int *max_clusters;  // not null: query the clusters the device holds instead of launching
};

template <int K, typename T, bool CSR, int TH>
int ring_go_t(const RingLaunch &R) {
    auto kern = k_reduced_ring<K, T, CSR, TH>;
    SPK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRingBytes));
    SPK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(R.nsys * R.ctas), (unsigned)R.nblk);
    cfg.blockDim = dim3(TH);
    cfg.dynamicSmemBytes = (size_t)R.slots * ring_stride<K>() * sizeof(double);
    cfg.stream = R.st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)R.ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (R.max_clusters) {
        SPK_CUDA(cudaOccupancyMaxActiveClusters(R.max_clusters, kern, &cfg));
        return SPK_OK;
    }
    SPK_CUDA(cudaLaunchKernelEx(&cfg, kern, R.tab, R.one));
    return SPK_OK;
}

template <int K, typename T, bool CSR>
int ring_go(const RingLaunch &R) {
    if constexpr (K <= 2)
        if (R.warps == 16) return ring_go_t<K, T, CSR, 512>(R);
    return ring_go_t<K, T, CSR, 256>(R);
}

int ring_launch(int K, int fp32, bool csr, const RingLaunch &R) {
    auto pick = [&](auto k) -> int {
        constexpr int kk = decltype(k)::value;
        if (fp32) return csr ? ring_go<kk, float, true>(R) : ring_go<kk, float, false>(R);
        return csr ? ring_go<kk, double, true>(R) : ring_go<kk, double, false>(R);
    };
    switch (K) {
        case 8: return pick(std::integral_constant<int, 8>{});
        case 4: return pick(std::integral_constant<int, 4>{});
        case 2: return pick(std::integral_constant<int, 2>{});
        default: return pick(std::integral_constant<int, 1>{});
    }
}

// The CTAs a cluster of this very launch may have: `want`, halved until the device can place one
// such cluster.  Up to 8 CTAs are portable; 16 need a partition of the chip with room for as
// many of the kernel's CTAs at this size (asked once per device and configuration).
int ring_ctas(int K, int fp32, bool csr, int want, int warps, int slots, int *ctas) {
    *ctas = want;
    if (want <= 8) return SPK_OK;
    static std::mutex mu;
    static std::map<std::array<int, 7>, int> known;
    int dev = 0;
    SPK_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> g(mu);
    const std::array<int, 7> key{dev, K, fp32, csr, want, K <= 2 ? warps : kRingWarps, slots};
    const auto at = known.find(key);
    if (at != known.end()) {
        *ctas = at->second;
        return SPK_OK;
    }
    for (; *ctas > 8; *ctas >>= 1) {
        int fits = 0;
        const RingLaunch R{nullptr, RingArgs{}, 1, 1, slots, *ctas, warps, nullptr, &fits};
        SPK_TRY(ring_launch(K, fp32, csr, R));
        if (fits > 0) break;
    }
    known[key] = *ctas;
    return SPK_OK;
}

template <typename T>
int csr_go(int K, const RedArgs *tab, const RedArgs &one, int nsys, cudaStream_t st) {
    switch (K) {
        case 1: k_reduced_csr<1, T><<<nsys, red_threads<1>(), 0, st>>>(tab, one); break;
        case 2: k_reduced_csr<2, T><<<nsys, red_threads<2>(), 0, st>>>(tab, one); break;
        case 4: k_reduced_csr<4, T><<<nsys, red_threads<4>(), 0, st>>>(tab, one); break;
        case 8: k_reduced_csr<8, T><<<nsys, red_threads<8>(), 0, st>>>(tab, one); break;
        case 16: k_reduced_csr<16, T><<<nsys, red_threads<16>(), 0, st>>>(tab, one); break;
        default: k_reduced_csr<32, T><<<nsys, red_threads<32>(), 0, st>>>(tab, one); break;
    }
    SPK_CUDA(cudaGetLastError());
    return SPK_OK;
}

RedArgs csr_args(const spk_system *s, void *work, double *red) {
    return RedArgs{s->d_red_rows.p, s->d_red_off.p, s->nlvl, s->mapRedX.p, s->IT.p, s->JT.p, s->T.p, work,
                   s->n, red, s->nRed};
}

}  // namespace

long long reduced_device_check() { return first_failed_check(); }

// Levels and row headers of the cluster solve from the kept rows (level by level,
// rows/off) and each level's first reduced unknown; left unbuilt when a level
// spans more unknowns than shared memory holds for one column.
int reduced_prepare(spk_system *s, const std::vector<int> &rows, const std::vector<int> &off,
                    const std::vector<int> &lvl_first) {
    // the tables of a system preprocessed again take the last ones' memory, as its records do
    s->red_ring = 0;
    s->red_full = 0;
    struct Unused {
        spk_system *s;
        ~Unused() {
            if (!s->red_full) s->red_dense.release();
            if (s->red_ring) return;
            s->d_red_lv.release();
            s->d_red_rr.release();
        }
    } unused{s};
    const int nl = s->nlvl, nk = s->nkept;
    const char *no = getenv("SPK_DISABLE_RING");  // test hook: the one-CTA solve
    if (!nk || (no && no[0] == '1')) return SPK_OK;
    cudaStream_t st = s->stream;
    std::vector<int> level(nk), span(2 * nl + 1, -1);  // first and last columns, nonzeros of the kept rows
    span[2 * nl] = 0;
    for (int li = 0; li < nl; li++) {
        span[li] = 2147483647;
        for (int q = off[li]; q < off[li + 1]; q++) level[q] = li;
    }
    DBuf<int> d_level(st), d_span(st);
    SPK_TRY(upload(d_level, level));
    SPK_TRY(upload(d_span, span));
    SPK_TRY(s->d_red_rr.reserve(nk));
    k_red_rows<<<blocks_for(nk), 256, 0, st>>>(nk, s->d_red_rows.p, s->mapRedX.p, s->IT.p, s->d_red_rr.p);
    k_red_span<<<blocks_for(nk), 256, 0, st>>>(nk, s->d_red_rr.p, d_level.p, s->JT.p, d_span.p, d_span.p + nl,
                                                  d_span.p + 2 * nl);
    SPK_CUDA(cudaGetLastError());
    SPK_CUDA(cudaMemcpyAsync(span.data(), d_span.p, sizeof(int) * (2 * nl + 1), cudaMemcpyDeviceToHost, st));
    SPK_CUDA(cudaStreamSynchronize(st));
    std::vector<RedLevel> lv(nl);
    long long tot = 0;
    int need = 1;
    for (int li = 0; li < nl; li++) {
        RedLevel &L = lv[li];
        L = RedLevel{off[li], off[li + 1] - off[li], span[li], span[nl + li] + 1 - span[li], lvl_first[li],
                     li ? lvl_first[li - 1] : s->nRed, tot};
        tot += (long long)L.nr * L.w;
        // live while the level runs: its unknowns up to its last column, and those
        // that enter with the next level
        need = std::max(need, L.c0 + L.w - (li + 1 < nl ? lvl_first[li + 1] : L.f0));
    }
    if (!ring_slots<1>(need)) return SPK_OK;
    static_assert(sizeof(RedLevel) == 8 * sizeof(int), "levels are stored as eight ints");
    SPK_TRY(s->d_red_lv.reserve(8 * (size_t)nl));
    SPK_CUDA(cudaMemcpyAsync(s->d_red_lv.p, lv.data(), sizeof(RedLevel) * nl, cudaMemcpyHostToDevice, st));
    if (tot <= 2ll * span[2 * nl]) {
        SPK_TRY(s->red_dense.reserve(tot));
        s->red_full = 1;
        SPK_CUDA(cudaMemsetAsync(s->red_dense.p, 0, sizeof(double) * tot, st));
        k_red_dense<<<(nk + 7) / 8, 256, 0, st>>>(nk, s->d_red_rr.p, d_level.p, s->JT.p, s->T.p,
                                                  (const RedLevel *)s->d_red_lv.p, s->red_dense.p);
        SPK_CUDA(cudaGetLastError());
    }
    SPK_CUDA(cudaStreamSynchronize(st));
    // a warp per row of an average level, at most 16 CTAs (fewer where a launch cannot place them: ring_ctas)
    const int avg = (nk + nl - 1) / nl;
    int c = 1;
    while (c < 16 && c * kRingWarps < avg) c <<= 1;
    s->red_ctas = c;
    s->red_warps = avg > 16 * kRingWarps ? 16 : kRingWarps;
    s->red_ring = need;
    return SPK_OK;
}

// The reduced solve of ncols columns of work (FP64, or FP32; U order, leading
// dimension n; whole blocks of up to 8 columns are allocated).
int reduced_solve(spk_system *s, int fp32, int ncols, void *work, cudaStream_t st) {
    if (s->red_ring) {
        const int k = ring_cols(s->red_ring, ncols), slots = ring_slots(k, s->red_ring);
        int ctas = 0;
        SPK_TRY(ring_ctas(k, fp32, !s->red_full, s->red_ctas, s->red_warps, slots, &ctas));
        const RingLaunch R{nullptr, ring_args(s, work, slots), 1, (ncols + k - 1) / k, slots, ctas, s->red_warps, st, nullptr};
        SPK_TRY(ring_launch(k, fp32, !s->red_full, R));
    } else {
        int K = 1;
        while (K < ncols) K <<= 1;
        const RedArgs a = csr_args(s, work, fp32 ? s->red_scratch : nullptr);
        SPK_TRY(fp32 ? csr_go<float>(K, nullptr, a, 1, st) : csr_go<double>(K, nullptr, a, 1, st));
    }
    s->launches++;
    return SPK_OK;
}

int red_plan_build(RedPlan &p, const std::vector<RedMember> &members, int K, int fp32) {
    p.K = K;
    p.fp32 = fp32;
    std::vector<RedArgs> csr;
    std::vector<RingArgs> ring[8];
    for (const RedMember &m : members) {
        if (!m.s->red_ring) {
            csr.push_back(csr_args(m.s, m.work, fp32 ? m.red : nullptr));
            continue;
        }
        const int k = ring_cols(m.s->red_ring, K), slots = ring_slots(k, m.s->red_ring);
        const int w = (k == 8 ? 0 : k == 4 ? 1 : k == 2 ? 2 : 3) + (m.s->red_full ? 0 : 4);
        ring[w].push_back(ring_args(m.s, m.work, slots));
        p.slots[w] = std::max(p.slots[w], slots);
        p.ctas[w] = std::max(p.ctas[w], m.s->red_ctas);
        p.warps[w] = std::max(p.warps[w], m.s->red_warps);
    }
    auto put = [](DBuf<char> &d, const void *src, size_t bytes) -> int {
        if (!bytes) return SPK_OK;
        SPK_TRY(d.alloc(bytes));
        SPK_CUDA(cudaMemcpy(d.p, src, bytes, cudaMemcpyHostToDevice));
        return SPK_OK;
    };
    int dev = 0, sms = 148;
    SPK_CUDA(cudaGetDevice(&dev));
    SPK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SPK_TRY(put(p.csr, csr.data(), sizeof(RedArgs) * csr.size()));
    p.ncsr = (int)csr.size();
    for (int w = 0; w < 8; w++) {
        SPK_TRY(put(p.ring[w], ring[w].data(), sizeof(RingArgs) * ring[w].size()));
        p.nring[w] = (int)ring[w].size();
        // smaller clusters rather than a second wave (two CTAs per SM)
        const int nb = K / (8 >> (w & 3));
        while (p.ctas[w] > 4 && (long long)p.ctas[w] * p.nring[w] * nb > 2ll * sms) p.ctas[w] >>= 1;
        if (p.nring[w]) SPK_TRY(ring_ctas(8 >> (w & 3), fp32, w >= 4, p.ctas[w], p.warps[w], p.slots[w], &p.ctas[w]));
    }
    return SPK_OK;
}

int red_plan_launch(const RedPlan &p, cudaStream_t st, long long *kernels) {
    if (p.ncsr) {
        const RedArgs none{};
        SPK_TRY(p.fp32 ? csr_go<float>(p.K, (const RedArgs *)p.csr.p, none, p.ncsr, st)
                       : csr_go<double>(p.K, (const RedArgs *)p.csr.p, none, p.ncsr, st));
        ++*kernels;
    }
    for (int w = 0; w < 8; w++) {
        if (!p.nring[w]) continue;
        const int k = 8 >> (w & 3);
        const RingLaunch R{(const RingArgs *)p.ring[w].p, RingArgs{}, p.nring[w], p.K / k, p.slots[w], p.ctas[w], p.warps[w], st,
                           nullptr};
        SPK_TRY(ring_launch(k, p.fp32, w >= 4, R));
        ++*kernels;
    }
    return SPK_OK;
}

}  // namespace spk
