// Checked builds (-DSPK_DEVICE_CHECKS): indexes of the solve kernels are bounds-checked; a
// failed check records (code, block, index) in the file's g_check (first one kept) and the
// access uses index 0 instead.  Off by default.  Codes: chain.cu 1 to 59, sweep.cu 60 to 79,
// sweep_rhs.cu 80 to 99, reduced.cu 100 to 119, residual.cu 120 to 139.
#pragma once

#include <cuda_runtime.h>

namespace spk {
namespace {

#ifdef SPK_DEVICE_CHECKS
__device__ unsigned long long g_check;
__device__ __noinline__ long long chk_fail(int code, long long i) {
    atomicCAS(&g_check, 0ull,
              ((unsigned long long)code << 48) | ((unsigned long long)(blockIdx.x & 0xffffff) << 24) |
                  (unsigned long long)(i & 0xffffff));
    return 0;
}
#define CK(i, n, code) \
    (((unsigned long long)(long long)(i) < (unsigned long long)(long long)(n)) ? (long long)(i) : chk_fail((code), (long long)(i)))
// a pointer into base[0, n); an unsigned index
#define CKP(p, base, n, code) ((base) + CK((p) - (base), (n), (code)))
#define CKU(i, n, code) ((unsigned)CK((i), (n), (code)))
inline long long first_failed_check() {
    unsigned long long v = 0;
    return cudaMemcpyFromSymbol(&v, g_check, sizeof(v)) == cudaSuccess ? (long long)v : -1;
}
#else
#define CK(i, n, code) (i)
#define CKP(p, base, n, code) (p)
#define CKU(i, n, code) (i)
inline long long first_failed_check() { return 0; }
#endif

}  // namespace
}  // namespace spk
