// The record of a tile of 16 rows (sweep.cu), which the records of many right-hand sides
// (sweep_rhs.cu) are made from, and what both kernels share: the ring of stages and its waits.
#pragma once

#include "spk_internal.cuh"

namespace spk {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr long long kWaitCycles = 1ll << 32;  // ~2 s: bound of a barrier wait

// record: W, 1 / diagonal, then the number of extra slots (low 16 bits) and the rows that have a
// column outside the tile (a bit each above them), the slots' values and offsets, the extra slots'
constexpr int kDiag = 1024;
constexpr int kExtra = kDiag + 128;
constexpr int kHead = kExtra + 16;

// Bytes of S slots per lane: values, and offsets in words (S even; four or two a word).
__host__ __device__ constexpr int slot_bytes(int S, bool wide) { return 256 * S + 128 * (wide ? S / 2 : (S + 3) / 4); }

__device__ __forceinline__ unsigned su32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool try_wait(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __noinline__ bool slow_wait(unsigned bar, unsigned parity) {
    const long long t0 = clock64();
    while (!try_wait(bar, parity))
        if (clock64() - t0 > kWaitCycles) return false;
    return true;
}

struct Ring {  // the stage a warp is at, and the parity of its next completion
    int slot = 0, parity = 0;
    __device__ void next(int ns) {
        if (++slot == ns) {
            slot = 0;
            parity ^= 1;
        }
    }
};

}  // namespace
}  // namespace spk
