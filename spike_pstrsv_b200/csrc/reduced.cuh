// Reduced solves of many systems in one launch sequence (reduced.cu), for the
// many-system groups.
#pragma once

#include "spk_internal.cuh"

namespace spk {

// Column blocks of one system: its work columns (FP64 or FP32, U order, leading
// dimension n) and, for FP32, an FP64 scratch of K x nRed.
struct RedMember {
    spk_system *s;
    void *work;
    double *red;
};

struct RedPlan {
    DBuf<char> csr, ring[8];  // argument tables: the one-CTA solve; clusters, by column block and layout
    int ncsr = 0, nring[8] = {}, slots[8] = {}, ctas[8] = {}, warps[8] = {};
    int K = 0, fp32 = 0;
};

int red_plan_build(RedPlan &p, const std::vector<RedMember> &members, int K, int fp32);
int red_plan_launch(const RedPlan &p, cudaStream_t st, long long *kernels);

}  // namespace spk
