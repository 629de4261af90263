// Fold of a row's partials inside a thread-block cluster.
//
// The CTAs that share an output row (the pieces of a unit's history and its ring part)
// form one cluster; each leaves its partial (unnormalised outputs, maximum, sum) in its
// own shared memory, and after a cluster barrier every CTA reads all partials of its
// share of the rows through distributed shared memory and writes finished outputs.  No
// partial goes to global memory and no second kernel is launched.
//
// The additions are those of merge_row (attn_fp32.cu) in the same order, so that both
// give the same bits: even and odd pieces in two chains, the denominator as the tree a
// warp reduction of eight lanes makes.
#pragma once

#include <cooperative_groups.h>

#include "kivi_common.cuh"

namespace kivi {

constexpr int kClusterFoldMax = 8;               // pieces of a row; a portable cluster has eight CTAs at most

struct ClusterOut {                              // where the outputs go; out == nullptr: partials to the workspace instead
    void* out;
    int out_dtype;
    float* lse;
};

// part_s [n_heads][D], ml_s [n_heads][2] in this CTA's shared memory (same place in every
// CTA of the cluster); row0: first output row of the cluster.  Every thread of every CTA
// of the cluster calls it.
__device__ __forceinline__ void cluster_fold(float* part_s, float* ml_s, int n_heads, int D, int64_t row0, const ClusterOut& to) {
    namespace cg = cooperative_groups;
    // What follows in the stream may become resident while the clusters fold: that hides
    // its launch, and by now few SMs are left to be unevenly taken.  32 units x 2k tokens,
    // attention calls back to back 9.6 us (let in at the kernel's start 12.2, at its end
    // 9.4), append and attention in turn 10.1 (10.1, 10.4); 64 x 512 8.2 (10.1, 8.7).
    cudaTriggerProgrammaticLaunchCompletion();
    cg::cluster_group cluster = cg::this_cluster();
    const int n = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    cluster.sync();
    const int quads = D / 4;
    for (int i = rank * blockDim.x + threadIdx.x; i < n_heads * quads; i += n * blockDim.x) {
        const int h = i / quads, d = 4 * (i - h * quads);
        float mv[kClusterFoldMax], den[kClusterFoldMax], w[kClusterFoldMax];
        float4 v[kClusterFoldMax];
        float M = -INFINITY;
#pragma unroll
        for (int s = 0; s < kClusterFoldMax; ++s) {
            mv[s] = -INFINITY; den[s] = 0.0f; v[s] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s < n) {
                const float2 ml = *reinterpret_cast<const float2*>(cluster.map_shared_rank(ml_s, s) + 2 * h);
                mv[s] = ml.x; den[s] = ml.y;
                v[s] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(part_s, s) + h * D + d);
                M = fmaxf(M, ml.x);
            }
        }
        float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
#pragma unroll
        for (int s = 0; s < kClusterFoldMax; ++s) {
            w[s] = mv[s] == -INFINITY ? 0.0f : exp2f(mv[s] - M);
            den[s] = fmaf(w[s], den[s], 0.0f);
        }
#pragma unroll
        for (int s = 0; s < kClusterFoldMax; s += 2) {
            a0.x = fmaf(v[s].x, w[s], a0.x); a0.y = fmaf(v[s].y, w[s], a0.y);
            a0.z = fmaf(v[s].z, w[s], a0.z); a0.w = fmaf(v[s].w, w[s], a0.w);
            a1.x = fmaf(v[s + 1].x, w[s + 1], a1.x); a1.y = fmaf(v[s + 1].y, w[s + 1], a1.y);
            a1.z = fmaf(v[s + 1].z, w[s + 1], a1.z); a1.w = fmaf(v[s + 1].w, w[s + 1], a1.w);
        }
        const float total = ((den[0] + den[4]) + (den[2] + den[6])) + ((den[1] + den[5]) + (den[3] + den[7]));
        const float inv = 1.0f / total;
        // natural-log sum of exponentials of the scaled scores (M and the sums live in the log2 domain)
        if (to.lse != nullptr && d == 0) to.lse[row0 + h] = (M + log2f(total)) * 0.6931471805599453f;
        store_quad(to.out, to.out_dtype, (row0 + h) * D + d,
                   make_float4((a0.x + a1.x) * inv, (a0.y + a1.y) * inv, (a0.z + a1.z) * inv, (a0.w + a1.w) * inv));
    }
    cluster.sync();                              // the others may still read this CTA's partial
}

}  // namespace kivi
