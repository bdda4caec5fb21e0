// egg_update_wide.cu -- eps-ball update + convergence flag, a warp per point.
//
// The same update as egg_update.cu (the reference's kernel_itr_grid_STAD5_5_1,
// src/algorithms/EGG_SynC.cu:551-763), for d > 4 and for small sets.  With many
// dimensions a cell holds about one point, an update meets thousands of
// candidate cells, few of them pass the box test (92 of 1,645 at 20k x 16D,
// 1,015 of 3,157 at 100k x 5D, first iteration), and 32 consecutive points
// share few of theirs; with few points, 32 to a warp leave the chip idle.  So
// a warp takes one point at a time (egg_point_walk.cuh): 20k x 16D updates
// 19.8 -> 3.3 ms a run, 100k x 5D 25.7 -> 13.6 ms for ten iterations, 10k x 2D
// 0.71 -> 0.24 ms a run (a thread per point before).  25k instructions per
// point at 100k x 5D; what is left is their issue and the chains of loads.
#include "egg_common.cuh"
#include "egg_kernels.h"
#include "egg_point_walk.cuh"

namespace egg {

namespace {

constexpr int kWideThreads = 128;
template <int DM, bool EX, int KB>
__global__ void __launch_bounds__(kWideThreads) k_update_wide(Geom g, Work w, int* __restrict__ counts, int per) {
    update_points_body<DM, EX, KB>(g, w, counts, per, blockIdx.x, gridDim.x);
}

// A batch's instances of one d > 8 may differ in their keys' width: a launch
// for each width takes the instances that have it (one kernel for both wants
// 252 registers at d = 16, where each alone wants 168).
template <int DM, bool EX, int KB>
__global__ void __launch_bounds__(kWideThreads) kb_update_wide(BatchArgs B) {
    batch_for(B, [&](const Geom& g, const Work& w, int bx, int gx) {
        if (DM > 8 && byte_keys(g) != (KB == 8)) return;
        update_points_body<DM, EX, KB>(g, w, nullptr, kWideBatchPer, bx, gx);
    });
}

}  // namespace

// Points per block of one instance.  Where every point is recomputed each
// wants a warp (the heavy ones, those of a dense cluster, sit together: 100k x
// 5D, ten iterations, 15.2 ms with one point per warp against 16.8 with two,
// 18.6 with four); from some 75,000 warps on, blocks that only settle kept
// points would be too many.
int wide_points_per_block(int n) {
    int per = kWideThreads;
    while (per > kWideThreads / 32 && (n + per - 1) / per < 148 * 128) per >>= 1;
    return per;
}

void launch_update_wide(const Exec& ex, int* counts, cudaStream_t st) {
    auto go = [&](auto one, auto batch, int lm) {
        const size_t smem = 16 * (2 * (size_t)ex.table_k() + 1) + 4 * (size_t)walk_floats(lm) * (kWideThreads / 32);
        if (ex.batch()) {
            if (smem > 36 * 1024) cudaFuncSetAttribute(batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            batch<<<ex.blocks(kShapeWide, kWideThreads), kWideThreads, smem, st>>>(ex.args(kShapeWide));
        } else {
            if (smem > 46 * 1024) cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            const int per = wide_points_per_block(ex.g->n);
            const int runs = per < 8 ? per : 8;  // whole runs of eight points
            const int blocks = ((ex.g->n + runs - 1) / runs + per / runs - 1) / (per / runs);
            one<<<blocks, kWideThreads, smem, st>>>(*ex.g, *ex.w, counts, per);
        }
    };
    // Every grid of 4 < d <= 16 has keys (16 bits a dimension hold any width), so
    // only more dimensions take the kernel for any d: 64-entry arrays, one load
    // per coordinate, 70 KB of shared memory per block.  Above 256 cells per
    // dimension, that kernel against these: a run of 100k x 5 at eps 0.012 98.1
    // and 29.8 ms, 20k x 8 at 0.02 8.7 and 4.5, 20k x 16 at 0.03 14.3 and 7.0.
    switch (ex.d) {
        case 2: go(k_update_wide<2, true, 16>, kb_update_wide<2, true, 16>, 2); return;
        case 3: go(k_update_wide<3, true, 16>, kb_update_wide<3, true, 16>, 3); return;
        case 4: go(k_update_wide<4, true, 16>, kb_update_wide<4, true, 16>, 4); return;
        case 5: go(k_update_wide<5, true, 16>, kb_update_wide<5, true, 16>, 5); return;
        case 6: go(k_update_wide<6, true, 16>, kb_update_wide<6, true, 16>, 6); return;
        case 7: go(k_update_wide<8, false, 16>, kb_update_wide<8, false, 16>, 8); return;
        case 8: go(k_update_wide<8, true, 16>, kb_update_wide<8, true, 16>, 8); return;
        default: break;
    }
    if (ex.d > kKeyDims) {
        go(k_update_wide<0, false, 16>, kb_update_wide<0, false, 16>, kMaxDims);
        return;
    }
    const bool k8 = ex.batch() ? ex.bt->key8 : byte_keys(*ex.g), k16 = ex.batch() ? ex.bt->key16 : !k8;
    if (ex.d == 16) {
        if (k8) go(k_update_wide<16, true, 8>, kb_update_wide<16, true, 8>, 16);
        if (k16) go(k_update_wide<16, true, 16>, kb_update_wide<16, true, 16>, 16);
    } else {
        if (k8) go(k_update_wide<16, false, 8>, kb_update_wide<16, false, 8>, 16);
        if (k16) go(k_update_wide<16, false, 16>, kb_update_wide<16, false, 16>, 16);
    }
}

}  // namespace egg
