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
template <int DM, bool EX>
__global__ void __launch_bounds__(kWideThreads) k_update_wide(Geom g, Work w, int* __restrict__ counts, int per) {
    update_points_body<DM, EX>(g, w, counts, per, blockIdx.x, gridDim.x);
}

template <int DM, bool EX>
__global__ void __launch_bounds__(kWideThreads) kb_update_wide(BatchArgs B) {
    batch_for(B, [&](const Geom& g, const Work& w, int bx, int gx) {
        update_points_body<DM, EX>(g, w, nullptr, kWideBatchPer, bx, gx);
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
    // byte keys need d <= 16 and at most 256 cells per dimension; a batch's
    // instances of one d may differ in that, so it takes the keys only where
    // every one has them
    const bool bytes = ex.batch() ? ex.bt->bytes : ex.w->cell_bytes != nullptr;
    if (ex.d == 2) go(k_update_wide<2, true>, kb_update_wide<2, true>, 2);
    else if (ex.d == 3) go(k_update_wide<3, true>, kb_update_wide<3, true>, 3);
    else if (ex.d == 4) go(k_update_wide<4, true>, kb_update_wide<4, true>, 4);
    else if (!bytes) go(k_update_wide<0, false>, kb_update_wide<0, false>, kMaxDims);
    else if (ex.d == 5) go(k_update_wide<5, true>, kb_update_wide<5, true>, 5);
    else if (ex.d == 6) go(k_update_wide<6, true>, kb_update_wide<6, true>, 6);
    else if (ex.d == 8) go(k_update_wide<8, true>, kb_update_wide<8, true>, 8);
    else if (ex.d == 16) go(k_update_wide<16, true>, kb_update_wide<16, true>, 16);
    else if (ex.d < 8) go(k_update_wide<8, false>, kb_update_wide<8, false>, 8);
    else go(k_update_wide<16, false>, kb_update_wide<16, false>, 16);
}

}  // namespace egg
