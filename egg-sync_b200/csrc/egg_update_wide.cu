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
#include "egg_host_common.h"
#include "egg_kernels.h"
#include "egg_point_walk.cuh"

namespace egg {

namespace {

template <int DM, bool EX, int KB>
__global__ void __launch_bounds__(kWideThreads) k_update_wide(Geom g, Work w, int* __restrict__ counts) {
    update_points_body<DM, EX, KB>(g, w, counts, g.wide_per, blockIdx.x, gridDim.x);
}

// Blocks per SM of the batched kernels: the walk's loads want warps, its arrays
// want registers.  200 instances with 4.9M points of five dimensions: 694 ms
// with the five blocks that 96 registers give, 619 with seven (72 registers, a
// few values spilled), 624 with eight, 716 with ten; 18 with 900,000 of six: 204
// with four, 177 with seven; 16 with 480,000 of eight: 79.4, 76.7 and 78.9 with
// four, five and six; eight with 80,000 of twelve: 25.9 with three, 23.2 with
// five; the others differ by less than the runs.
constexpr int wide_min_blocks(int dm, bool exact) {
    return dm == 5 || dm == 6 ? 7 : dm == 8 ? (exact ? 5 : 7) : dm == 16 ? (exact ? 4 : 5) : 5;
}

// A batch's instances of one d > 8 may differ in their keys' width: a launch
// for each width takes the instances that have it (one kernel for both wants
// 252 registers at d = 16, where each alone wants 168).
template <int DM, bool EX, int KB>
__global__ void __launch_bounds__(kWideThreads, wide_min_blocks(DM, EX)) kb_update_wide(BatchArgs B) {
    batch_for(B, [&](const Geom& g, const Work& w, int bx, int gx) {
        if (DM > 8 && byte_keys(g) != (KB == 8)) return;
        update_points_body<DM, EX, KB>(g, w, nullptr, g.wide_per, bx, gx);
    });
}

}  // namespace

void launch_update_wide(const Exec& ex, int* counts, cudaStream_t st) {
    const size_t table = 16 * (2 * (size_t)ex.table_k() + 1);
    auto smem_of = [&](int lm) { return table + 4 * (size_t)walk_floats(lm) * (kWideThreads / 32); };
    auto one = [&](auto kernel, int lm) {
        const size_t smem = smem_of(lm);
        if (smem > 46 * 1024) EGG_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<shape_blocks(kShapeWide, *ex.g), kWideThreads, smem, st>>>(*ex.g, *ex.w, counts);
    };
    // d <= 4 comes here from single calls only
    if (ex.d <= 4) {
        if (ex.d == 2) one(k_update_wide<2, true, 16>, 2);
        else if (ex.d == 3) one(k_update_wide<3, true, 16>, 3);
        else one(k_update_wide<4, true, 16>, 4);
        return;
    }
    auto go = [&](auto single, auto batch, int lm) {
        if (!ex.batch()) {
            one(single, lm);
            return;
        }
        const size_t smem = smem_of(lm);
        if (smem > 36 * 1024) EGG_CHECK(cudaFuncSetAttribute(batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        batch<<<ex.blocks(kShapeWide, kWideThreads), kWideThreads, smem, st>>>(ex.args(kShapeWide));
    };
    // Every grid of 4 < d <= 16 has keys (16 bits a dimension hold any width), so
    // only more dimensions take the kernel for any d: 64-entry arrays, one load
    // per coordinate, 70 KB of shared memory per block.  Above 256 cells per
    // dimension, that kernel against these: a run of 100k x 5 at eps 0.012 98.1
    // and 29.8 ms, 20k x 8 at 0.02 8.7 and 4.5, 20k x 16 at 0.03 14.3 and 7.0.
    switch (ex.d) {
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
