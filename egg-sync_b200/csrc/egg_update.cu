// egg_update.cu -- eps-ball synchronisation update + convergence flag.
//
// Replaces kernel_itr_grid_STAD5_5_1 of the reference
// (src/algorithms/EGG_SynC.cu:551-763) together with its pre-grid of
// neighbour outer cells (EGG_SynC.cu:368-536), which the dense outer_begin
// array makes unnecessary.
//
// For point p with own-cell corner c (c_l = g_l * side) and phi = x_p - c:
//   sum_{q in N(p)} sin(x_q - x_p) = cos(phi) * S - sin(phi) * (N - Cm)
// with S = sum sin(x_q - c), Cm = sum (1 - cos(x_q - c)), N = |N(p)|.
// A neighbour cell with dim ids g' (k = g' - g) whose points have offsets
// delta_q = x_q - g' * side contributes, through sin/cos tables of k * side,
//   S  += sin(k s) * (m - SM) + cos(k s) * SS
//   Cm += m * (1 - cos(k s)) + cos(k s) * SM + sin(k s) * SS
// where SS = sum sin(delta), SM = sum (1 - cos(delta)) over the counted
// points (the whole cell when it lies inside the eps-ball, the points that
// pass the distance test otherwise).  Every term is a small, well-conditioned
// quantity, so the FP32 result stays within ~1e-7 of the exact FP64 update.
//
// Cell classification, distance tests, the border rule and the flag follow
// the reference exactly (EGG_SynC.cu:583-597, 613-636, 666-681, 706-709).
//
// d <= 4 (more dimensions: egg_update_wide.cu).  Bound by instruction issue
// and by the latency of what is left of it, not by memory (the working set
// stays in L2).  Grouping the update's threads along a space-filling curve
// lets every warp walk in lockstep (before, 60% to 88% of the warps of the
// first iterations had their lanes walk one by one): update kernel over the
// first ten iterations, 1M x 3D 60 -> 40 ms, 250k x 3D 23.0 -> 15.0,
// 45,781 x 3D 9.5 -> 4.7, 100k x 4D 17.9 -> 8.2 ms, all bit-identical.
#include <climits>
#include <type_traits>

#include "egg_common.cuh"
#include "egg_host_common.h"
#include "egg_kernels.h"
#include "egg_point_walk.cuh"
#include "egg_stencil.cuh"

namespace egg {

namespace {

// reference half_count (EGG_SynC.cu:666-681) for a border point whose
// neighbourhood holds other fully covered cells: own cell plus the points
// within eps/2 in the other fully covered cells.
template <int D>
__device__ int half_count(const Geom& g, const Work& w, const float* x, const int* gi, int obase, int own, int own_cnt) {
    constexpr int d = D;
    int half = own_cnt;
    const int nst = w.st_count[0];
    for (int s = 0; s < nst; s++) {
        bool inb = true;
        for (int l = 0; l < g.od; l++) {
            int v = gi[l] + w.st_off[(size_t)s * g.od + l];
            inb = inb && (unsigned)v < (unsigned)g.width;
        }
        if (!inb) continue;
        const int o = obase + w.st_delta[s];
        int cb = w.outer_begin[o], ce = w.outer_begin[o + 1];
        if (cb >= ce) continue;
        if (g.od < d) {
            const int* keys = w.cell_dims + (size_t)g.od * g.ns;
            cb = lower_bound_i(keys, cb, ce, gi[g.od] - g.r - 1);
            ce = lower_bound_i(keys, cb, ce, gi[g.od] + g.r + 2);
        }
        for (int c = cb; c < ce; c++) {
            if (c == own) continue;
            float sm2 = 0.f, lg2 = 0.f;
            for (int l = 0; l < d; l++) box_terms(x[l], __ldg(w.cell_dims + (size_t)l * g.ns + c), g.side, sm2, lg2);
            if (!(lg2 <= g.t_eps)) continue;
            const int qb = __ldg(w.cell_start + c), qe = __ldg(w.cell_start + c + 1);
            float near2, far2;
            tight_box_dist2<D>(x, cell_box<D>(w, c, d), d, near2, far2);
            if (near2 > g.t_half) continue;
            if (far2 <= g.t_half) {
                half += qe - qb;
                continue;
            }
            for (int q = qb; q < qe; q++) {
                float d2 = 0.f;
                for (int l = 0; l < d; l++) d2 = dist_step(__ldg(w.X + (size_t)l * g.ns + q), x[l], d2);
                half += (d2 <= g.t_half);
            }
        }
    }
    return half;
}

}  // namespace

namespace {

#ifdef EGG_UPDATE_STATS
#define EGG_STAT(a, k, v) ((a).st[k] += (v))
#else
#define EGG_STAT(a, k, v) ((void)0)
#endif

// The outer column a walk is in: the box terms and cell offsets of the outer
// dimensions (l < od) are the same for every cell of the column, so they are
// formed once per column and point.  The box sums start with the outer
// dimensions, in the same order, so the totals round alike.
template <int D>
struct Col {
    float sm, lg;
    int kk[D];
};

// Lockstep walks read points from shared memory four at a time:
// with two in flight the loop waits on each load (1M x 3D: 42 -> 47 ms for
// the first ten iterations).  They want registers more than warps: five
// blocks of 128 threads per SM (96 registers) beat four (47 ms), six (80
// registers, 47 ms) and eight (64 registers, 45 ms); d = 4 keeps four blocks
// (100k x 4D: 12.4 ms against 13.5).
constexpr int kWalkUnroll = 4;
constexpr int update_min_blocks(int d, int threads) {
    const int m = (d <= 3 ? 640 : 512) / threads;
    return m > 0 ? m : 1;
}

template <int D>
struct Acc {
    float S[D];
    float Cm[D];
    int N;
    int partial_in;
#ifdef EGG_UPDATE_STATS
    unsigned st[kUStats];
#endif
};

// m counted points of a cell at offsets k (= cell dims - own dims) with
// SS = sum sin(delta), SM = sum (1 - cos(delta)) into the own-cell frame.
// tab[k + K] = sin(k side), cos(k side), 1 - cos(k side): one 16-byte load.
template <int D>
__device__ __forceinline__ void add_counted(Acc<D>& a, const int* kk, float m, const float* SS, const float* SM,
                                            const float4* tab, int K) {
#pragma unroll
    for (int l = 0; l < D; l++) {
        const float4 t = tab[kk[l] + K];
        const float ts = t.x, tc = t.y, tm = t.z;
        a.S[l] += ts * (m - SM[l]) + tc * SS[l];
        a.Cm[l] += m * tm + tc * SM[l] + ts * SS[l];
    }
}

// cell coordinate l from the packed 16-bit key, as a float without the
// integer-to-float unit: the 16 bits are the low mantissa of 2^23 + cd
__device__ __forceinline__ float key_dim_f(unsigned long long key, int l) {
    const unsigned word = (unsigned)(key >> (32 * (l >> 1)));
    const unsigned bits = __byte_perm(word, 0x4b000000u, (l & 1) ? 0x7432 : 0x7410);
    return __uint_as_float(bits) - 8388608.0f;
}
// box_terms with the cell coordinate as a float: the smaller square to sm,
// the larger to lg (equal squares are the same addend either way)
__device__ __forceinline__ void box_terms_f(float x, float cd, float side, float& sm, float& lg) {
    const float left = __fmaf_rn(cd, side, -x);
    const float right = __fmaf_rn(cd + 1.0f, side, -x);
    const float l2 = __fmul_rn(left, left), r2 = __fmul_rn(right, right);
    sm = __fadd_rn(sm, fminf(l2, r2));
    lg = __fadd_rn(lg, fmaxf(l2, r2));
}

// two floats of a register pair, added or subtracted in one instruction
// (each half rounds to nearest as the scalar operation does)
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// squared distance to a packed point, the operations and order of dist_step;
// nx holds -x in pairs
template <int D>
__device__ __forceinline__ float pair_dist2(const ulonglong2* v, const unsigned long long* nx, const float* x) {
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < pack_w(D); j++) {
        float e0, e1, e2 = 0.f, e3 = 0.f;
        unpack2(add2(v[j].x, nx[2 * j]), e0, e1);
        if (4 * j + 3 < D) {
            unpack2(add2(v[j].y, nx[2 * j + 1]), e2, e3);
        } else if (4 * j + 2 < D) {
            unpack2(v[j].y, e2, e3);
            e2 = __fsub_rn(e2, x[4 * j + 2 < D ? 4 * j + 2 : 0]);
        }
        acc = __fmaf_rn(e0, e0, acc);
        if (4 * j + 1 < D) acc = __fmaf_rn(e1, e1, acc);
        if (4 * j + 2 < D) acc = __fmaf_rn(e2, e2, acc);
        if (4 * j + 3 < D) acc = __fmaf_rn(e3, e3, acc);
    }
    return acc;
}

// tight_box_dist2 on a box record (lower, then upper corner) read in whole
// words, the differences of two dimensions at a time: lo - x and hi - x give
// the near gap max(lo - x, x - hi, 0) and the far gap max(|lo - x|, |hi - x|)
template <int D, bool kGlobal>
__device__ __forceinline__ void box_dist2(const unsigned long long* nx, const float* x, const ulonglong2* box,
                                          float& near2, float& far2) {
    float a2 = 0.f, b2 = 0.f;
#pragma unroll
    for (int j = 0; j < pack_w(D); j++) {
        const ulonglong2 L = kGlobal ? __ldg(box + j) : box[j];
        const ulonglong2 H = kGlobal ? __ldg(box + pack_w(D) + j) : box[pack_w(D) + j];
        float dl[4], dh[4];
        unpack2(add2(L.x, nx[2 * j]), dl[0], dl[1]);
        unpack2(add2(H.x, nx[2 * j]), dh[0], dh[1]);
        if (4 * j + 3 < D) {
            unpack2(add2(L.y, nx[2 * j + 1]), dl[2], dl[3]);
            unpack2(add2(H.y, nx[2 * j + 1]), dh[2], dh[3]);
        } else if (4 * j + 2 < D) {
            unpack2(L.y, dl[2], dl[3]);
            unpack2(H.y, dh[2], dh[3]);
            dl[2] = __fsub_rn(dl[2], x[4 * j + 2 < D ? 4 * j + 2 : 0]);
            dh[2] = __fsub_rn(dh[2], x[4 * j + 2 < D ? 4 * j + 2 : 0]);
        }
#pragma unroll
        for (int l = 0; l < 4; l++)
            if (4 * j + l < D) {
                const float near = fmaxf(fmaxf(dl[l], -dh[l]), 0.f), far = fmaxf(fabsf(dl[l]), fabsf(dh[l]));
                a2 = __fmaf_rn(near, near, a2);
                b2 = __fmaf_rn(far, far, b2);
            }
    }
    near2 = a2;
    far2 = b2;
}

// a sum record (a point's, a group's) added to the pairs av
template <int D, bool kGlobal>
__device__ __forceinline__ void add_point(unsigned long long* av, const ulonglong2* rec) {
#pragma unroll
    for (int j = 0; j < pack_s(D); j++) {
        const ulonglong2 t = kGlobal ? __ldg(rec + j) : rec[j];
        av[2 * j] = add2(av[2 * j], t.x);
        if (4 * j + 2 < 2 * D) av[2 * j + 1] = add2(av[2 * j + 1], t.y);
    }
}

// -x in pairs
template <int D>
__device__ __forceinline__ void negate_pairs(const float* x, unsigned long long* nx) {
#pragma unroll
    for (int k = 0; k < 2 * pack_w(D); k++)
        nx[k] = pack2(2 * k < D ? -x[2 * k < D ? 2 * k : 0] : 0.f, 2 * k + 1 < D ? -x[2 * k + 1 < D ? 2 * k + 1 : 0] : 0.f);
}

// ---------------------------------------------------------------------------
// The walk of a whole warp in lockstep (d <= 4).
//
// The warp takes the columns within r of any active lane's cell, each
// restricted in dimension od to the lanes' joint window.  Columns ascend and a
// column's cells ascend, so every lane meets its own candidates in the order
// of its own stencil; cells beyond its stencil it passes over (in the outer
// dimensions by their offset, elsewhere they fail its box test).  The
// candidates come 32 at a time, one per lane: each lane reads its cell's
// record, drops it when no active lane can count any of its points, and
// leaves it in shared memory otherwise.  Then the warp goes through the kept
// cells one by one, reading the records as broadcasts: no visit waits for a
// chain of loads, and the cells that only widen the joint window (40% of
// them) cost a thirty-second of a visit.
//
// With the joint box too wide the walk does not pay and returns false before
// any visit: for more than kUnionCols columns (points of an empty region), in
// tile order for too wide a joint region (kTileRoom), and
// in storage order (tiled false) when the lanes lie in several columns or
// spread over dimension od and more than kSpreadCells cells are around them
// (consecutive points of sparse columns are dozens of cells apart there).
// ---------------------------------------------------------------------------
constexpr int kUnionCols = 1024;
// In tile order a joint region of more than this many times one point's own
// (the curve leaves a cluster, or crosses an empty region) is not walked
// together either: few such warps, but thousands of candidates each held the
// whole launch (1M x 2D, eps 0.002, first update: 5.3 ms, 1.3 with 8 to 512; a
// run of 200k x 4D: 33.9 ms without, 48.3, 41.7, 37.7, 35.9, 34.0 and 34.0 with
// 8, 16, 32, 64, 128 and 512; one of 43,110 x 3D, eps 0.00065: 6.5, 4.6 with
// 128, 4.7 with 512).
constexpr float kTileRoom = 128.f;
// Whole rows of columns instead of columns where they hold at most this many
// cells per column: once the points have gathered, nearly every column of the
// hundreds around a warp is empty, and finding its few cells took 30 chained
// loads (update of 1M x 3D, 1,000 iterations: 103 ms by columns, 101 by rows;
// no difference between 1 and 16 cells per column; before that the window in
// dimension od leaves a column fewer candidates than its row).
constexpr int kRowFill = 4;
// In storage order, lanes in several columns walk together when the rows
// around them hold at most this many cells; else their points are walked one
// by one, 15 us for a warp's 32 (68,535 x 2D, 1,000 iterations: update 26.7 ms
// one by one, 15 together; 250k x 3D and 1M x 3D gain nothing from more
// cells, and with 64 lose 3% and 9%).
constexpr int kSpreadCells = 256;
// Points of a block at most (its list), and the blocks of a launch from which
// on a warp takes several rows in storage order: a full chip of them, five per
// SM.  1M x 3D, 1,000 iterations, update with 2, 4 and 8 rows: 87, 85, 76 ms.
// A batch's blocks go through its points by themselves (one row: 6 x 8 sweep
// 101.0 ms, rows by this rule 102.7).
constexpr int kListMax = 1024;
// Lanes of one place (a column, and near each other in dimension od) that are
// at least this many walk together when the whole warp does not (68,535 x 2D,
// eps 0.01, 417 iterations: update 10.2 ms without groups, 7.7 with groups of
// four and more, 8.2 with any).
constexpr int kGroupMin = 4;
constexpr int kRowBlocks = 148 * 5;
constexpr int kRowsAhead = 4;  // rows whose loads are in flight together

// shared memory of one warp, in 16-byte words: its joint box, 32 cell records (key, first
// point, points | box | sums), then 32 points (coordinates | sums); one dimension: 32 group records
__host__ __device__ constexpr int cell_words(int d) { return 1 + 2 * pack_w(d) + pack_s(d); }
__host__ __device__ constexpr int box_words(int d) { return (4 * (5 * d + 2) + 15) / 16; }
__host__ __device__ constexpr int warp_words(int d) {
    return box_words(d) + 32 * cell_words(d) + 32 * (pack_w(d) + pack_s(d)) + (d == 1 ? 32 * (pack_s(d) + 2 * pack_w(d)) : 0);
}

// float order as unsigned order, and back
__device__ __forceinline__ unsigned order_key(float x) {
    const unsigned u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float order_val(unsigned k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// what the screening of candidates needs of the warp's joint box: the same for
// all lanes, so it waits in shared memory (volatile: read where it is used)
// instead of in every lane's registers
template <int D>
struct WarpBox {
    int lo[D], hi[D], wide[D];
    float xl[D], xh[D];
    float mar, r2;
};

// One kept cell for the 32 lanes; a lane whose column is off (col.sm infinite)
// contributes nothing.  A group of points that some lane has to walk is
// brought into shared memory by the whole warp (one coalesced load per record
// word instead of a dependent load per point), then every walking lane reads
// the points as broadcasts.
template <int D, int OD>
__device__ __forceinline__ void visit_cell_warp(const Geom& g, const Work& w, const ulonglong2* rec, const float* x,
                                                const unsigned long long* nx, const int* gi, const Col<D>& col,
                                                Acc<D>& a, const float4* tab, int K, const volatile WarpBox<D>& B,
                                                ulonglong2* stage, int lane) {
    constexpr int PW = pack_w(D), PS = pack_s(D);
    const int od = OD > 0 ? OD : g.od;
    const ulonglong2 head = rec[0];
    const unsigned long long key = head.x;
    float sm2 = col.sm, lg2 = col.lg;
#pragma unroll
    for (int l = 0; l < D; l++)
        if (l >= od) box_terms_f(x[l], key_dim_f(key, l), g.side, sm2, lg2);
    const bool pass = sm2 <= g.t_eps;
    EGG_STAT(a, kUsCells, 1);
    if (!__any_sync(0xffffffffu, pass)) return;
    const int qb = (int)(unsigned)head.y, m_all = (int)(unsigned)(head.y >> 32);
    float near2, far2;
    box_dist2<D, false>(nx, x, rec + 1, near2, far2);
    const bool full = lg2 <= g.t_eps;
    const bool in = pass && (full || far2 <= g.t_eps);
    const bool straddle = pass && !in && !(near2 > g.t_eps);
    EGG_STAT(a, kUsSmallPass, pass);
    EGG_STAT(a, kUsFull, pass && full);
    EGG_STAT(a, kUsTightIn, in && !full);
    EGG_STAT(a, kUsTightOut, pass && !in && !straddle);
    if (!__any_sync(0xffffffffu, in || straddle)) return;
    // counted points and their sums: the whole cell's, or the walked ones
    unsigned long long av[2 * PS];
    int cnt = 0;
#pragma unroll
    for (int k = 0; k < 2 * PS; k++) av[k] = 0ull;
    if (in) {
#pragma unroll
        for (int j = 0; j < PS; j++) {
            const ulonglong2 t = rec[1 + 2 * PW + j];
            av[2 * j] = t.x;
            av[2 * j + 1] = t.y;
        }
        cnt = m_all;
    }
    if (__any_sync(0xffffffffu, straddle)) {
        const int qe = qb + m_all;
        const int kh = qb >> 5, kt = (qe - 1) >> 5;
        // points of group k; gr: its record (several groups only)
        auto visit_group = [&](int k, auto from, const ulonglong2* gr) {
            constexpr bool kGlobal = decltype(from)::value;
            const int sb = max(qb, k << 5), se = min(qe, (k << 5) + 32);
            const int m = se - sb;
            bool walk = straddle;
            if (kh != kt) {
                float n2, f2;
                box_dist2<D, kGlobal>(nx, x, gr + PS, n2, f2);
                const bool g_in = straddle && !(n2 > g.t_eps) && f2 <= g.t_eps;
                walk = straddle && !(n2 > g.t_eps) && !g_in;
                EGG_STAT(a, kUsGroupsOut, straddle && n2 > g.t_eps);
                EGG_STAT(a, kUsGroupsIn, g_in);
                if (g_in) {
                    add_point<D, kGlobal>(av, gr);
                    cnt += m;
                }
            }
            if (!__any_sync(0xffffffffu, walk)) return;
            __syncwarp();
            if (lane < m) {
                const ulonglong2* xp = reinterpret_cast<const ulonglong2*>(w.xp) + (size_t)(sb + lane) * PW;
#pragma unroll
                for (int j = 0; j < PW; j++) stage[lane * PW + j] = __ldg(xp + j);
                const ulonglong2* sp = reinterpret_cast<const ulonglong2*>(w.smp) + (size_t)(sb + lane) * PS;
#pragma unroll
                for (int j = 0; j < PS; j++) stage[32 * PW + lane * PS + j] = __ldg(sp + j);
            }
            __syncwarp();
            if (walk) {
                EGG_STAT(a, kUsPairs, m);
#pragma unroll kWalkUnroll
                for (int j = 0; j < m; j++) {
#ifdef EGG_UPDATE_STATS
                    {
                        const unsigned am_ = __activemask();
                        if ((threadIdx.x & 31) == __ffs(am_) - 1) a.st[kUsWalkSteps] += 1;
                    }
#endif
                    if (pair_dist2<D>(stage + j * PW, nx, x) <= g.t_eps) {
                        add_point<D, false>(av, stage + 32 * PW + j * PS);
                        cnt++;
                        EGG_STAT(a, kUsPairsIn, 1);
                    }
                }
            }
        };
        auto group = [&](int k) {
            return reinterpret_cast<const ulonglong2*>(group_rec<D>(w, k, (k == kh) ? 1 : 0, D));
        };
        if constexpr (D == 1) {
            // One dimension: cells of thousands of points.  Their groups come 32
            // at a time, one per lane, and stay where an active lane can count a
            // point of theirs (the screening of cells below); one load for all
            // lanes per group waited 600 cycles each (1M x 1 at eps 0.05, first
            // iteration: 15.0 ms, 5.4 with the screening, 5.5 with a thread per
            // point).
            constexpr int GW = PS + 2 * PW;
            ulonglong2* const recs = stage + 32 * (PW + PS);
            for (int k0 = kh; k0 <= kt; k0 += 32) {
                bool keep = k0 + lane <= kt;
                ulonglong2 r[GW];
                if (keep && kh != kt) {
                    const ulonglong2* gr = group(k0 + lane);
#pragma unroll
                    for (int j = 0; j < GW; j++) r[j] = __ldg(gr + j);
                    float lo, hi, skip;
                    unpack2(r[PS].x, lo, skip);
                    unpack2(r[PS + PW].x, hi, skip);
                    const float gap = fmaxf(fmaxf(lo - B.xh[0], B.xl[0] - hi) - B.mar, 0.f);
                    keep = !(gap * gap > g.t_eps * 1.0001f);
                }
                unsigned kept = __ballot_sync(0xffffffffu, keep);
                __syncwarp();  // the last chunk's records are read
                if (keep && kh != kt) {
#pragma unroll
                    for (int j = 0; j < GW; j++) recs[lane * GW + j] = r[j];
                }
                __syncwarp();
                for (; kept; kept &= kept - 1) {
                    const int src = __ffs(kept) - 1;
                    visit_group(k0 + src, std::false_type{}, recs + src * GW);
                }
            }
        } else {
            for (int k = kh; k <= kt; k++) visit_group(k, std::true_type{}, group(k));
        }
    }
    if (cnt) {
        float v[4 * PS];
        int kk[D];
#pragma unroll
        for (int j = 0; j < 2 * PS; j++) unpack2(av[j], v[2 * j], v[2 * j + 1]);
#pragma unroll
        for (int l = 0; l < D; l++) kk[l] = l < od ? col.kk[l] : (int)((key >> (16 * l)) & 0xffffu) - gi[l];
        // every offset is within the table: the lane passed the cell's box test
        add_counted<D>(a, kk, (float)cnt, v, v + D, tab, K);
        a.N += cnt;
        if (!full) a.partial_in += cnt;
    }
}

template <int D, int OD, bool tiled>
__device__ __forceinline__ bool walk_union(const Geom& g, const Work& w, const float* x, const int* gi, bool act,
                                           Acc<D>& a, const float4* tab, int K, ulonglong2* sh, int lane) {
    constexpr int PW = pack_w(D), PS = pack_s(D), CW = cell_words(D);
    const int od = OD > 0 ? OD : g.od;
    static_assert(sizeof(WarpBox<D>) <= 16 * box_words(D), "the joint box's words");
    volatile WarpBox<D>& B = *reinterpret_cast<WarpBox<D>*>(sh);
    ulonglong2* const cells = sh + box_words(D);
    ulonglong2* const stage = cells + 32 * CW;
    int ncol;
    bool spread;  // storage order, several columns: only with few candidates in all
    {
        float cols = 1.f, mar = 1.f, room = 1.f;
        const float inv_reach = 1.0f / (float)(2 * g.r + 1);
        bool one = true;
#pragma unroll
        for (int l = 0; l < D; l++) {
            const int lo = __reduce_min_sync(0xffffffffu, act ? gi[l] : INT_MAX);
            const int hi = __reduce_max_sync(0xffffffffu, act ? gi[l] : INT_MIN);
            const int wide = l < od ? min(g.width - 1, hi + g.r) - max(0, lo - g.r) + 1 : 1;
            cols *= (float)wide;
            room *= 1.0f + (float)(hi - lo) * inv_reach;
            if (l < od) one = one && lo == hi;
            if (l == od) one = one && hi - lo <= kLockZSpan;
            // the active lanes' bounding box, and a margin for the rounding of
            // the faces' offsets (relative to the coordinates)
            const float xl = order_val(__reduce_min_sync(0xffffffffu, act ? order_key(x[l]) : 0xffffffffu));
            const float xh = order_val(__reduce_max_sync(0xffffffffu, act ? order_key(x[l]) : 0u));
            mar = fmaxf(mar, fmaxf(fabsf(xl), fabsf(xh)));
            if (lane == 0) {
                B.lo[l] = lo;
                B.hi[l] = hi;
                B.wide[l] = wide;
                B.xl[l] = xl;
                B.xh[l] = xh;
            }
        }
        if ((tiled || !one) && cols > (float)kUnionCols) return false;
        if (tiled && room > kTileRoom) return false;
        spread = !tiled && !one;
        ncol = (int)cols;
        if (lane == 0) {
            const float inv = 1.0f / g.side;
            B.mar = mar * 4e-7f;
            B.r2 = g.t_eps * inv * inv * 1.002f;
        }
        __syncwarp();
    }
    unsigned long long nx[2 * PW];
    negate_pairs<D>(x, nx);
    Col<D> col;
    col.sm = col.lg = 0.f;
    // Whole rows (the columns of one row of dimension 0 follow each other, and
    // so do their cells) where they hold few cells, column by column otherwise.
    const int wide0 = od > 0 ? (int)B.wide[0] : 1;
    const int nrow = od > 1 ? ncol / wide0 : 1;
    int rowlen = 1;  // columns of a unit
    if (od > 0 && wide0 > 1) {
        bool few = true;
        int held = 0;
        for (int s0 = 0; s0 < nrow && few; s0 += 32) {
            int rem = s0 + lane, o = max(0, (int)B.lo[0] - g.r), m = 0;
#pragma unroll
            for (int l = 1; l < D; l++)
                if (l < od) {
                    const int wide = B.wide[l], q = rem / wide;
                    o += (max(0, (int)B.lo[l] - g.r) + rem - q * wide) * g.wpow[l];
                    rem = q;
                }
            if (s0 + lane < nrow) m = __ldg(w.outer_begin + o + wide0) - __ldg(w.outer_begin + o);
            held += __reduce_add_sync(0xffffffffu, m);
            few = od == D || held <= ncol * kRowFill;
        }
        if (few) rowlen = wide0;
        spread = spread && !(few && held <= kSpreadCells);
    }
    if (spread) return false;
    const int units = rowlen > 1 ? nrow : ncol;
    const int ob = 16 * od;
    const unsigned long long outer = ob >= 64 ? ~0ull : (1ull << ob) - 1ull;  // a packed key's outer coordinates
    for (int s0 = 0; s0 < units; s0 += 32) {
        // a column or a row per lane: its candidate cells [cb, ce)
        int cb = 0, ce = 0;
        {
            int rem = s0 + lane, o = rowlen > 1 ? max(0, (int)B.lo[0] - g.r) : 0;
            float exc = rem < units ? 0.f : INFINITY;
#pragma unroll
            for (int l = 0; l < D; l++)
                if (l < od && (l > 0 || rowlen == 1)) {
                    const int wide = B.wide[l], lo = B.lo[l];
                    const int q = rem / wide;
                    const int v = max(0, lo - g.r) + rem - q * wide;
                    rem = q;
                    o += v * g.wpow[l];
                    // no lane's cell is nearer than this many cells
                    const float gap = (float)max(max(lo - v, v - B.hi[l]), 0) - 1.001f;
                    exc += gap > 0.f ? gap * gap : 0.f;
                }
            if (exc <= B.r2) {
                cb = __ldg(w.outer_begin + o);
                ce = __ldg(w.outer_begin + o + rowlen);
                if (cb < ce && od < D && rowlen == 1) {
                    const int* keys = w.cell_dims + (size_t)od * g.ns;
                    cb = lower_bound_i(keys, cb, ce, B.lo[od < D ? od : 0] - g.r - 1);
                    ce = lower_bound_i(keys, cb, ce, B.hi[od < D ? od : 0] + g.r + 2);
                }
            }
        }
        // the chunk's candidates numbered through, unit by unit
        int upto = ce - cb;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, upto, k);
            if (lane >= k) upto += t;
        }
        const int total = __shfl_sync(0xffffffffu, upto, 31);
        const int shift = ce - upto;  // candidate f of this column is cell f + shift
        for (int f0 = 0; f0 < total; f0 += 32) {
            const int f = f0 + lane;
            bool keep = f < total;
            int nk;
            {
                // the column holding candidate f: the first with upto > f
                int src = 0;
#pragma unroll
                for (int k = 16; k > 0; k >>= 1) {
                    const int t = __shfl_sync(0xffffffffu, upto, src + k - 1);
                    if (t <= f) src += k;
                }
                src = min(src, 31);
                const int c = f + __shfl_sync(0xffffffffu, shift, src);
                unsigned long long key = 0;
                ulonglong2 bl[2 * PW];
                int qb = 0, qe = 0;
                if (keep) {
                    key = __ldg(w.cell_key + c);
                    qb = __ldg(w.cell_start + c);
                    qe = __ldg(w.cell_start + c + 1);
                    const ulonglong2* bp = reinterpret_cast<const ulonglong2*>(cell_box<D>(w, c, D));
#pragma unroll
                    for (int j = 0; j < 2 * PW; j++) bl[j] = __ldg(bp + j);
                    // no active lane passes the cell's box test, or no point of
                    // it is within eps of any (the tight box; a cell at the
                    // grid's edge also holds points beyond its own box and may
                    // count in full all the same)
                    float L[4 * PW], H[4 * PW], box2 = 0.f, tight2 = 0.f;
#pragma unroll
                    for (int j = 0; j < PW; j++) {
                        unpack2(bl[j].x, L[4 * j], L[4 * j + 1]);
                        unpack2(bl[j].y, L[4 * j + 2], L[4 * j + 3]);
                        unpack2(bl[PW + j].x, H[4 * j], H[4 * j + 1]);
                        unpack2(bl[PW + j].y, H[4 * j + 2], H[4 * j + 3]);
                    }
                    bool edge = false;
                    const float mar = B.mar, t_out = g.t_eps * 1.0001f;
#pragma unroll
                    for (int l = 0; l < D; l++) {
                        const float cd = key_dim_f(key, l), xl = B.xl[l], xh = B.xh[l];
                        const float gb = fmaxf(fmaxf(cd * g.side - xh, xl - (cd + 1.0f) * g.side) - mar, 0.f);
                        const float gt = fmaxf(fmaxf(L[l] - xh, xl - H[l]) - mar, 0.f);
                        box2 = fmaf(gb, gb, box2);
                        tight2 = fmaf(gt, gt, tight2);
                        edge = edge || cd == 0.f || cd >= (float)(g.width - 1);
                    }
                    keep = !(box2 > t_out) && (edge || !(tight2 > t_out));
                }
                const unsigned kept = __ballot_sync(0xffffffffu, keep);
                nk = __popc(kept);
                __syncwarp();  // the last chunk's records are read
                if (keep) {
                    ulonglong2* rec = cells + __popc(kept & ((1u << lane) - 1u)) * CW;
                    const ulonglong2* sp = reinterpret_cast<const ulonglong2*>(cell_sum<D>(w, c, D));
                    rec[0] = make_ulonglong2(key, (unsigned long long)(unsigned)qb |
                                                      ((unsigned long long)(unsigned)(qe - qb) << 32));
#pragma unroll
                    for (int j = 0; j < 2 * PW; j++) rec[1 + j] = bl[j];
#pragma unroll
                    for (int j = 0; j < PS; j++) rec[1 + 2 * PW + j] = __ldg(sp + j);
                }
                __syncwarp();
            }
            unsigned long long at = ~0ull;  // outer coordinates of the column col describes
#pragma unroll 1
            for (int j = 0; j < nk; j++) {
                const ulonglong2* rec = cells + j * CW;
#ifdef EGG_UPDATE_STATS
                const long long tv = clock64();
#endif
                const unsigned long long ck = rec[0].x & outer;
                if (ck != at) {
                    at = ck;
                    float sm = 0.f, lg = 0.f;
                    bool on = act;
#pragma unroll
                    for (int l = 0; l < D; l++)
                        if (l < od) {
                            const int k = (int)((ck >> (16 * l)) & 0xffffu) - gi[l];
                            col.kk[l] = k;
                            on = on && abs(k) <= g.r;
                            box_terms_f(x[l], key_dim_f(ck, l), g.side, sm, lg);
                        }
                    col.sm = on ? sm : INFINITY;
                    col.lg = lg;
                }
                visit_cell_warp<D, OD>(g, w, rec, x, nx, gi, col, a, tab, K, B, stage, lane);
#ifdef EGG_UPDATE_STATS
                if (lane == 0) {
                    a.st[kUsWarpVisits] += 1;
                    a.st[kUsCyclesVisits] += (unsigned)(clock64() - tv);
                }
#endif
            }
        }
    }
    return true;
}

}  // namespace

// One thread per point.  In tile order a warp's points are neighbours in
// space; otherwise they are 32 in a row of the storage order, the block's
// warps taking rows (several of them in a large set) from all over it (the
// points that still move late in a run sit together, and a block shares them
// out).  A warp none of whose points is touched keeps them all; one whose
// points are close enough walks their joint candidates in lockstep; of any
// other, in storage order, the groups of one place do so each, and the points
// left go on the block's list, whose warps take them one at a time
// (walk_point).  Every
// path visits a superset of the cells the reference visits and applies the
// reference's per-point box test to each, in the same order.
template <int D, int OD, bool tiled>
__device__ __forceinline__ void update_rows(const Geom& g, const Work& w, int* __restrict__ counts, int bx, int gx,
                                            int max_rows, float4* s_tab, int* s_list, int& s_count, volatile unsigned* state) {
    constexpr int d = D;
    // what a warp keeps across its walks waits in shared memory: the walk wants the registers
    volatile unsigned &s_heavy = state[0], &s_left = state[1], &s_grp = state[2], &s_listed = state[3];
    const int K = g.table_k, TW = 2 * K + 1;
    const int lane = threadIdx.x & 31;
    const int it = w.ctrl[kCtrlIter];
    // rows of 32 points per warp, and the blocks that takes (the others have none)
    const int rows = tiled ? 1 : min(max_rows, (gx + kRowBlocks - 1) / kRowBlocks), gxa = (gx + rows - 1) / rows;
    if (bx >= gxa) return;
    const int row0 = tiled ? bx * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5) : (int)(threadIdx.x >> 5) * rows * gxa + bx;
    // Rows none of whose points is touched are settled first, several at a
    // time: their loads overlap each other and the table's barrier (late in a
    // run nearly all of them).
    bool viol = false;
    unsigned heavy = 1u;
    if (!tiled && w.ctrl[kCtrlChanged] == 0 && counts == nullptr && w.ctrl[kCtrlForce] == 0) {
        heavy = 0;
        for (int k0 = 0; k0 < rows; k0 += kRowsAhead) {
            float xs[kRowsAhead][D];
            unsigned wv[kRowsAhead];
            unsigned long long nb[kRowsAhead];
#pragma unroll
            for (int k = 0; k < kRowsAhead; k++) {
                const int i = ((row0 + (k0 + k) * gxa) << 5) + lane;
                if (k0 + k < rows && i < g.n) {
                    wv[k] = w.warp_viol[i >> 5];
#pragma unroll
                    for (int l = 0; l < d; l++) xs[k][l] = w.X[(size_t)l * g.ns + i];
                }
            }
#pragma unroll
            for (int k = 0; k < kRowsAhead; k++) {
                const int i = ((row0 + (k0 + k) * gxa) << 5) + lane;
                nb[k] = 0;
                if (k0 + k < rows && i < g.n) {
                    int o = 0, z = 0;
#pragma unroll
                    for (int l = 0; l < d; l++) {
                        const int c = cell_dim(xs[k][l], g);
                        if (l < g.od) o += c * g.wpow[l];
                        if (l == g.od) z = c / g.zblk;
                    }
                    nb[k] = (w.need[o] >> z) & 1ull;
                }
            }
#pragma unroll
            for (int k = 0; k < kRowsAhead; k++) {
                const int i = ((row0 + (k0 + k) * gxa) << 5) + lane;
                if (__any_sync(0xffffffffu, nb[k] != 0)) {
                    heavy |= 1u << (k0 + k);
                } else if (k0 + k < rows && i < g.n) {
                    viol |= wv[k] != 0;
                    if (lane == 0) w.warp_moved[i >> 5] = 0;
                }
            }
        }
    } else if (rows > 1) {
        heavy = (1u << rows) - 1u;
    }
    for (int t = threadIdx.x; t < TW; t += blockDim.x)
        s_tab[t] = make_float4(w.table[t], w.table[TW + t], w.table[2 * TW + t], 0.f);
    if (threadIdx.x == 0) {
        s_count = 0;
        if (bx == 0) w.stamps[4 * it + 1] = globaltimer();
    }
    __syncthreads();
    if (!tiled && lane == 0) s_heavy = heavy;
    __syncwarp();
#pragma unroll 1
    while (true) {
        if constexpr (!tiled) {
            heavy = s_heavy;
            if (heavy == 0) break;
            __syncwarp();
            if (lane == 0) s_heavy = heavy & (heavy - 1);
        }
        const int t0 = ((row0 + (tiled ? 0 : (__ffs(heavy) - 1) * gxa)) << 5) + lane;
        if ((t0 & ~31) >= g.n) break;  // uniform across the warp
        const bool valid = t0 < g.n;
        const int tv = valid ? t0 : g.n - 1;  // lanes past n shadow the last point; their results are dropped
        const int i = tiled ? w.perm[tv] : tv;
        float x[D];
#pragma unroll
        for (int l = 0; l < d; l++) x[l] = w.X[(size_t)l * g.ns + i];
        bool bad = false;  // the point violates
        int gi[D];
        int obase = 0;
#pragma unroll
        for (int l = 0; l < d; l++) {
            gi[l] = cell_dim(x[l], g);
            if (l < g.od) obase += gi[l] * g.wpow[l];
        }
        // Incremental update: when no point of a point's stencil region moved
        // (old or new position) since the last update, every input of its
        // update is unchanged, so the result is the same bit for bit: it keeps
        // the position and the last violation bit.  The need bit is read again
        // where it is used, so nothing extra stays live over the walk.
        auto zblk_of = [&]() {
            int z = 0;
#pragma unroll
            for (int l = 0; l < d; l++)
                if (l == g.od) z = gi[l] / g.zblk;
            return z;
        };
        auto needs = [&]() {
            return valid && (counts != nullptr || w.ctrl[kCtrlForce] != 0 || ((w.need[obase] >> zblk_of()) & 1ull) != 0);
        };
        const unsigned nm = __ballot_sync(0xffffffffu, needs());
        Acc<D> a;
#pragma unroll
        for (int l = 0; l < d; l++) a.S[l] = a.Cm[l] = 0.f;
        a.N = a.partial_in = 0;
#ifdef EGG_UPDATE_STATS
        for (int k = 0; k < kUStats; k++) a.st[k] = 0;
        const long long t_walk0 = clock64();
#endif
        bool done = false;    // the point has its sums
        unsigned listed = 0;  // the lanes whose points go on the list
        if (nm) {
            if (lane == 0) atomicAdd(w.ctrl + kCtrlComputed, __popc(nm));
            ulonglong2* sh = reinterpret_cast<ulonglong2*>(s_tab + TW) + (threadIdx.x >> 5) * warp_words(D);
            if constexpr (tiled) {
                done = walk_union<D, OD, true>(g, w, x, gi, needs(), a, s_tab, K, sh, lane);
                if (!done) listed = nm;
            } else {
                // all together, or (storage order) by groups of one place
                if (lane == 0) {
                    s_left = s_grp = nm;
                    s_listed = 0;
                }
                __syncwarp();
                bool whole = true;
#pragma unroll 1
                while (true) {
                    const bool mine = (s_grp >> lane) & 1u;
                    const bool walked = walk_union<D, OD, false>(g, w, x, gi, mine, a, s_tab, K, sh, lane);
                    done = done || (walked && mine);
                    unsigned left = s_left, more = 0;
                    if (walked) left &= ~s_grp;
                    if (walked || whole) {
                        while (left) {  // the next group worth a walk
                            const int first = __ffs(left) - 1;
                            bool same = (left >> lane) & 1u;
#pragma unroll
                            for (int l = 0; l < D; l++) {
                                const int gf = __shfl_sync(0xffffffffu, gi[l], first);
                                same = same && abs(gi[l] - gf) <= (l < g.od ? 0 : l == g.od ? kLockZSpan / 2 : g.width);
                            }
                            const unsigned grp = __ballot_sync(0xffffffffu, same);
                            if (__popc(grp) >= kGroupMin) {
                                more = grp;
                                break;
                            }
                            left &= ~grp;
                            listed |= grp;
                        }
                    } else {
                        listed |= left;
                        left = 0;
                    }
                    listed |= s_listed;
                    __syncwarp();
                    if (lane == 0) {
                        s_left = left;
                        s_grp = more;
                        s_listed = listed;
                    }
                    __syncwarp();
                    whole = false;
                    if (more == 0) break;
                }
                listed = s_listed;
            }
            if ((listed >> lane) & 1u) s_list[atomicAdd(&s_count, 1)] = i;
        }
#ifdef EGG_UPDATE_STATS
        if (nm) {
            const long long dt = clock64() - t_walk0;
            const long long warp_dt = __reduce_max_sync(0xffffffffu, (unsigned)min(dt, 0x7fffffffLL));
            if (lane == 0) a.st[listed ? kUsCyclesLane : kUsCyclesShared] += (unsigned)warp_dt;
            if (lane == 0 && listed) a.st[kUsLaneWarps] = 1;
        }
#endif
        bool moved = false;
        if (valid && !needs()) {
            // Xn equals X unless this iteration rebuilt the grid (the grid
            // check copied Xn into X; a rebuild reorders X only).  A rebuild
            // reorders the points, and in tile order the storage warps' words
            // are not kept up: then the violation bit goes by original index.
            if (w.ctrl[kCtrlChanged] != 0)
                for (int l = 0; l < d; l++) w.Xn[(size_t)l * g.ns + i] = x[l];
            bad = tiled || w.ctrl[kCtrlChanged] != 0 ? w.viol_orig[w.orig[i]] != 0 : ((w.warp_viol[i >> 5] >> lane) & 1u) != 0;
        } else if (valid && done) {
            const int N = a.N;
            const float fN = (float)N;
            bool border = false;
            int onew = 0, zbnew = 0;
#pragma unroll
            for (int l = 0; l < d; l++) {
                border |= on_border_dim(x[l], g.side);
                const float corner = __fmul_rn((float)gi[l], g.side);
                const float phi = x[l] - corner;
                float sp, cp;
                sincosf(phi, &sp, &cp);
                const float A = cp * a.S[l] - sp * (fN - a.Cm[l]);
                const float xn = x[l] + A / fN;
                w.Xn[(size_t)l * g.ns + i] = xn;
                moved |= __float_as_uint(xn) != __float_as_uint(x[l]);
                if (l < g.od) onew += cell_dim(xn, g) * g.wpow[l];
                if (l == g.od) zbnew = cell_dim(xn, g) / g.zblk;
            }
            if (counts) counts[i] = N;
            // convergence flag, EGG_SynC.cu:706-709.  half_count <= N -
            // partial_in, so a border point with neighbours in a partial cell
            // always violates.
            const int own = w.cell_of[i];
            const int own_cnt = w.cell_start[own + 1] - w.cell_start[own];
            if (!border) bad = (N != own_cnt);
            else if (a.partial_in > 0) bad = true;
            else if (N == own_cnt) bad = false;
            else {
                bad = (N != half_count<D>(g, w, x, gi, obase, own, own_cnt));
                EGG_STAT(a, kUsHalfCount, 1);
            }
            w.viol_orig[w.orig[i]] = bad ? 1 : 0;
            if (moved) {
                unsigned long long* dcur = w.dirty[it & 1];
                atomicOr(dcur + obase, 1ull << zblk_of());
                atomicOr(dcur + onew, 1ull << zbnew);
            }
            EGG_STAT(a, kUsPoints, 1);
            EGG_STAT(a, kUsNeighbors, N);
        }
        // the storage warps whose points moved: the next grid check reads only
        // those (in tile order the cell-sums kernels of this iteration cleared
        // the marks; a listed point adds its own mark and bit below)
        const unsigned vb = __ballot_sync(0xffffffffu, bad), mb = __ballot_sync(0xffffffffu, moved);
        viol |= bad;
        if (tiled) {
            if (moved) w.warp_moved[i >> 5] = 1;
        } else if (lane == 0) {
            w.warp_moved[i >> 5] = mb != 0;
            if (nm || w.ctrl[kCtrlChanged] != 0) w.warp_viol[i >> 5] = vb;
        }
#ifdef EGG_UPDATE_STATS
        for (int k = 0; k < kUStats; k++) {
            unsigned long long v = a.st[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && v) atomicAdd(w.ustats + k, v);
        }
#endif
        if (tiled) break;
    }
    __syncthreads();
    const int todo = s_count;
    if (todo) {
        float* area = reinterpret_cast<float*>(s_tab + TW) + (threadIdx.x >> 5) * (4 * warp_words(D));
        viol |= update_listed_points<D, true, 16>(g, w, counts, s_tab, area, s_list, todo, !tiled);
    }
    if (__any_sync(0xffffffffu, viol) && lane == 0) {
        volatile int* f = w.ctrl + kCtrlFlag;
        if (*f != 0) *f = 0;
    }
}

// The two orders are compiled apart: one body for both cost the first
// iterations (tile order) 3% to 17%.
template <int D, int OD>
__device__ __forceinline__ void update_body(const Geom& g, const Work& w, int* __restrict__ counts, int bx, int gx,
                                            int max_rows) {
    extern __shared__ float4 s_tab[];  // sin, cos, 1 - cos of k * side; then each warp's area
    __shared__ int s_list[kListMax];
    __shared__ int s_count;
    __shared__ volatile unsigned s_state[8][4];
    volatile unsigned* const state = s_state[threadIdx.x >> 5];
    if constexpr (tile_dims(D)) {
        if (w.ctrl[kCtrlTiled] != 0) {
            update_rows<D, OD, true>(g, w, counts, bx, gx, max_rows, s_tab, s_list, s_count, state);
            return;
        }
    }
    update_rows<D, OD, false>(g, w, counts, bx, gx, max_rows, s_tab, s_list, s_count, state);
}

template <int D, int OD>
__global__ void __launch_bounds__(128, update_min_blocks(D, 128)) k_update(Geom g, Work w, int* __restrict__ counts) {
    update_body<D, OD>(g, w, counts, blockIdx.x, gridDim.x, kListMax / 128);
}

template <int D, int T>
__global__ void __launch_bounds__(T, update_min_blocks(D, T)) kb_update(BatchArgs B) {
    batch_for(B, [&](const Geom& g, const Work& w, int bx, int gx) { update_body<D, 0>(g, w, nullptr, bx, gx, 1); });
}

// need[] (zeroed by the grid-build check of this iteration) receives, over
// the stencil of every outer cell that the previous update marked dirty, the
// dirty blocks of dimension od widened by r + 1 cells on each side: exactly
// the points whose candidate cells (outer stencil, dimension od within
// r + 1 cells, for_candidates) can hold a moved point's old or new position.
// The dirty marks are cleared as they are consumed, so the array is clean
// again when the update after next writes it.
// A warp reads kNeedChunk outer cells at once; the lanes share the stencil
// entries of each dirty one (dirty cells cluster around the regions still
// moving, so a long run of them per warp would hold the whole launch).
// The dilation is closed-form: block b covers the blocks
// [b - ceil((r+1)/zblk), b + 1 + floor(r/zblk)], clipped to [0, nzb).
constexpr int kNeedChunk = 8;

__device__ __forceinline__ void need_body(const Geom& g, const Work& w, int bx, int gx) {
    const int it = w.ctrl[kCtrlIter];
    unsigned long long* prev = w.dirty[(it + 1) & 1];
    const int nst = w.st_count[0];
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int lo_sh = min(63, (g.r + g.zblk) / g.zblk), hi_sh = min(63, 1 + g.r / g.zblk);
    const unsigned long long full = g.nzb >= 64 ? ~0ull : (1ull << g.nzb) - 1ull;
    const long long stride = (long long)gx * wpb * kNeedChunk;
    // warp-uniform loop over chunks of outer cells
    for (long long o0 = ((long long)bx * wpb + (threadIdx.x >> 5)) * kNeedChunk; o0 < g.n_outer; o0 += stride) {
        const long long o = o0 + lane;
        const unsigned long long mine = (lane < kNeedChunk && o < g.n_outer) ? prev[o] : 0ull;
        if (mine) prev[o] = 0;
        unsigned todo = __ballot_sync(0xffffffffu, mine != 0);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const unsigned long long m = __shfl_sync(0xffffffffu, mine, src);
            const int oc = (int)o0 + src;
            unsigned long long dil = 0;
            for (int s = 0; s <= lo_sh; s++) dil |= m >> s;
            for (int s = 1; s <= hi_sh; s++) dil |= m << s;
            dil &= full;
            int co[32];
            int rem = oc;
            for (int l = 0; l < g.od; l++) {
                co[l] = rem % g.width;
                rem /= g.width;
            }
            for (int s = lane; s < nst; s += 32) {
                bool inb = true;
                for (int l = 0; l < g.od; l++) {
                    const int v = co[l] + __ldg(w.st_off + (size_t)s * g.od + l);
                    inb = inb && (unsigned)v < (unsigned)g.width;
                }
                if (inb) atomicOr(w.need + oc + __ldg(w.st_delta + s), dil);
            }
        }
    }
}

__global__ void k_need(Geom g, Work w) { need_body(g, w, blockIdx.x, gridDim.x); }

__global__ void kb_need(BatchArgs B) {
    batch_for(B, [&](const Geom& g, const Work& w, int bx, int gx) { need_body(g, w, bx, gx); });
}

void launch_need(const Exec& ex, cudaStream_t st) {
    if (ex.batch())
        kb_need<<<ex.blocks(kShapeCapOuter, 256), 256, 0, st>>>(ex.args(kShapeCapOuter));
    else
        k_need<<<ex.blocks(kShapeCapOuter, 256), 256, 0, st>>>(*ex.g, *ex.w);
}

template <int T>
void launch_update_batch(const Exec& ex, size_t smem, cudaStream_t st) {
    const int shape = T == 128 ? kShapeN128 : kShapeN256;
    // beside 13 KB of descriptors, list and state: 48 KB together need no opt-in
    auto go = [&](auto kernel) {
        if (smem > 32 * 1024) EGG_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kernel<<<ex.blocks(shape, T), T, smem, st>>>(ex.args(shape));
    };
    switch (ex.d) {
        case 1: go(kb_update<1, T>); break;
        case 2: go(kb_update<2, T>); break;
        case 3: go(kb_update<3, T>); break;
        case 4: go(kb_update<4, T>); break;
        default: break;  // d > 4: launch_update_wide
    }
}

void launch_update(const Exec& ex, int* counts, cudaStream_t st) {
    // below the tile order's size too few warps of 32 points are at hand to
    // fill the chip: a warp per point (10k x 2D)
    if (ex.d > 4 || (!ex.batch() && ex.g->point_walk)) {
        launch_update_wide(ex, counts, st);
        return;
    }
    const size_t stage = (size_t)warp_words(ex.d);  // 16-byte words per warp (point walks take less)
    const size_t smem = 16 * ((2 * (size_t)ex.table_k() + 1) + stage * (ex.update_threads() / 32));
    if (ex.batch()) {
        switch (ex.update_threads()) {
            case 128: launch_update_batch<128>(ex, smem, st); break;
            default: launch_update_batch<256>(ex, smem, st); break;
        }
    } else {
        // two outer dimensions are what n points give (width^2 <= n < width^3)
        // at nearly every eps in use: known to the compiler for d = 2, 3, 4
        const bool od2 = ex.g->od == 2;
        const int blocks = ex.blocks(kShapeN128, 128);
        auto go = [&](auto kernel) { kernel<<<blocks, 128, smem, st>>>(*ex.g, *ex.w, counts); };
        switch (ex.d) {
            case 1: go(k_update<1, 0>); break;
            case 2: od2 ? go(k_update<2, 2>) : go(k_update<2, 0>); break;
            case 3: od2 ? go(k_update<3, 2>) : go(k_update<3, 0>); break;
            case 4: od2 ? go(k_update<4, 2>) : go(k_update<4, 0>); break;
            default: break;  // d > 4: launch_update_wide
        }
    }
}

}  // namespace egg
