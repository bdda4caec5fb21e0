// egg_point_walk.cuh -- one point's update sums by a whole warp.
//
// The candidate cells of the point come 32 at a time, one per lane
// (consecutive cells: their keys are coalesced); those that pass the box test
// queue up in shared memory in candidate order; 32 queued cells at a time, a
// lane decides its cell (aggregate, skip or walk) and forms its contribution
// to the point's 2d sums; lane k then adds component k of the contributions
// in candidate order, so the sums round exactly as one thread's running sums
// do.  A point's latency is its candidates / 32 instead of all in a row.
#pragma once

#include "egg_common.cuh"

namespace egg {

// candidates of point i's cell `own`, 32 at a time in stencil and cell order;
// fn(c, valid) is called by all lanes together
template <typename F>
__device__ __forceinline__ void for_point_cells(const Geom& g, const Work& w, int own, int lane, F&& fn) {
    const int nst = w.st_count[0];
    const int obase = __ldg(w.cell_outer + own);
    const int* keys = w.cell_dims + (size_t)g.od * g.ns;
    const int z0 = g.od < g.d ? __ldg(keys + own) : 0;
    for (int s0 = 0; s0 < nst; s0 += 32) {
        const int s = s0 + lane;
        int cb = 0, ce = 0;
        if (s < nst) {
            bool inb = true;
            for (int l = 0; l < g.od; l++) {
                const int v = __ldg(w.cell_dims + (size_t)l * g.ns + own) + __ldg(w.st_off + (size_t)s * g.od + l);
                inb = inb && (unsigned)v < (unsigned)g.width;
            }
            if (inb) {
                const int o = obase + __ldg(w.st_delta + s);
                cb = __ldg(w.outer_begin + o);
                ce = __ldg(w.outer_begin + o + 1);
                if (cb < ce && g.od < g.d) {
                    cb = lower_bound_i(keys, cb, ce, z0 - g.r - 1);
                    ce = lower_bound_i(keys, cb, ce, z0 + g.r + 2);
                }
            }
        }
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
            int src = 0;  // the column holding candidate f: the first with upto > f
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) {
                const int t = __shfl_sync(0xffffffffu, upto, src + k - 1);
                if (t <= f) src += k;
            }
            const int c = f + __shfl_sync(0xffffffffu, shift, min(src, 31));
            fn(c, f < total);
        }
    }
}

constexpr int kWalkQueue = 64;

// shared floats of one warp: contributions [2 dm][33], sums [2 dm], queue
__host__ __device__ constexpr int walk_floats(int dm) { return 2 * dm * 33 + 2 * dm + kWalkQueue; }

#ifdef EGG_UPDATE_STATS
#define EGG_WSTAT(k, v) (st[k] += (v))
#else
#define EGG_WSTAT(k, v) ((void)0)
#endif

// What the walk knows a cell by.  DM: the dimensions the compiler knows the
// arrays by (0: any d, no keys); EX: d == DM exactly; KB: bits of a key's
// coordinate (8 only where DM > 8).
template <int DM, bool EX, int KB>
struct CellReader {
    static constexpr int LM = DM > 0 ? DM : kMaxDims;
    static constexpr int U = DM > 0 ? DM : 1;
    static constexpr int NW = DM <= 4 ? 2 : (DM > 8 && KB == 16 ? 8 : 4);  // words of a key

    static __device__ __forceinline__ void load_key(const Work& w, int c, unsigned* key) {
        if constexpr (DM > 0 && DM <= 4) {
            const unsigned long long v = __ldg(w.cell_key + c);
            key[0] = (unsigned)v;
            key[1] = (unsigned)(v >> 32);
        } else if constexpr (DM > 0) {
#pragma unroll
            for (int k = 0; k < NW / 4; k++) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(w.cell_wkey + (size_t)c * (4 * NW)) + k);
                key[4 * k] = v.x;
                key[4 * k + 1] = v.y;
                key[4 * k + 2] = v.z;
                key[4 * k + 3] = v.w;
            }
        }
    }
    static __device__ __forceinline__ int coord(const Geom& g, const Work& w, const unsigned* key, int c, int l) {
        if constexpr (DM > 0 && KB == 16) return (int)((key[l >> 1] >> (16 * (l & 1))) & 0xffffu);
        else if constexpr (DM > 0) return (int)((key[l >> 2] >> (8 * (l & 3))) & 255u);
        else return __ldg(w.cell_dims + (size_t)l * g.ns + c);
    }
    // the coordinate as a float: its bits are the low mantissa of 2^23 + cd
    static __device__ __forceinline__ float coord_f(const Geom& g, const Work& w, const unsigned* key, int c, int l) {
        if constexpr (DM > 0 && KB == 16)
            return __uint_as_float(__byte_perm(key[l >> 1], 0x4b000000u, (l & 1) ? 0x7432 : 0x7410)) - 8388608.0f;
        else if constexpr (DM > 0)
            return __uint_as_float(__byte_perm(key[l >> 2], 0x4b000000u, 0x7440 | (l & 3))) - 8388608.0f;
        else
            return (float)coord(g, w, key, c, l);
    }
    // the reference's box sums (EGG_SynC.cu:613-630) of cell c for x
    static __device__ __forceinline__ void box_sums(const Geom& g, const Work& w, int d, const float* x, int c,
                                                    float& sm2, float& lg2) {
        unsigned key[NW];
        load_key(w, c, key);
        sm2 = lg2 = 0.f;
#pragma unroll U
        for (int l = 0; l < LM; l++) {
            if (!EX && l >= d) break;
            const float cd = coord_f(g, w, key, c, l);
            const float left = __fmaf_rn(cd, g.side, -x[l]), right = __fmaf_rn(cd + 1.0f, g.side, -x[l]);
            const float l2 = __fmul_rn(left, left), r2 = __fmul_rn(right, right);
            sm2 = __fadd_rn(sm2, fminf(l2, r2));
            lg2 = __fadd_rn(lg2, fmaxf(l2, r2));
        }
    }
    // the first m floats of a record in whole words (d known to the compiler)
    static __device__ __forceinline__ void load_words(const float* rec, float* v, int m) {
#pragma unroll
        for (int k = 0; k < (2 * LM + 3) / 4; k++) {
            if (4 * k >= m) break;
            const float4 t = __ldg(reinterpret_cast<const float4*>(rec) + k);
            v[4 * k] = t.x;
            if (4 * k + 1 < 2 * LM) v[4 * k + 1] = t.y;
            if (4 * k + 2 < 2 * LM) v[4 * k + 2] = t.z;
            if (4 * k + 3 < 2 * LM) v[4 * k + 3] = t.w;
        }
    }
    // squared distances to the nearest and farthest point of a box record
    static __device__ __forceinline__ void box_near_far(int d, const float* x, const float* box, float& near2,
                                                        float& far2) {
        near2 = far2 = 0.f;
        const int bw = box_w(EX ? LM : d);
        float L[EX ? 2 * LM : 1], H[EX ? 2 * LM : 1];
        if constexpr (EX) {
            load_words(box, L, LM);
            load_words(box + bw, H, LM);
        }
#pragma unroll U
        for (int l = 0; l < LM; l++) {
            if (!EX && l >= d) break;
            const float dl = __fsub_rn(EX ? L[EX ? l : 0] : __ldg(box + l), x[l]);
            const float dh = __fsub_rn(EX ? H[EX ? l : 0] : __ldg(box + bw + l), x[l]);
            const float a = fmaxf(fmaxf(dl, -dh), 0.f), b = fmaxf(fabsf(dl), fabsf(dh));
            near2 = __fmaf_rn(a, a, near2);
            far2 = __fmaf_rn(b, b, far2);
        }
    }
};

// The sums S, Cm of the point at x (cell coordinates gi, cell own) into
// sums[0..LM) and sums[LM..2 LM) of the warp's shared area, |N(p)| and the
// points counted outside fully covered cells into N and partial_in (every
// lane).  All 32 lanes of the warp call it.
template <int DM, bool EX, int KB>
__device__ __forceinline__ void walk_point(const Geom& g, const Work& w, const float* x, const int* gi, int own,
                                           const float4* tab, float* area, int lane, int& N_out, int& partial_out,
                                           unsigned* st) {
    using R = CellReader<DM, EX, KB>;
    constexpr int LM = R::LM, U = R::U, SLOTS = (2 * LM + 31) / 32;
    const int d = EX ? DM : g.d;
    const int K = g.table_k;
    float* const terms = area;
    float* const sums = terms + 2 * LM * 33;
    int* const queue = reinterpret_cast<int*>(sums + 2 * LM);
    float acc[SLOTS];  // lane k: sum component k, k + 32, ... (S, then Cm)
#pragma unroll
    for (int j = 0; j < SLOTS; j++) acc[j] = 0.f;
    int N = 0, partial_in = 0;  // this lane's share

    // the first m <= 32 queued cells, a lane each
    auto flush = [&](int m) {
        int cnt = 0;
        bool full = false;
        float av[2 * LM];  // sums of the counted points: sin, then 1 - cos
        float *const as = av, *const am = av + LM;
        const int qv = lane < m ? queue[lane] : 0;
        const int c = qv & 0x7fffffff;
        if (lane < m) {
            float near2, far2;
            full = qv < 0;
            const int qb = __ldg(w.cell_start + c), qe = __ldg(w.cell_start + c + 1);
            R::box_near_far(d, x, w.cbox + (size_t)c * (2 * box_w(EX ? LM : d)), near2, far2);
            const bool in = full || far2 <= g.t_eps;
            EGG_WSTAT(kUsFull, full);
            EGG_WSTAT(kUsTightIn, in && !full);
            EGG_WSTAT(kUsTightOut, !in && near2 > g.t_eps);
            if (in) {
                const float* rec = w.csum + (size_t)c * sum_w(EX ? LM : d);
                if constexpr (EX) {
                    R::load_words(rec, av, 2 * LM);
                } else {
#pragma unroll U
                    for (int l = 0; l < LM; l++) {
                        if (l >= d) break;
                        as[l] = __ldg(rec + l);
                        am[l] = __ldg(rec + d + l);
                    }
                }
                cnt = qe - qb;
            } else if (!(near2 > g.t_eps)) {
#pragma unroll U
                for (int l = 0; l < LM; l++) {
                    if (!EX && l >= d) break;
                    as[l] = am[l] = 0.f;
                }
                const int kh = qb >> 5, kt = (qe - 1) >> 5;
                for (int k = kh; k <= kt; k++) {
                    const int sb = max(qb, k << 5), se = min(qe, (k << 5) + 32);
                    if (kh != kt) {
                        // a 32-point group of the cell: its tight box decides it wholesale
                        const float* rec = group_rec<0>(w, k, (k == kh) ? 1 : 0, EX ? LM : d);
                        float n2, f2;
                        R::box_near_far(d, x, rec + sum_w(EX ? LM : d), n2, f2);
                        if (n2 > g.t_eps) {
                            EGG_WSTAT(kUsGroupsOut, 1);
                            continue;
                        }
                        if (f2 <= g.t_eps) {
                            EGG_WSTAT(kUsGroupsIn, 1);
#pragma unroll U
                            for (int l = 0; l < LM; l++) {
                                if (!EX && l >= d) break;
                                as[l] += __ldg(rec + l);
                                am[l] += __ldg(rec + (EX ? LM : d) + l);
                            }
                            cnt += se - sb;
                            continue;
                        }
                    }
                    EGG_WSTAT(kUsPairs, se - sb);
                    for (int q = sb; q < se; q++) {
                        float d2 = 0.f;
                        if constexpr (EX && packed_dims(DM)) {
                            float xq[2 * LM], v[2 * LM];
                            R::load_words(reinterpret_cast<const float*>(w.xp) + (size_t)q * box_w(LM), xq, LM);
#pragma unroll
                            for (int l = 0; l < LM; l++) d2 = dist_step(xq[l], x[l], d2);
                            if (d2 <= g.t_eps) {
                                R::load_words(reinterpret_cast<const float*>(w.smp) + (size_t)q * sum_w(LM), v, 2 * LM);
#pragma unroll
                                for (int l = 0; l < 2 * LM; l++) av[l] += v[l];
                                cnt++;
                                EGG_WSTAT(kUsPairsIn, 1);
                            }
                        } else {
#pragma unroll U
                            for (int l = 0; l < LM; l++) {
                                if (!EX && l >= d) break;
                                d2 = dist_step(__ldg(w.X + (size_t)l * g.ns + q), x[l], d2);
                            }
                            if (d2 <= g.t_eps) {
                                const bool pk = packed_dims(d);
                                const float* ss = pk ? reinterpret_cast<const float*>(w.smp) + (size_t)q * sum_w(d) : w.sd + q;
                                const float* sm = pk ? ss + d : w.md + q;
                                const size_t step = pk ? 1 : (size_t)g.ns;
#pragma unroll U
                                for (int l = 0; l < LM; l++) {
                                    if (!EX && l >= d) break;
                                    as[l] += __ldg(ss + l * step);
                                    am[l] += __ldg(sm + l * step);
                                }
                                cnt++;
                                EGG_WSTAT(kUsPairsIn, 1);
                            }
                        }
                    }
                }
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, cnt > 0);
        if (cnt > 0) {
            // the contribution in the point's own-cell frame (every offset is
            // within the table: the cell passed the box test)
            float* t = terms + __popc(mask & ((1u << lane) - 1u));
            const float mf = (float)cnt;
            unsigned key[R::NW];
            R::load_key(w, c, key);
#pragma unroll U
            for (int l = 0; l < LM; l++) {
                if (!EX && l >= d) break;
                const float4 e = tab[R::coord(g, w, key, c, l) - gi[l] + K];
                const float ts = e.x, tc = e.y, tm = e.z;
                t[l * 33] = ts * (mf - am[l]) + tc * as[l];
                t[(LM + l) * 33] = mf * tm + tc * am[l] + ts * as[l];
            }
            N += cnt;
            if (!full) partial_in += cnt;
        }
        __syncwarp();
        const int nb = __popc(mask);
#pragma unroll
        for (int j = 0; j < SLOTS; j++) {
            const int k = lane + 32 * j;
            if (k < 2 * LM && (EX || (k < LM ? k < d : k - LM < d))) {
                float a = acc[j];
#pragma unroll 4
                for (int b = 0; b < nb; b++) a = __fadd_rn(a, terms[k * 33 + b]);
                acc[j] = a;
            }
        }
        __syncwarp();
    };

    int qn = 0;
    for_point_cells(g, w, own, lane, [&](int c, bool in_list) {
        bool pass = false, full = false;
        if (in_list) {
            float sm2, lg2;
            R::box_sums(g, w, d, x, c, sm2, lg2);
            pass = sm2 <= g.t_eps;
            full = lg2 <= g.t_eps;
            EGG_WSTAT(kUsCells, 1);
            EGG_WSTAT(kUsSmallPass, pass);
        }
        const unsigned m = __ballot_sync(0xffffffffu, pass);
        if (pass) queue[qn + __popc(m & ((1u << lane) - 1u))] = c | (full ? (int)0x80000000 : 0);
        qn += __popc(m);
        __syncwarp();
        if (qn >= 32) {
            flush(32);
            const int rest = lane < qn - 32 ? queue[32 + lane] : 0;
            __syncwarp();
            if (lane < qn - 32) queue[lane] = rest;
            qn -= 32;
            __syncwarp();
        }
    });
    if (qn > 0) flush(qn);
#pragma unroll
    for (int j = 0; j < SLOTS; j++) {
        const int k = lane + 32 * j;
        if (k < 2 * LM) sums[k] = acc[j];
    }
    N_out = __reduce_add_sync(0xffffffffu, N);
    partial_out = __reduce_add_sync(0xffffffffu, partial_in);
    __syncwarp();
}

// The update of the todo points of a block's list, a warp per point; `area`
// is the warp's shared memory.  words: the storage warps' violation words are
// in use (they hold a zero for the point).  Returns whether a point violates
// (every lane of the warp).
template <int DM, bool EX, int KB>
__device__ __forceinline__ bool update_listed_points(const Geom& g, const Work& w, int* __restrict__ counts,
                                                     const float4* tab, float* area, const int* list, int todo,
                                                     bool words) {
    using R = CellReader<DM, EX, KB>;
    constexpr int LM = R::LM, U = R::U;
    const int d = EX ? DM : g.d;
    const int lane = threadIdx.x & 31;
    const float* const sums = area + 2 * LM * 33;
    const int it = w.ctrl[kCtrlIter];
    bool any_viol = false;
    for (int e = threadIdx.x >> 5; e < todo; e += blockDim.x >> 5) {
        const int i = list[e];
        const int own = w.cell_of[i];
#ifdef EGG_UPDATE_STATS
        unsigned st[kUStats] = {};
#endif
        float x[LM];
        int gi[LM];
#pragma unroll U
        for (int l = 0; l < LM; l++) {
            if (!EX && l >= d) break;
            x[l] = w.X[(size_t)l * g.ns + i];
            gi[l] = __ldg(w.cell_dims + (size_t)l * g.ns + own);
        }
        int N, partial_in;
#ifdef EGG_UPDATE_STATS
        walk_point<DM, EX, KB>(g, w, x, gi, own, tab, area, lane, N, partial_in, st);
#else
        walk_point<DM, EX, KB>(g, w, x, gi, own, tab, area, lane, N, partial_in, nullptr);
#endif
        // the new position: lane l takes dimension l
        const float fN = (float)N;
        bool moved = false, border = false;
        int onew = 0, zbnew = 0;
        for (int l = lane; l < d; l += 32) {
            const float xl = w.X[(size_t)l * g.ns + i];
            const float corner = __fmul_rn((float)__ldg(w.cell_dims + (size_t)l * g.ns + own), g.side);
            const float phi = xl - corner;
            float sp, cp;
            sincosf(phi, &sp, &cp);
            const float A = cp * sums[l] - sp * (fN - sums[LM + l]);
            const float xn = xl + A / fN;
            w.Xn[(size_t)l * g.ns + i] = xn;
            moved |= __float_as_uint(xn) != __float_as_uint(xl);
            border |= on_border_dim(xl, g.side);
            if (l < g.od) onew += cell_dim(xn, g) * g.wpow[l];
            if (l == g.od) zbnew = cell_dim(xn, g) / g.zblk;
        }
        moved = __any_sync(0xffffffffu, moved);
        border = __any_sync(0xffffffffu, border);
        onew = __reduce_add_sync(0xffffffffu, onew);
        zbnew = __reduce_add_sync(0xffffffffu, zbnew);
        // convergence flag, EGG_SynC.cu:706-709.  half_count <= N - partial_in,
        // so a border point with neighbours in a partial cell always violates.
        const int own_b = w.cell_start[own], own_cnt = w.cell_start[own + 1] - own_b;
        bool viol;
        if (!border) {
            viol = N != own_cnt;
        } else if (partial_in > 0) {
            viol = true;
        } else if (N == own_cnt) {
            viol = false;
        } else {
            // reference half_count (EGG_SynC.cu:666-681): own cell plus the
            // points within eps/2 in the other fully covered cells
            int half = 0;
            for_point_cells(g, w, own, lane, [&](int c, bool in_list) {
                if (!in_list || c == own) return;
                float sm2, lg2, near2, far2;
                R::box_sums(g, w, d, x, c, sm2, lg2);
                if (!(lg2 <= g.t_eps)) return;
                const int qb = __ldg(w.cell_start + c), qe = __ldg(w.cell_start + c + 1);
                R::box_near_far(d, x, w.cbox + (size_t)c * (2 * box_w(d)), near2, far2);
                if (near2 > g.t_half) return;
                if (far2 <= g.t_half) {
                    half += qe - qb;
                    return;
                }
                for (int q = qb; q < qe; q++) {
                    float d2 = 0.f;
#pragma unroll U
                    for (int l = 0; l < LM; l++) {
                        if (!EX && l >= d) break;
                        d2 = dist_step(__ldg(w.X + (size_t)l * g.ns + q), x[l], d2);
                    }
                    half += d2 <= g.t_half;
                }
            });
            viol = N != own_cnt + __reduce_add_sync(0xffffffffu, half);
            EGG_WSTAT(kUsHalfCount, lane == 0);
        }
        any_viol |= viol;
        if (lane == 0) {
            if (counts) counts[i] = N;
            w.viol_orig[w.orig[i]] = viol ? 1 : 0;
            if (words && viol) atomicOr(w.warp_viol + (i >> 5), 1u << (i & 31));
            if (moved) {
                unsigned long long* dcur = w.dirty[it & 1];
                const int zb = g.od < d ? w.cell_dims[(size_t)g.od * g.ns + own] / g.zblk : 0;
                atomicOr(dcur + w.cell_outer[own], 1ull << zb);
                atomicOr(dcur + onew, 1ull << zbnew);
                w.warp_moved[i >> 5] = 1;  // cleared by this iteration's cell-sums kernels
            }
        }
        __syncwarp();
#ifdef EGG_UPDATE_STATS
        if (lane == 0) {
            st[kUsPoints] += 1;
            st[kUsNeighbors] += N;
        }
        for (int k = 0; k < kUStats; k++) {
            const unsigned v = __reduce_add_sync(0xffffffffu, st[k]);
            if (lane == 0 && v) atomicAdd(w.ustats + k, (unsigned long long)v);
        }
#endif
    }
    return any_viol;
}

// The update of the block's points, a warp per point that needs one.  The
// block settles `per` points (at most its threads): kept points as they are,
// the others go on a list that its warps share out.  Points come in runs of
// eight (a sector of every array) taken from all over the storage order,
// because those that still move sit together: late in a run the few hundred
// of them spread over as many blocks.
template <int DM, bool EX, int KB>
__device__ __forceinline__ void update_points_body(const Geom& g, const Work& w, int* __restrict__ counts, int per,
                                                   int bx, int gx) {
    using R = CellReader<DM, EX, KB>;
    constexpr int LM = R::LM;
    const int d = EX ? DM : g.d;
    extern __shared__ float4 s_tab[];  // sin, cos, 1 - cos of k * side; then each warp's area
    __shared__ int s_list[256];
    __shared__ int s_count;
    const int TW = 2 * g.table_k + 1;
    for (int t = threadIdx.x; t < TW; t += blockDim.x)
        s_tab[t] = make_float4(w.table[t], w.table[TW + t], w.table[2 * TW + t], 0.f);
    const int lane = threadIdx.x & 31;
    float* const area = reinterpret_cast<float*>(s_tab + TW) + (threadIdx.x >> 5) * walk_floats(LM);
    if (threadIdx.x == 0) {
        s_count = 0;
        if (bx == 0) w.stamps[4 * w.ctrl[kCtrlIter] + 1] = globaltimer();
    }
    __syncthreads();
    const int idx = threadIdx.x;
    const int iv = per < 8 ? bx * per + idx : (((idx >> 3) * gx + bx) << 3) + (idx & 7);
    bool any_viol = false;
    if (idx < per && iv < g.n) {
        const int c = w.cell_of[iv];
        const int zb = g.od < d ? w.cell_dims[(size_t)g.od * g.ns + c] / g.zblk : 0;
        if (counts != nullptr || w.ctrl[kCtrlForce] != 0 || ((w.need[w.cell_outer[c]] >> zb) & 1ull) != 0) {
            s_list[atomicAdd(&s_count, 1)] = iv;
        } else {
            // no moved point in its stencil region: it keeps its position and
            // its violation bit (bit-identical to recomputing)
            if (w.ctrl[kCtrlChanged] != 0)
                for (int l = 0; l < d; l++) w.Xn[(size_t)l * g.ns + iv] = w.X[(size_t)l * g.ns + iv];
            any_viol = w.viol_orig[w.orig[iv]] != 0;
        }
    }
    __syncthreads();
    const int todo = s_count;
    if (threadIdx.x == 0 && todo) atomicAdd(w.ctrl + kCtrlComputed, todo);
    any_viol |= update_listed_points<DM, EX, KB>(g, w, counts, s_tab, area, s_list, todo, false);
    if (__any_sync(0xffffffffu, any_viol) && lane == 0) {
        volatile int* f = w.ctrl + kCtrlFlag;
        if (*f != 0) *f = 0;
    }
}

}  // namespace egg
