// me_full_resolve.cu -- prediction-dependent tail of MotionEstimatorH264ImplFull.
//
// After the search every macroblock has its prediction-independent results
// (sub-pel vector and distortion, zero-vector distortion).  What is left is a
// function of the median prediction (Full.cpp:368-380 rounding, 401-446 tie
// rescan, 532-590 prediction distortion and GetBestVector), and the
// prediction depends on the left / above / above-right (else above-left)
// neighbours' final vectors: a DAG in raster order.
//
// The estimators whose evaluation is short (all but Ver2's Lagrangian
// overload) relax from the searched vectors to the fixed point, which is the
// sequential result: k_resolve_first, k_resolve_sweep, k_resolve_finish below.
//
// The Lagrangian overload, whose evaluation is a whole search, keeps every
// evaluation as a record {prediction, distortion at it, final vector, final
// distortion} in a small per-MB cache, so that a later visit with the same
// prediction is a lookup:
//
//   k_full_sweep0      every MB at once, prediction from the current vectors
//                      (initially the searched ones).
//   k_full_relax_sweep up to FullArgs::relax_sweeps launches, each re-evaluating the
//                      MBs whose prediction moved.  A sweep without change
//                      is the fixed point (k_full_relax_outcome writes the
//                      outputs).  Otherwise (long copy chains: the prediction
//                      wins and is copied along rows and columns)
//                      k_full_relax_outcome builds a dictionary of the frame's
//                      dominant vectors.
//   k_full_precompute, k_full_closure  records of every MB at every dictionary
//                      vector and at medians of its neighbours' possible vectors.
//   k_full_wave        one CTA replays the exact sequential order, pipelined
//                      by rows (below).
#include <cooperative_groups.h>

#include "me_cross_search.cuh"
#include "me_full_common.cuh"
#include "me_mrc_search.cuh"

namespace vppgpu {
namespace {
using namespace full;

constexpr int kEmpty = 0x7fffffff;  // no vector packs to this (|y| < 32767 quarter pels)
constexpr int kCacheRelax = 1;      // entries 1..3 round robin in relaxation
constexpr int kCacheDict = 4;       // entries 4..11 dictionary
constexpr int kCacheClosure = 12;   // entries 12..31 neighbour closure
constexpr int kSetMax = 6;          // possible final vectors kept per neighbour

__device__ __forceinline__ int4 empty_record() { return make_int4(kEmpty, 0, 0, 0); }

// Walk a tie tree held one word per lane (t0: words 0..31, t1: 32..): the
// outcome of the scan for rounded prediction (prx, pry).
__device__ __forceinline__ void tree_pick(int t0, int t1, int prx, int pry, int* mvx, int* mvy, int* minD)
{
    constexpr int RW = sizeof(TieRun) / sizeof(int);
    auto get = [&](int idx) {
        const int v0 = __shfl_sync(0xffffffffu, t0, idx & 31), v1 = __shfl_sync(0xffffffffu, t1, idx & 31);
        return idx < 32 ? v0 : v1;
    };
    int path = 0;
    for (int e = 0; e < TIE_DEPTH; e++) {
        if (e >= get(path * RW + TIE_DEPTH)) break;
        const int g = get(path * RW + e);
        const int cx = (int)(signed char)(g & 0xff) - prx, cy = (int)(signed char)((g >> 8) & 0xff) - pry;
        const int nx = (int)(signed char)((g >> 16) & 0xff) - prx, ny = (int)(signed char)((g >> 24) & 0xff) - pry;
        if ((cy * cy + cx * cx) - (ny * ny + nx * nx) >= 0) path |= 1 << e;
    }
    const int q = get(path * RW + TIE_DEPTH + 1);
    *mvx = mv_x(q);
    *mvy = mv_y(q);
    *minD = get(path * RW + TIE_DEPTH + 2);
}

// Exact-tie macroblocks: the integer scan depends on the rounded prediction.
// Walk the tie tree the search kernel kept (one load per lane), or, for the
// rare macroblock with more ties than the tree holds, replay the scan from
// the kept table and redo the sub-pel stage if the full-pel winner moved.
// Kept out of line.
__device__ __noinline__ void tie_path(const FullArgs& a, int k, int px, int py, int flags, int lane, int* mvx,
                                      int* mvy, int* minD)
{
    int prx = round_pred(px), pry = round_pred(py);
    if (prx == 0 && pry == 0) return;  // the search kernel already decided ties with (0,0)
    const int* tab = a.tables + (size_t)k * TAB * TAB;
    if (!(flags & FLAG_DEEP)) {
        constexpr int TW = TIE_RUNS * (int)(sizeof(TieRun) / sizeof(int));
        const int* tree = tab + TIE_ROW * TAB;
        const int t0 = __ldcg(tree + lane);
        const int t1 = lane < TW - 32 ? __ldcg(tree + 32 + lane) : 0;
        tree_pick(t0, t1, prx, pry, mvx, mvy, minD);
        return;
    }
    const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
    int xl, xr, yu, yd, mx, my, md, tie;
    full_range(n, m, a.W, a.H, a.motion_range, xl, xr, yu, yd);
    scan_table(GlobalTab{tab}, xl, xr, yu, yd, prx, pry, lane, &mx, &my, &md, &tie);
    int imv = a.spec_imv[k];
    if (mx != mv_x(imv) || my != mv_y(imv)) {
        if (a.intpel) {  // the integer-pel stage ends at the full-pel winner
            *mvx = 4 * mx;
            *mvy = 4 * my;
            *minD = md;
            return;
        }
        int qmx, qmy;
        subpel_refine_planes(a, n + mx, m + my, load_cur8(a, n, m, lane), lane, &md, &qmx, &qmy);
        *mvx = 4 * mx + qmx;
        *mvy = 4 * my + qmy;
        *minD = md;
    }
}

// Warp-level record lookup: lanes 0..KCACHE-1 each hold one record.
__device__ __forceinline__ bool cache_probe(const int4* c, int key, int lane, int4* rec)
{
    int4 e = lane < KCACHE ? __ldcg(c + lane) : empty_record();
    unsigned hit = __ballot_sync(0xffffffffu, e.x == key);
    if (!hit) return false;
    const int f = __ffs(hit) - 1;
    rec->x = key;
    rec->y = __shfl_sync(0xffffffffu, e.y, f);
    rec->z = __shfl_sync(0xffffffffu, e.z, f);
    rec->w = __shfl_sync(0xffffffffu, e.w, f);
    return true;
}

// The predictor multi-resolution estimators (kEst 1 Ver2, 2 Multires): the
// searched vector and distortion of tie MB k at prediction (px, py): from its
// tie tree, else a kept search whose tie decisions agree, else a new search
// (kept in slots 1..3; slot 0 holds the search at prediction (0, 0)).  One warp.
template <int kEst>
__device__ __noinline__ void pred_search_at(const FullArgs& a, int k, int px, int py, int lane, int* mvx, int* mvy,
                                            int* minD, mrc::Lattice* lt)
{
    if constexpr (kEst == cross::EST_CROSS) {
        // Cross: the tie tree, else a search at the rounded prediction (the
        // only way the prediction enters, MotionEstimatorH264ImplCross.cpp:393-405),
        // cached by it
        int tv, td;
        if (mrc::tie_tree_result(cross::EST_CROSS, static_cast<const mrc::V2TieRun*>(a.tie_runs) +
                                                       (size_t)k * mrc::V2_TIE_RUNS,
                                 px, py, lane, &tv, &td)) {
            *mvx = mv_x(tv);
            *mvy = mv_y(tv);
            *minD = td;
            return;
        }
        const int key = pack_mv(round_pred(px), round_pred(py));
        int4* sc = a.search_cache + (size_t)k * V2_SEARCH_CACHE;
        const int4 e = lane < V2_SEARCH_CACHE ? __ldcg(sc + lane) : make_int4(0, 0, 0, -1);
        const unsigned hit = __ballot_sync(0xffffffffu, e.w >= 0 && e.x == key);
        if (hit) {
            const int f = __ffs(hit) - 1;
            const int v = __shfl_sync(0xffffffffu, e.y, f);
            *mvx = mv_x(v);
            *mvy = mv_y(v);
            *minD = __shfl_sync(0xffffffffu, e.z, f);
            return;
        }
        const cross::CrossResult r =
            cross::cross_search(a, (k % a.cols) * 16, (k / a.cols) * 16, round_pred(px), round_pred(py), lane);
        *mvx = r.mvx;
        *mvy = r.mvy;
        *minD = r.min_d;
        const unsigned slot = 1 + ((unsigned)key * 2654435761u >> 30) % (V2_SEARCH_CACHE - 1);
        if (lane == 0) __stcg(sc + slot, make_int4(key, pack_mv(r.mvx, r.mvy), r.min_d, 1));
        __syncwarp();
        return;
    }
    int tv, td;
    // the Lagrangian overload's search depends on the whole prediction: no tie tree, kept searches by
    // their exact prediction
    if (kEst != mrc::EST_V2_LAMBDA &&
        mrc::tie_tree_result(kEst, static_cast<const mrc::V2TieRun*>(a.tie_runs) + (size_t)k * mrc::V2_TIE_RUNS, px,
                             py, lane, &tv, &td)) {
        *mvx = mv_x(tv);
        *mvy = mv_y(tv);
        *minD = td;
        return;
    }
    int4* sc = a.search_cache + (size_t)k * V2_SEARCH_CACHE;
    const int4 e = lane < V2_SEARCH_CACHE ? __ldcg(sc + lane) : make_int4(0, 0, 0, -1);
    const unsigned hit = __ballot_sync(0xffffffffu, e.w >= 0 && (kEst == mrc::EST_V2_LAMBDA
                                                                     ? e.x == pack_mv(px, py)
                                                                     : mrc::search_reusable(kEst, e.w, mv_x(e.x),
                                                                                            mv_y(e.x), px, py)));
    if (hit) {
        const int f = __ffs(hit) - 1;
        const int v = __shfl_sync(0xffffffffu, e.y, f);
        *mvx = mv_x(v);
        *mvy = mv_y(v);
        *minD = __shfl_sync(0xffffffffu, e.z, f);
        return;
    }
    bool bad = false;
    const mrc::MrcArgs& m = *static_cast<const mrc::MrcArgs*>(a.mrc);
    mrc::Lattice& LT = lt ? *lt : static_cast<mrc::Lattice*>(a.lattice)[k];
    const mrc::MbSearch r = mrc::search_pred<kEst>(m, LT, k / a.cols, k % a.cols, px, py, lane, bad);
    if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&a.ctrl->status, ST_OUT_OF_BOUNDS);
    *mvx = r.mvx;
    *mvy = r.mvy;
    *minD = r.min_d;
    const unsigned slot = 1 + ((unsigned)pack_mv(px, py) * 2654435761u >> 30) % (V2_SEARCH_CACHE - 1);
    if (lane == 0) __stcg(sc + slot, make_int4(pack_mv(px, py), pack_mv(r.mvx, r.mvy), r.min_d, r.tie));
    __syncwarp();
}

// Per-warp shared sub-pel lattices for the predictor estimators' searches at
// a prediction (8 warps per block); none for the full-search estimator.  The
// wavefront, which evaluates rarely, uses the per-MB scratch in global memory.
template <int kEst>
struct LatticeSlots {
    __device__ static mrc::Lattice* get(int warp)
    {
        __shared__ mrc::Lattice slots[8];
        return &slots[warp];
    }
};
template <>
struct LatticeSlots<0> {
    __device__ static mrc::Lattice* get(int) { return nullptr; }
};
template <>
struct LatticeSlots<6> {  // the SAD stage
    __device__ static mrc::Lattice* get(int) { return nullptr; }
};
template <>
struct LatticeSlots<cross::EST_CROSS> {
    __device__ static mrc::Lattice* get(int) { return nullptr; }
};

// Full evaluation of MB k by Ver2's Lagrangian overload (…MultiresCrossVer2.cpp:1162-1742) for raw prediction
// (px, py), one warp: the record {prediction, distortion at it, final vector, final distortion}.  Every MB is searched
// at its prediction (mrc::search_lambda); the final choice with the caller's lambda.
__device__ __noinline__ int4 evaluate(const FullArgs& a, int k, int px, int py, int lane, mrc::Lattice* lt = nullptr)
{
    const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
    const PredGeom g = pred_geom(n, m, a.W, a.H, px, py);
    const int4 sp = a.spec4[k];  // loads of spec and planes are independent: one round trip
    const int pd = plane_pred_distortion(a, n, m, g, lane);
    int mvx = mv_x(sp.x), mvy = mv_y(sp.x), minD = sp.y;
    const int zd = sp.z;
    if (sp.w & FLAG_TIE) pred_search_at<mrc::EST_V2_LAMBDA>(a, k, px, py, lane, &mvx, &mvy, &minD, lt);
    const int pos = best_of3_fast(mvx, mvy, minD, g.pcx, g.pcy, pd, zd, a.lambda, g.pcx, g.pcy);
    int4 rec;
    rec.x = pack_mv(px, py);
    rec.y = pd;
    if (pos == 0) {
        rec.z = pack_mv(mvx, mvy);
        rec.w = minD;
    } else if (pos == 1) {
        rec.z = pack_mv(g.pcx, g.pcy);
        rec.w = pd;
    } else {
        rec.z = pack_mv(0, 0);
        rec.w = zd;
    }
    return rec;
}

// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 4) k_full_sweep0(FullArgs a)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int k = blockIdx.x * 8 + wib;
    if (k >= a.nmb) return;
    int px, py;
    median_pred(a.final_mv, a.spec4[k].w, k, a.cols, &px, &py);
    const int4 rec = evaluate(a, k, px, py, lane, LatticeSlots<mrc::EST_V2_LAMBDA>::get(wib));
    if (lane < KCACHE) __stcg(a.cache + (size_t)k * KCACHE + lane, lane == 0 ? rec : empty_record());
    if (lane == 0) {
        a.pred_used[k] = rec.x;
        a.final_dist[k] = rec.w;
        __stcg(a.final_mv + k, rec.z);
    }
}

// ---------------------------------------------------------------------------
// State of the relaxation before sweep `upto` from the change counts of sweeps
// 1 .. upto-1: s > 0 when sweep s changed nothing (the fixed point), -1 when
// more than a few MBs still change and the counts stopped falling fast enough
// to reach zero within `limit` sweeps (they fall about geometrically while
// copy chains shorten; a ratio above 7/8, or a projection past the limit,
// gives up to the wavefront), 0 while
// the sweeps go on.  The sweep kernels and the outcome kernel evaluate the
// same counts with this one function, so they agree.
__device__ __forceinline__ int relax_status(const int* changed, int upto, int limit)
{
    int prev = 0;
    for (int s = 1; s < upto; s++) {
        const int c = *((const volatile int*)&changed[s]);
        if (c == 0) return s;
        if (s >= 3 && c > 32) {  // a few changes settle within a sweep or two: never give up on them
            const float r = (float)c / (float)prev;
            if (r >= 0.875f) return -1;
            if ((float)s + logf((float)c + 1.0f) / -logf(r) > (float)limit + 1.0f) return -1;
        }
        prev = c;
    }
    return 0;
}

constexpr int kHist = 4096;  // dictionary histogram slots
struct RelaxSmem {
    union {
        struct {
            int keys[kHist];
            int counts[kHist];
        } hist;
    } u;
    long long red_total[8];
    int red_count[8];
    int red_key[8];
    int red_val[8];
};

// One relaxation sweep: lane per MB (MBs gwarp + lane*nwarps ...) to find the
// MBs whose prediction moved, then the warp on each.  Skipped once an earlier
// sweep changed no vector (the fixed point is reached).
__global__ void __launch_bounds__(256, 4) k_full_relax_sweep(FullArgs a, int sweep)
{
    if (relax_status(a.changed, sweep, a.relax_sweeps) != 0) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gwarp = blockIdx.x * 8 + wib, nwarps = gridDim.x * 8;
    int changed = 0;
    for (int base = gwarp; base < a.nmb; base += 32 * nwarps) {
        const int k = base + lane * nwarps;
        int px = 0, py = 0, key = 0;
        bool moved = false;
        if (k < a.nmb) {
            median_pred(a.final_mv, __ldcg(&a.spec4[k].w), k, a.cols, &px, &py);
            key = pack_mv(px, py);
            moved = __ldcg(a.pred_used + k) != key;
        }
        unsigned todo = __ballot_sync(0xffffffffu, moved);
        while (todo) {
            const int f = __ffs(todo) - 1;
            todo &= todo - 1;
            const int kk = base + f * nwarps, fkey = __shfl_sync(0xffffffffu, key, f);
            const int fx = __shfl_sync(0xffffffffu, px, f), fy = __shfl_sync(0xffffffffu, py, f);
            int4* cache = a.cache + (size_t)kk * KCACHE;
            int4 rec;
            const bool hit = cache_probe(cache, fkey, lane, &rec);
            if (!hit) rec = evaluate(a, kk, fx, fy, lane, LatticeSlots<mrc::EST_V2_LAMBDA>::get(wib));
            if (lane == 0) {
                atomicAdd(&a.ctrl->relax_evals, 1);
                if (!hit) {
                    atomicAdd(&a.ctrl->relax_miss, 1);
                    __stcg(cache + kCacheRelax + (sweep % 3), rec);
                }
                __stcg(a.pred_used + kk, fkey);
                a.final_dist[kk] = rec.w;
                if (__ldcg(a.final_mv + kk) != rec.z) {
                    __stcg(a.final_mv + kk, rec.z);
                    changed++;
                }
            }
            __syncwarp();
        }
    }
    if (lane == 0 && changed) atomicAdd(&a.changed[sweep], changed);
}

// After the sweeps: a sweep that changed nothing means the vectors are the
// sequential result -- every block writes its MBs' outputs and adds their
// included distortions; otherwise block 0 finds the frame's dominant vectors
// for the wavefront's records.
__global__ void __launch_bounds__(256) k_full_relax_outcome(FullArgs a)
{
    __shared__ RelaxSmem S;
    const int status = relax_status(a.changed, a.relax_sweeps + 1, a.relax_sweeps);
    const int sweeps = status > 0 ? status : 0;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (sweeps) {
        long long tot = 0;
        int cnt = 0;
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.nmb; k += gridDim.x * blockDim.x) {
            const int fmv = __ldcg(a.final_mv + k);
            a.job->out_mv[k] = fmv;
            const int d = a.final_dist[k];
            if (a.job->out_dist) a.job->out_dist[k] = d;
            if (a.job->incl && a.job->incl[k]) {
                tot += d;
                cnt++;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
            cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
        }
        if (lane == 0 && cnt) {
            atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->total), (unsigned long long)tot);
            atomicAdd(&a.ctrl->count, cnt);
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.ctrl->sweeps = sweeps;
            a.ctrl->converged = 1;
        }
        return;
    }
    if (blockIdx.x != 0) return;
    for (int i = threadIdx.x; i < kHist; i += blockDim.x) {
        S.u.hist.keys[i] = kEmpty;
        S.u.hist.counts[i] = 0;
    }
    __syncthreads();
    for (int base = 0; base < a.nmb; base += 8 * blockDim.x) {  // uniform trip count: every lane shuffles
        const int k0 = base + threadIdx.x;
        int vals[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {  // eight loads in flight per thread
            const int k = k0 + u * blockDim.x;
            vals[u] = k < a.nmb ? __ldcg(a.final_mv + k) : kEmpty;
        }
#pragma unroll
        for (int u = 0; u < 8; u++) {
            // one insert per distinct vector of the warp (a pan makes most vectors equal:
            // per-lane atomics on one slot would serialise)
            const int v = vals[u];
            const unsigned same = __match_any_sync(0xffffffffu, v);
            if (v == kEmpty || (__ffs(same) - 1) != (int)(threadIdx.x & 31)) continue;
            // counts only steer which records are precomputed: a vector that finds
            // no slot within a few probes (frames with thousands of distinct
            // vectors) is left out
            unsigned h = ((unsigned)v * 2654435761u) >> 20;  // 12 bits
            for (int probe = 0; probe < 8; probe++) {
                int slot = (h + probe) & (kHist - 1);
                int prev = atomicCAS(&S.u.hist.keys[slot], kEmpty, v);
                if (prev == kEmpty || prev == v) {
                    atomicAdd(&S.u.hist.counts[slot], __popc(same));
                    break;
                }
            }
        }
    }
    __syncthreads();
    for (int d = 0; d < NDICT; d++) {
        int best_c = 0, best_k = kEmpty;
        for (int i = threadIdx.x; i < kHist; i += blockDim.x)
            if (S.u.hist.counts[i] > best_c) {
                best_c = S.u.hist.counts[i];
                best_k = i;
            }
        for (int o = 16; o > 0; o >>= 1) {
            int oc = __shfl_xor_sync(0xffffffffu, best_c, o), ok2 = __shfl_xor_sync(0xffffffffu, best_k, o);
            if (oc > best_c || (oc == best_c && ok2 < best_k)) {
                best_c = oc;
                best_k = ok2;
            }
        }
        if (lane == 0) {
            S.red_val[wib] = best_c;
            S.red_key[wib] = best_k;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int bc = 0, bk = kEmpty;
            for (int w = 0; w < 8; w++)
                if (S.red_val[w] > bc || (S.red_val[w] == bc && S.red_key[w] < bk)) {
                    bc = S.red_val[w];
                    bk = S.red_key[w];
                }
            a.dict[d] = bc > 0 ? S.u.hist.keys[bk] : kEmpty;
            if (bc > 0) S.u.hist.counts[bk] = 0;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) a.ctrl->sweeps = a.relax_sweeps;
}

// ---------------------------------------------------------------------------
// One warp per MB: records at every dictionary vector the MB's cache lacks.
__global__ void __launch_bounds__(256, 2) k_full_precompute(FullArgs a)
{
    if (*((volatile int*)&a.ctrl->converged)) return;
    __shared__ int dict[NDICT];
    if (threadIdx.x < NDICT) dict[threadIdx.x] = a.dict[threadIdx.x];
    __syncthreads();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int k = blockIdx.x * 8 + wib; k < a.nmb; k += gridDim.x * 8) {
        int4* cache = a.cache + (size_t)k * KCACHE;
        const int4 mine = __ldcg(cache + lane);
        for (int d = 0; d < NDICT; d++) {
            const int v = dict[d];
            if (v == kEmpty || __any_sync(0xffffffffu, mine.x == v)) continue;
            const int4 rec = evaluate(a, k, mv_x(v), mv_y(v), lane, LatticeSlots<mrc::EST_V2_LAMBDA>::get(wib));
            if (lane == 0) __stcg(cache + kCacheDict + d, rec);
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------------------
// Neighbour closure, one warp per MB.  The prediction of MB k is the median
// of the final vectors of A, B and C (or D); each of those is one of a few
// values: its current vector, its searched vector, zero, or the outcome of
// one of its records.  Medians of those per-neighbour sets, taken in order of
// plausibility (index sum), that MB k has no record for yet become records
// 12..31, evaluated here.  Then MB k's wavefront record is written.
// Wavefront record hashing: a prediction whose halves fit in signed 11 bits
// encodes to 22 bits; two distinct buckets of 4 per encoding.
__device__ __forceinline__ bool wave_encode(int key, unsigned* e)
{
    const int x = mv_x(key), y = mv_y(key);
    *e = (unsigned)(x & 0x7ff) | ((unsigned)(y & 0x7ff) << 11);
    return (unsigned)(x + 1024) < 2048u && (unsigned)(y + 1024) < 2048u;
}
__device__ __forceinline__ void wave_buckets(unsigned e, int* h1, int* h2)
{
    *h1 = (int)((e * 0x9e3779b1u) >> 28);
    *h2 = *h1 ^ (1 + (int)((e * 0xc2b2ae3du) >> 29));  // differs from h1
}

// Index triples (ia, ib, ic) < kSetMax^3 by index sum, then lexicographic,
// packed as ia | ib << 3 | ic << 6.
constexpr int kCombos = kSetMax * kSetMax * kSetMax;
struct ClosureOrder {
    short v[kCombos];
};
constexpr ClosureOrder make_closure_order()
{
    ClosureOrder o{};
    int n = 0;
    for (int sum = 0; sum <= 3 * (kSetMax - 1); sum++)
        for (int ia = 0; ia < kSetMax; ia++)
            for (int ib = 0; ib < kSetMax; ib++) {
                const int ic = sum - ia - ib;
                if (ic >= 0 && ic < kSetMax) o.v[n++] = (short)(ia | (ib << 3) | (ic << 6));
            }
    return o;
}
__constant__ const ClosureOrder kClosureOrder = make_closure_order();

struct ClosureSmem {
    unsigned tab[8][64];
    int cnt[8][16];
    int set[8][3][kSetMax];
    int nset[8][3];
    int fresh[8][KCACHE - kCacheClosure];
};

// Ordered, de-duplicated possible final vectors of MB x into set[0..n).
__device__ __forceinline__ int neighbour_set(const FullArgs& a, int x, int lane, int* set)
{
    int v = kEmpty;
    if (lane == 0) v = __ldcg(a.final_mv + x);
    else if (lane == 1) v = __ldcg(&a.spec4[x].x);
    else if (lane == 2) v = 0;
    else if (lane < 3 + kCacheClosure) {
        const int4 r = __ldcg(a.cache + (size_t)x * KCACHE + (lane - 3));
        if (r.x != kEmpty) v = r.z;
    }
    const bool valid = v != kEmpty;
    const unsigned vm = __ballot_sync(0xffffffffu, valid);
    const unsigned same = __match_any_sync(0xffffffffu, v);
    const bool keep = valid && (__ffs(same) - 1) == lane;
    const unsigned km = __ballot_sync(0xffffffffu, keep);
    const int rank = __popc(km & ((1u << lane) - 1u));
    if (keep && rank < kSetMax) set[rank] = v;
    (void)vm;
    __syncwarp();
    return min(__popc(km), kSetMax);
}

__global__ void __launch_bounds__(256, 2) k_full_closure(FullArgs a)
{
    if (*((volatile int*)&a.ctrl->converged)) return;
    __shared__ ClosureSmem S;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int cols = a.cols, rows = a.nmb / cols;
    for (int k = blockIdx.x * 8 + wib; k < a.nmb; k += gridDim.x * 8) {
        int4* cache = a.cache + (size_t)k * KCACHE;
        int4 mine = __ldcg(cache + lane);
        const int av = __ldcg(&a.spec4[k].w);
        // neighbour sets (an unavailable neighbour contributes zero, as in the median)
        const int r = k / cols, c = k - r * cols;
        (void)rows;
        const int nb[3] = {(av & AV_A) ? k - 1 : -1, (av & AV_B) ? k - cols : -1,
                           (av & AV_C) ? k - cols + 1 : ((av & AV_D) ? k - cols - 1 : -1)};
        for (int s = 0; s < 3; s++) {
            if (nb[s] >= 0) {
                const int n = neighbour_set(a, nb[s], lane, S.set[wib][s]);
                if (lane == 0) S.nset[wib][s] = n;
            } else if (lane == 0) {
                S.set[wib][s][0] = 0;
                S.nset[wib][s] = 1;
            }
        }
        __syncwarp();
        if (!(av & AV_B) && !(av & AV_C)) {
            // neither above nor above-right: B and C take A (median_from)
            for (int i = lane; i < kSetMax; i += 32) S.set[wib][1][i] = S.set[wib][2][i] = S.set[wib][0][i];
            if (lane == 0) S.nset[wib][1] = S.nset[wib][2] = S.nset[wib][0];
            __syncwarp();
        }
        const int nA = S.nset[wib][0], nB = S.nset[wib][1], nC = S.nset[wib][2];
        // combinations by index sum, 32 at a time
        int fresh = 0;
        for (int base = 0; base < kCombos && fresh < KCACHE - kCacheClosure; base += 32) {
            const int idx = base + lane;
            int ia = 0, ib = 0, ic = 0;
            bool ok = false;
            if (idx < kCombos) {
                const int code = kClosureOrder.v[idx];
                ia = code & 7;
                ib = (code >> 3) & 7;
                ic = (code >> 6) & 7;
                ok = ia < nA && ib < nB && ic < nC;
            }
            if (!__any_sync(0xffffffffu, ok)) continue;
            int key = kEmpty;
            if (ok) {
                const int A = S.set[wib][0][ia], B = S.set[wib][1][ib], C = S.set[wib][2][ic];
                key = pack_mv(median3(mv_x(A), mv_x(B), mv_x(C)), median3(mv_y(A), mv_y(B), mv_y(C)));
            }
            // new: not among the MB's records (including those added so far), first of its kind in the batch
            bool dup = !ok;
            for (int e = 0; e < KCACHE; e++) dup |= __shfl_sync(0xffffffffu, mine.x, e) == key;
            const unsigned same = __match_any_sync(0xffffffffu, key);
            const bool take = !dup && (__ffs(same) - 1) == lane;
            const unsigned tm = __ballot_sync(0xffffffffu, take);
            const int slot = fresh + __popc(tm & ((1u << lane) - 1u));
            if (take && slot < KCACHE - kCacheClosure) S.fresh[wib][slot] = key;
            __syncwarp();
            const int added = min(__popc(tm), KCACHE - kCacheClosure - fresh);
            if (lane >= kCacheClosure + fresh && lane < kCacheClosure + fresh + added)
                mine.x = S.fresh[wib][lane - kCacheClosure];
            fresh += added;
            __syncwarp();
        }
        // evaluate the new records
        for (int i = 0; i < fresh; i++) {
            const int key = S.fresh[wib][i];
            const int4 rec = evaluate(a, k, mv_x(key), mv_y(key), lane, LatticeSlots<mrc::EST_V2_LAMBDA>::get(wib));
            if (lane == kCacheClosure + i) mine = rec;
        }
        if (lane >= kCacheClosure) {
            if (lane < kCacheClosure + fresh) __stcg(cache + lane, mine);
        }
        // the wavefront record: entries hashed into 16 buckets of 4, each to
        // the emptier of its two buckets, in slot order (a record that does not
        // fit, or whose outcome is a clamped prediction, is left out: the
        // wavefront then evaluates that prediction itself)
        const int spec = __ldcg(&a.spec4[k].x);
        unsigned entry = 0xffffffffu;
        int h1 = 0, h2 = 0;
        if (mine.x != kEmpty) {
            const int code = mine.z == spec ? 0 : (mine.z == mine.x ? 1 : (mine.z == 0 ? 2 : 3));
            unsigned e;
            if (code < 3 && wave_encode(mine.x, &e)) {
                entry = e | ((unsigned)code << 22);
                wave_buckets(e, &h1, &h2);
            }
        }
        unsigned* tab = S.tab[wib];
        int* cnt = S.cnt[wib];
        tab[lane] = 0xffffffffu;
        tab[lane + 32] = 0xffffffffu;
        if (lane < 16) cnt[lane] = 0;
        __syncwarp();
        for (int i = 0; i < 32; i++) {
            if (lane == i && entry != 0xffffffffu) {
                const int c1 = cnt[h1], c2 = cnt[h2];
                const int b = c1 <= c2 ? h1 : h2, cb = c1 <= c2 ? c1 : c2;
                if (cb < 4) {
                    tab[4 * b + cb] = entry;
                    cnt[b] = cb + 1;
                }
            }
            __syncwarp();
        }
        WaveRec* wr = a.wave_rec + wave_rec_index(cols, r, c);
        reinterpret_cast<uint2*>(wr->slot)[lane] = make_uint2(tab[2 * lane], tab[2 * lane + 1]);
        if (lane == 0) {
            wr->spec = spec;
            wr->av = av;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Exact order, one CTA per group of up to WAVE_WARPS bands of 32 rows.
// Lane l of warp w owns row 32(band0+w) + l and handles column t - 2l at step
// t: its left neighbour is its own previous output, above / above-right /
// above-left are lane l-1's outputs of steps t-2, t-1 and t-3 (shuffles), so
// a warp advances 32 rows in lock step with no synchronisation.  Lane 0 takes
// the row above from warp w-1's lane 31 through shared memory, where each
// vector is its own flag (the array starts as kEmpty, which no vector packs
// to), or, for the first band of a launch, from the vectors the previous
// launch stored.  The 32 wavefront records of a step are contiguous (diagonal
// layout) and arrive by one bulk copy, kRing-1 steps ahead.  A step is a
// median, 32 key compares and, only for a lane whose prediction is in none of
// its records, a full evaluation by the whole warp.
constexpr int kWaveMaxWarps = WAVE_WARPS;
constexpr unsigned kWaveStepBytes = 32 * sizeof(WaveRec);

template <int kChunk>
__global__ void __launch_bounds__(kWaveMaxWarps * 32, 1) k_full_wave(FullArgs a, int band0, int last)
{
    if (*((volatile int*)&a.ctrl->converged)) return;
    extern __shared__ __align__(16) unsigned char wave_smem[];
    const int cols = a.cols, rows = a.nmb / a.cols, nw = blockDim.x >> 5;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // per warp: two buffers of kChunk steps (32 records a step), a barrier each
    WaveRec* ring = reinterpret_cast<WaveRec*>(wave_smem);                                // [nw][2][kChunk][32]
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(ring + nw * 2 * kChunk * 32);  // [nw][2]
    volatile int* edge = reinterpret_cast<int*>(bars + nw * 2);                           // [nw][cols]
    __shared__ int abort_flag;
    for (int i = threadIdx.x; i < nw * cols; i += blockDim.x) edge[i] = kEmpty;
    if (threadIdx.x < nw * 2) mbar_init(bars + threadIdx.x, 1);
    if (threadIdx.x == 0) abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    __syncthreads();

    const int band = band0 + w;
    const int r = 32 * band + lane;
    const bool row_ok = r < rows;
    const int lanes_used = min(32, rows - 32 * band);
    const int nsteps = cols + 2 * (lanes_used - 1);
    const int nchunks = (nsteps + kChunk - 1) / kChunk;
    const WaveRec* src = a.wave_rec + (size_t)band * (cols + 62) * 32;  // step t: src[32t .. 32t+31]
    WaveRec* mybuf = ring + w * 2 * kChunk * 32;
    unsigned long long* mybars = bars + w * 2;
    const volatile int* above = edge + (w - 1) * cols;                 // lane 0 of warps > 0
    const int* above_g = a.final_mv + (size_t)(32 * band - 1) * cols;  // lane 0 of warp 0 when band0 > 0

    auto issue = [&](int ci) {  // chunk ci into buffer ci & 1 (lane 0)
        const int steps = min(kChunk, nsteps - ci * kChunk);
        const unsigned bytes = (unsigned)steps * kWaveStepBytes;
        mbar_expect_tx(mybars + (ci & 1), bytes);
        bulk_load(mybuf + (ci & 1) * kChunk * 32, src + (size_t)ci * kChunk * 32, bytes, mybars + (ci & 1));
    };
    if (lane == 0) {
        issue(0);
        if (nchunks > 1) issue(1);
    }
    int issued = min(2, nchunks), consumed = 0;  // chunks of this warp
    // o1: this lane's output of step t-1 (its left neighbour at step t); s1, s2, s3: lane l-1's outputs of
    // steps t-1, t-2, t-3 (above-right, above, above-left at step t), received one shuffle per step
    int o1 = 0, s1 = 0, s2 = 0, s3 = 0;
    int pb = 0, pc = 0;          // lane 0: row above at columns c-1 and c (previous step's B and C)
    int misses = 0;
    bool stop = false;
    for (int t = 0; t < nsteps; t++) {
        const int ci = t / kChunk, ti = t - ci * kChunk;
        if (ti == 0) {
            long long it = 0;
            while (!mbar_try_wait(mybars + (ci & 1), (unsigned)(ci >> 1) & 1u))
                if (++it > a.spin_limit) {
                    stop = true;
                    break;
                }
            // a wait that ran out here, or lane 0's wait on the row above in the last chunk
            if (__any_sync(0xffffffffu, stop || *((volatile int*)&abort_flag))) {
                if (lane == 0) {
                    abort_flag = 1;
                    atomicOr(&a.ctrl->status, ST_TIMEOUT);
                }
                break;
            }
            consumed = ci + 1;
            // the other buffer held chunk ci-1, finished: refill it with chunk ci+1
            if (ci >= 1 && ci + 1 < nchunks) {
                if (lane == 0) issue(ci + 1);
                issued++;
            }
        }
        const int c = t - 2 * lane;
        const bool active = row_ok && c >= 0 && c < cols;
        const WaveRec& rec = mybuf[((ci & 1) * kChunk + ti) * 32 + lane];
        int B = s2, C = s1, D = s3;
        if (w > 0) {
            if (lane == 0 && active) {
                // warp w-1's lane 31 stores the row above: only column c+1 is new.  A wait that runs
                // out leaves this step's neighbours as they are (indices do not depend on them) and
                // ends the warp at the next chunk boundary.
                if (c == 0) {
                    long long it = 0;
                    while ((pc = above[0]) == kEmpty)
                        if (++it > a.spin_limit || *((volatile int*)&abort_flag)) {
                            stop = true;
                            abort_flag = 1;
                            break;
                        }
                    pb = 0;
                }
                int nc = 0;
                if (c + 1 < cols) {
                    long long it = 0;
                    while ((nc = above[c + 1]) == kEmpty)
                        if (++it > a.spin_limit || *((volatile int*)&abort_flag)) {
                            stop = true;
                            abort_flag = 1;
                            break;
                        }
                }
                D = pb;
                B = pc;
                C = nc;
                pb = pc;
                pc = nc;
            }
        } else if (band0 > 0 && lane == 0 && active) {
            B = __ldcg(above_g + c);
            C = c + 1 < cols ? __ldcg(above_g + c + 1) : 0;
            D = c >= 1 ? __ldcg(above_g + c - 1) : 0;
        }
        // the record lookup, straight-line in every lane (an inactive lane's record slot holds data of
        // some step, its result is not stored)
        const int key = median_packed(rec.av, o1, B, C, D);
        unsigned e;
        const bool inr = wave_encode(key, &e);
        int h1, h2;
        wave_buckets(e, &h1, &h2);
        const uint4 b1 = reinterpret_cast<const uint4*>(rec.slot)[h1];
        const uint4 b2 = reinterpret_cast<const uint4*>(rec.slot)[h2];
        // a table holds each prediction once: the matching entry's code + 1, else 0
        const unsigned m = 0xff3fffffu;
        auto code1 = [&](unsigned v) { return (v & m) == e ? ((v >> 22) & 3u) + 1u : 0u; };
        const unsigned k1 = max(max(code1(b1.x), code1(b1.y)), max(code1(b1.z), code1(b1.w)));
        const unsigned k2 = max(max(code1(b2.x), code1(b2.y)), max(code1(b2.z), code1(b2.w)));
        const unsigned k = max(k1, k2);
        const bool hit = inr && k != 0u;
        int out = k == 1u ? rec.spec : (k == 2u ? key : 0);
        unsigned miss = __ballot_sync(0xffffffffu, active && !hit);
        if (miss) {
            misses += __popc(miss);
            do {
                const int f = __ffs(miss) - 1;
                miss &= miss - 1;
                const int fkey = __shfl_sync(0xffffffffu, key, f);
                const int fk = (32 * band + f) * cols + (t - 2 * f);
                int4 rv;
                // a full search per miss: first the MB's records of this estimate (their final
                // vectors are searched ones, which the wavefront table leaves out)
                const int4 cr = __ldcg(a.cache + (size_t)fk * KCACHE + lane);
                const unsigned ch = __ballot_sync(0xffffffffu, cr.x == fkey);
                if (ch) {
                    const int src = __ffs(ch) - 1;
                    rv = make_int4(fkey, 0, __shfl_sync(0xffffffffu, cr.z, src), __shfl_sync(0xffffffffu, cr.w, src));
                } else {
                    rv = evaluate(a, fk, mv_x(fkey), mv_y(fkey), lane);
                }
                if (lane == f) {
                    out = rv.z;
                    a.final_mv[fk] = rv.z;
                    a.final_dist[fk] = rv.w;
                }
            } while (miss);
        }
        if (active) {
            a.wave_choice[r * cols + c] = hit ? key : kEmpty;
            if (lane == 31) {
                edge[w * cols + c] = out;
                a.final_mv[r * cols + c] = out;  // the next launch's first band reads this row
            }
        }
        o1 = out;
        s3 = s2;
        s2 = s1;
        s1 = __shfl_up_sync(0xffffffffu, out, 1);
    }
    // copies still in flight after an abort land before the CTA leaves; a
    // drain that gives up (only after a timeout) is reported as one too
    for (int ci = consumed; ci < issued; ci++) {
        long long it = 0;
        while (!mbar_try_wait(mybars + (ci & 1), (unsigned)(ci >> 1) & 1u))
            if (++it > a.spin_limit) {
                atomicOr(&a.ctrl->status, ST_TIMEOUT);
                break;
            }
    }
    if (lane == 0 && misses) atomicAdd(&a.ctrl->wave_miss, misses);
    __syncthreads();
    if (threadIdx.x == 0 && !abort_flag && last) a.ctrl->sweeps = a.relax_sweeps + 1000;
}

// Outputs of a wavefront-resolved frame, one thread per MB: the record each
// MB took (or the vector and distortion the wavefront evaluated), and the
// included-distortion average (Full.cpp:581-611).
__global__ void __launch_bounds__(256) k_full_wave_outputs(FullArgs a)
{
    if (*((volatile int*)&a.ctrl->converged) || (*((volatile int*)&a.ctrl->status) & ST_TIMEOUT)) return;
    long long tot = 0;
    int cnt = 0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.nmb; k += gridDim.x * blockDim.x) {
        const int key = a.wave_choice[k];
        int fmv = 0, d = 0;
        if (key != kEmpty) {
            const int4* cache = a.cache + (size_t)k * KCACHE;
            for (int e = 0; e < KCACHE; e++) {
                const int4 rec = __ldcg(cache + e);
                if (rec.x == key) {
                    fmv = rec.z;
                    d = rec.w;
                    break;
                }
            }
        } else {
            fmv = a.final_mv[k];
            d = a.final_dist[k];
        }
        a.final_mv[k] = fmv;
        a.final_dist[k] = d;
        a.job->out_mv[k] = fmv;
        if (a.job->out_dist) a.job->out_dist[k] = d;
        if (a.job->incl && a.job->incl[k]) {
            tot += d;
            cnt++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if ((threadIdx.x & 31) == 0 && cnt) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->total), (unsigned long long)tot);
        atomicAdd(&a.ctrl->count, cnt);
    }
}

// The included-distortion average, once every output block has added its sums.
__global__ void k_full_average(FullArgs a)
{
    if (*((volatile int*)&a.ctrl->status) & ST_TIMEOUT) return;
    const long long t = a.ctrl->total;
    const int c = a.ctrl->count;
    if (a.job->out_avg) *a.job->out_avg = c ? t / c : 0;
}

// ---------------------------------------------------------------------------
// The resolve of every estimator but Ver2's Lagrangian overload: an evaluation
// there is one round trip to L2 (the distortion at the prediction from the
// half-pel planes), so nothing is precomputed or kept; what counts is how many
// evaluations follow one another.
//
//   k_resolve_first   every MB at the median of the searched vectors
//   k_resolve_sweep   every MB whose prediction moved, over the whole GPU
//   k_resolve_finish  the rest, by one cluster
//
// k_resolve_finish keeps the frame's vectors in the shared memory of a cluster,
// a band of rows per CTA with the last row of the band above beside it, and
// works in rounds: every marked macroblock takes the median of its neighbours'
// vectors; those whose prediction moved are listed and evaluated, half a warp
// each, and where the vector changed it is replaced and its four dependents
// are marked.  After up to kFinishSub such rounds, fewer when nothing of the
// band moves, the cluster meets: the copies of the band's last row and the
// marks that the CTA above sent (distributed shared memory) count from then
// on.  The state always satisfies vector = f(prediction used), and a vector
// that changes marks all that read it, so a meeting after which nobody had
// work is the fixed point, which is the sequential result.  A median reads
// only earlier anti-diagonals c + 2r, so a meeting settles at least the first
// one that still moves: a frame takes at most cols + 2 rows meetings.
//
// What bounds a round is a chain: the L2 latency of an evaluation's samples (~800 cycles) and its instructions one
// after the other; a meeting costs ~1300 cycles more, which is why it waits for up to eight rounds (1080p pans with
// moving objects, a meeting after each round 440 us a frame, after up to eight 397; the record and wavefront kernels
// before 613).  While the distortions lie in shared memory (all but the largest frames) and no tie is deep, no round
// writes global memory: the barrier would wait for it.

// Sixteen consecutive bytes from any address, by two 16-byte loads: a warp's
// rows lie in 32 different lines, and the load unit takes a cycle or more for
// each line of an instruction (five word loads: 10 x 32 of them for the two
// samples of a quarter position, 0.35 us of a round).
__device__ __forceinline__ void load_row16(const unsigned char* p, unsigned* w)
{
    const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)15);
    const uint4 lo = __ldg(q), hi = __ldg(q + 1);
    const unsigned o = (unsigned)(reinterpret_cast<uintptr_t>(p) & 15), sh = 8 * (o & 3);
    const bool s2 = o & 8, s1 = o & 4;
    const unsigned a0 = s2 ? lo.z : lo.x, a1 = s2 ? lo.w : lo.y, a2 = s2 ? hi.x : lo.z, a3 = s2 ? hi.y : lo.w;
    const unsigned a4 = s2 ? hi.z : hi.x, a5 = s2 ? hi.w : hi.y;
    const unsigned v0 = s1 ? a1 : a0, v1 = s1 ? a2 : a1, v2 = s1 ? a3 : a2, v3 = s1 ? a4 : a3, v4 = s1 ? a5 : a4;
    w[0] = __funnelshift_r(v0, v1, sh);
    w[1] = __funnelshift_r(v1, v2, sh);
    w[2] = __funnelshift_r(v2, v3, sh);
    w[3] = __funnelshift_r(v3, v4, sh);
}

// The integer-pel SAD stage, resolved by the same kernels: its vector and distortion depend on the prediction
// only where the scan met a tie (MotionEstimatorH264ImplFull.cpp:424-441), and then only on the rounded one.
// (1920x1080: a frame 0.419 ms with a CTA that walked the anti-diagonals, a block barrier for each with ties,
// 0.234 so; 176x144 the same.)
constexpr int EST_SAD = 6;
// Whether a result at prediction pu may differ from that at `key`; flags: the MB's record.
template <int kEst>
__device__ __forceinline__ bool stale(int key, int pu, int flags)
{
    if constexpr (kEst == EST_SAD)
        return (flags & FLAG_TIE) && (round_pred(mv_x(key)) != round_pred(mv_x(pu)) ||
                                      round_pred(mv_y(key)) != round_pred(mv_y(pu)));
    return key != pu;
}

// One MB per half warp (16 lanes, a row of 16 samples each): the final vector
// and distortion of MB k (origin n, m) at prediction `key`, from its searched
// result `sp` and this lane's row of the input.  Lanes of a half without work
// (act false) pass any valid MB.
template <int kEst>
__device__ __forceinline__ int2 evaluate_half(const FullArgs& a, bool act, int k, int n, int m, int key, int4 sp,
                                              uint4 cur, int lane, mrc::Lattice* lt)
{
    const int px = mv_x(key), py = mv_y(key);
    PredGeom g{};
    int pd = 0;
    if constexpr (kEst != EST_SAD) {
        g = pred_geom(n, m, a.W, a.H, px, py);
        // qpel_block8's sixteen cases by bit fields: the plane (0 full pel, 1 b, 2 h, 3 j) and the column and
        // row offset of both averaged samples; the cases of one sample average it with itself
        const int s = g.fx | (g.fy << 2);
        constexpr unsigned kP1 = 0u | 0u << 2 | 1u << 4 | 0u << 6 | 0u << 8 | 1u << 10 | 3u << 12 | 1u << 14 | 2u << 16 |
                                 3u << 18 | 3u << 20 | 3u << 22 | 0u << 24 | 2u << 26 | 3u << 28 | 2u << 30;
        constexpr unsigned kP2 = 0u | 1u << 2 | 1u << 4 | 1u << 6 | 2u << 8 | 2u << 10 | 1u << 12 | 2u << 14 | 2u << 16 |
                                 2u << 18 | 3u << 20 | 2u << 22 | 2u << 24 | 1u << 26 | 1u << 28 | 1u << 30;
        constexpr unsigned kX1 = 1u << 3 | 1u << 15, kX2 = 1u << 7 | 1u << 11;
        constexpr unsigned kY1 = 1u << 12, kY2 = 1u << 13 | 1u << 14 | 1u << 15;
        const int p1 = (kP1 >> (2 * s)) & 3, p2 = (kP2 >> (2 * s)) & 3;
        const int at = (g.oy + (lane & 15) + PAD) * a.rstride + g.ox + PAD;
        const unsigned char* b1 = p1 ? a.hpel + (size_t)(p1 - 1) * a.plane_size : a.refp;
        const unsigned char* b2 = p2 ? a.hpel + (size_t)(p2 - 1) * a.plane_size : a.refp;
        b1 += at + (int)((kX1 >> s) & 1) + ((kY1 >> s) & 1 ? a.rstride : 0);
        b2 += at + (int)((kX2 >> s) & 1) + ((kY2 >> s) & 1 ? a.rstride : 0);
        unsigned w1[4], w2[4];
        load_row16(b1, w1);
        load_row16(b2, w2);
        const unsigned c4[4] = {cur.x, cur.y, cur.z, cur.w};
        // Cross: Tsd16x16PartialPath, the row's samples that lie on its path of 64 points
        uint4 mask = make_uint4(~0u, ~0u, ~0u, ~0u);
        if constexpr (kEst == cross::EST_CROSS)
            mask = __ldg(reinterpret_cast<const uint4*>(cross::c_path_rows.m[lane & 15]));
        const unsigned m4[4] = {mask.x, mask.y, mask.z, mask.w};
        unsigned acc = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned d = __vabsdiffu4(c4[i], __vavgu4(w1[i], w2[i]));
            acc = __dp4a(d & m4[i], d, acc);
        }
        const unsigned lo = __reduce_add_sync(0xffffffffu, lane < 16 ? acc : 0u);
        const unsigned hi = __reduce_add_sync(0xffffffffu, lane < 16 ? 0u : acc);
        pd = (int)(lane < 16 ? lo : hi);
    }
    int mvx = mv_x(sp.x), mvy = mv_y(sp.x), minD = sp.y;
    constexpr bool kScan = kEst == 0 || kEst == EST_SAD;  // ties decided at the rounded prediction (0, 0)
    const bool tie = act && (sp.w & FLAG_TIE) && (!kScan || round_pred(px) != 0 || round_pred(py) != 0);
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    if (ties) {  // rare: the searched vector depends on the prediction; a whole warp's work
#pragma unroll 1
        for (int h = 0; h < 2; h++) {
            if (!((ties >> (16 * h)) & 1u)) continue;
            const int hk = __shfl_sync(0xffffffffu, k, 16 * h), hx = __shfl_sync(0xffffffffu, px, 16 * h);
            const int hy = __shfl_sync(0xffffffffu, py, 16 * h), hf = __shfl_sync(0xffffffffu, sp.w, 16 * h);
            int tx = __shfl_sync(0xffffffffu, mvx, 16 * h), ty = __shfl_sync(0xffffffffu, mvy, 16 * h);
            int td = __shfl_sync(0xffffffffu, minD, 16 * h);
            if constexpr (kScan) tie_path(a, hk, hx, hy, hf, lane, &tx, &ty, &td);
            else pred_search_at<kEst>(a, hk, hx, hy, lane, &tx, &ty, &td, lt);
            if ((lane >> 4) == h) {
                mvx = tx;
                mvy = ty;
                minD = td;
            }
        }
    }
    if constexpr (kEst == EST_SAD) return make_int2(pack_mv(mvx, mvy), minD);  // no GetBestVector
    const int pos = best_of3_fast(mvx, mvy, minD, g.pcx, g.pcy, pd, sp.z, a.lambda, g.pcx, g.pcy,
                                  kEst == cross::EST_CROSS ? cross::PATH_NORM : 256);
    return pos == 0 ? make_int2(pack_mv(mvx, mvy), minD) : pos == 1 ? make_int2(pack_mv(g.pcx, g.pcy), pd)
                                                                    : make_int2(0, sp.z);
}

// This lane's row of MB (n, m)'s input.
__device__ __forceinline__ uint4 load_cur16(const FullArgs& a, int n, int m, int lane)
{
    return __ldg(reinterpret_cast<const uint4*>(a.src8 + (size_t)(m + (lane & 15)) * a.W + n));
}

// The median prediction from the vectors in global memory; the neighbours are
// read by position, beside the record that says which of them count.
__device__ __forceinline__ int median_global(const FullArgs& a, int k, int r, int c, int4* sp)
{
    const int cols = a.cols;
    *sp = __ldcg(a.spec4 + k);
    const int A = c > 0 ? __ldcg(a.final_mv + k - 1) : 0;
    const int B = r > 0 ? __ldcg(a.final_mv + k - cols) : 0;
    const int C = r > 0 && c + 1 < cols ? __ldcg(a.final_mv + k - cols + 1) : 0;
    const int D = r > 0 && c > 0 ? __ldcg(a.final_mv + k - cols - 1) : 0;
    return median_packed(sp->w, A, B, C, D);
}

template <int kEst>
__global__ void __launch_bounds__(256) k_resolve_first(const __grid_constant__ FullArgs a)
{
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int item = (blockIdx.x * 8 + wib) * 2 + (lane >> 4);
    const bool act = item < a.nmb;
    if (!__any_sync(0xffffffffu, act)) return;
    const int k = act ? item : 0, r = k / a.cols, c = k - r * a.cols;
    const uint4 cur = load_cur16(a, 16 * c, 16 * r, lane);
    int4 sp;
    const int key = median_global(a, k, r, c, &sp);
    const int2 out = evaluate_half<kEst>(a, act, k, 16 * c, 16 * r, key, sp, cur, lane, LatticeSlots<kEst>::get(wib));
    if (act && (lane & 15) == 0) {
        __stcg(a.pred_used + k, key);
        __stcg(a.final_dist + k, out.y);
        __stcg(a.final_mv + k, out.x);
    }
}

// One sweep over every MB: lane per MB (MBs gwarp + lane*nwarps ...) to find
// those whose prediction moved, then a half warp on each.  Skipped once an
// earlier sweep changed no vector.
template <int kEst>
__global__ void __launch_bounds__(256) k_resolve_sweep(const __grid_constant__ FullArgs a, int sweep)
{
    if (sweep > 1 && *((volatile int*)&a.changed[sweep - 1]) == 0) return;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gwarp = blockIdx.x * 8 + wib, nwarps = gridDim.x * 8;
    int changed = 0, evals = 0;
    for (int base = gwarp; base < a.nmb; base += 32 * nwarps) {
        const int k = base + lane * nwarps;
        int key = 0;
        int4 sp;
        bool moved = false;
        if (k < a.nmb) {
            const int r = k / a.cols;
            key = median_global(a, k, r, k - r * a.cols, &sp);
            moved = stale<kEst>(key, __ldcg(a.pred_used + k), sp.w);
        }
        unsigned todo = __ballot_sync(0xffffffffu, moved);
        while (todo) {
            const int f0 = __ffs(todo) - 1;
            todo &= todo - 1;
            const int f1 = todo ? __ffs(todo) - 1 : f0;
            const bool two = todo != 0;
            todo &= todo - 1;
            const int f = lane < 16 ? f0 : f1;
            const bool act = lane < 16 || two;
            const int kk = base + f * nwarps, r = kk / a.cols, c = kk - r * a.cols;
            const int fkey = __shfl_sync(0xffffffffu, key, f);
            int4 fsp;
            fsp.x = __shfl_sync(0xffffffffu, sp.x, f);
            fsp.y = __shfl_sync(0xffffffffu, sp.y, f);
            fsp.z = __shfl_sync(0xffffffffu, sp.z, f);
            fsp.w = __shfl_sync(0xffffffffu, sp.w, f);
            const uint4 cur = load_cur16(a, 16 * c, 16 * r, lane);
            const int old = __ldcg(a.final_mv + kk);
            const int2 out = evaluate_half<kEst>(a, act, kk, 16 * c, 16 * r, fkey, fsp, cur, lane,
                                                 LatticeSlots<kEst>::get(wib));
            if (act && (lane & 15) == 0) {
                __stcg(a.pred_used + kk, fkey);
                __stcg(a.final_dist + kk, out.y);
                if (old != out.x) __stcg(a.final_mv + kk, out.x);
                evals++;
                changed += old != out.x;
            }
            __syncwarp();
        }
    }
    evals = __reduce_add_sync(0xffffffffu, evals);
    changed = __reduce_add_sync(0xffffffffu, changed);
    if (lane == 0 && evals) {
        atomicAdd(&a.ctrl->relax_evals, evals);
        atomicAdd(&a.ctrl->relax_miss, evals);
        if (changed) atomicAdd(&a.changed[sweep], changed);
    }
}

constexpr int kFinishThreads = 512;
constexpr int kFinishHalves = kFinishThreads / 16;  // evaluations in flight per CTA
constexpr int kFinishSub = 8;                       // most rounds between two meetings of the cluster
constexpr int kFinishSmem = 220 * 1024;             // most dynamic shared memory of a CTA

// A CTA of the cluster holds `band` rows: per macroblock its vector, the
// prediction it was evaluated at, its distortion (`dist`; else that stays in
// global memory), a work entry, its neighbour mask and its mark; the row
// above the band, and the marks that arrive from there (two buffers).
struct FinishShape {
    int ctas, band, dist;
    size_t smem;
};
FinishShape finish_shape(int cols, int rows)
{
    FinishShape f;
    f.ctas = cols * rows <= kFinishThreads ? 1 : cols * rows <= 4 * kFinishThreads ? 4 : 8;
    for (;;) {
        f.band = (rows + f.ctas - 1) / f.ctas;
        const size_t n = (size_t)f.band * cols;
        f.dist = 1;
        f.smem = 4 * (3 * n + cols) + 4 * ((n + 3) / 4 * 4) + (size_t)(2 * cols + 3) / 4 * 4;
        if (f.smem <= (size_t)kFinishSmem) return f;
        if (f.ctas == 16) break;
        f.ctas = 16;  // beyond ~110000 macroblocks: the non-portable size
    }
    f.dist = 0;  // 8192 x 8192: 200 KB
    f.smem -= 4 * (size_t)f.band * cols;
    return f;
}

template <int kEst>
__global__ void __launch_bounds__(kFinishThreads, 1)
    k_resolve_finish(const __grid_constant__ FullArgs a, int first, int band, int keep_dist, int fresh)
{
    extern __shared__ __align__(16) int fin_smem[];
    __shared__ int s_n[2], s_any[3], s_evals[2], s_changed[RELAX_SWEEPS + 1];
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), ctas = (int)cluster.num_blocks();
    const int cols = a.cols, rows = a.nmb / cols;
    const int r0 = rank * band, nrow = max(0, min(rows - r0, band)), nloc = nrow * cols, k0 = r0 * cols;
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5, half = lane >> 4;
    const int most_loc = band * cols, quads = (most_loc + 3) >> 2;
    volatile int* s_fin = fin_smem;            // the row above the band, then the band
    int* s_pu = fin_smem + cols + most_loc;    // prediction used
    // marks, a byte each: macroblock i at byte 4 * (i % quads) + i / quads, so that neighbours lie in
    // different words
    unsigned* s_mark = reinterpret_cast<unsigned*>(s_pu + most_loc);
    unsigned char* s_av = reinterpret_cast<unsigned char*>(s_mark + quads);
    unsigned short* s_work = reinterpret_cast<unsigned short*>(s_av + 4 * quads);  // macroblocks whose prediction moved
    unsigned char* s_in = reinterpret_cast<unsigned char*>(s_work + 4 * quads);  // arriving marks of the first row, [2][cols]
    int* s_dist = reinterpret_cast<int*>(s_in + (2 * cols + 3) / 4 * 4);
    const bool has_below = rank + 1 < ctas;
    int* below = has_below ? cluster.map_shared_rank(fin_smem, rank + 1) : fin_smem;  // its row above the band
    unsigned char* below_in = has_below ? cluster.map_shared_rank(s_in, rank + 1) : s_in;
    const float per_col = 1.0f / (float)cols;

    auto mark = [&](int i) {  // i < 4 * quads
        const int q = i >= 2 * quads ? (i >= 3 * quads ? 3 : 2) : (i >= quads ? 1 : 0);
        reinterpret_cast<volatile unsigned char*>(s_mark)[4 * (i - q * quads) + q] = 1;
    };
    auto median_at = [&](int i) {  // local index; the row above is at i
        const int av = s_av[i], at = i + cols;
        const int A = (av & AV_A) ? s_fin[at - 1] : 0;
        const int B = (av & AV_B) ? s_fin[at - cols] : 0;
        const int C = (av & AV_C) ? s_fin[at - cols + 1] : 0;
        const int D = (!(av & AV_C) && (av & AV_D)) ? s_fin[at - cols - 1] : 0;
        return median_packed(av, A, B, C, D);
    };
    if (r0 > 0 && nrow > 0)
        for (int c = tid; c < cols; c += kFinishThreads) s_fin[c] = __ldcg(a.final_mv + k0 - cols + c);
#pragma unroll 2
    for (int i = tid; i < nloc; i += kFinishThreads) {
        if (kEst == EST_SAD && fresh) {  // the searched results are those at prediction (0, 0)
            const int4 sp = __ldcg(a.spec4 + k0 + i);
            s_fin[cols + i] = sp.x;
            s_pu[i] = 0;
            s_av[i] = (unsigned char)sp.w;
            s_dist[i] = sp.y;
            continue;
        }
        s_fin[cols + i] = __ldcg(a.final_mv + k0 + i);
        s_pu[i] = __ldcg(a.pred_used + k0 + i);
        s_av[i] = (unsigned char)__ldcg(&a.spec4[k0 + i].w);
        if (keep_dist) s_dist[i] = __ldcg(a.final_dist + k0 + i);
    }
    for (int i = tid; i < quads; i += kFinishThreads) s_mark[i] = 0x01010101u;
    for (int i = tid; i < 2 * cols; i += kFinishThreads) s_in[i] = 0;
    if (tid < 3) s_any[tid] = 0;
    if (tid < 2) s_n[tid] = s_evals[tid] = 0;
    if (tid <= RELAX_SWEEPS) s_changed[tid] = 0;
    cluster.sync();

    const int most = 64 * (cols + 2 * rows) + 65536;  // far above what the argument at the top allows
    int round = first;
    for (;; round++) {
        for (int sub = 0; sub < kFinishSub; sub++) {
            // list the marked macroblocks whose prediction moved
            int* n = &s_n[sub & 1];
            for (int q = tid; q < quads; q += kFinishThreads) {
                const unsigned m = s_mark[q];
                if (!m) continue;
                s_mark[q] = 0u;
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    const int i = q + b * quads;
                    if (((m >> (8 * b)) & 0xffu) && i < nloc && stale<kEst>(median_at(i), s_pu[i], s_av[i]))
                        s_work[atomicAdd(n, 1)] = (unsigned short)i;
                }
            }
            __syncthreads();
            const int nw = *n;
            if (nw == 0) break;
            if (tid == 0) {
                s_n[(sub + 1) & 1] = 0;
                s_evals[round > a.relax_sweeps] += nw;
            }
            if (tid < ctas) *cluster.map_shared_rank(&s_any[round % 3], tid) = 1;
            // a macroblock per half warp, the second halves after all the first: ties are the whole warp's work
            for (int w = 2 * wib; w < nw; w += kFinishHalves) {
                const bool act = w + half < nw;
                const int i = s_work[act ? w + half : w];
                const int lr = (int)(((float)i + 0.5f) * per_col);  // i / cols: never near a whole number
                const int r = r0 + lr, c = i - lr * cols, k = k0 + i;
                const int4 sp = __ldg(a.spec4 + k);
                const uint4 in = load_cur16(a, 16 * c, 16 * r, lane);
                // one reading of the neighbours for the half warp: others change meanwhile
                const int key = __shfl_sync(0xffffffffu, median_at(i), lane & 16);
                const int old = s_fin[cols + i];
                const int2 out = evaluate_half<kEst>(a, act, k, 16 * c, 16 * r, key, sp, in, lane, nullptr);
                const bool changed = act && old != out.x;
                const int d = lane & 15;
                if (act && d == 0) {
                    s_pu[i] = key;
                    if (keep_dist) s_dist[i] = out.y;
                    else __stcg(a.final_dist + k, out.y);
                    if (changed) {
                        s_fin[cols + i] = out.x;
                        if (lr == band - 1 && has_below) below[c] = out.x;
                        if (round <= a.relax_sweeps) atomicAdd(&s_changed[round], 1);
                    }
                }
                // its dependents, a lane each: right, below, below left, below right
                const int c2 = c + (d == 0 ? 1 : (d == 1 ? 0 : (d == 2 ? -1 : 1)));
                if (changed && d < 4 && c2 >= 0 && c2 < cols) {
                    if (d == 0) mark(i + 1);
                    else if (lr < band - 1) mark(i + cols + c2 - c);
                    else if (has_below) below_in[(round & 1) * cols + c2] = 1;
                }
                __syncwarp();
            }
            __syncthreads();
        }
        if (tid == 0) {
            s_n[0] = s_n[1] = 0;
            s_any[(round + 1) % 3] = 0;
        }
        cluster.sync();
        // what arrived before the meeting; the other buffer takes what follows it
        for (int c = tid; c < cols; c += kFinishThreads)
            if (s_in[(round & 1) * cols + c]) {
                s_in[(round & 1) * cols + c] = 0;
                mark(c);
            }
        __syncthreads();
        if (!*((volatile int*)&s_any[round % 3])) break;
        if (round - first > most) {
            if (tid == 0) atomicOr(&a.ctrl->status, ST_TIMEOUT);
            break;
        }
    }
    // outputs and the included-distortion average (Full.cpp:581-611)
    const JobDesc job = *a.job;
    long long tot = 0;
    int cnt = 0;
#pragma unroll 2
    for (int i = tid; i < nloc; i += kFinishThreads) {
        const int k = k0 + i, fmv = s_fin[cols + i], d = keep_dist ? s_dist[i] : __ldcg(a.final_dist + k);
        const int inc = job.incl ? job.incl[k] : 0;
        job.out_mv[k] = fmv;
        if (job.out_dist) job.out_dist[k] = d;
        if (inc) {
            tot += d;
            cnt++;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if (lane == 0 && cnt) {
        atomicAdd(reinterpret_cast<unsigned long long*>(&a.ctrl->total), (unsigned long long)tot);
        atomicAdd(&a.ctrl->count, cnt);
    }
    if (kEst != EST_SAD && tid == 0) {
        if (s_evals[0]) {
            atomicAdd(&a.ctrl->relax_evals, s_evals[0]);
            atomicAdd(&a.ctrl->relax_miss, s_evals[0]);
        }
        if (s_evals[1]) atomicAdd(&a.ctrl->wave_miss, s_evals[1]);
    }
    if (kEst != EST_SAD && tid <= RELAX_SWEEPS && s_changed[tid]) atomicAdd(&a.changed[tid], s_changed[tid]);
    cluster.sync();
    if (rank == 0 && tid == 0) {
        if constexpr (kEst != EST_SAD) {
            const int settled = round - 1;  // the last round (or sweep) with work
            const bool relaxed = a.relax_sweeps > 0 && settled <= a.relax_sweeps;
            a.ctrl->sweeps = relaxed ? (settled > 0 ? settled : 1) : a.relax_sweeps + 1000;
            a.ctrl->converged = relaxed;
        }
        const long long t = (long long)__ldcg(reinterpret_cast<const unsigned long long*>(&a.ctrl->total));
        const int n = __ldcg(&a.ctrl->count);
        if (job.out_avg) *job.out_avg = n ? t / n : 0;
    }
}

// Motion-compensated luma residual (MotionCompensatorH264ImplStd::Compensate,
// MotionCompensatorH264ImplStd.cpp:413-431: QuarterRead of the reference at
// the vector, a copy for full-pel vectors; then OverlayMem2Dv2::Sub16x16):
// one warp per macroblock, samples from the estimate's planes.
__global__ void __launch_bounds__(256) k_full_residual(FullArgs a, const int* __restrict__ mv, short* __restrict__ res)
{
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (k >= a.nmb) return;
    const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
    const int v = mv[k], mvx = mv_x(v), mvy = mv_y(v);
    const int qx = mvx % 4, qy = mvy % 4;  // C remainders, folded as QuarterRead does
    const int fx = qx < 0 ? qx + 4 : qx, fy = qy < 0 ? qy + 4 : qy;
    const int ox = n + mvx / 4 + (qx < 0 ? -1 : 0), oy = m + mvy / 4 + (qy < 0 ? -1 : 0);
    short* dst = res + (size_t)(m + (lane >> 1)) * a.W + n + 8 * (lane & 1);
    // a prediction more than 32 samples outside the picture would leave the
    // padded planes: flagged, residual zero
    if (ox < -32 || oy < -32 || ox > a.W + 16 || oy > a.H + 16) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
        if (lane == 0) atomicOr(&a.ctrl->status, ST_OUT_OF_BOUNDS);
        return;
    }
    const uint2 p = qpel_block8(a, ox, oy, fx, fy, lane);
    const uint2 c = load_cur8(a, n, m, lane);
    short vals[8];
#pragma unroll
    for (int b = 0; b < 4; b++) {
        vals[b] = (short)((int)((c.x >> (8 * b)) & 0xff) - (int)((p.x >> (8 * b)) & 0xff));
        vals[4 + b] = (short)((int)((c.y >> (8 * b)) & 0xff) - (int)((p.y >> (8 * b)) & 0xff));
    }
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(vals);
}

size_t wave_smem_bytes(int nw, int cols, int chunk)
{
    return (size_t)kWaveStepBytes * nw * 2 * chunk + sizeof(unsigned long long) * nw * 2 + sizeof(int) * (size_t)nw * cols;
}

constexpr int kWaveMaxCols = 512;  // 8192 / 16

}  // namespace

namespace {
template <int kEst>
int finish_prepare();
}

int full_resolve_prepare(vppgpu_ctx*)
{
    VPP_CUDA(cudaFuncSetAttribute(k_full_wave<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)wave_smem_bytes(3, kWaveMaxCols, 4)));
    VPP_CUDA(cudaFuncSetAttribute(k_full_wave<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)wave_smem_bytes(kWaveMaxWarps, kWaveMaxCols, 2)));
    int rc;
    if ((rc = finish_prepare<0>()) || (rc = finish_prepare<1>()) || (rc = finish_prepare<2>()) ||
        (rc = finish_prepare<cross::EST_CROSS>()) || (rc = finish_prepare<EST_SAD>()))
        return rc;
    return VPPGPU_OK;
}

namespace {

// Ver2's Lagrangian overload: an evaluation is a whole search, so records, dictionary and closure pay.
int resolve_launch_records(vppgpu_ctx* ctx, const FullArgs& args)
{
    const int rows = args.nmb / args.cols, nbands = (rows + 31) / 32;
    if (args.cols > kWaveMaxCols) return VPPGPU_ERR_UNSUPPORTED;
    k_full_sweep0<<<(args.nmb + 7) / 8, 256, 0, ctx->stream>>>(args);
    VPP_CHECK_LAUNCH(ctx);
    {
        // many warps, few MBs each: a sweep's latency is its busiest warp's evaluations
        const int want = (args.nmb + 7) / 8, cap = ctx->sm_count * args.relax_blocks_per_sm;
        for (int sweep = 1; sweep <= args.relax_sweeps; sweep++) {
            k_full_relax_sweep<<<want < cap ? want : cap, 256, 0, ctx->stream>>>(args, sweep);
            VPP_CHECK_LAUNCH(ctx);
        }
        const int ob = (args.nmb + 255) / 256, ocap = ctx->sm_count * 4;
        k_full_relax_outcome<<<ob < ocap ? ob : ocap, 256, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
    }
    {
        const int blocks = (args.nmb + 7) / 8, cap = ctx->sm_count * 8, grid = blocks < cap ? blocks : cap;
        k_full_precompute<<<grid, 256, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
        k_full_closure<<<grid, 256, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
    }
    for (int b0 = 0; b0 < nbands; b0 += kWaveMaxWarps) {
        const int nw = nbands - b0 < kWaveMaxWarps ? nbands - b0 : kWaveMaxWarps;
        const int last = b0 + nw == nbands;
        if (nw <= 3)
            k_full_wave<4><<<1, nw * 32, wave_smem_bytes(nw, args.cols, 4), ctx->stream>>>(args, b0, last);
        else
            k_full_wave<2><<<1, nw * 32, wave_smem_bytes(nw, args.cols, 2), ctx->stream>>>(args, b0, last);
        VPP_CHECK_LAUNCH(ctx);
    }
    {
        const int blocks = (args.nmb + 255) / 256, cap = ctx->sm_count * 4;
        k_full_wave_outputs<<<blocks < cap ? blocks : cap, 256, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
        k_full_average<<<1, 1, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
    }
    return VPPGPU_OK;
}

constexpr int kSadFresh = 2048;  // macroblocks; within the sizes whose distortions the cluster keeps

template <int kEst>
int resolve_launch(vppgpu_ctx* ctx, const FullArgs& args)
{
    // the SAD stage of a small frame starts the cluster from the searched results themselves
    const bool fresh = kEst == EST_SAD && args.nmb <= kSadFresh;
    if (!fresh) {
        k_resolve_first<kEst><<<(args.nmb + 15) / 16, 256, 0, ctx->stream>>>(args);
        VPP_CHECK_LAUNCH(ctx);
    }
    const int want = (args.nmb + 7) / 8, cap = ctx->sm_count * args.relax_blocks_per_sm;
    const int blocks = want < cap ? want : cap;
    const int sweeps = args.relax_sweeps < args.grid_sweeps ? args.relax_sweeps : args.grid_sweeps;
    for (int sweep = 1; sweep <= sweeps; sweep++) {
        k_resolve_sweep<kEst><<<blocks, 256, 0, ctx->stream>>>(args, sweep);
        VPP_CHECK_LAUNCH(ctx);
    }
    const FinishShape f = finish_shape(args.cols, args.nmb / args.cols);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.ctas);
    cfg.blockDim = dim3(kFinishThreads);
    cfg.dynamicSmemBytes = f.smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = f.ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    VPP_CUDA(cudaLaunchKernelEx(&cfg, k_resolve_finish<kEst>, args, sweeps + 1, f.band, f.dist, (int)fresh));
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

template <int kEst>
int finish_prepare()
{
    VPP_CUDA(cudaFuncSetAttribute(k_resolve_finish<kEst>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinishSmem));
    VPP_CUDA(cudaFuncSetAttribute(k_resolve_finish<kEst>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    return VPPGPU_OK;
}

}  // namespace

int full_resolve_launch(vppgpu_ctx* ctx, const FullArgs& args, int est)
{
    switch (est) {
    case 0: return resolve_launch<0>(ctx, args);
    case 1: return resolve_launch<1>(ctx, args);
    case 2: return resolve_launch<2>(ctx, args);
    case cross::EST_CROSS: return resolve_launch<cross::EST_CROSS>(ctx, args);
    case mrc::EST_V2_LAMBDA: return resolve_launch_records(ctx, args);
    default: return VPPGPU_ERR_INVALID_ARG;
    }
}

int sad_resolve_launch(vppgpu_ctx* ctx, const FullArgs& args)
{
    FullArgs a = args;
    a.relax_sweeps = a.grid_sweeps = 0;
    return resolve_launch<EST_SAD>(ctx, a);
}

int full_residual_launch(vppgpu_ctx* ctx, const FullArgs& args, const int* d_mv, short* d_res)
{
    k_full_residual<<<(args.nmb + 7) / 8, 256, 0, ctx->stream>>>(args, d_mv, d_res);
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

}  // namespace vppgpu
