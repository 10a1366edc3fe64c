// me_full.cu -- MotionEstimatorH264ImplFull on sm_103a.
//
// Reference: MotionEstimatorH264ImplFull::Estimate
// (src/CodecUtils/MotionEstimatorH264ImplFull.cpp:330-613).  Per 16x16
// macroblock: squared-error full search of +-R pels (running-best skip and
// prediction tie-break, :394-446), half-pel then quarter-pel refinement
// (:452-517), distortion at the median-predicted vector (:532-570) and a
// Lagrangian pick between best, predicted and zero vectors (:573-601).
//
// GB300 design
//   k_full_planes   one pass over tiles of the padded reference: int16 ->
//                   u8 (with a 0..255 check) and edge replication, the b / h /
//                   j half-pel planes (sub-pel stages, every distortion at a
//                   predicted vector) and the 16x16 block energies (the B^2 of
//                   every candidate's SSD = A^2 + B^2 - 2 sum(ab)); the input's
//                   byte packing rides along.
//   k_ssd_rowmin    (me_full_tc.cu) the minimum SSD of every 8 neighbouring
//                   candidates of every macroblock, by the tensor cores.
//   k_full_scan     a warp per MB: replays the reference's sequential raster
//                   scan, forming the SSDs of the few groups of candidates
//                   whose minimum and range can win, then the half-pel and
//                   quarter-pel refinement.
//   k_full_tietree  for the MBs whose scan met an exact tie, the whole table
//                   and the scan outcome of every tie decision pattern (the
//                   tie tree), read by the prediction-dependent stage.
//   k_sad_search    the SAD search's table: persistent, warp-specialised:
//                   compute warps build each macroblock's (2R+1)^2 table in
//                   shared memory (vabsdiff4, tiles staged by TMA tensor
//                   copies), a scan warp replays the scan over it.  Only the
//                   tables of tie macroblocks leave the SM.
//   resolve         (me_full_resolve.cu) the prediction-dependent tail:
//                   median prediction, tie rescans, prediction distortion
//                   and the Lagrangian pick, in the reference's raster order.
#include <string.h>

#include <cudaTypedefs.h>
#include <mutex>

#include "me_full_common.cuh"

namespace vppgpu {
namespace {
using namespace full;

// ---------------------------------------------------------------------------
// The frame's planes in one pass, a CTA per PL_TX x PL_TY tile of the padded
// reference (PAD samples of edge replication each side, OverlayExtMem2Dv2's
// extended boundary as a coordinate clamp):
//   refp    the padded reference as bytes (0..255 checked)
//   hpel    its H.264 half-pel planes, b (x half: 6-tap (1,-5,20,20,-5,1) on
//           the row, (+16) >> 5), h (y half, on the column) and j (centre:
//           the 6-tap over the unrounded vertical taps, (+512) >> 10), each
//           clipped to 0..255 -- the samples QuarterRead combines
//           (OverlayMem2Dv2.cpp:704-1052)
//   energy  (SSD search only) E(Y, X) = sum of squares of the 16x16 block at
//           (Y, X), its samples less 128, for Y <= PH-16, X <= PW-16: the B^2
//           term of every candidate's SSD = A^2 + B^2 - 2 sum(ab); below 2^23,
//           stored as the floats the row minima are formed with
// plus a share of the input's byte packing (src8, 0..255 checked).  The tile
// and its halo (2 before, 15 after in each direction) are staged once as
// bytes; taps read clamped coordinates, which differs from a clamped padded
// plane only within 3 samples of its border, never read (a prediction stays
// within 17 samples of the picture).
//
// What bounds it is instructions (29 MB move for a 1920x1080 frame, 4 us): taken a sample at a time it issued
// 11.9 million and took 23 us.  Samples stay packed: taps in 16-bit pairs, the centre's by dp2a, squares by
// dp4a; the four kinds of work of a phase are dealt to the warps as one list.
constexpr int PL_TX = 64, PL_TY = 32;
constexpr int PL_SW = PL_TX / 4 + 6, PL_SY = PL_TY + 17;  // staged words X0-4 .. X0+83, rows Y0-2 .. Y0+46
constexpr int PL_PITCH = PL_SW + 1;                       // odd: a column of rows lies in 32 banks
constexpr int PL_VW = PL_TX / 4 + 2;                      // words with vertical taps, X0-4 .. X0+67
constexpr int PL_EROWS = PL_TY + 15, PL_EPITCH = PL_TX + 4;

// Four samples of a row of shorts, columns c .. c+3 of a picture w wide (c and w multiples of 4), edges
// replicated; kWide: the row is 8-byte aligned.
template <bool kWide>
__device__ __forceinline__ unsigned load_samples4(const short* row, int c, int w, bool& bad)
{
    unsigned lo, hi;
    if (c < 0 || c >= w) {
        const unsigned v = (unsigned short)row[c < 0 ? 0 : w - 1];
        lo = hi = v | v << 16;
    } else if (kWide) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(row + c));
        lo = v.x;
        hi = v.y;
    } else {
        lo = (unsigned)(unsigned short)row[c] | (unsigned)(unsigned short)row[c + 1] << 16;
        hi = (unsigned)(unsigned short)row[c + 2] | (unsigned)(unsigned short)row[c + 3] << 16;
    }
    bad |= ((lo | hi) & 0xff00ff00u) != 0u;
    return __byte_perm(lo, hi, 0x6420);
}

template <bool kWide>
__device__ __forceinline__ void stage_planes(const short* ref16, int W, int H, int X0, int Y0, unsigned* px, bool& bad)
{
    for (int i = threadIdx.x; i < PL_SY * PL_SW; i += 256) {
        const int r = i / PL_SW, c = i - r * PL_SW;
        const int y = min(max(Y0 - 2 + r - PAD, 0), H - 1);
        px[r * PL_PITCH + c] = load_samples4<kWide>(ref16 + (size_t)y * W, X0 - 4 + 4 * c - PAD, W, bad);
    }
}

__global__ void __launch_bounds__(256) k_full_planes(const JobDesc* __restrict__ job, int W, int H, int rstride,
                                                     unsigned char* __restrict__ src8, unsigned char* __restrict__ refp,
                                                     unsigned char* __restrict__ hpel, size_t plane_size,
                                                     float* __restrict__ energy, int* status)
{
    __shared__ unsigned px[PL_SY * PL_PITCH];
    __shared__ __align__(16) unsigned vt[PL_TY * 2 * PL_VW];       // vertical sums + TAP_BIAS, pairs
    __shared__ __align__(16) int hs[PL_EROWS * PL_EPITCH];         // horizontal 16-sums of squares (energy)
    const short* __restrict__ ref16 = job->ref16;
    const int PW = rstride, PH = H + 2 * PAD;
    const int X0 = blockIdx.x * PL_TX, Y0 = blockIdx.y * PL_TY, tid = threadIdx.x;
    bool bad = false;
    // 1. stage: padded (Y, X) -> frame (clamp(Y - PAD), clamp(X - PAD))
    if ((reinterpret_cast<uintptr_t>(ref16) & 7) == 0) stage_planes<true>(ref16, W, H, X0, Y0, px, bad);
    else stage_planes<false>(ref16, W, H, X0, Y0, px, bad);
    // the input's byte packing, a share per CTA (8 samples per thread step, or 4 of a less aligned input)
    {
        const int nb = (int)(gridDim.x * gridDim.y), b = (int)(blockIdx.y * gridDim.x + blockIdx.x);
        const short* src16 = job->src16;
        if ((reinterpret_cast<uintptr_t>(src16) & 15) == 0) {
            const long long n = (long long)W * H / 8;
            for (long long j = (long long)b * 256 + tid; j < n; j += (long long)nb * 256) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(src16) + j);
                bad |= ((v.x | v.y | v.z | v.w) & 0xff00ff00u) != 0u;
                reinterpret_cast<uint2*>(src8)[j] = make_uint2(__byte_perm(v.x, v.y, 0x6420), __byte_perm(v.z, v.w, 0x6420));
            }
        } else {
            const long long n = (long long)W * H / 4;
            const unsigned* s = reinterpret_cast<const unsigned*>(src16);
            for (long long j = (long long)b * 256 + tid; j < n; j += (long long)nb * 256) {
                const unsigned lo = s[2 * j], hi = s[2 * j + 1];
                bad |= ((lo | hi) & 0xff00ff00u) != 0u;
                reinterpret_cast<unsigned*>(src8)[j] = __byte_perm(lo, hi, 0x6420);
            }
        }
    }
    if (__any_sync(0xffffffffu, bad) && (tid & 31) == 0) atomicOr(status, ST_PIXEL_RANGE);
    __syncthreads();
    // 2. vertical sums of rows Y0 .. Y0+31, four rows of a word per task; horizontal 16-sums of squares of rows
    //    Y0 .. Y0+46, 16 columns per task; the bytes and the b plane, a word per task
    constexpr int kV = PL_VW * PL_TY / 4, kE0 = (kV + 31) / 32 * 32, kE = 4 * 48, kB0 = kE0 + kE;
    for (int t = tid; t < kB0 + PL_TY * PL_TX / 4; t += 256) {
        if (t < kE0) {
            if (t >= kV) continue;
            const int g = t / PL_VW, wd = t - g * PL_VW;
            unsigned ev[9], od[9];
#pragma unroll
            for (int i = 0; i < 9; i++) {
                const unsigned w = px[(4 * g + i) * PL_PITCH + wd];
                ev[i] = w & 0x00ff00ffu;
                od[i] = (w >> 8) & 0x00ff00ffu;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const unsigned te = tap_pair(ev[i], ev[i + 1], ev[i + 2], ev[i + 3], ev[i + 4], ev[i + 5]);
                const unsigned to = tap_pair(od[i], od[i + 1], od[i + 2], od[i + 3], od[i + 4], od[i + 5]);
                *reinterpret_cast<uint2*>(vt + 2 * ((4 * g + i) * PL_VW + wd)) =
                    make_uint2(__byte_perm(te, to, 0x5410), __byte_perm(te, to, 0x7632));
            }
        } else if (t < kB0) {
            const int e = t - kE0, seg = e / 48, r = e - 48 * seg;
            if (!energy || r >= PL_EROWS) continue;
            unsigned x[8];
#pragma unroll
            for (int i = 0; i < 8; i++) x[i] = px[(r + 2) * PL_PITCH + 1 + 4 * seg + i] ^ 0x80808080u;
            int out[16];
#pragma unroll
            for (int s = 0; s < 4; s++) {
                int g[7];
#pragma unroll
                for (int i = 0; i < 7; i++) {
                    const int v = (int)(s ? __funnelshift_r(x[i], x[i + 1], 8 * s) : x[i]);
                    g[i] = __dp4a(v, v, 0);
                }
                int acc = g[0] + g[1] + g[2] + g[3];
                out[s] = acc;
#pragma unroll
                for (int q = 1; q < 4; q++) {
                    acc += g[q + 3] - g[q - 1];
                    out[4 * q + s] = acc;
                }
            }
            int4* d = reinterpret_cast<int4*>(hs + r * PL_EPITCH + 16 * seg);
#pragma unroll
            for (int q = 0; q < 4; q++) d[q] = make_int4(out[4 * q], out[4 * q + 1], out[4 * q + 2], out[4 * q + 3]);
        } else {
            const int r = (t - kB0) >> 4, q = (t - kB0) & 15, Y = Y0 + r, X = X0 + 4 * q;
            if (Y >= PH || X >= PW) continue;  // PW is a multiple of 16: a word is inside or outside whole
            const unsigned* p = px + (r + 2) * PL_PITCH + q;
            unsigned te, to;
            tap_row4(p[0], p[1], p[2], te, to);
            const size_t o = (size_t)Y * rstride + X;
            *reinterpret_cast<unsigned*>(refp + o) = p[1];
            *reinterpret_cast<unsigned*>(hpel + o) = scale_pair(te) | scale_pair(to) << 8;
        }
    }
    __syncthreads();
    // 3. the h and j planes, a word per task; vertical 16-sums of the squares, 16 rows of a column per task
    constexpr int kJ = PL_TY * PL_TX / 4;
    for (int t = tid; t < kJ + PL_TX * (PL_TY / 16); t += 256) {
        if (t < kJ) {
            const int r = t >> 4, q = t & 15, Y = Y0 + r, X = X0 + 4 * q;
            if (Y >= PH || X >= PW) continue;
            const unsigned* v = vt + 2 * (r * PL_VW + q);
            const uint2 c = *reinterpret_cast<const uint2*>(v + 2), n = *reinterpret_cast<const uint2*>(v + 4);
            const size_t o = (size_t)Y * rstride + X;
            *reinterpret_cast<unsigned*>(hpel + plane_size + o) = __byte_perm(scale_pair(c.x), scale_pair(c.y), 0x6420);
            *reinterpret_cast<unsigned*>(hpel + 2 * plane_size + o) = tap_centre4(v[1], c.x, c.y, n.x, n.y);
        } else if (energy) {
            const int c = (t - kJ) & (PL_TX - 1), r0 = 16 * ((t - kJ) / PL_TX), X = X0 + c;
            int acc = 0;
#pragma unroll
            for (int d = 0; d < 16; d++) acc += hs[(r0 + d) * PL_EPITCH + c];
#pragma unroll
            for (int r = r0; r < r0 + 16; r++) {
                if (r > r0) acc += hs[(r + 15) * PL_EPITCH + c] - hs[(r - 1) * PL_EPITCH + c];
                const int Y = Y0 + r;
                if (X <= PW - 16 && Y <= PH - 16) energy[(size_t)Y * rstride + X] = (float)acc;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// c + sum over the four bytes of |a - b| (unsigned bytes): the PTX SIMD
// video instruction with its accumulate form.
__device__ __forceinline__ unsigned sad4_add(unsigned a, unsigned b, unsigned c)
{
    unsigned d;
    asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// ---------------------------------------------------------------------------
// Search stage: one persistent CTA per slot (SEARCH_CTAS_PER_SM per SM),
// macroblocks blockIdx.x, blockIdx.x + gridDim.x, ...; warp-specialised.
//
//   compute warps      the SAD (OverlayMem2Dv2::Tad16x16,
//                      OverlayMem2Dv2.cpp:2655-2730) of all (2R+1)^2 full-pel
//                      candidates of a macroblock into a shared-memory table,
//                      with its row minima; warp 0 also stages the next
//                      macroblock's window and template (TMA tensor copies)
//   scan warp (1)      the reference's sequential raster scan over each
//                      table (prediction (0, 0) for ties, Full.cpp:394-446);
//                      tables of macroblocks whose scan met an exact tie go to
//                      global memory for their tie tree; then it releases the
//                      buffer, so the compute warps wait for a scan only when
//                      it falls two tables behind
//
// Two window buffers and two table buffers; the hand-offs are shared-memory
// barriers (mbarrier) whose waits are bounded: a wait that runs out sets
// ST_TIMEOUT and every role leaves, after the copies it issued landed.
// Launch shape, measured on 1080p frames: 8 candidate rows per thread with the
// template rows in two passes of the ring's period (a loop body small enough
// for the instruction cache), at 3 CTAs per SM, where the loop needs no spills.
constexpr int SEARCH_ROWS = 8;    // candidate rows per thread (the window-row ring's period)
constexpr int SEARCH_UNROLL = 8;  // template rows per unrolled loop body (a multiple of SEARCH_ROWS)
constexpr int SEARCH_WARPS = 64 / (2 * SEARCH_ROWS);  // compute warps: 2 row groups of a warp each
constexpr int SEARCH_THREADS = 32 * (SEARCH_WARPS + 1);
constexpr int SEARCH_CTAS_PER_SM = 3;
constexpr unsigned WIN_BYTES = WROWS * WSTRIDE + 256;     // window rows + template
// one window, 128-byte aligned, with room for a row 78 that the TMA box does
// not fill (only the unused candidate row 63 reads it)
constexpr int WIN_BUF = (WROWS * WSTRIDE + WSTRIDE + 127) / 128 * 128;
static_assert(SEARCH_UNROLL % SEARCH_ROWS == 0 && 16 % SEARCH_UNROLL == 0, "unroll must cover ring periods");

struct SearchSmem {
    alignas(128) int tab[2][TAB][TAB];  // rows 0 .. 2R: SADs (column 0: row minima)
    alignas(128) unsigned char win[2][WIN_BUF];  // WROWS rows of WSTRIDE bytes
    alignas(128) unsigned char cur[2][256];
    unsigned long long wfull[2];   // window b staged
    unsigned long long wfree[2];   // window b read by every compute thread
    unsigned long long tfull[2];   // table b written by every compute thread
    unsigned long long tempty[2];  // table b released by the scan warp
    int abort;
};

// Bounded wait for the phase of parity `par`; false when the search is
// abandoned (this wait ran out, or another role's did).
__device__ __forceinline__ bool search_wait(unsigned long long* bar, unsigned par, const FullArgs& a,
                                            volatile int* abort)
{
    long long it = 0;
    while (!mbar_try_wait(bar, par)) {
        if (*abort) return false;
        if (++it > a.spin_limit) {
            atomicOr(&a.ctrl->status, ST_TIMEOUT);
            *abort = 1;
            return false;
        }
    }
    return true;
}

// Wait (bounded, abort ignored) for the stagings [from, to) on a pair of
// barriers: copies must land before the CTA leaves.
__device__ __forceinline__ void search_drain(unsigned long long* bars, int from, int to, long long limit)
{
    for (int i = from; i < to; i++) {
        long long w = 0;
        while (!mbar_try_wait(&bars[i & 1], (unsigned)(i >> 1) & 1u) && ++w <= limit) {}
    }
}

__global__ void __launch_bounds__(SEARCH_THREADS, SEARCH_CTAS_PER_SM)
    k_sad_search(FullArgs a, const __grid_constant__ SearchMaps maps)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SearchSmem& S = *reinterpret_cast<SearchSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nit = (a.nmb - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;  // grid <= nmb: at least one
    volatile int* abort = &S.abort;
    if (tid == 0) {
        for (int b = 0; b < 2; b++) {
            mbar_init(&S.wfull[b], 1);
            mbar_init(&S.wfree[b], 32 * SEARCH_WARPS);
            mbar_init(&S.tfull[b], 32 * SEARCH_WARPS);
            mbar_init(&S.tempty[b], 32);
        }
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    auto mb_of = [&](int it) { return (int)blockIdx.x + it * (int)gridDim.x; };

    if (warp < SEARCH_WARPS) {
        // ---------------- compute warps ----------------
        // warp 0 stages the window + template of iteration `it` into buffer it & 1
        auto stage_window = [&](int it) {
            if (lane == 0) {
                const int b = it & 1, k = mb_of(it);
                const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
                mbar_expect_tx(&S.wfull[b], WIN_BYTES);
                tma_load_2d(S.win[b], &maps.win, n - 32 + PAD, m - 31 + PAD, &S.wfull[b]);
                tma_load_2d(S.cur[b], &maps.cur, n, m, &S.wfull[b]);
            }
        };
        int wissued = 0;  // warp 0: windows staged for iterations 0 .. wissued-1
        if (warp == 0) {
            stage_window(0);
            wissued = 1;
        }
        const int s = lane & 3, qg = (lane >> 2) & 3, ig = 2 * warp + (lane >> 4);
        const int ii0 = SEARCH_ROWS * ig;
        int it = 0;
        for (; it < nit; it++) {
            const int b = it & 1;
            const unsigned use = (unsigned)(it >> 1) & 1u;  // parity of this buffer's use
            if (warp == 0 && it + 1 < nit) {
                // window buffer b^1 was read in iteration it-1 (its first use: free from the start)
                if (!search_wait(&S.wfree[b ^ 1], ((unsigned)((it + 1) >> 1) & 1u) ^ 1u, a, abort)) break;
                stage_window(it + 1);
                wissued = it + 2;
            }
            if (!search_wait(&S.wfull[b], use, a, abort)) break;

            // vabsdiff4 with accumulate; each thread:
            // SEARCH_ROWS candidate rows x 4 word offsets, one byte shift s.  Each window
            // row is byte-aligned once for the thread's shift (funnel shifts: word i holds
            // bytes 4i+s .. 4i+s+3 of the thread's 32-byte slice) and kept in a ring of
            // SEARCH_ROWS rows; every 16-pixel row is then 4 of them against the
            // template row.
            unsigned acc[SEARCH_ROWS][4];
            {
                unsigned al[SEARCH_ROWS][7];
                auto load_row = [&](unsigned* dst, int r) {
                    const uint4* p = reinterpret_cast<const uint4*>(&S.win[b][r * WSTRIDE + 16 * qg]);
                    const uint4 x0 = p[0], x1 = p[1];
                    const unsigned w[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                    for (int i = 0; i < 7; i++) dst[i] = __funnelshift_r(w[i], w[i + 1], 8 * s);
                };
#pragma unroll
                for (int r = 0; r < SEARCH_ROWS; r++) load_row(al[r], ii0 + r);
#pragma unroll
                for (int r = 0; r < SEARCH_ROWS; r++)
#pragma unroll
                    for (int q = 0; q < 4; q++) acc[r][q] = 0u;
#pragma unroll 1
                for (int yq = 0; yq < 16; yq += SEARCH_UNROLL) {
#pragma unroll
                    for (int yu = 0; yu < SEARCH_UNROLL; yu++) {
                        const int y = yq + yu;
                        const uint4 t = *reinterpret_cast<const uint4*>(&S.cur[b][16 * y]);
                        const unsigned A[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
                        for (int r = 0; r < SEARCH_ROWS; r++) {
                            const unsigned* B = al[(r + yu) % SEARCH_ROWS];
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                unsigned c = acc[r][q];
#pragma unroll
                                for (int w = 0; w < 4; w++) c = sad4_add(A[w], B[q + w], c);
                                acc[r][q] = c;
                            }
                        }
                        if (y < 15) load_row(al[yu % SEARCH_ROWS], ii0 + y + SEARCH_ROWS);
                    }
                }
            }
            mbar_arrive(&S.wfree[b]);  // this thread is done with window b and its template

            if (!search_wait(&S.tempty[b], use ^ 1u, a, abort)) break;  // the scan warp released the table
            const int k = mb_of(it);
            const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
            int xl, xr, yu, yd;
            full_range(n, m, a.W, a.H, a.motion_range, xl, xr, yu, yd);
#pragma unroll
            for (int r = 0; r < SEARCH_ROWS; r++) {
                const int ii = ii0 + r;
                int v[4], mn = 0x7fffffff;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int jj = 16 * qg + 4 * q + s;
                    v[q] = (int)acc[r][q];
                    const int j = jj - RMAX - 1;
                    if (j >= xl && j <= xr) mn = min(mn, v[q]);
                }
#pragma unroll
                for (int o = 1; o < 16; o <<= 1) mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                if (ii < 2 * RMAX + 1) {
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int jj = 16 * qg + 4 * q + s;
                        S.tab[b][ii][jj] = jj == 0 ? mn : v[q];  // column 0 (outside every range): the row minimum
                    }
                }
            }
            mbar_arrive(&S.tfull[b]);
        }
        if (warp == 0) search_drain(S.wfull, it, wissued, a.spin_limit);
    } else {
        // ---------------- scan warp ----------------
        int it = 0;
        for (; it < nit; it++) {
            const int b = it & 1;
            const int k = mb_of(it);
            const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
            if (!search_wait(&S.tfull[b], (unsigned)(it >> 1) & 1u, a, abort)) break;
            int xl, xr, yu, yd, mx, my, minD, tie;
            full_range(n, m, a.W, a.H, a.motion_range, xl, xr, yu, yd);
            scan_table(SmemTab{S.tab[b]}, xl, xr, yu, yd, 0, 0, lane, &mx, &my, &minD, &tie);
            const int zero_d = S.tab[b][RMAX][RMAX + 1];
            if (tie) {  // its tie tree (and deep rescans) read the table from global memory
                int4* dst = reinterpret_cast<int4*>(a.tables + (size_t)k * TAB * TAB);
                const int4* src = reinterpret_cast<const int4*>(&S.tab[b][0][0]);
                for (int i = lane; i < (2 * RMAX + 1) * TAB / 4; i += 32) __stcg(dst + i, src[i]);
            }
            __syncwarp();
            mbar_arrive(&S.tempty[b]);
            if (lane == 0) {  // the full-pel result
                const int qmv = pack_mv(4 * mx, 4 * my);
                const int av = neighbour_mask(a.job->slice, k, a.cols, a.nmb / a.cols);
                a.spec4[k] = make_int4(qmv, minD, zero_d, (tie ? FLAG_TIE : 0) | av);
                a.spec_imv[k] = pack_mv(mx, my);
                __stcg(a.final_mv + k, qmv);
                if (tie) a.tie_list[atomicAdd(&a.ctrl->ntie, 1)] = k;
            }
        }
    }
}

// The window of the candidates of kMbs macroblocks of a row, the first at
// (n, m), in shared memory: WROWS rows from m - 31, columns n - 32 ..
// n + 16 kMbs + 31.  At these pitches (22 and 34 words) 16 rows at one column,
// and the word beside it, lie in 32 different banks.
__host__ __device__ constexpr int scan_pitch(int mbs) { return 64 + 16 * mbs + 8; }

// mbs: the macroblocks that are there; nthreads: a multiple of 16.
template <int kMbs>
__device__ __forceinline__ void stage_window(const FullArgs& a, int n, int m, int mbs, unsigned char* win, int tid,
                                             int nthreads)
{
    const unsigned char* src = a.refp + (size_t)(m - RMAX + PAD) * a.rstride + n - RMAX - 1 + PAD;
    constexpr int kPieces = kMbs + 4, kAcross = 8, kPitch = scan_pitch(kMbs);  // 16-byte pieces of a row
    static_assert(kPieces <= kAcross, "a row's pieces and the idle threads beside them");
    const int q = tid & (kAcross - 1), step = nthreads / kAcross;
    if (q >= mbs + 4) return;
#pragma unroll 5
    for (int r = tid / kAcross; r < WROWS; r += step) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + (size_t)r * a.rstride + 16 * q));
        uint2* d = reinterpret_cast<uint2*>(win + r * kPitch + 16 * q);
        d[0] = make_uint2(v.x, v.y);
        d[1] = make_uint2(v.z, v.w);
    }
}

// This lane's row of the template (row lane / 2).
__device__ __forceinline__ uint4 template_row(const FullArgs& a, int n, int m, int lane)
{
    return __ldg(reinterpret_cast<const uint4*>(a.src8 + (size_t)(m + (lane >> 1)) * a.W + n));
}

// The SSDs of the 8 candidates in table columns 8g .. 8g+7 of candidate row ii
// (i + RMAX): lane c < 8 gets column 8g + c.  One warp, a lane four candidates
// on one template row, which read five words of one window row.
template <int kPitch>
__device__ __forceinline__ int group_ssd(const unsigned char* win, uint4 t, int ii, int g, int lane)
{
    const unsigned* q = reinterpret_cast<const unsigned*>(win + (ii + (lane >> 1)) * kPitch + 8 * g + 4 * (lane & 1));
    const unsigned w[5] = {q[0], q[1], q[2], q[3], q[4]}, tw[4] = {t.x, t.y, t.z, t.w};
    unsigned acc[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int s = 0; s < 4; s++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned d = __vabsdiffu4(tw[i], s ? __funnelshift_r(w[i], w[i + 1], 8 * s) : w[i]);
            acc[s] = __dp4a(d, d, acc[s]);
        }
    // over the 16 template rows; a lane keeps two, then one of its candidates: 4 (lane & 1) + 2 (bit 4) + bit 3
    const bool b4 = lane & 16, b3 = lane & 8;
    const unsigned u0 = (b4 ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, b4 ? acc[0] : acc[2], 16);
    const unsigned u1 = (b4 ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, b4 ? acc[1] : acc[3], 16);
    unsigned v = (b3 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b3 ? u0 : u1, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return (int)__shfl_sync(0xffffffffu, v, ((lane >> 2) & 1) | ((lane & 2) << 3) | ((lane & 1) << 3));
}

// The reference's integer scan of each macroblock (prediction (0, 0) for ties,
// Full.cpp:394-446, see scan_table_t) and the half-pel then quarter-pel
// refinement around its winner (Full.cpp:452-517), one warp per macroblock:
// the prediction-independent result the resolve starts from.
//
// A group of 8 candidates (a.rowmin) can accept one only if its minimum is at
// or below the running minimum and some of its columns are in range of the
// running best (the skip rule adds the best's vector to the candidate's); once
// a tie is known, one that only ties must not lie farther out than the best.  A
// lane holds the minima of two candidate rows; the first row that has such a
// minimum is visited next, and only such groups' SSDs are formed: on a 1080p
// pan 6 rows and 7.5 groups a macroblock.
//
// What bounds it is latency with too few warps to hide it.  The macroblocks of a CTA are neighbours and share
// one window (22 KB a CTA, 36 warps an SM; a window and the minima kept for each warp, 24), and the refinement
// reads its planes from shared memory: 1920x1080, 48 -> 38 us (the refinement 6 of it, the window 4).
constexpr int SCAN_WARPS = 4;
__global__ void __launch_bounds__(32 * SCAN_WARPS, 8) k_full_scan(const __grid_constant__ FullArgs a)
{
    constexpr int kPitch = scan_pitch(SCAN_WARPS);
    __shared__ __align__(16) unsigned char s_win[WROWS * kPitch];
    __shared__ __align__(16) SubWindow s_sub[SCAN_WARPS];
    const int across = (a.cols + SCAN_WARPS - 1) / SCAN_WARPS, br = blockIdx.x / across;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, bc = SCAN_WARPS * (blockIdx.x - br * across);
    const int mbs = min(SCAN_WARPS, a.cols - bc), k = br * a.cols + bc + w;
    const int n = 16 * (bc + w), m = 16 * br;
    stage_window<SCAN_WARPS>(a, 16 * bc, m, mbs, s_win, threadIdx.x, 32 * SCAN_WARPS);
    const bool there = w < mbs;
    const uint4 t = template_row(a, there ? n : 16 * bc, m, lane);
    const uint2 cur = (lane & 1) ? make_uint2(t.z, t.w) : make_uint2(t.x, t.y);
    constexpr int kNone = 0x7fffffff;
    int xl, xr, yu, yd;
    full_range(n, m, a.W, a.H, a.motion_range, xl, xr, yu, yd);
    // A^2 of the samples less 128, which the minima are without
    const int c0 = (int)(cur.x ^ 0x80808080u), c1 = (int)(cur.y ^ 0x80808080u);
    const int energy = warp_sum(__dp4a(c0, c0, __dp4a(c1, c1, 0)));
    const int ga = (xl + 32) >> 3, gb = (xr + 32) >> 3;  // groups that hold candidates
    const float* minima = a.rowmin + ((size_t)k * 64 + yu + RMAX) * 8;  // candidate row yu's
    int rm[2] = {kNone, kNone};
    if (there) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const float4* q = reinterpret_cast<const float4*>(minima + 8 * min(lane + 32 * h, yd - yu));
            const float4 p0 = __ldg(q), p1 = __ldg(q + 1);
            const float f[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int g = 0; g < 8; g++)
                if (g >= ga && g <= gb) rm[h] = min(rm[h], energy + (int)f[g]);
        }
    }
    __syncthreads();
    if (!there) return;
    const unsigned char* win = s_win + 16 * w;
    const unsigned* at0 = reinterpret_cast<const unsigned*>(win + (RMAX + (lane >> 1)) * kPitch + RMAX + 1 + 8 * (lane & 1));
    const int zero_d = warp_sum(ssd8(cur, make_uint2(at0[0], at0[1])));

    int minD = zero_d, mx = 0, my = 0, tie = 0;
    int done = 0;  // rows yu .. yu+done-1 are behind the scan
    while (true) {
        const int r0 = yu + lane + my, r1 = r0 + 32;
        unsigned m0 = __ballot_sync(0xffffffffu, rm[0] <= minD && lane >= done && r0 >= yu && r0 <= yd &&
                                                     yu + lane <= yd);
        unsigned m1 = __ballot_sync(0xffffffffu, rm[1] <= minD && lane + 32 >= done && r1 >= yu && r1 <= yd &&
                                                     yu + lane + 32 <= yd);
        if (tie) {
            const int best = my * my + mx * mx, p0 = yu + lane, p1 = p0 + 32;
            m0 &= __ballot_sync(0xffffffffu, rm[0] < minD || best >= p0 * p0);
            m1 &= __ballot_sync(0xffffffffu, rm[1] < minD || best >= p1 * p1);
        }
        if (!m0 && !m1) break;
        const int off = m0 ? __ffs(m0) - 1 : 31 + __ffs(m1), i = yu + off;
        done = off + 1;
        const int gl = lane & 7, jl = 8 * gl - 32;  // lane g: the row's group g
        const int gmin = gl >= ga && gl <= gb ? energy + (int)__ldg(minima + 8 * off + gl) : kNone;
        unsigned left = 0xffu;  // groups not yet behind the scan
        while (i + my >= yu && i + my <= yd) {
            // the next group of the row that can accept, at the best as it is
            unsigned can = __ballot_sync(0xffffffffu, gmin <= minD && jl + 7 + mx >= xl && jl + mx <= xr) & left;
            if (tie) {
                const int jn = max(max(jl, -jl - 7), 0);  // the group's distance from column 0
                can &= __ballot_sync(0xffffffffu, gmin < minD || my * my + mx * mx >= i * i + jn * jn);
            }
            if (!can) break;
            const int g = __ffs(can) - 1;
            left &= ~((2u << g) - 1u);
            const int d = group_ssd<kPitch>(win, t, i + RMAX, g, lane);
            const int base = 8 * g - 32, j = base + lane;
            const bool valid = lane < 8 && j >= xl && j <= xr && !(i == 0 && j == 0);
            scan_piece(valid, d, i, j, base, xl, xr, yu, yd, 0, 0, minD, mx, my, tie);
        }
    }
    int qmx, qmy;
    subpel_refine_staged(a, s_sub[w], n, m, n + mx, m + my, lane, &minD, &qmx, &qmy);
    if (lane == 0) {
        const int qmv = pack_mv(4 * mx + qmx, 4 * my + qmy);
        const int av = neighbour_mask(a.job->slice, k, a.cols, a.nmb / a.cols);
        a.spec4[k] = make_int4(qmv, minD, zero_d, (tie ? FLAG_TIE : 0) | av);
        a.spec_imv[k] = pack_mv(mx, my);
        __stcg(a.final_mv + k, qmv);
        if (tie) a.tie_list[atomicAdd(&a.ctrl->ntie, 1)] = k;
    }
}

// ---------------------------------------------------------------------------
// Tie trees of the listed macroblocks (see TieRun), one CTA per MB: the table
// in shared memory (kSad: the search kept it; else formed here, warp p the rows
// p, p + 8, ..), warp p computes run p (forced scan, then the sub-pel stage of
// its winner when that is not the searched one).  FLAG_DEEP when a run
// reachable by some prediction met more ties than the tree holds (the
// prediction-dependent stage then rescans the kept table).
struct TieSmem {
    alignas(16) int tab[TAB][TAB];
    int run[TIE_RUNS][sizeof(TieRun) / sizeof(int)];
    int deep;
    alignas(16) unsigned char win[WROWS * scan_pitch(1)];
};

// The SSD table is made by more warps than have a run: a handful of macroblocks met a tie, so what counts is how
// long one takes (1920x1080, 17 of them, profiled: 22 us with 8 warps, 18 with 32).
constexpr int TIE_WARPS_SSD = 32;
template <bool kSad>
__global__ void __launch_bounds__(kSad ? TIE_RUNS * 32 : TIE_WARPS_SSD * 32) k_full_tietree(const __grid_constant__ FullArgs a)
{
    extern __shared__ __align__(16) unsigned char tie_smem[];
    TieSmem& S = *reinterpret_cast<TieSmem*>(tie_smem);
    const int tid = threadIdx.x, lane = tid & 31, p = tid >> 5;
    const int ntie = *((volatile int*)&a.ctrl->ntie);
    constexpr int kWords = (2 * RMAX + 1) * TAB / 4;
    for (int t = blockIdx.x; t < ntie; t += gridDim.x) {
        const int k = a.tie_list[t];
        const int n = (k % a.cols) * 16, m = (k / a.cols) * 16;
        int* gt = a.tables + (size_t)k * TAB * TAB;
        int xl, xr, yu, yd;
        full_range(n, m, a.W, a.H, a.motion_range, xl, xr, yu, yd);
        if constexpr (kSad) {
            for (int i = tid; i < kWords; i += blockDim.x)
                reinterpret_cast<int4*>(&S.tab[0][0])[i] = __ldcg(reinterpret_cast<const int4*>(gt) + i);
        } else {
            const uint4 tm = template_row(a, n, m, lane);
            stage_window<1>(a, n, m, 1, S.win, tid, blockDim.x);
            __syncthreads();
            for (int i = p; i < (2 * RMAX + 1) * (TAB / 8); i += TIE_WARPS_SSD) {
                const int ii = i / (TAB / 8), g = i % (TAB / 8), v = group_ssd<scan_pitch(1)>(S.win, tm, ii, g, lane);
                if (lane < 8) S.tab[ii][8 * g + lane] = v;
            }
            __syncthreads();
            table_row_minima(S.tab, xl, xr, yu, yd, p, TIE_WARPS_SSD, lane);
        }
        __syncthreads();
        const int4 sp = a.spec4[k];
        const int imv = a.spec_imv[k];
        if (kSad || p < TIE_RUNS) {
            int rmx, rmy, rmin, rt, nev, ev[TIE_DEPTH] = {0, 0, 0};
            scan_table_t<true>(SmemTab{S.tab}, xl, xr, yu, yd, 0, 0, p, lane, &rmx, &rmy, &rmin, &rt, &nev, ev);
            int rq = sp.x, rqmin = sp.y;
            if (nev >= 0 && (rmx != mv_x(imv) || rmy != mv_y(imv))) {  // (deeper runs are not read)
                int sx = 0, sy = 0;
                if (!kSad) subpel_refine_planes(a, n + rmx, m + rmy, load_cur8(a, n, m, lane), lane, &rmin, &sx, &sy);
                rq = pack_mv(4 * rmx + sx, 4 * rmy + sy);
                rqmin = rmin;
            }
            if (lane == 0) {
                S.run[p][0] = ev[0];
                S.run[p][1] = ev[1];
                S.run[p][2] = ev[2];
                S.run[p][3] = nev;
                S.run[p][4] = rq;
                S.run[p][5] = rqmin;
            }
        }
        __syncthreads();
        constexpr int RW = sizeof(TieRun) / sizeof(int);
        if (tid < TIE_RUNS * RW) gt[TIE_ROW * TAB + tid] = S.run[tid / RW][tid % RW];
        if (tid == 0) {
            // runs a prediction can reach: run p needs tie hb(p) met on the path of p without that bit
            bool reach[TIE_RUNS];
            bool deep = S.run[0][3] < 0;
            reach[0] = true;
            for (int q = 1; q < TIE_RUNS; q++) {
                const int hb = 31 - __clz(q), par = q & ~(1 << hb);
                const int pn = S.run[par][3] < 0 ? TIE_DEPTH + 1 : S.run[par][3];
                reach[q] = reach[par] && pn > hb;
                deep |= reach[q] && S.run[q][3] < 0;
            }
            if (deep) a.spec4[k].w = sp.w | FLAG_DEEP;
            S.deep = deep;
        }
        __syncthreads();
        if (!kSad && S.deep)
            for (int i = tid; i < kWords; i += blockDim.x)
                __stcg(reinterpret_cast<int4*>(gt) + i, reinterpret_cast<const int4*>(&S.tab[0][0])[i]);
        __syncthreads();
    }
}

// The words an estimate starts from: its job, the counters at zero.
__global__ void __launch_bounds__(256) k_set_job(JobDesc* dst, JobDesc v, int* ctrl, int* changed, int nchanged)
{
    if (threadIdx.x == 0) *dst = v;
    if (ctrl)
        for (int i = threadIdx.x; i < (int)(sizeof(MeCtrl) / sizeof(int)); i += 256) ctrl[i] = 0;
    for (int i = threadIdx.x; i < nchanged; i += 256) changed[i] = 0;
}

}  // namespace

int set_job(vppgpu_ctx* ctx, JobDesc* d_job, const JobDesc& v, MeCtrl* ctrl, int* changed, int nchanged)
{
    static_assert(sizeof(MeCtrl) % sizeof(int) == 0, "cleared by words");
    k_set_job<<<1, 256, 0, ctx->stream>>>(d_job, v, reinterpret_cast<int*>(ctrl), changed, nchanged);
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

int full_planes_launch(vppgpu_ctx* ctx, const FullArgs& args)
{
    const int PW = args.W + 2 * PAD, PH = args.H + 2 * PAD;
    dim3 grid((PW + PL_TX - 1) / PL_TX, (PH + PL_TY - 1) / PL_TY);
    k_full_planes<<<grid, 256, 0, ctx->stream>>>(args.job, args.W, args.H, args.rstride, (unsigned char*)args.src8,
                                                 (unsigned char*)args.refp, (unsigned char*)args.hpel, args.plane_size,
                                                 const_cast<float*>(args.energy), &args.ctrl->status);
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

namespace {

// The search's grid: SEARCH_CTAS_PER_SM persistent CTAs per SM, at most one per macroblock.
int search_grid(const vppgpu_ctx* ctx, int nmb)
{
    const int g = ctx->sm_count * SEARCH_CTAS_PER_SM;
    return nmb < g ? nmb : g;
}

PFN_cuTensorMapEncodeTiled_v12000 g_encode_tiled = nullptr;
std::once_flag g_encode_once;

// A 2-D tiled map over a row-major plane: width x height elements of
// `elem` bytes, `pitch` bytes per row, boxes of box_w x box_h elements, no
// swizzle (the box lands as box_h packed rows).
int encode_2d(CUtensorMap* map, const void* base, CUtensorMapDataType type, int elem, int width, int height,
              size_t pitch, int box_w, int box_h)
{
    std::call_once(g_encode_once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    if (!g_encode_tiled) return VPPGPU_ERR_NO_DEVICE;
    if (((uintptr_t)base & 15) || (pitch & 15) || ((size_t)box_w * elem) % 16) return VPPGPU_ERR_INVALID_ARG;
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)height};
    const cuuint64_t strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = g_encode_tiled(map, type, 2, const_cast<void*>(base), dims, strides, box, estr,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? VPPGPU_OK : VPPGPU_ERR_CUDA;
}

}  // namespace

int search_maps_encode(const FullArgs& a, SearchMaps* maps)
{
    memset(maps, 0, sizeof(*maps));
    const int PW = a.W + 2 * PAD, PH = a.H + 2 * PAD;
    int rc = encode_2d(&maps->win, a.refp, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, PW, PH, (size_t)a.rstride, WSTRIDE, WROWS);
    if (!rc) rc = encode_2d(&maps->cur, a.src8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, a.W, a.H, (size_t)a.W, 16, 16);
    return rc;
}

int full_launch(vppgpu_ctx* ctx, const FullArgs& args, int nmb, cudaEvent_t* ev)
{
    if (ev) VPP_CUDA(cudaEventRecord(ev[0], ctx->stream));
    int rc = full_planes_launch(ctx, args);  // with the block energies (args.energy)
    if (rc) return rc;
    if (ev) VPP_CUDA(cudaEventRecord(ev[1], ctx->stream));
    if ((rc = rowmin_launch(ctx, args))) return rc;
    if (ev) VPP_CUDA(cudaEventRecord(ev[2], ctx->stream));
    k_full_scan<<<(args.cols + SCAN_WARPS - 1) / SCAN_WARPS * (nmb / args.cols), 32 * SCAN_WARPS, 0, ctx->stream>>>(args);
    VPP_CHECK_LAUNCH(ctx);
    // as many CTAs as can have a macroblock: on flat or letterboxed content most of them tie
    k_full_tietree<false><<<min(ctx->sm_count, nmb), TIE_WARPS_SSD * 32, sizeof(TieSmem), ctx->stream>>>(args);
    VPP_CHECK_LAUNCH(ctx);
    if (ev) VPP_CUDA(cudaEventRecord(ev[3], ctx->stream));
    if ((rc = full_resolve_launch(ctx, args, 0))) return rc;
    if (ev) VPP_CUDA(cudaEventRecord(ev[4], ctx->stream));
    return VPPGPU_OK;
}

// The integer-pel SAD stage (FullArgs::intpel): planes, the SAD search (table,
// scan at prediction (0, 0), no sub-pel), tie trees, then the resolve.
int sad_launch(vppgpu_ctx* ctx, const FullArgs& args, const SearchMaps& maps, int nmb)
{
    int rc = full_planes_launch(ctx, args);
    if (rc) return rc;
    k_sad_search<<<search_grid(ctx, nmb), SEARCH_THREADS, sizeof(SearchSmem), ctx->stream>>>(args, maps);
    VPP_CHECK_LAUNCH(ctx);
    k_full_tietree<true><<<ctx->sm_count, TIE_RUNS * 32, sizeof(TieSmem), ctx->stream>>>(args);
    VPP_CHECK_LAUNCH(ctx);
    return sad_resolve_launch(ctx, args);
}

int full_prepare(vppgpu_ctx* ctx)
{
    VPP_CUDA(cudaFuncSetAttribute(k_sad_search, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SearchSmem)));
    VPP_CUDA(cudaFuncSetAttribute(k_full_tietree<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(TieSmem)));
    VPP_CUDA(cudaFuncSetAttribute(k_full_tietree<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(TieSmem)));
    int rc = rowmin_prepare();
    return rc ? rc : full_resolve_prepare(ctx);
}

}  // namespace vppgpu
