// me_mrc_search.cuh -- the macroblock search of the multi-resolution H.264
// estimators, shared by MotionEstimatorH264ImplMultiresCross and
// MotionEstimatorH264ImplMultiresCrossVer2 (me_mrc.cu) and by the
// prediction-dependent resolve (me_full_resolve.cu), which searches a
// Ver2 macroblock again when a tie makes its search depend on the prediction.
//
// The reference reads its extended-boundary level copies (borders 19 / 9 / 5)
// through overlays whose origins are clamped (OverlayExtMem2Dv2::SetOrigin)
// and, for the sub-pel window, past the overlay edge as flat row-major memory
// (a column beyond the row continues on the next row).  The device copies
// keep exactly that flat geometry, so the same addresses hold the same
// samples; a read outside a copy sets an error instead of reading.
//
// One warp searches one macroblock, and what bounds it is instructions issued.  Scored a candidate at a
// time over the warp, with a shuffle chain and a ballot for each partial distortion and the sub-pel window
// in shorts, a MultiresCross macroblock took 11.7 thousand (a 1280x720 frame 62 us; the Multires search of a
// 1920x1080 frame 174 us, its tie trees 60).  But a candidate's decision needs only two numbers of its own,
// its distortion and the smallest minimum that no phase of it rejects (phase_limit), so the candidates of
// an integer stage are scored independently, a lane each with packed bytes, and then settled in their order
// against the running minimum (settle); the sub-pel stages give a candidate four lanes, and their window
// is made two samples at a time: 3.5 thousand instructions, 20 us; 37 and 20 us.
#pragma once

#include "me_common.cuh"
#include "me_internal.h"

namespace vppgpu {
namespace mrc {
namespace {

constexpr int MRC_NOISE_FLOOR = 512;

struct Buf {
    const unsigned char* p;
    int w, h;  // flat row-major geometry
};

struct MrcArgs {
    int W, H, cols, nmb, rows_all, mode, motion_range;
    double lambda;  // MultiresCrossVer2's Lagrangian overload: its lambda
    Buf in0, in1, in2, e0, e1, e2;
    const unsigned char* incl;
    int* out_mv;
    int* out_dist;
    long long* out_avg;
    MeCtrl* ctrl;
};

// Overlay origin (OverlayMem2Dv2::SetOrigin / OverlayExtMem2Dv2::SetOrigin):
// buffer coordinates of block (x, y), clamped so that the block fits.
struct Org {
    int x, y;
};
__device__ __forceinline__ Org origin(const Buf& b, int bw, int bh, int eb, int x, int y)
{
    x += eb;
    y += eb;
    x = x < 0 ? 0 : (x > b.w - bw ? b.w - bw : x);
    y = y < 0 ? 0 : (y > b.h - bh ? b.h - bh : y);
    return Org{x, y};
}

// Flat read, as the reference addresses its buffers.
__device__ __forceinline__ int rd(const Buf& b, int r, int c, bool& bad)
{
    // level copies hold fewer than 2^31 samples; reads stay within a few rows of a
    // copy, so the flat index cannot overflow and a negative one compares as huge
    const unsigned f = (unsigned)(r * b.w + c);
    if (f >= (unsigned)(b.w * b.h)) {
        bad = true;
        return 0;
    }
    return __ldg(b.p + f);
}

// GetMotionRange of the multi-resolution estimators (…MultiresCross.cpp:1195-1262).
struct Level {
    int boundary, width, height, vec_range;
};
__device__ __forceinline__ void mr_range(const Level& L, int xpos, int ypos, int xoff, int yoff, int range, int& xl,
                                         int& xr, int& yu, int& yd)
{
    const int x = xpos + xoff, y = ypos + yoff, vr = L.vec_range;
    const int xlr = (xoff - range > -vr) ? range : (vr - 1) + xoff;
    const int xrr = (xoff + range < vr) ? range : (vr - 1) - xoff;
    const int yur = (yoff - range > -vr) ? range : (vr - 1) + yoff;
    const int ydr = (yoff + range < vr) ? range : (vr - 1) - yoff;
    xl = (x - xlr >= -L.boundary) ? -xlr : -(x + L.boundary);
    xr = (x + xrr < L.width) ? xrr : L.width - x;
    yu = (y - yur >= -L.boundary) ? -yur : -(y + L.boundary);
    yd = (y + ydr < L.height) ? ydr : L.height - y;
}

// ---------------------------------------------------------------------------
// Phase order of the partial distortion (OverlayMem2Dv2.cpp:79-80), p = 1..16: phase p sums the squared
// differences at rows phase_row + 4i, columns phase_col + 4j of the block, so the sixteen phases are the
// sixteen classes (row mod 4, column mod 4).  PartialLessThan rejects a candidate at the first phase with
// 16 * D_p > p * min (D_p: the sum of phases 1..p), with a value above min, and otherwise returns D_16.
// Whether any phase rejects is thus decided by one number of the candidate, the largest ceil(16 * D_p / p):
// it is accepted exactly when that is at most min.  s: the class sums, [4 * row + column].  (16 * D_16 of
// a 16x16 block of bytes is below 2^29.)
__device__ __forceinline__ void phase_limit(const unsigned (&s)[16], int& d, int& t)
{
    constexpr int kRow[16] = {0, 2, 0, 2, 1, 3, 1, 3, 0, 2, 1, 3, 0, 2, 1, 3};
    constexpr int kCol[16] = {0, 2, 2, 0, 1, 3, 3, 1, 1, 3, 0, 2, 3, 1, 2, 0};
    unsigned run = 0, top = 0;
#pragma unroll
    for (int p = 1; p <= 16; p++) {
        run += s[4 * kRow[p - 1] + kCol[p - 1]];
        top = max(top, (16u * run + (unsigned)(p - 1)) / (unsigned)p);
    }
    d = (int)run;
    t = (int)top;
}

// N words of a row of samples from any byte address: the aligned words around them.  Reads up to four
// bytes past them and three before, which stay inside the levels' scratch.
template <int N>
__device__ __forceinline__ void row_words(const unsigned char* p, unsigned (&w)[N])
{
    const unsigned* q = reinterpret_cast<const unsigned*>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)3);
    const unsigned sh = (unsigned)(reinterpret_cast<uintptr_t>(p) & 3) * 8;
    unsigned lo = __ldg(q);
#pragma unroll
    for (int i = 0; i < N; i++) {
        const unsigned hi = __ldg(q + i + 1);
        w[i] = __funnelshift_r(lo, hi, sh);
        lo = hi;
    }
}

// Squares of the bytes of four words of absolute differences, summed by byte position.
__device__ __forceinline__ void add_classes(unsigned d0, unsigned d1, unsigned d2, unsigned d3, unsigned* s)
{
    const unsigned a = __byte_perm(d0, d1, 0x5140), b = __byte_perm(d2, d3, 0x5140);
    const unsigned c = __byte_perm(d0, d1, 0x7362), e = __byte_perm(d2, d3, 0x7362);
    const unsigned k0 = __byte_perm(a, b, 0x5410), k1 = __byte_perm(a, b, 0x7632);
    const unsigned k2 = __byte_perm(c, e, 0x5410), k3 = __byte_perm(c, e, 0x7632);
    s[0] = __dp4a(k0, k0, s[0]);
    s[1] = __dp4a(k1, k1, s[1]);
    s[2] = __dp4a(k2, k2, s[2]);
    s[3] = __dp4a(k3, k3, s[3]);
}

// What a warp's search keeps in shared memory: the input blocks of levels 1 and 0, and the level-0
// reference around the centre of the last integer stage, rows and columns -5..+20 (22 with the word
// padding) of its block: all that the +-2 refinement and the sub-pel window of any of its winners read.
// Samples outside the copy are 0.
constexpr int WPITCH = 7;                   // words per row
constexpr int WROWS = 26;
struct Window {
    uint4 cur[16];
    uint2 cur1[8];
    unsigned win[WROWS * WPITCH + 2];  // (+2: the whole is a multiple of 16 bytes)
};
static_assert(sizeof(Window) % 16 == 0, "what a Lattice adds follows it at once");
// The sub-pel window (LoadHalfQuartPelWindow, …MultiresCross.cpp:1281-1349) as a lattice of 22 x 22 points
// (fr, fc), each with the four even quarter samples G (0,0), h (2,0), b (0,2), j (2,2); the block's sample
// (r, c) is point (3 + r, 3 + c).  h, b and j are byte planes of rows 2..19 in the window's columns; G is the
// window itself.  The reference scales h and b and copies G for rows and columns 2..18 only, which leaves
// (MultiresCross, Multires) the raw b in row 19, the raw h in column 19 and zeros for G there: raw holds h
// (rows 2..18) and row19 b, both + TAP_BIAS.  Ver2 completes that row and column.
constexpr int SUB_PLANE = 18 * WPITCH;
struct Lattice : Window {
    unsigned sub[3 * SUB_PLANE];            // h, b, j: row fr - 2
    unsigned raw[17 * 2 * WPITCH];          // pairs of shorts
    unsigned row19[2 * WPITCH];
};

// Words of 16 samples from byte column `col` of a row of the window or of a plane.
__device__ __forceinline__ void window_row(const unsigned* row, int col, unsigned (&w)[4])
{
    const unsigned* q = row + (col >> 2);
    const unsigned sh = (unsigned)(col & 3) * 8;
    unsigned lo = q[0];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned hi = q[i + 1];
        w[i] = __funnelshift_r(lo, hi, sh);
        lo = hi;
    }
}

// Distortion of the zero vector, the input block kept in L.cur on the way: lane = half a row.
__device__ __forceinline__ int zero_distortion(const MrcArgs& a, Window& L, Org oi, int n, int m, int lane)
{
    const int r = lane >> 1, c = 8 * (lane & 1);
    const Org o = origin(a.e0, 16, 16, 19, n, m);
    unsigned x[2], y[2];
    row_words(a.in0.p + (size_t)(oi.y + r) * a.in0.w + oi.x + c, x);
    row_words(a.e0.p + (size_t)(o.y + r) * a.e0.w + o.x + c, y);
    reinterpret_cast<uint2*>(L.cur)[lane] = make_uint2(x[0], x[1]);
    const unsigned d0 = __vabsdiffu4(x[0], y[0]), d1 = __vabsdiffu4(x[1], y[1]);
    return warp_sum((int)__dp4a(d1, d1, __dp4a(d0, d0, 0u)));
}

// Stage the window around block o of the level-0 copy: eight lanes a row, an aligned word each, joined
// with the next lane's.
__device__ __forceinline__ void stage_level0(const Buf& e0, Window& L, Org o, int lane)
{
    const int first = (o.y - 5) * e0.w + o.x - 5, size = e0.w * e0.h;
    if (first >= 0 && first + (WROWS - 1) * e0.w + 4 * WPITCH <= size) {
        const int wd = lane & 7;
#pragma unroll
        for (int i = 0; i < (WROWS + 3) / 4; i++) {
            const int r = min(4 * i + (lane >> 3), WROWS - 1);
            const uintptr_t u = reinterpret_cast<uintptr_t>(e0.p + first + r * e0.w);
            const unsigned v = __ldg(reinterpret_cast<const unsigned*>(u & ~(uintptr_t)3) + wd);
            const unsigned w = __funnelshift_r(v, __shfl_down_sync(0xffffffffu, v, 1), (unsigned)(u & 3) * 8);
            if (wd < WPITCH) L.win[r * WPITCH + wd] = w;
        }
    } else {
        for (int i = lane; i < WROWS * WPITCH; i += 32) {
            const int r = i / WPITCH, f = first + r * e0.w + 4 * (i - r * WPITCH);
            unsigned w = 0;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((unsigned)(f + k) < (unsigned)size) w |= (unsigned)__ldg(e0.p + f + k) << (8 * k);
            L.win[i] = w;
        }
    }
    __syncwarp();
}

// One lane's candidate: its distortion d and limit t (kPartial: phase_limit; else t = d).
__device__ __forceinline__ int score4(const unsigned (&cur)[4], const Buf& e, Org o)
{
    unsigned d = 0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        unsigned w[1];
        row_words(e.p + (size_t)(o.y + r) * e.w + o.x, w);
        const unsigned x = __vabsdiffu4(cur[r], w[0]);
        d = __dp4a(x, x, d);
    }
    return (int)d;
}

template <bool kPartial>
__device__ __forceinline__ void score8(const Window& L, const Buf& e, Org o, int& d, int& t)
{
    const unsigned char* p = e.p + (size_t)o.y * e.w + o.x;
    unsigned s[16] = {0u};
#pragma unroll
    for (int r = 0; r < 4; r++) {
        unsigned w[2], x[2];
        row_words(p + (size_t)r * e.w, w);
        row_words(p + (size_t)(r + 4) * e.w, x);
        const uint2 c = L.cur1[r], f = L.cur1[r + 4];
        const unsigned d0 = __vabsdiffu4(c.x, w[0]), d1 = __vabsdiffu4(c.y, w[1]);
        const unsigned d2 = __vabsdiffu4(f.x, x[0]), d3 = __vabsdiffu4(f.y, x[1]);
        if (kPartial) add_classes(d0, d1, d2, d3, s + 4 * r);
        else s[0] = __dp4a(d3, d3, __dp4a(d2, d2, __dp4a(d1, d1, __dp4a(d0, d0, s[0]))));
    }
    if (kPartial) phase_limit(s, d, t);
    else t = d = (int)s[0];
}

template <bool kPartial>
__device__ __forceinline__ void score16(const Window& L, int row, int col, int& d, int& t)
{
    unsigned s[16] = {0u};
#pragma unroll 1
    for (int i = 0; i < 16; i += 4)
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const uint4 c = L.cur[i + r];
            unsigned w[4];
            window_row(L.win + (row + i + r) * WPITCH, col, w);
            const unsigned d0 = __vabsdiffu4(c.x, w[0]), d1 = __vabsdiffu4(c.y, w[1]);
            const unsigned d2 = __vabsdiffu4(c.z, w[2]), d3 = __vabsdiffu4(c.w, w[3]);
            if (kPartial) add_classes(d0, d1, d2, d3, s + 4 * r);
            else s[0] = __dp4a(d3, d3, __dp4a(d2, d2, __dp4a(d1, d1, __dp4a(d0, d0, s[0]))));
        }
    if (kPartial) phase_limit(s, d, t);
    else t = d = (int)s[0];
}

// Decide the warp's candidates in lane order against the running minimum: a lane's candidate v (a packed
// offset) replaces it when its limit t is at most min, an equal distortion only if tie(x, y) returns
// false.  tie and take are called with the same arguments in every lane.
template <typename Tie, typename Take>
__device__ __forceinline__ void settle(bool valid, int d, int t, int v, int& min, Tie&& tie, Take&& take)
{
    unsigned todo = __ballot_sync(0xffffffffu, valid && t <= min);
    while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        const int dl = __shfl_sync(0xffffffffu, d, l), vl = __shfl_sync(0xffffffffu, v, l);
        if (dl == min) {
            if (tie(mv_x(vl), mv_y(vl))) continue;
        } else {
            min = dl;
            todo &= __ballot_sync(0xffffffffu, t <= dl);
        }
        take(mv_x(vl), mv_y(vl), dl);
    }
}

// A full search of the offsets [xl, xr] x [yu, yd] in raster order, the centre's distortion first, which
// starts the minimum.  score(x, y, d, t): a lane's candidate.
template <typename Score, typename Tie, typename Take>
__device__ __forceinline__ void raster(int xl, int xr, int yu, int yd, int& min, int lane, Score&& score, Tie&& tie,
                                       Take&& take)
{
    const int nx = xr - xl + 1, ny = yd - yu + 1, n = nx > 0 && ny > 0 ? nx * ny : 0;
    for (int e0 = 0; e0 <= n; e0 += 32) {
        const int e = e0 + lane - 1;  // -1: the centre
        const bool in = e >= 0 && e < n;
        const int r = in ? (int)((unsigned)e / (unsigned)nx) : 0;
        const int j = in ? xl + e - r * nx : 0, i = in ? yu + r : 0;
        int d, t;
        score(j, i, d, t);
        if (e0 == 0) min = __shfl_sync(0xffffffffu, d, 0);
        settle(in && (i || j), d, t, pack_mv(j, i), min, tie, take);
    }
}

// The four offsets of a cross step in the estimators' order: left, right, up, down.
__device__ __forceinline__ void cross_offset(int lane, int s, int& j, int& i)
{
    const int v = (lane & 1) ? s : -s;
    j = (lane & 2) ? 0 : v;
    i = (lane & 2) ? v : 0;
}

// The lattice whose row 0 is the window's row wy; its column 0 may be any of the window's columns 0..4.
template <bool kVer2>
__device__ __forceinline__ void build_lattice(Lattice& L, int wy, int lane)
{
    constexpr unsigned m = 0x00ff00ffu;
    unsigned *h = L.sub, *b = L.sub + SUB_PLANE, *jp = L.sub + 2 * SUB_PLANE;
    if (lane < 4 * WPITCH) {  // h, rows 2..18: a word column and five rows per lane
        const int g = lane / WPITCH, wd = lane - g * WPITCH;
        unsigned ev[10], od[10];
#pragma unroll
        for (int i = 0; i < 10; i++) {
            const unsigned w = L.win[(wy + 4 * g + i) * WPITCH + wd];
            ev[i] = w & m;
            od[i] = (w >> 8) & m;
        }
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const unsigned te = tap_pair(ev[i], ev[i + 1], ev[i + 2], ev[i + 3], ev[i + 4], ev[i + 5]);
            const unsigned to = tap_pair(od[i], od[i + 1], od[i + 2], od[i + 3], od[i + 4], od[i + 5]);
            const int at = (4 * g + i) * WPITCH + wd;
            L.raw[2 * at] = __byte_perm(te, to, 0x5410);
            L.raw[2 * at + 1] = __byte_perm(te, to, 0x7632);
            h[at] = scale_pair(te) | scale_pair(to) << 8;
        }
    }
    for (int i = lane; i < 18 * 6; i += 32) {  // b, rows 2..19: words 0..5 hold its columns 2..18
        const int r = i / 6, wd = i - 6 * r;
        const unsigned* q = L.win + (wy + 2 + r) * WPITCH + wd;
        unsigned te, to;
        tap_row4(wd ? q[-1] : 0u, q[0], q[1], te, to);
        b[r * WPITCH + wd] = scale_pair(te) | scale_pair(to) << 8;
        if (!kVer2 && r == 17) {
            L.row19[2 * wd] = __byte_perm(te, to, 0x5410);
            L.row19[2 * wd + 1] = __byte_perm(te, to, 0x7632);
        }
    }
    __syncwarp();
    for (int i = lane; i < 17 * 6; i += 32) {  // j, rows 2..18, from the raw h
        const int r = i / 6, wd = i - 6 * r;
        const unsigned* q = L.raw + 2 * (r * WPITCH + wd);
        jp[r * WPITCH + wd] = tap_centre4(wd ? q[-1] : 0u, q[0], q[1], q[2], q[3]);
    }
    __syncwarp();
}

// Where the samples of even quarter point (qr, qc) lie for block sample (0, 0): the word of the lattice
// their row starts at, and the byte column.
struct Point {
    int word, col;
};
__device__ __forceinline__ Point lattice_point(int wy, int wx, int qr, int qc)
{
    constexpr int win = 16 * 4 + 8 * 2, sub = (int)sizeof(Window) / 4;
    const int plane = ((qr >> 1) & 1) | (qc & 2);  // G, h, b, j
    const int fr = qr >> 2;
    return Point{plane ? sub + (plane - 1) * SUB_PLANE + (fr - 2) * WPITCH : win + (wy + fr) * WPITCH, wx + (qc >> 2)};
}

// Of the four lanes of a candidate, each with the class sums of one row class: settle the eight
// candidates (v, the lane's), strict improvements.
template <bool kPartial, typename Take>
__device__ __forceinline__ void settle_quads(const unsigned (&s)[4], int v, int& min, int lane, Take&& take)
{
    int d = (int)(s[0] + s[1] + s[2] + s[3]);
    d += __shfl_xor_sync(0xffffffffu, d, 1);
    d += __shfl_xor_sync(0xffffffffu, d, 2);
    if (!__any_sync(0xffffffffu, d < min)) return;
    int t = d;
    if (kPartial) {
        unsigned all[16];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) all[4 * r + c] = __shfl_sync(0xffffffffu, s[c], (lane & 28) | r);
        phase_limit(all, d, t);
    }
    settle((lane & 3) == 0 && d < min, d, t, v, min, [](int, int) { return true; }, take);
}

__device__ __forceinline__ int byte_of(unsigned w, int k) { return (int)((w >> (8 * k)) & 0xffu); }
__device__ __forceinline__ int raw_of(const unsigned* w, int i)
{
    return (int)reinterpret_cast<const unsigned short*>(w)[i] - TAP_BIAS;
}

// Half then quarter pel in the estimator's window around block o (…MultiresCross.cpp:875-941), strict
// improvements: eight candidates of a pass at once, four lanes each (a row class per lane).  The quarter
// samples are the averages of two even ones that LoadQuartPelWindow (…MultiresCross.cpp:1365-1389) pairs.
// take(qx, qy, d): an accepted quarter-pel offset.
template <bool kVer2, bool kPartial, typename Take>
__device__ __forceinline__ void subpel(Lattice& L, const Buf& e0, Org oc, Org o, int& min_d, int& qmx, int& qmy,
                                       int lane, bool& bad, Take&& take)
{
    const int wy = o.y - oc.y + 2, wx = o.x - oc.x + 2;
    // the reference reads the samples of all 22 x 22 points
    bad |= (o.y - 3) * e0.w + o.x - 3 < 0 || (o.y + 18) * e0.w + o.x + 18 >= e0.w * e0.h;
    build_lattice<kVer2>(L, wy, lane);
    const unsigned* words = reinterpret_cast<const unsigned*>(&L);
    const int rho = lane & 3, c9 = (lane >> 2) + (lane >= 16), sy = c9 / 3 - 1, sx = c9 - 3 * (c9 / 3) - 1;
    {
        const Point a = lattice_point(wy, wx, 12 + 2 * sy, 12 + 2 * sx);
        unsigned s[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = rho + 4 * i;
            const uint4 c = L.cur[r];
            unsigned w[4];
            window_row(words + a.word + r * WPITCH, a.col, w);
            add_classes(__vabsdiffu4(c.x, w[0]), __vabsdiffu4(c.y, w[1]), __vabsdiffu4(c.z, w[2]),
                        __vabsdiffu4(c.w, w[3]), s);
        }
        settle_quads<kPartial>(s, pack_mv(2 * sx, 2 * sy), min_d, lane, [&](int x, int y, int d) {
            qmx = x;
            qmy = y;
            take(x, y, d);
        });
    }
    const int hmx = qmx, hmy = qmy, qr = 12 + hmy, qc = 12 + hmx;
    Point a, b;
    if (sy == 0) {
        a = lattice_point(wy, wx, qr, qc + 2 * sx);
        b = lattice_point(wy, wx, qr, qc);
    } else {
        const Point up = lattice_point(wy, wx, qr + 2 * sy, qc);
        a = sy < 0 ? lattice_point(wy, wx, qr - 2, sx < 0 ? qc - 2 : qc) : (sx < 0 ? lattice_point(wy, wx, qr, qc - 2) : up);
        b = sx > 0 ? lattice_point(wy, wx, qr, qc + 2) : (sy > 0 && sx < 0 ? up : lattice_point(wy, wx, qr, qc));
    }
    // the incomplete row and column 19, met in block row 15 and column 15
    const bool row_edge = !kVer2 && hmy == 2 && sy > 0, col_edge = !kVer2 && hmx == 2 && sx > 0;
    unsigned s[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int r = rho + 4 * i;
        const uint4 c = L.cur[r];
        unsigned wa[4], wb[4];
        window_row(words + a.word + r * WPITCH, a.col, wa);
        window_row(words + b.word + r * WPITCH, b.col, wb);
        const unsigned cw[4] = {c.x, c.y, c.z, c.w};
        int edge = 0;  // column 19's sample
        if (col_edge && hmy) edge = raw_of(L.raw + 2 * WPITCH * ((qr >> 2) - 2 + r), wx + 19);
        if (i == 3 && row_edge && rho == 3) {
            const int at = wx + (qc >> 2);
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const int x = hmx ? raw_of(L.row19, at + k) : 0;
                const int y = k == 15 && col_edge ? edge : byte_of(sx < 0 ? wa[k >> 2] : wb[k >> 2], k & 3);
                const int e = byte_of(cw[k >> 2], k & 3) - ((x + y + 1) >> 1);
                s[k & 3] += (unsigned)(e * e);
            }
        } else {
            unsigned d[4];
#pragma unroll
            for (int k = 0; k < 4; k++) d[k] = __vabsdiffu4(cw[k], __vavgu4(wa[k], wb[k]));
            if (col_edge) {
                const int y = byte_of(sy == 0 ? wb[3] : wa[3], 3);
                const int e = byte_of(cw[3], 3) - ((edge + y + 1) >> 1);
                d[3] &= 0x00ffffffu;
                s[3] += (unsigned)(e * e);
            }
            add_classes(d[0], d[1], d[2], d[3], s);
        }
    }
    settle_quads<kPartial>(s, pack_mv(hmx + sx, hmy + sy), min_d, lane, [&](int x, int y, int d) {
        qmx = x;
        qmy = y;
        take(x, y, d);
    });
    __syncwarp();  // the lattice is reused by this warp's next search
}

// The input block of level 1 into L.cur1.
__device__ __forceinline__ void stage_level1(const MrcArgs& a, Window& L, int q, int p, int lane)
{
    const Org o = origin(a.in1, 8, 8, 0, q, p);
    if (lane < 16) {
        unsigned w[1];
        row_words(a.in1.p + (size_t)(o.y + (lane >> 1)) * a.in1.w + o.x + 4 * (lane & 1), w);
        reinterpret_cast<unsigned*>(L.cur1)[lane] = w[0];
    }
    __syncwarp();
}

// The input block of level 2, in every lane.
__device__ __forceinline__ void load_level2(const MrcArgs& a, int ll, int kk, unsigned (&cur)[4])
{
    const Org o = origin(a.in2, 4, 4, 0, ll, kk);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        unsigned w[1];
        row_words(a.in2.p + (size_t)(o.y + r) * a.in2.w + o.x, w);
        cur[r] = w[0];
    }
}

// ---------------------------------------------------------------------------
constexpr int TIE_L2 = 1, TIE_L1 = 2, TIE_L0 = 4;


// A search decides ties only with the prediction's vectors at the levels
// where its own trajectory met them, so a search made for prediction
// (ex, ey) whose trajectory tied at levels `tie` has the same trajectory, and
// result, for every prediction with the same vectors at those levels.
__device__ __forceinline__ int level_pred(int est, int p, int lvl);
__device__ __forceinline__ bool search_reusable(int est, int tie, int ex, int ey, int px, int py)
{
    for (int l = 0; l < 3; l++)
        if ((tie & (TIE_L0 >> l)) &&
            (level_pred(est, ex, l) != level_pred(est, px, l) || level_pred(est, ey, l) != level_pred(est, py, l)))
            return false;
    return true;
}

struct MbSearch {
    int zero_d, min_d, mvx, mvy;
    int tie;  // integer stages that met a candidate equal to their running minimum: TIE_L2 | TIE_L1 | TIE_L0
};

// Tie rule of the integer stages: an equal distortion replaces the current
// best (offset (rmx, rmy) from the centre (mx, my)) unless the candidate at
// (j, i) is farther from (px, py): (0, 0) for MultiresCross
// (…MultiresCross.cpp:741-746, 794, 857), the level's rounded prediction for
// Ver2 (…MultiresCrossVer2.cpp:778-786, 834-842, 906-914).
__device__ __forceinline__ bool farther(int mx, int my, int rmx, int rmy, int j, int i, int px, int py)
{
    const int cx = mx + rmx - px, cy = my + rmy - py, nx = mx + j - px, ny = my + i - py;
    return (cy * cy + cx * cx) - (ny * ny + nx * nx) < 0;
}

// The search of one macroblock, one warp, from the zero vector to the
// quarter-pel winner (…MultiresCross.cpp:612-941; …MultiresCrossVer2.cpp:643-992).
// kVer2: the completed sub-pel window.  skip(level, mx, my, rmx, rmy, j, i)
// decides an exact tie at an integer level: true keeps the current best
// (offset (rmx, rmy) from the centre (mx, my)), false takes the candidate at
// offset (j, i).  It is called with the same arguments in every lane.
template <bool kVer2, typename Skip, bool kH263 = false, typename Store>
__device__ MbSearch search_mb_with(const MrcArgs& a, Store& LT, int mbr, int mbc, Skip&& skip, int lane, bool& bad)
{
    const int m = 16 * mbr, n = 16 * mbc, p = 8 * mbr, q = 8 * mbc, kk = 4 * mbr, ll = 4 * mbc;
    const int w1 = a.W / 2, h1 = a.H / 2, w2 = w1 / 2, h2 = h1 / 2;
    const int l1_range = a.motion_range / 8, l2_range = l1_range / 2;
    const int lcl_l1_range = a.mode == 2 ? 2 : l1_range;
    const Level L0{16, a.W, a.H, a.motion_range / 4}, L1{8, w1, h1, l1_range}, L2{4, w2, h2, l2_range};
    MbSearch out;
    out.tie = 0;

    __syncwarp();
    out.zero_d = zero_distortion(a, LT, origin(a.in0, 16, 16, 0, n, m), n, m, lane);
    stage_level1(a, LT, q, p, lane);
    int mx = 0, my = 0, rmx = 0, rmy = 0, xl, xr, yu, yd;
    int min, lvl = 2;
    auto tie = [&](int j, int i) {
        out.tie |= TIE_L0 >> lvl;
        return skip(lvl, mx, my, rmx, rmy, j, i);
    };
    auto take = [&](int j, int i, int) {
        rmx = j;
        rmy = i;
    };

    if (a.mode == 2) {  // level 2 cross search (…MultiresCross.cpp:639-697)
        // Tsd4x4LessThan stops early only on a sum already above min: a full SSD decides the same
        unsigned cur2[4];
        load_level2(a, ll, kk, cur2);
        min = score4(cur2, a.e2, origin(a.e2, 4, 4, 5, ll, kk));
        mr_range(L2, ll, kk, 0, 0, l2_range - 1, xl, xr, yu, yd);
        for (int s = l2_range / 2; s > 0; s /= 2) {
            rmx = rmy = 0;
            int j, i;
            cross_offset(lane, s, j, i);
            const int d = score4(cur2, a.e2, origin(a.e2, 4, 4, 5, j + ll + mx, i + kk + my));
            settle(lane < 4 && i + my >= yu && i + my <= yd && j + mx >= xl && j + mx <= xr, d, d, pack_mv(j, i), min, tie,
                   take);
            mx += rmx;
            my += rmy;
        }
        mx <<= 1;
        my <<= 1;
    }

    // level 1 (…MultiresCross.cpp:699-816)
    lvl = 1;
    rmx = rmy = 0;
    auto score1 = [&](int j, int i, int& d, int& t) {
        score8<true>(LT, a.e1, origin(a.e1, 8, 8, 9, j + mx + q, i + my + p), d, t);
    };
    if (a.mode == 2) {
        mr_range(L1, q, p, mx, my, lcl_l1_range, xl, xr, yu, yd);
        raster(xl, xr, yu, yd, min, lane, score1, tie, take);
    } else {
        int t;
        score1(0, 0, min, t);
        for (int s = l1_range / 2; s > 0; s /= 2) {
            mr_range(L1, q, p, mx, my, lcl_l1_range - 1, xl, xr, yu, yd);
            rmx = rmy = 0;
            int j, i, d;
            cross_offset(lane, s, j, i);
            score1(j, i, d, t);
            settle(lane < 4 && i + my >= yu && i + my <= yd && j + mx >= xl && j + mx <= xr, d, t, pack_mv(j, i), min, tie,
                   take);
            mx += rmx;
            my += rmy;
        }
    }
    // the last level-1 refinement is added once more (…MultiresCross.cpp:815-816)
    mx = (mx + rmx) * 2;
    my = (my + rmy) * 2;

    // level 0 +-2 refinement (…MultiresCross.cpp:819-873)
    lvl = 0;
    rmx = rmy = 0;
    const Org oc = origin(a.e0, 16, 16, 19, n + mx, m + my);
    stage_level0(a.e0, LT, oc, lane);
    mr_range(L0, n, m, mx, my, 2, xl, xr, yu, yd);
    raster(xl, xr, yu, yd, min, lane,
           [&](int j, int i, int& d, int& t) {
               const Org c = origin(a.e0, 16, 16, 19, n + mx + j, m + my + i);
               score16<true>(LT, c.y - oc.y + 5, c.x - oc.x + 5, d, t);
           },
           tie, take);
    mx += rmx;
    my += rmy;
    const Org o = origin(a.e0, 16, 16, 19, n + mx, m + my);
    if constexpr (kH263) {
        // MotionEstimatorH263ImplMultiresCross (…H263ImplMultiresCross.cpp:885-940): the best of the
        // four diagonal half-pel corners, then the two points beside the winning corner (the full cross
        // if no corner won), each an OverlayMem2Dv2::HalfRead block (bilinear, +2 >> 2 diagonal, +1 >> 1
        // linear; the left neighbour for -1) of the level-0 reference, strict improvements; half pels.
        // Every sample read lies within 17 of the picture, where the border-19 copy holds the same edge
        // replication as the reference's border-17 one.  Four lanes a candidate, a row class each.
        bad |= (o.y - 1) * a.e0.w + o.x - 1 < 0 || (o.y + 16) * a.e0.w + o.x + 16 >= a.e0.w * a.e0.h;
        const int row = o.y - oc.y + 5, col = o.x - oc.x + 5, rho = lane & 3, k = lane >> 2;
        int hmx = 0, hmy = 0;
        auto half_stage = [&](int hx, int hy, bool valid) {
            unsigned s[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 c = LT.cur[rho + 4 * i];
                const unsigned cw[4] = {c.x, c.y, c.z, c.w};
                const unsigned* w = LT.win + (row + rho + 4 * i) * WPITCH;
                unsigned w00[4], w01[4], w10[4], w11[4], d[4];
                window_row(w, col, w00);
                window_row(w, col + hx, w01);
                window_row(w + hy * WPITCH, col, w10);
                window_row(w + hy * WPITCH, col + hx, w11);
#pragma unroll
                for (int e = 0; e < 4; e++) d[e] = __vabsdiffu4(cw[e], half4(w00[e], w01[e], w10[e], w11[e], hx, hy));
                add_classes(d[0], d[1], d[2], d[3], s);
            }
            if (!valid) s[0] = 0x10000000u;  // above any block's distortion
            settle_quads<true>(s, pack_mv(hx, hy), min, lane, [&](int x, int y, int) {
                hmx = x;
                hmy = y;
            });
        };
        half_stage((k & 1) ? 1 : -1, (k & 2) ? 1 : -1, k < 4);
        const int vx = hmx, vy = hmy;  // the winning corner
        if (vx || vy) half_stage((k & 1) ? vx : 0, (k & 1) ? 0 : vy, k < 2);
        else half_stage((k & 2) ? 0 : ((k & 1) ? 1 : -1), (k & 2) ? ((k & 1) ? 1 : -1) : 0, k < 4);
        __syncwarp();
        out.min_d = min;
        out.mvx = 2 * mx + hmx;
        out.mvy = 2 * my + hmy;
        return out;
    } else {
        int qmx = 0, qmy = 0;
        subpel<kVer2, true>(LT, a.e0, oc, o, min, qmx, qmy, lane, bad, [](int, int, int) {});
        out.min_d = min;
        out.mvx = mx * 4 + qmx;
        out.mvy = my * 4 + qmy;
        return out;
    }
}

// The search of MotionEstimatorH264ImplMultires (…Multires.cpp:644-906): full
// searches at level 2 (+-(range/16 - 1)) and level 1 (+-2 after level 2, else
// +-range/8), +-2 at level 0, half and quarter pel in the MultiresCross-style
// window; LessThan distortions, which decide exactly as full SSDs do.
template <typename Skip>
__device__ MbSearch search_mr_with(const MrcArgs& a, Lattice& LT, int mbr, int mbc, Skip&& skip, int lane, bool& bad)
{
    const int m = 16 * mbr, n = 16 * mbc, p = 8 * mbr, q = 8 * mbc, kk = 4 * mbr, ll = 4 * mbc;
    const int w1 = a.W / 2, h1 = a.H / 2, w2 = w1 / 2, h2 = h1 / 2;
    const int l1_range = a.motion_range / 8, l2_range = l1_range / 2;
    const int lcl_l1_range = a.mode == 2 ? 2 : l1_range;
    const Level L0{16, a.W, a.H, a.motion_range / 4}, L1{8, w1, h1, l1_range}, L2{4, w2, h2, l2_range};
    MbSearch out;
    out.tie = 0;
    __syncwarp();
    out.zero_d = zero_distortion(a, LT, origin(a.in0, 16, 16, 0, n, m), n, m, lane);
    stage_level1(a, LT, q, p, lane);
    int mx = 0, my = 0, rmx = 0, rmy = 0, xl, xr, yu, yd, min, lvl = 2;
    auto tie = [&](int j, int i) {
        out.tie |= TIE_L0 >> lvl;
        return skip(lvl, mx, my, rmx, rmy, j, i);
    };
    auto take = [&](int j, int i, int) {
        rmx = j;
        rmy = i;
    };

    if (a.mode == 2) {  // level 2 full search around (0, 0) (…Multires.cpp:667-731)
        unsigned cur2[4];
        load_level2(a, ll, kk, cur2);
        mr_range(L2, ll, kk, 0, 0, l2_range - 1, xl, xr, yu, yd);
        raster(xl, xr, yu, yd, min, lane,
               [&](int j, int i, int& d, int& t) { t = d = score4(cur2, a.e2, origin(a.e2, 4, 4, 5, ll + j, kk + i)); },
               tie, take);
        mx = rmx << 1;
        my = rmy << 1;
    }

    // level 1 around (mx, my) (…Multires.cpp:735-790)
    lvl = 1;
    rmx = rmy = 0;
    mr_range(L1, q, p, mx, my, lcl_l1_range, xl, xr, yu, yd);
    raster(xl, xr, yu, yd, min, lane,
           [&](int j, int i, int& d, int& t) {
               score8<false>(LT, a.e1, origin(a.e1, 8, 8, 9, j + mx + q, i + my + p), d, t);
           },
           tie, take);
    mx = (mx + rmx) * 2;
    my = (my + rmy) * 2;

    // level 0 +-2 (…Multires.cpp:792-849)
    lvl = 0;
    rmx = rmy = 0;
    const Org oc = origin(a.e0, 16, 16, 19, n + mx, m + my);
    stage_level0(a.e0, LT, oc, lane);
    mr_range(L0, n, m, mx, my, 2, xl, xr, yu, yd);
    raster(xl, xr, yu, yd, min, lane,
           [&](int j, int i, int& d, int& t) {
               const Org c = origin(a.e0, 16, 16, 19, n + mx + j, m + my + i);
               score16<false>(LT, c.y - oc.y + 5, c.x - oc.x + 5, d, t);
           },
           tie, take);
    mx += rmx;
    my += rmy;

    // half then quarter pel (…Multires.cpp:851-917), strict improvements, full distortions
    int qmx = 0, qmy = 0;
    subpel<false, false>(LT, a.e0, oc, origin(a.e0, 16, 16, 19, n + mx, m + my), min, qmx, qmy, lane, bad,
                         [](int, int, int) {});
    out.min_d = min;
    out.mvx = mx * 4 + qmx;
    out.mvy = my * 4 + qmy;
    return out;
}

// ---------------------------------------------------------------------------
// MultiresCrossVer2::Estimate(long*, void* lambda): every search level keeps
// its improvements in a five-slot list (Fifo(5) of include/GeneralUtils/Fifo.h,
// newest in slot 0; the first item after a reset fills every slot) and ends
// with GetBestVector over it.  Lane i < 5 of the searching warp holds slot i.
struct Fifo5 {
    int x, y, d;
    __device__ __forceinline__ void reset(int vx, int vy, int vd)
    {
        x = vx;
        y = vy;
        d = vd;
    }
    __device__ __forceinline__ void push(int vx, int vy, int vd, int lane)
    {
        x = __shfl_up_sync(0xffffffffu, x, 1);
        y = __shfl_up_sync(0xffffffffu, y, 1);
        d = __shfl_up_sync(0xffffffffu, d, 1);
        if (lane == 0) {
            x = vx;
            y = vy;
            d = vd;
        }
    }
};

// GetBestVector (include/CodecUtils/MotionEstimatorH264ImplMultiresCrossVer2.h:168-197):
// cost D/norm + lambda*sqrt(|v - ref|^2) in IEEE double, one rounding per
// operation as the reference's expression; slot 0 is costed at the current
// vector (mx, my) with lambda * 2^(level+2) / 16, slots 1..4 with the raw
// lambda; the slots in order, strict improvement.  Lanes 0..4 cost their slot
// at once.  Sets (mx, my) and returns the winning slot's distortion.
__device__ __forceinline__ int fifo_best(const Fifo5& f, double lambda, double norm, int level, int xr, int yr,
                                         int& mx, int& my, int lane)
{
    const double l = lane == 0 ? __ddiv_rn(__dmul_rn(lambda, (double)(1 << (level + 2))), 16.0) : lambda;
    const int vx = lane == 0 ? mx : f.x, vy = lane == 0 ? my : f.y;
    const double m2 = (double)((vx - xr) * (vx - xr) + (vy - yr) * (vy - yr));
    const double c = __dadd_rn(__ddiv_rn((double)f.d, norm), __dmul_rn(l, __dsqrt_rn(m2)));
    double best = __shfl_sync(0xffffffffu, c, 0);
    int bi = 0;
#pragma unroll
    for (int i = 1; i < 5; i++) {
        const double ci = __shfl_sync(0xffffffffu, c, i);
        if (ci < best) {
            best = ci;
            bi = i;
        }
    }
    const int nx = __shfl_sync(0xffffffffu, f.x, bi), ny = __shfl_sync(0xffffffffu, f.y, bi);
    if (bi) {
        mx = nx;
        my = ny;
    }
    return __shfl_sync(0xffffffffu, f.d, bi);
}

constexpr int TIE_ALL = TIE_L2 | TIE_L1 | TIE_L0;

// The search of the Lagrangian overload (…MultiresCrossVer2.cpp:1237-1676),
// one warp: the Ver2 search with GetBestVector towards the prediction's
// vector of each level (pl[2l], pl[2l+1]: level l's x, y, level 0 rounded;
// norms 16, 64, 256 at levels 2, 1, 0), at the end of the sub-pel stages towards the clamped
// quarter-pel prediction (pcx, pcy).  Unlike Estimate(long*), the cross mode
// adds its last level-1 refinement once only (…:1434-1499), and level 0
// continues from the list's choice.  Every result depends on the prediction:
// tie = TIE_ALL.
__device__ MbSearch search_lambda(const MrcArgs& a, Lattice& LT, int mbr, int mbc, const int* pl, int pcx, int pcy,
                                  int lane, bool& bad)
{
    const int m = 16 * mbr, n = 16 * mbc, p = 8 * mbr, q = 8 * mbc, kk = 4 * mbr, ll = 4 * mbc;
    const int w1 = a.W / 2, h1 = a.H / 2, w2 = w1 / 2, h2 = h1 / 2;
    const int l1_range = a.motion_range / 8, l2_range = l1_range / 2;
    const int lcl_l1_range = a.mode == 2 ? 2 : l1_range;
    const Level L0{16, a.W, a.H, a.motion_range / 4}, L1{8, w1, h1, l1_range}, L2{4, w2, h2, l2_range};
    const double lam = a.lambda;
    MbSearch out;
    out.tie = TIE_ALL;
    Fifo5 f;

    __syncwarp();
    out.zero_d = zero_distortion(a, LT, origin(a.in0, 16, 16, 0, n, m), n, m, lane);
    stage_level1(a, LT, q, p, lane);
    int mx = 0, my = 0, rmx = 0, rmy = 0, xl, xr, yu, yd, min, lvl = 2;
    auto tie = [&](int j, int i) { return farther(mx, my, rmx, rmy, j, i, pl[2 * lvl], pl[2 * lvl + 1]); };
    auto take = [&](int j, int i, int d) {
        rmx = j;
        rmy = i;
        f.push(j + mx, i + my, d, lane);
    };

    if (a.mode == 2) {  // level 2 cross search (…:1287-1370)
        // Tsd4x4LessThan stops early only on a sum already above min: a full SSD decides the same
        unsigned cur2[4];
        load_level2(a, ll, kk, cur2);
        min = score4(cur2, a.e2, origin(a.e2, 4, 4, 5, ll, kk));
        f.reset(0, 0, min);
        mr_range(L2, ll, kk, 0, 0, l2_range - 1, xl, xr, yu, yd);
        for (int s = l2_range / 2; s > 0; s /= 2) {
            rmx = rmy = 0;
            int j, i;
            cross_offset(lane, s, j, i);
            const int d = score4(cur2, a.e2, origin(a.e2, 4, 4, 5, j + ll + mx, i + kk + my));
            settle(lane < 4 && i + my >= yu && i + my <= yd && j + mx >= xl && j + mx <= xr, d, d, pack_mv(j, i), min, tie,
                   take);
            mx += rmx;
            my += rmy;
        }
        fifo_best(f, lam, 16.0, 2, pl[4], pl[5], mx, my, lane);
        mx <<= 1;
        my <<= 1;
    }

    // level 1 (…:1374-1502)
    lvl = 1;
    rmx = rmy = 0;
    auto score1 = [&](int j, int i, int& d, int& t) {
        score8<true>(LT, a.e1, origin(a.e1, 8, 8, 9, j + mx + q, i + my + p), d, t);
    };
    int t;
    score1(0, 0, min, t);
    f.reset(mx, my, min);
    if (a.mode == 2) {
        mr_range(L1, q, p, mx, my, lcl_l1_range, xl, xr, yu, yd);
        raster(xl, xr, yu, yd, min, lane, score1, tie, take);
        mx += rmx;
        my += rmy;
    } else {
        for (int s = l1_range / 2; s > 0; s /= 2) {
            mr_range(L1, q, p, mx, my, lcl_l1_range - 1, xl, xr, yu, yd);
            rmx = rmy = 0;
            int j, i, d;
            cross_offset(lane, s, j, i);
            score1(j, i, d, t);
            settle(lane < 4 && i + my >= yu && i + my <= yd && j + mx >= xl && j + mx <= xr, d, t, pack_mv(j, i), min, tie,
                   take);
            mx += rmx;
            my += rmy;
        }
    }
    fifo_best(f, lam, 64.0, 1, pl[2], pl[3], mx, my, lane);
    mx <<= 1;
    my <<= 1;

    // level 0 +-2 refinement (…:1503-1574)
    lvl = 0;
    rmx = rmy = 0;
    const Org oc = origin(a.e0, 16, 16, 19, n + mx, m + my);
    stage_level0(a.e0, LT, oc, lane);
    auto score0 = [&](int j, int i, int& d, int& t0) {
        const Org c = origin(a.e0, 16, 16, 19, n + mx + j, m + my + i);
        score16<true>(LT, c.y - oc.y + 5, c.x - oc.x + 5, d, t0);
    };
    score0(0, 0, min, t);
    f.reset(mx, my, min);
    mr_range(L0, n, m, mx, my, 2, xl, xr, yu, yd);
    raster(xl, xr, yu, yd, min, lane, score0, tie, take);
    mx += rmx;
    my += rmy;
    min = fifo_best(f, lam, 256.0, 0, pl[0], pl[1], mx, my, lane);

    // half then quarter pel in Ver2's window (…:1575-1662), strict improvements
    int mvx = mx * 4, mvy = my * 4, qmx = 0, qmy = 0;
    f.reset(mvx, mvy, min);
    const Org o = origin(a.e0, 16, 16, 19, n + mx, m + my);
    subpel<true, true>(LT, a.e0, oc, o, min, qmx, qmy, lane, bad,
                       [&](int x, int y, int d) { f.push(x + mvx, y + mvy, d, lane); });
    mvx += qmx;
    mvy += qmy;
    // towards the clamped quarter-pel prediction (…:1664-1677)
    out.min_d = fifo_best(f, lam, 256.0, 2, pcx, pcy, mvx, mvy, lane);
    out.mvx = mvx;
    out.mvy = mvy;
    return out;
}

// MultiresCross's tie rules: at level 2 the centre against the offset
// (…MultiresCross.cpp:673-679), elsewhere distances from (0, 0) (…:741-746, 857).
template <bool kH263 = false, typename Store>
__device__ __forceinline__ MbSearch search_mb_mrc(const MrcArgs& a, Store& LT, int mbr, int mbc, int lane,
                                                  bool& bad)
{
    auto skip = [](int lvl, int mx, int my, int rmx, int rmy, int j, int i) {
        return lvl == 2 ? (my * my + mx * mx) - (i * i + j * j) < 0 : farther(mx, my, rmx, rmy, j, i, 0, 0);
    };
    return search_mb_with<false, decltype(skip)&, kH263>(a, LT, mbr, mbc, skip, lane, bad);
}

// The prediction's vector at a pyramid level (quarter-pel component p):
// Ver2 rounds to level 0 and halves (…MultiresCrossVer2.cpp:627-642),
// Multires rounds to every level (…Multires.cpp:646-655).
constexpr int EST_VER2 = 1, EST_MULTIRES = 2, EST_V2_LAMBDA = 4;
__device__ __forceinline__ int level_pred(int est, int p, int lvl)
{
    if (est == EST_MULTIRES) {
        const int h = 2 << lvl;  // 2, 4, 8
        return p < 0 ? (p - h) / (2 * h) : (p + h) / (2 * h);
    }
    int v = p < 0 ? (p - 2) / 4 : (p + 2) / 4;
    for (int l = 0; l < lvl; l++) v /= 2;
    return v;
}

// Search of a predictor estimator (est) with ties decided by the distances
// from prediction (px, py) at each level.
template <int kEst>
__device__ __forceinline__ MbSearch search_pred(const MrcArgs& a, Lattice& LT, int mbr, int mbc, int px, int py,
                                                int lane, bool& bad)
{
    int pl[6];
    for (int l = 0; l < 3; l++) {
        pl[2 * l] = level_pred(kEst, px, l);
        pl[2 * l + 1] = level_pred(kEst, py, l);
    }
    if constexpr (kEst == EST_V2_LAMBDA) {
        // the prediction clamped to one macroblock outside the picture (…MultiresCrossVer2.cpp:1664-1675)
        const int n = 16 * mbc, m = 16 * mbr;
        int px0 = px / 4, py0 = py / 4;
        if (px0 + n > a.W) px0 = 16;
        if (px0 + n < -16) px0 = -16;
        if (py0 + m > a.H) py0 = 16;
        if (py0 + m < -16) py0 = -16;
        return search_lambda(a, LT, mbr, mbc, pl, 4 * px0 + px % 4, 4 * py0 + py % 4, lane, bad);
    }
    auto skip = [&pl](int lvl, int mx, int my, int rmx, int rmy, int j, int i) {
        return farther(mx, my, rmx, rmy, j, i, pl[2 * lvl], pl[2 * lvl + 1]);
    };
    if constexpr (kEst == EST_MULTIRES) return search_mr_with(a, LT, mbr, mbc, skip, lane, bad);
    else return search_mb_with<true>(a, LT, mbr, mbc, skip, lane, bad);
}

// Tie tree of a Ver2 macroblock: run r of eight decides its t-th tie (t < 3)
// by bit t of r (1 takes the candidate) and records the tie's level and the
// two vectors compared, current (cx, cy) and candidate (nx, ny) in level
// units, so that the decision for any prediction follows from them; runs
// sharing their low t bits share their first t ties.
constexpr int V2_TIE_RUNS = 8, V2_TIE_BITS = 3;
struct V2TieRun {
    int geo[V2_TIE_BITS];  // bytes: cx, cy, nx, ny (signed)
    int lvl;               // 2 bits per tie
    int nev;               // ties met (> V2_TIE_BITS: the tree is too deep)
    int mv;                // packed quarter-pel result
    int min_d;
    int pad;
};

template <int kEst>
__device__ __forceinline__ MbSearch search_run(const MrcArgs& a, Lattice& LT, int mbr, int mbc, int run,
                                               V2TieRun* rec, int lane, bool& bad)
{
    int t = 0, lvls = 0, geo[V2_TIE_BITS] = {0, 0, 0};
    bool wide = false;
    auto skip = [&](int lvl, int mx, int my, int rmx, int rmy, int j, int i) {
        const int cx = mx + rmx, cy = my + rmy, nx = mx + j, ny = my + i;
        const bool take = t < V2_TIE_BITS ? ((run >> t) & 1) : true;
        if (t < V2_TIE_BITS) {
            wide |= (unsigned)(cx + 128) > 255u || (unsigned)(cy + 128) > 255u || (unsigned)(nx + 128) > 255u ||
                    (unsigned)(ny + 128) > 255u;
            geo[t] = (cx & 0xff) | ((cy & 0xff) << 8) | ((nx & 0xff) << 16) | ((ny & 0xff) << 24);
            lvls |= lvl << (2 * t);
        }
        t++;
        return !take;
    };
    MbSearch r;
    if constexpr (kEst == EST_MULTIRES) r = search_mr_with(a, LT, mbr, mbc, skip, lane, bad);
    else r = search_mb_with<true>(a, LT, mbr, mbc, skip, lane, bad);
    if (lane == 0) {
        for (int e = 0; e < V2_TIE_BITS; e++) rec->geo[e] = geo[e];
        rec->lvl = lvls;
        rec->nev = wide ? 1000 : t;
        rec->mv = pack_mv(r.mvx, r.mvy);
        rec->min_d = r.min_d;
    }
    return r;
}

// The searched vector and distortion of a tie MB for prediction (px, py) from its tie tree; false when the
// tree is too deep.  One warp: half a run per lane, loaded at once (walked run by run, a tree of one tie
// was four round trips to L2, a microsecond of every evaluation).
__device__ __forceinline__ bool tie_tree_result(int est, const V2TieRun* runs, int ppx, int ppy, int lane, int* mv,
                                                int* min_d)
{
    static_assert(sizeof(V2TieRun) == 32 && V2_TIE_RUNS == 8, "two 16-byte words per run, half a warp of them");
    // even: {geo[0], geo[1], geo[2], lvl}, odd: {nev, mv, min_d, -}
    const int4 v = __ldcg(reinterpret_cast<const int4*>(runs) + (lane & 15));
    int run = 0;
    for (int t = 0; t < V2_TIE_BITS; t++) {
        if (t >= __shfl_sync(0xffffffffu, v.x, 2 * run + 1)) break;
        const int g = __shfl_sync(0xffffffffu, t == 0 ? v.x : (t == 1 ? v.y : v.z), 2 * run);
        const int lvl = (__shfl_sync(0xffffffffu, v.w, 2 * run) >> (2 * t)) & 3;
        const int cx = (signed char)(g & 0xff), cy = (signed char)((g >> 8) & 0xff);
        const int nx = (signed char)((g >> 16) & 0xff), ny = (signed char)(g >> 24);
        const int px = level_pred(est, ppx, lvl), py = level_pred(est, ppy, lvl);
        const bool skip = (cy - py) * (cy - py) + (cx - px) * (cx - px) < (ny - py) * (ny - py) + (nx - px) * (nx - px);
        run |= (skip ? 0 : 1) << t;
    }
    *mv = __shfl_sync(0xffffffffu, v.y, 2 * run + 1);
    *min_d = __shfl_sync(0xffffffffu, v.z, 2 * run + 1);
    return __shfl_sync(0xffffffffu, v.x, 2 * run + 1) <= V2_TIE_BITS;
}

}  // namespace
}  // namespace mrc
}  // namespace vppgpu
