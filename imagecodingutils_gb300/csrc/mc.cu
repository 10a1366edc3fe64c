// mc.cu -- MotionCompensatorH264ImplStd and the block add / subtract helpers
// on sm_103a.
//
// Reference: MotionCompensatorH264ImplStd::Compensate(pMotionList)
// (src/CodecUtils/MotionCompensatorH264ImplStd.cpp:323-473).  The reference
// copies the 4:2:0 reference frame into edge-extended temporaries and, block
// by block, overwrites the frame with the block each vector points at: luma
// 16x16 by OverlayMem2Dv2::QuarterRead at the quarter-pel vector, chroma 8x8
// by OverlayMem2Dv2::EighthRead at the same vector in eighth-pel units
// (bilinear, (z + 32) >> 6).  A zero vector leaves its block as it is.
//
// GB300 design: for compensation in place the frame is first copied to a
// stream-ordered temporary (the reference's temporaries), else read as it is;
// the output is computed from it in one launch, one warp per macroblock
// (luma window and the half-pel lattices its fraction reads in shared
// memory, then both chroma blocks).  The edge extension is a clamp of the sample coordinates,
// which gives the extended border's values for every vector within the
// reference's range.  Only full macroblock rows are compensated (the
// reference reads vectors past the end of its list for a partial bottom
// row); rows below keep the reference samples.
//
// The add-with-clip and subtract helpers (Add16x16WithClip255 /
// Add8x8WithClip255, Sub16x16 / Sub8x8, OverlayMem2Dv2.cpp:1195-1426) are
// elementwise over whole planes, 8 samples per thread with 16-byte accesses.
#include <cstdint>
#include <new>

#include "me_common.cuh"

namespace {

struct Plane {
    const short* p;
    int w, h;
};

constexpr int kMcWarps = 4;  // macroblocks per CTA, one warp each

// A macroblock's shared memory: its luma window from its first column (22 x 22 samples, two of margin on each side of
// the 17 x 17 the block reads), its 9 x 9 chroma windows (U, then V) from an even column, and what the j cases read:
// vertical 6-tap sums + TAP_BIAS of pairs of columns, or horizontal sums (any samples).  At 14 words a row, four rows
// apart eight words lie in the 32 banks.
struct McPairs {
    alignas(16) unsigned win[22][14];  // (written two words at a time)
    unsigned cwin[18][6];
    union {
        unsigned vt[16][12];
        int th[22][16];
    };
};

// QuarterRead per quarter case cs = fx | fy << 2: one sample, or the rounded average of two, from G (full-pel), b
// (horizontal half: 6-tap over a window row), h (vertical half: 6-tap down a window column) and j (centre).  Each
// entry: kind | offset << 3 of the first term, then << 8 of the second, the offset as dx | dy << 1.
enum : int { kTermG = 0, kTermB = 1, kTermH = 2, kTermJ = 3, kTermNone = 4 };
__constant__ int c_quarter_terms[16] = {
    kTermG | kTermNone << 8,                     kTermG | kTermB << 8,
    kTermB | kTermNone << 8,                     kTermG | 1 << 3 | kTermB << 8,
    kTermG | kTermH << 8,                        kTermB | kTermH << 8,
    kTermJ | kTermB << 8,                        kTermB | (kTermH | 1 << 3) << 8,
    kTermH | kTermNone << 8,                     kTermJ | kTermH << 8,
    kTermJ | kTermNone << 8,                     kTermJ | (kTermH | 1 << 3) << 8,
    kTermG | 2 << 3 | kTermH << 8,               kTermH | (kTermB | 2 << 3) << 8,
    kTermJ | (kTermB | 2 << 3) << 8,             kTermH | 1 << 3 | (kTermB | 2 << 3) << 8,
};

// the six-tap (1, -5, 20, 20, -5, 1) over samples s apart
template <int kS, typename T>
__device__ __forceinline__ int tap6(const T* p)
{
    return p[0] - 5 * p[kS] + 20 * p[2 * kS] + 20 * p[3 * kS] - 5 * p[4 * kS] + p[5 * kS];
}

// The block from windows of any samples, one at a time, lane (X = lane & 15, Y = lane >> 4 + 2t): a compact loop per
// kind of term (warp-uniform).  odd: the chroma windows begin at their second column.
__device__ __noinline__ void mc_any_samples(McPairs& L, int mvx, int mvy, bool odd, int lane, short* __restrict__ dst,
                                            int stride, short* __restrict__ du, short* __restrict__ dv, int cstride)
{
    constexpr int kP = 28, kC = 12;  // shorts a row
    const short* win = reinterpret_cast<const short*>(L.win);
    const int X = lane & 15, Y0 = lane >> 4, terms = c_quarter_terms[(mvx & 3) | (mvy & 3) << 2];
    if ((terms & 7) == kTermJ) {
#pragma unroll
        for (int t = 0; t < 11; t++) L.th[Y0 + 2 * t][X] = tap6<1>(win + (Y0 + 2 * t) * kP + X);
        __syncwarp();
    }
    const int nterm = (terms >> 8 & 7) == kTermNone ? 1 : 2;
    int acc[8];
#pragma unroll
    for (int t = 0; t < 8; t++) acc[t] = 0;
#pragma unroll 1
    for (int e = 0; e < nterm; e++) {
        const int term = terms >> (8 * e), kind = term & 7, dx = term >> 3 & 1, dy = term >> 4 & 1;
        const short* w = win + Y0 * kP + X;
        if (kind == kTermJ) {
            const int* tb = &L.th[Y0][X];
#pragma unroll
            for (int t = 0; t < 8; t++) acc[t] += clip255((tap6<16>(tb + 32 * t) + 512) >> 10);
        } else if (kind == kTermG) {
            w += (2 + dy) * kP + 2 + dx;
#pragma unroll
            for (int t = 0; t < 8; t++) acc[t] += w[2 * kP * t];
        } else if (kind == kTermB) {
            w += (2 + dy) * kP;
#pragma unroll
            for (int t = 0; t < 8; t++) acc[t] += clip255((tap6<1>(w + 2 * kP * t) + 16) >> 5);
        } else {
            w += 2 + dx;
#pragma unroll
            for (int t = 0; t < 8; t++) acc[t] += clip255((tap6<kP>(w + 2 * kP * t) + 16) >> 5);
        }
    }
#pragma unroll
    for (int t = 0; t < 8; t++)
        dst[(size_t)(Y0 + 2 * t) * stride + X] = (short)(nterm == 1 ? acc[t] : (acc[t] + 1) >> 1);
    // EighthRead of the chroma blocks: U rows 0-3, U rows 4-7, V rows 0-3, V rows 4-7
    const int fx = mvx & 7, fy = mvy & 7, x = lane & 7, y0 = lane >> 3;
    const int w00 = (8 - fx) * (8 - fy), w10 = fx * (8 - fy), w01 = (8 - fx) * fy, w11 = fx * fy;
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const int y = y0 + 4 * (t & 1);
        const short* p = reinterpret_cast<const short*>(L.cwin) + (9 * (t >> 1) + y) * kC + x + odd;
        const int v = (w00 * p[0] + w10 * p[1] + w01 * p[kC] + w11 * p[kC + 1] + 32) >> 6;
        (t < 2 ? du : dv)[(size_t)y * cstride + x] = (short)v;
    }
}

// The terms for a lane's pair of columns (2p, 2p + 1), rows r .. r + 3, pairs of samples 0..255; p: lane & 7.
__device__ __forceinline__ void mc_pair_term(const McPairs& L, int term, int r, int p, unsigned (&out)[4])
{
    const int kind = term & 7, dx = (term >> 3) & 1, dy = (term >> 4) & 1;
    if (kind == kTermG) {
        const unsigned* w = &L.win[r + 2 + dy][p + 1];
#pragma unroll
        for (int i = 0; i < 4; i++) out[i] = dx ? __funnelshift_r(w[14 * i], w[14 * i + 1], 16) : w[14 * i];
    } else if (kind == kTermB) {
        const unsigned* w = &L.win[r + 2 + dy][p];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned a = w[14 * i], b = w[14 * i + 1], c = w[14 * i + 2], d = w[14 * i + 3];
            out[i] = vppgpu::scale_pair(vppgpu::tap_pair(a, __funnelshift_r(a, b, 16), b, __funnelshift_r(b, c, 16), c,
                                                         __funnelshift_r(c, d, 16)));
        }
    } else if (kind == kTermH) {
        unsigned v[9];
        const unsigned* w = &L.win[r][p + 1];
#pragma unroll
        for (int i = 0; i < 9; i++) v[i] = dx ? __funnelshift_r(w[14 * i], w[14 * i + 1], 16) : w[14 * i];
#pragma unroll
        for (int i = 0; i < 4; i++)
            out[i] = vppgpu::scale_pair(vppgpu::tap_pair(v[i], v[i + 1], v[i + 2], v[i + 3], v[i + 4], v[i + 5]));
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned* w = &L.vt[r + i][p];
            out[i] = vppgpu::tap_centre2(w[0], w[1], w[2], w[3]);
        }
    }
}

// A pair of samples; kWide: 4-byte aligned.
template <bool kWide>
__device__ __forceinline__ void store_pair(short* d, unsigned v)
{
    if (kWide) {
        *reinterpret_cast<unsigned*>(d) = v;
    } else {
        d[0] = (short)v;
        d[1] = (short)(v >> 16);
    }
}

// One warp per macroblock: its 16x16 luma block and its two 8x8 chroma blocks.  What bounds it is latency and
// instructions: a sample at a time, the chroma blocks before the luma window was asked for, a 1920x1088 frame
// took 12.2 us (750 instructions a macroblock; its 13 MB are 2 us, a launch with nothing in it 4).  Here
// everything the vector points at is asked for at once and computed on pairs of samples: 10.1 us (525 instructions;
// 8, 12 and 14 CTAs an SM 10.5, 10.3 and 11.1).  kWide, 16-byte aligned frames: loads of 8 and 4 bytes.  Past the
// frame's edge the groups of samples that a load takes are inside or outside as a whole, so it costs the same; the
// macroblocks there by another path were the launch's tail (12.6).  Pairs hold samples of 0..255 (seen from the
// windows); macroblocks with others are computed from the same windows by mc_any_samples (a frame full of them
// 10.3 us; with a second staging of their own 16.3).  Frames at other alignments take loads of a sample, 12.3 us.
// Warp-synchronous: no block barrier.
template <bool kWide>
__global__ void __launch_bounds__(32 * kMcWarps, 10) k_mc_frame(const __grid_constant__ Plane ry,
                                                               const __grid_constant__ Plane ru,
                                                               const __grid_constant__ Plane rv,
                                                               const int* __restrict__ mv, int cols, int nmb,
                                                               short* __restrict__ oy, short* __restrict__ ou,
                                                               short* __restrict__ ov)
{
    __shared__ McPairs store[kMcWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int k = blockIdx.x * kMcWarps + w;
    if (k >= nmb) return;  // whole warps only
    const int mbr = k / cols, n = (k - mbr * cols) * 16, m = mbr * 16;
    const int v = __ldg(mv + k), mvx = vppgpu::mv_x(v), mvy = vppgpu::mv_y(v);
    if (!(mvx | mvy)) {  // a zero vector keeps the blocks
        if (kWide) {
            const size_t at = (size_t)(m + (lane >> 1)) * ry.w + n + 8 * (lane & 1);
            const uint4 y = __ldg(reinterpret_cast<const uint4*>(ry.p + at));
            const size_t cat = (size_t)((m >> 1) + (lane & 7)) * ru.w + (n >> 1);
            if (lane < 16) {
                const uint4 c = __ldg(reinterpret_cast<const uint4*>((lane < 8 ? ru.p : rv.p) + cat));
                *reinterpret_cast<uint4*>((lane < 8 ? ou : ov) + cat) = c;
            }
            *reinterpret_cast<uint4*>(oy + at) = y;
        } else {
            const size_t at = (size_t)(m + (lane >> 4)) * ry.w + n + (lane & 15);
            const size_t cat = (size_t)((m >> 1) + (lane >> 3)) * ru.w + (n >> 1) + (lane & 7);
            short y[8], c[4];
#pragma unroll
            for (int t = 0; t < 8; t++) y[t] = __ldg(ry.p + at + (size_t)(2 * t) * ry.w);
#pragma unroll
            for (int t = 0; t < 4; t++) c[t] = __ldg((t < 2 ? ru.p : rv.p) + cat + (size_t)(4 * (t & 1)) * ru.w);
#pragma unroll
            for (int t = 0; t < 8; t++) oy[at + (size_t)(2 * t) * ry.w] = y[t];
#pragma unroll
            for (int t = 0; t < 4; t++) (t < 2 ? ou : ov)[cat + (size_t)(4 * (t & 1)) * ru.w] = c[t];
        }
        return;
    }
    // floor quotients and remainders: what QuarterRead's and EighthRead's folding of negative ones gives
    const int ox = n + (mvx >> 2) - 2, oy0 = m + (mvy >> 2) - 2, cs = (mvx & 3) | (mvy & 3) << 2;
    const int cx = (n >> 1) + (mvx >> 3), cy = (m >> 1) + (mvy >> 3);
    McPairs& L = store[w];
    const int q = lane & 7, r4 = lane >> 3;
    const bool odd = kWide && (cx & 1);
    unsigned all = 0;
    if (kWide) {
        const bool inside = ox >= 0 && ox + 22 <= ry.w && cx >= 0 && cx + 9 <= ru.w;  // between the sides
        const int dx = ox & 3;
        uint2 y[6];
        unsigned c[5];
        // a group of four (two) samples of a row is inside the frame or outside it as a whole
        const int gx = (ox & ~3) + 4 * q, gc = (cx & ~1) + 2 * q;
        const short* py = ry.p + min(max(gx, 0), ry.w - 4);
        const int pc = min(max(gc, 0), ru.w - 2);
#pragma unroll
        for (int i = 0; i < 6; i++) {
            y[i] = make_uint2(0u, 0u);
            if (q < (dx + 25) >> 2 && r4 + 4 * i < 22)
                y[i] = __ldg(reinterpret_cast<const uint2*>(py + (size_t)min(max(oy0 + r4 + 4 * i, 0), ry.h - 1) * ry.w));
        }
#pragma unroll
        for (int i = 0; i < 5; i++) {
            const int r = r4 + 4 * i;
            c[i] = 0u;
            if (q < 5 && r < 18)
                c[i] = __ldg(reinterpret_cast<const unsigned*>(
                    (r < 9 ? ru.p : rv.p) + (size_t)min(max(cy + (r < 9 ? r : r - 9), 0), ru.h - 1) * ru.w + pc));
        }
        if (!inside) {  // the sides' samples repeated
#pragma unroll
            for (int i = 0; i < 6; i++) {
                const unsigned e = gx < 0 ? __byte_perm(y[i].x, 0u, 0x1010) : __byte_perm(y[i].y, 0u, 0x3232);
                if (gx < 0 || gx >= ry.w) y[i] = make_uint2(e, e);
            }
#pragma unroll
            for (int i = 0; i < 5; i++)
                if (gc < 0 || gc >= ru.w) c[i] = __byte_perm(c[i], 0u, gc < 0 ? 0x1010 : 0x3232);
        }
#pragma unroll
        for (int i = 0; i < 6; i++) {
            all |= y[i].x | y[i].y;
            const unsigned n0 = __shfl_down_sync(0xffffffffu, y[i].x, 1), n1 = __shfl_down_sync(0xffffffffu, y[i].y, 1);
            const unsigned a = dx & 2 ? y[i].y : y[i].x, b = dx & 2 ? n0 : y[i].y, d = dx & 2 ? n1 : n0;
            const unsigned sh = 16 * (dx & 1);
            if (q < 6 && r4 + 4 * i < 22)
                *reinterpret_cast<uint2*>(&L.win[r4 + 4 * i][2 * q]) =
                    make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, d, sh));
        }
#pragma unroll
        for (int i = 0; i < 5; i++) {
            all |= c[i];
            if (q < 5 && r4 + 4 * i < 18) L.cwin[r4 + 4 * i][q] = c[i];
        }
    } else {  // a column per lane: chroma (lanes 0-8 U, 16-24 V) and half the luma rows in flight together
        const Plane& P = lane < 16 ? ru : rv;
        const int cc = lane & 15, x = min(max(ox + lane, 0), ry.w - 1), xc = min(max(cx + cc, 0), ru.w - 1);
        short* win = reinterpret_cast<short*>(L.win) + lane;
        short* cw = reinterpret_cast<short*>(L.cwin) + 9 * 12 * (lane >> 4) + cc;
        short c[9];
#pragma unroll
        for (int r = 0; r < 9; r++)
            c[r] = cc < 9 ? __ldg(P.p + (size_t)min(max(cy + r, 0), ru.h - 1) * ru.w + xc) : (short)0;
#pragma unroll
        for (int h0 = 0; h0 < 22; h0 += 11) {
            short y[11];
#pragma unroll
            for (int r = 0; r < 11; r++)
                y[r] = lane < 22 ? __ldg(ry.p + (size_t)min(max(oy0 + h0 + r, 0), ry.h - 1) * ry.w + x) : (short)0;
#pragma unroll
            for (int r = 0; r < 11; r++) {
                all |= (unsigned short)y[r];
                if (lane < 22) win[28 * (h0 + r)] = y[r];
            }
        }
#pragma unroll
        for (int r = 0; r < 9; r++) {
            all |= (unsigned short)c[r];
            if (cc < 9) cw[12 * r] = c[r];
        }
    }
    const bool bytes = !__any_sync(0xffffffffu, (all & 0xff00ff00u) != 0u);
    __syncwarp();
    if (!bytes) {
        const size_t cat = (size_t)(m >> 1) * ru.w + (n >> 1);
        mc_any_samples(L, mvx, mvy, odd, lane, oy + (size_t)m * ry.w + n, ry.w, ou + cat, ov + cat, ru.w);
        return;
    }
    const int term = c_quarter_terms[cs], kind1 = term & 7, kind2 = (term >> 8) & 7;
    if (kind1 == kTermJ) {  // vertical sums of the window's words, two halves of eight rows
        if (lane < 24) {
            const int wd = lane < 12 ? lane : lane - 12, r0 = lane < 12 ? 0 : 8;
            unsigned x[13];
#pragma unroll
            for (int i = 0; i < 13; i++) x[i] = L.win[r0 + i][wd];
#pragma unroll
            for (int i = 0; i < 8; i++)
                L.vt[r0 + i][wd] = vppgpu::tap_pair(x[i], x[i + 1], x[i + 2], x[i + 3], x[i + 4], x[i + 5]);
        }
        __syncwarp();
    }
    const int r = 4 * r4;
    unsigned o[4];
    mc_pair_term(L, term, r, q, o);
    if (kind2 != kTermNone) {
        unsigned o2[4];
        mc_pair_term(L, term >> 8, r, q, o2);
#pragma unroll
        for (int i = 0; i < 4; i++) o[i] = ((o[i] + o2[i] + 0x00010001u) >> 1) & 0x00ff00ffu;
    }
    short* dst = oy + (size_t)(m + r) * ry.w + n + 2 * q;
#pragma unroll
    for (int i = 0; i < 4; i++) store_pair<kWide>(dst + (size_t)i * ry.w, o[i]);
    // chroma: a pair of columns of a row per lane and plane
    const int fx = mvx & 7, fy = mvy & 7, cr = lane >> 2, cp = lane & 3;
    const unsigned w00 = (8 - fx) * (8 - fy), w10 = fx * (8 - fy), w01 = (8 - fx) * fy, w11 = fx * fy;
    const size_t cat = (size_t)((m >> 1) + cr) * ru.w + (n >> 1) + 2 * cp;
#pragma unroll
    for (int pl = 0; pl < 2; pl++) {
        const unsigned *p0 = &L.cwin[9 * pl + cr][cp], *p1 = p0 + 6;
        const unsigned f0 = __funnelshift_r(p0[0], p0[1], 16), f1 = __funnelshift_r(p1[0], p1[1], 16);
        const unsigned s = w00 * (odd ? f0 : p0[0]) + w10 * (odd ? p0[1] : f0) + w01 * (odd ? f1 : p1[0]) +
                           w11 * (odd ? p1[1] : f1) + 0x00200020u;
        store_pair<kWide>((pl ? ov : ou) + cat, (s >> 6) & 0x00ff00ffu);
    }
}

// a = clip255(a + b) or a -= b, 8 samples per thread (16-byte accesses), the tail one by one.
template <bool kAdd>
__global__ void __launch_bounds__(256) k_plane_op(short* __restrict__ a, const short* __restrict__ b, long long n)
{
    const long long n8 = n >> 3;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += stride) {
        uint4 va = reinterpret_cast<const uint4*>(a)[i];
        const uint4 vb = __ldg(reinterpret_cast<const uint4*>(b) + i);
        short* sa = reinterpret_cast<short*>(&va);
        const short* sb = reinterpret_cast<const short*>(&vb);
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int r = kAdd ? sa[t] + sb[t] : sa[t] - sb[t];
            sa[t] = (short)(kAdd ? (r < 0 ? 0 : (r > 255 ? 255 : r)) : r);
        }
        reinterpret_cast<uint4*>(a)[i] = va;
    }
    for (long long i = 8 * n8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        const int r = kAdd ? a[i] + b[i] : a[i] - b[i];
        a[i] = (short)(kAdd ? (r < 0 ? 0 : (r > 255 ? 255 : r)) : r);
    }
}

int grid_for(vppgpu_ctx* ctx, long long work)
{
    long long g = (work + 255) / 256;
    const long long cap = (long long)ctx->sm_count * 16;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

struct vppgpu_mc {
    vppgpu_ctx* ctx;
    int W, H, range;
    short* d_tmp;  // the reference before compensation (Y, U, V)
    short* d_io;   // staging of the host entry point
    int* d_mv;
};

extern "C" {

int vppgpu_mc_create(vppgpu_ctx* ctx, int width, int height, int range, vppgpu_mc** out)
{
    if (!ctx || !out || width < 16 || height < 16 || (width % 16) || (height % 2) || range < 0)
        return VPPGPU_ERR_INVALID_ARG;
    *out = nullptr;
    int rc = vppgpu::bind(ctx);
    if (rc) return rc;
    vppgpu_mc* mc = new (std::nothrow) vppgpu_mc();
    if (!mc) return VPPGPU_ERR_OUT_OF_MEMORY;
    mc->ctx = ctx;
    mc->W = width;
    mc->H = height;
    mc->range = range;
    const size_t frame = (size_t)width * height * 3 / 2;
    const size_t nmb = (size_t)(width / 16) * (height / 16);
    if (cudaMalloc((void**)&mc->d_tmp, frame * sizeof(short)) != cudaSuccess ||
        cudaMalloc((void**)&mc->d_io, frame * sizeof(short)) != cudaSuccess ||
        cudaMalloc((void**)&mc->d_mv, (nmb ? nmb : 1) * sizeof(int)) != cudaSuccess) {
        cudaFree(mc->d_tmp);
        cudaFree(mc->d_io);
        delete mc;
        return VPPGPU_ERR_OUT_OF_MEMORY;
    }
    *out = mc;
    return VPPGPU_OK;
}

int vppgpu_mc_destroy(vppgpu_mc* mc)
{
    if (!mc) return VPPGPU_ERR_INVALID_ARG;
    cudaSetDevice(mc->ctx->device);
    cudaStreamSynchronize(mc->ctx->stream);
    cudaFree(mc->d_tmp);
    cudaFree(mc->d_io);
    cudaFree(mc->d_mv);
    delete mc;
    return VPPGPU_OK;
}

int vppgpu_mc_compensate_device(vppgpu_mc* mc, const short* d_ref_yuv, const short* d_mv, short* d_out_yuv)
{
    if (!mc || !d_ref_yuv || !d_mv || !d_out_yuv) return VPPGPU_ERR_INVALID_ARG;
    if (((uintptr_t)d_mv & 3) || ((uintptr_t)d_out_yuv & 1) || ((uintptr_t)d_ref_yuv & 1))
        return VPPGPU_ERR_INVALID_ARG;
    vppgpu_ctx* ctx = mc->ctx;
    int rc = vppgpu::bind(ctx);
    if (rc) return rc;
    const int W = mc->W, H = mc->H, cw = W / 2, ch = H / 2, cols = W / 16, rows = H / 16;
    const size_t ny = (size_t)W * H, nc = (size_t)cw * ch;
    // read from the frame itself unless the output overlaps it (then from a copy, as the reference does)
    const size_t frame = ny + 2 * nc;
    const short* src = d_ref_yuv;
    if (d_out_yuv < d_ref_yuv + frame && d_ref_yuv < d_out_yuv + frame) {
        VPP_CUDA(cudaMemcpyAsync(mc->d_tmp, d_ref_yuv, frame * sizeof(short), cudaMemcpyDeviceToDevice, ctx->stream));
        src = mc->d_tmp;
    }
    if (cols * rows > 0) {
        const Plane py{src, W, H}, pu{src + ny, cw, ch}, pv{src + ny + nc, cw, ch};
        const int grid = (cols * rows + kMcWarps - 1) / kMcWarps;
        const auto kernel = (((uintptr_t)src | (uintptr_t)d_out_yuv) & 15) == 0 ? k_mc_frame<true> : k_mc_frame<false>;
        kernel<<<grid, 32 * kMcWarps, 0, ctx->stream>>>(py, pu, pv, (const int*)d_mv, cols, cols * rows, d_out_yuv,
                                                        d_out_yuv + ny, d_out_yuv + ny + nc);
        VPP_CHECK_LAUNCH(ctx);
        ctx->launches++;
    }
    if (16 * rows < H) {  // rows below the last whole macroblock row keep the reference samples
        VPP_CUDA(cudaMemcpyAsync(d_out_yuv + (size_t)16 * rows * W, src + (size_t)16 * rows * W,
                                 (size_t)(H - 16 * rows) * W * sizeof(short), cudaMemcpyDeviceToDevice, ctx->stream));
        for (int p = 0; p < 2; p++) {
            const size_t o = ny + p * nc + (size_t)8 * rows * cw;
            VPP_CUDA(cudaMemcpyAsync(d_out_yuv + o, src + o, (size_t)(ch - 8 * rows) * cw * sizeof(short),
                                     cudaMemcpyDeviceToDevice, ctx->stream));
        }
    }
    return VPPGPU_OK;
}

int vppgpu_mc_compensate(vppgpu_mc* mc, short* yuv, const short* mv)
{
    if (!mc || !yuv || !mv) return VPPGPU_ERR_INVALID_ARG;
    vppgpu_ctx* ctx = mc->ctx;
    int rc = vppgpu::bind(ctx);
    if (rc) return rc;
    const size_t frame = (size_t)mc->W * mc->H * 3 / 2, nmb = (size_t)(mc->W / 16) * (mc->H / 16);
    VPP_CUDA(cudaMemcpyAsync(mc->d_io, yuv, frame * sizeof(short), cudaMemcpyHostToDevice, ctx->stream));
    VPP_CUDA(cudaMemcpyAsync(mc->d_mv, mv, nmb * sizeof(int), cudaMemcpyHostToDevice, ctx->stream));
    if ((rc = vppgpu_mc_compensate_device(mc, mc->d_io, (const short*)mc->d_mv, mc->d_io))) return rc;
    VPP_CUDA(cudaMemcpyAsync(yuv, mc->d_io, frame * sizeof(short), cudaMemcpyDeviceToHost, ctx->stream));
    VPP_CUDA(cudaStreamSynchronize(ctx->stream));
    return VPPGPU_OK;
}

static int plane_op(vppgpu_ctx* ctx, short* d_a, const short* d_b, long long n, bool add)
{
    if (!ctx || !d_a || !d_b || n < 0 || ((uintptr_t)d_a & 15) || ((uintptr_t)d_b & 15)) return VPPGPU_ERR_INVALID_ARG;
    int rc = vppgpu::bind(ctx);
    if (rc) return rc;
    if (n == 0) return VPPGPU_OK;
    const int g = grid_for(ctx, (n + 7) / 8);
    if (add)
        k_plane_op<true><<<g, 256, 0, ctx->stream>>>(d_a, d_b, n);
    else
        k_plane_op<false><<<g, 256, 0, ctx->stream>>>(d_a, d_b, n);
    VPP_CHECK_LAUNCH(ctx);
    ctx->launches++;
    return VPPGPU_OK;
}

int vppgpu_add_clip255_device(vppgpu_ctx* ctx, short* d_a, const short* d_b, long long n)
{
    return plane_op(ctx, d_a, d_b, n, true);
}

int vppgpu_sub_device(vppgpu_ctx* ctx, short* d_a, const short* d_b, long long n)
{
    return plane_op(ctx, d_a, d_b, n, false);
}

}  // extern "C"
