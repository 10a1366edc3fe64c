// colour.cu -- packed BGR24 -> planar YUV 4:2:0 (short planes) for sm_103a.
//
//   fixed point: FastFixedPointRGB24toYUV420Converter::Convert
//                (src/ImageUtils/FastFixedPointRGB24toYUV420Converter.cpp:94-169)
//   real:        RealRGB24toYUV420Converter::{NonFlip,Flip}Convert
//                (src/ImageUtils/RealRGB24toYUV420Converter.cpp:83-242)
//   real impl2:  RealRGB24toYUV420ConverterImpl2 (…ConverterImpl2.cpp:104-262)
//
// HBM-bound: 3 B in and 3 B out (Y + quarter-size U, V as int16) per pixel.
// The fixed-point kernel gives each thread four horizontally adjacent 2x2
// pixel blocks, so a row of its input is three aligned 8-byte loads and its
// luma output one 16-byte store.  The real converters' double arithmetic is
// done in integers where that provably gives the same; elsewhere they round
// after every operation (__dmul_rn/__dadd_rn) exactly like the reference's
// left-to-right evaluation with no FMA contraction.
#include "vppgpu_internal.cuh"

namespace {

// (int)(0.5 + c * 8192) as the reference's static_cast does (…FixedPoint….cpp:65-74).
constexpr int fixed_coef(double c) { return (int)(0.5 + c * (double)(2 << 12)); }
constexpr int kYr = fixed_coef(0.299), kYg = fixed_coef(0.587), kYb = fixed_coef(0.114);
constexpr int kUr = fixed_coef(-0.147), kUg = fixed_coef(-0.289), kUb = fixed_coef(0.436);
constexpr int kVr = fixed_coef(0.615), kVg = fixed_coef(-0.515), kVb = fixed_coef(-0.100);
static_assert(kYr + kYg + kYb == 8192 && kYr > 0 && kYg > 0 && kYb > 0, "a luma needs no clip");

__device__ __forceinline__ int clamp_s8(int x) { return min(max(x, -128), 127); }

__device__ __forceinline__ void fixed_pixel(int b, int g, int r, int& y, int& u, int& v)
{
    y = (kYr * r + kYg * g + kYb * b) >> 13;
    u += kUr * r + kUg * g + kUb * b;
    v += kVr * r + kVg * g + kVb * b;
}

__device__ __forceinline__ int fixed_chroma(int acc, int chr_off)
{
    int t = acc >> 13;
    t += t < 0 ? -2 : 2;
    return chr_off + clamp_s8(t >> 2);
}

__device__ __forceinline__ unsigned pack2(int a, int b) { return (unsigned)(a & 0xffff) | ((unsigned)b << 16); }

// Real converters: IEEE double, one rounding per operation, left to right.
__device__ __forceinline__ double lin3(double k0, double k1, double k2, double r, double g, double b)
{
    return __dadd_rn(__dadd_rn(__dmul_rn(k0, r), __dmul_rn(k1, g)), __dmul_rn(k2, b));
}

// One pixel's luma and one block's chroma term sums in double, the reference's order of operations.
// impl2: the mean is rounded in double.
__device__ __noinline__ int real_luma(unsigned p)
{
    const double b = (double)(p & 255u), g = (double)((p >> 8) & 255u), r = (double)((p >> 16) & 255u);
    return clip255(__double2int_rz(
        __dadd_rn(__dadd_rn(__dadd_rn(0.5, __dmul_rn(0.299, r)), __dmul_rn(0.587, g)), __dmul_rn(0.114, b))));
}
__device__ __forceinline__ int real_mean(double u, bool impl2)
{
    if (!impl2) {
        int iu = __double2int_rz(u);
        iu += iu < 0 ? -2 : 2;
        return iu / 4;
    }
    const double au = __ddiv_rn(u, 4.0);
    return __double2int_rz(u < 0.0 ? __dsub_rn(au, 0.5) : __dadd_rn(au, 0.5));
}
__device__ __noinline__ int real_chroma(unsigned p0, unsigned p1, unsigned p2, unsigned p3, double k0, double k1,
                                        double k2, bool impl2)
{
    const unsigned p[4] = {p0, p1, p2, p3};
    double u = 0.0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const double t = lin3(k0, k1, k2, (double)((p[q] >> 16) & 255u), (double)((p[q] >> 8) & 255u),
                              (double)(p[q] & 255u));
        u = q ? __dadd_rn(u, t) : t;
    }
    return real_mean(u, impl2);
}

// The same from integers.  The coefficients are thousandths, so the exact luma is n / 1000 and the exact chroma sum
// m / 1000, while the doubles are within 1e-11 of them: where no truncation lies on the exact value both truncate
// alike.  (A chroma sum of 0 truncates to 0 with either sign of an error.)
__device__ __forceinline__ int real_luma_int(unsigned p)
{
    constexpr unsigned lo = (114 & 255) | (587 & 255) << 8 | (299 & 255) << 16, hi = 0u | (587 >> 8) << 8 | (299 >> 8) << 16;
    const unsigned n = __dp4a(p, lo, (__dp4a(p, hi, 0u) << 8) + 500u), y = n / 1000u;
    return n == 1000u * y ? real_luma(p) : (int)y;
}
template <bool kImpl2>
__device__ __forceinline__ int real_chroma_int(const unsigned (&p)[4], int b, int g, int r, int k0, int k1, int k2)
{
    const int m = k0 * r + k1 * g + k2 * b;
    int iu;
    bool near;
    if (kImpl2) {
        const int t = m + (m < 0 ? -2000 : 2000);
        iu = t / 4000;
        near = t == 4000 * iu;
    } else {
        iu = m / 1000;
        near = m == 1000 * iu && m != 0;
        iu = (iu + (iu < 0 ? -2 : 2)) / 4;
    }
    // the reference's decimal constants, correctly rounded: what k / 1000 gives
    return near ? real_chroma(p[0], p[1], p[2], p[3], __ddiv_rn((double)k0, 1000.0), __ddiv_rn((double)k1, 1000.0),
                              __ddiv_rn((double)k2, 1000.0), kImpl2)
                : iu;
}

// Four 2x2 blocks per thread (8 pixels of two rows).  What bounds it beside memory is instructions: each byte by
// itself took 482 a thread, 36 us for sixteen 1920x1080 frames that move in 29.  A pixel is the low three bytes of a
// word cut out of the row; its fixed-point luma is two dp4a, by the high and the low bytes of the coefficients, and
// the chroma of a block comes from the sums of its four pixels: 353, 33 us.  The real converters (kKind)
// were bound by double arithmetic: 175 us for seven 996x568 frames, 29 from integers.
// kWide: width a multiple of 8 and aligned planes; else (width of 8 or more, luma 4-byte aligned) rows are read
// from any address as the aligned words around them, and the last group of a row ends at its end, sharing pixels
// with the one before (both write the same).
template <int kKind, bool kWide>
__global__ void __launch_bounds__(256) k_rgb_x8(const unsigned char* __restrict__ bgr, int w, int h, int chr_off, int flip,
                                               short* __restrict__ py, short* __restrict__ pu, short* __restrict__ pv)
{
    constexpr unsigned lo = (kYb & 255) | (kYg & 255) << 8 | (kYr & 255) << 16;
    constexpr unsigned hi = (kYb >> 8) | (kYg >> 8) << 8 | (kYr >> 8) << 16;
    size_t fpix = (size_t)w * h;
    const unsigned char* src = bgr + blockIdx.y * fpix * 3;
    short* Y = py + blockIdx.y * fpix;
    short* U = pu + blockIdx.y * (fpix / 4);
    short* V = pv + blockIdx.y * (fpix / 4);
    const unsigned groups_x = ((unsigned)w + 7) >> 3;
    const long long ngroups = (long long)groups_x * (h >> 1);
    for (long long gi = blockIdx.x * (long long)blockDim.x + threadIdx.x; gi < ngroups;
         gi += (long long)gridDim.x * blockDim.x) {
        const int yb = ngroups >> 32 ? (int)(gi / groups_x) : (int)((unsigned)gi / groups_x);
        const int x0 = min((int)(gi - (long long)yb * groups_x) * 8, w - 8), y0 = 2 * yb;
        unsigned px[2][8];
        uint4 lum[2];
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const int sy = kKind != VPPGPU_RGB_FIXED_POINT && flip ? h - 1 - (y0 + rr) : y0 + rr;
            const unsigned char* row = src + ((size_t)sy * w + x0) * 3;
            unsigned in[6];
            if (kWide) {
                const uint2* s = reinterpret_cast<const uint2*>(row);
                const uint2 a = __ldg(s), b = __ldg(s + 1), c = __ldg(s + 2);
                in[0] = a.x, in[1] = a.y, in[2] = b.x, in[3] = b.y, in[4] = c.x, in[5] = c.y;
            } else {
                const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(row) & 3);
                const unsigned* s = reinterpret_cast<const unsigned*>(row - off);
                unsigned v[7];
#pragma unroll
                for (int i = 0; i < 6; i++) v[i] = __ldg(s + i);
                v[6] = off ? __ldg(s + 6) : 0u;  // else past the row
#pragma unroll
                for (int i = 0; i < 6; i++) in[i] = __funnelshift_r(v[i], v[i + 1], 8 * off);
            }
#pragma unroll
            for (int g = 0; g < 2; g++) {  // twelve bytes are four pixels (the fourth byte of each: the next pixel's)
                px[rr][4 * g] = in[3 * g];
                px[rr][4 * g + 1] = __funnelshift_r(in[3 * g], in[3 * g + 1], 24);
                px[rr][4 * g + 2] = __funnelshift_r(in[3 * g + 1], in[3 * g + 2], 16);
                px[rr][4 * g + 3] = in[3 * g + 2] >> 8;
            }
            unsigned yv[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                yv[i] = kKind == VPPGPU_RGB_FIXED_POINT ? __dp4a(px[rr][i], lo, __dp4a(px[rr][i], hi, 0u) << 8) >> 13
                                                        : (unsigned)real_luma_int(px[rr][i]);
            lum[rr] = make_uint4(__byte_perm(yv[0], yv[1], 0x5410), __byte_perm(yv[2], yv[3], 0x5410),
                                 __byte_perm(yv[4], yv[5], 0x5410), __byte_perm(yv[6], yv[7], 0x5410));
        }
        int uo[4], vo[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned p[4] = {px[0][2 * k], px[0][2 * k + 1], px[1][2 * k], px[1][2 * k + 1]};
            unsigned br = 0, gs = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                br += p[q] & 0x00ff00ffu;
                gs = __dp4a(p[q], 0x00000100u, gs);
            }
            const int b = (int)(br & 0xffffu), g = (int)gs, r = (int)(br >> 16);
            if (kKind == VPPGPU_RGB_FIXED_POINT) {
                uo[k] = fixed_chroma(kUr * r + kUg * g + kUb * b, chr_off);
                vo[k] = fixed_chroma(kVr * r + kVg * g + kVb * b, chr_off);
            } else {
                uo[k] = chr_off + clamp_s8(real_chroma_int<kKind == VPPGPU_RGB_REAL_IMPL2>(p, b, g, r, -147, -289, 436));
                vo[k] = chr_off + clamp_s8(real_chroma_int<kKind == VPPGPU_RGB_REAL_IMPL2>(p, b, g, r, 615, -515, -100));
            }
        }
        size_t co = (size_t)yb * (w >> 1) + (x0 >> 1);
        if (kWide) {
#pragma unroll
            for (int rr = 0; rr < 2; rr++) *reinterpret_cast<uint4*>(Y + (size_t)(y0 + rr) * w + x0) = lum[rr];
            *reinterpret_cast<uint2*>(U + co) = make_uint2(pack2(uo[0], uo[1]), pack2(uo[2], uo[3]));
            *reinterpret_cast<uint2*>(V + co) = make_uint2(pack2(vo[0], vo[1]), pack2(vo[2], vo[3]));
        } else {
#pragma unroll
            for (int rr = 0; rr < 2; rr++) {
                unsigned* d = reinterpret_cast<unsigned*>(Y + (size_t)(y0 + rr) * w + x0);
                d[0] = lum[rr].x, d[1] = lum[rr].y, d[2] = lum[rr].z, d[3] = lum[rr].w;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                U[co + k] = (short)uo[k];
                V[co + k] = (short)vo[k];
            }
        }
    }
}

// Generic fixed-point path: one 2x2 block per thread (any even width).
__global__ void __launch_bounds__(256) k_rgb_fixed(const unsigned char* __restrict__ bgr, int w, int h,
                                                  int chr_off, short* __restrict__ py,
                                                  short* __restrict__ pu, short* __restrict__ pv)
{
    size_t fpix = (size_t)w * h;
    const unsigned char* src = bgr + blockIdx.y * fpix * 3;
    short* Y = py + blockIdx.y * fpix;
    short* U = pu + blockIdx.y * (fpix / 4);
    short* V = pv + blockIdx.y * (fpix / 4);
    int xb_n = w >> 1, yb_n = h >> 1;
    long long n = (long long)xb_n * yb_n;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int yb = (int)(i / xb_n), xb = (int)(i - (long long)yb * xb_n);
        int u = 0, v = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int yy = 2 * yb + (q >> 1), xx = 2 * xb + (q & 1);
            const unsigned char* t = src + ((size_t)yy * w + xx) * 3;
            int yv;
            fixed_pixel(t[0], t[1], t[2], yv, u, v);
            Y[(size_t)yy * w + xx] = (short)yv;
        }
        U[(size_t)yb * xb_n + xb] = (short)fixed_chroma(u, chr_off);
        V[(size_t)yb * xb_n + xb] = (short)fixed_chroma(v, chr_off);
    }
}

__global__ void __launch_bounds__(256) k_rgb_real(const unsigned char* __restrict__ bgr, int w, int h, int chr_off,
                                                 int flip, int impl2, short* __restrict__ py,
                                                 short* __restrict__ pu, short* __restrict__ pv)
{
    const double K00 = 0.299, K01 = 0.587, K02 = 0.114;
    const double K10 = -0.147, K11 = -0.289, K12 = 0.436;
    const double K20 = 0.615, K21 = -0.515, K22 = -0.100;
    size_t fpix = (size_t)w * h;
    const unsigned char* src = bgr + blockIdx.y * fpix * 3;
    short* Y = py + blockIdx.y * fpix;
    short* U = pu + blockIdx.y * (fpix / 4);
    short* V = pv + blockIdx.y * (fpix / 4);
    int xb_n = w >> 1, yb_n = h >> 1;
    long long n = (long long)xb_n * yb_n;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        int yb = (int)(i / xb_n), xb = (int)(i - (long long)yb * xb_n);
        double u = 0.0, v = 0.0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            int yy = 2 * yb + (q >> 1), xx = 2 * xb + (q & 1);
            int sy = flip ? (h - 1 - yy) : yy;
            const unsigned char* t = src + ((size_t)sy * w + xx) * 3;
            double b = (double)t[0], g = (double)t[1], r = (double)t[2];
            double yl = __dadd_rn(__dadd_rn(__dadd_rn(0.5, __dmul_rn(K00, r)), __dmul_rn(K01, g)), __dmul_rn(K02, b));
            Y[(size_t)yy * w + xx] = (short)clip255(__double2int_rz(yl));
            double uu = lin3(K10, K11, K12, r, g, b);
            double vv = lin3(K20, K21, K22, r, g, b);
            if (q == 0) {
                u = uu;
                v = vv;
            } else {
                u = __dadd_rn(u, uu);
                v = __dadd_rn(v, vv);
            }
        }
        int iu, iv;
        if (!impl2) {
            iu = __double2int_rz(u);
            iv = __double2int_rz(v);
            iu += iu < 0 ? -2 : 2;
            iv += iv < 0 ? -2 : 2;
            iu /= 4;
            iv /= 4;
        } else {
            double au = __ddiv_rn(u, 4.0), av = __ddiv_rn(v, 4.0);
            au = u < 0.0 ? __dsub_rn(au, 0.5) : __dadd_rn(au, 0.5);
            av = v < 0.0 ? __dsub_rn(av, 0.5) : __dadd_rn(av, 0.5);
            iu = __double2int_rz(au);
            iv = __double2int_rz(av);
        }
        U[(size_t)yb * xb_n + xb] = (short)(chr_off + clamp_s8(iu));
        V[(size_t)yb * xb_n + xb] = (short)(chr_off + clamp_s8(iv));
    }
}

template <bool kWide>
void launch_x8(vppgpu_ctx* ctx, int kind, const unsigned char* bgr, int nframes, int w, int h, int chr_off, int flip,
               short* y, short* u, short* v)
{
    const long long groups = (long long)((w + 7) >> 3) * (h >> 1), blocks = (groups + 255) / 256;
    const dim3 grid((unsigned)(blocks < 4096 ? blocks : 4096), nframes);
    if (kind == VPPGPU_RGB_FIXED_POINT)
        k_rgb_x8<VPPGPU_RGB_FIXED_POINT, kWide><<<grid, 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip, y, u, v);
    else if (kind == VPPGPU_RGB_REAL)
        k_rgb_x8<VPPGPU_RGB_REAL, kWide><<<grid, 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip, y, u, v);
    else
        k_rgb_x8<VPPGPU_RGB_REAL_IMPL2, kWide><<<grid, 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip, y, u, v);
}

int launch(vppgpu_ctx* ctx, int kind, const unsigned char* bgr, int nframes, int w, int h, int chr_off,
           int flip, short* y, short* u, short* v)
{
    const long long per = (long long)(w >> 1) * (h >> 1);
    // eight pixels a thread with 8- and 16-byte accesses, or 4-byte ones; a block a thread for what is left
    const uintptr_t out16 = (uintptr_t)y, out8 = (uintptr_t)u | (uintptr_t)v | (uintptr_t)bgr;
    if ((w & 7) == 0 && (out16 & 15) == 0 && (out8 & 7) == 0) {
        launch_x8<true>(ctx, kind, bgr, nframes, w, h, chr_off, flip != 0, y, u, v);
    } else if (w >= 8 && (out16 & 3) == 0 && ((uintptr_t)u & 1) == 0 && ((uintptr_t)v & 1) == 0) {
        launch_x8<false>(ctx, kind, bgr, nframes, w, h, chr_off, flip != 0, y, u, v);
    } else {
        const int gx = (int)(per + 255 < 4096 * 256 ? (per + 255) / 256 : 4096);
        if (kind == VPPGPU_RGB_FIXED_POINT)
            k_rgb_fixed<<<dim3(gx, nframes), 256, 0, ctx->stream>>>(bgr, w, h, chr_off, y, u, v);
        else
            k_rgb_real<<<dim3(gx, nframes), 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip != 0,
                                                                   kind == VPPGPU_RGB_REAL_IMPL2, y, u, v);
    }
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

int check(vppgpu_ctx* ctx, int kind, const void* bgr, int w, int h, const void* y, const void* u, const void* v)
{
    if (!ctx || !bgr || !y || !u || !v || w < 2 || h < 2 || (w & 1) || (h & 1)) return VPPGPU_ERR_INVALID_ARG;
    if (kind < VPPGPU_RGB_FIXED_POINT || kind > VPPGPU_RGB_REAL_IMPL2) return VPPGPU_ERR_INVALID_ARG;
    return VPPGPU_OK;
}

}  // namespace

extern "C" {

int vppgpu_rgb24_to_yuv420_device(vppgpu_ctx* ctx, int kind, const unsigned char* d_bgr, int w, int h,
                                  int chr_off, int flip, short* d_y, short* d_u, short* d_v)
{
    int rc = check(ctx, kind, d_bgr, w, h, d_y, d_u, d_v);
    if (rc) return rc;
    if ((rc = vppgpu::bind(ctx))) return rc;
    return launch(ctx, kind, d_bgr, 1, w, h, chr_off, flip, d_y, d_u, d_v);
}

int vppgpu_rgb24_to_yuv420_frames_device(vppgpu_ctx* ctx, int kind, const unsigned char* d_bgr, int nframes,
                                         int w, int h, int chr_off, int flip, short* d_y, short* d_u,
                                         short* d_v)
{
    int rc = check(ctx, kind, d_bgr, w, h, d_y, d_u, d_v);
    if (rc) return rc;
    if (nframes < 1 || nframes > 65535) return VPPGPU_ERR_INVALID_ARG;
    if ((rc = vppgpu::bind(ctx))) return rc;
    return launch(ctx, kind, d_bgr, nframes, w, h, chr_off, flip, d_y, d_u, d_v);
}

int vppgpu_rgb24_to_yuv420(vppgpu_ctx* ctx, int kind, const unsigned char* bgr, int w, int h, int chr_off,
                           int flip, short* y, short* u, short* v)
{
    int rc = check(ctx, kind, bgr, w, h, y, u, v);
    if (rc) return rc;
    if ((rc = vppgpu::bind(ctx))) return rc;
    size_t nin = (size_t)w * h * 3, ny = (size_t)w * h * 2, nc = (size_t)(w / 2) * (h / 2) * 2;
    unsigned char* d = nullptr;
    // 16-byte aligned sub-buffers
    size_t o_y = (nin + 255) & ~(size_t)255, o_u = o_y + ((ny + 255) & ~(size_t)255),
           o_v = o_u + ((nc + 255) & ~(size_t)255), tot = o_v + nc;
    VPP_CUDA(cudaMallocAsync((void**)&d, tot, ctx->stream));
    cudaError_t e = cudaMemcpyAsync(d, bgr, nin, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess) {
        rc = launch(ctx, kind, d, 1, w, h, chr_off, flip, (short*)(d + o_y), (short*)(d + o_u), (short*)(d + o_v));
        if (rc == VPPGPU_OK) e = cudaMemcpyAsync(y, d + o_y, ny, cudaMemcpyDeviceToHost, ctx->stream);
        if (rc == VPPGPU_OK && e == cudaSuccess) e = cudaMemcpyAsync(u, d + o_u, nc, cudaMemcpyDeviceToHost, ctx->stream);
        if (rc == VPPGPU_OK && e == cudaSuccess) e = cudaMemcpyAsync(v, d + o_v, nc, cudaMemcpyDeviceToHost, ctx->stream);
    }
    cudaFreeAsync(d, ctx->stream);
    cudaError_t e2 = cudaStreamSynchronize(ctx->stream);
    if (rc) return rc;
    if (e != cudaSuccess) return vppgpu::cuda_status(e);
    if (e2 != cudaSuccess) return vppgpu::cuda_status(e2);
    return VPPGPU_OK;
}

}  // extern "C"
