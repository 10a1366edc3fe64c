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

template <int kKind>
__device__ __forceinline__ unsigned pixel_luma(unsigned p)
{
    constexpr unsigned lo = (kYb & 255) | (kYg & 255) << 8 | (kYr & 255) << 16;
    constexpr unsigned hi = (kYb >> 8) | (kYg >> 8) << 8 | (kYr >> 8) << 16;
    return kKind == VPPGPU_RGB_FIXED_POINT ? __dp4a(p, lo, __dp4a(p, hi, 0u) << 8) >> 13 : (unsigned)real_luma_int(p);
}
// The chroma of a block from its pixels (row by row; the fourth byte of each is not read).
template <int kKind>
__device__ __forceinline__ void block_chroma(const unsigned (&p)[4], int chr_off, int& u, int& v)
{
    unsigned br = 0, gs = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        br += p[q] & 0x00ff00ffu;
        gs = __dp4a(p[q], 0x00000100u, gs);
    }
    const int b = (int)(br & 0xffffu), g = (int)gs, r = (int)(br >> 16);
    if (kKind == VPPGPU_RGB_FIXED_POINT) {
        u = fixed_chroma(kUr * r + kUg * g + kUb * b, chr_off);
        v = fixed_chroma(kVr * r + kVg * g + kVb * b, chr_off);
    } else {
        u = chr_off + clamp_s8(real_chroma_int<kKind == VPPGPU_RGB_REAL_IMPL2>(p, b, g, r, -147, -289, 436));
        v = chr_off + clamp_s8(real_chroma_int<kKind == VPPGPU_RGB_REAL_IMPL2>(p, b, g, r, 615, -515, -100));
    }
}

// Four 2x2 blocks per thread (8 pixels of two rows).  What bounds it beside memory is instructions: each byte by
// itself took 482 a thread, 36 us for sixteen 1920x1080 frames that move in 29.  A pixel is the low three bytes of a
// word cut out of the row; its fixed-point luma is two dp4a, by the high and the low bytes of the coefficients, and
// the chroma of a block comes from the sums of its four pixels: 353, 33 us.  The real converters (kKind)
// were bound by double arithmetic: 175 us for seven 996x568 frames, 29 from integers.
// Width a multiple of 8, aligned planes; 6 CTAs an SM (8: 33.1 us, 6: 32.8).
template <int kKind>
__global__ void __launch_bounds__(256, kKind == VPPGPU_RGB_FIXED_POINT ? 6 : 4)
    k_rgb_x8(const unsigned char* __restrict__ bgr, int w, int h, int chr_off, int flip,
                                               short* __restrict__ py, short* __restrict__ pu, short* __restrict__ pv)
{
    size_t fpix = (size_t)w * h;
    const unsigned char* src = bgr + blockIdx.y * fpix * 3;
    short* Y = py + blockIdx.y * fpix;
    short* U = pu + blockIdx.y * (fpix / 4);
    short* V = pv + blockIdx.y * (fpix / 4);
    const unsigned groups_x = (unsigned)w >> 3;
    const long long ngroups = (long long)groups_x * (h >> 1);
    for (long long gi = blockIdx.x * (long long)blockDim.x + threadIdx.x; gi < ngroups;
         gi += (long long)gridDim.x * blockDim.x) {
        const int yb = ngroups >> 32 ? (int)(gi / groups_x) : (int)((unsigned)gi / groups_x);
        const int x0 = (int)(gi - (long long)yb * groups_x) * 8, y0 = 2 * yb;
        unsigned px[2][8];
        uint4 lum[2];
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const int sy = kKind != VPPGPU_RGB_FIXED_POINT && flip ? h - 1 - (y0 + rr) : y0 + rr;
            const unsigned char* row = src + ((size_t)sy * w + x0) * 3;
            const uint2* s = reinterpret_cast<const uint2*>(row);
            const uint2 a = __ldg(s), b = __ldg(s + 1), c = __ldg(s + 2);
            const unsigned in[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
#pragma unroll
            for (int g = 0; g < 2; g++) {  // twelve bytes are four pixels (the fourth byte of each: the next pixel's)
                px[rr][4 * g] = in[3 * g];
                px[rr][4 * g + 1] = __funnelshift_r(in[3 * g], in[3 * g + 1], 24);
                px[rr][4 * g + 2] = __funnelshift_r(in[3 * g + 1], in[3 * g + 2], 16);
                px[rr][4 * g + 3] = in[3 * g + 2] >> 8;
            }
            unsigned yv[8];
#pragma unroll
            for (int i = 0; i < 8; i++) yv[i] = pixel_luma<kKind>(px[rr][i]);
            lum[rr] = make_uint4(__byte_perm(yv[0], yv[1], 0x5410), __byte_perm(yv[2], yv[3], 0x5410),
                                 __byte_perm(yv[4], yv[5], 0x5410), __byte_perm(yv[6], yv[7], 0x5410));
        }
        int uo[4], vo[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned p[4] = {px[0][2 * k], px[0][2 * k + 1], px[1][2 * k], px[1][2 * k + 1]};
            block_chroma<kKind>(p, chr_off, uo[k], vo[k]);
        }
        size_t co = (size_t)yb * (w >> 1) + (x0 >> 1);
#pragma unroll
        for (int rr = 0; rr < 2; rr++) *reinterpret_cast<uint4*>(Y + (size_t)(y0 + rr) * w + x0) = lum[rr];
        *reinterpret_cast<uint2*>(U + co) = make_uint2(pack2(uo[0], uo[1]), pack2(uo[2], uo[3]));
        *reinterpret_cast<uint2*>(V + co) = make_uint2(pack2(vo[0], vo[1]), pack2(vo[2], vo[3]));
    }
}

// Any even width and any alignment: one 2x2 block per thread, so that a warp's accesses are to neighbouring bytes
// whatever the row's address.  Two pixels of a row are six bytes from any address: the two or three aligned words
// around them.  (Eight pixels a thread in 4-byte accesses scattered a warp's stores: seven 996x568 frames by the real
// converter 29.5 us, 25.8 so; eight 1366x768 frames in fixed point 21 both ways.)
template <int kKind>
__global__ void __launch_bounds__(256) k_rgb_block(const unsigned char* __restrict__ bgr, int w, int h, int chr_off,
                                                  int flip, short* __restrict__ py, short* __restrict__ pu,
                                                  short* __restrict__ pv)
{
    const size_t fpix = (size_t)w * h;
    const unsigned char* src = bgr + blockIdx.y * fpix * 3;
    short* Y = py + blockIdx.y * fpix;
    short* U = pu + blockIdx.y * (fpix / 4);
    short* V = pv + blockIdx.y * (fpix / 4);
    const bool pairs = (reinterpret_cast<uintptr_t>(py) & 3) == 0;
    const unsigned xb_n = (unsigned)w >> 1;
    const long long n = (long long)xb_n * (h >> 1);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int yb = n >> 32 ? (int)(i / xb_n) : (int)((unsigned)i / xb_n), xb = (int)(i - (long long)yb * xb_n);
        unsigned p[4];
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const int yy = 2 * yb + rr, sy = kKind != VPPGPU_RGB_FIXED_POINT && flip ? h - 1 - yy : yy;
            const unsigned char* t = src + ((size_t)sy * w + 2 * xb) * 3;
            const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(t) & 3);
            const unsigned* s = reinterpret_cast<const unsigned*>(t - off);
            const unsigned v0 = __ldg(s), v1 = __ldg(s + 1), v2 = off == 3 ? __ldg(s + 2) : 0u;
            const unsigned a = __funnelshift_r(v0, v1, 8 * off), b = __funnelshift_r(v1, v2, 8 * off);
            p[2 * rr] = a;
            p[2 * rr + 1] = __funnelshift_r(a, b, 24);
            const unsigned y0 = pixel_luma<kKind>(p[2 * rr]), y1 = pixel_luma<kKind>(p[2 * rr + 1]);
            short* d = Y + (size_t)yy * w + 2 * xb;
            if (pairs) {
                *reinterpret_cast<unsigned*>(d) = y0 | y1 << 16;
            } else {
                d[0] = (short)y0;
                d[1] = (short)y1;
            }
        }
        int u, v;
        block_chroma<kKind>(p, chr_off, u, v);
        U[(size_t)yb * xb_n + xb] = (short)u;
        V[(size_t)yb * xb_n + xb] = (short)v;
    }
}

template <int kKind>
void launch_kind(vppgpu_ctx* ctx, const unsigned char* bgr, int nframes, int w, int h, int chr_off, int flip, short* y,
                 short* u, short* v)
{
    // Eight pixels a thread with 8- and 16-byte accesses where rows and planes are aligned to them.  A pixel of the
    // real kinds can be a chain of doubles (luma or chroma on a whole number), so theirs also have to fill the GPU, two
    // CTAs an SM: a 176x144 frame of colours in steps of 50 took 30.8 us by eight a thread and 11.4 by a block (10.3
    // before either); pictures, one 640x480 frame 8.2 and 6.1, one 1280x720 frame 8.3 both, one 1920x1080 frame 8.3
    // and 9.3, eight 33.0 and 45.2.
    const uintptr_t a16 = (uintptr_t)y, a8 = (uintptr_t)u | (uintptr_t)v | (uintptr_t)bgr;
    const long long eights = ((long long)(w >> 3) * (h >> 1) + 255) / 256 * nframes;
    const bool wide = (w & 7) == 0 && (a16 & 15) == 0 && (a8 & 7) == 0 &&
                      (kKind == VPPGPU_RGB_FIXED_POINT || eights >= 2 * ctx->sm_count);
    const long long work = (long long)(w >> (wide ? 3 : 1)) * (h >> 1), blocks = (work + 255) / 256;
    const dim3 grid((unsigned)(blocks < 4096 ? blocks : 4096), nframes);
    if (wide) k_rgb_x8<kKind><<<grid, 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip, y, u, v);
    else k_rgb_block<kKind><<<grid, 256, 0, ctx->stream>>>(bgr, w, h, chr_off, flip, y, u, v);
}

int launch(vppgpu_ctx* ctx, int kind, const unsigned char* bgr, int nframes, int w, int h, int chr_off,
           int flip, short* y, short* u, short* v)
{
    if (kind == VPPGPU_RGB_FIXED_POINT)
        launch_kind<VPPGPU_RGB_FIXED_POINT>(ctx, bgr, nframes, w, h, chr_off, flip != 0, y, u, v);
    else if (kind == VPPGPU_RGB_REAL)
        launch_kind<VPPGPU_RGB_REAL>(ctx, bgr, nframes, w, h, chr_off, flip != 0, y, u, v);
    else
        launch_kind<VPPGPU_RGB_REAL_IMPL2>(ctx, bgr, nframes, w, h, chr_off, flip != 0, y, u, v);
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
