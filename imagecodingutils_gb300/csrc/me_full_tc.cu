// me_full_tc.cu -- the SSD full search's table on the tensor cores: the
// minimum of every candidate row of every macroblock
// (MotionEstimatorH264ImplFull.cpp:394-446 compares the SSDs of the range's
// (2R+1)^2 candidates).
//
// SSD = A^2 + B^2 - 2 sum(ab): A^2 is the macroblock's, B^2 lies in the
// energy plane, and the cross terms sum(ab) are a contraction: 128 candidate
// positions x 256 pixels times 256 pixels x the macroblocks that search there.
// All three are formed from samples less 128 (the SSD does not change), which
// are whole numbers of at most 8 bits, exact in f16; products and their sums
// stay below 2^22 in magnitude, exact in the f32 accumulator in any order, and
// B^2 - 2 sum(ab) below 2^24.  The result is the integer result.
//
// Operands without an im2col copy: in the unswizzled K-major layout a core
// matrix is 8 rows of 16 bytes, 128 bytes in a row.  With 8 pixels (f16) per
// row, 64 consecutive pixels of a picture row are the core matrix of the
// positions x, x+8, .., x+56 at 8 of the block's columns; the block's other
// columns start 16 bytes on (the leading byte offset), the positions one
// picture row down a pitch on (the stride byte offset).  So one descriptor on
// plain picture rows gives the 128 positions {x0 + 8r} x {y0 .. y0+15} for one
// block row, and the block's next row is the same descriptor a pitch on: 16
// MMAs (M 128, N 32, K 16) accumulate the cross terms of a tile.  The eight
// phases x0 mod 8 need eight copies of the rows, each a pixel further, because
// operands start at 16-byte boundaries.
//
// A unit of work is 64 columns of positions and up to T tiles of 16 rows.  A
// tile is searched by macroblocks of 4 rows (-16 .. +32 from its top) and 7
// columns (-16 .. +80), so N = 4 x 8.  The accumulators of a tile are eight
// slots of 32 columns, one per phase (a lane is a position); two tiles' fit in
// TMEM.  Eight warps read them, each two macroblock rows of 32 positions, add
// the energies and keep, per macroblock, the minimum over the phases, i.e. over
// 8 neighbouring columns.  These minima of 8 candidates are the result (a row of
// candidates is 8 of them, aligned with the macroblock): the scan reads which
// rows, and which 8 candidates of a row, can win.
//
// Persistent, one CTA per SM: eight warps stage the next unit's operands and
// eight read the last tile's accumulators while one thread of each of four warps
// issues the MMAs of this one, two phases each, so that the MMAs run back to
// back.  The hand-offs are mbarriers with bounded waits, two of each kind: a
// unit's operands filled (every staging thread arrives) and freed (the four
// issuing threads' commits), a tile's accumulators full (the same commits) and
// empty (one arrival of each reading warp); at the end every issuing thread waits
// for its own MMAs (drain).
//
// Bound: the MMAs' read of the A operand, 4 KB at 128 bytes a cycle: 32 cycles
// each, 33 measured (N = 16 takes the same).  1080p, motionRange 128: 49 us, of
// which the MMAs 31, against 165 for the dp4a table it replaces (which ran at
// 0.6 of the dp4a rate); 4K 158 us, CIF 8.3.
#include "me_full_common.cuh"

namespace vppgpu {
namespace {
using namespace full;

constexpr int TC_EPI_WARPS = 8;         // the 128 positions of a tile, for two macroblock rows each
// MMA issue: a thread of each, two phases each.  A single thread issued an MMA every 41 to 67 cycles, by how the
// compiler formed the descriptors; two threads get the 33 that the A operand's read takes at nearly every one.
constexpr int TC_MMA_WARPS = 4;
constexpr int TC_FILL_WARPS = 8;
constexpr int TC_THREADS = 32 * (TC_EPI_WARPS + TC_MMA_WARPS + TC_FILL_WARPS);
// bytes of a picture row in shared memory: 72 f16 (144 bytes) at a pitch that keeps core matrices at 64-byte
// boundaries (pitches 144, 160, 176, 208 .. 288 took 1.23 times as long in an MMA loop, 128 as long as 192)
constexpr int TC_PITCH = 192;
constexpr int TC_CHUNKS = 9;            // 16-byte pieces of a row
constexpr int TC_PHASES = 8;
constexpr int TC_SLOTS = 2 * TC_PHASES; // accumulators: one per phase, of two tiles
constexpr int TC_N = 32;                // macroblocks of a tile: 4 rows x 8 columns
constexpr int TC_TMEM = TC_SLOTS * TC_N;
constexpr int TC_BROW = 16 * 256;       // bytes of a row of 8 templates: 16 x 2 core matrices
constexpr int TC_TILES = 2;
// f16 x f16 -> f32, A and B K-major, M 128, N 32
constexpr unsigned TC_IDESC = (1u << 4) | ((TC_N / 8) << 17) | ((128 / 16) << 24);

__host__ __device__ constexpr int tc_rows(int tiles) { return 16 * tiles + 15; }
__host__ __device__ constexpr int tc_buffer(int tiles)
{
    return TC_PHASES * tc_rows(tiles) * TC_PITCH + (tiles + 3) * TC_BROW;
}

// Shared-memory matrix descriptor, no swizzle: `lead` bytes between the two
// core matrices of K, `stride` bytes between core matrices of M or N.
__device__ __forceinline__ unsigned long long tc_desc(unsigned addr, unsigned lead, unsigned stride)
{
    return (unsigned long long)((addr >> 4) & 0x3fff) | ((unsigned long long)(lead >> 4) << 16) |
           ((unsigned long long)(stride >> 4) << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_mma(unsigned d, unsigned long long a, unsigned long long b, bool accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(TC_IDESC), "r"((int)accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(unsigned long long* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// 16 consecutive accumulator columns of this warp's 32 lanes.
__device__ __forceinline__ void tc_load16(unsigned addr, float* v)
{
    unsigned u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
          "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(u[i]);
}

// Two samples (bytes p of w, selected by the permutation `sel`) less 128, as f16.
__device__ __forceinline__ unsigned half2_less128(unsigned w, unsigned sel)
{
    unsigned h = __byte_perm(w, 0x64646464u, sel);  // 0x6400 | b: 1024 + b
    unsigned r;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(h), "r"(0x64806480u));  // - 1152
    return r;
}
__device__ __forceinline__ uint4 eight_less128(unsigned lo, unsigned hi)
{
    return make_uint4(half2_less128(lo, 0x4140), half2_less128(lo, 0x4342), half2_less128(hi, 0x4140),
                      half2_less128(hi, 0x4342));
}

// Tiles in column-window order, `high` of them in a window; a CTA takes a run
// of them (all CTAs' runs within one tile of each other), in units of up to
// TC_TILES neighbouring tiles that share their staged rows.
struct TcGrid {
    int high, run, more, phase;
};
struct TcUnit {
    int x0, y0, nt;  // first position, tiles
};

__global__ void __launch_bounds__(TC_THREADS, 1) k_ssd_rowmin(const __grid_constant__ FullArgs a, const TcGrid g)
{
    extern __shared__ __align__(128) unsigned char tc_raw[];
    __shared__ unsigned long long s_filled[2], s_freed[2], s_full[2], s_empty[2], s_drain;
    __shared__ unsigned s_tmem;
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rows = a.nmb / a.cols;
    constexpr int phase = tc_rows(TC_TILES) * TC_PITCH, buffer = tc_buffer(TC_TILES);
    // the first g.more CTAs take a tile more than the others
    const int first = (int)blockIdx.x * g.run + min((int)blockIdx.x, g.more);
    const int last = first + g.run + ((int)blockIdx.x < g.more ? 1 : 0);

    if (warp == TC_EPI_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_tmem)),
                     "r"(TC_TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < 2; b++) {
            mbar_init(&s_filled[b], 32 * TC_FILL_WARPS);
            mbar_init(&s_freed[b], TC_MMA_WARPS);
            mbar_init(&s_full[b], TC_MMA_WARPS);
            mbar_init(&s_empty[b], TC_EPI_WARPS);
        }
        mbar_init(&s_drain, TC_MMA_WARPS);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = s_tmem;
    volatile int* abort = &s_abort;
    // bounded wait by one thread; false when the work is given up
    auto wait = [&](unsigned long long* bar, unsigned par) {
        long long it = 0;
        while (!mbar_try_wait(bar, par)) {
            if ((++it & 15) == 0 && *abort) return false;
            if (it > a.spin_limit) {
                atomicOr(&a.ctrl->status, ST_TIMEOUT);
                *abort = 1;
                return false;
            }
        }
        return true;
    };
    // the same for a warp: one lane polls (polls are shared-memory accesses that the MMAs' operand reads wait for),
    // then every lane sees the phase complete
    auto wait_warp = [&](unsigned long long* bar, unsigned par) {
        int ok = 1;
        if (lane == 0) ok = wait(bar, par);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) mbar_try_wait(bar, par);
        return ok != 0;
    };
    auto unit_at = [&](int tau) {
        const int win = tau / g.high, ty = tau - win * g.high;
        return TcUnit{64 * win - 16, 16 * ty - 16, min(min(TC_TILES, last - tau), g.high - ty)};
    };

    if (warp >= TC_EPI_WARPS + TC_MMA_WARPS) {
        // ---------------- staging ----------------
        const int ft = tid - 32 * (TC_EPI_WARPS + TC_MMA_WARPS);
        const int PW = a.rstride, PH = a.H + 2 * PAD;
        constexpr int kA = (tc_rows(TC_TILES) * TC_CHUNKS + 32 * TC_FILL_WARPS - 1) / (32 * TC_FILL_WARPS);
        constexpr int kB = ((TC_TILES + 3) * 128 + 32 * TC_FILL_WARPS - 1) / (32 * TC_FILL_WARPS);
        int iu = 0;
        for (int tau = first; tau < last; iu++) {
            const TcUnit u = unit_at(tau);
            tau += u.nt;
            unsigned char* sA = tc_raw + (iu & 1) * buffer;
            unsigned char* sB = sA + TC_PHASES * phase;
            const int X0 = u.x0, Y0 = u.y0, na = tc_rows(u.nt) * TC_CHUNKS, nb = (u.nt + 3) * 128;
            // everything is read before the wait for the buffer: one round trip.  What lies outside the padded
            // plane belongs to positions outside every range: any samples do.  Templates: macroblock rows from
            // Y0 - 16, columns from X0 - 16; outside the frame the middle grey, zero as an operand.
            uint2 pa[kA][2];
            uint4 pb[kB];
#pragma unroll
            for (int k = 0; k < kA; k++) {
                const int i = min(ft + k * 32 * TC_FILL_WARPS, na - 1), r = i / TC_CHUNKS, q = i - r * TC_CHUNKS;
                const unsigned char* row = a.refp + (size_t)min(Y0 + r + PAD, PH - 1) * a.rstride;
                const int x = X0 + PAD + 8 * q;
                pa[k][0] = __ldg(reinterpret_cast<const uint2*>(row + min(x, PW - 8)));
                pa[k][1] = __ldg(reinterpret_cast<const uint2*>(row + min(x + 8, PW - 8)));
            }
#pragma unroll
            for (int k = 0; k < kB; k++) {
                const int i = ft + k * 32 * TC_FILL_WARPS, R = i >> 7, y = (i >> 3) & 15, q = i & 7;
                const int n = X0 - 16 + 16 * q, m = Y0 - 16 + 16 * R;
                pb[k] = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
                if (i < nb && n >= 0 && n < a.W && m >= 0 && m < 16 * rows)
                    pb[k] = __ldg(reinterpret_cast<const uint4*>(a.src8 + (size_t)(m + y) * a.W + n));
            }
            if (iu >= 2 && !wait_warp(&s_freed[iu & 1], (unsigned)((iu >> 1) - 1) & 1u)) break;
            // the picture rows from column X0, eight copies a pixel apart
#pragma unroll
            for (int k = 0; k < kA; k++) {
                const int i = ft + k * 32 * TC_FILL_WARPS, r = i / TC_CHUNKS, q = i - r * TC_CHUNKS;
                if (i >= na) break;
                const unsigned w[4] = {pa[k][0].x, pa[k][0].y, pa[k][1].x, pa[k][1].y};
#pragma unroll
                for (int f = 0; f < TC_PHASES; f++) {
                    const int b = f >> 2, s = 8 * (f & 3);
                    *reinterpret_cast<uint4*>(sA + f * phase + r * TC_PITCH + 16 * q) =
                        eight_less128(__funnelshift_r(w[b], w[b + 1], s), __funnelshift_r(w[b + 1], w[b + 2], s));
                }
            }
#pragma unroll
            for (int k = 0; k < kB; k++) {
                const int i = ft + k * 32 * TC_FILL_WARPS, R = i >> 7, y = (i >> 3) & 15, q = i & 7;
                if (i >= nb) break;
                unsigned char* d = sB + R * TC_BROW + y * 256 + q * 16;
                *reinterpret_cast<uint4*>(d) = eight_less128(pb[k].x, pb[k].y);
                *reinterpret_cast<uint4*>(d + 128) = eight_less128(pb[k].z, pb[k].w);
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the MMAs read what was written here
            mbar_arrive(&s_filled[iu & 1]);
        }
    } else if (warp >= TC_EPI_WARPS) {
        // ---------------- MMA issue: one thread of each issuing warp, its phases ----------------
        if (lane == 0) {
            constexpr int kF = TC_PHASES / TC_MMA_WARPS;
            const int f0 = kF * (warp - TC_EPI_WARPS), phase16 = g.phase >> 4;
            const unsigned base = smem_u32(tc_raw);
            bool go = true;
            int iu = 0, ti = 0;
            for (int tau = first; tau < last && go; iu++) {
                const int nt = unit_at(tau).nt;
                tau += nt;
                if (!(go = wait(&s_filled[iu & 1], (unsigned)(iu >> 1) & 1u))) break;
                tc_fence_after();
                const unsigned sa = base + (iu & 1) * buffer, sb = sa + TC_PHASES * phase;
                for (int t = 0; t < nt; t++, ti++) {
                    if (ti >= 2) {
                        if (!(go = wait(&s_empty[ti & 1], (unsigned)((ti >> 1) - 1) & 1u))) break;
                        tc_fence_after();
                    }
                    const unsigned d = tmem + ((ti & 1) * TC_PHASES + f0) * TC_N;
                    const unsigned long long da = tc_desc(sa + f0 * phase + 16 * t * TC_PITCH, 16, TC_PITCH);
                    const unsigned long long db = tc_desc(sb + t * TC_BROW, 128, TC_BROW);
                    // block row y: a picture row, and a row of templates, further; the phases' MMAs alternate, as
                    // those of one accumulator wait for each other
                    for (int y = 0; y < 16; y++)
#pragma unroll
                        for (int f = 0; f < kF; f++)
                            tc_mma(d + f * TC_N, da + f * phase16 + y * (TC_PITCH >> 4), db + y * (256 >> 4), y > 0);
                    tc_commit(&s_full[ti & 1]);
                }
                tc_commit(&s_freed[iu & 1]);
            }
            // every MMA has ended (an abandoned unit's too) before operands and accumulators are given back
            tc_commit(&s_drain);
            long long it = 0;
            while (!mbar_try_wait(&s_drain, 0) && ++it <= a.spin_limit) {}
        }
        __syncwarp();
    } else {
        // ---------------- accumulators to minima ----------------
        const int quarter = warp & 3, R0 = 2 * (warp >> 2);  // lanes of the accumulators, macroblock rows
        const int r = lane & 7, dy = 4 * quarter + (lane >> 3);
        const float kInf = __int_as_float(0x7f800000);
        int ti = 0, x_valid = 0;
        bool go = true;
        unsigned valid[2] = {0u, 0u};  // which phases of each macroblock column are candidates: bit 8 f + q
        for (int tau = first; tau < last && go; tau++, ti++) {
            const TcUnit u = unit_at(tau);
            const int X0 = u.x0, y = u.y0 + dy;
            if (tau == first || X0 != x_valid) {
                x_valid = X0;
                valid[0] = valid[1] = 0u;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const int n = X0 - 16 + 16 * q;
                    int xl, xr, yu, yd;
                    full_range(n, 0, a.W, a.H, a.motion_range, xl, xr, yu, yd);
                    if (n < 0 || n >= a.W) xr = xl - 1;
                    const int j0 = 8 * r + 16 - 16 * q;
#pragma unroll
                    for (int f = 0; f < TC_PHASES; f++)
                        if (j0 + f >= xl && j0 + f <= xr) valid[f >> 2] |= 1u << (8 * (f & 3) + q);
                }
            }
            const float* ep = a.energy + (size_t)min(y + PAD, a.H + 2 * PAD - 16) * a.rstride +
                              min(X0 + 8 * r + PAD, a.rstride - 8);
            const float4 e0 = __ldg(reinterpret_cast<const float4*>(ep));
            const float4 e1 = __ldg(reinterpret_cast<const float4*>(ep) + 1);
            const float e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
            float run[16];
#pragma unroll
            for (int c = 0; c < 16; c++) run[c] = kInf;
            go = wait_warp(&s_full[ti & 1], (unsigned)(ti >> 1) & 1u);
            if (!go) break;
            tc_fence_after();
            const unsigned acc = tmem + (ti & 1) * TC_PHASES * TC_N + 8 * R0 + ((unsigned)(32 * quarter) << 16);
#pragma unroll
            for (int f = 0; f < TC_PHASES; f++) {
                float d[16];
                tc_load16(acc + f * TC_N, d);
                const unsigned ok = valid[f >> 2] >> (8 * (f & 3));
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const bool in = (ok >> q) & 1u;
#pragma unroll
                    for (int R = 0; R < 2; R++) {
                        const float v = __fmaf_rn(-2.0f, d[8 * R + q], e[f]);
                        run[8 * R + q] = in ? fminf(run[8 * R + q], v) : run[8 * R + q];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[ti & 1]);
            // this lane's 8 columns are the group r + 6 - 2q of macroblock column q
            const int mc0 = (X0 >> 4) - 1;
#pragma unroll
            for (int R = 0; R < 2; R++) {
                const int mr = (u.y0 >> 4) - 1 + R0 + R, i = y - 16 * mr;
                if (mr < 0 || mr >= rows || i < -RMAX || i > RMAX) continue;
                float* dst = a.rowmin + ((ptrdiff_t)(mr * a.cols + mc0) * 64 + i + RMAX) * 8 + r + 6;
#pragma unroll
                for (int q = 0; q < 8; q++)
                    if ((unsigned)(r + 6 - 2 * q) < 8u && (unsigned)(mc0 + q) < (unsigned)a.cols)
                        __stcg(dst + q * (64 * 8 - 2), run[8 * R + q]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == TC_EPI_WARPS) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TC_TMEM) : "memory");
    }
}

}  // namespace

int rowmin_prepare()
{
    VPP_CUDA(cudaFuncSetAttribute(k_ssd_rowmin, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  2 * tc_buffer(TC_TILES)));
    return VPPGPU_OK;
}

int rowmin_launch(vppgpu_ctx* ctx, const FullArgs& args)
{
    // positions -16 .. W and -16 .. H
    TcGrid g;
    g.high = (args.H + 17 + 15) / 16;
    const int tiles = (args.W + 17 + 63) / 64 * g.high, grid = tiles < ctx->sm_count ? tiles : ctx->sm_count;
    g.phase = tc_rows(TC_TILES) * TC_PITCH;
    g.run = tiles / grid;
    g.more = tiles % grid;
    k_ssd_rowmin<<<grid, TC_THREADS, 2 * tc_buffer(TC_TILES), ctx->stream>>>(args, g);
    VPP_CHECK_LAUNCH(ctx);
    return VPPGPU_OK;
}

}  // namespace vppgpu
