// int16 convs, Gemms and products of small and middling tensors with the warp-level matrix instruction (mma.sync m16n8k32) on byte planes.
//
// Replaces dl::base::conv2d<int16_t,...> (esp-dl/dl/base/dl_base_conv2d.cpp) where the tensor-core tile kernel's two launches - its operands
// unrolled and split into byte planes in memory first - are most of the time: 4 x 40x40x64 -> 64, 3x3 took 12.3 us, 8 of them
// the packing and its launch.  Here the planes never reach memory: a block copies 64-element runs of its input
// pixels' windows and filter rows to shared memory as they are (asynchronous copies, three runs at a time, zero fill outside the image), a warp splits
// the words of a fragment into high and low bytes by byte permutes, and multiplies: x = 256 xh + xl with xh signed and xl unsigned, so a
// product is 65536 hh + 256 (hl + lh) + ll, four instructions of the matching signedness into three 32-bit accumulators, exact for
// reductions up to 16384 terms, put together in 64 bits.
// The order of the reduction is free as long as both operands agree: lane (g, t) takes the 16 consecutive elements 16t .. 16t + 15 of a run.  A run's 16-byte
// units lie XORed with the row, so a quarter warp's 16-byte reads meet no bank conflict.
// Bound by the latency of copies, fragments and products, one after the other, while there is a block an SM (4 of 40x40: matrix pipe 24 %, issue slots 43 %
// busy), by the matrix instruction (39 %), permutes and addresses (issue slots 53 %) together beyond that (256 of 28x28).  A barrier for three runs of
// the reduction instead of each, the next three on their way (both sides in turn, launches in a chain): 4 of 40x40x64 -> 64, 3x3 9.5 -> 8.1 us, 34 of 70x71x64 -> 24
// 69.9 -> 58.5, 8 of 40x40x64 13.4 -> 11.4, 8 of 10x10x256 -> 256 16.1 -> 14.5, 256 of 28x28x64 136 -> 124; one of 40x40x64 stays at 5.0.  (Two at a time in two / three
// groups took 1.06 / 1.07 times as long.)  Up to five runs are all asked for at the start (112x112x8 -> 16 at stride 2 3.0 -> 2.8; 80x80x32 stays at 4.8).
// The form of 64 x 64 spills 32 bytes, 64 x 32 4.
// us packed and here: 4 of 40x40x64 -> 64 12.3 / 8.1, one of them 12.4 / 5.0, 112x112x8 -> 16 at stride 2 12.3 / 2.8, 128x512x512 10.1 / 4.4.
#include "common.cuh"

#include <climits>
#include <mutex>

namespace espdl {

namespace {

constexpr int M16_RUN = 64; // elements of the reduction a stage

struct Mma16Params {
    const int16_t *in, *w;
    const long long *bias;
    const int32_t *ew;
    int16_t *out;
    int M, N, K, runs, tiles_n;
    int ic, ih, iw, oh, ow, kw, sh, sw, dh, dw, pt, pl, ips, ops;
    int e_shift_base, ew_scalar, per_channel, relu, half_even;
    int early; // the filter is a constant of the model: copied before the wait for the previous kernel
};

template <bool A_SIGNED, bool B_SIGNED>
__device__ __forceinline__ void mma_bytes(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
#define ESPDL_MMA(A, B)                                                                                                              \
    asm("mma.sync.aligned.m16n8k32.row.col.s32." A "." B ".s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};" \
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])                                                                             \
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1))
    if (A_SIGNED && B_SIGNED)
        ESPDL_MMA("s8", "s8");
    else if (A_SIGNED)
        ESPDL_MMA("s8", "u8");
    else if (B_SIGNED)
        ESPDL_MMA("u8", "s8");
    else
        ESPDL_MMA("u8", "u8");
#undef ESPDL_MMA
}

// 16 elements as 16 high and 16 low bytes.
struct Planes {
    uint4 hi, lo;
};
__device__ __forceinline__ Planes split_planes(uint32_t run, int row, int t)
{
    uint4 a, b;
    const uint32_t line = run + (uint32_t)row * 2u * M16_RUN, swz = (uint32_t)(row & 7);
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w) : "r"(line + 16u * ((2u * t) ^ swz)) : "memory");
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(line + 16u * ((2u * t + 1u) ^ swz)) : "memory");
    Planes p;
    p.hi = make_uint4(__byte_perm(a.x, a.y, 0x7531), __byte_perm(a.z, a.w, 0x7531), __byte_perm(b.x, b.y, 0x7531), __byte_perm(b.z, b.w, 0x7531));
    p.lo = make_uint4(__byte_perm(a.x, a.y, 0x6420), __byte_perm(a.z, a.w, 0x6420), __byte_perm(b.x, b.y, 0x6420), __byte_perm(b.z, b.w, 0x6420));
    return p;
}

// BM pixels x BN channels a block of eight warps, WM of them along the pixels (16 each), NT instructions' columns a warp.  PAR runs are waited for, met and
// multiplied together; GROUPS = 2: the next ones are on their way meanwhile, 1: they are all there are, all asked for at the start.
template <int WM, int NT, int PAR, int GROUPS>
__global__ void __launch_bounds__(256) conv_mma16_kernel(const __grid_constant__ Mma16Params p)
{
    constexpr int WN = 8 / WM, BM = 16 * WM, BN = 8 * NT * WN, ROWS = BM + BN, PER = (ROWS + 31) / 32; // rows of a stage, copied 32 at a time
    constexpr int STAGES = PAR * GROUPS, AHEAD = GROUPS == 1 ? PAR : STAGES - PAR;
    extern __shared__ __align__(128) uint8_t stage_mem[];
    grid_dep_launch(); // nothing is set up that the next kernel's blocks could disturb
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(stage_mem);
    const int tm = blockIdx.x / p.tiles_n, tn = blockIdx.x - tm * p.tiles_n;
    const int unit = threadIdx.x & 7, row0 = threadIdx.x >> 3; // the 16-byte unit of a run and the rows this thread copies

    // rows [0, BM) are pixels, [BM, ROWS) filter rows; a pixel's pointer is where its window's first tap would be
    const int16_t *from[PER];
    int iy0[PER], ix0[PER];
    bool real[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const int r = row0 + 32 * j;
        iy0[j] = ix0[j] = 0;
        if (r < BM) {
            const int m = tm * BM + r;
            real[j] = m < p.M;
            const int pix = real[j] ? m : 0, line = pix / p.ow, image = line / p.oh;
            iy0[j] = (line - image * p.oh) * p.sh - p.pt, ix0[j] = (pix - line * p.ow) * p.sw - p.pl;
            from[j] = p.in + ((long long)image * p.ih * p.iw + (long long)iy0[j] * p.iw + ix0[j]) * p.ips;
        } else {
            const int n = tn * BN + r - BM;
            real[j] = n < p.N && r < ROWS;
            from[j] = p.w + (long long)(real[j] ? n : 0) * p.K;
        }
    }
    int k = 8 * unit, c = k, dy = 0, dx = 0; // of this thread's unit in the next run to copy: its element of the reduction, channel and tap (in pixels)
    auto wrap = [&] {
        while (c >= p.ic) {
            c -= p.ic, dx += p.dw;
            if (dx == p.kw * p.dw)
                dx = 0, dy += p.dh;
        }
    };
    wrap();
    auto copy_to = [&](uint32_t to, int j, bool ok, const int16_t *at) {
        const int r = row0 + 32 * j;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + (uint32_t)r * 2u * M16_RUN + 16u * (uint32_t)(unit ^ (r & 7))), "l"(ok ? at : p.w), "r"(ok ? 16 : 0) : "memory");
    };
    auto stage_of = [&](int run) { return base + (uint32_t)(run % STAGES) * (ROWS * 2 * M16_RUN); };
    auto copy_filter = [&](int run) {
        const int at = run * M16_RUN + 8 * unit;
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (row0 + 32 * j >= BM && row0 + 32 * j < ROWS)
                copy_to(stage_of(run), j, real[j] && at < p.K, from[j] + at);
    };
    auto copy_pixels = [&](int run) {
        const long long tap = ((long long)dy * p.iw + dx) * p.ips + c;
#pragma unroll
        for (int j = 0; j < PER; j++)
            if (row0 + 32 * j < BM)
                copy_to(stage_of(run), j, real[j] && k < p.K && (unsigned)(iy0[j] + dy) < (unsigned)p.ih && (unsigned)(ix0[j] + dx) < (unsigned)p.iw, from[j] + tap);
        k += M16_RUN, c += M16_RUN;
        wrap();
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    if (p.early)
        for (int s = 0; s < min(AHEAD, p.runs); s++) copy_filter(s);
    grid_dep_wait();
    for (int s = 0; s < AHEAD; s++) { // runs beyond the reduction are zeros
        if (s < p.runs) {
            copy_pixels(s);
            if (!p.early)
                copy_filter(s);
        }
        if ((s + 1) % PAR == 0)
            commit();
    }

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, wm = warp % WM, wn = warp / WM;
    int hh[NT][4], mid[NT][4], ll[NT][4];
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) hh[j][i] = mid[j][i] = ll[j][i] = 0;
    for (int run0 = 0; run0 < p.runs; run0 += PAR) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GROUPS == 1 ? 0 : GROUPS - 2) : "memory");
        __syncthreads(); // these runs are there for all, and the stages of the runs before are read by all
        if (GROUPS > 1) { // on their way behind the products
#pragma unroll
            for (int u = 0; u < PAR; u++)
                if (run0 + AHEAD + u < p.runs) {
                    copy_pixels(run0 + AHEAD + u);
                    copy_filter(run0 + AHEAD + u);
                }
            commit();
        }
#pragma unroll
        for (int u = 0; u < PAR; u++) {
            if (run0 + u >= p.runs)
                break;
            const uint32_t at = stage_of(run0 + u);
            const Planes a0 = split_planes(at, 16 * wm + g, t), a1 = split_planes(at, 16 * wm + 8 + g, t);
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const Planes b = split_planes(at, BM + 8 * (NT * wn + j) + g, t);
                mma_bytes<true, true>(hh[j], a0.hi.x, a1.hi.x, a0.hi.y, a1.hi.y, b.hi.x, b.hi.y);
                mma_bytes<true, false>(mid[j], a0.hi.x, a1.hi.x, a0.hi.y, a1.hi.y, b.lo.x, b.lo.y);
                mma_bytes<false, false>(ll[j], a0.lo.x, a1.lo.x, a0.lo.y, a1.lo.y, b.lo.x, b.lo.y);
                mma_bytes<false, true>(mid[j], a0.lo.x, a1.lo.x, a0.lo.y, a1.lo.y, b.hi.x, b.hi.y);
                mma_bytes<true, true>(hh[j], a0.hi.z, a1.hi.z, a0.hi.w, a1.hi.w, b.hi.z, b.hi.w);
                mma_bytes<true, false>(mid[j], a0.hi.z, a1.hi.z, a0.hi.w, a1.hi.w, b.lo.z, b.lo.w);
                mma_bytes<false, false>(ll[j], a0.lo.z, a1.lo.z, a0.lo.w, a1.lo.w, b.lo.z, b.lo.w);
                mma_bytes<false, true>(mid[j], a0.lo.z, a1.lo.z, a0.lo.w, a1.lo.w, b.hi.z, b.hi.w);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    const bool words = (p.ops & 1) == 0 && ((uintptr_t)p.out & 3) == 0;
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int n = tn * BN + 8 * (NT * wn + j) + 2 * t;
        if (n >= p.N)
            continue;
        const bool two = n + 1 < p.N;
        int shift[2];
        long long bias[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int c = min(n + i, p.N - 1);
            shift[i] = max(-62, min(62, p.e_shift_base - (p.per_channel ? __ldg(p.ew + c) : p.ew_scalar)));
            bias[i] = p.bias ? __ldg(p.bias + c) : 0ll;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = tm * BM + 16 * wm + 8 * h + g;
            if (m >= p.M)
                continue;
            int q[2];
#pragma unroll
            for (int i = 0; i < 2; i++)
                q[i] = requant16((long long)hh[j][2 * h + i] * 65536 + (long long)mid[j][2 * h + i] * 256 + (long long)ll[j][2 * h + i], bias[i], shift[i], p.relu, p.half_even);
            int16_t *op = p.out + (long long)m * p.ops + n;
            if (words && two) {
                *(uint32_t *)op = ((uint32_t)q[0] & 0xffffu) | ((uint32_t)q[1] << 16);
            } else {
                op[0] = (int16_t)q[0];
                if (two)
                    op[1] = (int16_t)q[1];
            }
        }
    }
}

struct Mma16Plan {
    int bm, bn;
    float us;
};

// The tile by waves of as many blocks as an SM holds, each its start, its results, and its runs, which take their share of the matrix instructions or the
// latency of copies and fragments (4 of 40x40x64 -> 64, 3x3: 13.2 us with 64 x 64, 10.2 with 64 x 32, 12.0 with 32 x 32; 400x1152x128 14.5, 10.6, 7.9;
// 102400x576x64 70, 88, 112).  The choice against the other kernels looks at what 4500 layers took in the tile that they get, inputs in L2: a launch, a window's
// addresses, and the blocks of the SM that has most of them, as many at a time as fit, each its results and its runs beside others or their latency alone; of many
// blocks an SM's share and a part of the last wave.  Blocks of 32 x 32 that are one for nearly every SM take longer in a chain than fewer or more, as the next launch's begin
// beside them, several on each SM that has none (25 of 13x13x256 -> 16, 3x3 31 us in a chain, about 12 alone); inputs beyond L2 cost them.  Within 7 to 13 %
// (standard deviation) of 2700 other layers.
Mma16Plan mma16_plan(const espdl_conv_desc &d)
{
    static const struct {
        int bm, bn, resident;
        float start, block, run, latency; // us, of the choice
        float launch, window, results, beside, alone, every, rest, beyond;
    } shapes[3] = {{64, 64, 2, 1.3f, 1.8f, 0.42f, 0.85f, 2.4f, 0.57f, 1.83f, 0.427f, 0.5f, 0.5f, 0.25f, 0.0f},
                   {64, 32, 3, 1.3f, 1.2f, 0.263f, 0.5f, 1.35f, 0.83f, 0.84f, 0.256f, 0.74f, 0.74f, 0.28f, 0.0f},
                   {32, 32, 4, 1.0f, 1.0f, 0.2f, 0.22f, 0.0f, 0.31f, 1.77f, 0.267f, 0.267f, 0.49f, 0.13f, 2.4e-7f}};
    const float M = (float)d.n * d.out_h * d.out_w, runs = ceilf((float)d.kh * d.kw * d.in_c / M16_RUN);
    const float beyond = fmaxf(0.0f, M * d.kh * d.kw * d.in_c - 2.5e7f);
    const bool window = d.kh * d.kw > 1 || d.in_c % 16;
    Mma16Plan best = {0, 0, 1e30f};
    float least = 1e30f;
    for (const auto &s : shapes) {
        const float share = ceilf(M / s.bm) * ceilf((float)d.out_c / s.bn) / num_sms(), most = ceilf(share), side = fminf((float)s.resident, most);
        const float us = 2.0f + fmaxf(1.0f, share / s.resident) * (s.start + s.block * side + runs * fmaxf(s.latency, side * s.run));
        if (us < least) {
            const float alone = share > 0.8f && share <= 1.0f ? s.every : s.alone;
            const auto wave = [&](float blocks) { return s.results * blocks + runs * fmaxf(alone, blocks * s.beside); };
            const float full = floorf(most / s.resident), last = most - full * s.resident;
            least = us;
            best = {s.bm, s.bn, s.launch + (window ? s.window : 0.0f) + beyond * s.beyond + (share > 2 * s.resident ? (share / s.resident + s.rest) * wave((float)s.resident)
                                                                                              : full * wave((float)s.resident) + (last > 0 ? wave(last) : 0.0f))};
        }
    }
    return best;
}

template <int WM, int NT, int PAR, int GROUPS>
int launch_mma16_as(Mma16Params &p, cudaStream_t s)
{
    constexpr int BM = 16 * WM, BN = 8 * NT * (8 / WM), stage = (BM + BN) * 2 * M16_RUN;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] { attr_err = cudaFuncSetAttribute(conv_mma16_kernel<WM, NT, PAR, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, PAR * GROUPS * stage); });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(conv_mma16_kernel)");
    p.tiles_n = (p.N + BN - 1) / BN;
    launch_overlapped(conv_mma16_kernel<WM, NT, PAR, GROUPS>, dim3((unsigned)(p.tiles_n * ((p.M + BM - 1) / BM))), dim3(256), min(p.runs, PAR * GROUPS) * stage, s, p);
    count_launch();
    return check_launch("conv_mma16");
}

template <int WM, int NT>
int launch_mma16(Mma16Params &p, cudaStream_t s)
{
    return p.runs <= 5 ? launch_mma16_as<WM, NT, 5, 1>(p, s) : launch_mma16_as<WM, NT, 3, 2>(p, s);
}

} // namespace

bool conv2d_mma16_supported(const espdl_conv_desc &d)
{
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    if (d.dtype != ESPDL_DTYPE_INT16 || d.group != 1 || d.filter_image_stride != 0 || d.lut || d.residual)
        return false;
    if (d.in_c % 8 || ips % 8 || ((uintptr_t)d.input % 16) || ((uintptr_t)d.filter % 16))
        return false;
    const long long M = (long long)d.n * d.out_h * d.out_w, K = (long long)d.kh * d.kw * d.in_c;
    return M <= (1 << 24) && d.out_c <= (1 << 20) && K <= 16384 && (M + 31) / 32 * ((d.out_c + 31) / 32) <= (1 << 24);
}

float conv2d_mma16_estimate_us(const espdl_conv_desc &d) { return mma16_plan(d).us; }

int conv2d_mma16(const espdl_conv_desc &d, cudaStream_t s)
{
    const Mma16Plan plan = mma16_plan(d);
    Mma16Params p;
    p.in = (const int16_t *)d.input, p.w = (const int16_t *)d.filter, p.bias = (const long long *)d.bias, p.ew = d.filter_exponents, p.out = (int16_t *)d.output;
    p.M = d.n * d.out_h * d.out_w, p.N = d.out_c, p.K = d.kh * d.kw * d.in_c, p.runs = (p.K + M16_RUN - 1) / M16_RUN;
    p.ic = d.in_c, p.ih = d.in_h, p.iw = d.in_w, p.oh = d.out_h, p.ow = d.out_w, p.kw = d.kw;
    p.sh = d.stride_h, p.sw = d.stride_w, p.dh = d.dilation_h, p.dw = d.dilation_w, p.pt = d.pad_top, p.pl = d.pad_left;
    p.ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.e_shift_base = d.out_exponent - d.in_exponent, p.ew_scalar = d.filter_exponent, p.per_channel = d.per_channel;
    p.relu = d.activation == ESPDL_ACT_RELU, p.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.early = in_model_scope();
    if (plan.bm == 32)
        return launch_mma16<2, 1>(p, s);
    return plan.bn == 32 ? launch_mma16<4, 2>(p, s) : launch_mma16<4, 4>(p, s);
}

} // namespace espdl
