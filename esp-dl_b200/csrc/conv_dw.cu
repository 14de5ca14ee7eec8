// DepthwiseConv2D (group == channels), int8 and int16.
// Replaces dl::base::depthwise_conv2d<> (esp-dl/dl/base/dl_base_depthwise_conv2d.cpp:47-66,
// shell esp-dl/dl/base/dl_base.hpp:1209-2107): out[y,x,c] = epilogue(sum_{ky,kx} in[..,c] * w[ky,kx,c] + bias[c]).
//
// The op is bandwidth bound by design (9 MACs per byte read).  3x3 filters with stride 1 or 2 - the shapes of
// MobileNet-style networks - run on dw3x3_dp4a_kernel (a thread walks along a band of rows, dp4a over byte-transposed
// columns), other windows of 3x3, 5x5 and 7x7 on dwk_dp4a_kernel; other int8 shapes with C % 16 == 0 on dw_s8_vec16_kernel (16 channels per thread, 128-bit loads and
// stores, a warp reads and writes contiguous runs of the NHWC tensor), int16 3x3 and 5x5 on dw_run_s16_kernel, small ones
// and other int16 on dw_taps_kernel; everything else on dw_generic_kernel.
#include "common.cuh"

namespace espdl {

struct DwParams {
    int early; // filter, bias and exponents are constants of a model: read ahead of the previous kernel's end
    const void *in, *w, *bias;
    void *out;
    const int32_t *ew;
    const int8_t *lut;
    int lut_stride; // 0: one table, else entries between the tables of consecutive channels
    int n, ih, iw, c, oh, ow, kh, kw, sh, sw, dh, dw, pt, pl, ips, ops;
    int e_shift_base, ew_scalar, per_channel, relu, half_even;
    long long total;
    int chunks;
};

__device__ __forceinline__ int sbyte(uint32_t x, int i) { return (int)(int8_t)(x >> (8 * i)); }

__global__ void __launch_bounds__(256) dw_s8_vec16_kernel(DwParams p)
{
    grid_dep_launch();
    grid_dep_wait();
    const int8_t *__restrict__ in = (const int8_t *)p.in;
    const int8_t *__restrict__ w = (const int8_t *)p.w;
    const int32_t *__restrict__ bias = (const int32_t *)p.bias;
    int8_t *__restrict__ out = (int8_t *)p.out;
    for (long long item = blockIdx.x * (long long)blockDim.x + threadIdx.x; item < p.total;
         item += (long long)gridDim.x * blockDim.x) {
        long long ch_rem;
        const long long pix = div_rem(item, p.chunks, ch_rem);
        const int ch = (int)ch_rem * 16;
        int ox, oy, n;
        split_pixel(pix, p.ow, p.oh, ox, oy, n);
        int32_t acc[16];
#pragma unroll
        for (int j = 0; j < 16; j++) acc[j] = 0;
        for (int ky = 0; ky < p.kh; ky++) {
            const int iy = oy * p.sh + ky * p.dh - p.pt;
            if (iy < 0 || iy >= p.ih)
                continue;
            for (int kx = 0; kx < p.kw; kx++) {
                const int ix = ox * p.sw + kx * p.dw - p.pl;
                if (ix < 0 || ix >= p.iw)
                    continue;
                const uint4 a = __ldg((const uint4 *)(in + (((long long)n * p.ih + iy) * p.iw + ix) * p.ips + ch));
                const uint4 b = __ldg((const uint4 *)(w + ((long long)ky * p.kw + kx) * p.c + ch));
                const uint32_t av[4] = {a.x, a.y, a.z, a.w};
                const uint32_t bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int q = 0; q < 4; q++)
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[q * 4 + i] += sbyte(av[q], i) * sbyte(bv[q], i);
            }
        }
        uint32_t packed[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            uint32_t wd = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int c = ch + q * 4 + i;
                const int e = p.per_channel ? __ldg(p.ew + c) : p.ew_scalar;
                const int shift = max(-31, min(32, p.e_shift_base - e));
                int32_t v = requant8(acc[q * 4 + i], bias ? __ldg(bias + c) : 0, shift, p.relu, p.half_even);
                if (p.lut)
                    v = p.lut[(long long)c * p.lut_stride + ((uint8_t)v ^ 0x80u)];
                wd |= ((uint32_t)v & 0xffu) << (8 * i);
            }
            packed[q] = wd;
        }
        *(uint4 *)(out + pix * p.ops + ch) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
}

// K x K depthwise (5x5, 7x7), int8, any stride, dilation 1: a thread owns four consecutive channels of one output pixel.  All K*K words of its
// window are loaded before the first is used - small maps are bound by that latency -, groups of four taps are byte-transposed
// into one word per channel and meet the transposed filter, which the block keeps in shared memory, in one dp4a each: about three
// instructions a tap for four channels where the kernel above takes ten.  5x5 over 64 channels: 184x184 19.0 -> 12.9 us, 23x23 11.4 -> 2.4.
template <int K>
__global__ void __launch_bounds__(256) dwk_dp4a_kernel(DwParams p)
{
    constexpr int TAPS = K * K, GROUPS = (TAPS + 3) / 4;
    extern __shared__ uint32_t dwk_w[]; // [group][channel of the word][word]
    grid_dep_launch();
    if (!p.early)
        grid_dep_wait();
    const int words = p.c / 4;
    for (int i = threadIdx.x; i < GROUPS * words; i += 256) {
        const int g = i / words, c4 = i - g * words;
        uint32_t t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) t[j] = 4 * g + j < TAPS ? __ldg((const uint32_t *)((const int8_t *)p.w + (long long)(4 * g + j) * p.c) + c4) : 0u;
        const uint32_t lo0 = __byte_perm(t[0], t[1], 0x5140), lo1 = __byte_perm(t[2], t[3], 0x5140), hi0 = __byte_perm(t[0], t[1], 0x7362), hi1 = __byte_perm(t[2], t[3], 0x7362);
        dwk_w[(g * 4 + 0) * words + c4] = __byte_perm(lo0, lo1, 0x5410);
        dwk_w[(g * 4 + 1) * words + c4] = __byte_perm(lo0, lo1, 0x7632);
        dwk_w[(g * 4 + 2) * words + c4] = __byte_perm(hi0, hi1, 0x5410);
        dwk_w[(g * 4 + 3) * words + c4] = __byte_perm(hi0, hi1, 0x7632);
    }
    if (p.early)
        grid_dep_wait();
    __syncthreads();
    const unsigned total = (unsigned)(p.total); // words of the output, below 2^31
    for (unsigned item = blockIdx.x * 256u + threadIdx.x; item < total; item += gridDim.x * 256u) {
        const unsigned pix = item / (unsigned)words, c4 = item - pix * (unsigned)words, line = pix / (unsigned)p.ow, n = line / (unsigned)p.oh;
        const int ox = (int)(pix - line * (unsigned)p.ow), oy = (int)(line - n * (unsigned)p.oh);
        const int iy0 = oy * p.sh - p.pt, ix0 = ox * p.sw - p.pl;
        const int8_t *at = (const int8_t *)p.in + (((long long)n * p.ih + iy0) * p.iw + ix0) * p.ips + 4 * c4;
        uint32_t raw[GROUPS * 4];
        if (iy0 >= 0 && ix0 >= 0 && iy0 + K <= p.ih && ix0 + K <= p.iw) {
#pragma unroll
            for (int ky = 0; ky < K; ky++)
#pragma unroll
                for (int kx = 0; kx < K; kx++) raw[ky * K + kx] = __ldg((const uint32_t *)(at + ((long long)ky * p.iw + kx) * p.ips));
        } else {
#pragma unroll
            for (int ky = 0; ky < K; ky++)
#pragma unroll
                for (int kx = 0; kx < K; kx++) {
                    raw[ky * K + kx] = 0u;
                    if ((unsigned)(iy0 + ky) < (unsigned)p.ih && (unsigned)(ix0 + kx) < (unsigned)p.iw)
                        raw[ky * K + kx] = __ldg((const uint32_t *)(at + ((long long)ky * p.iw + kx) * p.ips));
                }
        }
#pragma unroll
        for (int t = TAPS; t < GROUPS * 4; t++) raw[t] = 0u;
        int acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int g = 0; g < GROUPS; g++) {
            const uint32_t lo0 = __byte_perm(raw[4 * g], raw[4 * g + 1], 0x5140), lo1 = __byte_perm(raw[4 * g + 2], raw[4 * g + 3], 0x5140);
            const uint32_t hi0 = __byte_perm(raw[4 * g], raw[4 * g + 1], 0x7362), hi1 = __byte_perm(raw[4 * g + 2], raw[4 * g + 3], 0x7362);
            const uint32_t *f = dwk_w + g * 4 * words + c4;
            acc[0] = __dp4a((int)__byte_perm(lo0, lo1, 0x5410), (int)f[0], acc[0]);
            acc[1] = __dp4a((int)__byte_perm(lo0, lo1, 0x7632), (int)f[words], acc[1]);
            acc[2] = __dp4a((int)__byte_perm(hi0, hi1, 0x5410), (int)f[2 * words], acc[2]);
            acc[3] = __dp4a((int)__byte_perm(hi0, hi1, 0x7632), (int)f[3 * words], acc[3]);
        }
        uint32_t wd = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int c = (int)c4 * 4 + i;
            const int e = p.per_channel ? __ldg(p.ew + c) : p.ew_scalar;
            const int shift = max(-31, min(32, p.e_shift_base - e));
            int32_t v = requant8(acc[i], p.bias ? __ldg((const int32_t *)p.bias + c) : 0, shift, p.relu, p.half_even);
            if (p.lut)
                v = p.lut[(long long)c * p.lut_stride + ((uint8_t)v ^ 0x80u)];
            wd |= ((uint32_t)v & 0xffu) << (8 * i);
        }
        *(uint32_t *)((int8_t *)p.out + (long long)pix * p.ops + 4 * c4) = wd;
    }
}

// 3x3 depthwise on dp4a, int8, dilation 1, stride S (1 or 2).
// dp4a sums four byte products, but a depthwise filter never sums across channels: the four bytes of a dp4a
// operand have to be four TAPS of one channel.  A thread owns four consecutive channels (one 32-bit word of an
// NHWC pixel) and a band of output rows, and walks along the row.  Each input column it meets (the band's input
// rows at one x) is byte-transposed once, eight PRMTs per four rows: word i of a group holds channel i of four
// vertically adjacent pixels.  Against the filter column (w[0][kx], w[1][kx], w[2][kx], 0) that word gives the
// output row whose window starts at the group's first row, against the same word shifted by one byte the next
// row (stride 1, two overlapping groups per band -> four output rows from six input rows).  With stride 2 the
// second output row of a band takes two taps from the group ((0,0,w0,w1)) and its third from a fifth input row,
// read untransposed with the tap placed in the byte of its channel.  Three transposed columns are live; per
// output that is 3 (S=1) or 4.5 (S=2) dp4a, about one PRMT, a shift, a max and half a pack.
// Rows outside the image walk along a row of zeros instead (g_dw_zero_row), so the walk has no per-load bounds
// checks and one step size; columns outside the image are skipped as a whole.  Three columns are always in flight
// (stride 1): with 16 warps per SM it is the bytes in flight, not the arithmetic, that set the speed.
constexpr int DW_ZERO_ROW_BYTES = 128 * 1024;
__device__ uint32_t g_dw_zero_row[DW_ZERO_ROW_BYTES / 4]; // never written: what rows outside the image read

template <int S>
struct DwCol {
    uint32_t t[S == 1 ? 2 : 1][4]; // [row group][channel]: four vertically adjacent pixels of that channel
    uint32_t extra;                // stride 2: the fifth input row, untransposed
};

template <int S>
__device__ __forceinline__ void dw_transpose_col(DwCol<S> &col, const uint32_t (&raw)[S == 1 ? 6 : 5])
{
    constexpr int PAIRS = S == 1 ? 3 : 2;
    uint32_t lo[PAIRS], hi[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; j++) {
        lo[j] = __byte_perm(raw[2 * j], raw[2 * j + 1], 0x5140); // channels 0,1 of the row pair, interleaved
        hi[j] = __byte_perm(raw[2 * j], raw[2 * j + 1], 0x7362); // channels 2,3
    }
#pragma unroll
    for (int g = 0; g < (S == 1 ? 2 : 1); g++) {
        col.t[g][0] = __byte_perm(lo[g], lo[g + 1], 0x5410);
        col.t[g][1] = __byte_perm(lo[g], lo[g + 1], 0x7632);
        col.t[g][2] = __byte_perm(hi[g], hi[g + 1], 0x5410);
        col.t[g][3] = __byte_perm(hi[g], hi[g + 1], 0x7632);
    }
    col.extra = S == 2 ? raw[S == 2 ? 4 : 0] : 0u;
}

// Band of a thread whose channels do not qualify for the one-add-one-shift epilogue (a shift below 1, a
// huge bias, half-even rounding or a fused table): plain loops with the general requantisation.  Kept out of line
// so that the walk below carries none of its registers.
__device__ __noinline__ void dw3x3_band_general(const DwParams &p, int S, int n, int c0, int oy0, int rows, int x_begin, int x_end)
{
    const int8_t *__restrict__ in = (const int8_t *)p.in + (long long)n * p.ih * p.iw * p.ips;
    int8_t *__restrict__ out = (int8_t *)p.out + (long long)n * p.oh * p.ow * p.ops;
    for (int oy = oy0; oy < min(p.oh, oy0 + rows); oy++)
        for (int ox = x_begin; ox < x_end; ox++)
            for (int i = 0; i < 4; i++) {
                const int c = c0 + i;
                int32_t acc = 0;
                for (int ky = 0; ky < 3; ky++)
                    for (int kx = 0; kx < 3; kx++) {
                        const int iy = oy * S - p.pt + ky, ix = ox * S - p.pl + kx;
                        if (iy >= 0 && iy < p.ih && ix >= 0 && ix < p.iw)
                            acc += (int)in[((long long)iy * p.iw + ix) * p.ips + c] * (int)((const int8_t *)p.w)[(ky * 3 + kx) * p.c + c];
                    }
                const int e = p.per_channel ? p.ew[c] : p.ew_scalar;
                const int shift = max(-31, min(32, p.e_shift_base - e));
                int32_t v = requant8(acc, p.bias ? ((const int32_t *)p.bias)[c] : 0, shift, p.relu, p.half_even);
                if (p.lut)
                    v = p.lut[(long long)c * p.lut_stride + ((uint8_t)v ^ 0x80u)];
                out[((long long)oy * p.ow + ox) * p.ops + c] = (int8_t)v;
            }
}

template <int S, bool EVEN>
__global__ void __launch_bounds__(128, 4) dw3x3_dp4a_kernel(DwParams p, int xsegs, int ytiles, int cols_per_thread)
{
    grid_dep_launch();
    if (!p.early)
        grid_dep_wait();
    constexpr int ROWS_IN = S == 1 ? 6 : 5;
    constexpr int ROWS_OUT = S == 1 ? 4 : 2;
    const int quads = p.c >> 2;
    const long long item = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (item >= p.total)
        return;
    const int cq = (int)(item % quads);
    long long r = item / quads;
    const int yt = (int)(r % ytiles);
    r /= ytiles;
    const int xs = (int)(r % xsegs);
    const int n = (int)(r / xsegs);
    const int c0 = cq * 4;

    // filter columns as dp4a operands: wv[kx][i] = (w[0][kx][i], w[1][kx][i], w[2][kx][i], 0)
    uint32_t wv[3][4], wv1[3][4], wsel[3][4];
#pragma unroll
    for (int kx = 0; kx < 3; kx++) {
        uint32_t f[3];
#pragma unroll
        for (int ky = 0; ky < 3; ky++) f[ky] = __ldg((const uint32_t *)((const int8_t *)p.w + (long long)(ky * 3 + kx) * p.c + c0));
        const uint32_t lo0 = __byte_perm(f[0], f[1], 0x5140), hi0 = __byte_perm(f[0], f[1], 0x7362);
        const uint32_t lo1 = __byte_perm(f[2], 0u, 0x5140), hi1 = __byte_perm(f[2], 0u, 0x7362);
        wv[kx][0] = __byte_perm(lo0, lo1, 0x5410);
        wv[kx][1] = __byte_perm(lo0, lo1, 0x7632);
        wv[kx][2] = __byte_perm(hi0, hi1, 0x5410);
        wv[kx][3] = __byte_perm(hi0, hi1, 0x7632);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            wv1[kx][i] = wv[kx][i] << (S == 1 ? 8 : 16);                           // the band's next output row
            wsel[kx][i] = S == 2 ? (f[2] & (0xffu << (8 * i))) : 0u;               // w[2][kx][i] in byte i
        }
    }
    int bias[4], shift[4];
    bool fast = !p.lut;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        bias[i] = p.bias ? __ldg((const int32_t *)p.bias + c0 + i) : 0;
        const int e = p.per_channel ? __ldg(p.ew + c0 + i) : p.ew_scalar;
        int bh, fs;
        fast = fast_constants(bias[i], p.e_shift_base - e, 9 << 14, EVEN, bh, fs) && fast;
        bias[i] = bh, shift[i] = fs;
    }
    const int oy0 = yt * ROWS_OUT;
    const int x_begin = xs * cols_per_thread, x_end = min(p.ow, x_begin + cols_per_thread);
    if (p.early)
        grid_dep_wait();
    if (!fast) {
        dw3x3_band_general(p, S, n, c0, oy0, ROWS_OUT, x_begin, x_end);
        return;
    }
    const int(&init)[4] = bias; // accumulators start from bias plus the rounding half
    const int floor_q = p.relu ? 0 : INT_MIN;
    const int iy0 = oy0 * S - p.pt;
    int ix = x_begin * S - p.pl; // column the row pointers stand on

    // one pointer per input row of the band; rows outside the image walk along the row of zeros
    const int8_t *rp[ROWS_IN];
    {
        const int8_t *img = (const int8_t *)p.in + (long long)n * p.ih * p.iw * p.ips + c0;
#pragma unroll
        for (int rr = 0; rr < ROWS_IN; rr++) {
            const int iy = iy0 + rr;
            const bool ok = iy >= 0 && iy < p.ih;
            rp[rr] = ok ? img + ((long long)iy * p.iw + ix) * p.ips : (const int8_t *)g_dw_zero_row + (long long)(ix + 2) * p.ips;
        }
    }
    int8_t *op = (int8_t *)p.out + (((long long)n * p.oh + oy0) * p.ow + x_begin) * p.ops + c0;
    const int orow = p.ow * p.ops;
    bool ovalid[ROWS_OUT];
#pragma unroll
    for (int ro = 0; ro < ROWS_OUT; ro++) ovalid[ro] = oy0 + ro < p.oh;

    uint32_t raw[ROWS_IN], raw2[ROWS_IN], raw3[ROWS_IN], raw4[ROWS_IN];
    auto load_col = [&](uint32_t (&dst)[ROWS_IN]) {
        const bool ok = ix >= 0 && ix < p.iw;
#pragma unroll
        for (int rr = 0; rr < ROWS_IN; rr++) {
            dst[rr] = ok ? __ldg((const uint32_t *)rp[rr]) : 0u;
            rp[rr] += p.ips;
        }
        ix++;
    };

    auto emit = [&](const DwCol<S> &k0, const DwCol<S> &k1, const DwCol<S> &k2) {
        int acc[ROWS_OUT][4];
#pragma unroll
        for (int kx = 0; kx < 3; kx++) {
            const DwCol<S> &k = kx == 0 ? k0 : (kx == 1 ? k1 : k2);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint32_t w = wv[kx][i], w1 = wv1[kx][i];
                if constexpr (S == 1) {
                    acc[0][i] = __dp4a((int)k.t[0][i], (int)w, kx == 0 ? init[i] : acc[0][i]);
                    acc[1][i] = __dp4a((int)k.t[0][i], (int)w1, kx == 0 ? init[i] : acc[1][i]);
                    acc[2][i] = __dp4a((int)k.t[1][i], (int)w, kx == 0 ? init[i] : acc[2][i]);
                    acc[3][i] = __dp4a((int)k.t[1][i], (int)w1, kx == 0 ? init[i] : acc[3][i]);
                } else {
                    acc[0][i] = __dp4a((int)k.t[0][i], (int)w, kx == 0 ? init[i] : acc[0][i]);
                    acc[1][i] = __dp4a((int)k.t[0][i], (int)w1, kx == 0 ? init[i] : acc[1][i]);
                    acc[1][i] = __dp4a((int)k.extra, (int)wsel[kx][i], acc[1][i]);
                }
            }
        }
#pragma unroll
        for (int ro = 0; ro < ROWS_OUT; ro++) {
            if (EVEN)
#pragma unroll
                for (int i = 0; i < 4; i++) acc[ro][i] += (acc[ro][i] >> shift[i]) & 1;
            const int q0 = max(acc[ro][0] >> shift[0], floor_q), q1 = max(acc[ro][1] >> shift[1], floor_q);
            const int q2 = max(acc[ro][2] >> shift[2], floor_q), q3 = max(acc[ro][3] >> shift[3], floor_q);
            uint32_t hi, wd;
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q3), "r"(q2));
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(wd) : "r"(q1), "r"(q0), "r"(hi));
            if (ovalid[ro])
                *(uint32_t *)(op + (long long)ro * orow) = wd;
        }
        op += p.ops;
    };

    DwCol<S> ca, cb, cc;
    if constexpr (S == 1) {
        // output x reads input columns x - pl + {0,1,2}: two columns prime the window, every step brings one in,
        // requested one step before it is needed
        load_col(raw);
        dw_transpose_col<S>(ca, raw);
        load_col(raw);
        dw_transpose_col<S>(cb, raw);
        load_col(raw);
        load_col(raw2);
        load_col(raw3);
        // three column registers and three load buffers rotate together: the pattern repeats every three outputs
        for (int x = x_begin; x < x_end; x += 3) {
            dw_transpose_col<S>(cc, raw);
            load_col(raw);
            emit(ca, cb, cc);
            if (x + 1 >= x_end)
                break;
            dw_transpose_col<S>(ca, raw2);
            load_col(raw2);
            emit(cb, cc, ca);
            if (x + 2 >= x_end)
                break;
            dw_transpose_col<S>(cb, raw3);
            load_col(raw3);
            emit(cc, ca, cb);
        }
    } else {
        // output x reads input columns 2x - pl + {0,1,2}; the last of them is the first of the next output
        load_col(raw);
        dw_transpose_col<S>(ca, raw);
        load_col(raw);
        load_col(raw2);
        load_col(raw3);
        load_col(raw4);
        // two pairs of load buffers alternate, so four columns are in flight
        for (int x = x_begin; x < x_end; x += 2) {
            dw_transpose_col<S>(cb, raw);
            dw_transpose_col<S>(cc, raw2);
            load_col(raw);
            load_col(raw2);
            emit(ca, cb, cc);
            if (x + 1 >= x_end)
                break;
            dw_transpose_col<S>(cb, raw3);
            dw_transpose_col<S>(ca, raw4);
            load_col(raw3);
            load_col(raw4);
            emit(cc, cb, ca);
        }
    }
}

template <typename T, typename ACC, typename BIAS>
__global__ void __launch_bounds__(256) dw_generic_kernel(DwParams p)
{
    grid_dep_launch();
    grid_dep_wait();
    const T *__restrict__ in = (const T *)p.in;
    const T *__restrict__ w = (const T *)p.w;
    const BIAS *__restrict__ bias = (const BIAS *)p.bias;
    T *__restrict__ out = (T *)p.out;
    for (long long item = blockIdx.x * (long long)blockDim.x + threadIdx.x; item < p.total;
         item += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(item % p.c);
        const long long pix = item / p.c;
        const int ox = (int)(pix % p.ow);
        const int oy = (int)((pix / p.ow) % p.oh);
        const int n = (int)(pix / ((long long)p.ow * p.oh));
        ACC acc = 0;
        for (int ky = 0; ky < p.kh; ky++) {
            const int iy = oy * p.sh + ky * p.dh - p.pt;
            if (iy < 0 || iy >= p.ih)
                continue;
            for (int kx = 0; kx < p.kw; kx++) {
                const int ix = ox * p.sw + kx * p.dw - p.pl;
                if (ix < 0 || ix >= p.iw)
                    continue;
                acc += (ACC)((int)in[(((long long)n * p.ih + iy) * p.iw + ix) * p.ips + c] *
                             (int)w[((long long)ky * p.kw + kx) * p.c + c]);
            }
        }
        const int e = p.per_channel ? p.ew[c] : p.ew_scalar;
        if (sizeof(T) == 1) {
            const int shift = max(-31, min(32, p.e_shift_base - e));
            int32_t v = requant8((int32_t)acc, bias ? (int32_t)bias[c] : 0, shift, p.relu, p.half_even);
            if (p.lut)
                v = p.lut[(long long)c * p.lut_stride + ((uint8_t)v ^ 0x80u)];
            out[pix * p.ops + c] = (T)v;
        } else {
            const int shift = max(-62, min(62, p.e_shift_base - e));
            out[pix * p.ops + c] = (T)requant16((long long)acc, bias ? (long long)bias[c] : 0ll, shift, p.relu, p.half_even);
        }
    }
}

// Any window, stride and dilation, int8 and int16, four channels of an output pixel a thread.  Eight taps' words are asked for before the first is used (one
// after the other, each waited for, three taps over 24 pixels took as long as a launch more), and meet in dot products: groups of four taps of a channel in
// dp4a, pairs in dp2a with the filter's high (signed) and low (unsigned) bytes - |sum| < 2^31 for 255 taps - where 64-bit multiply-adds a channel at a time
// took twice as long.  us before / after: int8 24x32, 1x3 4.6 / 2.4, 20x20x128 3x3 at dilation 2 7.0 / 3.2; int16 154 of 12x11x192 5x5 146 / 65,
// 64 of 56x56x96 3x3 421 / 178, 4 of 47x44x64 at stride 2 7.8 / 5.1 (large int16 maps of these windows have since a kernel of their own below).
template <typename T>
struct TapWord; // four channels
template <>
struct TapWord<int8_t> {
    uint32_t v;
};
template <>
struct TapWord<int16_t> {
    uint2 v;
};
__device__ __forceinline__ void clear(TapWord<int8_t> &w) { w.v = 0u; }
__device__ __forceinline__ void clear(TapWord<int16_t> &w) { w.v = make_uint2(0u, 0u); }
__device__ __forceinline__ void load(TapWord<int8_t> &w, const int8_t *p) { w.v = __ldg((const uint32_t *)p); }
__device__ __forceinline__ void load(TapWord<int16_t> &w, const int16_t *p) { w.v = __ldg((const uint2 *)p); }

struct TapSums {
    int hi[4], lo[4]; // int8: hi only
};
// Bytes of four words as one word per channel.
__device__ __forceinline__ void transpose4(const TapWord<int8_t> *t, uint32_t (&c)[4])
{
    const uint32_t lo0 = __byte_perm(t[0].v, t[1].v, 0x5140), lo1 = __byte_perm(t[2].v, t[3].v, 0x5140), hi0 = __byte_perm(t[0].v, t[1].v, 0x7362),
                   hi1 = __byte_perm(t[2].v, t[3].v, 0x7362);
    c[0] = __byte_perm(lo0, lo1, 0x5410), c[1] = __byte_perm(lo0, lo1, 0x7632), c[2] = __byte_perm(hi0, hi1, 0x5410), c[3] = __byte_perm(hi0, hi1, 0x7632);
}
__device__ __forceinline__ void add_taps(TapSums &s, const TapWord<int8_t> (&x)[8], const TapWord<int8_t> (&w)[8])
{
#pragma unroll
    for (int g = 0; g < 8; g += 4) {
        uint32_t a[4], b[4];
        transpose4(x + g, a), transpose4(w + g, b);
#pragma unroll
        for (int c = 0; c < 4; c++) s.hi[c] = __dp4a((int)a[c], (int)b[c], s.hi[c]);
    }
}
__device__ __forceinline__ void add_taps(TapSums &s, const TapWord<int16_t> (&x)[8], const TapWord<int16_t> (&w)[8])
{
#pragma unroll
    for (int g = 0; g < 8; g += 2)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint32_t x0 = c < 2 ? x[g].v.x : x[g].v.y, x1 = c < 2 ? x[g + 1].v.x : x[g + 1].v.y, w0 = c < 2 ? w[g].v.x : w[g].v.y, w1 = c < 2 ? w[g + 1].v.x : w[g + 1].v.y;
            const uint32_t a = __byte_perm(x0, x1, c & 1 ? 0x7632 : 0x5410), b = __byte_perm(w0, w1, c & 1 ? 0x6273 : 0x4051); // b: high bytes, low bytes
            asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(s.hi[c]) : "r"(a), "r"(b));
            asm("dp2a.hi.s32.u32 %0, %1, %2, %0;" : "+r"(s.lo[c]) : "r"(a), "r"(b));
        }
}

template <typename T>
__global__ void __launch_bounds__(128) dw_taps_kernel(DwParams p)
{
    grid_dep_launch();
    if (!p.early)
        grid_dep_wait();
    const T *__restrict__ in = (const T *)p.in;
    const T *__restrict__ w = (const T *)p.w;
    T *__restrict__ out = (T *)p.out;
    const unsigned words = (unsigned)p.c / 4, total = (unsigned)p.total;
    const int taps = p.kh * p.kw;
    bool first = true;
    for (unsigned item = blockIdx.x * blockDim.x + threadIdx.x; item < total; item += gridDim.x * blockDim.x, first = false) {
        const unsigned pix = item / words, ch = 4 * (item - pix * words), line = pix / (unsigned)p.ow, image = line / (unsigned)p.oh;
        const int iy0 = (int)(line - image * p.oh) * p.sh - p.pt, ix0 = (int)(pix - line * p.ow) * p.sw - p.pl;
        TapWord<T> wv[8];
#pragma unroll
        for (int t = 0; t < 8; t++) {
            clear(wv[t]);
            if (t < taps)
                load(wv[t], w + (long long)t * p.c + ch);
        }
        int shift[4];
        long long bias[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            shift[i] = p.e_shift_base - (p.per_channel ? __ldg(p.ew + ch + i) : p.ew_scalar);
            bias[i] = !p.bias ? 0ll : sizeof(T) == 1 ? (long long)__ldg((const int32_t *)p.bias + ch + i) : __ldg((const long long *)p.bias + ch + i);
        }
        if (p.early && first)
            grid_dep_wait();
        const T *from = in + (long long)image * p.ih * p.iw * p.ips + ch;
        TapSums s;
#pragma unroll
        for (int c = 0; c < 4; c++) s.hi[c] = s.lo[c] = 0;
        int ky = 0, kx = 0;
        for (int t0 = 0; t0 < taps; t0 += 8) {
            TapWord<T> xv[8];
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const int iy = iy0 + ky * p.dh, ix = ix0 + kx * p.dw;
                clear(xv[t]);
                if (t0 + t < taps && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw)
                    load(xv[t], from + ((long long)iy * p.iw + ix) * p.ips);
                if (++kx == p.kw)
                    kx = 0, ky++;
            }
            if (t0) {
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    clear(wv[t]);
                    if (t0 + t < taps)
                        load(wv[t], w + (long long)(t0 + t) * p.c + ch);
                }
            }
            add_taps(s, xv, wv);
        }
        int q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (sizeof(T) == 1) {
                q[i] = requant8(s.hi[i], (int)bias[i], max(-31, min(32, shift[i])), p.relu, p.half_even);
                if (p.lut)
                    q[i] = p.lut[(long long)(ch + i) * p.lut_stride + ((uint8_t)q[i] ^ 0x80u)];
            } else {
                q[i] = requant16((long long)s.hi[i] * 256 + s.lo[i], bias[i], max(-62, min(62, shift[i])), p.relu, p.half_even);
            }
        }
        T *to = out + (long long)pix * p.ops + ch;
        if (sizeof(T) == 1)
            *(uint32_t *)to = ((uint32_t)q[0] & 0xffu) | (((uint32_t)q[1] & 0xffu) << 8) | (((uint32_t)q[2] & 0xffu) << 16) | ((uint32_t)q[3] << 24);
        else
            *(uint2 *)to = make_uint2(((uint32_t)q[0] & 0xffffu) | ((uint32_t)q[1] << 16), ((uint32_t)q[2] & 0xffffu) | ((uint32_t)q[3] << 16));
    }
    if (first && p.early)
        grid_dep_wait();
}

// The sums' bytes in halves (HalvesParam): 256 hi + lo.
template <bool EVEN>
__device__ __forceinline__ int requant_halves(int hi, int lo, const HalvesParam &c)
{
    return shift_halves<EVEN>((hi >> 8) + (lo >> 16) + c.h, ((hi & 0xff) << 8) + (lo & 0xffff) + c.l, c);
}
__device__ __noinline__ int requant16_any(int hi, int lo, long long bias, int shift, int relu, int half_even)
{
    return requant16((long long)hi * 256 + lo, bias, max(-62, min(62, shift)), relu, half_even);
}

// int16, 3x3 and 5x5 at stride 1 and 2: four channels of four (two at stride 2) neighbouring outputs of a row a thread, so that a row's words, their pairs and the
// filter's bytes serve all of them and the results leave through 32-bit instructions; dw_taps_kernel spends most of its instructions on addresses, pads nine taps
// to sixteen and requantises in 64 bits.  Bound by the integer pipe (62 % busy, issue slots 59 %) with 4 to 6 warps a scheduler to cover its chains: constants
// worked out behind the sums leave registers for them (116 of 75x75x192 3x3 403 -> 336 us), as six blocks an SM do for 5x5 (361 -> 343), one wait for the launch before without the form that waits later (334 -> 306); a row's loads after
// the row before's products cost 3x3 a tenth, two outputs a thread instead of four a sixth.
// us dw_taps_kernel / here: 116 of 75x75x192 3x3 1141 / 306, 965 of 40x40x48 5x5 1170 / 323, 64 of 56x56x96 3x3 177 / 49, 313 of 30x33x96 at stride 2 73 / 29.
template <int K, int S, bool EVEN>
__global__ void __launch_bounds__(128, 6) dw_run_s16_kernel(DwParams p, int segs)
{
    constexpr int R = S == 1 ? 4 : 2, IN = (R - 1) * S + K;
    grid_dep_launch();
    grid_dep_wait();
    const unsigned words = (unsigned)p.c / 4, item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= (unsigned)p.total)
        return;
    const unsigned run = item / words, line = run / (unsigned)segs, image = line / (unsigned)p.oh;
    const int ch = 4 * (int)(item - run * words), ox = (int)(run - line * segs) * R, iy0 = (int)(line - image * p.oh) * S - p.pt, ix0 = ox * S - p.pl;
    const int16_t *from = (const int16_t *)p.in + (long long)image * p.ih * p.iw * p.ips + (long long)ix0 * p.ips + ch;
    const int16_t *w = (const int16_t *)p.w + ch;
    int hi[R][4], lo[R][4];
#pragma unroll
    for (int j = 0; j < R; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) hi[j][c] = lo[j][c] = 0;
#pragma unroll(K == 3 ? 3 : 1)
    for (int ky = 0; ky < K; ky++, w += K * p.c) {
        const int iy = iy0 + ky;
        if ((unsigned)iy >= (unsigned)p.ih)
            continue;
        const int16_t *row = from + (long long)iy * p.iw * p.ips;
        uint2 x[IN], f[K];
#pragma unroll
        for (int i = 0; i < IN; i++) {
            x[i] = make_uint2(0u, 0u);
            if ((unsigned)(ix0 + i) < (unsigned)p.iw)
                x[i] = __ldg((const uint2 *)(row + (long long)i * p.ips));
        }
#pragma unroll
        for (int i = 0; i < K; i++) f[i] = __ldg((const uint2 *)(w + i * p.c));
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int g = 0; g < K; g += 2) {
                const uint32_t f0 = c < 2 ? f[g].x : f[g].y, f1 = g + 1 < K ? (c < 2 ? f[g + 1 < K ? g + 1 : g].x : f[g + 1 < K ? g + 1 : g].y) : 0u;
                // high bytes, low bytes; the last tap of a row meets the two channels of its word as they lie
                const uint32_t b = g + 1 < K ? __byte_perm(f0, f1, c & 1 ? 0x6273 : 0x4051) : __byte_perm(f0, 0u, c & 1 ? 0x2434 : 0x4041);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const int i = j * S + g;
                    const uint32_t x0 = c < 2 ? x[i].x : x[i].y;
                    uint32_t a = x0;
                    if (g + 1 < K)
                        a = __byte_perm(x0, c < 2 ? x[i + 1 < IN ? i + 1 : i].x : x[i + 1 < IN ? i + 1 : i].y, c & 1 ? 0x7632 : 0x5410);
                    asm("dp2a.lo.s32.s32 %0, %1, %2, %0;" : "+r"(hi[j][c]) : "r"(a), "r"(b));
                    asm("dp2a.hi.s32.u32 %0, %1, %2, %0;" : "+r"(lo[j][c]) : "r"(a), "r"(b));
                }
            }
        }
    }
    HalvesParam k[4];
    bool fast = true;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int sh = p.e_shift_base - (p.per_channel ? __ldg(p.ew + ch + c) : p.ew_scalar);
        const long long b = p.bias ? __ldg((const long long *)p.bias + ch + c) : 0ll;
        fast = fast && halves_fit(b, sh);
        k[c] = halves_param<EVEN>(b, sh);
    }
    int16_t *to = (int16_t *)p.out + ((long long)line * p.ow + ox) * p.ops + ch;
#pragma unroll
    for (int j = 0; j < R; j++, to += p.ops) {
        if (ox + j >= p.ow)
            break;
        int q[4];
        if (fast) {
#pragma unroll
            for (int c = 0; c < 4; c++) q[c] = requant_halves<EVEN>(hi[j][c], lo[j][c], k[c]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++)
                q[c] = requant16_any(hi[j][c], lo[j][c], p.bias ? __ldg((const long long *)p.bias + ch + c) : 0ll,
                                     p.e_shift_base - (p.per_channel ? __ldg(p.ew + ch + c) : p.ew_scalar), p.relu, EVEN);
        }
        uint2 o;
        asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(o.x) : "r"(q[1]), "r"(q[0]));
        asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(o.y) : "r"(q[3]), "r"(q[2]));
        if (p.relu) {
            asm("max.s16x2 %0, %0, %1;" : "+r"(o.x) : "r"(0));
            asm("max.s16x2 %0, %0, %1;" : "+r"(o.y) : "r"(0));
        }
        *(uint2 *)to = o;
    }
}

template <int K, int S>
void launch_dw_run(const DwParams &p, int segs, unsigned blocks, cudaStream_t s)
{
    launch_overlapped(p.half_even ? dw_run_s16_kernel<K, S, true> : dw_run_s16_kernel<K, S, false>, dim3(blocks), dim3(128), 0, s, p, segs);
}

int conv2d_depthwise(const espdl_conv_desc &d, cudaStream_t s)
{
    DwParams p;
    p.in = d.input, p.w = d.filter, p.bias = d.bias, p.out = d.output, p.ew = d.filter_exponents, p.lut = d.lut, p.lut_stride = d.lut_channel_stride;
    p.n = d.n, p.ih = d.in_h, p.iw = d.in_w, p.c = d.in_c, p.oh = d.out_h, p.ow = d.out_w;
    p.kh = d.kh, p.kw = d.kw, p.sh = d.stride_h, p.sw = d.stride_w, p.dh = d.dilation_h, p.dw = d.dilation_w;
    p.pt = d.pad_top, p.pl = d.pad_left;
    p.ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.e_shift_base = d.out_exponent - d.in_exponent;
    p.ew_scalar = d.filter_exponent, p.per_channel = d.per_channel;
    p.relu = d.activation == ESPDL_ACT_RELU, p.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.early = in_model_scope();
    const long long pixels = (long long)d.n * d.out_h * d.out_w;
    const int threads = 256;
    const long long max_blocks = (long long)num_sms() * 32;
    const bool vec = d.dtype == ESPDL_DTYPE_INT8 && d.in_c % 16 == 0 && p.ips % 16 == 0 && p.ops % 16 == 0 &&
        ((uintptr_t)d.input % 16) == 0 && ((uintptr_t)d.output % 16) == 0 && ((uintptr_t)d.filter % 16) == 0;
    const bool words4 = d.dtype == ESPDL_DTYPE_INT8 && d.in_c % 4 == 0 && p.ips % 4 == 0 && p.ops % 4 == 0 && ((uintptr_t)d.input % 4) == 0 &&
        ((uintptr_t)d.output % 4) == 0 && ((uintptr_t)d.filter % 4) == 0;
    const size_t word = d.dtype == ESPDL_DTYPE_INT8 ? 4 : 8; // four channels
    const bool taps = d.in_c % 4 == 0 && p.ips % 4 == 0 && p.ops % 4 == 0 && (((uintptr_t)d.input | (uintptr_t)d.output | (uintptr_t)d.filter) % word) == 0 &&
        d.kh * d.kw <= 255 && pixels * (d.in_c / 4) < 1ll << 31;
    const bool k3 = words4 && d.kh == 3 && d.kw == 3 && d.dilation_h == 1 && d.dilation_w == 1 && d.stride_h == d.stride_w &&
        (d.stride_h == 1 || d.stride_h == 2);
    // Threads of a few pixels' work each: fewer of them than this leave the chip idle.  us by runs / dw_taps_kernel: 20x20x96 5x5 5.2 / 4.6, 28x28x96 5.2 / 4.9,
    // 40x40x96 5.2 / 7.6; 3x3 20x20x128 3.3 / 3.2, 28x28x96 3.2 / 3.4, 64 of 7x7x32 3.2 / 4.5; 28x28x128 at stride 2 2.9 / 3.1 (5x5 4.4 / 4.6).
    const int run = d.stride_h == 1 ? 4 : 2, segs = (d.out_w + run - 1) / run; // of dw_run_s16_kernel
    const long long run_items = (long long)d.n * d.out_h * segs * (d.in_c / 4);
    const bool runs = taps && d.dtype == ESPDL_DTYPE_INT16 && (d.kh == 3 || d.kh == 5) && d.kh == d.kw && d.dilation_h == 1 && d.dilation_w == 1 &&
        d.stride_h == d.stride_w && (d.stride_h == 1 || d.stride_h == 2) && run_items >= (d.kh == 5 && d.stride_h == 1 ? 40ll : 16ll) * num_sms();
    const long long filter_bytes = (d.kh * d.kw + 3ll) / 4 * 4 * d.in_c; // of dwk_dp4a_kernel
    if (k3 && ((long long)d.in_w + 10) * p.ips <= DW_ZERO_ROW_BYTES) {
        // a thread walks along a whole band of rows when the batch gives enough threads without cutting the band
        const int rows_out = d.stride_h == 1 ? 4 : 2;
        const int ytiles = (d.out_h + rows_out - 1) / rows_out;
        const long long per_seg = (long long)d.n * ytiles * (d.in_c / 4);
        const long long want = (long long)num_sms() * 2048;
        int cols = d.out_w;
        while (cols > 8 && per_seg * ((d.out_w + cols - 1) / cols) < want) cols = (cols + 1) / 2;
        // a small layer is bound by the latency of the walk: short runs, although each reads two columns of its neighbour again
        while (cols > 2 && per_seg * ((d.out_w + cols - 1) / cols) < (long long)num_sms() * 128) cols = (cols + 1) / 2;
        const int xsegs = (d.out_w + cols - 1) / cols;
        const long long items = per_seg * xsegs;
        p.total = items, p.chunks = 0;
        const long long blocks = (items + 127) / 128;
        if (blocks > 0x7fffffffll)
            return ESPDL_ERR_TOO_LARGE;
        if (d.stride_h == 1)
            launch_overlapped(p.half_even ? dw3x3_dp4a_kernel<1, true> : dw3x3_dp4a_kernel<1, false>, dim3((unsigned)blocks), dim3(128), 0, s, p, xsegs, ytiles, cols);
        else
            launch_overlapped(p.half_even ? dw3x3_dp4a_kernel<2, true> : dw3x3_dp4a_kernel<2, false>, dim3((unsigned)blocks), dim3(128), 0, s, p, xsegs, ytiles, cols);
    } else if (words4 && (d.kh == 3 || d.kh == 5 || d.kh == 7) && d.kh == d.kw && d.dilation_h == 1 && d.dilation_w == 1 && filter_bytes <= 48 * 1024 &&
               pixels * (d.in_c / 4) < (d.kh == 7 ? 1024ll * num_sms() : 1ll << 31)) { // 49 words a thread leave too few threads for large maps (16x56x56x96: 85 us, 58 below)
        p.chunks = 0;
        p.total = pixels * (d.in_c / 4);
        const long long blocks = min((p.total + 255) / 256, max_blocks);
        launch_overlapped(d.kh == 3 ? dwk_dp4a_kernel<3> : (d.kh == 5 ? dwk_dp4a_kernel<5> : dwk_dp4a_kernel<7>), dim3((unsigned)blocks), dim3(256), (size_t)filter_bytes, s, p);
    } else if (runs) {
        p.chunks = 0;
        p.total = run_items;
        const unsigned blocks = (unsigned)((run_items + 127) / 128);
        if (d.kh == 3)
            d.stride_h == 1 ? launch_dw_run<3, 1>(p, segs, blocks, s) : launch_dw_run<3, 2>(p, segs, blocks, s);
        else
            d.stride_h == 1 ? launch_dw_run<5, 1>(p, segs, blocks, s) : launch_dw_run<5, 2>(p, segs, blocks, s);
    } else if (taps && (d.dtype == ESPDL_DTYPE_INT16 || !vec || pixels * (d.in_c / 4) <= 1024ll * num_sms())) {
        // int8 beyond: sixteen channels a thread, whose address and epilogue cost a quarter (64x56x56x96 at dilation 2 67 us, 154 here; 4x40x40x64 7.1 / 6.7)
        p.chunks = 0;
        p.total = pixels * (d.in_c / 4);
        const long long blocks = min((p.total + 127) / 128, max_blocks * 2);
        launch_overlapped(d.dtype == ESPDL_DTYPE_INT8 ? dw_taps_kernel<int8_t> : dw_taps_kernel<int16_t>, dim3((unsigned)blocks), dim3(128), 0, s, p);
    } else if (vec) {
        p.chunks = d.in_c / 16;
        p.total = pixels * p.chunks;
        long long blocks = min((p.total + threads - 1) / threads, max_blocks);
        launch_overlapped(dw_s8_vec16_kernel, dim3((unsigned)blocks), dim3(threads), 0, s, p);
    } else {
        p.chunks = 0;
        p.total = pixels * d.in_c;
        long long blocks = min((p.total + threads - 1) / threads, max_blocks);
        if (d.dtype == ESPDL_DTYPE_INT8)
            launch_overlapped(dw_generic_kernel<int8_t, int32_t, int32_t>, dim3((unsigned)blocks), dim3(threads), 0, s, p);
        else
            launch_overlapped(dw_generic_kernel<int16_t, long long, long long>, dim3((unsigned)blocks), dim3(threads), 0, s, p);
    }
    count_launch();
    return check_launch("conv2d_depthwise");
}

} // namespace espdl
