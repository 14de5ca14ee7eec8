// CUDA-core Conv2D for every shape the tensor-core tile kernel does not take
// (filters larger than 1x1, channel counts that are not a multiple of 16, strides,
// dilation, int16 with a large K).  One thread owns one output pixel and a group of
// OCT consecutive output channels, so each input value it loads feeds OCT MACs; the
// int8 path reads four input channels per 32-bit load and uses dp4a.
//
// Replaces dl::base::conv2d<> for those shapes
// (esp-dl/dl/base/dl_base_conv2d.cpp:141-162 MAC loop, esp-dl/dl/base/dl_base.hpp:951-1022
// border handling, esp-dl/dl/base/dl_base_activate_buffer.hpp:27-73 epilogue).
#include "common.cuh"

namespace espdl {

struct ConvParams {
    const void *in, *w, *bias;
    void *out;
    const int32_t *ew;
    const int8_t *lut;
    int lut_stride; // 0: one table, else entries between the tables of consecutive channels
    const int8_t *res; // optional residual added to the result (a folded Add), or null
    int rps;           // residual pixel stride
    int n, ih, iw, ic, oh, ow, oc, kh, kw, sh, sw, dh, dw, pt, pl, ips, ops;
    int e_shift_base; // out_exponent - in_exponent; shift = base - e_w
    int ew_scalar, per_channel, relu, half_even;
    long long total; // number of (pixel, oc-group) work items
    int groups;      // oc groups per pixel
    int lanes;       // threads that share an item's reduction (a power of two up to 32)
    long long w_image; // elements between the filters of consecutive images (a batch of products), 0 = one filter
};

// The reduction of one work item (an output pixel, OCT output channels), whole or - SPLIT - this lane's share of it: words of VEC
// elements `sub`, sub + lanes, ... of the flattened window.
template <int OCT, int VEC, bool SPLIT, typename ACC, typename MulAdd>
__device__ __forceinline__ void simt_reduce(const ConvParams &p, int iy0, int ix0, long long in_image, long long w_first, int oc_left, long long wstride, int sub,
                                            ACC (&acc)[OCT], const MulAdd &mul_add)
{
    const int icw = p.ic / VEC;
    if constexpr (SPLIT) {
        const int words = p.kh * p.kw * icw;
#pragma unroll 4
        for (int q = sub; q < words; q += p.lanes) {
            const int tap = q / icw, c = (q - tap * icw) * VEC, ky = tap / p.kw, kx = tap - ky * p.kw;
            const int iy = iy0 + ky * p.dh, ix = ix0 + kx * p.dw;
            if ((unsigned)iy >= (unsigned)p.ih || (unsigned)ix >= (unsigned)p.iw)
                continue;
            const long long at = in_image + ((long long)iy * p.iw + ix) * p.ips + c, wt = w_first + (long long)q * VEC;
#pragma unroll
            for (int j = 0; j < OCT; j++)
                if (j < oc_left)
                    mul_add(at, wt + j * wstride, acc[j]);
        }
    } else {
        for (int ky = 0; ky < p.kh; ky++) {
            const int iy = iy0 + ky * p.dh;
            if (iy < 0 || iy >= p.ih)
                continue;
            for (int kx = 0; kx < p.kw; kx++) {
                const int ix = ix0 + kx * p.dw;
                if (ix < 0 || ix >= p.iw)
                    continue;
                const long long at = in_image + ((long long)iy * p.iw + ix) * p.ips, wt = w_first + ((long long)ky * p.kw + kx) * p.ic;
                for (int c = 0; c < icw; c++)
#pragma unroll
                    for (int j = 0; j < OCT; j++)
                        if (j < oc_left)
                            mul_add(at + c * VEC, wt + j * wstride + c * VEC, acc[j]);
            }
        }
    }
}

// Bound by the latency of the loads along a reduction: with few outputs a thread that walks its reduction alone takes 0.3 to 0.5 us
// per four elements (1x1024 by 1024: 143 us), so then `lanes` neighbouring threads share an item and add up by shuffles.
template <int OCT, bool DP4A, bool SPLIT>
__global__ void __launch_bounds__(256) conv_s8_kernel(ConvParams p)
{
    grid_dep_launch();
    grid_dep_wait();
    const int8_t *__restrict__ in = (const int8_t *)p.in;
    const int8_t *__restrict__ w = (const int8_t *)p.w;
    const int32_t *__restrict__ bias = (const int32_t *)p.bias;
    int8_t *__restrict__ out = (int8_t *)p.out;
    const long long wstride = (long long)p.kh * p.kw * p.ic; // elements per output channel
    const int lanes = SPLIT ? p.lanes : 1, sub = SPLIT ? (int)(threadIdx.x % lanes) : 0;
    const long long step = (long long)gridDim.x * blockDim.x / lanes;
    for (long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / lanes; __any_sync(0xffffffffu, first < p.total); first += step) {
        const bool live = first < p.total;
        const long long item = live ? first : p.total - 1;
        const int g = (int)(item % p.groups);
        const long long pix = item / p.groups;
        const int ox = (int)(pix % p.ow);
        const int oy = (int)((pix / p.ow) % p.oh);
        const int n = (int)(pix / ((long long)p.ow * p.oh));
        const int oc0 = g * OCT;
        int32_t acc[OCT];
#pragma unroll
        for (int j = 0; j < OCT; j++) acc[j] = 0;
        simt_reduce<OCT, DP4A ? 4 : 1, SPLIT>(p, oy * p.sh - p.pt, ox * p.sw - p.pl, (long long)n * p.ih * p.iw * p.ips, n * p.w_image + (long long)oc0 * wstride, p.oc - oc0,
                                              wstride, sub, acc, [&](long long at, long long wt, int32_t &sum) {
                                                  if (DP4A)
                                                      sum = __dp4a(__ldg((const int *)(in + at)), __ldg((const int *)(w + wt)), sum);
                                                  else
                                                      sum += (int)__ldg(in + at) * (int)__ldg(w + wt);
                                              });
        if (SPLIT)
            for (int d = lanes >> 1; d; d >>= 1)
#pragma unroll
                for (int j = 0; j < OCT; j++) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], d);
        int8_t *op = out + pix * p.ops + oc0;
#pragma unroll
        for (int j = 0; j < OCT; j++) {
            const int oc = oc0 + j;
            if (live && oc < p.oc && (!SPLIT || sub == j % lanes)) {
                const int e = p.per_channel ? p.ew[oc] : p.ew_scalar;
                const int shift = max(-31, min(32, p.e_shift_base - e));
                int32_t q = requant8(acc[j], bias ? bias[oc] : 0, shift, p.relu, p.half_even);
                if (p.lut)
                    q = p.lut[(long long)oc * p.lut_stride + ((uint8_t)q ^ 0x80u)];
                if (p.res)
                    q = sat8(q + (int)p.res[pix * p.rps + oc]);
                op[j] = (int8_t)q;
            }
        }
    }
}

template <int OCT, bool SPLIT>
__global__ void __launch_bounds__(256) conv_s16_kernel(ConvParams p)
{
    grid_dep_launch();
    grid_dep_wait();
    const int16_t *__restrict__ in = (const int16_t *)p.in;
    const int16_t *__restrict__ w = (const int16_t *)p.w;
    const long long *__restrict__ bias = (const long long *)p.bias;
    int16_t *__restrict__ out = (int16_t *)p.out;
    const long long wstride = (long long)p.kh * p.kw * p.ic;
    const int lanes = SPLIT ? p.lanes : 1, sub = SPLIT ? (int)(threadIdx.x % lanes) : 0;
    const long long step = (long long)gridDim.x * blockDim.x / lanes;
    for (long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / lanes; __any_sync(0xffffffffu, first < p.total); first += step) {
        const bool live = first < p.total;
        const long long item = live ? first : p.total - 1;
        const int g = (int)(item % p.groups);
        const long long pix = item / p.groups;
        const int ox = (int)(pix % p.ow);
        const int oy = (int)((pix / p.ow) % p.oh);
        const int n = (int)(pix / ((long long)p.ow * p.oh));
        const int oc0 = g * OCT;
        long long acc[OCT];
#pragma unroll
        for (int j = 0; j < OCT; j++) acc[j] = 0;
        simt_reduce<OCT, 1, SPLIT>(p, oy * p.sh - p.pt, ox * p.sw - p.pl, (long long)n * p.ih * p.iw * p.ips, n * p.w_image + (long long)oc0 * wstride, p.oc - oc0, wstride, sub,
                                   acc, [&](long long at, long long wt, long long &sum) {
                                       sum += (long long)((int)__ldg(in + at) * (int)__ldg(w + wt)); // |a*w| <= 2^30: exact in int32
                                   });
        if (SPLIT)
            for (int d = lanes >> 1; d; d >>= 1)
#pragma unroll
                for (int j = 0; j < OCT; j++) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], d);
        int16_t *op = out + pix * p.ops + oc0;
#pragma unroll
        for (int j = 0; j < OCT; j++) {
            const int oc = oc0 + j;
            if (live && oc < p.oc && (!SPLIT || sub == j % lanes)) {
                const int e = p.per_channel ? p.ew[oc] : p.ew_scalar;
                const int shift = max(-62, min(62, p.e_shift_base - e));
                op[j] = (int16_t)requant16(acc[j], bias ? bias[oc] : 0ll, shift, p.relu, p.half_even);
            }
        }
    }
}

// Stem-style convolutions (a handful of input channels, e.g. the 3-channel 3x3 stride-2 first layer of an image
// network): K = kh*kw*in_c is tiny, so the whole filter bank sits in shared memory packed four taps per 32-bit
// word, each thread gathers the K input bytes of ONE output pixel into registers once and then produces every
// output channel of that pixel with dp4a.  Output bytes of a pixel are contiguous, so stores are 128-bit.
constexpr int SMALL_MAX_WORDS = 16; // K <= 64
constexpr int SMALL_MAX_OC = 64;

template <int KH, int KW, int IC>
__global__ void __launch_bounds__(256) conv_s8_small_k_kernel(ConvParams p)
{
    grid_dep_launch();
    grid_dep_wait();
    __shared__ int w_s[SMALL_MAX_OC * SMALL_MAX_WORDS];
    __shared__ int bias_s[SMALL_MAX_OC];
    __shared__ int shift_s[SMALL_MAX_OC];
    constexpr int K = KH * KW * IC;
    constexpr int words = (K + 3) / 4;
    static_assert(words <= SMALL_MAX_WORDS, "filter too large for the small-K kernel");
    const int8_t *__restrict__ in = (const int8_t *)p.in;
    const int8_t *__restrict__ w = (const int8_t *)p.w;
    for (int i = threadIdx.x; i < p.oc * words; i += blockDim.x) {
        const int oc = i / words, wd = i % words;
        uint32_t v = 0;
        for (int b = 0; b < 4; b++) {
            const int k = wd * 4 + b;
            if (k < K)
                v |= ((uint32_t)(uint8_t)w[(long long)oc * K + k]) << (8 * b);
        }
        w_s[i] = (int)v;
    }
    for (int oc = threadIdx.x; oc < p.oc; oc += blockDim.x) {
        bias_s[oc] = p.bias ? ((const int32_t *)p.bias)[oc] : 0;
        const int e = p.per_channel ? p.ew[oc] : p.ew_scalar;
        shift_s[oc] = max(-31, min(32, p.e_shift_base - e));
    }
    __syncthreads();
    const long long pixels = (long long)p.n * p.oh * p.ow;
    const bool vec_store = (p.oc % 16 == 0) && (p.ops % 16 == 0) && (((uintptr_t)p.out) % 16 == 0);
    for (long long pix = blockIdx.x * (long long)blockDim.x + threadIdx.x; pix < pixels; pix += (long long)gridDim.x * blockDim.x) {
        const int ox = (int)(pix % p.ow);
        const int oy = (int)((pix / p.ow) % p.oh);
        const int n = (int)(pix / ((long long)p.ow * p.oh));
        int a[words];
#pragma unroll
        for (int i = 0; i < words; i++) a[i] = 0;
        // gather the K input bytes in filter order (ky, kx, c); taps outside the image stay 0
#pragma unroll
        for (int ky = 0; ky < KH; ky++) {
            const int iy = oy * p.sh + ky * p.dh - p.pt;
#pragma unroll
            for (int kx = 0; kx < KW; kx++) {
                const int ix = ox * p.sw + kx * p.dw - p.pl;
                const bool inside = iy >= 0 && iy < p.ih && ix >= 0 && ix < p.iw;
                const int8_t *ip = in + (((long long)n * p.ih + iy) * p.iw + ix) * p.ips;
#pragma unroll
                for (int c = 0; c < IC; c++) {
                    constexpr int dummy = 0;
                    (void)dummy;
                    const int k = (ky * KW + kx) * IC + c; // compile-time after unrolling: a[] stays in registers
                    const uint32_t v = inside ? (uint32_t)(uint8_t)__ldg(ip + c) : 0u;
                    a[k >> 2] |= (int)(v << (8 * (k & 3)));
                }
            }
        }
        int8_t *op = (int8_t *)p.out + pix * p.ops;
        for (int oc0 = 0; oc0 < p.oc; oc0 += 16) {
            uint32_t pk[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int oc = oc0 + j;
                if (oc < p.oc) {
                    int acc = 0;
                    const int *wr = w_s + oc * words;
#pragma unroll
                    for (int i = 0; i < words; i++) acc = __dp4a(a[i], wr[i], acc);
                    int q = requant8(acc, bias_s[oc], shift_s[oc], p.relu, p.half_even);
                    if (p.lut)
                        q = p.lut[(long long)oc * p.lut_stride + ((uint8_t)q ^ 0x80u)];
                    pk[j >> 2] |= ((uint32_t)q & 0xffu) << (8 * (j & 3));
                }
            }
            if (vec_store) {
                *(uint4 *)(op + oc0) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            } else {
                for (int j = 0; j < 16 && oc0 + j < p.oc; j++) op[oc0 + j] = (int8_t)(pk[j >> 2] >> (8 * (j & 3)));
            }
        }
    }
}

// Short windows with few output channels over large maps (the 2x2 convs of a text detector's first and last layers), int8: a thread owns an
// output pixel and four channels, the filter sits in shared memory as [chunk][channel of four][group], so that the lanes of a pixel
// read neighbouring chunks at once, and the loads of four chunks of the window are in flight together.  A tile kernel spends 1.3
// to 2.6 us per wave of 128-pixel tiles on these, nearly all of it on the tile's way through its pipeline, for 64 multiply-adds an
// output: 735x735x16 -> 1, 2x2 40 -> 13.5 us, 367x367x16 -> 16 18.5 -> 13.5, 368x368x8 -> 16 24.3 -> 12.1.
constexpr int NARROW_MAX_K = 144, NARROW_MAX_OC = 32;

template <typename U>
__global__ void __launch_bounds__(256) conv_s8_narrow_kernel(ConvParams p, int early)
{
    constexpr int CH = (int)sizeof(U), WORDS = CH / 4;
    struct alignas(CH) Chunk {
        int w[WORDS];
    };
    extern __shared__ __align__(16) uint8_t narrow_w[];
    Chunk *w_s = (Chunk *)narrow_w;
    grid_dep_launch();
    if (!early)
        grid_dep_wait();
    const int per_tap = p.ic / CH, chunks = p.kh * p.kw * per_tap, groups = p.groups;
    for (int i = threadIdx.x; i < chunks * 4 * groups; i += 256) {
        const int g = i % groups, j = i / groups % 4, q = i / groups / 4, oc = 4 * g + j;
        Chunk v = {};
        if (oc < p.oc) {
            const U t = __ldg((const U *)((const int8_t *)p.w + (long long)oc * chunks * CH) + q);
            v = *(const Chunk *)&t;
        }
        w_s[i] = v;
    }
    if (early)
        grid_dep_wait();
    __syncthreads();
    const unsigned total = (unsigned)p.total; // below 2^31
    for (unsigned item = blockIdx.x * 256u + threadIdx.x; item < total; item += gridDim.x * 256u) {
        const unsigned pix = item / (unsigned)groups, g = item - pix * (unsigned)groups, line = pix / (unsigned)p.ow, n = line / (unsigned)p.oh;
        const int iy0 = (int)(line - n * (unsigned)p.oh) * p.sh - p.pt, ix0 = (int)(pix - line * (unsigned)p.ow) * p.sw - p.pl;
        const int8_t *image = (const int8_t *)p.in + (long long)n * p.ih * p.iw * p.ips;
        int acc[4] = {0, 0, 0, 0};
        int ky = 0, kx = 0, c = 0; // of chunk q
#pragma unroll 1
        for (int q0 = 0; q0 < chunks; q0 += 4) {
            Chunk a[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int iy = iy0 + ky * p.dh, ix = ix0 + kx * p.dw;
                a[u] = {};
                if (q0 + u < chunks && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw) {
                    const U t = __ldg((const U *)(image + ((long long)iy * p.iw + ix) * p.ips) + c);
                    a[u] = *(const Chunk *)&t;
                }
                if (++c == per_tap) {
                    c = 0;
                    if (++kx == p.kw)
                        kx = 0, ky++;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (q0 + u >= chunks)
                    break;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const Chunk b = w_s[((q0 + u) * 4 + j) * groups + g];
#pragma unroll
                    for (int i = 0; i < WORDS; i++) acc[j] = __dp4a(a[u].w[i], b.w[i], acc[j]);
                }
            }
        }
        const int oc0 = (int)g * 4;
        int8_t *op = (int8_t *)p.out + (long long)pix * p.ops + oc0;
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int oc = min(oc0 + j, p.oc - 1);
            const int shift = max(-31, min(32, p.e_shift_base - (p.per_channel ? __ldg(p.ew + oc) : p.ew_scalar)));
            int q = requant8(acc[j], p.bias ? __ldg((const int32_t *)p.bias + oc) : 0, shift, p.relu, p.half_even);
            if (p.lut)
                q = p.lut[(long long)oc * p.lut_stride + ((uint8_t)q ^ 0x80u)];
            if (p.res)
                q = sat8(q + (int)p.res[(long long)pix * p.rps + oc]);
            word |= ((uint32_t)q & 0xffu) << (8 * j);
        }
        if (oc0 + 4 <= p.oc && (p.ops & 3) == 0 && ((uintptr_t)p.out & 3) == 0) {
            *(uint32_t *)op = word;
        } else {
            for (int j = 0; j < 4 && oc0 + j < p.oc; j++) op[j] = (int8_t)(word >> (8 * j));
        }
    }
}

static int narrow_chunk(const espdl_conv_desc &d)
{
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    const uintptr_t all = (uintptr_t)d.in_c | (uintptr_t)ips | (uintptr_t)d.input | (uintptr_t)d.filter;
    return all % 16 == 0 ? 16 : (all % 8 == 0 ? 8 : (all % 4 == 0 ? 4 : 0));
}

bool conv2d_narrow_supported(const espdl_conv_desc &d)
{
    return d.dtype == ESPDL_DTYPE_INT8 && d.group == 1 && d.filter_image_stride == 0 && d.kh * d.kw > 1 && d.kh * d.kw * d.in_c <= NARROW_MAX_K && d.out_c <= NARROW_MAX_OC &&
        narrow_chunk(d) && (long long)d.n * d.out_h * d.out_w * ((d.out_c + 3) / 4) < (1ll << 31);
}

// A thread's instructions - a dot product per word and channel, about fourteen per chunk, sixty for the ends - at the measured issue rate.
float conv2d_narrow_estimate_us(const espdl_conv_desc &d)
{
    const double items = (double)d.n * d.out_h * d.out_w * ((d.out_c + 3) / 4), K = d.kh * d.kw * d.in_c;
    return (float)(2.0 + items * (K + 14 * K / narrow_chunk(d) + 60) / (num_sms() * 4 * 32 * 430.0));
}

static bool simt_dp4a(const espdl_conv_desc &d)
{
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    return d.dtype == ESPDL_DTYPE_INT8 && d.in_c % 4 == 0 && ips % 4 == 0 && ((uintptr_t)d.input % 4) == 0 && ((uintptr_t)d.filter % 4) == 0 && d.filter_image_stride % 4 == 0;
}

// Threads per item: until the GPU has work for all its schedulers, or a thread's share is down to four words (from twelve words on:
// six ran 6.2 us whole and 8.9 us split).
static int simt_lanes(const espdl_conv_desc &d)
{
    const long long items = (long long)d.n * d.out_h * d.out_w * ((d.out_c + 3) / 4), words = (long long)d.kh * d.kw * d.in_c / (simt_dp4a(d) ? 4 : 1);
    int lanes = 1;
    // (short reductions sooner: 504 pixels x 192 channels of 27 words took 13.7 us over four lanes, 10.4 whole)
    while (words >= 12 && lanes < 32 && words > 4 * lanes && items * lanes < (long long)num_sms() * (words < 64 ? 128 : 1024)) lanes *= 2;
    return lanes;
}

float conv2d_simt_estimate_us(const espdl_conv_desc &d)
{
    const double macs = (double)d.n * d.out_h * d.out_w * d.out_c * d.kh * d.kw * d.in_c, words = (double)d.kh * d.kw * d.in_c / (simt_dp4a(d) ? 4 : 1) / simt_lanes(d);
    const double rate = d.dtype == ESPDL_DTYPE_INT16 ? 0.5e6 : (simt_dp4a(d) ? 2.2e6 : 0.8e6); // multiply-adds per us, measured
    return (float)(3.0 + words * 0.3 + macs / rate);
}

static void fill_params(const espdl_conv_desc &d, ConvParams &p)
{
    p.res = (const int8_t *)d.residual, p.rps = d.residual_pixel_stride ? d.residual_pixel_stride : d.out_c;
    p.in = d.input, p.w = d.filter, p.bias = d.bias, p.out = d.output, p.ew = d.filter_exponents, p.lut = d.lut, p.lut_stride = d.lut_channel_stride;
    p.n = d.n, p.ih = d.in_h, p.iw = d.in_w, p.ic = d.in_c, p.oh = d.out_h, p.ow = d.out_w, p.oc = d.out_c;
    p.kh = d.kh, p.kw = d.kw, p.sh = d.stride_h, p.sw = d.stride_w, p.dh = d.dilation_h, p.dw = d.dilation_w;
    p.pt = d.pad_top, p.pl = d.pad_left;
    p.w_image = d.filter_image_stride;
    p.ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.e_shift_base = d.out_exponent - d.in_exponent;
    p.ew_scalar = d.filter_exponent, p.per_channel = d.per_channel;
    p.relu = d.activation == ESPDL_ACT_RELU, p.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.groups = (d.out_c + 3) / 4;
    p.total = (long long)d.n * d.out_h * d.out_w * p.groups;
}

int conv2d_narrow(const espdl_conv_desc &d, cudaStream_t s)
{
    ConvParams p;
    fill_params(d, p);
    p.lanes = 1;
    const unsigned grid = (unsigned)min((p.total + 255) / 256, (long long)num_sms() * 32);
    const size_t smem = (size_t)p.groups * 4 * d.kh * d.kw * d.in_c;
    const int chunk = narrow_chunk(d);
    launch_overlapped(chunk == 16 ? conv_s8_narrow_kernel<uint4> : (chunk == 8 ? conv_s8_narrow_kernel<uint2> : conv_s8_narrow_kernel<uint32_t>), dim3(grid), dim3(256), smem, s, p,
                      (int)in_model_scope());
    count_launch();
    return check_launch("conv2d_narrow");
}

int conv2d_simt(const espdl_conv_desc &d, cudaStream_t s)
{
    ConvParams p;
    fill_params(d, p);
    constexpr int OCT = 4;
    const int threads = 256;
    p.lanes = simt_lanes(d);
    long long blocks = (p.total * p.lanes + threads - 1) / threads;
    const long long max_blocks = (long long)num_sms() * 32;
    if (blocks > max_blocks)
        blocks = max_blocks;
    if (d.dtype == ESPDL_DTYPE_INT8 && !d.filter_image_stride && d.out_c <= SMALL_MAX_OC && d.kh == 3 && d.kw == 3 && (d.in_c == 3 || d.in_c == 1 || d.in_c == 4)) {
        const long long pixels = (long long)d.n * d.out_h * d.out_w;
        const unsigned grid = (unsigned)min((pixels + threads - 1) / threads, max_blocks);
        if (d.in_c == 3)
            launch_overlapped(conv_s8_small_k_kernel<3, 3, 3>, dim3(grid), dim3(threads), 0, s, p);
        else if (d.in_c == 1)
            launch_overlapped(conv_s8_small_k_kernel<3, 3, 1>, dim3(grid), dim3(threads), 0, s, p);
        else
            launch_overlapped(conv_s8_small_k_kernel<3, 3, 4>, dim3(grid), dim3(threads), 0, s, p);
    } else if (d.dtype == ESPDL_DTYPE_INT8) {
        const bool dp4a = simt_dp4a(d), split = p.lanes > 1;
        launch_overlapped(dp4a ? (split ? conv_s8_kernel<OCT, true, true> : conv_s8_kernel<OCT, true, false>)
                               : (split ? conv_s8_kernel<OCT, false, true> : conv_s8_kernel<OCT, false, false>),
                          dim3((unsigned)blocks), dim3(threads), 0, s, p);
    } else {
        launch_overlapped(p.lanes > 1 ? conv_s16_kernel<OCT, true> : conv_s16_kernel<OCT, false>, dim3((unsigned)blocks), dim3(threads), 0, s, p);
    }
    count_launch();
    return check_launch("conv2d_simt");
}

} // namespace espdl
