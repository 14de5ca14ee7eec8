// Small int8 convs, Gemms and products with the warp-level matrix instruction (mma.sync m16n8k32).
//
// The tile kernels start a TMA pipeline, tensor memory and eighteen warps per CTA and issue M = 128 instructions one after the other:
// right for large products, but a layer of one image (a few hundred pixels) is then all start-up - 3.1 us
// for next to nothing, 0.35 us more for every 128 bytes of the reduction (7x7x960 -> 160: 5.9 us, 10x10x128 -> 256 3x3 stride 2:
// 8.9 us) against 1.2 us for an empty kernel.  Here a warp computes a tile of (16 MT) x (8 NT) outputs straight from global
// memory (everything involved sits in L2), up to eight warps share a tile's reduction and add up through shared memory, and the first
// part of the filter and the epilogue's constants are in registers before the kernel waits for the one before it.  Bound by
// latency: one trip to L2 for the input, the reduction's last instruction, one exchange, the store.
//
// Fragments: the order of the reduction is free as long as both operands agree, so lane (g, t) of a warp takes 16 consecutive bytes at
// 64 * step + 16 * t of row g (input pixel or filter row): one 128-bit load per row and step, words 0, 1 feed the first
// instruction and words 2, 3 the second.  A window's taps are consecutive runs of the reduction; with Cin a multiple of 16 a chunk never
// leaves its tap.  ALIGN = 4: word loads, a word never leaves its tap (Cin a multiple of 4).  ALIGN = 1: any channel count (first
// layers): a filter row's taps are one run of KW * Cin bytes in the input too, padded here to whole chunks; a chunk is read as the five
// aligned words around it, shifted, and masked where it crosses the image's edge (27 images 192x96x3 -> 16, 7x7: 129 us before).
#include "common.cuh"

#include <climits>

namespace espdl {

namespace {

constexpr int MMA_WARPS = 8;

struct MmaParams {
    const int8_t *in, *w, *lut, *res;
    const int32_t *bias, *ew;
    int8_t *out;
    int M, N, K;                  // output pixels (per image of a batch of products), channels, reduction
    int steps;                    // 64-byte steps of the reduction
    int run, run_chunks;          // ALIGN 1: bytes of a filter row and its chunks
    int split;                    // warps that share a tile's reduction: 1, 2, 4 or 8
    int tiles_n, tiles;           // tiles of a matrix
    int ic, ih, iw, oh, ow, kw, sh, sw, dh, dw, pt, pl, ips, ops, rps, lut_stride;
    long long w_image;            // batch of products: elements from one image's filter to the next (gridDim.y images)
    int e_shift_base, ew_scalar, per_channel, relu, half_even;
    int acc_bound; // of |sum|, see fast_constants
    int early; // the filter is a constant of the model: loaded before the wait for the previous kernel
};

__device__ __forceinline__ void mma_s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16 bytes of a dense row of K bytes at offset k; zero past its end.
template <int ALIGN>
__device__ __forceinline__ uint4 dense_chunk(const int8_t *row, int k, int K)
{
    if (ALIGN == 16)
        return k < K ? __ldg((const uint4 *)(row + k)) : make_uint4(0u, 0u, 0u, 0u);
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = k + 4 * i < K ? __ldg((const uint32_t *)(row + k + 4 * i)) : 0u;
    return make_uint4(v[0], v[1], v[2], v[3]);
}

// Four channels outside the one-add-one-shift form.
__device__ __noinline__ uint32_t general_word(const MmaParams &p, const int (&v)[4], int oc0)
{
    uint32_t word = 0;
#pragma unroll 1 // rare: four copies of the form are half of a small kernel's code
    for (int i = 0; i < 4; i++) {
        const int n = min(oc0 + i, p.N - 1);
        const int shift = max(-31, min(32, p.e_shift_base - (p.per_channel ? __ldg(p.ew + n) : p.ew_scalar)));
        word |= ((uint32_t)requant8(v[i], p.bias ? __ldg(p.bias + n) : 0, shift, p.relu, p.half_even) & 0xffu) << (8 * i);
    }
    return word;
}

// 16 bytes from any address; words without a byte in [lo, hi) are not read.
__device__ __forceinline__ uint4 unaligned_chunk(const int8_t *at, const int8_t *lo, const int8_t *hi)
{
    const uint32_t *base = (const uint32_t *)((uintptr_t)at & ~(uintptr_t)3);
    const uint32_t sh = 8u * ((uint32_t)(uintptr_t)at & 3u);
    uint32_t w[5];
#pragma unroll
    for (int i = 0; i < 5; i++) w[i] = (const int8_t *)(base + i) < hi && (const int8_t *)(base + i + 1) > lo ? __ldg(base + i) : 0u;
    return make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh), __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
}

// The first `have` of 16 bytes from any address, all of them readable.
__device__ __forceinline__ uint4 inside_chunk(const int8_t *at, int have)
{
    const uint32_t *base = (const uint32_t *)((uintptr_t)at & ~(uintptr_t)3);
    const int m = (int)((uintptr_t)at & 3);
    uint32_t w[5];
#pragma unroll
    for (int i = 0; i < 5; i++) w[i] = 4 * i < have + m ? __ldg(base + i) : 0u;
    return make_uint4(__funnelshift_r(w[0], w[1], 8 * m), __funnelshift_r(w[1], w[2], 8 * m), __funnelshift_r(w[2], w[3], 8 * m), __funnelshift_r(w[3], w[4], 8 * m));
}

// Bytes [from, to) of a chunk stay, the others become zero.
__device__ __forceinline__ uint4 keep_bytes(uint4 v, int from, int to)
{
    if (from <= 0 && to >= 16)
        return v;
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int a = min(max(from - 4 * i, 0), 4), b = min(max(to - 4 * i, 0), 4);
        const uint32_t below_b = b == 4 ? 0xffffffffu : (1u << (8 * b)) - 1u, below_a = a == 4 ? 0xffffffffu : (1u << (8 * a)) - 1u;
        w[i] &= below_b & ~below_a;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

template <int MT, int NT, bool WINDOW, int ALIGN>
__global__ void __launch_bounds__(32 * MMA_WARPS) conv_mma_kernel(const __grid_constant__ MmaParams p)
{
    constexpr int ROWS = 16 * MT, COLS = 8 * NT, PITCH = NT == 1 ? 8 : COLS + 8; // the pitch keeps the fragments' stores off one another's banks
    constexpr int DEPTH = MT * NT <= 2 ? 4 : 2;                                  // steps whose loads are in flight together
    __shared__ __align__(16) int part[MMA_WARPS][ROWS * PITCH];
    grid_dep_launch(); // nothing is set up that the next kernel's blocks could disturb
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int kpart = warp & (p.split - 1), slot = warp / p.split;
    const int tile = blockIdx.x * (MMA_WARPS / p.split) + slot;
    const bool active = tile < p.tiles;
    const int tm = active ? tile / p.tiles_n : 0, tn = active ? tile - tm * p.tiles_n : 0;
    const int8_t *w = p.w + blockIdx.y * p.w_image;
    const long long image0 = (long long)blockIdx.y * p.M; // first output pixel of this matrix

    if (!p.early)
        grid_dep_wait();
    uint4 b[DEPTH][NT];
    auto load_b = [&](int s0) {
#pragma unroll
        for (int d = 0; d < DEPTH; d++)
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const int s = s0 + d * p.split, n = tn * COLS + 8 * j + g;
                b[d][j] = make_uint4(0u, 0u, 0u, 0u);
                if (active && s < p.steps && n < p.N) {
                    if constexpr (ALIGN == 1) {
                        const int q = 4 * s + t, ky = q / p.run_chunks, off = 16 * (q - ky * p.run_chunks), have = min(16, p.run - off);
                        const int8_t *at = w + (long long)n * p.K + ky * p.run + off;
                        if (ky * p.run < p.K)
                            b[d][j] = keep_bytes(unaligned_chunk(at, at, at + have), 0, have);
                    } else {
                        b[d][j] = dense_chunk<ALIGN>(w + (long long)n * p.K, 64 * s + 16 * t, p.K);
                    }
                }
            }
    };
    load_b(kpart);
    // epilogue: a thread takes four neighbouring channels, the same ones in every row it visits
    constexpr int QUADS = COLS / 4;
    const int e_lane = kpart * 32 + lane, cq = e_lane % QUADS, oc0 = tn * COLS + 4 * cq;
    int bias_half[4], shift[4];
    bool fast = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int n = min(oc0 + i, p.N - 1);
        fast = fast_constants(p.bias ? __ldg(p.bias + n) : 0, p.e_shift_base - (p.per_channel ? __ldg(p.ew + n) : p.ew_scalar), p.acc_bound, p.half_even,
                              bias_half[i], shift[i]) && fast;
    }
    // the input rows of this lane's fragments
    const int8_t *row[MT][2];
    int iy0[MT][2], ix0[MT][2];
    bool row_ok[MT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = tm * ROWS + 16 * i + 8 * h + g;
            row_ok[i][h] = active && m < p.M;
            const long long pix = image0 + (row_ok[i][h] ? m : 0);
            if (WINDOW) {
                // at most 2^24 pixels: divisions of 32 bits (of 64 they were a tenth of a first layer's instructions)
                const unsigned line = (unsigned)pix / (unsigned)p.ow, image = line / (unsigned)p.oh;
                const int ox = (int)((unsigned)pix - line * (unsigned)p.ow), oy = (int)(line - image * (unsigned)p.oh);
                iy0[i][h] = oy * p.sh - p.pt, ix0[i][h] = ox * p.sw - p.pl;
                row[i][h] = p.in + (long long)image * p.ih * p.iw * p.ips;
            } else {
                row[i][h] = p.in + pix * p.ips;
            }
        }
    if (p.early)
        grid_dep_wait();

    int acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[i][j][k] = 0;

    for (int s0 = kpart; s0 < p.steps; s0 += DEPTH * p.split) {
        if (s0 != kpart)
            load_b(s0);
        uint4 a[DEPTH][MT][2];
#pragma unroll
        for (int d = 0; d < DEPTH; d++) {
            const int k = 64 * (s0 + d * p.split) + 16 * t;
            if constexpr (ALIGN == 1) {
                // what lies behind the run meets zeros of the filter; only the image's edges have to read as zero
                const int q = k / 16, ky = q / p.run_chunks, off = 16 * (q - ky * p.run_chunks), width = p.iw * p.ic;
#pragma unroll
                for (int i = 0; i < MT; i++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int iy = iy0[i][h] + ky * p.dh, x = ix0[i][h] * p.ic + off;
                        a[d][i][h] = make_uint4(0u, 0u, 0u, 0u);
                        if (row_ok[i][h] && ky * p.run < p.K && (unsigned)iy < (unsigned)p.ih && x + 16 > 0 && x < width) {
                            const int8_t *line = row[i][h] + iy * width;
                            if (x >= 0 && x + 16 <= width)
                                a[d][i][h] = inside_chunk(line + x, min(16, p.run - off));
                            else
                                a[d][i][h] = keep_bytes(unaligned_chunk(line + x, line, line + width), -x, width - x);
                        }
                    }
            } else if (!WINDOW) {
#pragma unroll
                for (int i = 0; i < MT; i++)
#pragma unroll
                    for (int h = 0; h < 2; h++) a[d][i][h] = row_ok[i][h] ? dense_chunk<ALIGN>(row[i][h], k, p.K) : make_uint4(0u, 0u, 0u, 0u);
            } else {
                constexpr int PIECES = ALIGN == 16 ? 1 : 4;
                uint32_t v[MT][2][4];
#pragma unroll
                for (int q = 0; q < PIECES; q++) {
                    const int kq = k + 4 * q;
                    const int tap = kq / p.ic, c = kq - tap * p.ic, ky = tap / p.kw, kx = tap - ky * p.kw;
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int iy = iy0[i][h] + ky * p.dh, ix = ix0[i][h] + kx * p.dw;
                            const bool in = row_ok[i][h] && kq < p.K && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
                            const int8_t *at = row[i][h] + ((long long)iy * p.iw + ix) * p.ips + c;
                            if (ALIGN == 16)
                                a[d][i][h] = in ? __ldg((const uint4 *)at) : make_uint4(0u, 0u, 0u, 0u);
                            else
                                v[i][h][q] = in ? __ldg((const uint32_t *)at) : 0u;
                        }
                }
                if (ALIGN != 16)
#pragma unroll
                    for (int i = 0; i < MT; i++)
#pragma unroll
                        for (int h = 0; h < 2; h++) a[d][i][h] = make_uint4(v[i][h][0], v[i][h][1], v[i][h][2], v[i][h][3]);
            }
        }
#pragma unroll
        for (int d = 0; d < DEPTH; d++) {
            if (s0 + d * p.split >= p.steps)
                break;
#pragma unroll
            for (int i = 0; i < MT; i++)
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    mma_s8(acc[i][j], a[d][i][0].x, a[d][i][1].x, a[d][i][0].y, a[d][i][1].y, b[d][j].x, b[d][j].y);
                    mma_s8(acc[i][j], a[d][i][0].z, a[d][i][1].z, a[d][i][0].w, a[d][i][1].w, b[d][j].z, b[d][j].w);
                }
        }
    }
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) {
            *(int2 *)&part[warp][(16 * i + g) * PITCH + 8 * j + 2 * t] = make_int2(acc[i][j][0], acc[i][j][1]);
            *(int2 *)&part[warp][(16 * i + 8 + g) * PITCH + 8 * j + 2 * t] = make_int2(acc[i][j][2], acc[i][j][3]);
        }
    if (p.split > 1)
        __syncthreads();
    else
        __syncwarp();
    if (!active)
        return;
    const bool words = (p.ops & 3) == 0 && ((uintptr_t)p.out & 3) == 0 && oc0 + 4 <= p.N;
    const int floor_q = p.relu ? 0 : INT_MIN;
#pragma unroll 2
    for (int e = e_lane; e < ROWS * QUADS; e += p.split * 32) {
        const int r = e / QUADS, m = tm * ROWS + r;
        if (m >= p.M || oc0 >= p.N)
            continue;
        int4 sum = make_int4(0, 0, 0, 0);
        for (int k = 0; k < p.split; k++) {
            const int4 v = *(const int4 *)&part[slot * p.split + k][r * PITCH + 4 * cq];
            sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
        }
        const int v[4] = {sum.x, sum.y, sum.z, sum.w};
        const long long pix = image0 + m;
        int8_t *op = p.out + pix * p.ops + oc0;
        uint32_t word = 0;
        if (fast) {
            int q[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int w = __viaddmax_s32(v[i], bias_half[i], floor_q);
                q[i] = (w + ((w >> shift[i]) & p.half_even)) >> shift[i];
            }
            uint32_t hi;
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q[3]), "r"(q[2]));
            asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(word) : "r"(q[1]), "r"(q[0]), "r"(hi));
        } else {
            word = general_word(p, v, oc0);
        }
        if (p.lut || p.res) {
            uint32_t out = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int q = (int)(int8_t)(word >> (8 * i));
                const int n = min(oc0 + i, p.N - 1);
                if (p.lut)
                    q = __ldg(p.lut + (long long)n * p.lut_stride + ((uint8_t)q ^ 0x80u));
                if (p.res)
                    q = sat8(q + (int)p.res[pix * p.rps + n]);
                out |= ((uint32_t)q & 0xffu) << (8 * i);
            }
            word = out;
        }
        if (words) {
            *(uint32_t *)op = word;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (oc0 + i < p.N)
                    op[i] = (int8_t)(word >> (8 * i));
        }
    }
}

struct MmaPlan {
    int mt, nt, split;
    float us;
};

bool is_window(const espdl_conv_desc &d)
{
    return d.kh != 1 || d.kw != 1 || d.stride_h != 1 || d.stride_w != 1 || d.pad_top || d.pad_bottom || d.pad_left || d.pad_right;
}

int mma_align(const espdl_conv_desc &d)
{
    const int ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    const uintptr_t a = (uintptr_t)d.input | (uintptr_t)d.filter | (uintptr_t)ips | (uintptr_t)d.in_c | (uintptr_t)d.filter_image_stride;
    if (a % 4 == 0)
        return a % 16 == 0 ? 16 : 4;
    return ips == d.in_c && d.dilation_w == 1 && d.filter_image_stride == 0 ? 1 : 0;
}

int mma_steps(const espdl_conv_desc &d)
{
    return mma_align(d) == 1 ? (d.kh * ((d.kw * d.in_c + 15) / 16) + 3) / 4 : (d.kh * d.kw * d.in_c + 63) / 64;
}

// Tile and split with the least estimated time.  The estimate is a fit (12 % rms) to 106 timings of chains of 21 layers over all
// shapes and splits, 0.1 to 240 M multiply-adds: a trip to memory per batch of loads and an epilogue per tile share, times the
// rounds of blocks, and the issue of loads and stores by all warps of an SM.  2 x 4 tiles were never the best by more than 3 %.
MmaPlan mma_plan(const espdl_conv_desc &d)
{
    const bool batched = d.filter_image_stride != 0;
    const long long M = (batched ? 1ll : (long long)d.n) * d.out_h * d.out_w, images = batched ? d.n : 1;
    const int steps = mma_steps(d);
    const float loads = mma_align(d) == 16 ? 1.f : (mma_align(d) == 4 ? 4.f : 8.f), window = is_window(d) ? (mma_align(d) == 4 ? 0.2f : 0.0168f) : 0.f; // words find their tap one by one
    static const int shapes[3][2] = {{1, 1}, {1, 2}, {2, 2}};
    MmaPlan best = {0, 0, 0, 1e30f};
    for (const auto &s : shapes) {
        const int mt = s[0], nt = s[1], depth = mt * nt <= 2 ? 4 : 2;
        const float tiles = (float)images * (float)((M + 16 * mt - 1) / (16 * mt)) * (float)((d.out_c + 8 * nt - 1) / (8 * nt));
        for (int split = 1; split <= MMA_WARPS && split <= steps; split *= 2) {
            const int own = (steps + split - 1) / split;
            const float warps = tiles * split / num_sms(), rounds = max(1.f, warps / 16.f); // of an SM, which holds sixteen
            const float us = 0.54f + rounds * (1.f * ((own + depth - 1) / depth) + 0.288f * mt * nt / split + 0.0037f * own * mt * nt) + (split > 1 ? 0.136f : 0.f) +
                warps * (own * (0.0059f * (2 * mt + nt) * loads + window) + 0.0251f * mt * nt);
            if (us < best.us)
                best = {mt, nt, split, us};
        }
    }
    return best;
}

template <int MT, int NT>
void launch_mma(const MmaParams &p, bool window, int align, int images, cudaStream_t s)
{
    const int per_block = MMA_WARPS / p.split;
    const dim3 grid((unsigned)((p.tiles + per_block - 1) / per_block), (unsigned)images);
    const auto kernel = align == 1 ? conv_mma_kernel<MT, NT, true, 1>
        : window                   ? (align == 16 ? conv_mma_kernel<MT, NT, true, 16> : conv_mma_kernel<MT, NT, true, 4>)
                                   : (align == 16 ? conv_mma_kernel<MT, NT, false, 16> : conv_mma_kernel<MT, NT, false, 4>);
    launch_overlapped(kernel, grid, dim3(32 * MMA_WARPS), 0, s, p);
}

} // namespace

bool conv2d_mma_supported(const espdl_conv_desc &d)
{
    if (d.dtype != ESPDL_DTYPE_INT8 || d.group != 1 || mma_align(d) == 0 || d.filter_image_stride < 0)
        return false;
    const bool batched = d.filter_image_stride != 0;
    if (batched && (is_window(d) || d.n > 65535))
        return false;
    const long long M = (batched ? 1ll : (long long)d.n) * d.out_h * d.out_w;
    return M <= (1 << 24) && (long long)d.kh * d.kw * d.in_c <= (1 << 17);
}

float conv2d_mma_estimate_us(const espdl_conv_desc &d) { return mma_plan(d).us; }

int conv2d_mma(const espdl_conv_desc &d, cudaStream_t s)
{
    const bool batched = d.filter_image_stride != 0;
    const MmaPlan plan = mma_plan(d);
    MmaParams p;
    p.in = (const int8_t *)d.input, p.w = (const int8_t *)d.filter, p.lut = d.lut, p.res = (const int8_t *)d.residual;
    p.bias = (const int32_t *)d.bias, p.ew = d.filter_exponents, p.out = (int8_t *)d.output;
    p.M = (batched ? 1 : d.n) * d.out_h * d.out_w, p.N = d.out_c, p.K = d.kh * d.kw * d.in_c;
    p.steps = mma_steps(d), p.split = plan.split;
    p.run = d.kw * d.in_c, p.run_chunks = (p.run + 15) / 16;
    p.tiles_n = (p.N + 8 * plan.nt - 1) / (8 * plan.nt), p.tiles = p.tiles_n * ((p.M + 16 * plan.mt - 1) / (16 * plan.mt));
    p.ic = d.in_c, p.ih = d.in_h, p.iw = d.in_w, p.oh = d.out_h, p.ow = d.out_w, p.kw = d.kw;
    p.sh = d.stride_h, p.sw = d.stride_w, p.dh = d.dilation_h, p.dw = d.dilation_w, p.pt = d.pad_top, p.pl = d.pad_left;
    p.ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, p.ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    p.rps = d.residual_pixel_stride ? d.residual_pixel_stride : d.out_c, p.lut_stride = d.lut_channel_stride;
    p.w_image = d.filter_image_stride;
    p.e_shift_base = d.out_exponent - d.in_exponent, p.ew_scalar = d.filter_exponent, p.per_channel = d.per_channel;
    p.relu = d.activation == ESPDL_ACT_RELU, p.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    // 2^14 a term: beyond 65536 the sum alone may reach 2^31 and the rounding's half leave 32 bits, which no channel may risk
    p.acc_bound = p.K <= 65536 ? p.K << 14 : INT_MAX;
    p.early = in_model_scope();
    const bool window = is_window(d);
    const int align = mma_align(d), images = batched ? d.n : 1;
    if (plan.mt == 2)
        launch_mma<2, 2>(p, window, align, images, s);
    else if (plan.nt == 2)
        launch_mma<1, 2>(p, window, align, images, s);
    else
        launch_mma<1, 1>(p, window, align, images, s);
    count_launch();
    return check_launch("conv_mma");
}

} // namespace espdl
