// Operand packing for the products that the tile kernel cannot read in place: rows of K elements become rows of Kp = K
// rounded up to 16 bytes, with the window of a convolution unrolled (a row is one output pixel), for
//   int16   two byte planes per operand.  The input splits into a signed high and an unsigned low byte (x = 256*hi + lo); the filter
//           is shifted into the unsigned range first, w + 32768 = 256*uh + ul, so that its two planes have ONE signedness and
//           the tile kernel multiplies a plane of the input by both in one instruction of twice the width; what the shift adds,
//           32768 * (sum of the input row), is taken off again in the epilogue with the row sums written here.
//   int8    the rows themselves (reductions that are no multiple of 16, windows over channel counts that are none).
// Bound by memory traffic: every source element is read once per window position it appears in (from L1 / L2 mostly), every
// plane written once, 16 bytes per thread and store.  A group of lanes owns a row - as many as it has 16-element chunks, up to
// a warp - so a row's sum is a shuffle away.
#include "common.cuh"

namespace espdl {

namespace {

struct PackParams {
    const void *in, *w;
    int8_t *a_hi, *b_hi;
    uint8_t *a_lo, *b_lo; // int16
    int *row_sum;         // int16: one per row of A
    int rows, N, K, Kp, lanes;
    long long row0; // first output pixel
    int ih, iw, ic, oh, ow, kw, sh, sw, dh, dw, pt, pl, ips;
};

__device__ __forceinline__ uint32_t pack4(const int *v) { return (uint32_t)(v[0] & 255) | ((uint32_t)(v[1] & 255) << 8) | ((uint32_t)(v[2] & 255) << 16) | ((uint32_t)v[3] << 24); }

__device__ __forceinline__ uint4 pack16(const int (&v)[16]) { return make_uint4(pack4(v), pack4(v + 4), pack4(v + 8), pack4(v + 12)); }

// 16 consecutive elements of a dense row; `vec`: 16-byte loads are in order.
template <typename T>
__device__ __forceinline__ void dense16(const T *src, int count, bool vec, int (&v)[16])
{
    if (vec && count >= 16) {
        alignas(16) T t[16];
        *(uint4 *)t = __ldg((const uint4 *)src);
        if (sizeof(T) == 2)
            *(uint4 *)(t + 8) = __ldg((const uint4 *)(src + 8));
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = t[j];
    } else {
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = j < count ? (int)src[j] : 0;
    }
}

// 16 int16 elements (their words) as 16 high and 16 low bytes, and their sum: byte permutes and dot products, a sixth of the instructions
// that shifts and masks of single elements take (3x3 windows over 64 channels, 25600 pixels, packed and multiplied: 33.2 -> 23.5 us).
__device__ __forceinline__ int split16(const uint4 a, const uint4 b, uint4 &hi, uint4 &lo)
{
    hi = make_uint4(__byte_perm(a.x, a.y, 0x7531), __byte_perm(a.z, a.w, 0x7531), __byte_perm(b.x, b.y, 0x7531), __byte_perm(b.z, b.w, 0x7531));
    lo = make_uint4(__byte_perm(a.x, a.y, 0x6420), __byte_perm(a.z, a.w, 0x6420), __byte_perm(b.x, b.y, 0x6420), __byte_perm(b.z, b.w, 0x6420));
    const int high = __dp4a((int)hi.x, 0x01010101, __dp4a((int)hi.y, 0x01010101, __dp4a((int)hi.z, 0x01010101, __dp4a((int)hi.w, 0x01010101, 0))));
    const unsigned low = __dp4a(lo.x, 0x01010101u, __dp4a(lo.y, 0x01010101u, __dp4a(lo.z, 0x01010101u, __dp4a(lo.w, 0x01010101u, 0u))));
    return high * 256 + (int)low;
}

template <typename T, bool WINDOW>
__global__ void __launch_bounds__(256) pack_kernel(PackParams p)
{
    grid_dep_launch(); // what this writes is read by the tile kernel's loads only, all of which wait for it (TcParams::filter_early)
    grid_dep_wait();
    const int lane = threadIdx.x & 31, sub = lane % p.lanes, per_warp = 32 / p.lanes;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long groups = ((long long)p.rows + p.N + per_warp - 1) / per_warp;
    const bool vec_w = p.K % 16 == 0 && ((uintptr_t)p.w & 15) == 0;
    const bool vec_in = p.ips % 16 == 0 && p.ic % 16 == 0 && ((uintptr_t)p.in & 15) == 0;
    for (long long g = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5); g < groups; g += warps) {
        const long long row = g * per_warp + lane / p.lanes;
        const bool is_b = row >= p.rows, live = row < (long long)p.rows + p.N;
        int sum = 0;
        if (live && is_b) {
            const long long n = row - p.rows;
#pragma unroll 2
            for (int k = sub * 16; k < p.Kp; k += p.lanes * 16) {
                if (sizeof(T) == 2 && vec_w) {
                    const uint4 *at = (const uint4 *)((const T *)p.w + n * p.K + k);
                    uint4 hi, lo;
                    split16(__ldg(at), __ldg(at + 1), hi, lo);
                    hi.x ^= 0x80808080u, hi.y ^= 0x80808080u, hi.z ^= 0x80808080u, hi.w ^= 0x80808080u; // + 32768
                    *(uint4 *)(p.b_hi + n * p.Kp + k) = hi;
                    *(uint4 *)(p.b_lo + n * p.Kp + k) = lo;
                    continue;
                }
                int v[16];
                dense16((const T *)p.w + n * p.K + k, p.K - k, vec_w, v);
                if (sizeof(T) == 2) {
                    int hi[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const int u = k + j < p.K ? v[j] + 32768 : 0;
                        hi[j] = u >> 8, v[j] = u;
                    }
                    *(uint4 *)(p.b_hi + n * p.Kp + k) = pack16(hi);
                    *(uint4 *)(p.b_lo + n * p.Kp + k) = pack16(v);
                } else {
                    *(uint4 *)(p.b_hi + n * p.Kp + k) = pack16(v);
                }
            }
        } else if (live) {
            const long long pix = p.row0 + row;
            const T *src = (const T *)p.in + pix * p.ips;
            int iy0 = 0, ix0 = 0;
            if (WINDOW) {
                const unsigned line = (unsigned)pix / (unsigned)p.ow, image = line / (unsigned)p.oh; // fewer than 2^31 pixels
                const int ox = (int)((unsigned)pix - line * (unsigned)p.ow), oy = (int)(line - image * (unsigned)p.oh);
                src = (const T *)p.in + (long long)image * p.ih * p.iw * p.ips;
                iy0 = oy * p.sh - p.pt, ix0 = ox * p.sw - p.pl;
            }
#pragma unroll 2
            for (int k = sub * 16; k < p.Kp; k += p.lanes * 16) {
                if (sizeof(T) == 2 && vec_in && (WINDOW || k + 16 <= p.K)) {
                    const T *at = src + k;
                    bool in = true;
                    if (WINDOW) { // a chunk never leaves its tap
                        const int tap = k / p.ic, ky = tap / p.kw, iy = iy0 + ky * p.dh, ix = ix0 + (tap - ky * p.kw) * p.dw;
                        in = k < p.K && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
                        at = src + ((long long)iy * p.iw + ix) * p.ips + (k - tap * p.ic);
                    }
                    uint4 x0 = make_uint4(0, 0, 0, 0), x1 = x0, hi, lo;
                    if (in)
                        x0 = __ldg((const uint4 *)at), x1 = __ldg((const uint4 *)at + 1);
                    sum += split16(x0, x1, hi, lo);
                    *(uint4 *)(p.a_hi + row * p.Kp + k) = hi;
                    *(uint4 *)(p.a_lo + row * p.Kp + k) = lo;
                    continue;
                }
                int v[16];
                if (!WINDOW) {
                    dense16(src + k, p.K - k, vec_in, v);
                } else {
                    int tap = k / p.ic, c = k - tap * p.ic;
                    int ky = tap / p.kw, kx = tap - ky * p.kw;
                    int iy = iy0 + ky * p.dh, ix = ix0 + kx * p.dw;
                    bool in = (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
                    const T *at = src + ((long long)iy * p.iw + ix) * p.ips;
                    if (vec_in) { // a chunk never leaves its tap
                        if (in && k < p.K) {
                            dense16(at + c, 16, true, v);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] = 0;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            v[j] = in && k + j < p.K ? (int)at[c] : 0;
                            if (++c == p.ic) {
                                c = 0;
                                if (++kx == p.kw)
                                    kx = 0, ky++;
                                iy = iy0 + ky * p.dh, ix = ix0 + kx * p.dw;
                                in = (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw;
                                at = src + ((long long)iy * p.iw + ix) * p.ips;
                            }
                        }
                    }
                }
                if (sizeof(T) == 2) {
                    int hi[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) hi[j] = v[j] >> 8, sum += v[j];
                    *(uint4 *)(p.a_hi + row * p.Kp + k) = pack16(hi);
                    *(uint4 *)(p.a_lo + row * p.Kp + k) = pack16(v);
                } else {
                    *(uint4 *)(p.a_hi + row * p.Kp + k) = pack16(v);
                }
            }
        }
        if (sizeof(T) == 2) {
            for (int d = p.lanes >> 1; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            if (live && !is_b && sub == 0)
                p.row_sum[row] = sum;
        }
    }
}

} // namespace

int pack_operands(const espdl_conv_desc &d, long long row0, int rows, bool filter, const PackedOperands &o, cudaStream_t s)
{
    PackParams p;
    p.in = d.input, p.w = d.filter;
    p.a_hi = (int8_t *)o.a_hi, p.a_lo = (uint8_t *)o.a_lo, p.b_hi = (int8_t *)o.b_hi, p.b_lo = (uint8_t *)o.b_lo, p.row_sum = o.row_sum;
    p.rows = rows, p.N = filter ? d.out_c : 0, p.K = d.kh * d.kw * d.in_c, p.Kp = o.Kp, p.row0 = row0;
    p.ih = d.in_h, p.iw = d.in_w, p.ic = d.in_c, p.oh = d.out_h, p.ow = d.out_w, p.kw = d.kw;
    p.sh = d.stride_h, p.sw = d.stride_w, p.dh = d.dilation_h, p.dw = d.dilation_w, p.pt = d.pad_top, p.pl = d.pad_left;
    p.ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c;
    p.lanes = 1;
    while (p.lanes < 32 && p.lanes * 16 < p.Kp) p.lanes *= 2;
    // 36 chunks over 32 lanes are two rounds, the second nearly empty; over 8 lanes five: fewer lanes while that fills them better
    auto used = [&](int lanes) { return (p.Kp / 16 + lanes - 1) / lanes * lanes; };
    while (p.lanes > 4 && used(p.lanes / 2) * 6 < used(p.lanes) * 5) p.lanes /= 2;
    const long long groups = ((long long)p.rows + p.N + 32 / p.lanes - 1) / (32 / p.lanes);
    const unsigned blocks = (unsigned)min((groups + 7) / 8, (long long)num_sms() * 16);
    const bool window = d.kh != 1 || d.kw != 1 || d.stride_h != 1 || d.stride_w != 1 || d.pad_top || d.pad_bottom || d.pad_left || d.pad_right;
    if (d.dtype == ESPDL_DTYPE_INT16)
        launch_overlapped(window ? pack_kernel<int16_t, true> : pack_kernel<int16_t, false>, dim3(blocks), dim3(256), 0, s, p);
    else
        launch_overlapped(window ? pack_kernel<int8_t, true> : pack_kernel<int8_t, false>, dim3(blocks), dim3(256), 0, s, p);
    count_launch();
    return check_launch("pack_operands");
}

} // namespace espdl
