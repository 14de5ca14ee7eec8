// RMSNormalization and LayerNormalization over the trailing axes of an int8 / int16 tensor.
// Replaces dl::module::RMSNormalization::forward_int8 / forward_int16 with dl::base::rms_norm
// (esp-dl/dl/module/include/dl_module_rms_normalization.hpp:57-113, esp-dl/dl/base/dl_base_norm.cpp:9-38) and the
// quantized branch of dl::module::LayerNormalization::forward_template
// (esp-dl/dl/module/include/dl_module_layer_normalization.hpp:141-214).
//
// A warp owns one row.  Integer sums (the row sum, the sum of squares) are exact, so the lanes split them and combine
// with shuffles.  LayerNormalization's variance is an fp32 sum whose result depends on the order of the additions: the
// lanes compute the squared differences of 32 consecutive elements in parallel and then every lane adds the 32 values
// in element order, so the sum is the reference's sequential sum bit for bit.  Every fp32 product, sum and quotient is
// rounded on its own (no fused multiply-add), as in the reference built without contraction.
#include "rows.cuh"

#include <climits>
#include <mutex>

namespace espdl {

namespace {

struct NormParams {
    const void *in, *scale, *bias;
    void *out, *mean, *inv_std;
    int op, half_even, len;
    long long rows;
    float in_scale, out_rescale, scale_scale, bias_scale, mean_rescale, inv_std_rescale, epsilon;
    float one = 1.0f; // see add_product2
};

// math::sqrt_newton (esp-dl/dl/math/include/dl_math.hpp:83-97); the iteration ends by itself, the cap only bounds it
__device__ __forceinline__ float sqrt_newton_dev(float x)
{
    if (x == 0.f)
        return 0.f;
    float r = x;
    for (int it = 0; it < 100; it++) {
        const float last = r;
        r = __fmul_rn(__fadd_rn(last, __fdiv_rn(x, last)), 0.5f);
        if (!(fabsf(__fsub_rn(r, last)) > 0.00001f))
            break;
    }
    return r;
}

template <typename T>
__device__ __forceinline__ void store_q(T *p, long long i, int q)
{
    p[i] = (T)(sizeof(T) == 1 ? sat8(q) : sat16(q));
}

// V consecutive elements of a row as one 32-bit word: 4 int8 or 2 int16.
template <typename T>
struct Word {
    static constexpr int V = 4 / (int)sizeof(T);
    uint32_t w;
    __device__ __forceinline__ int get(int i) const
    {
        return sizeof(T) == 1 ? (int)(int8_t)(w >> (8 * i)) : (int)(int16_t)(w >> (16 * i));
    }
    __device__ __forceinline__ void set(int i, int q)
    {
        if (sizeof(T) == 1)
            w |= ((uint32_t)sat8(q) & 0xffu) << (8 * i);
        else
            w |= ((uint32_t)sat16(q) & 0xffffu) << (16 * i);
    }
};

// Rows whose length is a multiple of V and whose pointers are word aligned: every lane moves whole words.  The
// variance terms of 32 * V consecutive elements go through shared memory (one float4 / float2 per lane) and every lane
// then adds them in element order from broadcast reads, which costs a quarter of the shuffles of the scalar form.
template <typename T>
__device__ __forceinline__ void norm_row_words(const NormParams &p, const T *x, T *y, long long row, int lane, float *stage)
{
    constexpr int V = Word<T>::V;
    const int words = p.len / V;
    const uint32_t *xw = (const uint32_t *)x;
    uint32_t *yw = (uint32_t *)y;
    if (p.op == ESPDL_NORM_RMS) {
        long long ss = 0;
        for (int j = lane; j < words; j += 32) {
            Word<T> a{xw[j]};
#pragma unroll
            for (int i = 0; i < V; i++) ss += (long long)(a.get(i) * a.get(i));
        }
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float fsum = sizeof(T) == 1 ? __int2float_rn((int)ss) : __ll2float_rn(ss);
        const float mean_sq = __fdiv_rn(__fmul_rn(fsum, __fmul_rn(p.in_scale, p.in_scale)), __int2float_rn(p.len));
        float rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, p.epsilon)));
        rms = __fmul_rn(rms, __fmul_rn(p.in_scale, p.out_rescale));
        const float *sc = (const float *)p.scale;
        const bool sc_vec = ((uintptr_t)sc % (4 * V)) == 0;
        for (int j = lane; j < words; j += 32) {
            Word<T> a{xw[j]}, r{0u};
            float s4[V];
            if (sc_vec && V == 4) {
                const float4 t = *(const float4 *)(sc + j * V);
                s4[0] = t.x, s4[1] = t.y, s4[V - 2] = t.z, s4[V - 1] = t.w;
            } else if (sc_vec) {
                const float2 t = *(const float2 *)(sc + j * V);
                s4[0] = t.x, s4[1] = t.y;
            } else {
#pragma unroll
                for (int i = 0; i < V; i++) s4[i] = sc[j * V + i];
            }
#pragma unroll
            for (int i = 0; i < V; i++) r.set(i, fround(__fmul_rn(__fmul_rn(__int2float_rn(a.get(i)), rms), s4[i]), p.half_even));
            yw[j] = r.w;
        }
        return;
    }
    int sum = 0;
    for (int j = lane; j < words; j += 32) {
        Word<T> a{xw[j]};
#pragma unroll
        for (int i = 0; i < V; i++) sum += a.get(i);
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    float mean = (float)((double)sum * 1.0 / (double)p.len);
    if (p.mean && lane == 0)
        store_q((T *)p.mean, row, fround(__fmul_rn(__fmul_rn(mean, p.mean_rescale), p.in_scale), p.half_even));
    float var = 0.f;
    for (int base = 0; base < words; base += 32) {
        const int j = base + lane;
        float d2[V];
#pragma unroll
        for (int i = 0; i < V; i++) d2[i] = 0.f;
        if (j < words) {
            Word<T> a{xw[j]};
#pragma unroll
            for (int i = 0; i < V; i++) {
                const float d = __fsub_rn(__int2float_rn(a.get(i)), mean);
                d2[i] = __fmul_rn(d, d);
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < V; i++) stage[lane * V + i] = d2[i];
        __syncwarp();
        const int n = min(32, words - base) * V;
        for (int k = 0; k < n; k += V) { // one broadcast read of V terms, added in element order
            if (V == 4) {
                const float4 t = *(const float4 *)(stage + k);
                var = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(var, t.x), t.y), t.z), t.w);
            } else {
                const float2 t = *(const float2 *)(stage + k);
                var = __fadd_rn(__fadd_rn(var, t.x), t.y);
            }
        }
    }
    mean = __fmul_rn(mean, p.in_scale);
    var = __fmul_rn(var, __fmul_rn(p.in_scale, p.in_scale));
    var = __fdiv_rn(var, __int2float_rn(p.len));
    const float inv_std = __fdiv_rn(1.0f, sqrt_newton_dev(__fadd_rn(var, p.epsilon)));
    if (p.inv_std && lane == 0)
        store_q((T *)p.inv_std, row, fround(__fmul_rn(inv_std, p.inv_std_rescale), p.half_even));
    const T *sc = (const T *)p.scale, *bi = (const T *)p.bias;
    for (int j = lane; j < words; j += 32) {
        Word<T> a{xw[j]}, r{0u};
#pragma unroll
        for (int i = 0; i < V; i++) {
            const int e = j * V + i;
            const float xv = __fmul_rn(__int2float_rn(a.get(i)), p.in_scale);
            const float normalized = __fmul_rn(__fsub_rn(xv, mean), inv_std);
            const float sv = sc ? __fmul_rn(__int2float_rn((int)sc[e]), p.scale_scale) : 1.0f;
            const float bv = bi ? __fmul_rn(__int2float_rn((int)bi[e]), p.bias_scale) : 0.0f;
            r.set(i, fround(__fmul_rn(__fadd_rn(__fmul_rn(normalized, sv), bv), p.out_rescale), p.half_even));
        }
        yw[j] = r.w;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) norm_kernel(NormParams p, int early)
{
    if (early)
        grid_dep_launch();
    grid_dep_wait();
    __shared__ __align__(16) float stage_all[8][128];
    const bool words_ok = p.len % Word<T>::V == 0 && ((uintptr_t)p.in % 4) == 0 && ((uintptr_t)p.out % 4) == 0;
    const int lane = threadIdx.x & 31;
    const long long warp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5, warps = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = warp; row < p.rows; row += warps) {
        const T *x = (const T *)p.in + row * p.len;
        T *y = (T *)p.out + row * p.len;
        if (words_ok) {
            norm_row_words<T>(p, x, y, row, lane, stage_all[threadIdx.x >> 5]);
            continue;
        }
        if (p.op == ESPDL_NORM_RMS) {
            // int8: int32 sum of squares (as dl::base::reduce_l2 returns it), int16: int64
            long long ss = 0;
            for (int j = lane; j < p.len; j += 32) ss += (long long)((int)x[j] * (int)x[j]);
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float fsum = sizeof(T) == 1 ? __int2float_rn((int)ss) : __ll2float_rn(ss);
            const float mean_sq = __fdiv_rn(__fmul_rn(fsum, __fmul_rn(p.in_scale, p.in_scale)), __int2float_rn(p.len));
            float rms = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean_sq, p.epsilon)));
            rms = __fmul_rn(rms, __fmul_rn(p.in_scale, p.out_rescale));
            const float *sc = (const float *)p.scale;
            for (int j = lane; j < p.len; j += 32)
                store_q(y, j, fround(__fmul_rn(__fmul_rn(__int2float_rn((int)x[j]), rms), sc[j]), p.half_even));
        } else {
            int sum = 0;
            for (int j = lane; j < p.len; j += 32) sum += (int)x[j];
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            float mean = (float)((double)sum * 1.0 / (double)p.len);
            if (p.mean && lane == 0)
                store_q((T *)p.mean, row, fround(__fmul_rn(__fmul_rn(mean, p.mean_rescale), p.in_scale), p.half_even));
            float var = 0.f;
            for (int base = 0; base < p.len; base += 32) {
                const int j = base + lane;
                float d2 = 0.f;
                if (j < p.len) {
                    const float d = __fsub_rn(__int2float_rn((int)x[j]), mean);
                    d2 = __fmul_rn(d, d);
                }
                const int n = min(32, p.len - base);
                for (int k = 0; k < n; k++) var = __fadd_rn(var, __shfl_sync(0xffffffffu, d2, k));
            }
            mean = __fmul_rn(mean, p.in_scale);
            var = __fmul_rn(var, __fmul_rn(p.in_scale, p.in_scale));
            var = __fdiv_rn(var, __int2float_rn(p.len));
            const float inv_std = __fdiv_rn(1.0f, sqrt_newton_dev(__fadd_rn(var, p.epsilon)));
            if (p.inv_std && lane == 0)
                store_q((T *)p.inv_std, row, fround(__fmul_rn(inv_std, p.inv_std_rescale), p.half_even));
            const T *sc = (const T *)p.scale, *bi = (const T *)p.bias;
            for (int j = lane; j < p.len; j += 32) {
                const float xv = __fmul_rn(__int2float_rn((int)x[j]), p.in_scale);
                const float normalized = __fmul_rn(__fsub_rn(xv, mean), inv_std);
                const float sv = sc ? __fmul_rn(__int2float_rn((int)sc[j]), p.scale_scale) : 1.0f;
                const float bv = bi ? __fmul_rn(__int2float_rn((int)bi[j]), p.bias_scale) : 0.0f;
                const float r = __fadd_rn(__fmul_rn(normalized, sv), bv);
                store_q(y, j, fround(__fmul_rn(r, p.out_rescale), p.half_even));
            }
        }
    }
}

// A code to a float without a conversion instruction (these run at an eighth of the rate of the others, and the results below need one an
// element already).  A code with its sign bit flipped, put under the exponent of 2^23, is 2^23 + 128 + x (32768 for int16); that and x are
// exact.
template <typename T>
__device__ __forceinline__ float code_to_float(uint32_t flipped, int k)
{
    if (sizeof(T) == 1)
        return __fsub_rn(__uint_as_float(__byte_perm(flipped, 0x4b000000u, 0x7440u | (uint32_t)k)), 8388736.f);
    return __fsub_rn(__uint_as_float(__byte_perm(flipped, 0x4b000000u, k ? 0x7432u : 0x7410u)), 8421376.f);
}

// Two floats of one instruction: every operation rounds each as the scalar one does, at half the issue slots.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pair(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void split(F2 x, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// a + b where a is a product: with a factor of one that the compiler cannot see, because it contracts packed products and sums, whatever rounding they
// name (20 of 77 M results differed).
__device__ __forceinline__ F2 add_product2(F2 a, F2 b, F2 one) { return fma2(a, one, b); }

// Codes k and k + 1 of a word (see code_to_float).
template <typename T>
__device__ __forceinline__ F2 codes_to_floats(uint32_t flipped, int k)
{
    if (sizeof(T) == 1)
        return add2(pair(__uint_as_float(__byte_perm(flipped, 0x4b000000u, 0x7440u | (uint32_t)k)), __uint_as_float(__byte_perm(flipped, 0x4b000000u, 0x7441u + (uint32_t)k))),
                    pair(-8388736.f, -8388736.f));
    return add2(pair(__uint_as_float(__byte_perm(flipped, 0x4b000000u, 0x7410u)), __uint_as_float(__byte_perm(flipped, 0x4b000000u, 0x7432u))), pair(-8421376.f, -8421376.f));
}

// The squared differences of a 16-byte unit of codes from the row's mean.
template <typename T>
__device__ __forceinline__ void unit_squares(uint4 w, F2 minus_mean, float (&d2)[16 / sizeof(T)])
{
    constexpr int V = Word<T>::V;
    constexpr uint32_t FLIP = sizeof(T) == 1 ? 0x80808080u : 0x80008000u;
    const uint32_t x[4] = {w.x ^ FLIP, w.y ^ FLIP, w.z ^ FLIP, w.w ^ FLIP};
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int k = 0; k < V; k += 2) {
            const F2 d = add2(codes_to_floats<T>(x[j], k), minus_mean);
            split(mul2(d, d), d2[j * V + k], d2[j * V + k + 1]);
        }
}

// The ordered sum of a row's squared differences, `units` 16-byte units: the next unit's squares are made beside the chain of this one's additions, which
// alone is four cycles an element (100352 rows of 768: 57.3 us pair by pair, 54.9).  Its registers leave four blocks an SM, see launch_layer_rows.
template <typename T>
__device__ __forceinline__ float ordered_squares(const uint4 *row, int units, float mean)
{
    const F2 minus_mean = pair(-mean, -mean);
    float a[16 / sizeof(T)], b[16 / sizeof(T)], var = 0.f;
    unit_squares<T>(row[0], minus_mean, a);
    int i = 1;
    for (; i + 1 < units; i += 2) {
        const uint4 wb = row[i], wa = row[i + 1];
        unit_squares<T>(wb, minus_mean, b);
#pragma unroll
        for (int k = 0; k < 16 / (int)sizeof(T); k++) var = __fadd_rn(var, a[k]);
        unit_squares<T>(wa, minus_mean, a);
#pragma unroll
        for (int k = 0; k < 16 / (int)sizeof(T); k++) var = __fadd_rn(var, b[k]);
    }
    if (i < units)
        unit_squares<T>(row[i], minus_mean, b);
#pragma unroll
    for (int k = 0; k < 16 / (int)sizeof(T); k++) var = __fadd_rn(var, a[k]);
    if (i < units) {
#pragma unroll
        for (int k = 0; k < 16 / (int)sizeof(T); k++) var = __fadd_rn(var, b[k]);
    }
    return var;
}

// One word of results from one of codes (sign bits flipped): sv, bv are its columns' scale and bias.
template <typename T, bool EVEN>
__device__ __forceinline__ uint32_t norm_word(uint32_t codes, F2 minus_mean, F2 inv_std, const F2 *sv, const F2 *bv, F2 in_scale, F2 rescale, F2 half, F2 one)
{
    constexpr int V = Word<T>::V;
    int q[V];
#pragma unroll
    for (int k = 0; k < V; k += 2) {
        // products with a power of two are exact, so a fused multiply-add there rounds as the separate operations do
        const F2 d = fma2(codes_to_floats<T>(codes, k), in_scale, minus_mean);
        const F2 y = add_product2(mul2(mul2(d, inv_std), sv[k / 2]), bv[k / 2], one);
        float a, b;
        split(EVEN ? mul2(y, rescale) : fma2(y, rescale, half), a, b);
        q[k] = EVEN ? __float2int_rn(a) : __float2int_rd(a), q[k + 1] = EVEN ? __float2int_rn(b) : __float2int_rd(b);
    }
    uint32_t w;
    if (V == 4) {
        uint32_t hi;
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(q[V - 1]), "r"(q[V - 2]));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(q[1]), "r"(q[0]), "r"(hi));
    } else {
        asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(w) : "r"(q[1]), "r"(q[0]));
    }
    return w;
}

// LayerNormalization with the rows of a block side by side in shared memory.  The variance is an ordered fp32 sum, so a row
// costs `len` dependent additions whoever does them; a warp per row made all 32 lanes do the same ones.  Here a thread walks one
// row (row pitch an odd number of words: thread r reading word i of row r meets no bank conflict), 32 rows of a warp side by
// side, and the normalising pass gives every thread fixed columns, whose scale and bias stay in registers while it goes
// down the rows.  Bound by instruction issue (100352 rows of 768: 101 -> 80 us with asynchronous copies in, codes to floats without conversions, all
// threads in the normalising pass and as many blocks as there are groups of rows; 80 -> 69 with two elements an instruction).
// Rows of whole aligned 16-byte units have a pitch of an odd number of those: copies and a row's reads are of 16 bytes then, a quarter warp's
// without bank conflicts as well (69 -> 63 us).  A thread copies down its columns and normalises two (int16: four) words of a row at a time, scale and bias are
// converted as words of codes: what is done for a word besides its arithmetic was a third of all instructions (63.6 -> 57.3 us; int16 114 -> 92, 200000 rows of
// 64 21.3 -> 12.8).  Copying, summing and normalising take 9, 17 and 31 us of these 57, hardly beside each other although blocks are independent; a warp that
// copies and sums the next rows while eight normalise these was slower (80: the one warp's chain of additions is in the way).
// WORDS: rows are whole aligned words in global memory; otherwise the block's rows, one contiguous run of bytes, are dealt out to
// and collected from the padded rows byte by byte.  UNITS: rows of whole 16-byte units, 2: their squares made ahead, 3: results that begin at any word; forms of their own, because what a block fetches of a kernel's code
// counts in the shortest launches (6250 rows of 16: 3.77 us, 3.99 with both forms in one kernel).
template <typename T, bool WORDS, bool EVEN, int UNITS>
__global__ void __launch_bounds__(256) layer_rows_kernel(NormParams p, int R, int pitch, int across, int across16, int early)
{
    if (early)
        grid_dep_launch();
    grid_dep_wait();
    constexpr int V = Word<T>::V;
    constexpr uint32_t FLIP = sizeof(T) == 1 ? 0x80808080u : 0x80008000u;
    extern __shared__ __align__(16) uint32_t rows_s[]; // R x pitch words, then per row {mean, 1 / std}
    float2 *stats = (float2 *)(rows_s + (size_t)R * pitch + ((R * pitch) & 1));
    const int words = (p.len + V - 1) / V, row_bytes = p.len * (int)sizeof(T);
    const long long groups = (p.rows + R - 1) / R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (long long g = blockIdx.x; g < groups; g += gridDim.x) {
        const long long r0 = g * R;
        const int nr = (int)min((long long)R, p.rows - r0);
        const uint32_t *src = (const uint32_t *)((const T *)p.in + r0 * p.len); // R is a multiple of 4: word aligned
        const int total = nr * row_bytes;
        __syncthreads();
        if (WORDS) {
            // asynchronous copies: all of the block's rows in flight at once (with loads through registers a block spent half its time here)
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(rows_s);
            if (UNITS) { // a thread copies down its columns
                const int columns = words / 4, wide = min(across16, columns), down = 256 / wide, first = threadIdx.x / wide;
                if (first < down)
                    for (int c = threadIdx.x % wide; c < columns; c += wide) {
                        uint32_t at = to + 4u * (uint32_t)(first * pitch + 4 * c);
                        const uint32_t *from = src + (long long)first * words + 4 * c;
                        for (int rr = first; rr < nr; rr += down, at += 4u * (uint32_t)(down * pitch), from += (long long)down * words)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at), "l"(from) : "memory");
                    }
            } else
                for (int rr = warp; rr < nr; rr += 8)
                    for (int i = lane; i < words; i += 32)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + 4u * (uint32_t)(rr * pitch + i)), "l"(src + (long long)rr * words + i) : "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            deal_rows<T>(src, total, row_bytes, rows_s, pitch);
        }
        __syncthreads();
        const int own = threadIdx.x;
        if (own < nr) {
            const uint32_t *row = rows_s + own * pitch;
            const int full = p.len / V;
            int sum = 0;
            auto add_word = [&](uint32_t w) {
                Word<T> a{w};
                if (V == 4) {
                    sum = __dp4a((int)a.w, 0x01010101, sum);
                } else {
#pragma unroll
                    for (int k = 0; k < V; k++) sum += a.get(k);
                }
            };
            if (UNITS)
                for (int i = 0; i < full; i += 4) {
                    const uint4 w = *(const uint4 *)(row + i);
                    add_word(w.x), add_word(w.y), add_word(w.z), add_word(w.w);
                }
            else
                for (int i = 0; i < full; i++) add_word(row[i]);
            Word<T> last{full < words ? row[full] : 0u};
#pragma unroll
            for (int k = 0; k < V; k++)
                if (full * V + k < p.len)
                    sum += last.get(k);
            float mean = (float)((double)sum * 1.0 / (double)p.len);
            float var = 0.f;
            auto add = [&](float x) {
                const float d = __fsub_rn(x, mean);
                var = __fadd_rn(var, __fmul_rn(d, d));
            };
            const F2 minus_mean = pair(-mean, -mean);
            auto add_squares = [&](uint32_t w) {
                w ^= FLIP;
#pragma unroll
                for (int k = 0; k < V; k += 2) {
                    const F2 d = add2(codes_to_floats<T>(w, k), minus_mean);
                    float a, b;
                    split(mul2(d, d), a, b);
                    var = __fadd_rn(__fadd_rn(var, a), b);
                }
            };
            if (UNITS == 2)
                var = ordered_squares<T>((const uint4 *)row, full / 4, mean);
            else if (UNITS)
                for (int i = 0; i < full; i += 4) {
                    const uint4 w = *(const uint4 *)(row + i);
                    add_squares(w.x), add_squares(w.y), add_squares(w.z), add_squares(w.w);
                }
            else
#pragma unroll 4
                for (int i = 0; i < full; i++) add_squares(row[i]);
#pragma unroll
            for (int k = 0; k < V; k++)
                if (full * V + k < p.len)
                    add(code_to_float<T>(last.w ^ FLIP, k));
            const long long out_row = r0 + own;
            if (p.mean)
                store_q((T *)p.mean, out_row, fround(__fmul_rn(__fmul_rn(mean, p.mean_rescale), p.in_scale), p.half_even));
            mean = __fmul_rn(mean, p.in_scale);
            var = __fmul_rn(var, __fmul_rn(p.in_scale, p.in_scale));
            var = __fdiv_rn(var, __int2float_rn(p.len));
            const float inv_std = __fdiv_rn(1.0f, sqrt_newton_dev(__fadd_rn(var, p.epsilon)));
            if (p.inv_std)
                store_q((T *)p.inv_std, out_row, fround(__fmul_rn(inv_std, p.inv_std_rescale), p.half_even));
            stats[own] = make_float2(mean, inv_std);
        }
        __syncthreads();
        const T *sc = (const T *)p.scale, *bi = (const T *)p.bias;
        uint32_t *dst = (uint32_t *)((T *)p.out + r0 * p.len);
        const F2 in_scale = pair(p.in_scale, p.in_scale), rescale = pair(p.out_rescale, p.out_rescale), half = pair(0.5f, 0.5f), one = pair(p.one, p.one);
        // scale and bias of a thread's columns, from element e on
        auto constants = [&](int e, F2 &s, F2 &b) {
            float s2[2], b2[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int at = min(e + h, p.len - 1);
                s2[h] = sc ? __fmul_rn(__int2float_rn((int)sc[at]), p.scale_scale) : 1.0f;
                b2[h] = bi ? __fmul_rn(__int2float_rn((int)bi[at]), p.bias_scale) : 0.0f;
            }
            s = pair(s2[0], s2[1]), b = pair(b2[0], b2[1]);
        };
        auto word = [&](uint32_t codes, F2 minus_mean, F2 inv_std, const F2 *sv, const F2 *bv) {
            return norm_word<T, EVEN>(codes, minus_mean, inv_std, sv, bv, in_scale, rescale, half, one);
        };
        // W words of a row a thread: a whole 16-byte unit where rows are made of these, so that addresses, bounds and the row's figures cost a quarter as much
        constexpr int W = UNITS ? (sizeof(T) == 1 ? 2 : 4) : 1;
        const int columns = words / W, down = 256 / across; // threads along a row, rows at a time
        const int first_row = threadIdx.x / across;
        for (int c = threadIdx.x % across; c < columns && first_row < down; c += across) {
            F2 sv[W * V / 2], bv[W * V / 2];
            if (W * sizeof(uint32_t) % 8 == 0 && sc && bi && (((uintptr_t)sc | (uintptr_t)bi) & 15) == 0) { // whole words of codes, as the rows' own
                const F2 s_scale = pair(p.scale_scale, p.scale_scale), b_scale = pair(p.bias_scale, p.bias_scale);
#pragma unroll
                for (int i = 0; i < W; i++) {
                    const uint32_t sw = ((const uint32_t *)sc)[c * W + i] ^ FLIP, bw = ((const uint32_t *)bi)[c * W + i] ^ FLIP;
#pragma unroll
                    for (int k = 0; k < V; k += 2) {
                        sv[(i * V + k) / 2] = mul2(codes_to_floats<T>(sw, k), s_scale);
                        bv[(i * V + k) / 2] = mul2(codes_to_floats<T>(bw, k), b_scale);
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < W * V; k += 2) constants(c * W * V + k, sv[k / 2], bv[k / 2]);
            }
            const uint32_t *from = rows_s + first_row * pitch + c * W;
            uint32_t *to = dst + (long long)first_row * words + c * W;
#pragma unroll(W == 1 ? 2 : 1)
            for (int rr = first_row; rr < nr; rr += down, from += down * pitch, to += (long long)down * words) {
                const float2 st = stats[rr];
                const F2 minus_mean = pair(-st.x, -st.x), inv_std = pair(st.y, st.y);
                if (W == 2) {
                    const uint2 x = *(const uint2 *)from;
                    uint2 y;
                    y.x = word(x.x ^ FLIP, minus_mean, inv_std, sv, bv);
                    y.y = word(x.y ^ FLIP, minus_mean, inv_std, sv + V / 2, bv + V / 2);
                    if (UNITS == 3)
                        to[0] = y.x, to[1] = y.y;
                    else
                        *(uint2 *)to = y;
                } else if (W == 4) {
                    const uint4 x = *(const uint4 *)from;
                    uint4 y;
                    y.x = word(x.x ^ FLIP, minus_mean, inv_std, sv, bv);
                    y.y = word(x.y ^ FLIP, minus_mean, inv_std, sv + V / 2, bv + V / 2);
                    y.z = word(x.z ^ FLIP, minus_mean, inv_std, sv + V, bv + V);
                    y.w = word(x.w ^ FLIP, minus_mean, inv_std, sv + 3 * V / 2, bv + 3 * V / 2);
                    if (UNITS == 3)
                        to[0] = y.x, to[1] = y.y, to[2] = y.z, to[3] = y.w;
                    else
                        *(uint4 *)to = y;
                } else {
                    const uint32_t y = word(*from ^ FLIP, minus_mean, inv_std, sv, bv);
                    if (WORDS)
                        *to = y;
                    else
                        rows_s[rr * pitch + c] = y;
                }
            }
        }
        if (!WORDS) {
            __syncthreads();
            collect_rows<T>(dst, total, row_bytes, rows_s, pitch);
        }
    }
}

template <typename T>
int launch_layer_rows(const NormParams &p, int R, int pitch, cudaStream_t s)
{
    const bool words = p.len % Word<T>::V == 0;
    const size_t smem = ((size_t)R * pitch + 1) * 4 + (size_t)R * sizeof(float2);
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] {
        for (auto k : {layer_rows_kernel<T, true, false, 0>, layer_rows_kernel<T, true, true, 0>, layer_rows_kernel<T, false, false, 0>, layer_rows_kernel<T, false, true, 0>,
                       layer_rows_kernel<T, true, false, 1>, layer_rows_kernel<T, true, true, 1>, layer_rows_kernel<T, true, false, 2>, layer_rows_kernel<T, true, true, 2>,
                       layer_rows_kernel<T, true, false, 3>, layer_rows_kernel<T, true, true, 3>})
            if (attr_err == cudaSuccess)
                attr_err = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
    });
    if (attr_err != cudaSuccess)
        return set_cuda_error(attr_err, "cudaFuncSetAttribute(layer_rows_kernel)");
    const long long groups = (p.rows + R - 1) / R;
    // Squares ahead of their sum where the rows leave four blocks an SM or the launch has no more (7812 rows of 1024 11.3 us, 10.8 so); beyond that the blocks that
    // its registers cost are worth more: us ahead / not, 58593 rows of 1024 48.9 / 45.6, 104166 of 576 44.4 / 42.7, int16 58593 of 512 38.9 / 34.7, 234375 of
    // 128 29.0 / 27.9.  int8 at five blocks is even (156250 of 384 40.2 / 40.4, 187500 of 320 39.4 / 40.6).
    const int blocks = (int)(227 * 1024 / (smem + 1024));
    const bool ahead = groups <= 4ll * num_sms() || blocks < (sizeof(T) == 1 ? 6 : 5);
    const auto kernel = pitch % 4 == 0 ? ((uintptr_t)p.out % 16 != 0 ? (p.half_even ? layer_rows_kernel<T, true, true, 3> : layer_rows_kernel<T, true, false, 3>)
                                              : ahead ? (p.half_even ? layer_rows_kernel<T, true, true, 2> : layer_rows_kernel<T, true, false, 2>)
                                                      : (p.half_even ? layer_rows_kernel<T, true, true, 1> : layer_rows_kernel<T, true, false, 1>))
        : words                        ? (p.half_even ? layer_rows_kernel<T, true, true, 0> : layer_rows_kernel<T, true, false, 0>)
                                       : (p.half_even ? layer_rows_kernel<T, false, true, 0> : layer_rows_kernel<T, false, false, 0>);
    // Threads along a row: all of its columns, or a part of them at a time where that leaves fewer threads without work; a pass converts the constants of its
    // columns first, about two rows' work (8370 rows of 264, whose 66 words are three rows at once or seven in two passes: 6.8 us in one, 7.9 in two).
    const int columns = (p.len + Word<T>::V - 1) / Word<T>::V / (pitch % 4 != 0 ? 1 : sizeof(T) == 1 ? 2 : 4);
    const auto spread = [R](int columns, int first) {
        int across = 1, least = INT_MAX;
        for (int passes = (columns + 255) / 256; passes <= 8; passes++) {
            const int a = (columns + passes - 1) / passes, down = 256 / a, cost = passes * (first + (R + down - 1) / down);
            if (cost < least)
                least = cost, across = a;
        }
        return across;
    };
    const int across = spread(columns, 2), across16 = spread(max(1, (p.len + Word<T>::V - 1) / Word<T>::V / 4), 0); // (the units that are copied)
    launch_mover(kernel, dim3((unsigned)min(groups, (long long)num_sms() * 64)), dim3(256), smem, s, p, R, pitch, across, across16);
    count_launch();
    return check_launch("layer norm");
}

} // namespace

} // namespace espdl

using namespace espdl;

extern "C" int espdl_b200_norm(const espdl_norm_desc *d, void *stream)
{
    if (!d || !d->input || !d->output || d->rows < 0 || d->len <= 0)
        return ESPDL_ERR_INVALID_ARG;
    if (d->op != ESPDL_NORM_RMS && d->op != ESPDL_NORM_LAYER && d->op != ESPDL_NORM_LP)
        return ESPDL_ERR_INVALID_ARG;
    if (d->op == ESPDL_NORM_RMS && !d->scale)
        return ESPDL_ERR_INVALID_ARG;
    if (d->dtype != ESPDL_DTYPE_INT8 && d->dtype != ESPDL_DTYPE_INT16)
        return ESPDL_ERR_UNSUPPORTED;
    for (int e : {d->in_exponent, d->out_exponent, d->scale_exponent, d->bias_exponent, d->mean_exponent, d->inv_std_dev_exponent})
        if (e > 30 || e < -30)
            return ESPDL_ERR_INVALID_ARG;
    if (d->rows == 0)
        return ESPDL_OK;
    if (d->op == ESPDL_NORM_LP)
        return lp_norm_op(*d, (cudaStream_t)stream);
    NormParams p;
    p.in = d->input, p.out = d->output, p.scale = d->scale, p.bias = d->bias, p.mean = d->mean, p.inv_std = d->inv_std_dev;
    p.op = d->op, p.half_even = d->round_mode == ESPDL_ROUND_HALF_EVEN, p.len = d->len, p.rows = d->rows;
    p.in_scale = dl_scale(d->in_exponent), p.out_rescale = dl_rescale(d->out_exponent);
    p.scale_scale = dl_scale(d->scale_exponent), p.bias_scale = dl_scale(d->bias_exponent);
    p.mean_rescale = dl_rescale(d->mean_exponent), p.inv_std_rescale = dl_rescale(d->inv_std_dev_exponent);
    p.epsilon = d->epsilon;
    if (d->op == ESPDL_NORM_LAYER && ((uintptr_t)d->input % 4) == 0 && ((uintptr_t)d->output % 4) == 0) {
        // rows a block: 48 KB of them (four blocks an SM keep eight warps at their rows), fewer where that leaves SMs without a block
        const int V = d->dtype == ESPDL_DTYPE_INT8 ? 4 : 2, words = (d->len + V - 1) / V;
        const bool units = d->len % (4 * V) == 0 && ((uintptr_t)d->input % 16) == 0;
        const int pitch = units ? 4 * (words / 4 | 1) : words | 1;
        const long long fit = (50 * 1024) / ((long long)pitch * 4 + 8), share = (d->rows + num_sms() - 1) / num_sms();
        const int R = (int)min(min(256ll, max(fit, (96 * 1024) / ((long long)pitch * 4 + 8) >= 32 ? 32ll : 0ll)), max(32ll, share)) / 32 * 32;
        // long rows: a block of 32 takes its time whatever else there is (11 us for 768 int8, 18 int16), a warp per row is faster below some waves of rows
        const long long few = d->len <= 128 ? 256 : (long long)num_sms() * (V == 4 ? 24 : 32);
        if (R >= 32 && d->rows >= few)
            return d->dtype == ESPDL_DTYPE_INT8 ? launch_layer_rows<int8_t>(p, R, pitch, (cudaStream_t)stream) : launch_layer_rows<int16_t>(p, R, pitch, (cudaStream_t)stream);
    }
    const long long blocks = (d->rows + 7) / 8; // eight rows (warps) per block
    const unsigned grid = (unsigned)min(blocks, (long long)num_sms() * 8);
    if (d->dtype == ESPDL_DTYPE_INT8)
        launch_mover(norm_kernel<int8_t>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, p);
    else
        launch_mover(norm_kernel<int16_t>, dim3(grid), dim3(256), 0, (cudaStream_t)stream, p);
    count_launch();
    return check_launch("norm");
}
