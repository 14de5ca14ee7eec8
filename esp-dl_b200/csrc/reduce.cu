// Reductions over any set of axes of an int8 / int16 tensor: ReduceMean, ReduceSum, ReduceMax, ReduceMin, ReduceL1,
// ReduceSumSquare, ReduceL2 (dl_module_reduce_l1.hpp, dl_module_reduce_sum_square.hpp, dl_module_reduce_l2.hpp), ReduceProd,
// ReduceLogSum, ReduceLogSumExp (dl_module_reduce_prod.hpp, dl_module_reduce_log_sum.hpp, dl_module_reduce_log_sum_exp.hpp).
// Replaces dl::module::ReduceBase::forward_template and the reduce functions of the modules built on it
// (esp-dl/dl/module/include/dl_module_reduce_base.hpp:121-262, dl_module_reduce_mean.hpp:17-45, dl_module_reduce_sum.hpp:
// 17-42), and average pools over whole images.  Two kernels.  channel_reduce_kernel: one run of reduced axes between kept ones (the
// usual spatial mean of an NHWC map) from 2 KB an image on, integer accumulations; pixels shared by the threads of a block and the
// blocks of a cluster.  reduce_kernel: everything else, a thread owns one output element and walks the reduced axes.  Integer sums
// are exact, so the order does not matter; the mean's fp32 expression is evaluated in the reference's order.  The floating-point
// accumulations (the product, the sum of exponentials) are not associative: the walk visits the reduced elements in the reference's
// order (row-major over the reduced axes), one thread per output.
#include "common.cuh"
#include "reduce_plan.cuh"

#include <climits>
#include <cooperative_groups.h>
#include <cstring>
#include <type_traits>

namespace espdl {

namespace {

struct ReduceParams {
    const void *in;
    void *out;
    int op, half_even, e_in, e_out;
    int nk, nr;            // kept / reduced axes
    int ksize[6], rsize[6];
    long long kstride[6], rstride[6];
    long long outputs, count;
    const float *exp_table;
    float scale; // AVERAGE_POOL: 2^e_in / area * 2^-e_out as the reference forms it
};

constexpr int AVERAGE_POOL = 100; // an average pool over the whole image, beside the espdl_reduce_op_t values

// tool::round of a float that may be no int32 (NaN, infinity): such a value converts to the minimum on x86
__device__ __forceinline__ long long fround_x86(float v, int half_even)
{
    if (!(fabsf(v) < 2147483520.f))
        return (long long)INT_MIN;
    return fround(v, half_even);
}

// The output code of one integer accumulation (every operator but the product and the sum of exponentials).
template <typename ACC>
__device__ __forceinline__ long long finish_integer(const ReduceParams &p, ACC acc)
{
    if (p.op == ESPDL_REDUCE_MEAN) {
        // tool::round(tmp * input_scale / count * output_scale), all in fp32
        float f = __fmul_rn((float)acc, dl_scale(p.e_in));
        f = __fdiv_rn(f, (float)(unsigned long long)p.count);
        f = __fmul_rn(f, dl_rescale(p.e_out));
        return fround(f, p.half_even);
    }
    if (p.op == AVERAGE_POOL) // int8: the reference sums in int32, int16: in int64; both convert the sum to fp32
        return fround_half_up(__fmul_rn(sizeof(ACC) == 4 ? __int2float_rn((int)acc) : __ll2float_rn((long long)acc), p.scale));
    if (p.op == ESPDL_REDUCE_L2) {
        // math::sqrt_newton (dl_math.hpp:83-97): r = (r + x / r) * 0.5 until |r - last| <= 1e-5, every step rounded to fp32
        const float x = __fmul_rn(sizeof(ACC) == 4 ? __int2float_rn((int)acc) : __ll2float_rn((long long)acc), dl_scale(2 * p.e_in));
        float r = x;
        if (x != 0.f) {
            for (int it = 0; it < 100; it++) {
                const float last = r;
                r = __fmul_rn(__fadd_rn(last, __fdiv_rn(x, last)), 0.5f);
                if (!(fabsf(__fsub_rn(r, last)) > 0.00001f))
                    break;
            }
        }
        return fround(__fmul_rn(r, dl_rescale(p.e_out)), p.half_even);
    }
    if (p.op == ESPDL_REDUCE_LOG_SUM) {
        // static_cast<float>(sum * input_scale): the integer sum becomes a float before the multiplication
        const float sumf = sizeof(ACC) == 4 ? __int2float_rn((int)acc) : __ll2float_rn((long long)acc);
        return fround_x86(__fmul_rn(logf(__fmul_rn(sumf, dl_scale(p.e_in))), dl_rescale(p.e_out)), p.half_even);
    }
    if (p.op == ESPDL_REDUCE_SUM || p.op == ESPDL_REDUCE_L1 || p.op == ESPDL_REDUCE_SUM_SQUARE) {
        const int shift = max(-62, min(62, p.e_out - (p.op == ESPDL_REDUCE_SUM_SQUARE ? 2 * p.e_in : p.e_in)));
        return sizeof(ACC) == 4 ? (long long)shift_round32((int32_t)acc, max(-31, min(32, shift)), p.half_even)
                                : shift_round64((long long)acc, shift, p.half_even);
    }
    return (long long)acc;
}

// How an element enters an integer accumulation.
enum Fold { FOLD_SUM, FOLD_MAX, FOLD_MIN, FOLD_ABS, FOLD_SQUARE };

__host__ __device__ __forceinline__ Fold fold_of(int op)
{
    switch (op) {
    case ESPDL_REDUCE_MAX: return FOLD_MAX;
    case ESPDL_REDUCE_MIN: return FOLD_MIN;
    case ESPDL_REDUCE_L1: return FOLD_ABS;
    case ESPDL_REDUCE_SUM_SQUARE:
    case ESPDL_REDUCE_L2: return FOLD_SQUARE;
    default: return FOLD_SUM;
    }
}

template <typename ACC>
__device__ __forceinline__ ACC fold_element(Fold f, ACC acc, ACC v)
{
    if (f == FOLD_MAX)
        return acc > v ? acc : v;
    if (f == FOLD_MIN)
        return acc < v ? acc : v;
    if (f == FOLD_ABS)
        return acc + (v < 0 ? -v : v);
    if (f == FOLD_SQUARE)
        return acc + (ACC)((int)v * (int)v);
    return acc + v;
}

template <typename ACC>
__device__ __forceinline__ ACC fold_partial(Fold f, ACC a, ACC b)
{
    return f == FOLD_MAX ? (a > b ? a : b) : (f == FOLD_MIN ? (a < b ? a : b) : a + b);
}

template <typename T, typename ACC>
__device__ __forceinline__ ACC fold_start(Fold f)
{
    return f == FOLD_MAX ? (ACC)(sizeof(T) == 1 ? -128 : -32768) : (f == FOLD_MIN ? (ACC)(sizeof(T) == 1 ? 127 : 32767) : (ACC)0);
}

template <typename T, typename ACC>
__global__ void __launch_bounds__(256) reduce_kernel(ReduceParams p, int early)
{
    if (early)
        grid_dep_launch();
    grid_dep_wait();
    const T *in = (const T *)p.in;
    T *out = (T *)p.out;
    const int lo = sizeof(T) == 1 ? -128 : -32768, hi = sizeof(T) == 1 ? 127 : 32767;
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < p.outputs; o += (long long)gridDim.x * blockDim.x) {
        long long base = 0, rem = o;
        for (int k = p.nk - 1; k >= 0; k--) {
            base += (rem % p.ksize[k]) * p.kstride[k];
            rem /= p.ksize[k];
        }
        int idx[6] = {0, 0, 0, 0, 0, 0};
        long long off = base;
        const Fold f = fold_of(p.op);
        ACC acc = fold_start<T, ACC>(f);
        float facc = p.op == ESPDL_REDUCE_PROD ? 1.f : 0.f; // int8 product, both sums of exponentials
        double dacc = 1.0;                                   // int16 product
        const float in_scale = dl_scale(p.e_in);
        for (long long i = 0; i < p.count; i++) {
            const ACC v = (ACC)in[off];
            if (p.op == ESPDL_REDUCE_PROD) {
                const float t = __fmul_rn((float)(int)v, in_scale);
                if (sizeof(T) == 1)
                    facc = __fmul_rn(facc, t);
                else
                    dacc = __dmul_rn(dacc, (double)t);
            } else if (p.op == ESPDL_REDUCE_LOG_SUM_EXP) {
                facc = __fadd_rn(facc, sizeof(T) == 1 ? p.exp_table[(int)v + 128] : expf(__fmul_rn((float)(int)v, in_scale)));
            } else {
                acc = fold_element<ACC>(f, acc, v);
            }
            for (int r = p.nr - 1; r >= 0; r--) { // odometer over the reduced axes
                off += p.rstride[r];
                if (++idx[r] < p.rsize[r])
                    break;
                off -= (long long)p.rsize[r] * p.rstride[r];
                idx[r] = 0;
            }
        }
        long long q;
        if (p.op == ESPDL_REDUCE_PROD) {
            if (sizeof(T) == 1) {
                q = fround_x86(__fmul_rn(facc, dl_rescale(p.e_out)), p.half_even);
            } else {
                // the fp64 product times the fp32 scale, rounded as a double (floor(v + 0.5), or to nearest even)
                const double v = __dmul_rn(dacc, (double)dl_rescale(p.e_out));
                q = !(fabs(v) < 2147483647.0) ? (long long)INT_MIN : (p.half_even ? (long long)__double2ll_rn(v) : (long long)floor(__dadd_rn(v, 0.5)));
            }
        } else if (p.op == ESPDL_REDUCE_LOG_SUM_EXP) {
            q = fround_x86(__fmul_rn(logf(facc), dl_rescale(p.e_out)), p.half_even);
        } else {
            q = finish_integer<ACC>(p, acc);
        }
        out[o] = (T)max((long long)lo, min((long long)hi, q));
    }
}

// Reduction over the middle axis of [outer][count][C] (the spatial mean / pool of NHWC maps), integer operators.
// Bound by memory: every input byte once.  A thread per output walked `count` elements one after another, a byte each, with
// C threads at work per image (a 184x184x32 map took 2.2 ms, 5 GB/s); here a thread owns V = 16 bytes of channels and every
// rows-th pixel, eight loads in flight, the partial results meet in shared memory, and with few images up to eight
// thread blocks of a cluster share one (their partials are read through distributed shared memory by the first).
// Integer sums and extrema do not depend on the order.
template <typename T, int V, typename ACC, Fold F>
__device__ __forceinline__ void fold_vector(ACC (&acc)[V], const T *v)
{
    if constexpr (sizeof(T) == 1 && V % 4 == 0 && F == FOLD_SUM) { // byte sums: dp4a against one-hot selectors
#pragma unroll
        for (int j = 0; j < V; j++) acc[j] = __dp4a(((const int *)v)[j / 4], 1 << (8 * (j % 4)), acc[j]);
    } else {
#pragma unroll
        for (int j = 0; j < V; j++) acc[j] = fold_element<ACC>(F, acc[j], (ACC)v[j]);
    }
}

template <typename T, int V, typename ACC, Fold F, int THREADS>
__global__ void __launch_bounds__(THREADS) channel_reduce_kernel(ReduceParams p, int C, int slice_lanes, int slices, int rows, int early)
{
    namespace cg = cooperative_groups;
    __shared__ ACC part[V * THREADS]; // [channel of the lane][thread]: consecutive threads in consecutive words
    cg::cluster_group cluster = cg::this_cluster();
    const int cl = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const long long item = blockIdx.x / cl;
    const long long image = item / slices;
    const int slice = (int)(item - image * slices);
    const int tx = threadIdx.x % slice_lanes, ty = threadIdx.x / slice_lanes;
    const int c0 = (slice * slice_lanes + tx) * V;
    const bool active = ty < rows && c0 < C;
    const ACC start = fold_start<T, ACC>(F);
    ACC acc[V];
#pragma unroll
    for (int j = 0; j < V; j++) acc[j] = start;
    if (early)
        grid_dep_launch();
    grid_dep_wait();
    if (active) {
        struct alignas(V * sizeof(T)) Vec {
            T v[V];
        };
        const T *src = (const T *)p.in + image * p.count * C + c0;
        const long long step = (long long)rows * cl;
        long long r = (long long)rank * rows + ty;
        auto take = [&](auto depth) { // `depth` loads in flight: a lone image is bound by their latency
            constexpr int D = decltype(depth)::value;
            for (; r + (D - 1) * step < p.count; r += D * step) {
                Vec w[D];
#pragma unroll
                for (int u = 0; u < D; u++) w[u] = *(const Vec *)(src + (r + u * step) * C);
#pragma unroll
                for (int u = 0; u < D; u++) fold_vector<T, V, ACC, F>(acc, w[u].v);
            }
        };
        take(std::integral_constant<int, 8>{});
        take(std::integral_constant<int, 2>{});
        take(std::integral_constant<int, 1>{});
    }
    // Lanes of a warp that own the same channels (a power of two of them to a pixel) meet first (27 images of 24x12x32: 4.5 us with all of the
    // meeting in shared memory, 2.6 this way), each step leaving a lane with half as many
    // channels to add: V - 1 exchanges in all.  Then one row of partials per warp, or, where pixels do not divide a warp, per thread row.
    const bool halving = (slice_lanes & (slice_lanes - 1)) == 0 && slice_lanes <= 32;
    int rows_left;
    if (halving) {
        int col = 0;
        bool holds = true;
        const int lane = threadIdx.x & 31;
        auto step = [&](auto level, auto width) { // `width` channels before the step
            constexpr int off = 16 >> decltype(level)::value, W = decltype(width)::value;
            if (off < slice_lanes)
                return;
            const bool up = lane & off;
            if constexpr (W > 1) {
#pragma unroll
                for (int j = 0; j < W / 2; j++) {
                    const ACC other = __shfl_xor_sync(0xffffffffu, up ? acc[j] : acc[j + W / 2], off);
                    acc[j] = fold_partial<ACC>(F, up ? acc[j + W / 2] : acc[j], other);
                }
                col += up ? W / 2 : 0;
            } else {
                acc[0] = fold_partial<ACC>(F, acc[0], __shfl_xor_sync(0xffffffffu, acc[0], off));
                holds = holds && !up;
            }
        };
        step(std::integral_constant<int, 0>{}, std::integral_constant<int, V>{});
        step(std::integral_constant<int, 1>{}, std::integral_constant<int, (V > 2 ? V / 2 : 1)>{});
        step(std::integral_constant<int, 2>{}, std::integral_constant<int, (V > 4 ? V / 4 : 1)>{});
        step(std::integral_constant<int, 3>{}, std::integral_constant<int, (V > 8 ? V / 8 : 1)>{});
        step(std::integral_constant<int, 4>{}, std::integral_constant<int, (V > 16 ? V / 16 : 1)>{});
        int width = V;
        for (int off = 16; off >= slice_lanes && width > 1; off >>= 1) width >>= 1;
        rows_left = THREADS / 32;
#pragma unroll
        for (int j = 0; j < V; j++)
            if (j < width && holds)
                part[(col + j) * THREADS + (threadIdx.x >> 5) * slice_lanes + tx] = acc[j];
    } else {
#pragma unroll
        for (int j = 0; j < V; j++) part[j * THREADS + threadIdx.x] = acc[j];
        int half = 1;
        while (half < rows) half <<= 1;
        for (half >>= 1; half; half >>= 1) {
            __syncthreads();
            if (ty < half && ty + half < rows) {
                const int other = threadIdx.x + half * slice_lanes;
#pragma unroll
                for (int j = 0; j < V; j++) part[j * THREADS + threadIdx.x] = fold_partial<ACC>(F, part[j * THREADS + threadIdx.x], part[j * THREADS + other]);
            }
        }
        rows_left = 1;
    }
    __syncthreads();
    const int lo = sizeof(T) == 1 ? -128 : -32768, hi = sizeof(T) == 1 ? 127 : 32767;
    const int cols = min(slice_lanes * V, C - slice * slice_lanes * V);
    for (int col = threadIdx.x; col < cols; col += THREADS) {
        const int at = (col % V) * THREADS + col / V;
        ACC sum = part[at];
#pragma unroll 4
        for (int r = 1; r < rows_left; r++) sum = fold_partial<ACC>(F, sum, part[at + r * slice_lanes]);
        if (cl > 1) {
            part[at] = sum;
            continue;
        }
        const long long q = finish_integer<ACC>(p, sum);
        ((T *)p.out)[image * C + slice * slice_lanes * V + col] = (T)max((long long)lo, min((long long)hi, q));
    }
    if (cl > 1)
        cluster.sync();
    if (cl > 1 && rank == 0) {
        for (int col = threadIdx.x; col < cols; col += THREADS) {
            const int at = (col % V) * THREADS + col / V;
            ACC sum = part[at];
#pragma unroll 4
            for (int k = 1; k < cl; k++) sum = fold_partial<ACC>(F, sum, cluster.map_shared_rank(part, k)[at]);
            const long long q = finish_integer<ACC>(p, sum);
            ((T *)p.out)[image * C + slice * slice_lanes * V + col] = (T)max((long long)lo, min((long long)hi, q));
        }
    }
    if (cl > 1)
        cluster.sync(); // no block leaves while its partials may still be read
}

template <typename T, int V, typename ACC, int THREADS>
int launch_channel_reduce(const ReduceParams &p, long long outer, int C, cudaStream_t s)
{
    const ReducePlan plan = reduce_plan(outer, p.count, C, V, THREADS, num_sms());
    if (plan.rows < 1)
        return ESPDL_ERR_UNSUPPORTED;
    const int slice_lanes = plan.slice_lanes, slices = plan.slices, rows = plan.rows, cl = plan.cluster;
    const long long items = outer * slices;
    if (items * cl > 0x7fffffffll)
        return ESPDL_ERR_TOO_LARGE;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items * cl)), cfg.blockDim = dim3(THREADS), cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cl, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 2 : 1;
    auto launch = [&](auto kernel) {
        if (cl > 8)
            cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchKernelEx(&cfg, kernel, p, C, slice_lanes, slices, rows, (int)in_model_scope());
    };
    switch (fold_of(p.op)) {
    case FOLD_SUM: launch(channel_reduce_kernel<T, V, ACC, FOLD_SUM, THREADS>); break;
    case FOLD_MAX: launch(channel_reduce_kernel<T, V, ACC, FOLD_MAX, THREADS>); break;
    case FOLD_MIN: launch(channel_reduce_kernel<T, V, ACC, FOLD_MIN, THREADS>); break;
    case FOLD_ABS: launch(channel_reduce_kernel<T, V, ACC, FOLD_ABS, THREADS>); break;
    case FOLD_SQUARE: launch(channel_reduce_kernel<T, V, ACC, FOLD_SQUARE, THREADS>); break;
    }
    count_launch();
    return check_launch("channel reduce");
}

// Below 2 KB an image keeps too few of a block's threads busy: a thread per output then (reduce_kernel, pool_kernel).
bool channel_reduce_pays(long long count, int C, int elem_size) { return count * C * elem_size >= 2048; }

template <typename T, typename ACC>
int channel_reduce(const ReduceParams &p, long long outer, int C, cudaStream_t s)
{
    const uintptr_t a = (uintptr_t)p.in | (uintptr_t)(C * sizeof(T));
    // a few large images: more than 8 loads a thread with eight blocks of 256 each, and SMs left for sixteen of 512
    // (184x184x64, one image: about 20 -> 9.5 us)
    if (a % 16 == 0 && outer <= num_sms() / 16 && p.count * C * (long long)sizeof(T) >= 8ll * 8 * 256 * 16)
        return launch_channel_reduce<T, 16 / sizeof(T), ACC, 512>(p, outer, C, s);
    if (a % 16 == 0)
        return launch_channel_reduce<T, 16 / sizeof(T), ACC, 256>(p, outer, C, s);
    if (a % 4 == 0)
        return launch_channel_reduce<T, 4 / sizeof(T), ACC, 256>(p, outer, C, s);
    return launch_channel_reduce<T, 1, ACC, 256>(p, outer, C, s);
}

} // namespace

bool average_pool_whole_supported(const espdl_pool_desc &d)
{
    const long long pixels = (long long)d.in_h * d.in_w;
    return d.op != ESPDL_POOL_MAX && channel_reduce_pays(pixels, d.c, d.dtype == ESPDL_DTYPE_INT8 ? 1 : 2);
}

int average_pool_whole(const espdl_pool_desc &d, float scale, cudaStream_t s)
{
    ReduceParams p;
    memset(&p, 0, sizeof(p));
    p.in = d.input, p.out = d.output, p.op = AVERAGE_POOL, p.scale = scale, p.count = (long long)d.in_h * d.in_w;
    return d.dtype == ESPDL_DTYPE_INT8 ? channel_reduce<int8_t, int32_t>(p, d.n, d.c, s) : channel_reduce<int16_t, long long>(p, d.n, d.c, s);
}

int reduce_op(const espdl_reduce_desc &d, cudaStream_t s)
{
    if (!d.input || !d.output || d.ndim < 1 || d.ndim > 6 || d.op < 0 || d.op > ESPDL_REDUCE_LOG_SUM_EXP)
        return ESPDL_ERR_INVALID_ARG;
    if (d.op == ESPDL_REDUCE_LOG_SUM_EXP && d.dtype == ESPDL_DTYPE_INT8 && !d.exp_table)
        return ESPDL_ERR_INVALID_ARG;
    if (d.dtype != ESPDL_DTYPE_INT8 && d.dtype != ESPDL_DTYPE_INT16)
        return ESPDL_ERR_UNSUPPORTED;
    ReduceParams p;
    p.in = d.input, p.out = d.output, p.op = d.op, p.half_even = d.round_mode == ESPDL_ROUND_HALF_EVEN;
    p.e_in = d.in_exponent, p.e_out = d.out_exponent;
    p.exp_table = d.exp_table, p.scale = 0.f;
    p.nk = p.nr = 0, p.outputs = 1, p.count = 1;
    long long stride = 1;
    long long strides[6];
    for (int i = d.ndim - 1; i >= 0; i--) {
        if (d.shape[i] <= 0)
            return ESPDL_ERR_INVALID_ARG;
        strides[i] = stride;
        stride *= d.shape[i];
    }
    for (int i = 0; i < d.ndim; i++) {
        if (d.reduce[i]) {
            p.rsize[p.nr] = d.shape[i], p.rstride[p.nr] = strides[i], p.nr++;
            p.count *= d.shape[i];
        } else {
            p.ksize[p.nk] = d.shape[i], p.kstride[p.nk] = strides[i], p.nk++;
            p.outputs *= d.shape[i];
        }
    }
    if (abs(p.e_in) > 30 || abs(p.e_out) > 30)
        return ESPDL_ERR_UNSUPPORTED;
    // [outer][count][C]: one run of reduced axes between kept ones (unit axes may stand anywhere)
    const bool ordered = d.op == ESPDL_REDUCE_PROD || d.op == ESPDL_REDUCE_LOG_SUM_EXP; // sums in floating point keep the reference's order
    long long outer = 1, inner = 1;
    int state = 0; // 0: leading kept axes, 1: reduced, 2: trailing kept
    for (int i = 0; i < d.ndim && state < 3; i++) {
        if (d.shape[i] == 1)
            continue;
        if (d.reduce[i])
            state = state <= 1 ? 1 : 3;
        else if (state == 0)
            outer *= d.shape[i];
        else
            state = 2, inner *= d.shape[i];
    }
    if (!ordered && state < 3 && inner <= 65536 && channel_reduce_pays(p.count, (int)inner, d.dtype == ESPDL_DTYPE_INT8 ? 1 : 2))
        return d.dtype == ESPDL_DTYPE_INT8 ? channel_reduce<int8_t, int32_t>(p, outer, (int)inner, s)
                                           : channel_reduce<int16_t, long long>(p, outer, (int)inner, s);
    const long long blocks = (p.outputs + 255) / 256;
    const int grid = (int)(blocks < (long long)num_sms() * 8 ? blocks : (long long)num_sms() * 8);
    if (d.dtype == ESPDL_DTYPE_INT8)
        launch_mover(reduce_kernel<int8_t, int32_t>, dim3(grid), dim3(256), 0, s, p);
    else
        launch_mover(reduce_kernel<int16_t, long long>, dim3(grid), dim3(256), 0, s, p);
    count_launch();
    return check_launch("reduce");
}


// ------------------------------------------------------------------------------------------ Pad
// dl::module::Pad (esp-dl/dl/module/include/dl_module_pad.hpp:10-100; per-axis rules of esp-dl/dl/base/dl_base_pad.cpp:18-66).
namespace {

struct PadParams {
    const void *in;
    void *out;
    int ndim, mode;
    int ishape[6], oshape[6], begin[6];
    long long istride[6];
    long long total;
    long long constant;
};

template <typename T>
__global__ void __launch_bounds__(256) pad_kernel(PadParams p, int early)
{
    if (early)
        grid_dep_launch();
    grid_dep_wait();
    const T *in = (const T *)p.in;
    T *out = (T *)p.out;
    for (long long o = blockIdx.x * (long long)blockDim.x + threadIdx.x; o < p.total; o += (long long)gridDim.x * blockDim.x) {
        long long rem = o, off = 0;
        bool inside = true;
        for (int k = p.ndim - 1; k >= 0; k--) {
            int i = (int)(rem % p.oshape[k]) - p.begin[k];
            rem /= p.oshape[k];
            const int n = p.ishape[k];
            if (i < 0 || i >= n) {
                if (p.mode == ESPDL_PAD_CONSTANT)
                    inside = false;
                else if (p.mode == ESPDL_PAD_EDGE)
                    i = i < 0 ? 0 : n - 1;
                else
                    i = i < 0 ? -i : 2 * (n - 1) - i; // mirror, the edge element is not repeated
                i = max(0, min(n - 1, i));
            }
            off += (long long)i * p.istride[k];
        }
        out[o] = inside ? in[off] : (T)p.constant;
    }
}

} // namespace

int pad_op(const espdl_pad_desc &d, cudaStream_t s)
{
    if (!d.input || !d.output || d.ndim < 1 || d.ndim > 6 || d.mode < 0 || d.mode > 2)
        return ESPDL_ERR_INVALID_ARG;
    if (d.elem_size != 1 && d.elem_size != 2 && d.elem_size != 4)
        return ESPDL_ERR_UNSUPPORTED;
    PadParams p;
    p.in = d.input, p.out = d.output, p.ndim = d.ndim, p.mode = d.mode, p.constant = d.constant, p.total = 1;
    long long stride = 1;
    for (int i = d.ndim - 1; i >= 0; i--) {
        if (d.shape[i] <= 0 || d.pad_begin[i] < 0 || d.pad_end[i] < 0)
            return ESPDL_ERR_INVALID_ARG;
        if (d.mode == ESPDL_PAD_REFLECT && (d.pad_begin[i] >= d.shape[i] || d.pad_end[i] >= d.shape[i]))
            return ESPDL_ERR_INVALID_ARG;
        p.ishape[i] = d.shape[i], p.begin[i] = d.pad_begin[i], p.oshape[i] = d.shape[i] + d.pad_begin[i] + d.pad_end[i];
        p.istride[i] = stride;
        stride *= d.shape[i];
        p.total *= p.oshape[i];
    }
    const long long blocks = (p.total + 255) / 256;
    const int grid = (int)(blocks < (long long)num_sms() * 16 ? blocks : (long long)num_sms() * 16);
    if (d.elem_size == 1)
        launch_mover(pad_kernel<int8_t>, dim3(grid), dim3(256), 0, s, p);
    else if (d.elem_size == 2)
        launch_mover(pad_kernel<int16_t>, dim3(grid), dim3(256), 0, s, p);
    else
        launch_mover(pad_kernel<int32_t>, dim3(grid), dim3(256), 0, s, p);
    count_launch();
    return check_launch("pad");
}

} // namespace espdl
