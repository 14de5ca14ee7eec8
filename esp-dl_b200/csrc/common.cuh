// Shared device/host helpers of the B200 backend: ESP-DL's exact rounding and
// saturation rules as device functions, status plumbing and launch accounting.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/espdl_b200.h"

namespace espdl {

// ---------------------------------------------------------------- host state
int set_cuda_error(cudaError_t e, const char *what); // records text, returns ESPDL_ERR_CUDA
int set_error_text(int status, const char *fmt, ...); // records text for espdl_b200_last_error, returns status
void count_launch(int n = 1);
int num_sms();
// Work counters of a persistent kernel that hands out its tiles dynamically: two zero-initialised words {next tile,
// CTAs done} in device memory that no other launch in flight uses - one pair per stream, or per stream and capture sequence
// while `s` is being captured into a graph (launches of one stream, and the nodes captured on one stream, run one after
// the other; two graphs, and the branches of one, may run side by side).  The kernel's last CTA writes both words back to zero.  Null when no pair is left: the
// kernel then walks its tiles in the fixed order.
unsigned *sched_counters(cudaStream_t s);
int lp_norm_op(const espdl_norm_desc &d, cudaStream_t s); // sequence_ops.cu
// Records the most recent failed launch (cudaGetLastError) if any.
int check_launch(const char *what);
// Programmatic dependent launch: the kernel may become resident while the previous kernel of the stream is still
// draining (its CTAs take an SM as soon as one is free and run their prologue: barriers, TMEM, per-channel constants).
// Such a kernel calls grid_dep_wait() before it reads or writes anything a previous kernel touches, and
// grid_dep_launch() once its own CTA is set up.  ESPDL_B200_NO_PDL=1 launches them the plain way.
bool pdl_enabled();

template <typename... KArgs, typename... Args>
cudaError_t launch_overlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr, cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// The kernels that move or rewrite tensors (elementwise operators, pools, copies, reductions ...) start with grid_dep_wait() and
// take a last argument `early`: whether they let the next kernel's blocks become resident at once.  Inside a model's plan, whose
// parameters no launch writes, the conv kernels read theirs (filter, bias, exponents, table) before they wait; outside of it a caller of
// the C ABI may have written them just before, with espdl_b200_copy or a kernel of its own: both sides are `early` only inside.
bool in_model_scope();

template <typename... KArgs, typename... Args>
cudaError_t launch_mover(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args &&...args)
{
    return launch_overlapped(kernel, grid, block, smem, s, args..., (int)in_model_scope());
}

#ifdef __CUDACC__
// Blocks until every kernel this one depends on has finished and its writes are visible to this grid.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// This CTA no longer minds the next kernel's CTAs becoming resident.
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// A bounded wait ran out: `word` is host memory.
__device__ __forceinline__ void report_timeout(int *word)
{
    if (word)
        atomicExch_system(word, ESPDL_ERR_TIMEOUT);
}
#endif

#define ESPDL_CUDA_TRY(call)                                \
    do {                                                    \
        cudaError_t e__ = (call);                           \
        if (e__ != cudaSuccess)                             \
            return ::espdl::set_cuda_error(e__, #call);     \
    } while (0)

// Descriptor checks shared by every conv entry point (abi.cu); ESPDL_OK or the status to return.
int conv_validate(const espdl_conv_desc *d);

// kernels behind the C ABI (one translation unit each)
int conv2d_simt(const espdl_conv_desc &d, cudaStream_t s);
int conv2d_narrow(const espdl_conv_desc &d, cudaStream_t s); // short windows, few output channels
bool conv2d_narrow_supported(const espdl_conv_desc &d);
float conv2d_narrow_estimate_us(const espdl_conv_desc &d);
float conv2d_simt_estimate_us(const espdl_conv_desc &d); // about what it takes, for the choice against packed operands
int conv2d_depthwise(const espdl_conv_desc &d, cudaStream_t s);
bool conv2d_tc_supported(const espdl_conv_desc &d);
bool overlaps(const espdl_conv_desc &d); // do results lie where inputs do?  Channels side by side in the same rows don't
size_t conv2d_tc_workspace_bytes(const espdl_conv_desc &d);
int conv2d_tc(const espdl_conv_desc &d, void *workspace, size_t workspace_bytes, cudaStream_t s, const long long *peer_delta = nullptr,
              int n_peer = 0, int *row_sums = nullptr); // peer_delta: byte distances to copies of the output on other GPUs that receive every row as well
// Packed operands of the tile kernel (pack.cu): rows of Kp bytes, Kp a multiple of 16; int16 operands as two planes.
struct PackedOperands {
    void *a_hi, *a_lo, *b_hi, *b_lo;
    int *row_sum; // int16: sum of every row of A
    int Kp;
};
// Packs output pixels [row0, row0 + rows) and, with `filter`, the filter.
int pack_operands(const espdl_conv_desc &d, long long row0, int rows, bool filter, const PackedOperands &o, cudaStream_t s);
// Convs and products that run on the tile kernel once their operands are packed: reductions that are no multiple of 16, int16
// windows, channel counts that are no multiple of 16.
bool conv2d_packed_supported(const espdl_conv_desc &d);
size_t conv2d_packed_workspace_bytes(const espdl_conv_desc &d);
int conv2d_packed(const espdl_conv_desc &d, void *workspace, size_t workspace_bytes, cudaStream_t s);
// Small int8 convs and products with warp-level matrix instructions (conv_mma.cu); the estimate decides against the tile kernels.
bool conv2d_mma_supported(const espdl_conv_desc &d);
float conv2d_mma_estimate_us(const espdl_conv_desc &d);
int conv2d_mma(const espdl_conv_desc &d, cudaStream_t s);
// The same for int16, split into byte planes in registers (conv_mma16.cu).
bool conv2d_mma16_supported(const espdl_conv_desc &d);
float conv2d_mma16_estimate_us(const espdl_conv_desc &d);
int conv2d_mma16(const espdl_conv_desc &d, cudaStream_t s);
// Each translation unit with bounded device-side waits keeps the address of ONE status word in pinned, device-mapped host
// memory: a wait that runs out stores ESPDL_ERR_TIMEOUT there, and espdl_b200_stream_sync reads it as ordinary memory.
// (A device word per unit, copied back at every synchronisation, cost seven blocking copies: 60 us of a 160 us pass.)
int bind_device_error(int *word);
int bind_device_error_stem(int *word);
int bind_device_error_band(int *word);
int bind_device_error_dw(int *word);
int bind_device_error_dw_mma(int *word);
int bind_device_error_conv(int *word);
int bind_device_error_block(int *word);
int bind_device_error_dwpw(int *word);
int image_preprocess(const espdl_image_desc &d, cudaStream_t s);
int detect_candidates(const espdl_detect_desc &d, cudaStream_t s);
int reduce_op(const espdl_reduce_desc &d, cudaStream_t s);
// average over whole images, as a reduction (reduce.cu)
bool average_pool_whole_supported(const espdl_pool_desc &d);
int average_pool_whole(const espdl_pool_desc &d, float scale, cudaStream_t s);
int pad_op(const espdl_pad_desc &d, cudaStream_t s);
bool fused_block_supported(const espdl_block_desc &d);
int fused_block_tc(const espdl_block_desc &d, cudaStream_t s);
bool fused_dwpw_supported(const espdl_block_desc &d, bool has_expand); // depthwise -> pointwise pair without an expand conv
int fused_dwpw(const espdl_block_desc &d, cudaStream_t s);
bool conv2d_conv_tc_supported(const espdl_conv_desc &d);
int conv2d_conv_tc(const espdl_conv_desc &d, cudaStream_t s);
bool conv2d_dw_tma_supported(const espdl_conv_desc &d);
int conv2d_dw_tma(const espdl_conv_desc &d, cudaStream_t s);
bool conv2d_dw_tma_whole(const espdl_conv_desc &d); // its tiles have all channels of a pixel
bool conv2d_dw_mma_supported(const espdl_conv_desc &d); // 3x3 at stride 1 on the warp-level matrix instruction (conv_dw_mma.cu)
bool conv2d_dw_mma_pays(const espdl_conv_desc &d);
int conv2d_dw_mma(const espdl_conv_desc &d, cudaStream_t s);
bool conv2d_stem_tc_supported(const espdl_conv_desc &d);
int conv2d_stem_tc(const espdl_conv_desc &d, cudaStream_t s);
// 3x3 conv with 8 or 16 input channels: banded-filter tensor-core kernel over 128-byte row windows (conv_band_tc.cu)
bool conv2d_band_tc_supported(const espdl_conv_desc &d);
int conv2d_band_tc(const espdl_conv_desc &d, cudaStream_t s);

// ------------------------------------------------------------- device math
// dl::tool::shift_and_round on a 32-bit accumulator (int8 operators).
//   shift > 0 : HALF_UP   floor((v + 2^(s-1)) / 2^s)  ==  (v >> s) + bit (s-1) of v
//               HALF_EVEN floor, +1 if remainder > half or (== half and quotient odd)
//   shift <= 0: (int64)v << -shift, saturated to int32
// Callers guarantee shift >= -31.
__device__ __forceinline__ int32_t shift_round32(int32_t v, int shift, int half_even)
{
    if (shift > 31) // |v| is at most 2^31, half a step of 2^32, and that tie goes to 0 either way
        v = 0, shift = 31;
    if (shift > 0) {
        int32_t q = v >> shift;
        if (!half_even) {
            q += (v >> (shift - 1)) & 1;
        } else {
            const int32_t rem = v & ((1 << shift) - 1);
            const int32_t half = 1 << (shift - 1);
            q += (rem > half || (rem == half && (q & 1))) ? 1 : 0;
        }
        return q;
    }
    const long long s = (long long)v << (-shift);
    return (int32_t)max(min(s, (long long)INT32_MAX), (long long)INT32_MIN);
}

// Same on a 64-bit accumulator (int16 operators); |shift| <= 62.
__device__ __forceinline__ long long shift_round64(long long v, int shift, int half_even)
{
    if (shift > 0) {
        long long q = v >> shift;
        if (!half_even) {
            q += (v >> (shift - 1)) & 1;
        } else {
            const long long rem = v & ((1ll << shift) - 1);
            const long long half = 1ll << (shift - 1);
            q += (rem > half || (rem == half && (q & 1))) ? 1 : 0;
        }
        return q;
    }
    return (long long)((unsigned long long)v << (-shift));
}

// Constants of the one-add-one-shift int8 epilogue, q = (acc + bias_half) >> shift with bias_half = bias + 2^(s-1) (one less
// for half to even, see shift_fast in tc_common.cuh).  It equals the wrapping 32-bit bias add and 64-bit rounding shift of
// the reference as long as nothing leaves 32 bits, i.e. |bias| + |acc| + 2^(s-1) < 2^31; `acc_bound` bounds |acc| (2^14 per
// term of the sum).  A shift beyond 31 - channels whose weights were all but zero when the model was quantised; model files
// have shifts up to 39 and saturated biases there - gives 0 for every 32-bit sum: a positive constant below 2^31 shifted
// out completely.  Returns false for channels that need the general form (shift < 1, a bias close to the type's ends).
__device__ __forceinline__ bool fast_constants(int bias, int s, int acc_bound, int half_even, int &bias_half, int &shift)
{
    if (s > 31) {
        bias_half = 1 << 29, shift = 31;
        return acc_bound <= (1 << 29);
    }
    const int sh = max(1, s);
    const unsigned half = 1u << (sh - 1);
    bias_half = (int)((unsigned)bias + half - (half_even ? 1u : 0u));
    shift = sh;
    return s >= 1 && (long long)abs((long long)bias) + acc_bound + (long long)half <= 2147483647ll;
}

__device__ __forceinline__ int32_t sat8(int32_t v) { return max(-128, min(127, v)); }
__device__ __forceinline__ int32_t sat16(int32_t v) { return max(-32768, min(32767, v)); }
__device__ __forceinline__ long long sat16_64(long long v) { return max(-32768ll, min(32767ll, v)); }

// int8 conv epilogue: bias (wrapping 32-bit add), shift/round, ReLU, saturate.
__device__ __forceinline__ int32_t requant8(int32_t acc, int32_t bias, int shift, int relu, int half_even)
{
    int32_t v = shift_round32((int32_t)((uint32_t)acc + (uint32_t)bias), shift, half_even);
    if (relu)
        v = max(v, 0);
    return sat8(v);
}

__device__ __forceinline__ int32_t requant16(long long acc, long long bias, int shift, int relu, int half_even)
{
    long long v = shift_round64(acc + bias, shift, half_even);
    if (relu)
        v = max(v, 0ll);
    return (int32_t)sat16_64(v);
}

// dl::tool::round(float) on generic targets: (int)floorf((float)((double)v + 0.5)).
// A single correctly rounded fp32 add gives the same float as the double sum
// narrowed to float (the double sum of two floats whose exponents differ by less
// than 29 is exact), so one __fadd_rn reproduces it without fp64.
__device__ __forceinline__ int fround_half_up(float v) { return (int)floorf(__fadd_rn(v, 0.5f)); }
// ESP32-P4: fcvt.w.s with round-to-nearest-even.
__device__ __forceinline__ int fround_half_even(float v) { return __float2int_rn(v); }
__device__ __forceinline__ int fround(float v, int half_even) { return half_even ? fround_half_even(v) : fround_half_up(v); }

// int16's epilogue after the sums in 32-bit instructions (64-bit sums, shifts and comparisons took more than twice as many): sum + bias + 2^(s-1) as H * 65536 + L,
// L in 16 bits, H bounded so that the shift leaves what saturates.  1 <= s <= 31, |bias| < 2^45, H below 2^30.
struct alignas(16) HalvesParam { // of a channel
    int h, l;  // bias + 2^(s-1)
    int limit; // |H| beyond it is outside int16 after the shift
    int shift;
};
__device__ __forceinline__ bool halves_fit(long long bias, int shift) { return shift >= 1 && shift <= 31 && bias < (1ll << 45) && bias > -(1ll << 45); }
template <bool EVEN>
__device__ __forceinline__ HalvesParam halves_param(long long bias, int shift)
{
    const int s = max(1, min(31, shift));
    const long long add = bias + (1ll << (s - 1)) - (EVEN ? 1 : 0);
    return {(int)(add >> 16), (int)(add & 0xffff), (int)((32768ll << max(0, s - 16)) - 1), s};
}
// (sum + bias + 2^(s-1)) >> s, the constants added: l with what it carries.
template <bool EVEN>
__device__ __forceinline__ int shift_halves(int h, int l, const HalvesParam &c)
{
    h += l >> 16;
    if (EVEN) { // a tie is rounded up only where that gives an even number
        const uint32_t q = __funnelshift_r(__byte_perm((uint32_t)l, (uint32_t)h, 0x5410), (uint32_t)(h >> 16), c.shift);
        l = (l & 0xffff) + (int)(q & 1u);
        h += l >> 16;
    }
    h = max(min(h, c.limit), ~c.limit);
    return (int)__funnelshift_r(__byte_perm((uint32_t)l, (uint32_t)h, 0x5410), (uint32_t)(h >> 16), c.shift);
}

// a / b and what is left, a >= 0, b > 0.  A 64-bit division is some hundred instructions; a few of them were a third of the time of a small launch, most tensors'
// indices fit 32 bits.
__device__ __forceinline__ long long div_rem(long long a, long long b, long long &rem)
{
    if (((a | b) >> 32) == 0) {
        const unsigned q = (unsigned)a / (unsigned)b;
        rem = (unsigned)a - q * (unsigned)b;
        return q;
    }
    const long long q = a / b;
    rem = a - q * b;
    return q;
}

// Column, row and image of an output pixel.
__device__ __forceinline__ void split_pixel(long long pix, int ow, int oh, int &x, int &y, int &n)
{
    long long rem_x, rem_y;
    n = (int)div_rem(div_rem(pix, ow, rem_x), oh, rem_y);
    x = (int)rem_x, y = (int)rem_y;
}

// DL_SCALE / DL_RESCALE: exact powers of two as floats.
__host__ __device__ __forceinline__ float dl_scale(int e) { return e > 0 ? (float)(1 << e) : 1.0f / (float)(1 << -e); }
__host__ __device__ __forceinline__ float dl_rescale(int e) { return e > 0 ? 1.0f / (float)(1 << e) : (float)(1 << -e); }

} // namespace espdl
