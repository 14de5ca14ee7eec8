// C ABI: life cycle, memory and the conv2d dispatcher (include/espdl_b200.h).
#include "common.cuh"
#include "tile_counters.cuh"

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <cmath>
#include <mutex>
#include <map>

namespace espdl {

static thread_local char g_last_error[512] = "";
static std::atomic<uint64_t> g_launches{0};
static int g_device = -1;
static int g_num_sms = 0;
static int *g_error_word = nullptr; // pinned, mapped: written by device-side waits that ran out
static std::mutex g_ws_mutex;
static void *g_ws = nullptr; // cached scratch of espdl_b200_conv2d (int16 limb planes)
static size_t g_ws_bytes = 0;
// Scratch of espdl_b200_conv2d for calls that can do without: a few streams keep one each, the least recently used makes room.
struct StreamScratch {
    unsigned long long stream = 0, used = 0; // the stream's id (never given to another one), the call that used it last
    void *p = nullptr;
    size_t bytes = 0;
};
static StreamScratch g_stream_scratch[4];
static unsigned long long g_scratch_calls = 0;

int set_cuda_error(cudaError_t e, const char *what)
{
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s", what, cudaGetErrorString(e));
    return ESPDL_ERR_CUDA;
}

int set_error_text(int status, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
    return status;
}

void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

int num_sms() { return g_num_sms > 0 ? g_num_sms : 148; }

namespace {
constexpr int SCHED_PAIRS = 2048;
__device__ unsigned g_sched_words[2 * SCHED_PAIRS]; // zero at load; every kernel leaves its pair zero
std::mutex g_sched_mutex;
TileCounters g_sched_pairs(SCHED_PAIRS);
std::map<cudaGraphExec_t, unsigned long long> g_graph_capture; // whose capture a graph came from, while it lives

// The capture that `s` is in, 0 for none; false where that cannot be asked.
bool capture_of(cudaStream_t s, unsigned long long &id)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    id = 0;
    if (cudaStreamGetCaptureInfo(s, &cs, &id) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (cs != cudaStreamCaptureStatusActive)
        id = 0;
    return true;
}
}

unsigned *sched_counters(cudaStream_t s)
{
    static unsigned *base = nullptr;
    static const bool off = getenv("ESPDL_B200_STATIC_TILES") != nullptr;
    if (off)
        return nullptr;
    unsigned long long id = 0;
    if (!capture_of(s, id))
        return nullptr;
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    if (!base) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_sched_words) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        base = (unsigned *)p;
    }
    // branches of one graph are captured on streams of their own and may run side by side
    const int pair = g_sched_pairs.get(id, s);
    return pair < 0 ? nullptr : base + 2 * pair;
}

int check_launch(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return set_cuda_error(e, what);
    return ESPDL_OK;
}

} // namespace espdl

using namespace espdl;

extern "C" {

int espdl_b200_init(int device)
{
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0) {
        snprintf(g_last_error, sizeof(g_last_error), "no CUDA device: %s", cudaGetErrorString(e));
        return ESPDL_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= count)
        return ESPDL_ERR_INVALID_ARG;
    if (g_device >= 0 && g_device != device)
        // one device per process: the cached scratch and the SM count belong to the device of the first call
        return set_error_text(ESPDL_ERR_INVALID_ARG, "espdl_b200_init(%d): this process is bound to device %d; call espdl_b200_shutdown first",
                              device, g_device);
    ESPDL_CUDA_TRY(cudaSetDevice(device));
    if (g_device == device)
        return ESPDL_OK; // done before: the properties of a device take milliseconds to ask for
    cudaDeviceProp prop;
    ESPDL_CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (prop.major != 10) {
        snprintf(g_last_error, sizeof(g_last_error), "device %d is sm_%d%d; this library holds sm_100a code only", device,
                 prop.major, prop.minor);
        return ESPDL_ERR_NO_DEVICE;
    }
    if (!g_error_word) {
        ESPDL_CUDA_TRY(cudaHostAlloc((void **)&g_error_word, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
        *g_error_word = 0;
    }
    int *word = nullptr; // the word as the device addresses it
    ESPDL_CUDA_TRY(cudaHostGetDevicePointer((void **)&word, g_error_word, 0));
    for (int (*bind)(int *) : {bind_device_error, bind_device_error_stem, bind_device_error_band, bind_device_error_dw, bind_device_error_dw_mma, bind_device_error_conv,
                               bind_device_error_block, bind_device_error_dwpw}) {
        const int st = bind(word);
        if (st)
            return st;
    }
    g_device = device;
    g_num_sms = prop.multiProcessorCount;
    return ESPDL_OK;
}

void espdl_b200_shutdown(void)
{
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if (g_ws) {
        cudaFree(g_ws);
        g_ws = nullptr;
        g_ws_bytes = 0;
    }
    for (StreamScratch &slot : g_stream_scratch) {
        if (slot.p)
            cudaFree(slot.p);
        slot = StreamScratch();
    }
    g_device = -1;
}

const char *espdl_b200_strerror(int status)
{
    switch (status) {
    case ESPDL_OK: return "ok";
    case ESPDL_ERR_INVALID_ARG: return "invalid argument";
    case ESPDL_ERR_UNSUPPORTED: return "unsupported combination";
    case ESPDL_ERR_CUDA: return "CUDA call failed";
    case ESPDL_ERR_NO_DEVICE: return "no usable sm_100 device";
    case ESPDL_ERR_NO_MEM: return "out of device memory";
    case ESPDL_ERR_TIMEOUT: return "device-side wait timed out";
    case ESPDL_ERR_TOO_LARGE: return "size beyond the fixed maximum";
    default: return "unknown status";
    }
}

const char *espdl_b200_last_error(void) { return g_last_error; }

int espdl_b200_arena_alloc(size_t bytes, void **dptr)
{
    if (!dptr)
        return ESPDL_ERR_INVALID_ARG;
    *dptr = nullptr;
    cudaError_t e = cudaMalloc(dptr, bytes ? bytes : 16);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return ESPDL_ERR_NO_MEM;
    }
    if (e != cudaSuccess)
        return set_cuda_error(e, "cudaMalloc");
    return ESPDL_OK;
}

int espdl_b200_arena_free(void *dptr)
{
    if (dptr)
        ESPDL_CUDA_TRY(cudaFree(dptr));
    return ESPDL_OK;
}

int espdl_b200_upload(void *dst_dev, const void *src_host, size_t bytes, void *stream)
{
    if ((!dst_dev || !src_host) && bytes)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaMemcpyAsync(dst_dev, src_host, bytes, cudaMemcpyHostToDevice, (cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_download(void *dst_host, const void *src_dev, size_t bytes, void *stream)
{
    if ((!dst_host || !src_dev) && bytes)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaMemcpyAsync(dst_host, src_dev, bytes, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return ESPDL_OK;
}

} // extern "C"
namespace espdl {
static thread_local int g_model_scope = 0;
static thread_local bool g_overlap = true;
bool in_model_scope() { return g_model_scope > 0; }

bool pdl_enabled()
{
    static const bool on = !getenv("ESPDL_B200_NO_PDL");
    return on && g_overlap;
}
} // namespace espdl
extern "C" {

void espdl_b200_model_scope(int enter) { g_model_scope += enter ? 1 : -1; }
void espdl_b200_overlap(int on) { g_overlap = on != 0; }

int espdl_b200_download_rows(void *dst_host, const void *src_dev, size_t row_bytes, size_t src_stride_bytes, size_t rows, void *stream)
{
    if ((!dst_host || !src_dev) && row_bytes && rows)
        return ESPDL_ERR_INVALID_ARG;
    if (src_stride_bytes < row_bytes)
        return ESPDL_ERR_INVALID_ARG;
    if (!row_bytes || !rows)
        return ESPDL_OK;
    ESPDL_CUDA_TRY(cudaMemcpy2DAsync(dst_host, row_bytes, src_dev, src_stride_bytes, row_bytes, rows, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_memset(void *dst_dev, int value, size_t bytes, void *stream)
{
    ESPDL_CUDA_TRY(cudaMemsetAsync(dst_dev, value, bytes, (cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_stream_sync(void *stream)
{
    ESPDL_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    // a tile kernel whose bounded wait expired left its status in the mapped word
    const int dev = g_error_word && *(volatile int *)g_error_word ? __atomic_exchange_n(g_error_word, 0, __ATOMIC_SEQ_CST) : 0;
    if (dev) {
        snprintf(g_last_error, sizeof(g_last_error), "a device-side bounded wait expired in the tensor-core tile kernel");
        return dev;
    }
    return ESPDL_OK;
}

int espdl_b200_host_alloc(size_t bytes, void **hptr)
{
    if (!hptr)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaMallocHost(hptr, bytes ? bytes : 16));
    return ESPDL_OK;
}

int espdl_b200_host_free(void *hptr)
{
    if (hptr)
        ESPDL_CUDA_TRY(cudaFreeHost(hptr));
    return ESPDL_OK;
}

uint64_t espdl_b200_launch_count(void) { return g_launches.load(); }

int espdl_b200_mem_info(size_t *free_bytes, size_t *total_bytes)
{
    size_t f = 0, t = 0;
    ESPDL_CUDA_TRY(cudaMemGetInfo(&f, &t));
    if (free_bytes)
        *free_bytes = f;
    if (total_bytes)
        *total_bytes = t;
    return ESPDL_OK;
}

int espdl_b200_stream_create(void **stream)
{
    if (!stream)
        return ESPDL_ERR_INVALID_ARG;
    cudaStream_t s;
    ESPDL_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    *stream = (void *)s;
    return ESPDL_OK;
}

int espdl_b200_stream_destroy(void *stream)
{
    if (!stream)
        return ESPDL_OK;
    unsigned long long id = 0;
    if (capture_of((cudaStream_t)stream, id) && !id && cudaStreamQuery((cudaStream_t)stream) == cudaSuccess) {
        std::lock_guard<std::mutex> lock(g_sched_mutex);
        g_sched_pairs.give_back_stream(stream);
    }
    cudaGetLastError(); // work in flight: its pair stays taken
    ESPDL_CUDA_TRY(cudaStreamDestroy((cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_event_create(void **event)
{
    if (!event)
        return ESPDL_ERR_INVALID_ARG;
    cudaEvent_t e;
    ESPDL_CUDA_TRY(cudaEventCreate(&e));
    *event = (void *)e;
    return ESPDL_OK;
}

int espdl_b200_event_destroy(void *event)
{
    if (event)
        ESPDL_CUDA_TRY(cudaEventDestroy((cudaEvent_t)event));
    return ESPDL_OK;
}

int espdl_b200_event_record(void *event, void *stream)
{
    if (!event)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaEventRecord((cudaEvent_t)event, (cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_event_elapsed_ms(void *start, void *stop, float *ms)
{
    if (!start || !stop || !ms)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaEventSynchronize((cudaEvent_t)stop));
    ESPDL_CUDA_TRY(cudaEventElapsedTime(ms, (cudaEvent_t)start, (cudaEvent_t)stop));
    return ESPDL_OK;
}

int espdl_b200_event_sync(void *event)
{
    if (!event)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaEventSynchronize((cudaEvent_t)event));
    return ESPDL_OK;
}

int espdl_b200_stream_wait_event(void *stream, void *event)
{
    if (!event)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaStreamWaitEvent((cudaStream_t)stream, (cudaEvent_t)event, 0));
    return ESPDL_OK;
}

int espdl_b200_device_copy(void *dst_dev, const void *src_dev, size_t bytes, void *stream)
{
    if ((!dst_dev || !src_dev) && bytes)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaMemcpyAsync(dst_dev, src_dev, bytes, cudaMemcpyDeviceToDevice, (cudaStream_t)stream));
    return ESPDL_OK;
}

int espdl_b200_graph_begin(void *stream)
{
    if (!stream)
        return ESPDL_ERR_INVALID_ARG; // the legacy default stream cannot be captured
    ESPDL_CUDA_TRY(cudaStreamBeginCapture((cudaStream_t)stream, cudaStreamCaptureModeThreadLocal));
    return ESPDL_OK;
}

int espdl_b200_graph_end(void *stream, void **graph)
{
    if (!stream || !graph)
        return ESPDL_ERR_INVALID_ARG;
    unsigned long long id = 0;
    capture_of((cudaStream_t)stream, id);
    cudaGraph_t g = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaError_t e = cudaStreamEndCapture((cudaStream_t)stream, &g);
    const char *what = "cudaStreamEndCapture";
    if (e == cudaSuccess) {
        what = "cudaGraphInstantiate";
        e = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
    }
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    if (e != cudaSuccess) {
        g_sched_pairs.give_back_capture(id); // nothing of it was ever launched
        return set_cuda_error(e, what);
    }
    g_graph_capture[exec] = id;
    *graph = (void *)exec;
    return ESPDL_OK;
}

int espdl_b200_graph_launch(void *graph, void *stream)
{
    if (!graph)
        return ESPDL_ERR_INVALID_ARG;
    ESPDL_CUDA_TRY(cudaGraphLaunch((cudaGraphExec_t)graph, (cudaStream_t)stream));
    return ESPDL_OK;
}

static int graph_destroy(void *graph, bool idle)
{
    if (!graph)
        return ESPDL_OK;
    {
        std::lock_guard<std::mutex> lock(g_sched_mutex);
        auto it = g_graph_capture.find((cudaGraphExec_t)graph);
        if (it != g_graph_capture.end()) {
            if (idle && it->second)
                g_sched_pairs.give_back_capture(it->second);
            g_graph_capture.erase(it);
        }
    }
    ESPDL_CUDA_TRY(cudaGraphExecDestroy((cudaGraphExec_t)graph));
    return ESPDL_OK;
}

int espdl_b200_graph_destroy(void *graph) { return graph_destroy(graph, false); }
int espdl_b200_graph_destroy_idle(void *graph) { return graph_destroy(graph, true); }

int espdl_b200_tile_counters(void)
{
    std::lock_guard<std::mutex> lock(g_sched_mutex);
    return g_sched_pairs.taken();
}

} // extern "C"

// ------------------------------------------------------------------ conv2d
// Checks every conv entry point makes before anything is planned or launched: pointers, extents, the output size
// the reference derives, exponent pointers that the kernels will dereference, and the supported enumerators.
int espdl::conv_validate(const espdl_conv_desc *d)
{
    if (!d || !d->input || !d->filter || !d->output)
        return ESPDL_ERR_INVALID_ARG;
    if (d->dtype != ESPDL_DTYPE_INT8 && d->dtype != ESPDL_DTYPE_INT16)
        return ESPDL_ERR_UNSUPPORTED;
    if (d->n < 0 || d->in_h <= 0 || d->in_w <= 0 || d->in_c <= 0 || d->out_c <= 0 || d->out_h <= 0 || d->out_w <= 0)
        return ESPDL_ERR_INVALID_ARG;
    if (d->kh <= 0 || d->kw <= 0 || d->stride_h <= 0 || d->stride_w <= 0 || d->dilation_h <= 0 || d->dilation_w <= 0)
        return ESPDL_ERR_INVALID_ARG;
    if (d->pad_top < 0 || d->pad_bottom < 0 || d->pad_left < 0 || d->pad_right < 0)
        return ESPDL_ERR_INVALID_ARG;
    if (d->group != 1 && !(d->group == d->in_c && d->out_c == d->in_c))
        return ESPDL_ERR_UNSUPPORTED;
    if (d->per_channel && !d->filter_exponents)
        return ESPDL_ERR_INVALID_ARG;
    if (d->activation != ESPDL_ACT_LINEAR && d->activation != ESPDL_ACT_RELU)
        return ESPDL_ERR_UNSUPPORTED;
    if (d->round_mode != ESPDL_ROUND_HALF_UP && d->round_mode != ESPDL_ROUND_HALF_EVEN)
        return ESPDL_ERR_INVALID_ARG;
    if (d->lut && d->dtype != ESPDL_DTYPE_INT8)
        return ESPDL_ERR_UNSUPPORTED;
    if (d->lut_channel_stride != 0 && (!d->lut || d->lut_channel_stride < 256))
        return ESPDL_ERR_INVALID_ARG;
    if ((d->in_pixel_stride && d->in_pixel_stride < d->in_c) || (d->out_pixel_stride && d->out_pixel_stride < d->out_c))
        return ESPDL_ERR_INVALID_ARG;
    if (d->filter_image_stride != 0 && d->group != 1)
        return ESPDL_ERR_INVALID_ARG;
    if (d->residual && (d->dtype != ESPDL_DTYPE_INT8 || d->group != 1 || d->kh != 1 || d->kw != 1 || d->stride_h != 1 || d->stride_w != 1 ||
                        (d->residual_pixel_stride && d->residual_pixel_stride < d->out_c)))
        return ESPDL_ERR_UNSUPPORTED; // the folded Add is implemented for pointwise int8 convs / Gemm
    // output extents must be the ones the reference derives (dl_module_conv.hpp:81-102)
    const int oh = (d->in_h + d->pad_top + d->pad_bottom - d->dilation_h * (d->kh - 1) - 1) / d->stride_h + 1;
    const int ow = (d->in_w + d->pad_left + d->pad_right - d->dilation_w * (d->kw - 1) - 1) / d->stride_w + 1;
    if (oh != d->out_h || ow != d->out_w)
        return ESPDL_ERR_INVALID_ARG;
    if (!d->per_channel) {
        const int shift = d->out_exponent - d->filter_exponent - d->in_exponent;
        const int lim = d->dtype == ESPDL_DTYPE_INT8 ? 31 : 62;
        if (shift > lim || shift < -lim)
            return ESPDL_ERR_INVALID_ARG;
    }
    return ESPDL_OK;
}

// 3x3 depthwise tensors, in outputs, below which the kernel without the TMA pipeline is the faster one.  In a model's stream of overlapping
// launches up to 16 M at stride 1 and 2 M at stride 2 (14x14x384 1.7 against 4.1 us, 16 images of 56x56x144 5.8 / 7.9; 64 of 28x28x192 at stride
// 2 5.6 / 5.2); launched one by one, where it has no previous kernel to hide its first loads behind, up to 1 M and 256 K (16 of
// 28x28x192 6.3 / 5.3).
static long long dw_small(int stride)
{
    return stride == 1 ? (espdl::in_model_scope() ? 16ll << 20 : 1ll << 20) : (espdl::in_model_scope() ? 2ll << 20 : 256ll << 10);
}

// Depthwise on the matrix instruction?
static bool runs_dw_mma(const espdl_conv_desc &d, bool small)
{
    const char *knob = getenv("ESPDL_B200_DW_MMA"); // 0: never, always: wherever it can run
    if (d.kernel != ESPDL_KERNEL_AUTO || (knob && *knob == '0') || getenv("ESPDL_B200_NO_DW_TMA"))
        return false;
    if (knob && *knob == 'a')
        return conv2d_dw_mma_supported(d);
    return !small && !getenv("ESPDL_B200_DEBUG_WAIT_EXPIRY") && !getenv("ESPDL_B200_DW_TMA_NARROW") && conv2d_dw_mma_pays(d);
}

// Short windows with few output channels: the CUDA cores where every other kernel would take longer.  The tile kernel's time is that of its waves
// of 128-pixel tiles, each its taps' loads one after the other and its rows' epilogue (from 2x2 and 3x3 windows of 33 to 540 thousand pixels); the
// warp-level instructions take about twice their estimate where chunks are words.
static bool runs_narrow(const espdl_conv_desc &d)
{
    const char *knob = getenv("ESPDL_B200_NARROW"); // 0: never, always: wherever it can run
    if (d.kernel != ESPDL_KERNEL_AUTO || d.n <= 0 || !conv2d_narrow_supported(d) || (knob && *knob == '0'))
        return false;
    if (knob && *knob == 'a')
        return true;
    if (conv2d_stem_tc_supported(d) || conv2d_band_tc_supported(d) || (d.in_c % 8 && d.kh * d.kw * d.in_c > 64)) // longer windows of words: packed operands
        return false;
    const float us = conv2d_narrow_estimate_us(d);
    const float mma = conv2d_mma_supported(d) ? conv2d_mma_estimate_us(d) : 8.f;
    if (mma < 8.f && mma * (d.in_c % 16 ? 2.f : 1.f) < 1.1f * us)
        return false;
    const double waves = ceil((double)d.n * d.out_h * d.out_w / 128 / num_sms());
    return us < (conv2d_conv_tc_supported(d) ? 2.5 + waves * (0.6 + 0.17 * d.kh * d.kw + 0.045 * d.out_c) : (double)conv2d_simt_estimate_us(d));
}

// Small enough for the warp-level matrix instructions?
static bool runs_mma(const espdl_conv_desc &d)
{
    const char *knob = getenv("ESPDL_B200_SMALL_MMA"); // 0: never, always: wherever it can run
    if (d.kernel != ESPDL_KERNEL_AUTO || d.n <= 0 || !conv2d_mma_supported(d) || (knob && *knob == '0'))
        return false;
    if (knob && *knob == 'a')
        return true;
    // What the kernel that would run otherwise takes for a small layer, from the same chains of launches (us): a start-up of 2.5
    // to 4, and 0.33 for every 128 bytes of the reduction that its matrix instructions walk one after the other.  Large layers
    // are decided by this estimate's growth: tile kernels stay below 6 us up to 200 M multiply-adds.
    const int cin_blocks = (d.in_c + 127) / 128, ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    float other;
    if (conv2d_stem_tc_supported(d))
        other = 4.f;
    else if (conv2d_band_tc_supported(d) && d.filter_image_stride == 0)
        other = 6.f;
    else if (d.filter_image_stride == 0 && conv2d_conv_tc_supported(d))
        other = d.stride_h == 1 && d.dilation_h == 1 && cin_blocks == 1 && d.in_c % 32 == 0 && d.in_c != 96 && d.out_c <= 256 ? 3.9f : 2.5f + 0.33f * d.kh * d.kw * cin_blocks;
    else if (conv2d_tc_supported(d))
        // (rows that no TMA store can address leave a tile by warps: 560 products with rows of whole words within 0.6 % of the faster of the two on average, 1.1 % with 9e-6 as for others,
        // 1930x640x176 into rows of 184 5.2 us there, 8.2 here; 2050 with other rows 0.7 %, and lower costs made dozens of them slower: by 2e-6 10352x240x100 took 7.7 there,
        // 5.9 here, 4557x976x53 8.5 / 5.6)
        other = 3.4f + 0.33f * (cin_blocks - 1) + (ops % 16 ? (ops % 4 ? 9e-6f : 4e-6f) * d.n * d.out_h * d.out_w * d.out_c : 0.f);
    else
        // packed operands: two launches, one pass over the unrolled rows; no kernel's start-up is worth waiting for beyond that
        return conv2d_mma_estimate_us(d) < (conv2d_packed_supported(d) ? min(9.f + (d.in_c % 16 == 0 ? 2.5e-7f : 3.5e-6f) * (float)d.n * d.out_h * d.out_w * d.kh * d.kw * d.in_c, conv2d_simt_estimate_us(d))
                                                                       : conv2d_simt_estimate_us(d));
    return conv2d_mma_estimate_us(d) < min(other, 8.f);
}

bool espdl::overlaps(const espdl_conv_desc &d)
{
    const long long es = d.dtype == ESPDL_DTYPE_INT16 ? 2 : 1, ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    const long long in_bytes = (((long long)d.n * d.in_h * d.in_w - 1) * ips + d.in_c) * es, out_bytes = (((long long)d.n * d.out_h * d.out_w - 1) * ops + d.out_c) * es;
    const long long ahead = (long long)((intptr_t)d.output - (intptr_t)d.input);
    if (ahead >= in_bytes || -ahead >= out_bytes)
        return false;
    const long long row = ips * es, into = (ahead % row + row) % row; // of the output into the input's row
    return !(ips == ops && into >= d.in_c * es && into + d.out_c * es <= row);
}

// Can int16 layers run on the warp-level instructions?  Without scratch for packed operands (a caller's choice, or a stream under capture) they do wherever they can.
static bool may_mma16(const espdl_conv_desc &d, bool product)
{
    const char *knob = getenv("ESPDL_B200_MMA16"); // 0: never, always: wherever it can run
    return d.dtype == ESPDL_DTYPE_INT16 && d.kernel == ESPDL_KERNEL_AUTO && d.n > 0 && conv2d_mma16_supported(d) && !(knob && *knob == '0') && !(product && overlaps(d));
}

// int16 on the warp-level instructions, where the other kernels take longer.  Packing and the tile kernel: two launches, the reduction's length, the
// rows packed (more where they and their planes are beyond L2), the results, rows that leave by warps and tiles of 16 columns, the products, and of windows the taps
// and units that groups of eight channels cut; from 4300 layers, 10 % (standard deviation) off them.  2000 others take 0.6 % longer than with the faster kernel of
// the two each time; 3.8 % with the line as it was before either kernel's last changes (us here / there: 49 of 101x104x24 -> 24, 3x3 112 / 305, 120067x48x8 13 / 24; 2028x6400x48 51 / 30).
// The products' rate is a third of theirs: 4096x1024x1024 23 us there, 64 here; 45 of 11x11x256 -> 80, 3x3 20 / 33.
// Eight-element reductions are padded to 64 here, and the CUDA cores read many of them at once (29585x8x1 3.2 / 7.0, 12164x8x17 5.0 /
// 6.0; 5977x8x5 3.6 / 3.3, 1088x8x192 8.9 / 3.8).  A product whose results overwrite its inputs stays with the tile kernel, which has copied those before it writes.
static bool runs_mma16(const espdl_conv_desc &d)
{
    const bool product = conv2d_tc_supported(d);
    if (!may_mma16(d, product))
        return false;
    const char *knob = getenv("ESPDL_B200_MMA16");
    if (knob && *knob == 'a')
        return true;
    const float M = (float)d.n * d.out_h * d.out_w, K = (float)d.kh * d.kw * d.in_c, us = conv2d_mma16_estimate_us(d);
    if (!product && !conv2d_packed_supported(d))
        return us < conv2d_simt_estimate_us(d) && !(K <= 8 && d.out_c <= 64 && M >= 7000);
    const int ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    const float N = (float)d.out_c, beyond = fmaxf(0.0f, M * K - 2.5e7f), by_warps = ops % 8 || d.out_c % 8 ? 1.0f : 0.0f, narrow = d.out_c <= 16 ? 1.0f : 0.0f;
    const float tile = product ? 6.4f + 3.11e-3f * K + 5.4e-7f * M * K + 4.09e-7f * beyond + 1.91e-6f * M * N + 1.95e-9f * M * K * N + by_warps * M * (8.4e-5f + 4.6e-7f * N) + narrow * M * 4.2e-5f
                               : 6.9f + 2.67e-3f * K + 4.33e-7f * M * K + 5.41e-7f * beyond + 2.12e-6f * M * N + 1.65e-9f * M * K * N + by_warps * M * 1.1e-4f + narrow * M * 2.5e-5f +
            1.28e-5f * M * d.kh * d.kw + (d.in_c % 16 ? 6.81e-7f * M * K : 0.0f);
    return us < 0.95f * tile; // 5040x800x96, 5x5: 13.3 us there, 15.5 here; 6400x576x64, 3x3 10.4 / 8.2
}

// Shapes no kernel reads in place, large enough for packed operands to pay (a caller without the scratch gets the CUDA-core kernel).
static bool runs_packed(const espdl_conv_desc &d)
{
    return d.kernel == ESPDL_KERNEL_AUTO && d.n > 0 && !conv2d_stem_tc_supported(d) && !conv2d_band_tc_supported(d) && !conv2d_conv_tc_supported(d) &&
        !conv2d_tc_supported(d) && conv2d_packed_supported(d);
}

// Image i of a batch of products.
static espdl_conv_desc product_of_image(const espdl_conv_desc &d, int i)
{
    const size_t es = d.dtype == ESPDL_DTYPE_INT16 ? 2 : 1;
    const long long ips = d.in_pixel_stride ? d.in_pixel_stride : d.in_c, ops = d.out_pixel_stride ? d.out_pixel_stride : d.out_c;
    espdl_conv_desc one = d;
    one.n = 1, one.filter_image_stride = 0;
    one.input = (const char *)d.input + (size_t)i * d.in_h * d.in_w * ips * es;
    one.filter = (const char *)d.filter + (size_t)i * d.filter_image_stride * es;
    one.output = (char *)d.output + (size_t)i * d.out_h * d.out_w * ops * es;
    return one;
}

// Scratch of a batch of int16 products that runs one after the other on the tile kernel, 0 where one launch of the CUDA cores over all
// of them is as fast.  A slice takes the packing's and the tile kernel's start, 6.3 to 9.1 us, the CUDA cores 0.62 to 0.86 M
// multiply-adds a us, 0.27 M where 32 threads read filter rows a multiple of 64 bytes apart.  One by one against together, us: 8 slices of
// 512x512x512 72 / 3927, 2 of 256x64x256 15 / 17, 64 of 400x32x400 469 / 1199; 64 of 128x64x128 482 / 249, of 400x400x32 576 / 383.
static size_t one_by_one_bytes(const espdl_conv_desc &d)
{
    if (d.kernel != ESPDL_KERNEL_AUTO || d.dtype != ESPDL_DTYPE_INT16 || d.filter_image_stride <= 0 || d.n < 1)
        return 0;
    const espdl_conv_desc one = product_of_image(d, 0);
    const double macs = (double)d.out_h * d.out_w * d.in_c * d.out_c;
    if (4 + d.n * macs / (d.in_c % 32 == 0 && d.out_c >= 128 ? 0.27e6 : 0.7e6) < d.n * (8.5 + macs / 2e8))
        return 0;
    return conv2d_tc_supported(one) ? conv2d_tc_workspace_bytes(one) : (conv2d_packed_supported(one) ? conv2d_packed_workspace_bytes(one) : 0);
}

// The scratch that `s` keeps, at least `need` bytes; null (the call does without) while the stream is being captured, whose graph would
// keep the address, and where there is no memory.  g_ws_mutex is held.
static StreamScratch *stream_scratch(cudaStream_t s, size_t need)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone || cudaStreamGetId(s, &id) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    StreamScratch *slot = g_stream_scratch;
    for (StreamScratch &c : g_stream_scratch) {
        if (c.p && c.stream == id) {
            slot = &c;
            break;
        }
        if (c.used < slot->used)
            slot = &c;
    }
    if (!slot->p || slot->stream != id || slot->bytes < need) {
        // what still runs on the old block ends first: its own stream's work, or that of a stream which may be gone
        if (slot->p && (slot->stream == id ? cudaStreamSynchronize(s) : cudaDeviceSynchronize()) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        if (slot->p)
            cudaFree(slot->p);
        *slot = StreamScratch();
        if (cudaMalloc(&slot->p, need) != cudaSuccess) {
            cudaGetLastError();
            slot->p = nullptr;
            return nullptr;
        }
        slot->stream = id, slot->bytes = need;
    }
    slot->used = ++g_scratch_calls;
    return slot;
}

extern "C" {

int espdl_b200_conv2d_workspace_bytes(const espdl_conv_desc *desc, size_t *bytes)
{
    if (!bytes)
        return ESPDL_ERR_INVALID_ARG;
    *bytes = 0;
    int st = conv_validate(desc);
    if (st)
        return st;
    if (desc->kernel == ESPDL_KERNEL_SIMT || desc->group != 1 || runs_narrow(*desc) || runs_mma(*desc) || (runs_mma16(*desc) && !conv2d_tc_supported(*desc)))
        return ESPDL_OK;
    if (desc->filter_image_stride != 0 && !conv2d_tc_supported(*desc))
        *bytes = one_by_one_bytes(*desc);
    else if (conv2d_tc_supported(*desc))
        *bytes = conv2d_tc_workspace_bytes(*desc);
    else if (runs_packed(*desc))
        *bytes = conv2d_packed_workspace_bytes(*desc);
    return ESPDL_OK;
}

int espdl_b200_conv2d_is_small(const espdl_conv_desc *desc)
{
    // ungrouped it has to beat the tile kernel on grouped rows, 3.4 us and up
    return conv_validate(desc) == ESPDL_OK && runs_mma(*desc) && conv2d_mma_estimate_us(*desc) < 3.6f ? 1 : 0;
}

int espdl_b200_conv2d_ws(const espdl_conv_desc *desc, void *workspace, size_t workspace_bytes, void *stream)
{
    int st = conv_validate(desc);
    if (st)
        return st;
    if (g_device < 0)
        return ESPDL_ERR_NO_DEVICE;
    if (desc->n == 0)
        return ESPDL_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (desc->group != 1) {
        // Depthwise convs have no tensor-core tile kernel
        if (desc->kernel == ESPDL_KERNEL_TCGEN05)
            return ESPDL_ERR_UNSUPPORTED;
        // 3x3 int8 with 16-byte channel runs: the TMA-fed kernels; ESPDL_KERNEL_SIMT asks for the kernels that read global
        // memory directly, which also run small layers (dw_small)
        const bool small = desc->kernel == ESPDL_KERNEL_AUTO && (long long)desc->n * desc->out_h * desc->out_w * desc->out_c < dw_small(desc->stride_h) && desc->kh == 3 &&
            !getenv("ESPDL_B200_DEBUG_WAIT_EXPIRY") && !getenv("ESPDL_B200_DW_TMA_NARROW");
        if (runs_dw_mma(*desc, small))
            return conv2d_dw_mma(*desc, s);
        if (desc->kernel != ESPDL_KERNEL_SIMT && !small && conv2d_dw_tma_supported(*desc))
            return conv2d_dw_tma(*desc, s);
        return conv2d_depthwise(*desc, s);
    }
    if (runs_narrow(*desc))
        return conv2d_narrow(*desc, s);
    if (runs_mma(*desc))
        return conv2d_mma(*desc, s);
    if (runs_mma16(*desc)) {
        // products declare the tile kernel's scratch whichever kernel runs them, and are refused without it or where it is not aligned
        const size_t need = conv2d_tc_supported(*desc) ? conv2d_tc_workspace_bytes(*desc) : 0;
        return need > workspace_bytes || (need && (!workspace || (uintptr_t)workspace % 16)) ? ESPDL_ERR_INVALID_ARG : conv2d_mma16(*desc, s);
    }
    if (desc->kernel != ESPDL_KERNEL_SIMT && conv2d_stem_tc_supported(*desc))
        return conv2d_stem_tc(*desc, s); // 3x3 stride-2 RGB first layer: banded-filter tensor-core kernel
    if (desc->filter_image_stride != 0) {
        // a batch of matrix products: image i multiplies by the filter at filter + i * filter_image_stride
        if (desc->kh != 1 || desc->kw != 1 || desc->stride_h != 1 || desc->stride_w != 1 || desc->pad_top || desc->pad_bottom ||
            desc->pad_left || desc->pad_right || desc->filter_image_stride < 0)
            return ESPDL_ERR_INVALID_ARG;
        if (desc->kernel != ESPDL_KERNEL_SIMT && conv2d_tc_supported(*desc))
            return conv2d_tc(*desc, workspace, workspace_bytes, s);
        if (desc->kernel == ESPDL_KERNEL_TCGEN05)
            return ESPDL_ERR_UNSUPPORTED;
        const size_t one_by_one = one_by_one_bytes(*desc);
        if (one_by_one && workspace && workspace_bytes >= one_by_one) {
            for (int i = 0; i < desc->n && !st; i++) {
                const espdl_conv_desc one = product_of_image(*desc, i);
                st = conv2d_tc_supported(one) ? conv2d_tc(one, workspace, workspace_bytes, s) : conv2d_packed(one, workspace, workspace_bytes, s);
            }
            return st;
        }
        return conv2d_simt(*desc, s); // all products in one launch (one per image: 128 launches, 1.5 ms, for the attention of 64 images)
    }
    if (desc->kernel != ESPDL_KERNEL_SIMT && conv2d_band_tc_supported(*desc))
        return conv2d_band_tc(*desc, s); // 3x3 with 8 or 16 input channels: banded filter over 128-byte row windows
    const bool conv_tc_ok = conv2d_conv_tc_supported(*desc);
    if (conv_tc_ok && desc->kernel != ESPDL_KERNEL_SIMT)
        return conv2d_conv_tc(*desc, s); // filters larger than 1x1 (or strided): implicit GEMM over the taps
    const bool tc_ok = conv2d_tc_supported(*desc);
    if (desc->kernel == ESPDL_KERNEL_TCGEN05 && !tc_ok)
        return ESPDL_ERR_UNSUPPORTED;
    if (tc_ok && desc->kernel != ESPDL_KERNEL_SIMT) {
        const size_t need = conv2d_tc_workspace_bytes(*desc);
        if (need > workspace_bytes || (need && !workspace))
            return ESPDL_ERR_INVALID_ARG;
        return conv2d_tc(*desc, workspace, workspace_bytes, s);
    }
    if (runs_packed(*desc) && workspace && workspace_bytes >= conv2d_packed_workspace_bytes(*desc))
        return conv2d_packed(*desc, workspace, workspace_bytes, s);
    if (runs_packed(*desc) && may_mma16(*desc, false) && conv2d_mma16_estimate_us(*desc) < conv2d_simt_estimate_us(*desc))
        return conv2d_mma16(*desc, s);
    return conv2d_simt(*desc, s);
}

int espdl_b200_conv2d(const espdl_conv_desc *desc, void *stream)
{
    size_t need = 0;
    int st = espdl_b200_conv2d_workspace_bytes(desc, &need);
    if (st)
        return st;
    if (need == 0)
        return espdl_b200_conv2d_ws(desc, nullptr, 0, stream);
    if (g_device >= 0 && runs_mma16(*desc))
        return conv2d_mma16(*desc, (cudaStream_t)stream);
    std::lock_guard<std::mutex> lock(g_ws_mutex);
    if (!conv2d_tc_supported(*desc)) { // the CUDA cores run it as it is, the scratch only makes it faster
        StreamScratch *scratch = stream_scratch((cudaStream_t)stream, need);
        return espdl_b200_conv2d_ws(desc, scratch ? scratch->p : nullptr, scratch ? scratch->bytes : 0, stream);
    }
    // int16 Gemms and pointwise convs: the cached scratch is shared by all of them, which are serialised on the host here and must be
    // ordered on the device by the caller's streams.
    if (need > g_ws_bytes) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (may_mma16(*desc, true) && cudaStreamIsCapturing((cudaStream_t)stream, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone)
            return conv2d_mma16(*desc, (cudaStream_t)stream); // nothing can be allocated now
        if (g_ws) {
            ESPDL_CUDA_TRY(cudaDeviceSynchronize());
            ESPDL_CUDA_TRY(cudaFree(g_ws));
            g_ws = nullptr;
            g_ws_bytes = 0;
        }
        cudaError_t e = cudaMalloc(&g_ws, need);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return ESPDL_ERR_NO_MEM;
        }
        g_ws_bytes = need;
    }
    return espdl_b200_conv2d_ws(desc, g_ws, g_ws_bytes, stream);
}

int espdl_b200_gemm_scatter(const espdl_conv_desc *desc, void *const *peer_outputs, int n_peers, void *stream)
{
    if (n_peers < 0 || n_peers > 7 || (n_peers > 0 && !peer_outputs))
        return ESPDL_ERR_INVALID_ARG;
    const int st = conv_validate(desc);
    if (st)
        return st;
    if (g_device < 0)
        return ESPDL_ERR_NO_DEVICE;
    if (desc->dtype != ESPDL_DTYPE_INT8 || desc->lut || desc->residual || desc->filter_image_stride != 0 || !conv2d_tc_supported(*desc))
        return ESPDL_ERR_UNSUPPORTED;
    if (desc->n == 0)
        return ESPDL_OK;
    long long delta[7] = {0, 0, 0, 0, 0, 0, 0};
    for (int i = 0; i < n_peers; i++) {
        if (!peer_outputs[i] || ((uintptr_t)peer_outputs[i] % 16) != ((uintptr_t)desc->output % 16))
            return set_error_text(ESPDL_ERR_INVALID_ARG, "espdl_b200_gemm_scatter: peer output %d is null or aligned differently from the local output", i);
        delta[i] = (long long)((intptr_t)peer_outputs[i] - (intptr_t)desc->output);
    }
    return conv2d_tc(*desc, nullptr, 0, (cudaStream_t)stream, delta, n_peers);
}

int espdl_b200_ipc_export(const void *dptr, void *handle64)
{
    if (!dptr || !handle64)
        return ESPDL_ERR_INVALID_ARG;
    static_assert(sizeof(cudaIpcMemHandle_t) == 64, "the C ABI passes IPC handles as 64 bytes");
    ESPDL_CUDA_TRY(cudaIpcGetMemHandle((cudaIpcMemHandle_t *)handle64, const_cast<void *>(dptr)));
    return ESPDL_OK;
}

int espdl_b200_ipc_open(const void *handle64, void **dptr)
{
    if (!handle64 || !dptr)
        return ESPDL_ERR_INVALID_ARG;
    cudaIpcMemHandle_t h;
    memcpy(&h, handle64, sizeof(h));
    ESPDL_CUDA_TRY(cudaIpcOpenMemHandle(dptr, h, cudaIpcMemLazyEnablePeerAccess));
    return ESPDL_OK;
}

int espdl_b200_ipc_close(void *dptr)
{
    if (dptr)
        ESPDL_CUDA_TRY(cudaIpcCloseMemHandle(dptr));
    return ESPDL_OK;
}

int espdl_b200_fused_block(const espdl_block_desc *desc, void *stream)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    if (!desc->input || !desc->output || !desc->dw_filter || !desc->project_filter || desc->n < 0)
        return ESPDL_ERR_INVALID_ARG;
    if (desc->n == 0)
        return ESPDL_OK;
    // a depthwise -> pointwise pair (no expand conv) has a kernel of its own
    if (!desc->expand_filter && fused_dwpw_supported(*desc, false))
        return fused_dwpw(*desc, (cudaStream_t)stream);
    return fused_block_tc(*desc, (cudaStream_t)stream);
}

int espdl_b200_image_preprocess(const espdl_image_desc *desc, void *stream)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    return image_preprocess(*desc, (cudaStream_t)stream);
}

int espdl_b200_detect_candidates(const espdl_detect_desc *desc, void *stream)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    return detect_candidates(*desc, (cudaStream_t)stream);
}

int espdl_b200_reduce(const espdl_reduce_desc *desc, void *stream)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    return reduce_op(*desc, (cudaStream_t)stream);
}

int espdl_b200_pad(const espdl_pad_desc *desc, void *stream)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    return pad_op(*desc, (cudaStream_t)stream);
}

int espdl_b200_fused_block_supported(const espdl_block_desc *desc)
{
    if (!desc)
        return ESPDL_ERR_INVALID_ARG;
    if (desc->reserved[0] == 0 && fused_dwpw_supported(*desc, false))
        return ESPDL_OK;
    return fused_block_supported(*desc) ? ESPDL_OK : ESPDL_ERR_UNSUPPORTED;
}

} // extern "C"
