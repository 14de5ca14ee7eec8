/* A stand-in for libespdl_b200.so that needs no GPU: device memory is host memory, streams, events and graphs are numbers, no
 * operator computes anything, and the calls whose order and arguments matter are written to $FAKE_DEVICE_LOG, a line each.
 * Questions about kernels (scratch, small layers) go to the real library ($REAL_DEVICE_LIB), which answers them on the host.
 * Operators without a line of their own are generated by the test from the host library's undefined symbols. */
#include <dlfcn.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "espdl_b200.h"

static FILE *log_file;
static void *real;
static int scope, overlapped = 1;
static long handles = 1;

static void line(const char *fmt, ...)
{
    if (!log_file)
        log_file = fopen(getenv("FAKE_DEVICE_LOG"), "w");
    va_list ap;
    va_start(ap, fmt);
    vfprintf(log_file, fmt, ap);
    va_end(ap);
    fputc('\n', log_file);
    fflush(log_file);
}

static void *real_symbol(const char *name)
{
    if (!real)
        real = dlopen(getenv("REAL_DEVICE_LIB"), RTLD_NOW | RTLD_LOCAL);
    return real ? dlsym(real, name) : NULL;
}

int espdl_b200_init(int device) { return device; }
const char *espdl_b200_strerror(int s) { return s ? "error" : "ok"; }
const char *espdl_b200_last_error(void) { return ""; }

int espdl_b200_arena_alloc(size_t bytes, void **p)
{
    const char *limit = getenv("FAKE_ARENA_LIMIT");
    line("alloc bytes=%zu", bytes);
    if (limit && bytes > strtoull(limit, NULL, 10))
        return ESPDL_ERR_NO_MEM;
    *p = aligned_alloc(256, (bytes + 511) / 256 * 256);
    return *p ? ESPDL_OK : ESPDL_ERR_NO_MEM;
}
int espdl_b200_arena_free(void *p) { free(p); return 0; }
int espdl_b200_host_alloc(size_t bytes, void **p) { *p = aligned_alloc(256, (bytes + 511) / 256 * 256); return 0; }
int espdl_b200_host_free(void *p) { free(p); return 0; }
int espdl_b200_upload(void *d, const void *s, size_t n, void *st) { line("upload stream=%p dst=%p", st, d); memcpy(d, s, n); return 0; }
int espdl_b200_download(void *d, const void *s, size_t n, void *st) { line("download stream=%p src=%p", st, s); memcpy(d, s, n); return 0; }
int espdl_b200_memset(void *d, int v, size_t n, void *st) { (void)st; memset(d, v, n); return 0; }

int espdl_b200_stream_create(void **s)
{
    const char *limit = getenv("FAKE_STREAM_LIMIT");
    static int made;
    if (limit && made >= atoi(limit))
        return ESPDL_ERR_CUDA;
    made++;
    *s = (void *)(handles++);
    return 0;
}
int espdl_b200_stream_destroy(void *s) { line("stream_destroy stream=%p", s); return 0; }
int espdl_b200_event_create(void **e) { *e = (void *)(handles++); return 0; }
int espdl_b200_event_record(void *e, void *s) { line("record event=%p stream=%p", e, s); return 0; }
int espdl_b200_stream_wait_event(void *s, void *e) { line("wait event=%p stream=%p", e, s); return 0; }
int espdl_b200_graph_begin(void *s) { line("graph_begin stream=%p", s); return 0; }
int espdl_b200_graph_end(void *s, void **g) { *g = (void *)(handles++); line("graph_end stream=%p graph=%p", s, *g); return 0; }
int espdl_b200_graph_launch(void *g, void *s) { line("graph_launch graph=%p stream=%p", g, s); return 0; }
int espdl_b200_graph_destroy(void *g) { line("graph_destroy graph=%p", g); return 0; }
void espdl_b200_model_scope(int enter) { scope += enter ? 1 : -1; }
void espdl_b200_overlap(int on) { overlapped = on; }

int espdl_b200_conv2d_workspace_bytes(const espdl_conv_desc *d, size_t *bytes)
{
    return ((int (*)(const espdl_conv_desc *, size_t *))real_symbol("espdl_b200_conv2d_workspace_bytes"))(d, bytes);
}
int espdl_b200_conv2d_is_small(const espdl_conv_desc *d) { return ((int (*)(const espdl_conv_desc *))real_symbol("espdl_b200_conv2d_is_small"))(d); }

int espdl_b200_conv2d_ws(const espdl_conv_desc *d, void *ws, size_t ws_bytes, void *s)
{
    size_t need = 0;
    espdl_b200_conv2d_workspace_bytes(d, &need);
    line("conv stream=%p ws=%p ws_bytes=%zu need=%zu scope=%d overlap=%d in=%p filter=%p out=%p n=%d m=%d k=%d oc=%d image_stride=%d", s, ws, ws_bytes, need, scope,
         overlapped, d->input, d->filter, d->output, d->n, d->out_h * d->out_w, d->in_c * d->kh * d->kw, d->out_c, d->filter_image_stride);
    return 0;
}
int espdl_b200_copy(const espdl_copy_desc *d, void *s) { line("copy stream=%p src=%p dst=%p scope=%d", s, d->src, d->dst, scope); return 0; }
