// Capturing a model's plan as a CUDA graph, with independent branches side by side.
//
// A graph replayed as one chain runs a launch at a time.  With one image most launches occupy a fraction of the SMs for a few
// microseconds, and networks with branches (a detector's heads, the parallel streams of a re-identification block) then
// take the sum of all launches instead of the longest path through them.  Here every step depends only on the earlier
// steps whose device memory it meets (read after write, write after read, write after write, at byte level, channel slices by
// their columns), steps are dealt out to a few capture streams accordingly, and events carry the dependencies that
// cross streams.  Model::build says where branches are used.
#include <algorithm>
#include <cstring>

#include "dl_model_base.hpp"
#include "espdl_b200.h"

namespace dl {

namespace {

struct Access {
    const char *base = nullptr;
    size_t row = 0, pitch = 0, rows = 1; // pitch 0: one dense run of `row` bytes
    bool write = false;
    const char *end() const { return base + (pitch ? (rows - 1) * pitch : 0) + row; }
};

bool overlap(const Access &a, const Access &b)
{
    if (a.end() <= b.base || b.end() <= a.base)
        return false;
    if (!a.pitch || a.pitch != b.pitch)
        return true;
    // rows of the same pitch: columns [0, a.row) against [d, d + b.row), wrapping at the pitch
    const ptrdiff_t diff = b.base - a.base, p = (ptrdiff_t)a.pitch;
    const size_t d = (size_t)(((diff % p) + p) % p);
    return d < a.row || d + b.row > a.pitch;
}

Access access_of(TensorBase *t, bool write)
{
    Access a;
    a.base = (const char *)t->device, a.write = write;
    const size_t es = dtype_sizeof(t->dtype);
    if (t->row_stride) {
        a.row = (size_t)t->shape.back() * es, a.pitch = (size_t)t->row_stride * es;
        a.rows = a.row ? t->get_bytes() / a.row : 0;
    } else {
        a.row = t->get_bytes();
    }
    return a;
}

struct Item {
    int step = -1;            // a step of the plan, or
    TensorBase *io = nullptr; // an upload / download of this tensor
    bool upload = false;
    std::vector<Access> accesses;
    std::vector<int> after; // the items it directly depends on
    int stream = 0;
    bool chained = false; // its only dependency is the item before it on its stream
    bool event = false;   // items on other streams wait for it
};

} // namespace

// Steps [first, last) of the plan - and, with `io`, the copies of the graph inputs in front and of the outputs behind - as an
// executable graph.
esp_err_t Model::capture_plan(int first, int last, bool io, void **graph)
{
    ModelContext *ctx = m_model_context;
    const char *arena = (const char *)m_arena, *arena_end = arena + m_arena_bytes;
    std::vector<Item> items;
    auto copy_item = [&](TensorBase *t, bool upload) {
        Item it;
        it.io = t, it.upload = upload;
        it.accesses.push_back(access_of(t, upload));
        items.push_back(it);
    };
    if (io)
        for (auto &kv : m_inputs)
            if (kv.second->data)
                copy_item(kv.second, true);
    for (int s = first; s < last; s++) {
        Item it;
        it.step = s;
        auto add = [&](const std::string &name, bool write) {
            TensorBase *t = ctx->get_tensor(name);
            if (t && t->device && (const char *)t->device >= arena && (const char *)t->device < arena_end)
                it.accesses.push_back(access_of(t, write));
        };
        for (const std::string &name : m_module_inputs[s]) add(name, false);
        for (const std::string &name : m_module_outputs[s]) add(name, true);
        if (m_execution_plan[s]->workspace_bytes(ctx) && ctx->workspace) { // the scratch that steps share
            Access a;
            a.base = (const char *)ctx->workspace, a.row = ctx->workspace_bytes, a.write = true;
            it.accesses.push_back(a);
        }
        items.push_back(it);
    }
    if (io)
        for (auto &kv : m_outputs)
            if (kv.second->data)
                copy_item(kv.second, false);

    // direct dependencies: walking back from an item, every earlier one that it meets and that is no ancestor of a later such
    const int n = (int)items.size();
    const int words = (n + 63) / 64;
    std::vector<uint64_t> ancestors((size_t)n * words, 0);
    auto is_ancestor = [&](int i, int j) { return (ancestors[(size_t)j * words + i / 64] >> (i % 64)) & 1; };
    for (int j = 0; j < n; j++)
        for (int i = j - 1; i >= 0; i--) {
            if (is_ancestor(i, j))
                continue;
            bool meets = !m_branches;
            for (const Access &a : items[j].accesses)
                for (const Access &b : items[i].accesses)
                    meets = meets || ((a.write || b.write) && overlap(a, b));
            if (!meets)
                continue;
            items[j].after.push_back(i);
            for (int w = 0; w < words; w++) ancestors[(size_t)j * words + w] |= ancestors[(size_t)i * words + w];
            ancestors[(size_t)j * words + i / 64] |= 1ull << (i % 64);
        }
    // streams: behind the latest dependency that is still the end of its stream, else on a stream whose end is an ancestor, else on a
    // fresh one, else on the one that ended longest ago
    const int limit = m_branches ? MAX_BRANCHES : 1;
    std::vector<int> tail(limit, -1);
    for (int j = 0; j < n; j++) {
        int s = -1;
        for (int d : items[j].after) // descending
            if (s < 0 && tail[items[d].stream] == d)
                s = items[d].stream;
        for (int k = 0; k < limit && s < 0; k++)
            if (tail[k] >= 0 && is_ancestor(tail[k], j))
                s = k;
        for (int k = 0; k < limit && s < 0; k++)
            if (tail[k] < 0)
                s = k;
        if (s < 0)
            s = (int)(std::min_element(tail.begin(), tail.end()) - tail.begin());
        items[j].chained = items[j].after.empty() ? tail[s] < 0 && s == 0 : items[j].after.size() == 1 && tail[s] == items[j].after[0];
        items[j].stream = s, tail[s] = j;
        for (int d : items[j].after)
            if (items[d].stream != s)
                items[d].event = true;
    }
    while ((int)m_branch_streams.size() < limit - 1) {
        void *s = nullptr;
        const int made = espdl_b200_stream_create(&s);
        if (made) {
            m_status = made;
            return ESP_FAIL;
        }
        m_branch_streams.push_back(s);
    }
    std::vector<void *> streams = {ctx->stream};
    streams.insert(streams.end(), m_branch_streams.begin(), m_branch_streams.end());
    std::vector<void *> events(n + 1, nullptr); // events[n]: the start
    int st = espdl_b200_graph_begin(ctx->stream);
    if (st) {
        m_status = st;
        return ESP_FAIL;
    }
    auto record = [&](int i, void *stream) {
        if (!st) st = espdl_b200_event_create(&events[i]);
        if (!st) st = espdl_b200_event_record(events[i], stream);
    };
    if (limit > 1)
        record(n, streams[0]);
    std::vector<bool> joined(limit, false);
    joined[0] = true;
    for (int j = 0; j < n && !st; j++) {
        const Item &it = items[j];
        void *stream = streams[it.stream];
        if (!joined[it.stream]) { // a stream joins the capture by waiting for one of its events
            st = espdl_b200_stream_wait_event(stream, events[n]);
            joined[it.stream] = true;
        }
        for (int d : it.after)
            if (!st && items[d].stream != it.stream)
                st = espdl_b200_stream_wait_event(stream, events[d]);
        if (!it.chained || m_plain_launches)
            espdl_b200_overlap(0); // joins: plain edges
        if (!st && it.io) {
            st = it.upload ? espdl_b200_upload(it.io->device, it.io->data, it.io->get_bytes(), stream)
                           : espdl_b200_download(it.io->data, it.io->device, it.io->get_bytes(), stream);
        } else if (!st) {
            void *own = ctx->stream;
            ctx->stream = stream;
            if (execute(it.step, it.step + 1) != ESP_OK)
                st = m_status ? m_status : ESPDL_ERR_CUDA;
            ctx->stream = own;
        }
        espdl_b200_overlap(1);
        if (it.event)
            record(j, stream);
    }
    for (int k = 1; k < limit && !st; k++)
        if (tail[k] >= 0) {
            if (!events[tail[k]])
                record(tail[k], streams[k]);
            if (!st) st = espdl_b200_stream_wait_event(streams[0], events[tail[k]]);
        }
    const int end = espdl_b200_graph_end(ctx->stream, graph);
    for (void *e : events)
        if (e)
            espdl_b200_event_destroy(e);
    if (st || end) {
        m_status = st ? st : end;
        return ESP_FAIL;
    }
    return ESP_OK;
}

} // namespace dl
