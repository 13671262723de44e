// Engine lifecycle, workspace layout and the C ABI of the k-truss path.
//
// kt_ktruss / kt_decompose take host buffers like the reference's ktruss() (kernel.h:12):
// they copy the graph to the device, run the device pipeline and copy the result back.
// kt_engine_* take device buffers and leave the data in HBM.

#include <algorithm>
#include <chrono>
#include <cstring>
#include <mutex>
#include <vector>

#include "kt_device.cuh"
#include "kt_engine.h"

namespace kt {

int check_cuda(cudaError_t err, const char* what) {
    if (err == cudaSuccess) return KT_OK;
    int code = (err == cudaErrorMemoryAllocation) ? KT_ERR_DEVICE_ALLOC
               : (err == cudaErrorNoDevice || err == cudaErrorInsufficientDriver) ? KT_ERR_NO_DEVICE
                                                                                 : KT_ERR_CUDA;
    return fail(code, "%s: %s", what, cudaGetErrorString(err));
}

int check_launch(kt_engine*, const char* what) { return check_cuda(cudaGetLastError(), what); }

namespace {

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

struct Carver {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t count) {
        T* p = reinterpret_cast<T*>(base ? base + off : nullptr);
        off += align_up(sizeof(T) * (count ? count : 1));
        return p;
    }
};

}  // namespace

// Lays out every array of the engine for the given capacity inside `base`; with base == nullptr
// it only measures.  `staging` adds the host-transfer buffers of the host-buffer entry points.
size_t carve(kt_engine* e, char* base, uint32_t n, uint64_t N, bool staging) {
    const uint64_t m = N / 2 + 1;
    const uint64_t keys = std::max<uint64_t>(N, n);
    // look-back words for sorts of any size up to the capacity
    const uint64_t look_cap = std::max(look_words(keys), look_words(std::min(keys, kSmallSort)));
    Carver c{base};
    e->key_a = c.take<uint64_t>(keys);
    e->key_b = c.take<uint64_t>(keys);
    e->val_a = c.take<uint32_t>(N);
    e->val_b = c.take<uint32_t>(N);
    e->deg = c.take<uint32_t>(n);
    e->rank = c.take<uint32_t>(n);
    e->s_ptr = c.take<uint32_t>((size_t)n + 1);
    e->s_len = c.take<uint32_t>((size_t)n + 1);
    e->s_split = c.take<uint32_t>((size_t)n + 1);
    e->o_ptr = c.take<uint32_t>((size_t)n + 1);
    e->s_col = c.take<uint32_t>(N);
    e->s_eid = c.take<uint32_t>(N);
    e->o_col = c.take<uint32_t>(m);
    e->o_fence = c.take<uint32_t>(m / 32 + 2);  // every 32nd oriented column
    e->e_src = c.take<uint32_t>(m);
    e->sup = c.take<uint32_t>(m + 4);  // read four at a time
    e->rnd = c.take<uint32_t>(m);
    e->tr = c.take<uint32_t>(m);
    e->q0 = c.take<uint32_t>(m);
    e->q1 = c.take<uint32_t>(m);
    e->cap_chunks = (uint32_t)std::min<uint64_t>(m + 4096, 0xfffff000u);
    e->chunks0 = c.take<uint4>(e->cap_chunks);
    e->chunks1 = c.take<uint4>(e->cap_chunks);
    e->cap_rounds = (uint32_t)std::min<uint64_t>(m + 2, 1u << 22);
    e->round_size = c.take<uint32_t>(e->cap_rounds);
    e->round_level = c.take<uint32_t>(e->cap_rounds);
    e->round_ns = c.take<uint32_t>(e->cap_rounds);
    e->cap_levels = (uint32_t)std::min<uint64_t>(m + 2, 1u << 16);
    e->level_k = c.take<uint32_t>(e->cap_levels);
    e->level_alive = c.take<uint32_t>(e->cap_levels);
    e->level_ns = c.take<uint32_t>(e->cap_levels);
    e->level_front = c.take<uint32_t>(e->cap_levels);
    e->sel_stats = c.take<uint32_t>(32);
    e->sel_part = c.take<uint64_t>((size_t)kSelMaxBlocks * 10);
    e->sel_feat = c.take<float>(KT_SELECTOR_FEATURES);
    e->sel_choice = c.take<uint32_t>(1);
    e->look = c.take<unsigned long long>(look_cap);
    e->look_cap = look_cap;
    e->digit_counts = c.take<uint32_t>(kCountWords);
    if (staging) {
        e->in_src = c.take<uint32_t>(N);
        e->in_dst = c.take<uint32_t>(N);
        e->out_u32 = c.take<uint32_t>(N);
        e->out_u8 = c.take<uint8_t>(N);
    }
    return c.off;
}

void drop_replay(kt_engine* e) {
    if (e->replay) cudaGraphExecDestroy(e->replay);
    e->replay = nullptr;
    e->replay_direct = false;
}

// Records a successful device-buffer call for kt_engine_replay; a different call drops the
// captured pipeline of the previous one.
void remember(kt_engine* e, const kt_engine::LastCall& c) {
    const kt_engine::LastCall& l = e->last;
    if (l.kind != c.kind || l.src != c.src || l.dst != c.dst || l.entries != c.entries || l.n != c.n ||
        l.truss != c.truss || l.k_max != c.k_max || l.k != c.k || l.keep != c.keep)
        drop_replay(e);
    e->last = c;
    e->last.list_need = e->list_need;
}

void forget(kt_engine* e) {
    drop_replay(e);
    e->last = kt_engine::LastCall{};
}

int reserve(kt_engine* e, uint32_t max_nodes, uint64_t max_entries) {
    if (max_nodes <= e->cap_nodes && max_entries <= e->cap_entries && e->arena) return KT_OK;
    max_nodes = std::max(max_nodes, e->cap_nodes);
    max_entries = std::max(max_entries, e->cap_entries);
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    if (e->arena) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize before resize"))) return rc;
        drop_replay(e);  // the captured pipeline points into the old workspace
        cudaFree(e->arena);
        e->arena = nullptr;
        e->arena_bytes = 0;
    }
    const size_t bytes = carve(e, nullptr, max_nodes, max_entries, true);
    void* p = nullptr;
    if ((rc = check_cuda(alloc_device(e, &p, bytes), "allocate engine workspace"))) {
        e->cap_nodes = 0;
        e->cap_entries = 0;
        return rc;
    }
    e->arena = p;
    e->arena_bytes = bytes;
    carve(e, static_cast<char*>(p), max_nodes, max_entries, true);
    // the selector's block ticket starts at zero; its last block clears it again on every call
    if ((rc = check_cuda(cudaMemsetAsync(e->sel_stats, 0, sizeof(uint32_t) * 32, e->stream), "clear ticket")))
        return rc;
    e->cap_nodes = max_nodes;
    e->cap_entries = max_entries;
    reserve_small_lists(e, max_entries / 2);
    return KT_OK;
}

}  // namespace kt

using kt::check_cuda;
using kt::fail;

namespace {

std::mutex g_default_mu;
kt_engine* g_default = nullptr;

// The engine used by the host-buffer entry points (device 0, created on first use).
int default_engine(kt_engine** out) {
    std::lock_guard<std::mutex> lock(g_default_mu);
    if (!g_default) {
        int rc = kt_engine_create(0, &g_default);
        if (rc) return rc;
    }
    *out = g_default;
    return KT_OK;
}

double now_ms() {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

int record_start(kt_engine* e) {
    e->emit_timed = false;
    return check_cuda(cudaEventRecord(e->ev_start, e->stream), "record start");
}

int record(kt_engine* e, cudaEvent_t ev) { return check_cuda(cudaEventRecord(ev, e->stream), "record event"); }

// Ends a call: the stop event, then the control block to the host (the call's one read, unless its
// triangle count was needed); waits for both and returns an input error.
int record_stop(kt_engine* e) {
    int rc = check_cuda(cudaEventRecord(e->ev_stop, e->stream), "record stop");
    if (rc) return rc;
    e->ctrl_fresh = false;
    if ((rc = kt::sync_and_check(e))) return rc;
    e->ctrl_fresh = true;
    float a = 0, b = 0, c = 0, d = 0;
    if ((rc = check_cuda(cudaEventElapsedTime(&a, e->ev_start, e->ev_select), "elapsed time")) ||
        (rc = check_cuda(cudaEventElapsedTime(&d, e->ev_select, e->ev_built), "elapsed time")) ||
        (rc = check_cuda(cudaEventElapsedTime(&b, e->ev_built, e->ev_counted), "elapsed time")) ||
        (rc = check_cuda(cudaEventElapsedTime(&c, e->ev_counted, e->ev_stop), "elapsed time")))
        return rc;
    e->stats.build_ms = a;
    e->stats.select_ms = d;
    e->stats.support_ms = b;
    e->stats.peel_ms = c;
    e->stats.last_ms = a + b + c + d;
    e->stats.emit_ms = 0;
    if (e->emit_timed &&
        (rc = check_cuda(cudaEventElapsedTime(&e->stats.emit_ms, e->ev_peeled, e->ev_stop), "elapsed time")))
        return rc;
    e->emit_timed = false;
    return KT_OK;
}

// Device time of the input and output copies of a host-buffer call (events ev_copy[0..3]; the
// stream must have drained).
int copy_times(kt_engine* e) {
    int rc = check_cuda(cudaEventElapsedTime(&e->stats.copy_in_ms, e->ev_copy[0], e->ev_copy[1]), "elapsed time");
    if (!rc) rc = check_cuda(cudaEventElapsedTime(&e->stats.copy_out_ms, e->ev_copy[2], e->ev_copy[3]), "elapsed time");
    return rc;
}

int fill_graph_stats(kt_engine* e) {
    e->stats.num_nodes = e->n;
    e->stats.num_edges = e->m;
    e->stats.kernel_launches = e->launches;
    return KT_OK;
}

// A batch's vertex ranges and where its graphs' k_max go.
struct Batch {
    const uint32_t* offsets;
    uint32_t graphs;
    uint32_t* k_max;
};

// Device pipeline for the decomposition (inputs on the device).
int run_decompose(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n,
                  uint32_t* d_truss, uint32_t* d_k_max, const Batch* batch = nullptr) {
    int rc;
    if ((rc = record_start(e))) return rc;
    // (the selector's statistics need a checked graph)
    if ((rc = kt::build_graph(e, d_src, d_dst, entries, n, e->selector != nullptr))) return rc;
    if ((rc = record(e, e->ev_select))) return rc;
    if ((rc = kt::select_schedule(e))) return rc;
    if ((rc = record(e, e->ev_built))) return rc;
    if ((rc = kt::count_support(e))) return rc;
    if ((rc = record(e, e->ev_counted))) return rc;
    if ((rc = kt::peel_decompose(e))) return rc;
    if ((rc = record(e, e->ev_peeled))) return rc;
    e->emit_timed = true;
    if ((rc = kt::emit_truss_per_entry(e, d_truss, d_k_max))) return rc;
    if (batch && (rc = kt::emit_graph_kmax(e, d_src, d_dst, batch->offsets, batch->graphs, d_truss, batch->k_max)))
        return rc;
    if ((rc = record_stop(e))) return rc;
    return fill_graph_stats(e);
}

// The single-k pipeline after the build, by the engine's variant: the engine's peel (oriented by
// degree or by index; recount all = the schedule's recount rounds, affected = decrements only), or
// count-and-delete passes (undirected capped counts; tiled counts).
int single_k_body(kt_engine* e, uint32_t k) {
    int rc;
    const kt_variant& v = e->variant;
    if (v.input_format == KT_FORMAT_TILED_COOCSR) return kt::ktruss_tiled(e, k, v.recount == KT_RECOUNT_ALL,
                                                                        v.directedness == KT_UNDIRECTED);
    if (v.directedness == KT_UNDIRECTED) return kt::ktruss_undirected(e, k, v.recount == KT_RECOUNT_ALL, 8);
    if (k >= 3 && (rc = kt::count_support(e))) return rc;
    if (!e->trusted && (rc = record(e, e->ev_counted))) return rc;
    const uint32_t saved = e->sched.recount_percent;
    if (v.recount == KT_RECOUNT_AFFECTED) e->sched.recount_percent = 0;
    rc = kt::peel_single_k(e, k);
    e->sched.recount_percent = saved;
    return rc;
}

// Whether the variant's single-k pipeline runs without host reads after the build (capturable).
bool single_k_capturable(const kt_engine* e) {
    return e->variant.input_format != KT_FORMAT_TILED_COOCSR && e->variant.directedness != KT_UNDIRECTED;
}

int run_ktruss(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t entries, uint32_t n, uint32_t k,
               uint8_t* d_keep) {
    int rc;
    if ((rc = record_start(e))) return rc;
    e->orient_by_index = e->variant.directedness == KT_DIRECTED_BY_INDEX;
    rc = kt::build_graph(e, d_src, d_dst, entries, n, !single_k_capturable(e));
    e->orient_by_index = false;
    if (rc) return rc;
    if ((rc = record(e, e->ev_select))) return rc;
    if ((rc = record(e, e->ev_built))) return rc;
    if ((rc = single_k_body(e, k))) return rc;
    if (!single_k_capturable(e) && (rc = record(e, e->ev_counted))) return rc;
    if ((rc = kt::emit_keep(e, d_keep))) return rc;
    if ((rc = record_stop(e))) return rc;
    return fill_graph_stats(e);
}

// The device pipeline of the remembered call, for a trusted run (its input passed the checks
// of the call itself): no host reads, so it can be captured into a CUDA graph.
int replay_pipeline(kt_engine* e) {
    const kt_engine::LastCall& c = e->last;
    int rc;
    if (c.kind == 1 && (rc = kt::build_graph(e, c.src, c.dst, c.entries, c.n, false))) return rc;
    if (c.kind == 1 && (rc = kt::select_schedule(e))) return rc;  // on the device: capturable
    if (c.kind == 1)
        return (rc = kt::count_support(e)) || (rc = kt::peel_decompose(e)) ||
                       (rc = kt::emit_truss_per_entry(e, c.truss, c.k_max))
                   ? rc
                   : KT_OK;
    e->orient_by_index = e->variant.directedness == KT_DIRECTED_BY_INDEX;
    rc = kt::build_graph(e, c.src, c.dst, c.entries, c.n, false);
    e->orient_by_index = false;
    if (rc || (rc = single_k_body(e, c.k)) || (rc = kt::emit_keep(e, c.keep))) return rc;
    return KT_OK;
}

// Captures the remembered call's pipeline once (CUDA graph; if the capture is refused, later
// replays launch the pipeline directly), then launches it between the start and stop events.
int replay(kt_engine* e, int sync) {
    if (!e->last.kind) return fail(KT_ERR_INVALID_ARG, "kt_engine_replay: no decomposition or single-k call to repeat");
    int rc;
    if (!e->replay && !e->replay_direct && e->last.kind == 2 && !single_k_capturable(e))
        e->replay_direct = true;  // variant passes read a flag per pass: launched directly
    if (!e->replay && !e->replay_direct) {
        const uint64_t l0 = e->launches;
        cudaGraph_t g = nullptr;
        e->trusted = true;
        rc = check_cuda(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal), "begin capture");
        if (!rc) {
            const int body = replay_pipeline(e);
            const cudaError_t end = cudaStreamEndCapture(e->stream, &g);
            rc = body ? body : check_cuda(end, "capture the pipeline");
        }
        e->trusted = false;
        e->replay_launches = e->launches - l0;
        e->launches = l0;
        e->replay_peel_mode = e->peel_mode;
        if (!rc) rc = check_cuda(cudaGraphInstantiate(&e->replay, g, 0), "instantiate the pipeline graph");
        if (g) cudaGraphDestroy(g);
        if (rc) {
            // capture errors leave the context usable: fall back to direct launches
            (void)cudaGetLastError();
            kt::clear_error();
            e->replay = nullptr;
            e->replay_direct = true;
        }
    }
    if ((rc = record_start(e))) return rc;
    if (e->replay_direct) {
        e->trusted = true;
        rc = replay_pipeline(e);
        e->trusted = false;
        if (rc) return rc;
    } else {
        if ((rc = check_cuda(cudaGraphLaunch(e->replay, e->stream), "launch the pipeline graph"))) return rc;
        e->launches += e->replay_launches;
    }
    if ((rc = check_cuda(cudaEventRecord(e->ev_stop, e->stream), "record stop"))) return rc;
    e->peel_mode = e->replay_peel_mode;
    e->ctrl_fresh = false;
    e->peel_timed = false;
    e->stats_ready = false;
    e->stats.build_ms = e->stats.select_ms = e->stats.support_ms = e->stats.peel_ms = 0;
    e->replay_timing = true;
    fill_graph_stats(e);
    if (!sync) return KT_OK;
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
    return kt::finish_stats(e);
}

int check_coo(const kt_coo* g, const char* what) {
    if (!g) return fail(KT_ERR_INVALID_ARG, "%s: null graph", what);
    if (g->num_edges && (!g->src_idx || !g->dst_idx)) return fail(KT_ERR_INVALID_ARG, "%s: null edge arrays", what);
    return KT_OK;
}

}  // namespace

extern "C" {

int kt_engine_create(int device, kt_engine** out) {
    if (!out) return fail(KT_ERR_INVALID_ARG, "kt_engine_create: null output");
    *out = nullptr;
    int count = 0;
    int rc = check_cuda(cudaGetDeviceCount(&count), "cudaGetDeviceCount");
    if (rc) return rc;
    if (device < 0 || device >= count) return fail(KT_ERR_NO_DEVICE, "device %d not present (%d devices)", device, count);
    if ((rc = check_cuda(cudaSetDevice(device), "cudaSetDevice"))) return rc;
    kt_engine* e = new kt_engine();
    e->device = device;
    e->lists_allowed = true;
    if ((rc = check_cuda(cudaDeviceGetAttribute(&e->num_sms, cudaDevAttrMultiProcessorCount, device), "SM count")) ||
        (rc = check_cuda(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking), "create stream")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_start), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_stop), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_built), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_counted), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_select), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_peeled), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_copy[0]), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_copy[1]), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_copy[2]), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_copy[3]), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_peel0), "create event")) ||
        (rc = check_cuda(cudaEventCreate(&e->ev_peel1), "create event")) ||
        (rc = check_cuda(cudaMalloc(&e->ctrl, sizeof(uint32_t) * kt::kCtrlWords), "allocate control block")) ||
        (rc = check_cuda(cudaMallocHost(&e->h_ctrl, sizeof(uint32_t) * kt::kCtrlWords), "allocate host mirror"))) {
        kt_engine_destroy(e);
        return rc;
    }
    *out = e;
    return KT_OK;
}

int kt_engine_destroy(kt_engine* e) {
    if (!e) return KT_OK;
    cudaSetDevice(e->device);
    if (e->stream) cudaStreamSynchronize(e->stream);
    kt::drop_replay(e);
    if (e->arena) cudaFree(e->arena);
    if (e->aux) cudaFree(e->aux);
    if (e->tile_off) cudaFree(e->tile_off);
    if (e->ingest) cudaFree(e->ingest);
    if (e->lists) cudaFree(e->lists);
    if (e->ctrl) cudaFree(e->ctrl);
    if (e->h_ctrl) cudaFreeHost(e->h_ctrl);
    if (e->ev_start) cudaEventDestroy(e->ev_start);
    if (e->ev_stop) cudaEventDestroy(e->ev_stop);
    if (e->ev_built) cudaEventDestroy(e->ev_built);
    if (e->ev_counted) cudaEventDestroy(e->ev_counted);
    if (e->ev_select) cudaEventDestroy(e->ev_select);
    if (e->ev_peeled) cudaEventDestroy(e->ev_peeled);
    for (cudaEvent_t ev : e->ev_copy)
        if (ev) cudaEventDestroy(ev);
    if (e->ev_peel0) cudaEventDestroy(e->ev_peel0);
    if (e->ev_peel1) cudaEventDestroy(e->ev_peel1);
    if (e->stream) cudaStreamDestroy(e->stream);
    delete e;
    return KT_OK;
}

void* kt_engine_stream(kt_engine* e) { return e ? (void*)e->stream : nullptr; }

int kt_engine_reserve(kt_engine* e, uint32_t max_nodes, uint64_t max_entries) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_reserve: null engine");
    if (max_entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    return kt::reserve(e, max_nodes, max_entries);
}

int kt_engine_set_list_limit(kt_engine* e, uint64_t bytes) {
    kt::clear_error();
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_list_limit: null engine");
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    e->list_limit = bytes;
    if (e->list_cap * sizeof(uint2) > bytes) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
        kt::free_lists(e);
    }
    if (e->arena) kt::reserve_small_lists(e, e->cap_entries / 2);
    return KT_OK;
}

int kt_engine_get_list_limit(kt_engine* e, uint64_t* bytes, uint64_t* held) {
    kt::clear_error();
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_get_list_limit: null engine");
    if (bytes) *bytes = e->list_limit;
    if (held) *held = e->list_cap * sizeof(uint2);
    return KT_OK;
}

int kt_engine_decompose(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                        uint32_t num_nodes, uint32_t* d_truss, uint32_t* d_k_max, int sync) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_decompose: null engine");
    if (num_entries && (!d_src || !d_dst || !d_truss)) return fail(KT_ERR_INVALID_ARG, "kt_engine_decompose: null buffer");
    kt::clear_error();
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    if ((rc = run_decompose(e, d_src, d_dst, num_entries, num_nodes, d_truss, d_k_max))) {
        kt::forget(e);  // only a call that passed its checks is repeated
        return rc;
    }
    kt_engine::LastCall c;
    c.kind = 1, c.src = d_src, c.dst = d_dst, c.entries = num_entries, c.n = num_nodes, c.truss = d_truss, c.k_max = d_k_max;
    kt::remember(e, c);
    if (sync) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
        return kt::finish_stats(e);
    }
    return KT_OK;
}

int kt_engine_ktruss(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                     uint32_t num_nodes, uint32_t k, uint8_t* d_keep, int sync) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_ktruss: null engine");
    if (num_entries && (!d_src || !d_dst || !d_keep)) return fail(KT_ERR_INVALID_ARG, "kt_engine_ktruss: null buffer");
    kt::clear_error();
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    if ((rc = run_ktruss(e, d_src, d_dst, num_entries, num_nodes, k, d_keep))) {
        kt::forget(e);
        return rc;
    }
    kt_engine::LastCall c;
    c.kind = 2, c.src = d_src, c.dst = d_dst, c.entries = num_entries, c.n = num_nodes, c.k = k, c.keep = d_keep;
    kt::remember(e, c);
    if (sync) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
        return kt::finish_stats(e);
    }
    return KT_OK;
}

int kt_engine_replay(kt_engine* e, int sync) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_replay: null engine");
    kt::clear_error();
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    return replay(e, sync);
}

int kt_engine_replay_mode(const kt_engine* e) { return !e ? 0 : e->replay ? 1 : e->replay_direct ? 2 : 0; }

kt_schedule kt_schedule_default(void) { return kt_schedule{8, 32, 85, 50, 0}; }

kt_variant kt_variant_default(void) {
    return kt_variant{KT_DIRECTED_BY_DEGREE, KT_FORMAT_COOCSR, KT_RECOUNT_ALL, 512, 8, 8};
}

int kt_engine_set_variant(kt_engine* e, const kt_variant* v) {
    kt::clear_error();
    if (!e || !v) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_variant: null argument");
    if (v->directedness < KT_UNDIRECTED || v->directedness > KT_DIRECTED_BY_DEGREE ||
        v->input_format < KT_FORMAT_COOCSR || v->input_format > KT_FORMAT_TILED_COOCSR ||
        v->recount < KT_RECOUNT_ALL || v->recount > KT_RECOUNT_AFFECTED)
        return fail(KT_ERR_INVALID_ARG, "kt_engine_set_variant: bad enum value");
    if (v->block_size < 1 || v->block_size > 1024)
        return fail(KT_ERR_INVALID_ARG, "block_size must be 1..1024 (got %u)", v->block_size);
    if (v->num_tiles < 1 || v->num_tiles > 4096 || v->num_parallel_tiles < 1)
        return fail(KT_ERR_INVALID_ARG, "num_tiles must be 1..4096 and num_parallel_tiles >= 1");
    e->variant = *v;
    kt::drop_replay(e);
    return KT_OK;
}

int kt_engine_get_variant(kt_engine* e, kt_variant* v) {
    kt::clear_error();
    if (!e || !v) return fail(KT_ERR_INVALID_ARG, "kt_engine_get_variant: null argument");
    *v = e->variant;
    return KT_OK;
}

int kt_engine_set_schedule(kt_engine* e, const kt_schedule* s) {
    kt::clear_error();
    if (!e || !s) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_schedule: null argument");
    const uint32_t g = s->support_group, w = s->chunk_width;
    if (g != 0 && g != 4 && g != 8 && g != 16 && g != 32)
        return fail(KT_ERR_INVALID_ARG, "support_group must be 0 (vertex hash), 4, 8, 16 or 32 (got %u)", g);
    if (w != 8 && w != 16 && w != 32) return fail(KT_ERR_INVALID_ARG, "chunk_width must be 8, 16 or 32 (got %u)", w);
    if (s->compact_percent > 99)
        return fail(KT_ERR_INVALID_ARG, "compact_percent must be 0..99 (got %u)", s->compact_percent);
    if (s->recount_percent > 100)
        return fail(KT_ERR_INVALID_ARG, "recount_percent must be 0..100 (got %u)", s->recount_percent);
    if (s->peel_blocks > 2) return fail(KT_ERR_INVALID_ARG, "peel_blocks must be 0, 1 or 2 (got %u)", s->peel_blocks);
    e->sched = *s;
    kt::drop_replay(e);  // a replay captures the pipeline again with this schedule
    return KT_OK;
}

int kt_engine_set_wait_limit(kt_engine* e, uint64_t base_ns, uint32_t ns_per_unit) {
    kt::clear_error();
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_wait_limit: null engine");
    if (base_ns < 1000) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_wait_limit: base below 1 microsecond");
    e->wait_base_ns = base_ns;
    e->wait_ns_per_unit = ns_per_unit;
    kt::drop_replay(e);  // a captured pipeline holds the old limits
    return KT_OK;
}

int kt_engine_get_wait_limit(kt_engine* e, uint64_t* base_ns, uint32_t* ns_per_unit) {
    kt::clear_error();
    if (!e || !base_ns || !ns_per_unit) return fail(KT_ERR_INVALID_ARG, "kt_engine_get_wait_limit: null argument");
    *base_ns = e->wait_base_ns;
    *ns_per_unit = (uint32_t)e->wait_ns_per_unit;
    return KT_OK;
}

int kt_engine_get_schedule(kt_engine* e, kt_schedule* s) {
    kt::clear_error();
    if (!e || !s) return fail(KT_ERR_INVALID_ARG, "kt_engine_get_schedule: null argument");
    *s = e->sched;
    return KT_OK;
}

int kt_last_stats(kt_stats* stats) {
    kt::clear_error();
    if (!stats) return fail(KT_ERR_INVALID_ARG, "kt_last_stats: null argument");
    kt_engine* e = nullptr;
    int rc = default_engine(&e);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    return kt_engine_stats(e, stats);
}

int kt_set_schedule(const kt_schedule* s) {
    kt_engine* e = nullptr;
    int rc = default_engine(&e);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    return kt_engine_set_schedule(e, s);
}

int kt_set_list_limit(uint64_t bytes) {
    kt_engine* e = nullptr;
    int rc = default_engine(&e);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    return kt_engine_set_list_limit(e, bytes);
}

int kt_get_list_limit(uint64_t* bytes, uint64_t* held) {
    kt_engine* e = nullptr;
    int rc = default_engine(&e);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    return kt_engine_get_list_limit(e, bytes, held);
}

int kt_get_schedule(kt_schedule* s) {
    kt_engine* e = nullptr;
    int rc = default_engine(&e);
    if (rc) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    return kt_engine_get_schedule(e, s);
}

uint32_t kt_schedule_grid(kt_schedule* out, uint32_t cap) {
    const uint32_t count = KT_SELECTOR_SCHEDULES;  // 3 groups x 3 widths x 2 compactions x 2 recounts
    for (uint32_t i = 0; out && i < count && i < cap; ++i) {
        kt_schedule s{0, 0, 0, 0, 0};
        kt::grid_schedule(i, &s.support_group, &s.chunk_width, &s.compact_percent, &s.recount_percent);
        out[i] = s;
    }
    return count;
}

namespace {

int autotune(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries, uint32_t num_nodes,
             const kt_schedule* candidates, uint32_t num_candidates, uint32_t repeats, float* ms, kt_schedule* best,
             bool batch) {
    kt::clear_error();
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_autotune: null engine");
    if (num_entries && (!d_src || !d_dst)) return fail(KT_ERR_INVALID_ARG, "kt_engine_autotune: null buffer");
    if (repeats == 0) return fail(KT_ERR_INVALID_ARG, "kt_engine_autotune: repeats must be >= 1");
    kt::forget(e);
    kt_schedule grid[36];
    if (!candidates) {
        num_candidates = kt_schedule_grid(grid, 36);
        candidates = grid;
    }
    if (num_candidates == 0) return fail(KT_ERR_INVALID_ARG, "kt_engine_autotune: no candidates");
    const kt_schedule saved = e->sched;
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    // support count and peel of one run (the rows are compacted in place while peeling, so every run
    // builds the CSR again)
    const auto run = [&](float* t) {
        int rc;
        if ((rc = kt::build_graph(e, d_src, d_dst, num_entries, num_nodes, true)) || (rc = record(e, e->ev_built)) ||
            (rc = kt::count_support(e)) || (rc = kt::peel_decompose(e)) || (rc = record(e, e->ev_stop)) ||
            (rc = check_cuda(cudaEventSynchronize(e->ev_stop), "synchronize")) ||
            (rc = check_cuda(cudaEventElapsedTime(t, e->ev_built, e->ev_stop), "elapsed time")))
            return rc;
        return kt::finish_stats(e);
    };
    // what but the support group a schedule says has no effect on a decomposition from lists
    const auto same_walks = [](const kt_schedule& a, const kt_schedule& b) {
        return a.chunk_width == b.chunk_width && a.compact_percent == b.compact_percent &&
               a.recount_percent == b.recount_percent && a.peel_blocks == b.peel_blocks;
    };
    uint32_t best_i = 0;
    std::vector<float> times(num_candidates);
    e->batch_call = batch;  // the peel's launch shape follows the call being tuned
    float first = 0;
    rc = run(&first);  // not counted: it makes the list buffer, and shows whether the graph takes lists
    const bool lists = e->m != 0 && e->list_need != 0;
    for (uint32_t i = 0; i < num_candidates && !rc; ++i) {
        if ((rc = kt_engine_set_schedule(e, &candidates[i]))) break;
        uint32_t same = 0;  // an earlier candidate that ran the same kernels
        while (same < i && !(lists && candidates[same].support_group == candidates[i].support_group)) ++same;
        if (same < i) {
            times[i] = times[same];
        } else {
            for (uint32_t r = 0; r < repeats && !rc; ++r) {
                float t = 0;
                if (!(rc = run(&t))) times[i] = r == 0 || t < times[i] ? t : times[i];
            }
        }
        if (rc) break;
        if (ms) ms[i] = times[i];
        const kt_schedule& b = candidates[best_i];
        if (i == 0 || times[i] < times[best_i] ||
            (lists && candidates[i].support_group == b.support_group && same_walks(candidates[i], saved) &&
             !same_walks(b, saved)))
            best_i = i;
    }
    e->batch_call = false;
    if (rc) {
        e->sched = saved;
        return rc;
    }
    e->sched = candidates[best_i];
    if (best) *best = candidates[best_i];
    return KT_OK;
}

}  // namespace

int kt_engine_autotune(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                       uint32_t num_nodes, const kt_schedule* candidates, uint32_t num_candidates, uint32_t repeats,
                       float* ms, kt_schedule* best) {
    return autotune(e, d_src, d_dst, num_entries, num_nodes, candidates, num_candidates, repeats, ms, best, false);
}

int kt_engine_autotune_batch(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                             uint32_t num_nodes, const kt_schedule* candidates, uint32_t num_candidates,
                             uint32_t repeats, float* ms, kt_schedule* best) {
    return autotune(e, d_src, d_dst, num_entries, num_nodes, candidates, num_candidates, repeats, ms, best, true);
}

int kt_engine_tiled_coocsr(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                           uint32_t num_nodes, uint32_t tiles_per_dim, uint32_t* d_tile_src_ptr, uint32_t* d_src_out,
                           uint32_t* d_dst_out) {
    kt::clear_error();
    if (!e || !d_tile_src_ptr || (num_entries && (!d_src || !d_dst || !d_src_out || !d_dst_out)))
        return fail(KT_ERR_INVALID_ARG, "kt_engine_tiled_coocsr: null argument");
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    return kt::tiled_coocsr(e, d_src, d_dst, num_entries, num_nodes, tiles_per_dim, d_tile_src_ptr, d_src_out,
                            d_dst_out);
}

int kt_engine_symmetrize(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                         uint32_t num_nodes, uint32_t* d_src_out, uint32_t* d_dst_out, uint64_t capacity,
                         uint64_t* num_out) {
    kt::clear_error();
    if (!e || !num_out || (num_entries && (!d_src || !d_dst || (capacity && (!d_src_out || !d_dst_out)))))
        return fail(KT_ERR_INVALID_ARG, "kt_engine_symmetrize: null argument");
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    return kt::symmetrize(e, d_src, d_dst, num_entries, num_nodes, d_src_out, d_dst_out, capacity, num_out);
}

int kt_engine_set_selector(kt_engine* e, kt_selector* s) {
    kt::clear_error();
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_set_selector: null engine");
    e->selector = s;
    kt::drop_replay(e);
    return KT_OK;
}

int kt_engine_features(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                       uint32_t num_nodes, float* features) {
    kt::clear_error();
    if (!e || !features) return fail(KT_ERR_INVALID_ARG, "kt_engine_features: null argument");
    if (num_entries && (!d_src || !d_dst)) return fail(KT_ERR_INVALID_ARG, "kt_engine_features: null buffer");
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc || (rc = kt::build_graph(e, d_src, d_dst, num_entries, num_nodes, true)) ||
        (rc = kt::graph_features(e, nullptr)) ||
        (rc = check_cuda(cudaMemcpyAsync(features, e->sel_feat, sizeof(float) * KT_SELECTOR_FEATURES,
                                         cudaMemcpyDeviceToHost, e->stream), "read features")))
        return rc;
    return check_cuda(cudaStreamSynchronize(e->stream), "synchronize");
}

int kt_engine_selftest_wait_timeout(kt_engine* e, int wait, uint64_t timeout_ns) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_selftest_wait_timeout: null engine");
    if (timeout_ns == 0 || timeout_ns > 5000000000ull)
        return fail(KT_ERR_INVALID_ARG, "timeout must be in (0, 5 s]");
    if (wait < KT_WAIT_GRID_BARRIER || wait > KT_WAIT_LOOK_BACK)
        return fail(KT_ERR_INVALID_ARG, "kt_engine_selftest_wait_timeout: unknown wait %d", wait);
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    e->stats_ready = true;  // the probe leaves no peel statistics behind
    return wait == KT_WAIT_GRID_BARRIER   ? kt::barrier_timeout_probe(e, timeout_ns)
           : wait == KT_WAIT_LIST_BARRIER ? kt::list_timeout_probe(e, timeout_ns)
                                          : kt::look_timeout_probe(e, timeout_ns);
}

int kt_engine_selftest_barrier_timeout(kt_engine* e, uint64_t timeout_ns) {
    return kt_engine_selftest_wait_timeout(e, KT_WAIT_GRID_BARRIER, timeout_ns);
}

int kt_engine_round_log(kt_engine* e, uint32_t* size, uint32_t* level, uint32_t* ns, uint32_t cap,
                        uint32_t* num_rounds) {
    if (!e || !num_rounds) return fail(KT_ERR_INVALID_ARG, "kt_engine_round_log: null argument");
    int rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize");
    if (rc) return rc;
    if ((rc = kt::finish_stats(e))) return rc;
    const uint32_t R = e->stats.num_rounds;
    *num_rounds = R;
    const uint32_t c = std::min<uint32_t>(std::min<uint32_t>(cap, R), e->cap_rounds > 0 ? e->cap_rounds - 1 : 0);
    if (c == 0) return KT_OK;
    uint32_t* dst[3] = {size, level, ns};
    uint32_t* src[3] = {e->round_size, e->round_level, e->round_ns};
    for (int i = 0; i < 3; ++i)
        if (dst[i] && (rc = check_cuda(cudaMemcpy(dst[i], src[i] + 1, sizeof(uint32_t) * c, cudaMemcpyDeviceToHost),
                                       "read round log")))
            return rc;
    return KT_OK;
}

int kt_engine_level_log(kt_engine* e, uint32_t* k, uint32_t* alive, uint32_t* ns, uint32_t* frontier, uint32_t cap,
                        uint32_t* num_levels) {
    if (!e || !num_levels) return fail(KT_ERR_INVALID_ARG, "kt_engine_level_log: null argument");
    int rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize");
    if (rc) return rc;
    if ((rc = kt::finish_stats(e))) return rc;
    const uint32_t L = e->stats.num_levels;
    *num_levels = L;
    const uint32_t c = std::min<uint32_t>(std::min<uint32_t>(cap, L), e->cap_levels);
    if (c == 0) return KT_OK;
    uint32_t* dst[4] = {k, alive, ns, frontier};
    uint32_t* src[4] = {e->level_k, e->level_alive, e->level_ns, e->level_front};
    for (int i = 0; i < 4; ++i)
        if (dst[i] &&
            (rc = check_cuda(cudaMemcpy(dst[i], src[i], sizeof(uint32_t) * c, cudaMemcpyDeviceToHost), "read level log")))
            return rc;
    return KT_OK;
}

int kt_engine_stats(kt_engine* e, kt_stats* stats) {
    if (!e || !stats) return fail(KT_ERR_INVALID_ARG, "kt_engine_stats: null argument");
    int rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize");
    if (rc) return rc;
    if ((rc = kt::finish_stats(e))) return rc;
    e->stats.kernel_launches = e->launches;
    *stats = e->stats;
    return KT_OK;
}

int kt_engine_decompose_batch(kt_engine* e, const uint32_t* d_src, const uint32_t* d_dst, uint64_t num_entries,
                              uint32_t num_nodes, const uint32_t* d_vertex_offsets, uint32_t num_graphs,
                              uint32_t* d_truss_per_entry, uint32_t* d_k_max_per_graph, int sync) {
    if (!e) return fail(KT_ERR_INVALID_ARG, "kt_engine_decompose_batch: null engine");
    if (!d_vertex_offsets || !d_k_max_per_graph || num_graphs == 0 ||
        (num_entries && (!d_src || !d_dst || !d_truss_per_entry)))
        return fail(KT_ERR_INVALID_ARG, "kt_engine_decompose_batch: null buffer or no graphs");
    kt::clear_error();
    int rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice");
    if (rc) return rc;
    // the union of disjoint graphs: its truss numbers are each graph's own
    kt::forget(e);
    e->batch_call = true;
    const Batch batch{d_vertex_offsets, num_graphs, d_k_max_per_graph};
    rc = run_decompose(e, d_src, d_dst, num_entries, num_nodes, d_truss_per_entry, nullptr, &batch);
    e->batch_call = false;
    if (rc) return rc;
    if (sync) {
        if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
        return kt::finish_stats(e);
    }
    return KT_OK;
}

int kt_decompose_batch(const uint32_t* src, const uint32_t* dst, uint64_t num_entries, uint32_t num_nodes,
                       const uint32_t* vertex_offsets, uint32_t num_graphs, uint32_t* truss_per_entry,
                       uint32_t* k_max_per_graph) {
    if (!vertex_offsets || !k_max_per_graph || num_graphs == 0 || (num_entries && (!src || !dst || !truss_per_entry)))
        return fail(KT_ERR_INVALID_ARG, "kt_decompose_batch: null buffer or no graphs");
    for (uint32_t g = 0; g < num_graphs; ++g)
        if (vertex_offsets[g] > vertex_offsets[g + 1])
            return fail(KT_ERR_INVALID_ARG, "kt_decompose_batch: vertex offsets decrease at graph %u", g);
    if (vertex_offsets[num_graphs] != num_nodes)
        return fail(KT_ERR_INVALID_ARG, "kt_decompose_batch: last vertex offset %u != num_nodes %u",
                    vertex_offsets[num_graphs], num_nodes);
    if (num_entries >= 0xffffffffull) return fail(KT_ERR_TOO_LARGE, "more than 2^32-2 entries");
    kt::clear_error();
    kt_engine* e = nullptr;
    int rc;
    if ((rc = default_engine(&e))) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    kt::forget(e);  // host-buffer calls overwrite the staging buffers a replay would read
    if ((rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice"))) return rc;
    if ((rc = kt::reserve(e, std::max(num_nodes, e->cap_nodes), std::max(num_entries, e->cap_entries)))) return rc;
    const size_t need = 2 * (size_t)num_graphs + 1;
    if (e->aux_words < need) {
        if (e->aux) cudaFree(e->aux);
        e->aux = nullptr;
        e->aux_words = 0;
        if ((rc = check_cuda(kt::alloc_device(e, (void**)&e->aux, sizeof(uint32_t) * need), "allocate batch staging")))
            return rc;
        e->aux_words = need;
    }
    uint32_t* d_off = e->aux;
    uint32_t* d_kmax = e->aux + num_graphs + 1;
    const uint64_t N = num_entries;
    if ((rc = record(e, e->ev_copy[0])) ||
        (rc = check_cuda(cudaMemcpyAsync(d_off, vertex_offsets, sizeof(uint32_t) * (num_graphs + 1),
                                         cudaMemcpyHostToDevice, e->stream), "H2D")))
        return rc;
    if (N && ((rc = check_cuda(cudaMemcpyAsync(e->in_src, src, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D")) ||
              (rc = check_cuda(cudaMemcpyAsync(e->in_dst, dst, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D"))))
        return rc;
    if ((rc = record(e, e->ev_copy[1]))) return rc;
    e->batch_call = true;
    const Batch batch{d_off, num_graphs, d_kmax};
    rc = run_decompose(e, e->in_src, e->in_dst, N, num_nodes, e->out_u32, nullptr, &batch);
    e->batch_call = false;
    if (rc) return rc;
    if ((rc = record(e, e->ev_copy[2]))) return rc;
    if (N && (rc = check_cuda(cudaMemcpyAsync(truss_per_entry, e->out_u32, N * 4, cudaMemcpyDeviceToHost, e->stream),
                              "D2H")))
        return rc;
    if ((rc = check_cuda(cudaMemcpyAsync(k_max_per_graph, d_kmax, sizeof(uint32_t) * num_graphs,
                                         cudaMemcpyDeviceToHost, e->stream), "D2H")) ||
        (rc = record(e, e->ev_copy[3])) || (rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize")))
        return rc;
    if ((rc = kt::finish_stats(e))) return rc;
    return copy_times(e);
}

int kt_decompose(const kt_coo* graph, uint32_t* truss_per_entry, uint32_t* k_max, const kt_config* config) {
    int rc = check_coo(graph, "kt_decompose");
    if (rc) return rc;
    if (graph->num_edges && !truss_per_entry) return fail(KT_ERR_INVALID_ARG, "kt_decompose: null output");
    if (config && config->processor == KT_PROCESSOR_CPU)
        return fail(KT_ERR_UNSUPPORTED, "processor cpu: this library runs the GPU path only");
    kt::clear_error();
    kt_engine* e = nullptr;
    if ((rc = default_engine(&e))) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    kt::forget(e);  // host-buffer calls overwrite the staging buffers a replay would read
    if ((rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice"))) return rc;
    const uint64_t N = graph->num_edges;
    if ((rc = kt::reserve(e, std::max(graph->num_nodes, e->cap_nodes), std::max(N, e->cap_entries)))) return rc;
    if ((rc = record(e, e->ev_copy[0]))) return rc;
    if (N) {
        if ((rc = check_cuda(cudaMemcpyAsync(e->in_src, graph->src_idx, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D")) ||
            (rc = check_cuda(cudaMemcpyAsync(e->in_dst, graph->dst_idx, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D")))
            return rc;
    }
    if ((rc = record(e, e->ev_copy[1]))) return rc;
    if ((rc = run_decompose(e, e->in_src, e->in_dst, N, graph->num_nodes, e->out_u32, nullptr))) return rc;
    if ((rc = record(e, e->ev_copy[2]))) return rc;
    if (N && (rc = check_cuda(cudaMemcpyAsync(truss_per_entry, e->out_u32, N * 4, cudaMemcpyDeviceToHost, e->stream), "D2H")))
        return rc;
    if ((rc = record(e, e->ev_copy[3]))) return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
    if ((rc = kt::finish_stats(e)) || (rc = copy_times(e))) return rc;
    if (k_max) *k_max = e->stats.k_max;
    return KT_OK;
}

int kt_ktruss(const kt_coo* graph, kt_coo* truss, const kt_config* config) {
    int rc = check_coo(graph, "kt_ktruss");
    if (rc) return rc;
    if (!truss || !config) return fail(KT_ERR_INVALID_ARG, "kt_ktruss: null truss or config");
    if (config->processor == KT_PROCESSOR_CPU)
        return fail(KT_ERR_UNSUPPORTED, "processor cpu: this library runs the GPU path only");
    if (config->processor != KT_PROCESSOR_GPU || config->directedness < 0 || config->directedness > 2 ||
        config->input_format < 0 || config->input_format > 1 || config->recount < 0 || config->recount > 1)
        return fail(KT_ERR_INVALID_ARG, "kt_ktruss: bad enum value in config");
    if (truss->capacity < graph->num_edges || (graph->num_edges && (!truss->src_idx || !truss->dst_idx)))
        return fail(KT_ERR_CAPACITY, "truss capacity %u below %u entries", truss->capacity, graph->num_edges);
    kt::clear_error();
    kt_engine* e = nullptr;
    if ((rc = default_engine(&e))) return rc;
    std::lock_guard<std::mutex> lock(g_default_mu);
    kt::forget(e);  // host-buffer calls overwrite the staging buffers a replay would read
    if ((rc = check_cuda(cudaSetDevice(e->device), "cudaSetDevice"))) return rc;
    // the reference's variant switches select the single-k path (-d, -f, -r, -b, -t, -y)
    const kt_variant variant{config->directedness, config->input_format, config->recount,
                             config->block_size ? config->block_size : 512u,
                             config->num_tiles ? config->num_tiles : 8u,
                             config->num_parallel_tiles ? config->num_parallel_tiles : 8u};
    if ((rc = kt_engine_set_variant(e, &variant))) return rc;
    const uint64_t N = graph->num_edges;
    const int verbose = config->verbosity >= 1;
    double t0 = now_ms();
    if ((rc = kt::reserve(e, std::max(graph->num_nodes, e->cap_nodes), std::max(N, e->cap_entries)))) return rc;
    if (N) {
        if ((rc = check_cuda(cudaMemcpyAsync(e->in_src, graph->src_idx, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D")) ||
            (rc = check_cuda(cudaMemcpyAsync(e->in_dst, graph->dst_idx, N * 4, cudaMemcpyHostToDevice, e->stream), "H2D")) ||
            (rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize")))
            return rc;
    }
    if (verbose) printf("    Copy COO graph to GPU: %f ms\n", now_ms() - t0);
    // -w warm-up and -x timed runs (kernel_ddc.cu:227-244); each run rebuilds the graph from
    // the input entries, so every run is the full device pipeline.
    const uint32_t runs = config->num_warmup_runs + config->num_timed_runs;
    // Runs after the first repeat it on the same input: kt_engine_replay's CUDA graph.
    for (uint32_t i = 0; i < (runs ? runs : 1); ++i) {
        if (verbose) printf("    Performing K-truss\n");
        if (i == 0) {
            if ((rc = run_ktruss(e, e->in_src, e->in_dst, N, graph->num_nodes, config->k, e->out_u8))) return rc;
            kt_engine::LastCall c;
            c.kind = 2, c.src = e->in_src, c.dst = e->in_dst, c.entries = N, c.n = graph->num_nodes, c.k = config->k,
            c.keep = e->out_u8;
            kt::remember(e, c);
            if ((rc = kt::finish_stats(e))) return rc;
        } else if ((rc = replay(e, 1))) {
            return rc;
        }
        if (config->verbosity == 0 && i >= config->num_warmup_runs) {
            kt_print_config_csv(config);
            printf("%f ms\n", e->stats.last_ms);
        }
        if (verbose) printf("\033[0;32m        Total K-truss time: %f ms\n\033[0m", e->stats.last_ms);
    }
    t0 = now_ms();
    std::vector<uint8_t> keep(N);
    if (N && (rc = check_cuda(cudaMemcpyAsync(keep.data(), e->out_u8, N, cudaMemcpyDeviceToHost, e->stream), "D2H")))
        return rc;
    if ((rc = check_cuda(cudaStreamSynchronize(e->stream), "synchronize"))) return rc;
    uint32_t w = 0;
    for (uint64_t i = 0; i < N; ++i)
        if (keep[i]) {
            truss->src_idx[w] = graph->src_idx[i];
            truss->dst_idx[w] = graph->dst_idx[i];
            ++w;
        }
    truss->num_edges = w;
    truss->num_nodes = graph->num_nodes;
    if (verbose) printf("    Copy COO truss from GPU: %f ms\n", now_ms() - t0);
    return KT_OK;
}

}  // extern "C"
