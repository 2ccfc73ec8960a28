// Runtime: device/stream selection, status, the pooled stream-ordered allocator and the
// host<->device transfers behind the memory entries of the boundary
// (reference: engine_cuda/src/cuda_bindings.cpp:23-170, which calls cudaMalloc / cudaFree /
// cudaMemcpy directly on every call).
//
// Allocator: freed blocks are kept in per-size free lists and handed out again for the same
// rounded size.  All work runs on one stream, so a block returned by cuda_free may be reused
// by the next allocation without waiting: every kernel that still reads it was enqueued earlier.
#include "common.cuh"
#include <algorithm>
#include <cstdarg>
#include <cstdlib>
#include <cstring>
#include <string>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace seera {

// Configuration by environment, read once when the library is first used:
//   SEERA_PRECISION   0..5   initial precision mode of the contractions (default 3: bf16x6 on the tensor cores - fp32-class
//                            products over fp32's whole exponent range, so that a caller who never heard of
//                            seera_set_precision still runs on tcgen05 kernels and still matches the fp32 reference)
//   SEERA_PAIR_TILES  0|1    the "pair_tiles" option (TMA-fed GEMMs as clusters of two CTAs on 256-row tiles)
//   SEERA_SM_RESERVE  n      SMs the persistent kernels leave free (the "sm_reserve" option)
//   SEERA_TC_WAIT_MS  n      budget of the bounded waits inside the tensor-core kernels, in milliseconds (default 2000)
static Runtime make_runtime() {
    Runtime r;
    r.precision = 3;
    if (const char *e = getenv("SEERA_PRECISION")) {
        int m = atoi(e);
        if (m >= 0 && m <= 5 && e[0] >= '0' && e[0] <= '5') r.precision = m;
    }
    if (const char *e = getenv("SEERA_PAIR_TILES")) r.pair_tiles = atoi(e) != 0;
    if (const char *e = getenv("SEERA_TC_WAIT_MS")) {
        long long ms = atoll(e);
        if (ms > 0) r.tc_wait_clocks = (unsigned long long)ms * 2000000ull;      // ~2e6 clocks per millisecond
    }
    return r;
}
Runtime &rt() { static Runtime r = make_runtime(); return r; }

int fail(int code, const char *fmt, ...) {
    Runtime &r = rt();
    va_list ap; va_start(ap, fmt);
    vsnprintf(r.err, sizeof(r.err), fmt, ap);
    va_end(ap);
    r.status = code;
    return code;
}

int check_cuda(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return SEERA_OK;
    return fail(SEERA_E_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int ensure_init() {
    if (rt().device >= 0) return SEERA_OK;
    return seera_init(0);
}

namespace {
// A recorded optimizer update: its node and a copy of its launch, kept so that the scalars can be replaced.
struct OptNode {
    cudaGraphNode_t node;
    OptLaunch launch;
    size_t at = 0;                                      // its place among the launches of the recording
};
struct GraphRec {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<std::pair<void *, size_t>> blocks;      // every block handed out while the graph was captured
    uint64_t kernels = 0;                               // kernel launches recorded in the graph
    uint64_t launches_at_begin = 0;
    bool collectives = false;                           // the recording holds launches of the data-parallel communicator
    std::vector<OptNode> optimizers;                    // recorded optimizer updates, whose scalars change from replay to replay
    std::vector<int> finish_slots;                      // counters of the recorded launches that finish in their last block
    bool lost_update = false;                           // ... one of which is not among them
    size_t noted = 0;                                   // launches recorded, and a hash of their kernels and grids
    uint64_t hash = 1469598103934665603ull;
    uint64_t row = 0;                                   // the hash if the nodes are those launches, one after the other; else 0
};
static std::vector<GraphRec *> &live_graphs() { static std::vector<GraphRec *> v; return v; }
struct Pool {
    std::map<size_t, std::vector<void *>> free_lists;   // rounded size -> cached blocks
    std::unordered_map<void *, size_t> live;            // every block handed out -> rounded size
    size_t reserved = 0;
    // stream capture: blocks used inside a captured step stay reserved for the graph that replays it
    bool capturing = false;
    std::map<size_t, std::vector<void *>> cap_free;     // freed during capture: reusable only inside the capture
    std::unordered_map<void *, GraphRec *> owner;       // block -> graph whose replay writes it
    GraphRec *cur = nullptr;
};
Pool &pool() { static Pool p; return p; }

size_t round_size(size_t n) {
    if (n == 0) n = 1;
    if (n <= (1u << 20)) return (n + 511) & ~size_t(511);                 // 512 B granules up to 1 MiB
    return (n + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);        // 2 MiB granules above
}
}  // namespace

// Per-launch profile (seera_profile_enable): launches bracketed by profile_begin / profile_end[_bytes] are timed with
// events on the engine's stream and booked under a tag.  Contractions book FLOPs and a kind (0 forward, 1 data gradient,
// 2 weight gradient, 4 both in one launch, from the entry name's "(dX)" / "(dW)" / "(dX+dW)" suffix); bandwidth-bound passes book
// their algorithmic bytes (kind 3).  Nothing is recorded while a graph is being captured.
struct ProfRec { cudaEvent_t a, b; double work; int kind; const char *tag; };
struct ProfAgg { int kind = 0; uint64_t n = 0; double ms = 0, work = 0; };
struct Prof { bool on = false; std::vector<ProfRec> recs; cudaEvent_t pending = nullptr; std::map<std::string, ProfAgg> table; };
static Prof &prof() { static Prof p; return p; }

void profile_begin() {
    Prof &p = prof();
    if (!p.on || rt().capturing) return;
    cudaEventCreate(&p.pending);
    cudaEventRecord(p.pending, rt().stream);
}
static int profile_kind(const char *name) {
    const char *of = name ? strrchr(name, '(') : nullptr;
    if (!of) return name && strcmp(name, "conv2d_act_bwd") == 0 ? 2 : 0;       // the short-patch layer backward forms only the weight gradient
    if (!strcmp(of, "(dX)") || !strcmp(of, "(dA)")) return 1;
    if (!strcmp(of, "(dW)") || !strcmp(of, "(dB)")) return 2;
    return !strcmp(of, "(dX+dW)") || !strcmp(of, "(dA+dB)") ? 4 : 0;
}
static void profile_close(double work, int kind, const char *tag) {
    Prof &p = prof();
    if (!p.on || !p.pending) return;
    ProfRec r{p.pending, nullptr, work, kind, tag ? tag : "?"};
    cudaEventCreate(&r.b);
    cudaEventRecord(r.b, rt().stream);
    p.recs.push_back(r);
    p.pending = nullptr;
}
void profile_end(double flops, const char *name) { profile_close(flops, profile_kind(name), name); }
void profile_end_bytes(double bytes, const char *tag) { profile_close(bytes, 3, tag); }

// Resolves the recorded events into the per-tag table (waits for them).
static void profile_collect() {
    Prof &p = prof();
    for (auto &r : p.recs) {
        float e = 0.f;
        cudaEventSynchronize(r.b);
        cudaEventElapsedTime(&e, r.a, r.b);
        ProfAgg &g = p.table[std::string(r.tag)];
        g.kind = r.kind; g.n++; g.ms += e; g.work += r.work;
        cudaEventDestroy(r.a); cudaEventDestroy(r.b);
    }
    p.recs.clear();
}

// An optimizer update is being recorded into the open capture: its node is the one the stream's next work will depend on.  One whose node
// cannot be named would keep the scalars that it was recorded with: an error, here and where scalars are set.
int graph_note_optimizer(const OptLaunch &launch) {
    Pool &p = pool();
    if (!p.capturing || !p.cur) return SEERA_OK;
    cudaStreamCaptureStatus st;
    const cudaGraphNode_t *deps = nullptr;
    size_t n = 0;
    const cudaError_t e = cudaStreamGetCaptureInfo_v2(rt().stream, &st, nullptr, nullptr, &deps, &n);
    if (rt().graph_test_lose_update) n = 2;
    rt().graph_test_lose_update = false;                // one update only
    if (e == cudaSuccess && n == 1) {
        p.cur->optimizers.push_back({deps[0], launch, p.cur->noted - 1});
        return SEERA_OK;
    }
    cudaGetLastError();
    p.cur->lost_update = true;
    return fail(SEERA_E_CUDA, "a recorded optimizer update has no node of its own (%zu dependencies): its scalars could not be replaced", n);
}

// Executable graphs of recordings that have been destroyed, for the next recording of the same kernels and grids in a row (another would run
// slower on them than on its own, see batch.cu): updating one takes 8 us where making one takes 125 and destroying it 110 (14 launches; a
// short training run records its step once).  At most SPARES_MAX; seera_pool_trim gives them back.  Nodes are named by the graph an
// executable was made from, which stays with it.
namespace {
constexpr size_t SPARES_MAX = 4;
struct Spare {
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    std::vector<OptNode> optimizers;
    uint64_t row;
};
std::vector<Spare> &spares() { static std::vector<Spare> v; return v; }
}  // namespace
// A launch, fill or copy goes into the open recording (batch.cu, which sees them all).
void graph_note_launch(const void *func, dim3 grid, dim3 block, size_t smem) {
    GraphRec *g = pool().cur;
    if (!g) return;
    auto mix = [g](uint64_t v) { g->hash = (g->hash ^ v) * 1099511628211ull; g->hash ^= g->hash >> 32; };
    mix((uint64_t)(uintptr_t)func);
    mix(((uint64_t)grid.x << 32) ^ ((uint64_t)grid.y << 16) ^ grid.z);
    mix(((uint64_t)smem << 32) ^ ((uint64_t)block.x << 16) ^ (block.y << 8) ^ block.z);
    g->noted++;
}
// The number of nodes of a graph if each follows the one before it, else 0.
static size_t chain_length(cudaGraph_t g) {
    size_t nodes = 0, edges = 0, roots = 0;
    if (cudaGraphGetNodes(g, nullptr, &nodes) != cudaSuccess || cudaGraphGetEdges(g, nullptr, nullptr, &edges) != cudaSuccess ||
        cudaGraphGetRootNodes(g, nullptr, &roots) != cudaSuccess || !nodes || roots != 1 || edges != nodes - 1) {
        cudaGetLastError();
        return 0;
    }
    std::vector<cudaGraphNode_t> from(edges), to(edges);
    if (edges && cudaGraphGetEdges(g, from.data(), to.data(), &edges) != cudaSuccess) { cudaGetLastError(); return 0; }
    std::sort(from.begin(), from.end());
    return std::adjacent_find(from.begin(), from.end()) == from.end() ? nodes : 0;       // nothing has two successors
}
static void spares_trim(size_t keep) {
    auto &v = spares();
    while (v.size() > keep) {
        cudaGraphExecDestroy(v.front().exec);
        cudaGraphDestroy(v.front().graph);
        v.erase(v.begin());
    }
}
static void take_spare(GraphRec *g) {
    auto &v = spares();
    for (size_t i = v.size(); i-- > 0;) {
        if (v[i].row != g->row || v[i].optimizers.size() != g->optimizers.size()) continue;
        bool same = true;
        for (size_t k = 0; k < g->optimizers.size(); k++) same &= v[i].optimizers[k].at == g->optimizers[k].at;
        if (!same) continue;
        Spare sp = v[i];
        v.erase(v.begin() + (long)i);
        cudaGraphExecUpdateResultInfo info;
        if (cudaGraphExecUpdate(sp.exec, g->graph, &info) == cudaSuccess) {
            cudaGraphDestroy(g->graph);
            g->graph = sp.graph;
            g->exec = sp.exec;
            for (size_t k = 0; k < sp.optimizers.size(); k++) g->optimizers[k].node = sp.optimizers[k].node;
            return;
        }
        cudaGetLastError();                             // other launches: not for this recording, nor known to be for any other
        cudaGraphExecDestroy(sp.exec);
        cudaGraphDestroy(sp.graph);
    }
}
// The caller has waited for the graph's last launch.
static void keep_spare(GraphRec *g) {
    if (!g->exec || !g->graph || !g->row) return;
    spares_trim(SPARES_MAX - 1);
    spares().push_back({g->graph, g->exec, g->optimizers, g->row});
    g->graph = nullptr;
    g->exec = nullptr;
}

// Slot 0 serves the library's own stream, whose launches follow one another, the next ones a caller's stream each (streams have numbers that
// are not given twice), and the rest are for recordings, which may be replayed beside all of them.
namespace {
constexpr int FINISH_STREAMS = 64;
struct FinishSlots {
    std::unordered_map<unsigned long long, int> streams;
    std::vector<int> free;
    FinishSlots() { for (int i = FINISH_SLOTS - 1; i >= FINISH_STREAMS; i--) free.push_back(i); }
};
FinishSlots &finish_slots() { static FinishSlots s; return s; }
}  // namespace
int finish_slot() {
    Pool &p = pool();
    FinishSlots &f = finish_slots();
    if (p.capturing && p.cur) {
        if (f.free.empty()) return -1;
        p.cur->finish_slots.push_back(f.free.back());
        f.free.pop_back();
        return p.cur->finish_slots.back();
    }
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(rt().stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) { cudaGetLastError(); return -1; }
    if (rt().stream == rt().own_stream) return 0;
    unsigned long long id = 0;
    if (cudaStreamGetId(rt().stream, &id) != cudaSuccess) { cudaGetLastError(); return -1; }
    auto it = f.streams.find(id);
    if (it != f.streams.end()) return it->second;
    if (f.streams.size() + 1 >= (size_t)FINISH_STREAMS) return -1;
    const int slot = (int)f.streams.size() + 1;
    f.streams[id] = slot;
    return slot;
}

void *scratch_alloc(size_t bytes) { return seera_cuda_malloc(bytes); }
void scratch_free(void *p) { seera_cuda_free(p); }

}  // namespace seera

namespace seera {
// dp.cu: a collective is being recorded into the open capture
void graph_note_collective() {
    Pool &p = pool();
    if (p.capturing && p.cur) p.cur->collectives = true;
}
// dp.cu, before the communicator goes away: the library that runs the collectives keeps per-recording state alive as long as a
// recording that holds its launches exists, and tearing the communicator down waits for that state.  The executable graphs are
// destroyed here; their handles stay valid for seera_graph_destroy, and seera_graph_launch on them reports an error.
void graphs_with_collectives_release() {
    if (rt().stream) cudaStreamSynchronize(rt().stream);
    for (GraphRec *g : live_graphs()) {
        if (!g->collectives) continue;
        if (g->exec) { cudaGraphExecDestroy(g->exec); g->exec = nullptr; }
        if (g->graph) { cudaGraphDestroy(g->graph); g->graph = nullptr; }
    }
}
}  // namespace seera

using namespace seera;

static void pinned_trim();
static void pinned_other_streams();

extern "C" {

int seera_init(int device) {
    Runtime &r = rt();
    if (r.device == device && r.stream) return SEERA_OK;
    // one device per process: the stream, the memory pool, the tensor-core status word and the profiler events all belong to
    // the device of the first call
    if (r.device >= 0 && r.device != device)
        return fail(SEERA_E_ARG, "seera_init: this process already runs on device %d (one device per process; asked for %d)", r.device, device);
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0)
        return fail(SEERA_E_CUDA, "seera_init: no CUDA device (%s)", cudaGetErrorString(e));
    if (device < 0 || device >= n) return fail(SEERA_E_ARG, "seera_init: device %d of %d", device, n);
    if (int s = check_cuda(cudaSetDevice(device), "cudaSetDevice")) return s;
    cudaDeviceProp p;
    if (int s = check_cuda(cudaGetDeviceProperties(&p, device), "cudaGetDeviceProperties")) return s;
    r.sm_count = r.sm_physical = p.multiProcessorCount;
    if (!r.own_stream)
        if (int s = check_cuda(cudaStreamCreateWithFlags(&r.own_stream, cudaStreamNonBlocking), "cudaStreamCreate")) return s;
    r.stream = r.own_stream;
    r.device = device;
    if (const char *e = getenv("SEERA_SM_RESERVE")) {
        int n = atoi(e);
        if (n > 0 && n < r.sm_physical) r.sm_count = r.sm_physical - n;
    }
    return SEERA_OK;
}

int seera_synchronize(void) {
    SEERA_ENSURE();
    if (int s = batch_flush()) return s;
    if (rt().capturing) return fail(SEERA_E_ARG, "synchronize: not allowed while a graph is being captured");
    return check_cuda(cudaStreamSynchronize(rt().stream), "cudaStreamSynchronize");
}

int seera_set_stream(void *s) {
    SEERA_ENSURE();
    if (int e = batch_flush()) return e;
    pinned_other_streams();
    rt().stream = s ? reinterpret_cast<cudaStream_t>(s) : rt().own_stream;
    return SEERA_OK;
}
void *seera_get_stream(void) { return ensure_init() || batch_flush() ? nullptr : (void *)rt().stream; }
const char *seera_last_error(void) { return rt().err; }
int seera_last_status(void) { return rt().status; }
void seera_clear_status(void) { rt().status = 0; rt().err[0] = 0; }
uint64_t seera_launch_count(void) { return rt().launches; }
int seera_device_sm_count(void) { return ensure_init() ? 0 : rt().sm_count; }
void *seera_event_create(void) {
    if (ensure_init()) return nullptr;
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return (void *)e;
}
int seera_event_record(void *ev) {
    SEERA_ENSURE();
    if (!ev) return fail(SEERA_E_ARG, "event_record: null");
    if (int s = batch_flush()) return s;
    return check_cuda(cudaEventRecord((cudaEvent_t)ev, rt().stream), "cudaEventRecord");
}
float seera_event_elapsed_ms(void *a, void *b) {
    if (!a || !b) return -1.f;
    if (cudaEventSynchronize((cudaEvent_t)b) != cudaSuccess) { check_cuda(cudaGetLastError(), "cudaEventSynchronize"); return -1.f; }
    float ms = -1.f;
    if (cudaEventElapsedTime(&ms, (cudaEvent_t)a, (cudaEvent_t)b) != cudaSuccess) { cudaGetLastError(); return -1.f; }
    return ms;
}
int seera_event_destroy(void *ev) { return ev ? check_cuda(cudaEventDestroy((cudaEvent_t)ev), "cudaEventDestroy") : SEERA_OK; }

int seera_profile_enabled(void) { return seera::prof().on ? 1 : 0; }
int seera_profile_enable(int on) {
    auto &p = seera::prof();
    if (int s = batch_flush()) return s;
    if (on && !p.on) { seera::profile_collect(); p.table.clear(); }      // a new session starts from an empty table
    p.on = on != 0;
    return SEERA_OK;
}
// Sums over the kinds below `kinds` (5: all contractions), each kind in its own place or all of them in the first.
static void profile_sum(int kinds, bool apart, uint64_t *n, double *ms, double *flops) {
    seera::profile_collect();
    for (auto &kv : seera::prof().table) {
        const auto &g = kv.second;
        if (g.kind == 3 || g.kind >= kinds) continue;
        const int k = apart ? g.kind : 0;
        n[k] += g.n; ms[k] += g.ms; flops[k] += g.work;
    }
}
int seera_profile_read_kinds(uint64_t *launches3, double *ms3, double *flops3) {
    SEERA_ENSURE();
    uint64_t n[3] = {0, 0, 0};
    double t[3] = {0, 0, 0}, f[3] = {0, 0, 0};
    profile_sum(3, true, n, t, f);
    for (int k = 0; k < 3; k++) {
        if (launches3) launches3[k] = n[k];
        if (ms3) ms3[k] = t[k];
        if (flops3) flops3[k] = f[k];
    }
    return SEERA_OK;
}
int seera_profile_read(uint64_t *launches, double *ms, double *flops) {
    SEERA_ENSURE();
    uint64_t n = 0;
    double t = 0, f = 0;
    profile_sum(5, false, &n, &t, &f);
    if (launches) *launches = n;
    if (ms) *ms = t;
    if (flops) *flops = f;
    seera::prof().table.clear();
    return SEERA_OK;
}
int seera_profile_report(char *buf, size_t size) {
    SEERA_ENSURE();
    if (!buf || size < 2) return fail(SEERA_E_ARG, "profile_report: no buffer");
    seera::profile_collect();
    size_t off = 0;
    buf[0] = 0;
    for (auto &kv : seera::prof().table) {
        const auto &g = kv.second;
        int w = snprintf(buf + off, size - off, "%s\t%d\t%llu\t%.6f\t%.6e\n", kv.first.c_str(), g.kind, (unsigned long long)g.n, g.ms, g.work);
        if (w < 0 || (size_t)w >= size - off) { buf[off] = 0; return fail(SEERA_E_LIMIT, "profile_report: buffer of %zu bytes is too small", size); }
        off += (size_t)w;
    }
    return SEERA_OK;
}

int seera_set_precision(int mode) {
    if (mode < 0 || mode > 5) return fail(SEERA_E_ARG, "seera_set_precision: mode %d", mode);
    rt().precision = mode;
    return SEERA_OK;
}
int seera_get_precision(void) { return rt().precision; }

void *seera_cuda_malloc(size_t n_bytes) {
    if (ensure_init()) return nullptr;
    Pool &p = pool();
    size_t sz = round_size(n_bytes);
    if (p.capturing) {
        auto ic = p.cap_free.find(sz);
        if (ic != p.cap_free.end() && !ic->second.empty()) {
            void *b = ic->second.back();
            ic->second.pop_back();
            p.live[b] = sz;
            return b;
        }
    }
    auto it = p.free_lists.find(sz);
    if (it != p.free_lists.end() && !it->second.empty()) {
        void *b = it->second.back();
        it->second.pop_back();
        p.live[b] = sz;
        if (p.capturing) { p.owner[b] = p.cur; p.cur->blocks.push_back({b, sz}); }
        return b;
    }
    // A pass that has to grow the pool (a new model's first) runs launch by launch from here: held back, its launches would wait out
    // every cudaMalloc of the pass, where the device can work through them meanwhile.
    if (batch_flush()) return nullptr;
    void *b = nullptr;
    cudaError_t e = cudaMalloc(&b, sz);
    if (e != cudaSuccess) {            // give cached blocks back to the driver and retry once
        cudaGetLastError();
        seera_pool_trim();
        e = cudaMalloc(&b, sz);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        fail(SEERA_E_OOM, "cuda_malloc(%zu): %s", n_bytes, cudaGetErrorString(e));
        return nullptr;
    }
    p.reserved += sz;
    p.live[b] = sz;
    if (p.capturing) { p.owner[b] = p.cur; p.cur->blocks.push_back({b, sz}); }
    return b;
}
void *seera_cuda_malloc_f32(int n) { return n < 0 ? nullptr : seera_cuda_malloc((size_t)n * 4); }
void *seera_cuda_malloc_i32(int n) { return n < 0 ? nullptr : seera_cuda_malloc((size_t)n * 4); }
void *seera_cuda_malloc_i16(int n) { return n < 0 ? nullptr : seera_cuda_malloc((size_t)n * 2); }

int seera_cuda_free(void *ptr) {
    if (!ptr) return SEERA_OK;
    Pool &p = pool();
    auto it = p.live.find(ptr);
    if (it == p.live.end()) return fail(SEERA_E_ARG, "cuda_free(%p): not a live block of this pool", ptr);
    if (ptr == rt().scaled_grad) rt().scaled_grad = nullptr;
    auto ow = p.owner.find(ptr);
    if (ow != p.owner.end()) {
        // a block a captured graph writes on every replay: reusable inside that capture, otherwise kept aside
        if (p.capturing && ow->second == p.cur) p.cap_free[it->second].push_back(ptr);
    } else {
        p.free_lists[it->second].push_back(ptr);
    }
    p.live.erase(it);
    return SEERA_OK;
}

int seera_pool_trim(void) {
    Pool &p = pool();
    if (int s = batch_flush()) return s;
    if (rt().stream) cudaStreamSynchronize(rt().stream);
    for (auto &kv : p.free_lists) {
        for (void *b : kv.second) { cudaFree(b); p.reserved -= kv.first; }
        kv.second.clear();
    }
    batch_trim();
    spares_trim(0);
    pinned_trim();
    return SEERA_OK;
}
size_t seera_pool_bytes_reserved(void) { return pool().reserved; }

int seera_graph_begin(void) {
    SEERA_ENSURE();
    Pool &p = pool();
    if (p.capturing) return fail(SEERA_E_ARG, "graph_begin: a capture is already open");
    if (int s = batch_flush()) return s;
    if (int s = check_cuda(cudaStreamBeginCapture(rt().stream, cudaStreamCaptureModeRelaxed), "cudaStreamBeginCapture")) return s;
    rt().scaled_grad = nullptr;
    p.cur = new GraphRec();
    p.cur->launches_at_begin = rt().launches;
    p.cap_free.clear();
    p.capturing = true;
    rt().capturing = true;
    return SEERA_OK;
}

void *seera_graph_end(void) {
    Pool &p = pool();
    if (!p.capturing) { fail(SEERA_E_ARG, "graph_end: no capture is open"); return nullptr; }
    p.capturing = false;
    rt().capturing = false;
    rt().scaled_grad = nullptr;
    p.cap_free.clear();
    GraphRec *g = p.cur;
    p.cur = nullptr;
    g->kernels = rt().launches - g->launches_at_begin;
    rt().launches = g->launches_at_begin;               // recorded, not executed
    cudaError_t e = cudaStreamEndCapture(rt().stream, &g->graph);
    if (e == cudaSuccess && !g->collectives) {
        if (chain_length(g->graph) == g->noted) g->row = g->hash | 1;
        if (g->row) take_spare(g);
    }
    if (e == cudaSuccess && !g->exec) e = cudaGraphInstantiate(&g->exec, g->graph, 0);
    if (e != cudaSuccess) {
        check_cuda(e, "graph_end");
        cudaGetLastError();
        seera_graph_destroy(g);
        return nullptr;
    }
    live_graphs().push_back(g);
    return g;
}

int seera_graph_launch(void *graph) {
    SEERA_ENSURE();
    GraphRec *g = static_cast<GraphRec *>(graph);
    if (int s = batch_flush()) return s;
    if (!g || !g->exec) return fail(SEERA_E_ARG, "graph_launch: not a captured graph (or one whose communicator has been finalized)");
    rt().launches += g->kernels;
    return check_cuda(cudaGraphLaunch(g->exec, rt().stream), "cudaGraphLaunch");
}

int seera_graph_destroy(void *graph) {
    GraphRec *g = static_cast<GraphRec *>(graph);
    if (!g) return SEERA_OK;
    Pool &p = pool();
    batch_flush();
    if (rt().stream) cudaStreamSynchronize(rt().stream);
    keep_spare(g);
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    for (auto &b : g->blocks) {
        p.owner.erase(b.first);
        if (!p.live.count(b.first)) p.free_lists[b.second].push_back(b.first);   // idle: back to the general pool
    }
    for (int s : g->finish_slots) finish_slots().free.push_back(s);
    auto &lg = live_graphs();
    for (size_t i = 0; i < lg.size(); i++)
        if (lg[i] == g) { lg.erase(lg.begin() + (long)i); break; }
    delete g;
    return SEERA_OK;
}
int seera_is_capturing(void) { return pool().capturing ? 1 : 0; }

int seera_graph_set_scalars(void *graph, const float *values, int n) {
    GraphRec *g = static_cast<GraphRec *>(graph);
    if (!g || !g->exec || !values) return fail(SEERA_E_ARG, "graph_set_scalars: not a captured graph");
    if (g->lost_update) return fail(SEERA_E_ARG, "graph_set_scalars: the recording holds an update whose scalars cannot be replaced");
    for (OptNode &o : g->optimizers) {
        if (n != o.launch.n_scalars) return fail(SEERA_E_ARG, "graph_set_scalars: %d values for an update of %d", n, o.launch.n_scalars);
        memcpy(o.launch.scalars, values, (size_t)n * sizeof(float));
        cudaKernelNodeParams kp = {};
        void *args[OptLaunch::MAX_ARGS];
        optimizer_node_params(o.launch, kp, args);
        if (int s = check_cuda(cudaGraphExecKernelNodeSetParams(g->exec, o.node, &kp), "cudaGraphExecKernelNodeSetParams")) return s;
    }
    return SEERA_OK;
}

// Page-locked host blocks.  The driver takes milliseconds to pin and unpin a block (3 ms for 200 KB measured; a training loop of
// eight steps took 1 to 7 ms for its five blocks and 0.9 ms for the steps), so freed blocks are kept for the next request of
// their rounded size, up to PINNED_KEPT_MAX bytes; seera_pool_trim gives them back.  A kept block is handed out again once the work that
// was queued when it was freed has passed, since a copy may still be reading it.
}  // extern "C"
static cudaStream_t copy_stream(int *status);
namespace {
constexpr size_t PINNED_KEPT_MAX = size_t(256) << 20;
struct PinnedBlock { void *p; cudaEvent_t compute, copy; };
struct Pinned {
    std::mutex mu;
    std::unordered_map<void *, size_t> live;
    std::map<size_t, std::vector<PinnedBlock>> kept;
    size_t kept_bytes = 0;
    bool other_streams = false;                         // seera_set_stream was used: a copy may be queued on a stream not watched here
};
Pinned &pinned() { static Pinned p; return p; }
size_t pinned_round(size_t n) {                       // powers of two from a page up to 1 MiB, then 2 MiB granules
    if (n > (size_t(1) << 20)) return (n + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1);
    size_t r = 4096;
    while (r < n) r <<= 1;
    return r;
}
void pinned_drop(PinnedBlock &b) {
    cudaEventDestroy(b.compute); cudaEventDestroy(b.copy);
    cudaFreeHost(b.p);
}
}  // namespace
static void pinned_other_streams() { pinned().other_streams = true; }
static void pinned_trim() {
    Pinned &k = pinned();
    std::lock_guard<std::mutex> lock(k.mu);
    for (auto &kv : k.kept) for (PinnedBlock &b : kv.second) pinned_drop(b);
    k.kept.clear();
    k.kept_bytes = 0;
}
extern "C" {
void *seera_host_alloc_pinned(size_t n) {
    if (ensure_init()) return nullptr;
    Pinned &k = pinned();
    const size_t sz = pinned_round(n);
    std::lock_guard<std::mutex> lock(k.mu);
    auto it = k.kept.find(sz);
    if (it != k.kept.end())
        for (size_t i = 0; i < it->second.size(); i++) {
            PinnedBlock b = it->second[i];
            if (cudaEventQuery(b.compute) != cudaSuccess || cudaEventQuery(b.copy) != cudaSuccess) { cudaGetLastError(); continue; }
            it->second.erase(it->second.begin() + (long)i);
            k.kept_bytes -= sz;
            cudaEventDestroy(b.compute); cudaEventDestroy(b.copy);
            k.live[b.p] = sz;
            return b.p;
        }
    void *p = nullptr;
    if (cudaMallocHost(&p, sz) != cudaSuccess) { cudaGetLastError(); fail(SEERA_E_OOM, "cudaMallocHost(%zu)", n); return nullptr; }
    k.live[p] = sz;
    return p;
}
int seera_host_free_pinned(void *p) {
    if (!p) return SEERA_OK;
    if (int s = batch_flush()) return s;
    Pinned &k = pinned();
    std::lock_guard<std::mutex> lock(k.mu);
    auto it = k.live.find(p);
    const size_t sz = it == k.live.end() ? 0 : it->second;
    if (sz) k.live.erase(it);
    int st = SEERA_OK;
    cudaStream_t cs = nullptr;
    if (sz && !k.other_streams && !rt().capturing && rt().stream && k.kept_bytes + sz <= PINNED_KEPT_MAX && (cs = copy_stream(&st))) {
        PinnedBlock b{p, nullptr, nullptr};
        bool ok = cudaEventCreateWithFlags(&b.compute, cudaEventDisableTiming) == cudaSuccess;
        if (ok && cudaEventCreateWithFlags(&b.copy, cudaEventDisableTiming) != cudaSuccess) { cudaEventDestroy(b.compute); ok = false; }
        if (ok && (cudaEventRecord(b.compute, rt().stream) != cudaSuccess || cudaEventRecord(b.copy, cs) != cudaSuccess)) {
            cudaEventDestroy(b.compute); cudaEventDestroy(b.copy);
            ok = false;
        }
        if (ok) {
            k.kept[sz].push_back(b);
            k.kept_bytes += sz;
            return SEERA_OK;
        }
        cudaGetLastError();
    }
    return check_cuda(cudaFreeHost(p), "cudaFreeHost");
}

int seera_cuda_memcopy_devicetodevice(void *dst, const void *src, int num_elem) {
    SEERA_ENSURE();
    if (num_elem < 0 || !dst || !src) return fail(SEERA_E_ARG, "memcopy_devicetodevice: bad argument");
    return check_cuda(cudaMemcpyAsync(dst, src, (size_t)num_elem * sizeof(float), cudaMemcpyDeviceToDevice, rt().stream),
                      "cudaMemcpyAsync d2d");
}
int seera_cuda_memset(void *ptr, int value, size_t n_bytes) {
    SEERA_ENSURE();
    if (!ptr) return fail(SEERA_E_ARG, "cuda_memset: null");
    return check_cuda(cudaMemsetAsync(ptr, value, n_bytes, rt().stream), "cudaMemsetAsync");
}

void *seera_to_device(const void *host, size_t n_bytes) {
    void *d = seera_cuda_malloc(n_bytes);
    if (!d) return nullptr;
    if (n_bytes && seera_upload(d, host, n_bytes)) { seera_cuda_free(d); return nullptr; }
    return d;
}
int seera_upload(void *dev, const void *host, size_t n_bytes) {
    SEERA_ENSURE();
    if (!dev || !host) return fail(SEERA_E_ARG, "upload: null");
    if (int s = batch_flush()) return s;
    // From pageable memory the runtime stages the copy before returning, so the caller may reuse
    // `host` at once; from pinned memory the copy is asynchronous and ordered on the stream.
    return check_cuda(cudaMemcpyAsync(dev, host, n_bytes, cudaMemcpyHostToDevice, rt().stream), "cudaMemcpyAsync h2d");
}
// ---- measurement aid: hold the stream for a while so that the launches that follow queue up behind it ---------
// Events recorded around a kernel in an eagerly launched sequence otherwise also time the host's gaps between launches.
__global__ void stream_delay_kernel(long long clocks) {
    const long long t0 = clock64();
    while (clock64() - t0 < clocks) {}          // bounded by `clocks` (at most 0.1 s worth, see below)
}
int seera_stream_delay(int microseconds) {
    SEERA_ENSURE();
    if (microseconds < 0 || microseconds > 100000) return fail(SEERA_E_ARG, "stream_delay: 0..100000 microseconds");
    if (int s = batch_flush()) return s;
    if (rt().capturing) return fail(SEERA_E_ARG, "stream_delay: not allowed while a graph is being captured");
    int khz = 0;
    if (cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, rt().device) != cudaSuccess || khz <= 0) { cudaGetLastError(); khz = 1500000; }
    stream_delay_kernel<<<1, 1, 0, rt().stream>>>((long long)microseconds * khz / 1000);
    SEERA_LAUNCH_CHECK("stream_delay");
    return SEERA_OK;
}

// ---- copy stream: host<->device transfers that overlap the compute stream -----------------------------------
// One extra non-blocking stream per process.  Ordering against the compute stream is explicit: each fence records an
// event at the current tail of one stream and makes the other wait for it, so "everything queued so far" is the unit.
}  // extern "C"
static cudaStream_t copy_stream(int *status) {
    static cudaStream_t cs[64] = {nullptr};
    const int dev = rt().device & 63;
    if (!cs[dev]) {
        cudaError_t e = cudaStreamCreateWithFlags(&cs[dev], cudaStreamNonBlocking);
        if (e != cudaSuccess) { *status = check_cuda(e, "cudaStreamCreate(copy)"); return nullptr; }
    }
    return cs[dev];
}
extern "C" {
static int fence(cudaStream_t from, cudaStream_t to, const char *what) {
    cudaEvent_t ev;
    if (int s = check_cuda(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), what)) return s;
    cudaError_t e = cudaEventRecord(ev, from);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(to, ev, 0);
    cudaEventDestroy(ev);              // released once the recorded work has completed
    return check_cuda(e, what);
}
static int copy_guard(const char *what) {
    if (rt().capturing) return fail(SEERA_E_ARG, "%s: not allowed while a graph is being captured", what);
    return batch_flush();
}
int seera_copy_upload(void *dev, const void *pinned_host, size_t n_bytes) {
    SEERA_ENSURE();
    if (!dev || !pinned_host) return fail(SEERA_E_ARG, "copy_upload: null");
    if (int s = copy_guard("copy_upload")) return s;
    int st = SEERA_OK; cudaStream_t cs = copy_stream(&st); if (!cs) return st;
    return check_cuda(cudaMemcpyAsync(dev, pinned_host, n_bytes, cudaMemcpyHostToDevice, cs), "cudaMemcpyAsync h2d (copy stream)");
}
int seera_copy_download(void *pinned_host, const void *dev, size_t n_bytes) {
    SEERA_ENSURE();
    if (!dev || !pinned_host) return fail(SEERA_E_ARG, "copy_download: null");
    if (int s = copy_guard("copy_download")) return s;
    int st = SEERA_OK; cudaStream_t cs = copy_stream(&st); if (!cs) return st;
    return check_cuda(cudaMemcpyAsync(pinned_host, dev, n_bytes, cudaMemcpyDeviceToHost, cs), "cudaMemcpyAsync d2h (copy stream)");
}
int seera_copy_wait_compute(void) {
    SEERA_ENSURE();
    if (int s = copy_guard("copy_wait_compute")) return s;
    int st = SEERA_OK; cudaStream_t cs = copy_stream(&st); if (!cs) return st;
    return fence(rt().stream, cs, "copy_wait_compute");
}
int seera_compute_wait_copy(void) {
    SEERA_ENSURE();
    if (int s = copy_guard("compute_wait_copy")) return s;
    int st = SEERA_OK; cudaStream_t cs = copy_stream(&st); if (!cs) return st;
    return fence(cs, rt().stream, "compute_wait_copy");
}
int seera_copy_synchronize(void) {
    SEERA_ENSURE();
    if (int s = copy_guard("copy_synchronize")) return s;
    int st = SEERA_OK; cudaStream_t cs = copy_stream(&st); if (!cs) return st;
    return check_cuda(cudaStreamSynchronize(cs), "cudaStreamSynchronize(copy)");
}

int seera_to_host(void *host, const void *dev, size_t n_bytes) {
    SEERA_ENSURE();
    if (!dev || !host) return fail(SEERA_E_ARG, "to_host: null");
    if (int s = batch_flush()) return s;
    if (rt().capturing) return fail(SEERA_E_ARG, "to_host: not allowed while a graph is being captured");
    if (int s = check_cuda(cudaMemcpyAsync(host, dev, n_bytes, cudaMemcpyDeviceToHost, rt().stream), "cudaMemcpyAsync d2h")) return s;
    return check_cuda(cudaStreamSynchronize(rt().stream), "cudaStreamSynchronize");
}

}  // extern "C"
