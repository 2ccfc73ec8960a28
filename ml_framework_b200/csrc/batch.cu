// Batches: many launches, one submission (seera_batch_begin / _end).
//
// A launch costs the host about 2.8 us here, and separate launches leave the device 1-2 us between kernels.  Inside a batch the library's
// launches are therefore noted down - kernel, grid, a copy of its arguments: 0.1 us - and handed over together as a graph.  The executable
// graph of a batch is kept, for the next batch of the same kernels and grids in a row; that one has to replace only the launches whose
// arguments differ from the time before (0.25 us each; none in a loop that finds its buffers again).  14 launches: 5 us of host time if
// all of them differ, 1.5 if none does, against 39 one by one; 50 launches: 16 against 141.
//
// The stream is not captured meanwhile.  A capture would forbid every other thread of the process to synchronise the device (and lose the
// batch if one did), would take in what a caller enqueues on the stream by itself, and costs twice as much (0.25 us a launch, and 0.45
// for comparing an executable with the captured graph).  The library's launches are seen by the linker instead: build.py resolves
// cudaLaunchKernel, cudaLaunchKernelExC, cudaMemsetAsync and cudaMemcpyAsync of this library's objects to the functions below.
//
// Kernels and grids are never replaced in an executable: from then on it runs slower, also back at what it was made of (an autoencoder step
// of 64 images 236 us, 251 with the executable of a step of 8, of the same kernels; then 182 for 174 at 8).  A row of kernels and grids
// is given an executable the second time it comes by, while BATCH_KEPT_MAX leave room or one of them has been passed over by BATCH_STALE
// batches; any other batch is launched call by call.  Nothing here waits for the device: an executable graph that is destroyed while it
// runs is freed when it ends.
#include <algorithm>
#include <cstring>
#include <memory>
#include <new>
#include <unordered_map>
#include <unordered_set>
#include <vector>

#include "common.cuh"

extern "C" {
cudaError_t __real_cudaLaunchKernel(const void *func, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t stream);
cudaError_t __real_cudaLaunchKernelExC(const cudaLaunchConfig_t *config, const void *func, void **args);
cudaError_t __real_cudaMemsetAsync(void *dst, int value, size_t bytes, cudaStream_t stream);
cudaError_t __real_cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind kind, cudaStream_t stream);
}

namespace seera {
namespace {

struct alignas(64) Chunk { unsigned char b[64]; };
struct Op {
    enum Kind : unsigned { KERNEL, FILL, COPY } kind;
    unsigned cluster, value;            // blocks of a cluster (1: none); the byte of a fill
    const void *what, *src;             // kernel, or destination; source of a copy
    dim3 grid, block;
    size_t bytes;                       // dynamic shared memory, or length
    size_t at, chunks;                  // the arguments among `data`
    bool same_launch(const Op &o) const {
        return kind == o.kind && (kind != KERNEL || (cluster == o.cluster && what == o.what && bytes == o.bytes && grid.x == o.grid.x &&
                                                     grid.y == o.grid.y && grid.z == o.grid.z && block.x == o.block.x && block.y == o.block.y &&
                                                     block.z == o.block.z));
    }
    bool same_memory(const Op &o) const { return value == o.value && what == o.what && src == o.src && bytes == o.bytes; }
};
struct Row {
    std::vector<Op> ops;
    std::vector<Chunk> data;
};
// Where a kernel's arguments lie in its parameter block.
struct Layout {
    std::vector<std::pair<size_t, size_t>> args;      // offset, size
    size_t chunks = 0;
};
struct Kept {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<cudaGraphNode_t> nodes;
    Row now;                                            // what the executable holds
    uint64_t used = 0;
    ~Kept() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
    }
};
struct State {
    bool open = false;                                  // launches of the thread `owner` on `stream` are noted down
    const int *owner = nullptr;
    bool parted = false;                                // a first part of the batch has been submitted
    uint64_t tag = 0, inner_at = 0;                     // ... and the launch count where the batch directly inside began
    cudaStream_t stream = nullptr;
    Row row;
    cudaEvent_t last = nullptr;                         // behind the last batch
    std::unordered_map<uint64_t, std::unique_ptr<Kept>> kept;
    std::unordered_set<uint64_t> sighted;               // rows that have come by once
    uint64_t clock = 0, replaced = 0;                   // batches submitted; when an executable last made room for another
    std::unordered_map<const void *, Layout> layouts;
    std::vector<void *> argv;
};
constexpr size_t BATCH_KEPT_MAX = 64, BATCH_SIGHTED_MAX = 4096;
// An executable takes 125 us to make and 110 to destroy (14 launches): one in BATCH_TURN batches may go for another.
constexpr uint64_t BATCH_STALE = 1024, BATCH_TURN = 64;
// The first pass inside a batch that makes this many launches is submitted at its end if the device has finished the batch before: a
// step that is waited for would else run host and device one after the other (VGG at 100 images: 557 -> 474 us).  Below that the
// second submission (6 us) costs a small network more than the device's head start gives.
constexpr uint64_t BATCH_PART = 12;
thread_local int depth = 0;                             // batches that this thread has begun and not ended; its address names the thread
State &st() { static State &s = *new State; return s; }          // not destroyed: the driver may be gone before

const Layout &layout_of(const void *func) {
    State &b = st();
    auto it = b.layouts.find(func);
    if (it != b.layouts.end()) return it->second;
    Layout l;
    size_t off, size, end = 0;
    while (cudaFuncGetParamInfo(func, l.args.size(), &off, &size) == cudaSuccess) {
        l.args.push_back({off, size});
        end = std::max(end, off + size);
    }
    cudaGetLastError();                                 // the index behind the last argument
    l.chunks = (end + sizeof(Chunk) - 1) / sizeof(Chunk);
    return b.layouts.emplace(func, std::move(l)).first->second;
}
void **arguments(const Op &op, Row &row) {
    State &b = st();
    const Layout &l = layout_of(op.what);
    unsigned char *p = op.chunks ? row.data[op.at].b : nullptr;
    b.argv.resize(l.args.size() + 1);
    for (size_t i = 0; i < l.args.size(); i++) b.argv[i] = p + l.args[i].first;
    return b.argv.data();
}

void note_kernel(const void *func, dim3 grid, dim3 block, void **args, size_t smem, unsigned cluster) {
    Row &r = st().row;
    const Layout &l = layout_of(func);
    const size_t at = r.data.size();
    r.data.resize(at + l.chunks, Chunk{});
    for (size_t i = 0; i < l.args.size(); i++) memcpy(r.data[at].b + l.args[i].first, args[i], l.args[i].second);
    r.ops.push_back({Op::KERNEL, cluster, 0, func, nullptr, grid, block, smem, at, l.chunks});
}

cudaError_t launch_alone(const Op &op, Row &row, cudaStream_t stream) {
    if (op.kind == Op::FILL) return __real_cudaMemsetAsync(const_cast<void *>(op.what), (int)op.value, op.bytes, stream);
    if (op.kind == Op::COPY) return __real_cudaMemcpyAsync(const_cast<void *>(op.what), op.src, op.bytes, cudaMemcpyDeviceToDevice, stream);
    if (op.cluster == 1) return __real_cudaLaunchKernel(op.what, op.grid, op.block, arguments(op, row), op.bytes, stream);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = op.grid; cfg.blockDim = op.block; cfg.dynamicSmemBytes = op.bytes; cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = op.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    return __real_cudaLaunchKernelExC(&cfg, op.what, arguments(op, row));
}
cudaKernelNodeParams node_params(const Op &op, Row &row) {
    cudaKernelNodeParams kp = {};
    kp.func = const_cast<void *>(op.what);
    kp.gridDim = op.grid; kp.blockDim = op.block; kp.sharedMemBytes = (unsigned)op.bytes;
    kp.kernelParams = arguments(op, row);
    return kp;
}
cudaError_t add_node(Kept &k, const Op &op, Row &row) {
    cudaGraphNode_t node = nullptr;
    const cudaGraphNode_t *before = k.nodes.empty() ? nullptr : &k.nodes.back();
    const size_t n = k.nodes.empty() ? 0 : 1;
    cudaError_t e;
    if (op.kind == Op::KERNEL) {
        const cudaKernelNodeParams kp = node_params(op, row);
        e = cudaGraphAddKernelNode(&node, k.graph, before, n, &kp);
        if (e == cudaSuccess && op.cluster > 1) {
            cudaKernelNodeAttrValue v = {};
            v.clusterDim.x = op.cluster; v.clusterDim.y = 1; v.clusterDim.z = 1;
            e = cudaGraphKernelNodeSetAttribute(node, cudaLaunchAttributeClusterDimension, &v);
        }
    } else if (op.kind == Op::FILL) {
        const cudaMemsetParams mp = {const_cast<void *>(op.what), 0, op.value, 1, op.bytes, 1};
        e = cudaGraphAddMemsetNode(&node, k.graph, before, n, &mp);
    } else {
        e = cudaGraphAddMemcpyNode1D(&node, k.graph, before, n, const_cast<void *>(op.what), op.src, op.bytes, cudaMemcpyDeviceToDevice);
    }
    if (e == cudaSuccess) k.nodes.push_back(node);
    return e;
}
cudaError_t replace_node(Kept &k, size_t i, const Op &op, Row &row) {
    if (op.kind == Op::KERNEL) {
        const cudaKernelNodeParams kp = node_params(op, row);
        return cudaGraphExecKernelNodeSetParams(k.exec, k.nodes[i], &kp);
    }
    if (op.kind == Op::FILL) {
        const cudaMemsetParams mp = {const_cast<void *>(op.what), 0, op.value, 1, op.bytes, 1};
        return cudaGraphExecMemsetNodeSetParams(k.exec, k.nodes[i], &mp);
    }
    return cudaGraphExecMemcpyNodeSetParams1D(k.exec, k.nodes[i], const_cast<void *>(op.what), op.src, op.bytes, cudaMemcpyDeviceToDevice);
}

uint64_t key_of(uint64_t tag, const Row &row) {
    uint64_t h = 1469598103934665603ull ^ tag;
    auto mix = [&h](uint64_t v) { h = (h ^ v) * 1099511628211ull; h ^= h >> 32; };
    for (const Op &o : row.ops) {
        mix(o.kind * 64 + o.cluster);
        if (o.kind != Op::KERNEL) continue;
        mix((uint64_t)(uintptr_t)o.what);
        mix(((uint64_t)o.grid.x << 32) ^ ((uint64_t)o.grid.y << 16) ^ o.grid.z);
        mix(((uint64_t)o.bytes << 32) ^ ((uint64_t)o.block.x << 16) ^ (o.block.y << 8) ^ o.block.z);
    }
    return h;
}
// Gives a kept executable the row's arguments; false: it is not one for the row, or no longer.
bool bring_up(Kept &k, Row &row) {
    if (k.now.ops.size() != row.ops.size()) return false;
    for (size_t i = 0; i < row.ops.size(); i++)
        if (!row.ops[i].same_launch(k.now.ops[i])) return false;
    for (size_t i = 0; i < row.ops.size(); i++) {       // the same kernels: the same places among the arguments
        const Op &o = row.ops[i];
        const bool args = o.chunks && memcmp(&row.data[o.at], &k.now.data[o.at], o.chunks * sizeof(Chunk)) != 0;
        if (!args && o.same_memory(k.now.ops[i])) continue;
        if (replace_node(k, i, o, row) != cudaSuccess) { cudaGetLastError(); return false; }
        k.now.ops[i] = o;
        if (args) std::copy_n(row.data.begin() + (long)o.at, o.chunks, k.now.data.begin() + (long)o.at);
    }
    return true;
}
bool make(Kept &k, Row &row) {
    if (cudaGraphCreate(&k.graph, 0) != cudaSuccess) { cudaGetLastError(); return false; }
    for (const Op &o : row.ops)
        if (add_node(k, o, row) != cudaSuccess) { cudaGetLastError(); return false; }
    if (cudaGraphInstantiate(&k.exec, k.graph, 0) != cudaSuccess) { cudaGetLastError(); return false; }
    k.now = row;
    return true;
}
// Room for one more executable?
bool room() {
    State &b = st();
    if (b.kept.size() < BATCH_KEPT_MAX) return true;
    auto old = b.kept.begin();
    for (auto i = b.kept.begin(); i != b.kept.end(); ++i) if (i->second->used < old->second->used) old = i;
    if (b.clock - old->second->used <= BATCH_STALE || b.clock - b.replaced < BATCH_TURN) return false;
    b.replaced = b.clock;
    b.kept.erase(old);
    return true;
}

// The executable for what has been noted down, with its arguments, or null.
const Kept *executable(bool whole) {
    State &b = st();
    const uint64_t key = key_of(b.tag, b.row);
    Kept *k = nullptr;
    try {
        auto it = b.kept.find(key);
        if (it != b.kept.end()) {
            k = it->second.get();
            if (!bring_up(*k, b.row)) {
                b.kept.erase(it);
                return nullptr;
            }
        } else if (whole && !b.sighted.insert(key).second && room()) {
            auto fresh = std::make_unique<Kept>();
            if (!make(*fresh, b.row)) return nullptr;
            k = fresh.get();
            b.kept[key] = std::move(fresh);
        }
        if (b.sighted.size() > BATCH_SIGHTED_MAX) b.sighted.clear();
    } catch (const std::bad_alloc &) {                   // no host memory for one: call by call
        b.kept.clear();
        return nullptr;
    }
    if (k) k->used = b.clock;
    return k;
}

// Hands over what has been noted down.  `whole`: all of a batch, whose executable is worth keeping.
int submit(bool whole) {
    State &b = st();
    if (!b.open) return SEERA_OK;
    b.open = false;
    Row &row = b.row;
    cudaError_t e = cudaSuccess;
    if (!row.ops.empty()) {
        ++b.clock;
        const Kept *k = executable(whole);
        if (k) {
            e = cudaGraphLaunch(k->exec, b.stream);
        } else {
            for (size_t i = 0; i < row.ops.size() && e == cudaSuccess; i++) e = launch_alone(row.ops[i], row, b.stream);
        }
        row.ops.clear();
        row.data.clear();
        if (e == cudaSuccess && (b.last || cudaEventCreateWithFlags(&b.last, cudaEventDisableTiming) == cudaSuccess))
            e = cudaEventRecord(b.last, b.stream);
    }
    if (e == cudaSuccess) return SEERA_OK;
    cudaGetLastError();
    return check_cuda(e, "batch");
}
void open(uint64_t tag) {
    State &b = st();
    b.open = true;
    b.owner = &depth;
    b.tag = tag;
    b.stream = rt().stream;
}
// Notes a launch down, or, where there is no memory for that or another thread launches on the stream, submits what there is and says no.
template <class Note>
bool noted(cudaStream_t stream, Note note) {
    State &b = st();
    if (!b.open || stream != b.stream) return false;
    if (b.owner != &depth) { submit(false); return false; }
    const size_t ops = b.row.ops.size();
    try {
        note();
        return true;
    } catch (const std::bad_alloc &) {
        b.row.ops.resize(ops);
        submit(false);
        return false;
    }
}
}  // namespace

int batch_flush() { return submit(false); }
void batch_trim() {
    st().kept.clear();
    st().sighted.clear();
}

cudaError_t allow_smem(const void *kernel, size_t bytes) {
    static std::unordered_map<const void *, size_t> limits;
    size_t &now = limits[kernel];
    if (bytes <= (now ? now : 32 * 1024)) return cudaSuccess;           // (48 KB with what the kernel has of its own are always allowed)
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) now = bytes;
    return e;
}

}  // namespace seera

using namespace seera;

extern "C" {

// The library's own launches arrive here.
cudaError_t __wrap_cudaLaunchKernel(const void *func, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t stream) {
    if (noted(stream, [&] { note_kernel(func, grid, block, args, smem, 1); })) return cudaSuccess;
    if (rt().capturing) graph_note_launch(func, grid, block, smem);
    return __real_cudaLaunchKernel(func, grid, block, args, smem, stream);
}
cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *config, const void *func, void **args) {
    const bool cluster = config->numAttrs == 1 && config->attrs[0].id == cudaLaunchAttributeClusterDimension &&
                         config->attrs[0].val.clusterDim.y == 1 && config->attrs[0].val.clusterDim.z == 1;
    const unsigned c = cluster ? config->attrs[0].val.clusterDim.x : 1;
    if (config->numAttrs == 0 || cluster) {
        if (noted(config->stream, [&] { note_kernel(func, config->gridDim, config->blockDim, args, config->dynamicSmemBytes, c); })) return cudaSuccess;
    } else if (st().open && config->stream == st().stream) {
        submit(false);
    }
    if (rt().capturing) graph_note_launch(func, config->gridDim, config->blockDim, config->dynamicSmemBytes + ((size_t)c << 24));
    return __real_cudaLaunchKernelExC(config, func, args);
}
cudaError_t __wrap_cudaMemsetAsync(void *dst, int value, size_t bytes, cudaStream_t stream) {
    if (bytes && noted(stream, [&] { st().row.ops.push_back({Op::FILL, 1, (unsigned)value & 255u, dst, nullptr, {}, {}, bytes, 0, 0}); }))
        return cudaSuccess;
    if (rt().capturing) graph_note_launch(nullptr, {}, {}, 1);
    return __real_cudaMemsetAsync(dst, value, bytes, stream);
}
cudaError_t __wrap_cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind kind, cudaStream_t stream) {
    if (kind != cudaMemcpyDeviceToDevice) {
        if (st().open && stream == st().stream) submit(false);
    } else if (bytes && noted(stream, [&] { st().row.ops.push_back({Op::COPY, 1, 0, dst, src, {}, {}, bytes, 0, 0}); })) {
        return cudaSuccess;
    }
    if (rt().capturing) graph_note_launch(nullptr, {}, {}, 2);
    return __real_cudaMemcpyAsync(dst, src, bytes, kind, stream);
}

int seera_batch_begin(uint64_t tag) {
    SEERA_ENSURE();
    State &b = st();
    if (depth++ > 0) {
        if (depth == 2) b.inner_at = rt().launches;
        return SEERA_OK;
    }
    if (int s = submit(false)) return s;                // another thread's: the rest of it goes call by call
    b.parted = false;
    if (rt().capturing || seera_profile_enabled() || rt().stream == nullptr) return SEERA_OK;
    cudaStreamCaptureStatus status;
    if (cudaStreamIsCapturing(rt().stream, &status) != cudaSuccess || status != cudaStreamCaptureStatusNone) { cudaGetLastError(); return SEERA_OK; }
    open(tag);
    return SEERA_OK;
}
int seera_batch_end(void) {
    State &b = st();
    if (depth == 0) return fail(SEERA_E_ARG, "batch_end: no batch is open");
    --depth;
    if (!b.open || b.owner != &depth) return SEERA_OK;
    if (depth == 0) return submit(true);
    if (b.parted || depth > 1 || rt().launches - b.inner_at < BATCH_PART) return SEERA_OK;
    if (b.last && cudaEventQuery(b.last) != cudaSuccess) { cudaGetLastError(); return SEERA_OK; }
    b.parted = true;
    if (int s = submit(true)) return s;
    open(b.tag);
    return SEERA_OK;
}
int seera_batches_kept(void) { return (int)st().kept.size(); }

}  // extern "C"
