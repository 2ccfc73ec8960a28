// Shared host-side state and helpers for the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include "seera_b200.h"

namespace seera {

struct Runtime {
    int device = -1;
    int sm_count = 148;                 // SMs the kernels size their grids for (physical count minus the "sm_reserve" option)
    int sm_physical = 148;
    cudaStream_t stream = nullptr;      // the stream every kernel is enqueued on
    cudaStream_t own_stream = nullptr;
    int precision = 0;                  // set from SEERA_PRECISION (default 3) when the runtime is created
    unsigned long long tc_wait_clocks = 4000000000ull;      // budget of a bounded wait inside a tensor-core kernel (~2 s)
    int tc_test_skip_load = -1;         // test hook ("tc_test_skip_load" option): see TmaGemmParams::skip_load
    bool graph_test_lose_update = false;        // test hook ("graph_test_lose_update" option): the next recorded update cannot name its node
    bool dense_tma = true;              // Dense GEMMs in modes 1/2: TMA-fed kernel (false: in-kernel conversion kernel)
    int tile_n_cap2 = 128;              // widest accumulator tile with two operand copies per stage (bf16x3)
    int tile_n_cap3 = 128;              // ... with three (bf16x6)
    bool pool_short_patch = false;      // fold a 2x2 max-pool into the tensor-core short-patch forward kernel too (its epilogue warps become the
                                        // bottleneck: off; 3 x 3 unit-stride layers fold it into the fp32 stencil kernel regardless)
    bool wgrad_single = true;           // precision mode 4: weight gradients from the first fp16 copy of each operand alone
    bool skinny_gemm = true;            // Dense products of at most 16 output columns: exact fp32 on the CUDA cores in every mode
    int mma_issuers = 0;                // cap on the MMA-issuing threads of the TMA-fed GEMM kernel (0: none; 1 or 2)
    bool pair_tiles = false;            // TMA-fed GEMMs as clusters of two CTAs on 256-row tiles where the plan finds it pays
    bool conv_tma = true;               // convolutions in modes 1-3: TMA im2col kernel (false: in-kernel gather kernel)
    // the loss gradient whose largest entry the loss head has already turned into the dynamic factor (grad_scale_of_loss then has
    // nothing left to do for it)
    const float *scaled_grad = nullptr;
    long long scaled_n = 0;
    bool capturing = false;             // a stream capture (seera_graph_begin) is open
    bool tc_used = false;               // a tensor-core kernel ran since the status word was last read
    int status = 0;
    uint64_t launches = 0;
    char err[512] = {0};
};
Runtime &rt();
int fail(int code, const char *fmt, ...);       // records the status + message, returns code
int check_cuda(cudaError_t e, const char *what);
int ensure_init();

// Grid for a grid-stride kernel over `work_items` with `threads` per block: enough blocks to cover
// the work once, capped at a whole number of waves (8 resident 256-thread CTAs per SM).
inline int stride_grid(long long work_items, int threads = 256) {
    long long need = (work_items + threads - 1) / threads;
    long long cap = (long long)rt().sm_count * 8;
    if (need < 1) need = 1;
    return (int)(need < cap ? need : cap);
}

inline void count_launch(int n = 1) { rt().launches += n; }

// out[c] = sum over s < splits of partial[s * n + c], added in a fixed order (the same bits on every run).  A block owns 32
// consecutive columns; its warps take the splits w, w + warps, ... (128-byte coalesced reads), then their sums are added in warp
// order.  Columns at or beyond n_first go to out2 (may be null).  What such a launch waits for is the chain of reads of one warp: up to
// 32 warps keep it at a few reads however many splits there are (288 columns of 296 splits: 8 us with 8 warps).
static __global__ void __launch_bounds__(1024) sum_splits_kernel(const float *__restrict__ partial, float *__restrict__ out,
                                                                 float *__restrict__ out2, int n_first, int n, int splits) {
    __shared__ float sm[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5, c = blockIdx.x * 32 + lane;
    float t = 0.f;
    if (c < n)
        for (int s = warp; s < splits; s += 8 * warps) {
            float v[8];                                       // all of them requested before the first is added
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = s + k * warps < splits ? __ldg(partial + (long long)(s + k * warps) * n + c) : 0.f;
#pragma unroll
            for (int k = 0; k < 8; k++) t += v[k];
        }
    sm[warp][lane] = t;
    __syncthreads();
    if (warp == 0 && c < n) {
        float r = sm[0][lane];
        for (int w = 1; w < warps; w++) r += sm[w][lane];
        if (c < n_first) out[c] = r;
        else if (out2) out2[c - n_first] = r;
    }
}
inline void launch_sum_splits(const float *partial, float *out, int n, int splits, cudaStream_t st, float *out2 = nullptr, int n_first = -1) {
    const int threads = splits <= 64 ? 256 : (splits <= 128 ? 512 : 1024);
    sum_splits_kernel<<<(n + 31) / 32, threads, 0, st>>>(partial, out, out2, n_first < 0 ? n : n_first, n, splits);
    count_launch();
}

#define SEERA_ENSURE()                      \
    do {                                    \
        int _s = seera::ensure_init();      \
        if (_s) return _s;                  \
    } while (0)

#define SEERA_LAUNCH_CHECK(name)                                                   \
    do {                                                                           \
        seera::count_launch();                                                     \
        cudaError_t _e = cudaGetLastError();                                       \
        if (_e != cudaSuccess) return seera::check_cuda(_e, name);                 \
    } while (0)

// Two fp32 multiply-adds per instruction (each half rounded as fmaf rounds): the way to the full fp32 rate on sm_100.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Contraction profile (seera_profile_enable): bracket a launch sequence with events and book its FLOPs.
void profile_begin();
void profile_end_bytes(double bytes, const char *tag);      // a bandwidth-bound pass: its algorithmic bytes
void profile_end(double flops, const char *name = nullptr);    // name ending in (dX)/(dA) or (dW)/(dB) books the launch as a backward product

// Brackets the launches of a bandwidth-bound pass for the profile: constructed before them, destroyed after them.
struct ProfBytes {
    double bytes;
    const char *tag;
    ProfBytes(double b, const char *t) : bytes(b), tag(t) { profile_begin(); }
    ~ProfBytes() { profile_end_bytes(bytes, tag); }
};

// An optimizer launch, described so that a recorded one can be given other scalars (runtime.cu, fused.cu).
struct OptLaunch {
    static constexpr int MAX_ARGS = 16;
    int kind;                      // 0 Adam, 1 SGD
    float *w; const float *g; float *m, *v;
    long long n; bool vec; int grid;
    float scalars[9]; int n_scalars;
};
int graph_note_optimizer(const OptLaunch &launch);
void graph_note_launch(const void *func, dim3 grid, dim3 block, size_t smem);
// kernel, grid, block and argument pointers of the launch (the pointers point into `launch`)
void optimizer_node_params(const OptLaunch &launch, cudaKernelNodeParams &kp, void **args);

// runtime.cu: which of the counters kept at zero a launch that finishes in its last block may use (fused.cu); -1: none.
constexpr int FINISH_SLOTS = 256;
int finish_slot();

// Device float[2]: {dynamic factor of the fp16 gradient copies, its inverse}; both 1 until a loss head sets them (fused.cu).
float *grad_scale_words();

// batch.cu: hands the launches of an open seera_batch_begin to the device; the rest of that batch is launched one by one.  Called
// before whatever has to come behind them: a wait, a copy from or to host memory, an event, another recording.
int batch_flush();
void batch_trim();                          // gives back the executable graphs kept for further batches
// Lets a kernel be launched with up to `bytes` of dynamic shared memory.  The limit is the kernel's and not a launch's: it is only ever
// raised, since a launch that has been noted down comes after this call.
cudaError_t allow_smem(const void *kernel, size_t bytes);

// Pool-backed scratch for internal use (split-K partials, operand shadows).
void graph_note_collective();              // runtime.cu: the open capture records a collective
void graphs_with_collectives_release();     // runtime.cu: destroy the executable graphs that hold collectives (before the communicator goes)
void *scratch_alloc(size_t bytes);
void scratch_free(void *p);

}  // namespace seera
