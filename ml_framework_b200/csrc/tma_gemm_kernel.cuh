// TMA-fed tcgen05 GEMM kernel, tensor-map helpers and bf16 shadow conversion shared by the Dense and the
// convolution entry points.
#pragma once
#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "contraction_functors.cuh"
#include "tc_epilogue.cuh"
#include "tc_ptx.cuh"

namespace seera {


// ---- tensor maps -----------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || !p) {
            cudaGetLastError();
            return nullptr;
        }
        fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// bf16 row-major matrix [rows, cols] with pitch ld (elements, multiple of 8): 2-D map, inner dimension = cols.
// Box = box_inner x box_outer elements, 128-byte swizzle (64-byte for 32 elements), out-of-range elements read as zero.
inline int make_map_2d(CUtensorMap *m, const void *base, int rows, int cols, int ld, int box_inner, int box_outer) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return fail(SEERA_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, box_inner == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(SEERA_E_CUDA, "cuTensorMapEncodeTiled failed (%d) for %dx%d ld %d box %dx%d", (int)r, rows, cols, ld,
                                       box_inner, box_outer);
    return SEERA_OK;
}

// ---- fp32 -> bf16 shadows -----------------------------------------------------------------------------------
// NS = 1: hi = bf16(x).  NS = 2: plus lo = bf16(x - hi).  NS = 3: plus lo2 = bf16(x - hi - lo) (24 mantissa bits).
struct Shadow {
    __nv_bfloat16 *p[3] = {nullptr, nullptr, nullptr};      // 16-bit containers: bf16 or fp16 by `enc`
    int rows = 0, cols = 0, ld = 0;
    Enc enc{0, 1.f, nullptr};
};

}  // namespace seera
// ---- layers that hand their 16-bit operand copies from call to call --------------------------------------------------------
// Row-major copies of one [rows, cols] matrix (activations of a Dense layer, its weight matrix, a convolution's filters as
// [F][tap][channel]), kept by the caller between the forward and the backward call of a layer, or written by one layer's epilogue
// for the next layer's forward.
struct seera_rows {
    seera::Shadow s;
    int ns;
};
namespace seera {
// The copies if they serve a product of `ns` copies of a [rows, cols] matrix of this class in the present encoding, else null.
const Shadow *rows_usable(const seera_rows *h, int ns, int rows, int cols, int cls);

// Classes of tensor, for the scale of an fp16 encoding: activations are O(1) after He / Glorot initialisation, weights a
// few hundredths, gradients of a batch-mean loss 1e-6 .. 1e-2.  With the factors 2^4 / 2^8 / 2^12 the second copy of a
// value stays a normal fp16 number down to a magnitude of 2^-7 / 2^-11 / 2^-15 (below that its absolute error is
// 2^-29 / 2^-33 / 2^-37, far under the products' own rounding); values saturate at 4094 / 255.9 / 15.99 - data beyond
// that belongs in the bf16 modes 2 and 3, which keep fp32's exponent range.
enum { CLS_ACT = 0, CLS_WEIGHT = 1, CLS_GRAD = 2 };

template <int NS>
__global__ void __launch_bounds__(256) shadow_rows_kernel(const float *__restrict__ src, long long src_ld, int rows, int cols,
                                                          __nv_bfloat16 *__restrict__ d0, __nv_bfloat16 *__restrict__ d1,
                                                          __nv_bfloat16 *__restrict__ d2, int ld, Enc enc, FastDiv by_groups) {
    // one thread per 8 consecutive elements of a row; ld is a multiple of 8 so the 16-byte stores are aligned
    long long groups_per_row = ld >> 3, total = (long long)rows * groups_per_row;
    long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nthr = (long long)gridDim.x * blockDim.x;
    const bool small = total < (1ll << 31);       // then the row index is one multiply and a shift instead of a 64-bit division
    for (long long g = tid; g < total; g += nthr) {
        int r = small ? by_groups.div((int)g) : (int)(g / groups_per_row), c0 = (int)(g - (long long)r * groups_per_row) * 8;
        const float *s = src + (long long)r * src_ld + c0;
        float v[8];
        if (c0 + 8 <= cols && ((reinterpret_cast<uintptr_t>(s) & 15) == 0)) {
            float4 a = __ldg(reinterpret_cast<const float4 *>(s)), b = __ldg(reinterpret_cast<const float4 *>(s) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = (c0 + i < cols) ? __ldg(s + i) : 0.f;
        }
        long long o = (long long)r * ld + c0;
        store_split8<NS>(v, enc, d0 + o, d1 + o, d2 + o);
    }
}

// Precision modes 1 / 2 / 3: one, two, three bf16 copies (1, 3, 6 products).  Mode 4: two fp16 copies (3 products).
// Mode 5: one fp16 copy (1 product) - the first copy of a mode-4 set, so copies kept by a mode-4 forward serve a mode-5 backward.
inline int precision_copies() { int m = rt().precision; return m == 4 ? 2 : (m == 5 ? 1 : (m < 1 ? 1 : (m > 3 ? 3 : m))); }
inline Enc enc_for(int cls) {
    if (rt().precision != 4 && rt().precision != 5) return Enc{0, 1.f, nullptr};
    static const float scale[3] = {16.f, 256.f, 4096.f};
    return Enc{1, scale[cls], cls == CLS_GRAD ? grad_scale_words() : nullptr};
}
// Copies a weight-gradient product uses.  Its rounding stays in that one tensor (nothing downstream of dW in the backward
// pass reads it), so with the "wgrad_single" option the fp16 split mode forms dW from the first copy of each operand alone:
// one product instead of three, 2e-4 of rounding in dW.
inline int wgrad_copies(int ns) { return (rt().wgrad_single && rt().precision == 4) ? 1 : ns; }
// The inverse of an operand's dynamic factor, for the epilogue (null: none).
inline const float *enc_dinv(const Enc &a, const Enc &b) { return (a.dscale || b.dscale) ? grad_scale_words() + 1 : nullptr; }

inline int alloc_shadow(Shadow &s, int rows, int cols, int ns) {
    s.rows = rows; s.cols = cols; s.ld = (cols + 7) / 8 * 8;
    for (int i = 0; i < ns; i++) {
        s.p[i] = (__nv_bfloat16 *)scratch_alloc((size_t)rows * s.ld * 2);
        if (!s.p[i]) return SEERA_E_OOM;
    }
    return SEERA_OK;
}
inline void free_shadow(Shadow &s) {
    for (int i = 0; i < 3; i++) { if (s.p[i]) scratch_free(s.p[i]); s.p[i] = nullptr; }
}
// Row-major fp32 [rows, cols] -> bf16 shadows of the same layout (pitch rounded up to 8 elements).
inline int make_shadow(const float *src, int rows, int cols, int ns, Shadow &s, int cls) {
    if (int e = alloc_shadow(s, rows, cols, ns)) return e;
    s.enc = enc_for(cls);
    if (s.enc.dscale)          // an fp32 gradient tensor handed in from outside: its own largest entry sets the dynamic factor
        if (int e = seera_grad_scale_update(src, (long long)rows * cols)) return e;
    long long groups = (long long)rows * (s.ld / 8);
    int grid = stride_grid(groups);
    cudaStream_t st = rt().stream;
    ProfBytes pb(4.0 * rows * cols + 2.0 * ns * rows * s.ld, "shadow_rows");
    if (ns == 1) shadow_rows_kernel<1><<<grid, 256, 0, st>>>(src, cols, rows, cols, s.p[0], s.p[1], s.p[2], s.ld, s.enc, fast_div(s.ld / 8));
    else if (ns == 2) shadow_rows_kernel<2><<<grid, 256, 0, st>>>(src, cols, rows, cols, s.p[0], s.p[1], s.p[2], s.ld, s.enc, fast_div(s.ld / 8));
    else shadow_rows_kernel<3><<<grid, 256, 0, st>>>(src, cols, rows, cols, s.p[0], s.p[1], s.p[2], s.ld, s.enc, fast_div(s.ld / 8));
    count_launch();
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, "shadow_rows");
}

// ---- TMA + mbarrier PTX -------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst_smem, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
// im2col-mode load from an NHWC tensor: {c, w, h, n} is the channel offset and the position of the filter
// window's corner for the FIRST pixel of the column; {off_w, off_h} selects the filter tap.  The copy walks
// pixelsPerColumn window positions (w fastest, then h, then n) and fetches channelsPerPixel channels of each.
__device__ __forceinline__ void tma_load_im2col(uint32_t dst_smem, const CUtensorMap *map, int c, int w, int h, int n,
                                                int off_w, int off_h, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6], {%7, %8};"
                 ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(w), "r"(h), "r"(n), "r"(bar),
                   "h"((unsigned short)off_w), "h"((unsigned short)off_h) : "memory");
}

// ---- CTA pairs (tcgen05 cta_group::2): two CTAs of a cluster share one 256-row accumulator tile -------------------------
// Each CTA stages its own 128 rows of A and its own half of B's columns; the MMA, issued by the even CTA alone, reads the
// shared memory of both, and each CTA's TMEM receives its 128 rows of the result.  Per CTA and k-step that is
// (128 + N/2) operand rows loaded for 128 x N of output instead of (128 + N): the L2 -> shared-memory stream, which bounds
// the split-product kernels, shrinks by a quarter to a third.  No multicast load is involved: every CTA issues plain
// tensor copies into its own shared memory; only their completion is counted on the even CTA's barrier, and the
// tcgen05.commit that frees a stage or publishes an accumulator arrives on both CTAs' barriers.
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    __syncwarp();        // the single-thread roles left their warps diverged
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// shared::cluster address of the same variable in the CTA of rank `rank`
__device__ __forceinline__ uint32_t mapa_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void st_cluster_f4(uint32_t cluster_addr, float x, float y, float z, float w) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
// arrives on the barrier at this shared-memory offset in BOTH CTAs of the pair once the MMAs issued so far have finished
__device__ __forceinline__ void umma2_commit_both(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
// tensor copies of a CTA of a pair: into its own shared memory, completion counted on `bar`, a shared::cluster address
__device__ __forceinline__ void tma2_load_2d(uint32_t dst_smem, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma2_load_im2col(uint32_t dst_smem, const CUtensorMap *map, int c, int w, int h, int n,
                                                 int off_w, int off_h, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.im2col.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6], {%7, %8};"
                 ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(w), "r"(h), "r"(n), "r"(bar),
                   "h"((unsigned short)off_w), "h"((unsigned short)off_h) : "memory");
}

// MN-major operand tile: 64 contiguous row-index elements (128 bytes) per k line, 8 k lines per 1024-byte
// atom; atoms of the next 64 row indices start box_bytes later.
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t addr, uint32_t box_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((box_bytes >> 4) & 0x3FFF) << 16;   // leading byte offset: next 64 elements along M/N
    d |= (uint64_t)(1024 >> 4) << 32;                   // stride byte offset: next 8 k lines
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// 32 contiguous row-index elements (64 bytes, 64-byte swizzle) per k line: atoms of 512 bytes, the next 32 row indices box_bytes later.
__device__ __forceinline__ uint64_t umma_desc_sw64_mn(uint32_t addr, uint32_t box_bytes) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)((box_bytes >> 4) & 0x3FFF) << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
           (uint64_t)4 << 61;
}

// How the producer forms the A tile of a stage:
//   TMA_A_ROWS    2-D map of a row-major matrix [M, K], read along its rows (K-major)
//   TMA_A_COLS    2-D map of a row-major matrix [K, M], read along its columns (MN-major, two 64-wide boxes)
//   TMA_A_IM2COL  im2col map of an NHWC tensor; M = output pixels, K = (tap, channel): one tap x 64 channels
//                 per stage (K-major).  B is then [N, (tap, channel)] read along its rows.
//   TMA_A_TAPS    im2col map of an NHWC tensor; M = (tap, channel), K = output pixels: 64 pixels per stage,
//                 two boxes of 64 channels (MN-major).  B is then [pixels, N] read along its columns.
// Tensors of up to 32 channels take boxes of 32 (`narrow`) in the two im2col modes, half of a box of 64 being padding:
//   IM2COL        two taps a stage, each 128 rows of 64 bytes with the 64-byte swizzle; B likewise, two boxes of 32 (or the 32 filters of
//                 each tap below one another, read along its columns).  An odd last tap stands beside zeros from beyond the channels.
//   TAPS          M = (tap, 32 channels), four boxes a tile
enum { TMA_A_ROWS = 0, TMA_A_COLS = 1, TMA_A_IM2COL = 2, TMA_A_TAPS = 3 };

// A launch of several output phases of a strided data gradient (functors with kPhases = 4): the same tiles for each phase, each with its own
// maps, taps and window corner.
constexpr int TMA_PHASES = 4;
template <class CS, class = void> struct phases_of { static constexpr int value = 1; };
template <class CS> struct phases_of<CS, std::void_t<decltype(CS::kPhases)>> { static constexpr int value = CS::kPhases; };
// Functors of the convolutions, whose products may take narrow boxes.
template <class CS, class = void> struct narrow_of { static constexpr bool value = false; };
template <class CS> struct narrow_of<CS, std::void_t<decltype(CS::kNarrow)>> { static constexpr bool value = true; };
struct TmaMaps { CUtensorMap a[3], b[3]; };
template <int N> struct TmaMapSet { TmaMaps of[N]; };
struct TmaPhase { int K, taps, S, pw, ph, a, b; FastDiv by_S; };      // contraction, its taps and their columns, lower padding; the phase (a, b)

struct TmaGemmParams {
    int M, N, K, kchunk, splits, bn, stages;
    int first;               // tiles before this launch's (a product's last tiles, too few for a round, go to clusters)
    int tiles;               // end of this launch's tiles
    int a_mode, b_mn;        // b_mn = 1: B read along its contiguous row index (MN-major)
    int pair;                // 1: launched as clusters of two CTAs sharing 256-row tiles (tcgen05 cta_group::2)
    int issuers;             // 1 or 2 threads issue the MMAs of a k-step (the K = 16 slices dealt round robin), each into its own
                             // accumulator; the epilogue adds the accumulators up
    int shared;              // CTAs of a cluster that share one tile, each with its part of the contraction (1: none)
    int forward;             // a layer's output: ReLU and pools decide on these sums (tma_plan)
    int joined;              // split products with B's first two copies side by side as one operand of 2 x bn columns (below)
    // convolution geometry for the im2col modes
    int OW, OHW;             // output width and pixels per image of the traversal
    int sw, sh, pw, ph;      // window stride and lower padding
    int S, taps;             // filter width and R*S
    int cpad, cchunks;       // channel pitch of the weight rows / channels rounded up to 64, in chunks of 64
    int narrow;              // boxes of 32 channels (above)
    int wflip;               // TMA_A_IM2COL with b_mn: B is [channel of A][tap][wflip columns], its taps in reverse order (a data
                             // gradient that reads the forward's filter copies as they are)
    int phases;              // of a launch with several (0: none); the tiles of phase z follow those of phase z - 1
    TmaPhase phase[TMA_PHASES];
    float *partial;
    int *status;
    unsigned long long wait_clocks;   // budget of every bounded wait in the kernel
    int skip_load;           // test hook: the producer of CTA 0 leaves out the loads of this k-step (-1: none), so that the
                             // waits downstream of it run out and the kernel has to report and unwind
    const float *dinv;       // device word holding the inverse of the gradient operand's dynamic factor (null: none)
    float out_scale;         // the accumulator is multiplied by this before bias / activation / store: 1 / (scale_a * scale_b)
    int a_fp16, b_fp16;      // operand formats: 0 bf16, 1 fp16
    const float *bias;       // per-column bias added before the store, or null
    int act;                 // activation applied before the store (0 = none)
    int pool_on;             // 1: rows are pixels of a layer output that is only consumed through a 2x2 max-pool: store that instead
    PoolOut pool;
    FastDiv by_mtiles, by_ntiles, by_OHW, by_OW, by_S, by_cchunks;      // filled by launch_tma_gemm
};

// warps 0 and 3: TMA producers of A and B; warps 1-2: MMA issuers (the first p.issuers of them); warp 3 allocates TMEM; warps 4-11:
// epilogue, two warps per TMEM lane quarter, which take its 32-column chunks alternately.  One warp per quarter drained a 128 x 128 tile in about the
// time of twice its main loop (VGG, 128 filters at 16 x 16: launch 80 us, main loop alone 37 us).
constexpr int TG_THREADS = 384, TG_EPI_WARP0 = 4, TG_EPI_WARPS = 8;

// Persistent kernel: each CTA walks tiles  id = blockIdx.x, blockIdx.x + gridDim.x, ...  (m-tile fastest, then n-tile,
// then K split).  The operand ring keeps streaming across tile boundaries and the accumulator is double-buffered in
// TMEM, so the epilogue of tile i overlaps the main loop of tile i+1.
//
// What an MMA costs (a loop of MMAs alone, clocks per K = 16 slice of 128 rows): the larger of N / 2 on the tensor pipe and
// 32 + N / 4 for its operands, which come from shared memory at 128 bytes a clock (4 KB of A, 32 N bytes of B): 40 / 48 / 64 / 128 at
// N = 32 / 64 / 128 / 256.  One thread keeps up with that; commits cost nothing measurable.
//
// Split products (NS = 2: A0 B0 + A0 B1 + A1 B0; NS = 3: the six products down to 2^-16 of the first) therefore take B0 and B1, which
// lie one after the other in a stage, as ONE operand of 2 x bn columns wherever that is at most 256 wide: A0 is read once for two
// products, whose sums go to two accumulators side by side.  A slice of NS = 2 takes 64 + 48 clocks instead of 3 x 48 at
// bn = 64 (88 for 120 at 32), one of NS = 3 2 x 64 + 2 x 48 instead of 288; at bn = 128 the tensor pipe bounds both forms, but the joined one
// leaves a fifth of the reads of shared memory to the epilogue (131072 x 128 x 576 with the pool: 48.3 -> 47.5 us; NS = 3 at
// bn = 64, 25600 x 64 x 1152: 34.3 -> 31.8).  Sums in two accumulators are also shorter chains: 1.92e-6 -> 1.02e-6 of error at NS = 3
// against float64, 1.08e-6 -> 7.1e-7 at NS = 2 on fp16 (512 x 64 x 576).  The epilogue adds the two accumulators; TMEM holds 2 buffers x 2 x bn columns (at most 512).
//
// Products of one copy with N <= 128, and the forward ones in six products that tma_plan names, are issued by two threads (lane 0 of
// warps 1 and 2), which take the K = 16 slices of a k-step alternately, each into an accumulator of its own (MMAs of different threads are
// not ordered among themselves), and commit to the stage's "empty" and the tile's "accumulator full" barriers, which count `issuers` arrivals.
// (NARROW apart from the rest: its branches in the producer and the issuer cost the others 5 % of a launch.)
template <int NS, class CS, bool PAIR, bool NARROW>
__global__ void __launch_bounds__(TG_THREADS, 1)
tma_gemm_kernel(const __grid_constant__ TmaMapSet<phases_of<CS>::value> maps, CS cs, TmaGemmParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[2 * 8 + 4];      // full[8], empty[8], tfull[2], tempty[2]
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag;

    const int t = threadIdx.x, lane = t & 31;
    const int warp = __shfl_sync(0xffffffffu, t >> 5, 0);       // the same in all lanes, and known to be
    const int bn = p.bn, stages = p.stages;
    // PAIR: the two CTAs of a cluster work on one tile of 256 rows; `rank` 0 (the even CTA) issues its MMAs
    constexpr int TM = PAIR ? 2 * TC_BM : TC_BM;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    // a tile shared by the CTAs of a cluster: `part` is this CTA's share of its contraction (one tile per cluster)
    const int shared = PAIR ? 1 : p.shared, part = shared > 1 ? (int)cluster_ctarank() : 0;
    const int worker = p.first + (PAIR ? (int)(blockIdx.x >> 1) : (shared > 1 ? (int)blockIdx.x / shared : (int)blockIdx.x));
    const int nworkers = PAIR ? (int)(gridDim.x >> 1) : (shared > 1 ? (int)gridDim.x / shared : (int)gridDim.x);
    const int bh = PAIR ? bn >> 1 : bn;                       // columns of B this CTA stages
    const int mtiles = (p.M + TM - 1) / TM, ntiles = (p.N + bn - 1) / bn;
    const int total_tiles = p.tiles;
    const bool a_mn = p.a_mode == TMA_A_COLS || p.a_mode == TMA_A_TAPS;

    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t a_bytes = TC_BM * 128, b_bytes = (uint32_t)bh * 128;
    const uint32_t stage_bytes = (uint32_t)NS * (a_bytes + b_bytes);
    const uint32_t smem0 = smem_u32(smem);
    auto a_tile = [&](int s, int i) { return smem0 + (uint32_t)s * stage_bytes + (uint32_t)i * a_bytes; };
    auto b_tile = [&](int s, int i) { return smem0 + (uint32_t)s * stage_bytes + (uint32_t)NS * a_bytes + (uint32_t)i * b_bytes; };
    unsigned char *epi_smem = smem + (size_t)stages * stage_bytes;   // one EPI_WARP_SMEM per epilogue warp after the ring
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[8]), tfull0 = smem_u32(&bars[16]), tempty0 = smem_u32(&bars[18]);
    const int issuers = PAIR ? 1 : p.issuers;
    const bool joined = !PAIR && NS >= 2 && p.joined;
    const int nacc = joined ? 2 : issuers;                    // accumulators of a buffer, bn columns apart
    const uint32_t tmem_cols = (uint32_t)(2 * nacc * bn < 32 ? 32 : 2 * nacc * bn);

    if (t == 0) {
        abort_flag = 0;
        for (int s = 0; s < stages; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, issuers); }
        for (int b = 0; b < 2; b++) { mbar_init(tfull0 + 8 * b, issuers); mbar_init(tempty0 + 8 * b, PAIR ? 2 * TG_EPI_WARPS : TG_EPI_WARPS); }
        fence_mbar_init();
        fence_async_smem();
    }
    if (warp == 3) { if (PAIR) tmem_alloc2(smem_u32(&tmem_base_slot), tmem_cols); else tmem_alloc(smem_u32(&tmem_base_slot), tmem_cols); }
    tc_fence_before();
    if (PAIR) cluster_sync_all(); else __syncthreads();        // the peer's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int *abortp = &abort_flag;

    // tile id -> origin and K range
    auto tile_origin = [&](int id, int &m0, int &n0, int &kbeg, int &ktiles, int &z) {
        int rest = p.by_mtiles.div(id), mt = id - rest * mtiles;
        z = p.by_ntiles.div(rest);
        int nt = rest - z * ntiles;
        m0 = mt * TM + (int)rank * TC_BM; n0 = nt * bn;         // this CTA's own 128 rows
        kbeg = (z + part) * p.kchunk;                           // (z is 0 where a cluster shares a tile)
        int kend = min(p.K, kbeg + p.kchunk);
        if (phases_of<CS>::value > 1) { kbeg = 0; kend = p.phase[z].K; }
        ktiles = (kend - kbeg + TC_BK - 1) / TC_BK;
    };

    if (warp == 0 || warp == 3) {
        // ---------------- TMA producers: warp 0 loads A, warp 3 (once it has allocated TMEM) B ----------------
        // What a producer issues per k-step bounds the launches of one copy per operand, and those whose columns are few: one warp for both
        // operands that found its coordinates by division took 75 ns more a k-step for a dozen instructions
        // (weight gradient 576 x 128 x 131072 31.5 -> 27.9 us, 2304 x 256 x 50176 48.5 -> 44.2, data gradient 131072 x 64 x 1152 56 -> 52.9).
        const bool leader = elect_one();
        auto ld2d = [&](uint32_t dst, const CUtensorMap *m, int x, int y, uint32_t bar) {
            if (PAIR) tma2_load_2d(dst, m, x, y, bar); else tma_load_2d(dst, m, x, y, bar);
        };
        auto ldim = [&](uint32_t dst, const CUtensorMap *m, int c, int w, int h, int n, int ow, int oh, uint32_t bar) {
            if (PAIR) tma2_load_im2col(dst, m, c, w, h, n, ow, oh, bar); else tma_load_im2col(dst, m, c, w, h, n, ow, oh, bar);
        };
        int it = 0;
        int s = 0;                                            // ring slot and its phase, carried across tiles
        uint32_t ph = 0;
        bool alive = true;
        const int c64 = p.cchunks * 64;
        for (int id = worker; id < total_tiles && alive; id += nworkers) {
            int m0, n0, kbeg, ktiles, z;
            tile_origin(id, m0, n0, kbeg, ktiles, z);
            const TmaMaps &own = maps.of[phases_of<CS>::value > 1 ? z : 0];
            int S = p.S, taps = p.taps, pw = p.pw, phh = p.ph;
            FastDiv by_S = p.by_S;
            if (phases_of<CS>::value > 1) { S = p.phase[z].S; taps = p.phase[z].taps; pw = p.phase[z].pw; phh = p.phase[z].ph; by_S = p.phase[z].by_S; }
            // im2col, M = pixels: the tap and channel of the next k-step, counted on from the first one's
            int tap = 0, c0 = 0, r = 0, sx = 0;
            if (p.a_mode == TMA_A_IM2COL) {
                const int ktile = kbeg >> 6;
                tap = NARROW ? 2 * ktile : p.by_cchunks.div(ktile);
                c0 = NARROW ? 0 : (ktile - tap * p.cchunks) * 64;
                r = by_S.div(tap); sx = tap - r * S;
            }
            auto next_tap = [&]() { tap++; if (++sx == S) { sx = 0; r++; } };
            if (warp == 0) {
                const CUtensorMap *mA = own.a;
                // window corner of this tile's first output pixel
                int pix_img = 0, pix_w = 0, pix_h = 0;
                if (p.a_mode == TMA_A_IM2COL) {
                    pix_img = p.by_OHW.div(m0);
                    const int rem = m0 - pix_img * p.OHW, oh = p.by_OW.div(rem), ow = rem - oh * p.OW;
                    pix_w = ow * p.sw - pw; pix_h = oh * p.sh - phh;
                }
                // im2col, M = (tap, channel): the boxes of this tile, and the first pixel of the next k-step
                constexpr int BOXES = NARROW ? 4 : 2, BOX = TC_BM / BOXES;             // rows of a box: channels of one tap
                int box_c[BOXES] = {}, box_s[BOXES] = {}, box_r[BOXES] = {}, img = 0, rem = 0;
                bool box_ok[BOXES] = {};
                uint32_t tx_bytes = PAIR ? 2u * stage_bytes : stage_bytes;     // a pair counts both CTAs' bytes on the even CTA's barrier
                if (p.a_mode == TMA_A_TAPS) {
#pragma unroll
                    for (int b = 0; b < BOXES; b++) {
                        const int mb = m0 + BOX * b, at = NARROW ? mb >> 5 : p.by_cchunks.div(mb >> 6);
                        box_ok[b] = at < p.taps;
                        box_c[b] = NARROW ? 0 : mb - at * c64; box_r[b] = p.by_S.div(at); box_s[b] = at - box_r[b] * p.S;
                        if (!box_ok[b]) tx_bytes -= (uint32_t)NS * (uint32_t)(BOX * 128);
                    }
                    if (PAIR && rank == 0) {                       // the peer's boxes beyond the last tap are not loaded either
                        for (int b = 0; b < 2; b++) {
                            const int mb = m0 + TC_BM + 64 * b, at = p.by_cchunks.div(mb >> 6);
                            if (at >= p.taps) tx_bytes -= (uint32_t)NS * 8192u;
                        }
                    }
                    img = p.by_OHW.div(kbeg); rem = kbeg - img * p.OHW;
                }
                for (int kt = 0; kt < ktiles; kt++, it++) {
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1u, abortp, p.status, 1, p.wait_clocks)) { alive = false; break; }
                    const int k0 = kbeg + kt * TC_BK;
                    const uint32_t bar = PAIR ? mapa_rank(full0 + 8 * s, 0) : full0 + 8 * s;
                    const bool skip = p.skip_load >= 0 && blockIdx.x == 0 && it == p.skip_load;      // test hook: this stage never fills
                    if (leader && !skip) {
                        if (rank == 0) mbar_expect_tx(full0 + 8 * s, tx_bytes);
                        if (p.a_mode == TMA_A_ROWS) {
#pragma unroll
                            for (int i = 0; i < NS; i++) ld2d(a_tile(s, i), &mA[i], k0, m0, bar);
                        } else if (p.a_mode == TMA_A_COLS) {
#pragma unroll
                            for (int i = 0; i < NS; i++)
                                for (int b = 0; b < 2; b++) ld2d(a_tile(s, i) + b * 8192, &mA[i], m0 + 64 * b, k0, bar);
                        } else if (p.a_mode == TMA_A_IM2COL) {
#pragma unroll
                            for (int h = 0; h < (NARROW ? 2 : 1); h++) {
                                const bool in = !NARROW || tap < taps;             // else: zeros, from beyond the channels
#pragma unroll
                                for (int i = 0; i < NS; i++)
                                    ldim(a_tile(s, i) + h * 8192, &mA[i], in ? c0 : 32, pix_w, pix_h, pix_img, in ? sx : 0, in ? r : 0, bar);
                                if (NARROW) next_tap();
                            }
                        } else {
                            const int oh = p.by_OW.div(rem), ow = rem - oh * p.OW, w = ow * p.sw - p.pw, h = oh * p.sh - p.ph;
#pragma unroll
                            for (int i = 0; i < NS; i++)
#pragma unroll
                                for (int b = 0; b < BOXES; b++)
                                    if (box_ok[b]) ldim(a_tile(s, i) + b * (BOX * 128), &mA[i], box_c[b], w, h, img, box_s[b], box_r[b], bar);
                        }
                    }
                    if (p.a_mode == TMA_A_IM2COL) {
                        if (NARROW) { if (!leader || skip) { next_tap(); next_tap(); } }
                        else if ((c0 += 64) == c64) { c0 = 0; next_tap(); }
                    } else if (p.a_mode == TMA_A_TAPS) {
                        if (p.OHW >= TC_BK) { if ((rem += TC_BK) >= p.OHW) { rem -= p.OHW; img++; } }
                        else { img = p.by_OHW.div(k0 + TC_BK); rem = k0 + TC_BK - img * p.OHW; }
                    }
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            } else {
                const CUtensorMap *mB = own.b;
                const int nb0 = n0 + (int)rank * bh;               // this CTA's own columns of B
                for (int kt = 0; kt < ktiles; kt++, it++) {
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1u, abortp, p.status, 1, p.wait_clocks)) { alive = false; break; }
                    const uint32_t bar = PAIR ? mapa_rank(full0 + 8 * s, 0) : full0 + 8 * s;
                    const bool skip = p.skip_load >= 0 && blockIdx.x == 0 && it == p.skip_load;
                    if (leader && !skip) {
                        if (NARROW && p.a_mode == TMA_A_IM2COL) {
#pragma unroll
                            for (int h = 0; h < 2; h++) {
                                const int at = tap + h;
                                const bool in = at < taps;
#pragma unroll
                                for (int i = 0; i < NS; i++) {
                                    if (p.b_mn) {
                                        for (int b = 0; b < bh / 64; b++)
                                            ld2d(b_tile(s, i) + b * 8192 + h * 4096, &mB[i], (in ? (taps - 1 - at) * p.wflip : 0) + nb0 + 64 * b, in ? 0 : 32, bar);
                                    } else {
                                        ld2d(b_tile(s, 0) + (uint32_t)(h * NS + i) * (b_bytes >> 1), &mB[i], at * p.cpad, nb0, bar);
                                    }
                                }
                            }
                        } else {
                            // B's coordinate along the contraction, and where its columns begin
                            int bk = kbeg + kt * TC_BK, bx = 0;
                            if (p.a_mode == TMA_A_IM2COL) {
                                if (p.b_mn) { bk = c0; bx = (taps - 1 - tap) * p.wflip; }
                                else bk = tap * p.cpad + c0;
                            }
                            if (p.b_mn) {
#pragma unroll
                                for (int i = 0; i < NS; i++)
                                    for (int b = 0; b < bh / 64; b++) ld2d(b_tile(s, i) + b * 8192, &mB[i], bx + nb0 + 64 * b, bk, bar);
                            } else {
#pragma unroll
                                for (int i = 0; i < NS; i++) ld2d(b_tile(s, i), &mB[i], bk, nb0, bar);
                            }
                        }
                    }
                    if (p.a_mode == TMA_A_IM2COL) {
                        if (NARROW) tap += 2;
                        else if ((c0 += 64) == c64) { c0 = 0; tap++; }
                    }
                    if (++s == stages) { s = 0; ph ^= 1u; }
                }
            }
        }
        if (*abortp && rank == 0) {
            // give copies already in flight a bounded chance to land before the CTA's shared memory goes away
            for (int k = it - stages < 0 ? 0 : it - stages; k < it; k++) {
                unsigned long long t0 = clock64();
                if (p.skip_load >= 0 && blockIdx.x == 0 && k == p.skip_load) continue;      // nothing was issued for it
                while (!mbar_try_wait(full0 + 8 * (k % stages), (uint32_t)(k / stages) & 1u) && clock64() - t0 < p.wait_clocks) {}
            }
        }
        __syncwarp();
    } else if (warp >= 1 && warp <= issuers && rank == 0) {
        // ---------------- MMA issuers (in the even CTA of a pair) ----------------
        const bool leader = elect_one();
        const int me = warp - 1;
        uint32_t idesc = umma_idesc_16bit(bn, p.a_fp16, p.b_fp16) | ((uint32_t)(a_mn ? 1 : 0) << 15) | ((uint32_t)p.b_mn << 16);
        if (PAIR) idesc = (idesc & ~(31u << 24)) | ((uint32_t)(TM >> 4) << 24);          // M = 256 over the two CTAs
        const uint32_t idesc2 = umma_idesc_16bit(2 * bn, p.a_fp16, p.b_fp16) | ((uint32_t)(a_mn ? 1 : 0) << 15) | ((uint32_t)p.b_mn << 16);
        // bytes from slice 0 to the next K = 16 slice and to the third
        const bool a64 = NARROW, b64 = NARROW && !p.b_mn;
        const uint32_t a_step = a_mn ? (a64 ? 1024u : 2048u) : 32u, b_step = p.b_mn ? 2048u : 32u;
        const uint32_t a_far = a64 && !a_mn ? 8192u : 2 * a_step, b_far = b64 ? (uint32_t)NS * (b_bytes >> 1) : 2 * b_step;
        // split products kept: hi*hi | + hi*lo, lo*hi | + hi*lo2, lo2*hi, lo*lo
        constexpr int NPROD = NS == 1 ? 1 : (NS == 2 ? 3 : 6);
        const int pa[6] = {0, 0, 1, 0, 2, 1}, pb[6] = {0, 1, 0, 2, 0, 1};
        bool alive = true;
        int local = 0;
        int s = 0;                                            // ring slot and its phase, carried across tiles
        uint32_t ph = 0;
        // descriptors of copy 0 / slice 0 in slot 0; the others differ only in the start-address field (16-byte units),
        // which never carries out of its 14 bits for addresses inside the CTA's shared memory
        const uint32_t a_step16 = a_step >> 4, b_step16 = b_step >> 4, a_copy16 = a_bytes >> 4, b_copy16 = b64 ? b_bytes >> 5 : b_bytes >> 4;
        const uint32_t a_far16 = a_far >> 4, b_far16 = b_far >> 4;
        auto at = [](int jj, uint32_t step, uint32_t far) { return NARROW ? (uint32_t)(jj & 1) * step + (uint32_t)(jj >> 1) * far : (uint32_t)jj * step; };
        const uint64_t da0 = (a64 ? (a_mn ? umma_desc_sw64_mn(a_tile(0, 0), 4096) : umma_desc_sw64(a_tile(0, 0)))
                                  : (a_mn ? umma_desc_sw128_mn(a_tile(0, 0), 8192) : umma_desc_sw128(a_tile(0, 0)))) + (uint32_t)me * a_step16;
        const uint64_t db0 = (p.b_mn ? umma_desc_sw128_mn(b_tile(0, 0), 8192) : (b64 ? umma_desc_sw64(b_tile(0, 0)) : umma_desc_sw128(b_tile(0, 0)))) +
                             (uint32_t)me * b_step16;
        const uint32_t stage16 = stage_bytes >> 4;
        for (int id = worker; id < total_tiles && alive; id += nworkers, local++) {
            int m0, n0, kbeg, ktiles, z;
            tile_origin(id, m0, n0, kbeg, ktiles, z);
            const int buf = local & 1;
            // the epilogue must have drained this accumulator buffer (two tiles ago)
            alive = mbar_wait(tempty0 + 8 * buf, (((uint32_t)local >> 1) & 1u) ^ 1u, abortp, p.status, 4, p.wait_clocks);
            if (!alive) break;
            tc_fence_after();
            const uint32_t d_tmem = tmem_base + (uint32_t)((buf * nacc + me) * bn);
            uint32_t acc = 0;
            for (int kt = 0; kt < ktiles && alive; kt++) {
                alive = mbar_wait(full0 + 8 * s, ph, abortp, p.status, 2, p.wait_clocks);
                if (!alive) break;
                tc_fence_after();
                const uint64_t das = da0 + (uint32_t)s * stage16, dbs = db0 + (uint32_t)s * stage16;
                // the K = 16 slices of this thread (da0 / db0 already point at its first one), fully unrolled either way: one thread
                // keeps up with the pipe only while an MMA costs it a few instructions
                auto slice = [&](uint64_t dsa, uint64_t dsb, bool first) {
                    uint64_t da[NS], db[NS];
#pragma unroll
                    for (int i = 0; i < NS; i++) { da[i] = dsa + (uint32_t)i * a_copy16; db[i] = dsb + (uint32_t)i * b_copy16; }
#pragma unroll
                    for (int q = 0; q < NPROD; q++) {
                        const bool open = first && q == 0;        // only the k-step's first product can start the accumulator
                        if (PAIR) umma2_bf16(d_tmem, da[pa[q]], db[pb[q]], idesc, open ? acc : 1u);
                        else if (open) umma_bf16(d_tmem, da[pa[q]], db[pb[q]], idesc, acc);
                        else umma_bf16_add(d_tmem, da[pa[q]], db[pb[q]], idesc);
                    }
                };
                // the same with B0 and B1 as one operand: hi*(hi, lo) | lo*(hi, lo) and the two with a third copy, or lo*hi
                auto slice_joined = [&](uint64_t dsa, uint64_t dsb, bool first) {
                    umma_bf16(d_tmem, dsa, dsb, idesc2, first ? acc : 1u);
                    if (NS == 2) {
                        umma_bf16_add(d_tmem + (uint32_t)bn, dsa + a_copy16, dsb, idesc);
                    } else {
                        umma_bf16_add(d_tmem, dsa + a_copy16, dsb, idesc2);
                        umma_bf16_add(d_tmem + (uint32_t)bn, dsa, dsb + 2u * b_copy16, idesc);
                        umma_bf16_add(d_tmem + (uint32_t)bn, dsa + 2u * a_copy16, dsb, idesc);
                    }
                };
                if (leader) {
                if (NS >= 2 && joined) {
#pragma unroll
                    for (int jj = 0; jj < TC_BK / 16; jj++)
                        slice_joined(das + at(jj, a_step16, a_far16), dbs + at(jj, b_step16, b_far16), jj == 0);
                } else if (issuers == 2) {
#pragma unroll
                    for (int jj = 0; jj < TC_BK / 32; jj++) slice(das + at(2 * jj, a_step16, a_far16), dbs + at(2 * jj, b_step16, b_far16), jj == 0);
                } else {
#pragma unroll
                    for (int jj = 0; jj < TC_BK / 16; jj++)
                        slice(das + at(jj, a_step16, a_far16), dbs + at(jj, b_step16, b_far16), jj == 0);
                }
                if (PAIR) umma2_commit_both(empty0 + 8 * s); else umma_commit(empty0 + 8 * s);
                }
                acc = 1;
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
            if (alive && leader) { if (PAIR) umma2_commit_both(tfull0 + 8 * buf); else umma_commit(tfull0 + 8 * buf); }   // accumulator complete
        }
    } else if (warp >= TG_EPI_WARP0 && shared == 1) {
        // ---------------- epilogue: warp w drains TMEM lane quarter w % 4, every second 32-column chunk ----------------
        const int q = warp & 3, half = (warp - TG_EPI_WARP0) >> 2;
        float *stage = reinterpret_cast<float *>(epi_smem + (size_t)(warp - TG_EPI_WARP0) * EPI_WARP_SMEM);
        const float out_scale = p.dinv ? p.out_scale * __ldg(p.dinv) : p.out_scale;
        int local = 0;
        const uint32_t tempty_at = PAIR ? mapa_rank(tempty0, 0) : tempty0;      // the even CTA's barrier counts both epilogues
        for (int id = worker; id < total_tiles; id += nworkers, local++) {
            int m0, n0, kbeg, ktiles, z;
            tile_origin(id, m0, n0, kbeg, ktiles, z);
            const int buf = local & 1, c_first = bn == 32 ? (half ^ buf) * 32 : half * 32;     // one chunk a tile: the halves take tiles in turn
            // (a longer budget than the issuers', so that a stage that never fills is reported by the role that waits for it)
            if (!mbar_wait(tfull0 + 8 * buf, ((uint32_t)local >> 1) & 1u, abortp, p.status, 3, p.wait_clocks + (p.wait_clocks >> 2))) break;
            tc_fence_after();
            // the accumulator goes back to the issuers as soon as its last chunk is in registers
            auto release = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) { if (PAIR) mbar_arrive_cluster(tempty_at + 8 * buf); else mbar_arrive(tempty0 + 8 * buf); }
            };
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * nacc * bn + c_first);
            if constexpr (phases_of<CS>::value > 1) { cs.a = p.phase[z].a; cs.b = p.phase[z].b; }
            if (c_first >= bn)
                release();
            else if (p.pool_on)
                drain_accumulator_pooled(taddr, m0 + q * 32, n0, c_first, bn, 64, p.M, p.N, p.bias, p.act, p.pool, stage, out_scale, nacc,
                                         (uint32_t)bn, release);
            else
                drain_accumulator(taddr, m0 + q * 32, n0, c_first, bn, 64, p.M, p.N, cs, p.partial, (long long)z * p.M * p.N, stage, p.bias,
                                  p.act, out_scale, nacc, (uint32_t)bn, release);
        }
    }
    if (!PAIR && shared > 1) {
        // ---------------- a tile of a cluster: chunk ci (32 x 32) is added up and finished by CTA ci % shared ----------------
        // Each CTA writes its sums of a chunk into the shared memory of that CTA, where the ring is done with.  What the tile's 64 KB
        // cost between SMs is 2 us either way; reading the others' shares instead measured 0.3 to 1.5 us slower (and keeps every CTA
        // until it has been read), bulk copies the same.
        const bool epi = warp >= TG_EPI_WARP0;
        const int ew = warp - TG_EPI_WARP0, cols = bn >> 5;
        const bool done = epi && mbar_wait(tfull0, 0, abortp, p.status, 3, p.wait_clocks + (p.wait_clocks >> 2));
        tc_fence_after();
        cluster_sync_all();                                    // every CTA's ring is free
        if (done) {
            const int q = warp & 3;
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c = (ew >> 2) * 32; c < bn; c += 64) {
                float v[32];
                tmem_ld32_sum(taddr + (uint32_t)c, v, nacc, (uint32_t)bn);
                const int ci = q * cols + (c >> 5), slot = ci / shared, owner = ci - slot * shared;
                const uint32_t dst = mapa_rank(smem0 + (uint32_t)(((slot * shared + part) * 256 + lane) * 16), (uint32_t)owner);
#pragma unroll
                for (int k = 0; k < 8; k++) st_cluster_f4(dst + 512u * k, v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            }
        }
        cluster_sync_all();                                    // every share is where it is added up, in the order of the shares
        if (epi) {
            float *stage = reinterpret_cast<float *>(epi_smem + (size_t)ew * EPI_WARP_SMEM);
            const float out_scale = p.dinv ? p.out_scale * __ldg(p.dinv) : p.out_scale;
            int m0, n0, kbeg, ktiles, z;
            tile_origin(worker, m0, n0, kbeg, ktiles, z);
#pragma unroll 1
            for (int slot = ew, ci = slot * shared + part; ci < 4 * cols; slot += TG_EPI_WARPS, ci += TG_EPI_WARPS * shared) {
                const float4 *src = reinterpret_cast<const float4 *>(smem) + slot * shared * 256 + lane;
                float v[32];
#pragma unroll
                for (int k = 0; k < 32; k++) v[k] = 0.f;
#pragma unroll 1
                for (int r = 0; r < shared; r++, src += 256) {
#pragma unroll
                    for (int k = 0; k < 8; k++) { const float4 x = src[32 * k]; v[4 * k] += x.x; v[4 * k + 1] += x.y; v[4 * k + 2] += x.z; v[4 * k + 3] += x.w; }
                }
                const int q = ci / cols, row = m0 + q * 32, n = n0 + (ci - q * cols) * 32;
                if (row >= p.M || n >= p.N) continue;
                if (p.pool_on) put_chunk_pooled(v, row, n, p.M, p.N, p.bias, p.act, p.pool, stage, out_scale);
                else put_chunk(v, row, n, p.M, p.N, cs, stage, p.bias, p.act, out_scale);
            }
        }
    }
    tc_fence_before();
    if (PAIR) cluster_sync_all(); else __syncthreads();        // neither CTA's shared memory or TMEM goes away while the other still uses it
    if (warp == 3) { if (PAIR) tmem_dealloc2(tmem_base, tmem_cols); else tmem_dealloc(tmem_base, tmem_cols); }
}

// Sum of the split partials in split order (in `zg` interleaved chains that are added in chain order), then the epilogue's transform.
// A block's eight warps are zg chains x 8 / zg groups of 128 consecutive outputs, four per lane where the row length allows: with one
// output per thread and one chain the launch took the time of `splits` dependent reads (5 to 8 us for 20 to 37 splits).
template <class CS, bool VEC>
__global__ void __launch_bounds__(256) tma_splitk_reduce_kernel(const float *__restrict__ partial, CS cs, int M, int N, int splits,
                                                                const float *__restrict__ bias, int act, float scale,
                                                                const float *__restrict__ dinv, int zg, FastDiv by_N) {
    constexpr int V = VEC ? 4 : 1;
    __shared__ float sm[8][32 * V];
    if (dinv) scale *= __ldg(dinv);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, groups = 8 / zg, chain = warp / groups, grp = warp - chain * groups;
    const long long total = (long long)M * N, stride = (long long)gridDim.x * groups * 32 * V;
    const bool small = total < (1ll << 31);       // 32-bit index arithmetic then: the 64-bit division costs more than the loads
    for (long long base = (long long)blockIdx.x * groups * 32 * V; base < total; base += stride) {
        const long long i = base + (grp * 32 + lane) * V;
        float s[V];
#pragma unroll
        for (int k = 0; k < V; k++) s[k] = 0.f;
        if (i < total) {
            for (int z0 = chain; z0 < splits; z0 += 8 * zg) {
                float q[8][V];                            // all of them requested before the first is added
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    const int z = z0 + b * zg;
                    if (VEC) {
                        const float4 r = z < splits ? __ldg(reinterpret_cast<const float4 *>(partial + (long long)z * total + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
                        q[b][0] = r.x; q[b][1 % V] = r.y; q[b][2 % V] = r.z; q[b][3 % V] = r.w;
                    } else {
                        q[b][0] = z < splits ? __ldg(partial + (long long)z * total + i) : 0.f;
                    }
                }
#pragma unroll
                for (int b = 0; b < 8; b++)
#pragma unroll
                    for (int k = 0; k < V; k++) s[k] += q[b][k];
            }
        }
        if (zg > 1) {
#pragma unroll
            for (int k = 0; k < V; k++) sm[warp][k * 32 + lane] = s[k];
            __syncthreads();
            if (chain == 0)
                for (int w = 1; w < zg; w++)
#pragma unroll
                    for (int k = 0; k < V; k++) s[k] += sm[w * groups + grp][k * 32 + lane];
        }
        if (chain == 0 && i < total) {
            const int m = small ? by_N.div((int)i) : (int)(i / N), n = (int)(i - (long long)m * N);
#pragma unroll
            for (int k = 0; k < V; k++) {
                float v = s[k] * scale;
                if (bias) v += __ldg(bias + n + k);
                cs(m, n + k, epilogue_act(v, act));
            }
        }
        if (zg > 1) __syncthreads();
    }
}
template <class CS>
void launch_splitk_reduce(const TmaGemmParams &p, const CS &cs, int splits, cudaStream_t st) {
    const bool vec = (p.N & 3) == 0;
    const long long outs = (long long)p.M * p.N / (vec ? 4 : 1);
    // chains: as long as each keeps a batch of eight reads and there are not yet four blocks' worth of outputs per SM
    int zg = 1;
    while (zg < 8 && splits >= 16 * zg && outs * zg < (long long)rt().sm_count * 4 * 256) zg *= 2;
    const long long per_block = 256 / zg;
    const long long need = (outs + per_block - 1) / per_block, cap = (long long)rt().sm_count * 8;
    const int grid = (int)(need < cap ? need : cap);
    if (vec) tma_splitk_reduce_kernel<CS, true><<<grid, 256, 0, st>>>(p.partial, cs, p.M, p.N, splits, p.bias, p.act, p.out_scale, p.dinv, zg, fast_div(p.N));
    else tma_splitk_reduce_kernel<CS, false><<<grid, 256, 0, st>>>(p.partial, cs, p.M, p.N, splits, p.bias, p.act, p.out_scale, p.dinv, zg, fast_div(p.N));
    count_launch();
}

int *tc_status_word();

inline int tma_pick_bn(int N, int ns, int b_mn) {
    int bn = N <= 32 ? 32 : (N <= 64 ? 64 : (N <= 128 ? 128 : 256));
    if (b_mn && bn < 64) bn = 64;
    if (ns == 2 && bn > rt().tile_n_cap2) bn = rt().tile_n_cap2;
    if (ns >= 3 && bn > rt().tile_n_cap3) bn = rt().tile_n_cap3;
    // at least two stages of ns * (128 + bn) * 128 bytes must fit beside the epilogue staging
    while (bn > 32 && 2 * (size_t)ns * (TC_BM + bn) * 128 > 225 * 1024 - TG_EPI_WARPS * EPI_WARP_SMEM - 1024) bn >>= 1;
    return bn;
}

// Estimated time of a k-step: its MMAs (see tma_gemm_kernel) or its loads, at the 1.75 GHz that the tensor pipe's load leaves.
inline double tma_kstep_us(int bn, int ns, int joined, size_t stage_bytes) {
    auto mma = [](int n) { return n >= 128 ? n / 2 : 32 + n / 4; };
    const int products = ns == 1 ? 1 : (ns == 2 ? 3 : 6);
    const int slice = joined ? (ns == 2 ? mma(2 * bn) + mma(bn) : 2 * (mma(2 * bn) + mma(bn))) : products * mma(bn);
    const double loads = 180. + (double)stage_bytes / 140.;
    return (4. * slice > loads ? 4. * slice : loads) / 1750.;
}

// How many clusters of `size` CTAs of one SM each the chip holds at once (GPU processing clusters lose what is left over of their SMs).
int clusters_at_once(int size);

// Shared memory of a launch: bytes of a stage, stages that fit beside the epilogue's staging (227 KB per CTA on sm_100a; 2 KB are kept
// for the kernel's static shared memory and alignment slack).
inline size_t tma_stage_bytes(const TmaGemmParams &p, int bn, int ns) { return (size_t)ns * (TC_BM * 128 + (size_t)(p.pair ? bn / 2 : bn) * 128); }
inline int tma_stages(size_t stage) {
    const int n = (int)((225 * 1024 - TG_EPI_WARPS * EPI_WARP_SMEM - 1024) / stage);
    return n > 8 ? 8 : n;
}

// How a product's contraction is shared out at an accumulator width, by estimated time (microseconds past a launch's start).  A tile's way
// out takes 1 us for 128 columns.
//   one CTA a tile:     rounds of tiles over the SMs, each its k-steps and a tile's way out
//   a cluster a tile:   2 to 8 CTAs share the k-steps and add up through each other's shared memory, 2 us for 128 columns and 0.25 for
//                       each CTA; for as many tiles as clusters of that size fit on the chip at once
//   split with partial sums (allow_split): items of (tile, part) in rounds, a second launch of 3 us that adds the parts up, and
//                       the parts' way to L2 and back, 4 (2 parts + 1) M N bytes at 5 TB/s
// Where the tiles of a last round are few, that round goes to clusters too, as a launch of its own (6 us): 12432 x 256 x
// 2304 in six products (148 + 48 tiles) 75 -> 67 us.
// At least two k-steps for every CTA.  Ties go to fewer parts.  1600 x 256 x 2304 in six products (26 tiles,
// 38 us by one CTA each): 23.5 / 18.6 / 16.8 / 16.2 us by clusters of 2 / 3 / 4 / 5; 1000 x 1024 x 784 (64 tiles) 20.3 -> 15.1.  For 128 x
// 128 x 2304 (one tile, 37.5) clusters of 8 take 12.5 and a split of 18 with its reduction 7.5 + 4.2.
struct TmaShare {
    double us = 0.;
    int splits = 1, shared = 1;                    // parts in memory; CTAs a tile
    long long rest = 0;                            // tiles of a last round in clusters of
    int rest_shared = 0;
};
// The counts of parts worth trying for `ksteps` k-steps: after `parts`, the next one whose longest part is shorter (0: none).  Those between
// leave parts without work, or as long as before: 2048 k-steps have 81 such counts up to 256.
inline int tma_next_parts(int ksteps, int parts) {
    const int per = (ksteps + parts - 1) / parts;
    return per > 1 ? (ksteps + per - 2) / (per - 1) : 0;
}
inline TmaShare tma_share(const TmaGemmParams &p, int bn, int joined, int ns, bool allow_split) {
    TmaShare r;
    const size_t stage = tma_stage_bytes(p, bn, ns);
    const int stages = tma_stages(stage), tm = p.pair ? 2 * TC_BM : TC_BM;
    const int sms = p.pair ? rt().sm_count / 2 : rt().sm_count, ksteps = (p.K - 1) / TC_BK + 1;      // workers: CTAs, or pairs of them
    const long long tiles = (long long)((p.M - 1) / tm + 1) * ((p.N - 1) / bn + 1);
    // Weight gradients of convolutions: their loads of A take 0.36 us a k-step and copy at any width, and their outputs lie a filter's taps
    // apart, one sector each: 8 us for a tile of 128 columns by one CTA.
    const bool taps = p.a_mode == TMA_A_TAPS;
    const double mma_us = tma_kstep_us(bn, ns, joined, stage), kstep_us = taps && mma_us < 0.36 * ns ? 0.36 * ns : mma_us;
    const double out_us = bn / 128., scatter_us = taps ? 8. * out_us : 0.;
    auto rounds_us = [&](long long items, int per, double scatter) {
        const long long up = items + sms - 1;                     // (a 64-bit division takes several times a 32-bit one)
        const double rounds = up < (1ll << 32) ? (double)((unsigned)up / (unsigned)sms) : (double)(up / sms);
        return rounds * (per * kstep_us + out_us + scatter);
    };
    // the cluster size that finishes `n` tiles first, if that is before `t`
    auto clusters = [&](long long n, double &t) {
        int size = 0;
        for (int c = 2; c <= 8 && 2 * c <= ksteps && n * c <= sms && !p.pair; c++) {
            const unsigned chunks = (unsigned)bn / 8;
            if ((chunks + c - 1) / c * c * (size_t)4096 > stages * stage) continue;        // every share of a CTA's chunks, where the ring was
            const int per = (ksteps + c - 1) / c;
            if ((c - 1) * per >= ksteps) continue;
            const double u = per * kstep_us + 1. + (2. + 0.25 * c) * out_us + scatter_us / c;
            if (u < t && n <= clusters_at_once(c)) { t = u; size = c; }
        }
        return size;
    };
    r.us = rounds_us(tiles, ksteps, scatter_us);
    if (const int c = clusters(tiles, r.us)) r.shared = c;
    if (tiles > sms && tiles % sms) {
        double last = rounds_us(1, ksteps, scatter_us) - 6.;
        r.rest_shared = clusters(tiles % sms, last);
        if (r.rest_shared) { r.rest = tiles % sms; r.us = rounds_us(tiles - r.rest, ksteps, scatter_us) + 6. + last; }
    }
    if (allow_split) {
        const double pass_us = (double)p.M * p.N * 4. / 5e6, sum_us = 3. + (taps ? (double)p.M * p.N / (1750. * sms) : 0.);
        // no count takes less than the k-steps evenly over the SMs (a little off that, for the roundings on the way)
        const double least_us = (double)tiles * ksteps / sms * kstep_us * (1. - 1e-6) + sum_us;
        const int maxs = ksteps / 2 < 256 ? ksteps / 2 : 256;
        for (int parts = 2; parts && parts <= maxs; parts = tma_next_parts(ksteps, parts)) {
            const double way_us = (2. * parts + 1.) * pass_us;
            if (least_us + way_us >= r.us) break;
            const double t = rounds_us(tiles * parts, (ksteps + parts - 1) / parts, 0.) + sum_us + way_us;
            if (t < r.us) { r.us = t; r.splits = parts; r.shared = 1; r.rest = 0; }
        }
    }
    return r;
}

// Chooses the accumulator width and whether the launch runs as CTA pairs; sets p.bn and p.pair from p.M, p.N, p.b_mn and returns how the
// contraction is shared out, for launch_tma_gemm.  Every call of a program that runs eagerly pays for this, so each width is estimated once
// (2.7 GHz Xeon, a plan: 576 x 128 x 131072 in one product 7.2 -> 1.0 us, the same x 25600 in six 5.3 -> 0.7, 1152 x 256 x 6400 in six 1.6 -> 0.2).
// Pairs pay when the operand stream bounds the kernel (the split modes: per CTA and k-step 128 + N/2 operand rows instead of
// 128 + N) and there are enough 256-row tiles to keep 74 pairs busy; a launch that may split its contraction always has.
inline TmaShare tma_plan(TmaGemmParams &p, int ns, bool allow_split) {
    p.bn = tma_pick_bn(p.N, ns, p.b_mn);
    p.pair = 0;
    // split products: one thread, B's first two copies as one operand; the others: two threads where TMEM has room for
    // their accumulators (2 buffers x issuers x bn <= 512 columns), one for 256-column instructions.
    // Outputs of a layer in six products keep the order of sums that two threads give, but for convolutions of 128 columns: another order
    // moves the ReLU and pool decisions that lie on a tie, and programs that follow a run from version to version see that (a network with
    // batch normalisation: 1e-3 to 1e-2 of a first-layer gradient in one of ten seeds).  It costs 1.5 us of 14 at 32768 x 64 x 288 and
    // nothing for Dense layers; at 128 columns the joined form is 3 % faster (198912 x 128 x 576: 126 -> 122 us).  Products of few tiles have
    // another order all the same, where a cluster shares the contraction: there it halves the time.
    auto joined = [&](int bn) { return ns >= 2 && bn <= 128 && !(ns == 3 && p.forward && (p.a_mode != TMA_A_IM2COL || bn < 128)); };
    // Half the width gives twice the tiles, which is worth its extra loads of A where the wider ones leave SMs without work or a long way out
    // of the accumulators: 1000 x 1024 x 1024 in one product, 256 columns 12.4, 128 columns 9.3 us; 3136 x 512 x 4608 20.9 against 24.2.
    // (A width changes no order of sums by itself; convolutions in six products are joined at 128 columns and not below.)
    TmaShare how;
    auto share = [&](int bn) { return p.phases ? TmaShare{} : tma_share(p, bn, joined(bn), ns, allow_split); };
    if (!rt().pair_tiles) {
        how = share(p.bn);
        if (!p.phases && !(ns == 3 && p.forward && p.a_mode == TMA_A_IM2COL))
            while (p.bn >= 128) {
                const TmaShare half = share(p.bn / 2);
                if (half.us + 0.5 >= how.us) break;
                p.bn /= 2;
                how = half;
            }
    }
    p.joined = joined(p.bn);
    p.issuers = p.bn <= 128 && !p.joined ? 2 : 1;
    if (rt().mma_issuers && rt().mma_issuers < p.issuers) p.issuers = rt().mma_issuers;
    if (!rt().pair_tiles) return how;
    int bn = p.bn;
    if (ns == 2 && p.N > 128) bn = 256;               // a pair stages half of B per CTA: 2 x (16 + 16) KB per stage, three stages
    const long long pair_tiles = (long long)((p.M + 2 * TC_BM - 1) / (2 * TC_BM)) * ((p.N + bn - 1) / bn);
    if (ns > 2 || rt().sm_count < 4 || p.narrow || bn < 64 || (p.b_mn && bn < 128) || p.M < 2 * TC_BM ||
        (!allow_split && pair_tiles < rt().sm_count / 2)) return share(p.bn);
    p.bn = bn;
    p.pair = !p.phases;                               // (phases share a launch of single CTAs)
    p.joined = 0;
    return p.phases ? how : tma_share(p, p.bn, 0, ns, allow_split);
}

// Launches the kernel on prepared tensor maps.  p.M, p.N, p.K (contraction length in elements), a_mode, b_mn, bn
// and the geometry fields must be set; kchunk, stages, partial and status are filled here.  `how` is what tma_plan returned.
template <class CS>
int launch_tma_gemm(const TmaMapSet<phases_of<CS>::value> &maps, TmaGemmParams p, const CS &cs, int ns, const TmaShare &how, double flops,
                    const char *name) {
    if (p.issuers != 2 || p.pair || p.joined || 4 * p.bn > 512) p.issuers = 1;      // TMEM has 512 columns
    const int tm = p.pair ? 2 * TC_BM : TC_BM;
    const size_t stage = tma_stage_bytes(p, p.bn, ns);
    const int stages = tma_stages(stage);
    if (stages < 2) return fail(SEERA_E_LIMIT, "%s: tile does not fit shared memory", name);
    size_t smem = stage * stages + TG_EPI_WARPS * EPI_WARP_SMEM + 1024;
    const long long tiles = (long long)((p.M + tm - 1) / tm) * ((p.N + p.bn - 1) / p.bn), ksteps = (p.K + TC_BK - 1) / TC_BK;
    int splits = p.phases ? p.phases : how.splits;
    const long long rest = how.rest;
    p.shared = how.shared;
    const int parts = p.shared > 1 ? p.shared : (p.phases ? 1 : splits);
    p.kchunk = (int)((ksteps + parts - 1) / parts) * TC_BK;
    if (!p.phases) splits = p.shared > 1 ? 1 : (p.K + p.kchunk - 1) / p.kchunk;
    p.splits = splits;
    p.stages = stages;
    p.by_mtiles = fast_div((p.M + tm - 1) / tm); p.by_ntiles = fast_div((p.N + p.bn - 1) / p.bn);
    p.by_OHW = fast_div(p.OHW); p.by_OW = fast_div(p.OW); p.by_S = fast_div(p.S); p.by_cchunks = fast_div(p.cchunks);
    p.status = tc_status_word();
    p.wait_clocks = rt().tc_wait_clocks;
    p.skip_load = rt().tc_test_skip_load;
    rt().tc_test_skip_load = -1;                 // one launch only
    p.partial = nullptr;
    if (splits > 1 && !p.phases) {
        p.partial = (float *)scratch_alloc((size_t)splits * p.M * p.N * sizeof(float));
        if (!p.partial) return SEERA_E_OOM;
    }
    long long all_tiles = tiles * splits;
    const long long workers = p.pair ? rt().sm_count / 2 : rt().sm_count;
    p.first = 0;
    p.tiles = (int)(all_tiles - rest);
    dim3 grid((unsigned)((p.tiles < workers ? p.tiles : workers) * (p.pair ? 2 : 1)));     // persistent: one CTA per SM at most
    if (p.shared > 1) grid.x = (unsigned)(tiles * p.shared);
    unsigned cluster = p.pair ? 2u : (unsigned)p.shared;
    cudaStream_t st = rt().stream;
    cudaError_t e;
    profile_begin();
#define SEERA_TMA_LAUNCH(NSV, PAIRV, NARROWV)                                                                              \
    {                                                                                                                      \
        auto kern = tma_gemm_kernel<NSV, CS, PAIRV, NARROWV>;                                                              \
        e = allow_smem((const void *)kern, 225 * 1024);                                                                    \
        if (e == cudaSuccess) {                                                                                            \
            cudaLaunchConfig_t cfg = {};                                                                                   \
            cfg.gridDim = grid; cfg.blockDim = dim3(TG_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = st;             \
            cudaLaunchAttribute attr[1];                                                                                   \
            attr[0].id = cudaLaunchAttributeClusterDimension;                                                              \
            attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;                \
            cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 1 : 0;                                                          \
            e = cudaLaunchKernelEx(&cfg, kern, maps, cs, p);                                                               \
            if (e == cudaSuccess) e = cudaGetLastError();                                                                  \
        }                                                                                                                  \
    }
    for (int turn = 0; turn < (rest ? 2 : 1); turn++) {
        if (turn) {
            if (e != cudaSuccess) break;
            p.first = p.tiles; p.tiles = (int)all_tiles; p.shared = how.rest_shared; p.skip_load = -1;
            p.kchunk = (int)((ksteps + how.rest_shared - 1) / how.rest_shared) * TC_BK;
            grid.x = (unsigned)(rest * how.rest_shared); cluster = (unsigned)how.rest_shared;
        }
        constexpr bool N = narrow_of<CS>::value;
        if (p.pair) { if (ns == 1) SEERA_TMA_LAUNCH(1, true, false) else SEERA_TMA_LAUNCH(2, true, false) }
        else if (N && p.narrow) { if (ns == 1) SEERA_TMA_LAUNCH(1, false, N) else if (ns == 2) SEERA_TMA_LAUNCH(2, false, N) else SEERA_TMA_LAUNCH(3, false, N) }
        else if (ns == 1) SEERA_TMA_LAUNCH(1, false, false) else if (ns == 2) SEERA_TMA_LAUNCH(2, false, false) else SEERA_TMA_LAUNCH(3, false, false)
        count_launch();
    }
#undef SEERA_TMA_LAUNCH
    if (e == cudaSuccess && p.partial) {
        launch_splitk_reduce(p, cs, splits, st);
        e = cudaGetLastError();
    }
    if (p.partial) scratch_free(p.partial);
    profile_end(flops, name);
    rt().tc_used = true;
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, name);
}

// Dense: A operand shadow `sa`; a_mn = 0: sa is [M, K] (read along its rows); a_mn = 1: sa is [K, M].  Likewise B with N.
template <class CS>
int run_tma_gemm(const Shadow &sa, int a_mn, const Shadow &sb, int b_mn, const CS &cs, int M, int N, int K,
                 bool allow_split, const char *name, const float *bias = nullptr, int act = 0, int copies = 0) {
    const int ns = copies ? copies : precision_copies();
    TmaGemmParams p{};
    p.bias = bias; p.act = act;
    p.M = M; p.N = N; p.K = K; p.a_mode = a_mn ? TMA_A_COLS : TMA_A_ROWS; p.b_mn = b_mn;
    p.forward = !a_mn && b_mn;                    // C = A B
    p.a_fp16 = sa.enc.fmt; p.b_fp16 = sb.enc.fmt; p.out_scale = 1.f / (sa.enc.scale * sb.enc.scale);
    p.dinv = enc_dinv(sa.enc, sb.enc);
    const TmaShare how = tma_plan(p, ns, allow_split);
    TmaMapSet<1> set;
    TmaMaps &maps = set.of[0];
    for (int i = 0; i < 3; i++) {
        int j = i < ns ? i : 0;
        // K-major: inner dimension = K (cols of the shadow), box 64 x rows-of-tile; MN-major: inner = M/N, box 64 x 64 k lines
        if (int s = make_map_2d(&maps.a[i], sa.p[j], sa.rows, sa.cols, sa.ld, 64, a_mn ? 64 : TC_BM)) return s;
        if (int s = make_map_2d(&maps.b[i], sb.p[j], sb.rows, sb.cols, sb.ld, 64, b_mn ? 64 : (p.pair ? p.bn / 2 : p.bn))) return s;
    }
    return launch_tma_gemm(set, p, cs, ns, how, 2.0 * M * N * (double)K, name);
}

}  // namespace seera
