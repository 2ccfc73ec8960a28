// 3 x 3 unit-stride convolution with one to three input channels + bias + activation + 2x2 / stride-2 max-pool on the tensor cores: the
// first layer of an image network at a batch that fills the chip.
//
// As fp32 multiply-adds the layer is bound by the fp32 pipe (conv3x3_pool_kernel: 56 us for 3 -> 64 channels, 512 images of 32 x 32, whose
// traffic is 100 MB = 15 us; the multiply-adds alone take 26).  This kernel takes 35 us (777 images with three copies: 95 -> 52), bound by
// what the epilogue warps issue; producers and products alone take 26 for 777.  Here a tile is 128 pool windows, and each of the four positions inside
// the window is a GEMM of its own, [128 windows, 9 C] x [9 C, F], into its own quarter of the accumulator: the TMEM lane is the window,
// so that the four values that the pool compares sit in one thread and the pooled values of a warp are 32 neighbours in memory.
//   producers   8 warps, two groups of four; thread = window.  It reads the window's 4 x 4 x C patch once (48 values), and for each
//               position writes one 64-value row: the bf16 copies of its 9 C values, first copy | second copy, and the third one in a
//               row of its own.  Three copies hold all 24 bits of an fp32 value.
//   MMA         one warp: per position the six products of the copies that matter (those left out are below 2^-24), K = 32 each
//   epilogue    8 warps, two per lane quarter that take turns by tile, 16 filters at a time: bias, activation, maximum and its index (the
//               first maximum wins), pooled values, indices and the channels-last copies for the next convolution
// Each position has a stage for its operand rows, the accumulator is double-buffered; the CTA is persistent.
// The result is fp32-class in every mode: all copies are made whatever the mode's own number is.
// Values that have no bf16 copies (infinities, NaNs, and what rounds to infinity) would leave NaNs behind, which the maximum passes over: a
// producer that meets one makes all products of the window NaN, and the epilogue forms such a window again in fp32, in the order of
// conv3x3_pool_kernel.  So it does with every window if it is a filter that holds such a value.  (Finite values whose result lies in the last
// 2^-8 below fp32's largest may still overflow: the leading copies' product is that much larger at most.)
#include "conv_first.cuh"
#include "internal.h"
#include "tma_gemm_kernel.cuh"

namespace seera {

constexpr int PT_STAGES = 4 /* one per position of the window */, PT_PRODUCER_WARPS = 8, PT_EPI_WARPS = 8;
constexpr int PT_THREADS = 32 * (PT_PRODUCER_WARPS + 1 + PT_EPI_WARPS);
constexpr uint32_t PT_A_TILE = TC_BM * 128, PT_STAGE = 2 * PT_A_TILE;
constexpr int PT_ROW = 64 + 4;                 // floats of a window's row in an epilogue warp's staging
constexpr size_t PT_SMEM = 1024 + 2 * 64 * 128 + PT_STAGES * (size_t)PT_STAGE + (64 + PT_EPI_WARPS * 32 * PT_ROW) * sizeof(float);

struct PoolTcGeom {
    int C, H, W, F, OHq, OWq, Pq, ph, pw, windows, tiles, bn, act;
    FastDiv by_Pq, by_OWq;
};

constexpr float PT_LARGEST = 3.38e38f;         // up to it a value has finite bf16 copies

__device__ __forceinline__ uint32_t pt_offset(int row, int chunk) { return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4); }
// 16 columns of this warp's 32 lanes, requested
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, float *v) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

template <int C, int ACT>
__global__ void __launch_bounds__(PT_THREADS, 1)
conv_pool_tc_kernel(const float *__restrict__ X, const float *__restrict__ Wt, const float *__restrict__ bias, PoolOut po, PoolTcGeom g,
                    int *status) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long bars[3 * PT_STAGES + 4];      // full, empty of even and of odd tiles, tfull[2], tempty[2]
    __shared__ uint32_t tmem_base_slot;
    __shared__ int abort_flag, filters_bad;
    constexpr int K = 9 * C, CHUNKS = (K + 15) / 16 * 2, SLICES = CHUNKS / 2;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, f_base = blockIdx.y * 64;
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *b_base = smem, *a_base = smem + 2 * 64 * 128;
    float *bk = reinterpret_cast<float *>(a_base + PT_STAGES * (size_t)PT_STAGE);
    const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[PT_STAGES]), tfull0 = smem_u32(&bars[3 * PT_STAGES]), tempty0 = tfull0 + 16;
    uint32_t cols = 32;
    while (cols < (uint32_t)(8 * g.bn)) cols <<= 1;

    if (t == 0) {
        abort_flag = 0;
        filters_bad = 0;
        for (int s = 0; s < PT_STAGES; s++) mbar_init(full0 + 8 * s, 4);
        for (int s = 0; s < 2 * PT_STAGES; s++) mbar_init(empty0 + 8 * s, 1);
        for (int b = 0; b < 2; b++) { mbar_init(tfull0 + 8 * b, 1); mbar_init(tempty0 + 8 * b, 4); }
        fence_mbar_init();
    }
    __syncthreads();
    for (int e = t; e < g.bn; e += PT_THREADS) bk[e] = bias ? __ldg(bias + f_base + e) : 0.f;
    // filters: row f = first copy | second copy, and the third copy in the tile behind
    for (int e = t; e < g.bn * CHUNKS; e += PT_THREADS) {
        const int row = e / CHUNKS, kg = e - row * CHUNKS;
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int k = kg * 8 + i;
            v[i] = k < K ? __ldg(Wt + (long long)(f_base + row) * K + k) : 0.f;
            if (!(fabsf(v[i]) <= PT_LARGEST)) filters_bad = 1;
        }
        *reinterpret_cast<uint4 *>(b_base + pt_offset(row, kg)) = split_chunk(v);
        *reinterpret_cast<uint4 *>(b_base + pt_offset(row, kg + 4)) = split_chunk(v);
        *reinterpret_cast<uint4 *>(b_base + 64 * 128 + pt_offset(row, kg)) = split_chunk(v);
    }
    fence_async_smem();
    if (warp == PT_PRODUCER_WARPS) tmem_alloc(smem_u32(&tmem_base_slot), cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_base_slot;
    volatile int *abortp = &abort_flag;

    if (warp < PT_PRODUCER_WARPS) {
        // ---------------- producers: group of four warps = every other tile of the CTA, thread = window ----------------
        const int group = warp >> 2, row = t & 127, plane = g.H * g.W;
        for (int it = group, tile = blockIdx.x + group * gridDim.x; tile < g.tiles; it += 2, tile += 2 * gridDim.x) {
            const int wi = min(tile * TC_BM + row, g.windows - 1), n = g.by_Pq.div(wi), rem = wi - n * g.Pq, qr = g.by_OWq.div(rem);
            const int ih0 = 2 * qr - g.ph, iw0 = 2 * (rem - qr * g.OWq) - g.pw;
            const float *xn = X + (long long)n * C * plane + (long long)ih0 * g.W + iw0;
            float v[C][4][4];
            bool bad = false;
#pragma unroll
            for (int c = 0; c < C; c++)
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const bool in = (unsigned)(ih0 + i) < (unsigned)g.H && (unsigned)(iw0 + j) < (unsigned)g.W;
                        v[c][i][j] = in ? __ldg(xn + c * plane + i * g.W + j) : 0.f;
                        bad |= !(fabsf(v[c][i][j]) <= PT_LARGEST);
                    }
            bool gave_up = false;
#pragma unroll
            for (int p = 0; p < 4; p++) {
                // A tile's use of a stage waits until the tile before it, the other group's, has been read out of it.  Even and odd tiles have
                // barriers of their own, so that each group sees every phase of the one it waits on.
                if (it > 0 && !mbar_wait(empty0 + 8 * (((it - 1) & 1) * PT_STAGES + p), (uint32_t)((it - 1) >> 1) & 1u, abortp, status, 1)) {
                    gave_up = true;
                    break;
                }
                const int s = p;
                unsigned char *a = a_base + (size_t)s * PT_STAGE;
#pragma unroll
                for (int kg = 0; kg < CHUNKS; kg++) {
                    float u[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int k = kg * 8 + i, c = k / 9, r = (k % 9) / 3, q = k % 3;
                        u[i] = k < K ? v[c < C ? c : 0][(p >> 1) + r][(p & 1) + q] : 0.f;
                    }
                    if (kg == 0 && bad) u[0] = __int_as_float(0x7fffffff);
                    *reinterpret_cast<uint4 *>(a + pt_offset(row, kg)) = split_chunk(u);
                    *reinterpret_cast<uint4 *>(a + pt_offset(row, kg + 4)) = split_chunk(u);
                    *reinterpret_cast<uint4 *>(a + PT_A_TILE + pt_offset(row, kg)) = split_chunk(u);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * s);
            }
            if (gave_up) break;
        }
    } else if (warp == PT_PRODUCER_WARPS) {
        // ---------------- MMA issuer: a converged warp, one lane of which issues ----------------
        const uint32_t idesc = umma_idesc_bf16(g.bn);
        const bool leader = elect_one();
        int it = 0;
        for (int tile = blockIdx.x; tile < g.tiles; tile += gridDim.x, it++) {
            const int buf = it & 1;
            if (!mbar_wait(tempty0 + 8 * buf, (((uint32_t)it >> 1) & 1u) ^ 1u, abortp, status, 4)) break;
            bool gave_up = false;
            for (int p = 0; p < 4; p++) {
                const int s = p;
                if (!mbar_wait(full0 + 8 * s, (uint32_t)it & 1u, abortp, status, 2)) { gave_up = true; break; }
                tc_fence_after();
                if (leader) {
                    const uint32_t d = tmem_base + (uint32_t)((buf * 4 + p) * g.bn), a = smem_u32(a_base) + s * PT_STAGE, b = smem_u32(b_base);
                    uint32_t acc = 0;
#pragma unroll
                    for (int j = 0; j < SLICES; j++) {
                        const uint64_t a0 = umma_desc_sw128(a + 32 * j), a1 = umma_desc_sw128(a + 64 + 32 * j), a2 = umma_desc_sw128(a + PT_A_TILE + 32 * j);
                        const uint64_t b0 = umma_desc_sw128(b + 32 * j), b1 = umma_desc_sw128(b + 64 + 32 * j), b2 = umma_desc_sw128(b + 64 * 128 + 32 * j);
                        umma_bf16(d, a0, b0, idesc, acc);
                        acc = 1;
                        umma_bf16_add(d, a0, b1, idesc);
                        umma_bf16_add(d, a1, b0, idesc);
                        umma_bf16_add(d, a0, b2, idesc);
                        umma_bf16_add(d, a2, b0, idesc);
                        umma_bf16_add(d, a1, b1, idesc);
                    }
                    umma_commit(empty0 + 8 * ((it & 1) * PT_STAGES + s));
                    if (p == 3) umma_commit(tfull0 + 8 * buf);
                }
                __syncwarp();
            }
            if (gave_up) break;
        }
    } else {
        // ---------------- epilogue: lane quarter warp % 4 (= the warp's rank in the CTA modulo 4), every other tile ----------------
        // The pooled values also go through shared memory, so that eight lanes write the 128 bytes a window owns in each channels-last copy.
        const int q = warp & 3, ew = warp - PT_PRODUCER_WARPS - 1, half = ew >> 2;
        float *stage = bk + 64 + ew * 32 * PT_ROW;
        for (int it = half, tile = blockIdx.x + half * gridDim.x; tile < g.tiles; it += 2, tile += 2 * gridDim.x) {
            const int buf = half;                         // = it & 1
            if (!mbar_wait(tfull0 + 8 * buf, ((uint32_t)it >> 1) & 1u, abortp, status, 3)) break;
            tc_fence_after();
            const int w0 = tile * TC_BM + q * 32, wi = w0 + lane, wl = min(wi, g.windows - 1), n = g.by_Pq.div(wl), rem = wl - n * g.Pq;
            const bool live = wi < g.windows;
            float *op = po.pooled + ((long long)n * g.F + f_base) * g.Pq + rem;
            int *om = po.mask + ((long long)n * g.F + f_base) * g.Pq + rem;
            const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 4 * g.bn);
            bool again = filters_bad != 0;
            for (int f0 = 0; f0 < g.bn; f0 += 16) {
                float z[4][16];
#pragma unroll
                for (int p = 0; p < 4; p++) tmem_ld16_issue(at + (uint32_t)(p * g.bn + f0), z[p]);
                tmem_ld_wait();
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int f = 0; f < 16; f++) asm volatile("" : "+f"(z[p][f]));
                if (f0 + 16 >= g.bn) {                    // the accumulator has been read: the issuer may have it while the rest goes on
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty0 + 8 * buf);
                }
#pragma unroll
                for (int f = 0; f < 16; f++) {
                    const float b = bk[f0 + f];
                    float m = -3.402823466e+38f;
                    int id = 0;
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        float x = z[p][f] + b;
                        if (ACT != SEERA_ACT_RELU) x = epilogue_act(x, ACT);
                        if (x > m) { m = x; id = p; }
                    }
                    // relu after the maximum: the same value and, since a window without a positive entry is all zeros, the same index
                    if (ACT == SEERA_ACT_RELU && !(m > 0.f)) { m = 0.f; id = 0; }
                    stage[lane * PT_ROW + f0 + f] = m;
                    if (live) { op[(unsigned)((f0 + f) * g.Pq)] = m; om[(unsigned)((f0 + f) * g.Pq)] = id; }
                }
                again |= z[0][0] != z[0][0];
            }
            if (again) {                                  // the window in fp32 (not while z is held: the accumulator reads need its registers)
                const int qr = g.by_OWq.div(rem), ih0 = 2 * qr - g.ph, iw0 = 2 * (rem - qr * g.OWq) - g.pw;
                const float *xn = X + (long long)n * C * g.H * g.W, *wk = Wt + (long long)f_base * K;
#pragma unroll 1
                for (int f = 0; f < g.bn; f++, wk += K) {
                    float m = -3.402823466e+38f;
                    int id = 0;
#pragma unroll 1
                    for (int p = 0; p < 4; p++) {
                        float x = 0.f;
#pragma unroll 1
                        for (int k = 0; k < K; k++) {
                            const int c = k / 9, ih = ih0 + (p >> 1) + (k % 9) / 3, iw = iw0 + (p & 1) + k % 3;
                            const bool in = (unsigned)ih < (unsigned)g.H && (unsigned)iw < (unsigned)g.W;
                            x = fmaf(in ? __ldg(xn + ((long long)c * g.H + ih) * g.W + iw) : 0.f, __ldg(wk + k), x);
                        }
                        x += bk[f];
                        if (ACT != SEERA_ACT_RELU) x = epilogue_act(x, ACT);
                        if (x > m) { m = x; id = p; }
                    }
                    if (ACT == SEERA_ACT_RELU && !(m > 0.f)) { m = 0.f; id = 0; }
                    stage[lane * PT_ROW + f] = m;
                    if (live) { op[(unsigned)(f * g.Pq)] = m; om[(unsigned)(f * g.Pq)] = id; }
                }
            }
            __syncwarp();
            if (po.copy[0]) {
                __syncwarp();
                const int per = g.bn >> 3, rows = min(32, g.windows - w0) * per;        // 8 filters each
                for (int e = lane; e < rows; e += 32) {
                    const int r = e / per, f = (e - r * per) * 8;
                    const float4 x = *reinterpret_cast<const float4 *>(stage + r * PT_ROW + f), y = *reinterpret_cast<const float4 *>(stage + r * PT_ROW + f + 4);
                    float u[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
                    const long long c = (long long)(w0 + r) * po.Cp + f_base + f;
                    store_split8_n(u, po.ns, po.enc, po.copy[0] + c, po.copy[1] + c, po.copy[2] + c);
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == PT_PRODUCER_WARPS) tmem_dealloc(tmem_base, cols);
}

// For F a multiple of 16 up to 64, or of 64 beyond; from a tile for every SM on (100 images of 3 x 32 x 32 into 64 filters: 14.4 against
// 15.2 us; below that the fp32 kernel's start is shorter).
bool conv_pool_tc_applies(int NB, int C, int H, int W, int F, int R, int S, int sh, int sw, int ph, int pw) {
    const int OH = H + 2 * ph - 2, OW = W + 2 * pw - 2;
    if (rt().precision < 1 || !rt().conv_tma || R != 3 || S != 3 || sh != 1 || sw != 1 || ph < 0 || pw < 0 || C < 1 || C > 3) return false;
    if (F < 32 || (F <= 64 ? F % 16 != 0 : F % 64 != 0) || F > 4096 || OH < 2 || OW < 2 || (OH & 1) || (OW & 1)) return false;
    const long long windows = (long long)NB * (OH / 2) * (OW / 2);
    return windows < (1ll << 31) - 128 && (long long)C * H * W < (1ll << 30) && windows * ((F + 63) / 64) >= (long long)TC_BM * rt().sm_count;
}

int conv_pool_tc(const float *X, const float *Wt, const float *bias, const PoolOut &pool, int NB, int C, int H, int W, int F, int ph, int pw, int act,
                 const char *name) {
    PoolTcGeom g{};
    g.C = C; g.H = H; g.W = W; g.F = F; g.ph = ph; g.pw = pw; g.act = act;
    g.OHq = (H + 2 * ph - 2) / 2; g.OWq = (W + 2 * pw - 2) / 2; g.Pq = g.OHq * g.OWq;
    g.windows = NB * g.Pq; g.tiles = (g.windows + TC_BM - 1) / TC_BM; g.bn = F < 64 ? F : 64;
    g.by_Pq = fast_div(g.Pq); g.by_OWq = fast_div(g.OWq);
    const int chunks = F < 64 ? 1 : F / 64;
    int gx = rt().sm_count / chunks;
    if (gx < 1) gx = 1;
    if (gx > g.tiles) gx = g.tiles;
    profile_begin();
    cudaError_t e = cudaSuccess;
    auto launch = [&](auto kern) {
        e = allow_smem((const void *)kern, PT_SMEM);
        if (e == cudaSuccess) kern<<<dim3((unsigned)gx, (unsigned)chunks), PT_THREADS, PT_SMEM, rt().stream>>>(X, Wt, bias, pool, g, tc_status_word());
    };
#define SEERA_PT(CV) \
    if (act == SEERA_ACT_RELU) launch(conv_pool_tc_kernel<CV, SEERA_ACT_RELU>); \
    else if (act == SEERA_ACT_SIGMOID) launch(conv_pool_tc_kernel<CV, SEERA_ACT_SIGMOID>); \
    else if (act == SEERA_ACT_TANH) launch(conv_pool_tc_kernel<CV, SEERA_ACT_TANH>); \
    else launch(conv_pool_tc_kernel<CV, SEERA_ACT_NONE>);
    if (C == 1) { SEERA_PT(1) } else if (C == 2) { SEERA_PT(2) } else { SEERA_PT(3) }
#undef SEERA_PT
    count_launch();
    if (e == cudaSuccess) e = cudaGetLastError();
    profile_end(2.0 * NB * (4.0 * g.Pq) * (double)F * C * 9, name);
    rt().tc_used = true;
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, name);
}

}  // namespace seera
