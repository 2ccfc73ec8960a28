// Nearest 2x2 unpooling followed by a 3 x 3 unit-stride transposed convolution with padding 1 onto ONE channel (the end of an
// autoencoder), without the unpooled tensor: exact fp32 on the CUDA cores, everything read and written at the low resolution.
//
// The 3 x 3 window of an output pixel covers 2 x 2 low-resolution pixels, which ones depends on the pixel's parity.  So
//   forward   the four outputs of a low pixel are 2 x 2 sums over its 3 x 3 neighbourhood with filters that are sums of the
//             3 x 3 filter's weights: 16 multiply-adds per channel instead of 36;
//   dX        the gradient of a low pixel is a 4 x 4 window of the output gradient against a 4 x 4 filter of such sums;
//   dW        a low pixel meets every tap with the sum of the output gradient over a 2 x 2 box: nine box sums per pixel serve all
//             channels.
// All three are bound by one pass over the low-resolution tensor.  At 256 x 32 x 32 x 32 (33 MB; unpooled 134 MB) this replaces an unpooling
// pass, a stencil over 134 MB, a weight gradient over 134 MB, a data gradient that writes 134 MB and its folding: 46 + 71 + 50 + 23 + 45 us.
#include "common.cuh"
#include "internal.h"
#include "tc_epilogue.cuh"

namespace seera {

constexpr int UC_CMAX = 512;          // input channels (the combined filters sit in shared memory, 64 bytes a channel)

__device__ __forceinline__ void uc_cp4(float *dst, const float *src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(take ? 4 : 0) : "memory");
}
__device__ __forceinline__ void uc_cp16(float *dst, const float *src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(take ? 16 : 0) : "memory");
}
__device__ __forceinline__ void uc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void uc_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Both kernels stream their input through a ring of cp.async stages: with loads into registers an SM had 8 KB on their way, which at a
// microsecond of latency is a fifth of the memory's rate (68 and 67 us at the size above).

// Forward: a block takes 16 rows x 32 columns of one image (warp = two rows, which share two of their four input rows and every filter
// read; lane = column); a stage holds FCH channels of that patch with its border.
constexpr int FBAND = 16, FCH = 4, FROWS = FBAND + 2, FPITCH = 40, FSTAGES = 4;       // column c of the patch at c + 4: interior rows are 16-byte aligned
__global__ void __launch_bounds__(256) unpool_convt_fwd_kernel(const float *__restrict__ x, const float *__restrict__ Wt,
                                                               const float *__restrict__ bias, float *__restrict__ y, int C, int H, int W,
                                                               int act, int segs, int bands, int items, int vec, FastDiv by_segs,
                                                               FastDiv by_bands, FastDiv by_chunks) {
    extern __shared__ __align__(16) float sm[];           // stages, then [C][a][b][low row][low column] combined filters
    float *ew = sm + FSTAGES * FCH * FROWS * FPITCH;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, chunks = by_chunks.d;
    const int my_items = ((int)items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, steps = my_items * chunks;
    const int plane = H * W;
    // the pieces of a stage this thread copies: eight of four columns and the two border columns per row
    constexpr int VPER = (FCH * FROWS * 10 + 255) / 256;
    int vch[VPER], vrow[VPER], vcol[VPER], vdst[VPER], voff[VPER];
#pragma unroll
    for (int k3 = 0; k3 < VPER; k3++) {
        const int e = t + 256 * k3, r = e / 10, p = e - 10 * r;
        vch[k3] = r / FROWS;
        vrow[k3] = e < FCH * FROWS * 10 ? r - vch[k3] * FROWS : -1;
        vcol[k3] = p < 8 ? 4 * p : (p == 8 ? -1 : 32);
        vdst[k3] = r * FPITCH + 4 + vcol[k3];
        voff[k3] = vch[k3] * plane + vrow[k3] * W + vcol[k3];
    }
    auto request = [&](int step) {
        const int k = by_chunks.div(step), chunk = step - k * chunks, item = blockIdx.x + k * gridDim.x;
        const int q = by_segs.div(item), seg = item - q * segs, n = by_bands.div(q), band = q - n * bands;
        const int i0 = band * FBAND - 1, j0 = seg * 32;
        float *st = sm + (step % FSTAGES) * (FCH * FROWS * FPITCH);
        const float *xn = x + (long long)n * C * plane;
        if (vec) {
            const int at = chunk * FCH * plane + i0 * W + j0;
#pragma unroll
            for (int k3 = 0; k3 < VPER; k3++) {
                const bool in = vrow[k3] >= 0 && chunk * FCH + vch[k3] < C && (unsigned)(i0 + vrow[k3]) < (unsigned)H &&
                                (unsigned)(j0 + vcol[k3]) < (unsigned)W;
                if (vrow[k3] >= 0) {
                    float *dst = st + vdst[k3];
                    const float *src = xn + (in ? at + voff[k3] : 0);
                    if (vcol[k3] >= 0 && vcol[k3] < 32) uc_cp16(dst, src, in); else uc_cp4(dst, src, in);
                }
            }
        } else {
            for (int e = t; e < FCH * FROWS * 34; e += 256) {
                const int r = e / 34, col = e - 34 * r - 1, ch = r / FROWS, i = i0 + r - ch * FROWS, c = chunk * FCH + ch;
                const bool in = c < C && (unsigned)i < (unsigned)H && (unsigned)(j0 + col) < (unsigned)W;
                uc_cp4(st + r * FPITCH + 4 + col, xn + (in ? c * plane + i * W + j0 + col : 0), in);
            }
        }
    };
    for (int s = 0; s < FSTAGES - 1; s++) { if (s < steps) request(s); uc_commit(); }
    for (int e = t; e < C * 16; e += 256) {
        const int c = e >> 4, a = (e >> 3) & 1, b = (e >> 2) & 1, dr = (e >> 1) & 1, dc = e & 1;
        // low rows of parity a: a = 0: i - 1 by tap row 2, i by tap rows 0 and 1; a = 1: i by tap rows 1 and 2, i + 1 by tap row 0
        const int r0 = a ? (dr ? 0 : 1) : (dr ? 0 : 2), r1 = a ? (dr ? 0 : 2) : (dr ? 1 : 2);
        const int t0 = b ? (dc ? 0 : 1) : (dc ? 0 : 2), t1 = b ? (dc ? 0 : 2) : (dc ? 1 : 2);
        float s = 0.f;
        for (int r = r0; r <= r1; r++)
            for (int k = t0; k <= t1; k++) s += __ldg(Wt + c * 9 + r * 3 + k);
        ew[e] = s;
    }
    const float b0 = bias ? __ldg(bias) : 0.f;
    float o[2][4];
#pragma unroll
    for (int k = 0; k < 4; k++) o[0][k] = o[1][k] = 0.f;
    for (int step = 0; step < steps; step++) {
        uc_wait<FSTAGES - 2>();
        __syncthreads();
        if (step + FSTAGES - 1 < steps) request(step + FSTAGES - 1);
        uc_commit();
        const int k = by_chunks.div(step), chunk = step - k * chunks;
        const float *st = sm + (step % FSTAGES) * (FCH * FROWS * FPITCH) + 2 * warp * FPITCH + 4 + lane;
        const float *wc = ew + chunk * FCH * 16;
#pragma unroll
        for (int ch = 0; ch < FCH; ch++) {
            if (chunk * FCH + ch >= C) break;
            const float *p = st + ch * (FROWS * FPITCH);
            float l[4], v[4], r[4];
#pragma unroll
            for (int h = 0; h < 4; h++) { l[h] = p[h * FPITCH - 1]; v[h] = p[h * FPITCH]; r[h] = p[h * FPITCH + 1]; }
            const float4 w00 = *reinterpret_cast<const float4 *>(wc + ch * 16), w01 = *reinterpret_cast<const float4 *>(wc + ch * 16 + 4);
            const float4 w10 = *reinterpret_cast<const float4 *>(wc + ch * 16 + 8), w11 = *reinterpret_cast<const float4 *>(wc + ch * 16 + 12);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                o[h][0] = fmaf(w00.x, l[h], fmaf(w00.y, v[h], fmaf(w00.z, l[h + 1], fmaf(w00.w, v[h + 1], o[h][0]))));
                o[h][1] = fmaf(w01.x, v[h], fmaf(w01.y, r[h], fmaf(w01.z, v[h + 1], fmaf(w01.w, r[h + 1], o[h][1]))));
                o[h][2] = fmaf(w10.x, l[h + 1], fmaf(w10.y, v[h + 1], fmaf(w10.z, l[h + 2], fmaf(w10.w, v[h + 2], o[h][2]))));
                o[h][3] = fmaf(w11.x, v[h + 1], fmaf(w11.y, r[h + 1], fmaf(w11.z, v[h + 2], fmaf(w11.w, r[h + 2], o[h][3]))));
            }
        }
        if (chunk == chunks - 1) {
            const int item = blockIdx.x + k * gridDim.x, q = by_segs.div(item), seg = item - q * segs, n = by_bands.div(q), band = q - n * bands;
            const int j = seg * 32 + lane;
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int i = band * FBAND + 2 * warp + h;
                if (i < H && j < W) {
                    float *out = y + ((long long)n * 2 * H + 2 * i) * 2 * W + 2 * j;
                    *reinterpret_cast<float2 *>(out) = make_float2(epilogue_act(o[h][0] + b0, act), epilogue_act(o[h][1] + b0, act));
                    *reinterpret_cast<float2 *>(out + 2 * W) = make_float2(epilogue_act(o[h][2] + b0, act), epilogue_act(o[h][3] + b0, act));
                }
#pragma unroll
                for (int k = 0; k < 4; k++) o[h][k] = 0.f;
            }
        }
    }
}

// Backward: lane = column, warp = four channels of the block's 32 (blockIdx.y), a stage = BROWS rows x 32 columns of one image (all 32
// channels) with the output gradient over them.  A pixel's 4 x 4 gradient window is read once per warp and serves both gradients.
// Partial sums of dW: [block][C][9].
constexpr int BROWS = 4, BSTAGES = 3, BDROWS = 2 * BROWS + 2, BDPITCH = 72;      // gradient column h of the window at h + 4
constexpr int BSTAGE = 32 * BROWS * 32 + BDROWS * BDPITCH;
__global__ void __launch_bounds__(256, 2) unpool_convt_bwd_kernel(const float *__restrict__ x, const float *__restrict__ Wt,
                                                               const float *__restrict__ dz, float *__restrict__ dx, float *__restrict__ partial,
                                                               int C, int H, int W, int segs, int bands, int items, int vec, FastDiv by_segs,
                                                               FastDiv by_bands) {
    extern __shared__ __align__(16) float sm[];
    __shared__ __align__(16) float ew[32][16];            // combined filters of this block's channels
    __shared__ float red[32][9];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, cb = blockIdx.y * 32, plane = H * W;
    auto where = [&](int item, int &n, int &i0, int &j0) {
        const int q = by_segs.div(item), seg = item - q * segs;
        n = by_bands.div(q); i0 = (q - n * bands) * BROWS; j0 = seg * 32;
    };
    auto request = [&](int item, int slot) {
        int n, i0, j0;
        where(item, n, i0, j0);
        float *st = sm + slot * BSTAGE, *sd = st + 32 * BROWS * 32;
        const float *xn = x + ((long long)n * C + cb) * plane, *dn = dz + (long long)n * 4 * plane;
        const int W2 = 2 * W;
        if (vec) {
#pragma unroll
            for (int e0 = 0; e0 < 32 * BROWS * 8; e0 += 256) {
                const int e = e0 + t, p = e & 7, r = (e >> 3) & (BROWS - 1), ch = e / (8 * BROWS);
                const bool in = cb + ch < C && i0 + r < H && j0 + 4 * p < W;
                uc_cp16(st + (ch * BROWS + r) * 32 + 4 * p, xn + (in ? ch * plane + (i0 + r) * W + j0 + 4 * p : 0), in);
            }
            if (t < BDROWS * 18) {                        // 16 pieces of four columns and the two border columns
                const int r = t / 18, p = t - 18 * r, h = 2 * i0 - 1 + r, col = p < 16 ? 4 * p : (p == 16 ? -1 : 64);
                const bool in = (unsigned)h < (unsigned)(2 * H) && (unsigned)(2 * j0 + col) < (unsigned)W2;
                const float *src = dn + (in ? h * W2 + 2 * j0 + col : 0);
                float *dst = sd + r * BDPITCH + 4 + col;
                if (p < 16) uc_cp16(dst, src, in); else uc_cp4(dst, src, in);
            }
        } else {
            for (int e = t; e < 32 * BROWS * 32; e += 256) {
                const int p = e & 31, r = (e >> 5) & (BROWS - 1), ch = e / (32 * BROWS);
                const bool in = cb + ch < C && i0 + r < H && j0 + p < W;
                uc_cp4(st + e, xn + (in ? ch * plane + (i0 + r) * W + j0 + p : 0), in);
            }
            for (int e = t; e < BDROWS * 66; e += 256) {
                const int r = e / 66, col = e - 66 * r - 1, h = 2 * i0 - 1 + r;
                const bool in = (unsigned)h < (unsigned)(2 * H) && (unsigned)(2 * j0 + col) < (unsigned)W2;
                uc_cp4(sd + r * BDPITCH + 4 + col, dn + (in ? h * W2 + 2 * j0 + col : 0), in);
            }
        }
    };
    for (int s = 0; s < BSTAGES - 1; s++) {
        if ((int)(blockIdx.x + s * gridDim.x) < items) request(blockIdx.x + s * gridDim.x, s);
        uc_commit();
    }
    for (int e = t; e < 32 * 16; e += 256) {
        const int c = cb + (e >> 4), u = (e >> 2) & 3, v = e & 3;
        float s = 0.f;
        if (c < C)
            for (int r = max(0, u - 1); r <= min(2, u); r++)
                for (int q = max(0, v - 1); q <= min(2, v); q++) s += __ldg(Wt + c * 9 + r * 3 + q);
        ew[e >> 4][e & 15] = s;
    }
    float acc[4][9];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < 9; i++) acc[k][i] = 0.f;
    const int c0 = cb + warp * 4;
    int slot = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        uc_wait<BSTAGES - 2>();
        __syncthreads();
        const int ahead = item + (BSTAGES - 1) * gridDim.x;
        if (ahead < items) request(ahead, slot == 0 ? BSTAGES - 1 : slot - 1);
        uc_commit();
        int n, i0, j0;
        where(item, n, i0, j0);
        const float *st = sm + slot * BSTAGE + warp * 4 * BROWS * 32 + lane, *sd = sm + slot * BSTAGE + 32 * BROWS * 32 + 2 * lane + 4;
        const bool in = j0 + lane < W;
        float *dxp = dx ? dx + ((long long)n * C + c0) * plane + (long long)i0 * W + j0 + lane : nullptr;
        float d[4][4];                                    // window rows 2i - 1 .. 2i + 2, columns 2j - 1 .. 2j + 2
        auto row = [&](int r, float *o) {
            const float *p = sd + r * BDPITCH;
            const float2 m = *reinterpret_cast<const float2 *>(p);
            o[0] = p[-1]; o[1] = m.x; o[2] = m.y; o[3] = p[2];
        };
        row(0, d[2]); row(1, d[3]);
#pragma unroll
        for (int i = 0; i < BROWS; i++) {
#pragma unroll
            for (int k = 0; k < 4; k++) { d[0][k] = d[2][k]; d[1][k] = d[3][k]; }
            row(2 * i + 2, d[2]); row(2 * i + 3, d[3]);
            if (dx && in && i0 + i < H) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (c0 + k < C) {
                        float s = 0.f;
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const float4 w4 = *reinterpret_cast<const float4 *>(&ew[warp * 4 + k][4 * u]);
                            s = fmaf(w4.x, d[u][0], fmaf(w4.y, d[u][1], fmaf(w4.z, d[u][2], fmaf(w4.w, d[u][3], s))));
                        }
                        dxp[(long long)k * plane + i * W] = s;
                    }
                }
            }
            float xv[4], cols[4][3];                      // (pixels outside the image hold zeros)
#pragma unroll
            for (int k = 0; k < 4; k++) xv[k] = st[(k * BROWS + i) * 32];
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int s = 0; s < 3; s++) cols[u][s] = d[u][s] + d[u][s + 1];
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int s = 0; s < 3; s++) {
                    const float box = cols[r][s] + cols[r + 1][s];
#pragma unroll
                    for (int k = 0; k < 4; k++) acc[k][3 * r + s] = fmaf(xv[k], box, acc[k][3 * r + s]);
                }
        }
        if (++slot == BSTAGES) slot = 0;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int i = 0; i < 9; i++) {
            float v = acc[k][i];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red[warp * 4 + k][i] = v;
        }
    __syncthreads();
    for (int e = t; e < 32 * 9; e += 256)
        if (cb + e / 9 < C) partial[(long long)blockIdx.x * C * 9 + cb * 9 + e] = red[e / 9][e % 9];
}

}  // namespace seera

using namespace seera;

extern "C" {

// H, W: the low-resolution size.
int seera_unpool2_convT_fusable(int N, int Cin, int H, int W, int Cout, int KH, int KW, int sh, int sw, int ph, int pw) {
    return N >= 1 && Cin >= 1 && Cin <= UC_CMAX && H >= 1 && W >= 1 && Cout == 1 && KH == 3 && KW == 3 && sh == 1 && sw == 1 && ph == 1 && pw == 1 &&
           (long long)N * Cin * H * W * 4 < (1ll << 31) && !ensure_init() && rt().precision != 0;
}

int seera_unpool2_convT_bias_act_fwd(const float *x, const float *w, const float *bias, float *y, int N, int Cin, int H, int W, int act) {
    SEERA_ENSURE();
    if (!x || !w || !y || !seera_unpool2_convT_fusable(N, Cin, H, W, 1, 3, 3, 1, 1, 1, 1)) return fail(SEERA_E_ARG, "unpool2_convT_fwd: bad argument");
    if (reinterpret_cast<uintptr_t>(y) & 7) return fail(SEERA_E_ARG, "unpool2_convT_fwd: output not 8-byte aligned");
    const int segs = (W + 31) / 32, bands = (H + FBAND - 1) / FBAND, items = N * bands * segs, chunks = (Cin + FCH - 1) / FCH;
    const size_t smem = ((size_t)FSTAGES * FCH * FROWS * FPITCH + (size_t)Cin * 16) * sizeof(float);
    const int cap = rt().sm_count * 4;                    // resident blocks
    const int vec = (W & 3) == 0 && aligned16(x);
    cudaError_t e = allow_smem((const void *)unpool_convt_fwd_kernel, smem);
    if (e != cudaSuccess) return check_cuda(e, "unpool2_convT_fwd");
    profile_begin();
    unpool_convt_fwd_kernel<<<items < cap ? items : cap, 256, smem, rt().stream>>>(x, w, bias, y, Cin, H, W, act, segs, bands, items, vec,
                                                                               fast_div(segs), fast_div(bands), fast_div(chunks));
    SEERA_LAUNCH_CHECK("unpool2_convT_fwd");
    profile_end(2.0 * N * 4 * H * W * (double)Cin * 9, "unpool2_convT_fwd");
    return SEERA_OK;
}

// y: the layer output (2H x 2W), g its gradient; dx (may be null) at the low resolution.
int seera_unpool2_convT_act_bwd(const float *w, const float *x, const float *y, const float *g, float *dx, float *dw, float *db, int N, int Cin,
                                int H, int W, int act) {
    SEERA_ENSURE();
    if (!x || !w || !g || !dw || !db || (act != SEERA_ACT_NONE && !y) || !seera_unpool2_convT_fusable(N, Cin, H, W, 1, 3, 3, 1, 1, 1, 1))
        return fail(SEERA_E_ARG, "unpool2_convT_bwd: bad argument");
    const int n_out = N * 4 * H * W;
    float *dz = (float *)scratch_alloc((size_t)n_out * sizeof(float));
    if (!dz) return SEERA_E_OOM;
    int s = seera_act_bias_bwd(g, y, dz, db, n_out, 1, 4 * H * W, act);
    const int chunks = (Cin + 31) / 32, segs = (W + 31) / 32, bands = (H + BROWS - 1) / BROWS, items = N * bands * segs;
    int blocks = rt().sm_count * 2 / chunks;              // resident blocks
    if (blocks > (items + 1) / 2) blocks = (items + 1) / 2;
    if (blocks < 1) blocks = 1;
    float *partial = s ? nullptr : (float *)scratch_alloc((size_t)blocks * Cin * 9 * sizeof(float));
    if (!s && !partial) s = SEERA_E_OOM;
    if (!s) {
        profile_begin();
        const size_t smem = (size_t)BSTAGES * BSTAGE * sizeof(float);
        cudaError_t e = allow_smem((const void *)unpool_convt_bwd_kernel, smem);
        if (e == cudaSuccess)
            unpool_convt_bwd_kernel<<<dim3((unsigned)blocks, (unsigned)chunks), 256, smem, rt().stream>>>(
                x, w, dz, dx, partial, Cin, H, W, segs, bands, items, (W & 3) == 0 && aligned16(x) && aligned16(dz), fast_div(segs), fast_div(bands));
        count_launch();
        launch_sum_splits(partial, dw, Cin * 9, blocks, rt().stream);
        if (e == cudaSuccess) e = cudaGetLastError();
        profile_end(2.0 * N * 4 * H * W * (double)Cin * 9 * (dx ? 2 : 1), dx ? "unpool2_convT_bwd(dX+dW)" : "unpool2_convT_bwd(dW)");
        if (e != cudaSuccess) s = check_cuda(e, "unpool2_convT_bwd");
    }
    if (partial) scratch_free(partial);
    scratch_free(dz);
    return s;
}

}  // extern "C"
