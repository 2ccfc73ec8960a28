// Weight and bias gradient of a 3 x 3 convolution with one to four input channels (the first layer of an image network, the last
// of an autoencoder), exact fp32 on the CUDA cores; a layer of little work with more channels goes in groups of four (conv_small.cu).
//
// The gradient arrives through a 2x2 / stride-2 max-pool (pooled gradient, argmax index, pooled output) or at full resolution (with
// the layer output); activation slope and pool routing are applied on the way in.  A UNIT is a 2 x 2 block of output pixels with the
// (3 + stride)^2 input values per channel that its four patches share.  A lane owns a filter and keeps its row of dW in
// registers, twice: the two halves of a packed multiply-add take the same product of two neighbouring units.  A block walks tiles of 32
// units through a ring of cp.async stages:
//   * inputs [unit pair][value][2], so that 16 bytes are two values of both units, read by all lanes at once;
//   * gradients [filter][unit], which a lane reads along its own row;
// and per unit pair, channel and input row the values go against the four positions' gradients: 4 x 9 x C packed multiply-adds for 8 x C
// 16-byte reads.  With the pool three of four gradients are zero; multiplying by them is still cheaper than fetching each
// lane's own patch (per lane and position that is as many bytes from shared memory, which is what bounds it).
// A pass over the inputs and gradients is all the memory traffic there is; what a block issues is a third copies and two thirds
// products, so copies go 16 bytes at a time where the gradient's rows allow it.
// Each block writes one partial sum per filter and tap, added in block order: the result does not depend on scheduling.
//
// Against the tensor-core form (first_tc_wgrad_kernel, bound by the warps that gather, split and swizzle patches and gradients), which
// keeps the other short patches: 64 filters, 3 channels, 512 images of 32 x 32 through the pool 70 -> 61 us; 8 filters, 1 channel, 64 of
// 28 x 28 through the pool 10 -> 3.2 us; 32 filters at full resolution, 3 channels, 128 of 32 x 32 33 -> 23 us, 1 channel, stride 2,
// 256 of 64 x 64 52 -> 25 us.
#include "conv_first.cuh"
#include "internal.h"

namespace seera {

constexpr int DW_UNITS = 32;

__device__ __forceinline__ void dw_cp4(uint32_t dst, const void *src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(take ? 4 : 0) : "memory");
}
__device__ __forceinline__ void dw_cp8(uint32_t dst, const void *src, bool take) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(take ? 8 : 0) : "memory");
}

__device__ __forceinline__ void dw_cp16(uint32_t dst, const void *src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(take ? 16 : 0) : "memory");
}

template <int C, int ST, int FL, bool POOLED>
struct DwShape {
    static constexpr int K = 9 * C, KP = (K + 1 + 3) / 4 * 4;       // taps, and columns of a partial sum: taps, bias, padding
    static constexpr int ROWS = 3 + ST, COLS = (3 + ST + 1) / 2 * 2, NRAW = C * ROWS * (3 + ST);     // rows padded to an even length
    static constexpr int PAIR = 2 * C * ROWS * COLS + 4;            // floats of a unit pair's inputs
    // floats of a filter's row: one per unit and array through the pool; else per unit pair two pixel rows of four pixels
    static constexpr int VROW = POOLED ? DW_UNITS + 4 : 4 * DW_UNITS + 4;
    static constexpr int ARRAYS = POOLED ? 3 : 2;
    // floats of a stage that holds the gradient rows of `vf` filters
    __host__ __device__ static constexpr int stage(int vf) { return (DW_UNITS / 2) * PAIR + ARRAYS * vf * VROW; }
    static constexpr int RED = 8 * 32 * KP;
};

template <int C, int ST, int FL, bool POOLED>
__global__ void __launch_bounds__(256, 2) first_dw_kernel(const float *__restrict__ X, DzSource src, float *__restrict__ partial, FirstGeom g,
                                                          int units, int ntiles, int stages, int vf, FastDiv by_units, FastDiv by_cols) {
    // blockIdx.z: group of C of the g.C input channels
    using Sh = DwShape<C, ST, FL, POOLED>;
    constexpr int KP = Sh::KP, K = Sh::K, VROW = Sh::VROW, ROWS = Sh::ROWS, COLS = Sh::COLS, SUB = 32 / FL;
    extern __shared__ __align__(16) float sm[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c_first = blockIdx.z * C, c_here = min(C, g.C - c_first);
    const int f0 = blockIdx.y * FIRST_FC, FC = min(vf, g.F - f0), STAGE = Sh::stage(vf);
    const int plane = g.H * g.W, P = g.OH * g.OW, Pq = P >> 2, ucols = by_cols.d;
    const bool sloped = src.act != SEERA_ACT_NONE;
    const float *pa = POOLED ? src.gp : (src.dz ? src.dz : src.g), *pb = POOLED ? src.yp : src.y;
    // how many consecutive values of a gradient row one copy takes
    const uintptr_t at_all = reinterpret_cast<uintptr_t>(pa) | (sloped ? reinterpret_cast<uintptr_t>(pb) : 0) |
                             (POOLED ? reinterpret_cast<uintptr_t>(src.mask) : 0);
    const int run = POOLED ? ((Pq & 3) == 0 && (at_all & 15) == 0 ? 4 : 1)
                           : ((g.OW & 3) == 0 && (at_all & 15) == 0 ? 4 : ((g.OW & 1) == 0 && (at_all & 7) == 0 ? 2 : 1));

    // (lanes beyond the last filter compute on whatever their rows hold; their sums go nowhere)
    auto request = [&](int tile, int s) {
        const int u = tile * DW_UNITS + lane;
        const bool live = u < units;
        const int ul = live ? u : 0, n = by_units.div(ul), rem = ul - n * by_units.d, ur = by_cols.div(rem), uc = rem - ur * ucols;
        const int oh = 2 * ur, ow = 2 * uc, ih0 = oh * ST - g.ph, iw0 = ow * ST - g.pw;
        const float *xn = X + ((long long)n * g.C + c_first) * plane;
        float *stage = sm + s * STAGE;
        const uint32_t d0 = (uint32_t)__cvta_generic_to_shared(stage + (lane >> 1) * Sh::PAIR + (lane & 1));
        bool colok[3 + ST];
#pragma unroll
        for (int j = 0; j < 3 + ST; j++) colok[j] = (unsigned)(iw0 + j) < (unsigned)g.W;
#pragma unroll
        for (int r0 = 0; r0 < C * ROWS; r0 += 8) {
            const int rr = r0 + warp, c = rr / ROWS, i = rr - c * ROWS;
            if (rr < C * ROWS) {
                const bool rowok = live && c < c_here && (unsigned)(ih0 + i) < (unsigned)g.H;
                const int off = c * plane + (ih0 + i) * g.W + iw0;
#pragma unroll
                for (int j = 0; j < 3 + ST; j++) {
                    const bool in = rowok && colok[j];
                    dw_cp4(d0 + 8u * (uint32_t)(rr * COLS + j), xn + (in ? off + j : 0), in);
                }
            }
        }
        // gradients; a lane without a unit copies nothing from the address of unit 0
        const uint32_t v0 = (uint32_t)__cvta_generic_to_shared(stage + (DW_UNITS / 2) * Sh::PAIR);
        const uint32_t ARR = 4u * (uint32_t)(vf * VROW);
        if (POOLED && run == 4) {                // thread = (four windows, filter)
            const int q = t & 7, v = tile * DW_UNITS + 4 * q;
            const bool lv = v < units;
            const int vl = lv ? v : 0, vn = by_units.div(vl);
            const long long at = ((long long)vn * g.F + f0) * Pq + (vl - vn * by_units.d);
            for (int f = t >> 3; f < FC; f += 32) {
                const uint32_t d = v0 + 4u * (uint32_t)(f * VROW + 4 * q);
                const long long o = at + (long long)f * Pq;
                dw_cp16(d, pa + o, lv);
                dw_cp16(d + ARR, src.mask + o, lv);
                if (sloped) dw_cp16(d + 2 * ARR, pb + o, lv);
            }
        } else if (POOLED) {
            const long long at = ((long long)n * g.F + f0) * Pq + rem;
            for (int f = warp; f < FC; f += 8) {
                const uint32_t d = v0 + 4u * (uint32_t)(f * VROW + lane);
                const long long o = at + (long long)f * Pq;
                dw_cp4(d, pa + o, live);
                dw_cp4(d + ARR, src.mask + o, live);
                if (sloped) dw_cp4(d + 2 * ARR, pb + o, live);
            }
        } else if (run == 4) {                   // thread = (unit pair, filter): four pixels of two rows
            const int q = t & 15, v = tile * DW_UNITS + 2 * q;
            const bool lv = v < units;
            const int vl = lv ? v : 0, vn = by_units.div(vl), vr = vl - vn * by_units.d, vu = by_cols.div(vr), vc = vr - vu * ucols;
            const bool l1 = lv && 2 * vu + 1 < g.OH;
            const long long at = ((long long)vn * g.F + f0) * P + (long long)(2 * vu) * g.OW + 2 * vc;
            const int down = l1 ? g.OW : 0;
            for (int f = t >> 4; f < FC; f += 16) {
                const uint32_t d = v0 + 4u * (uint32_t)(f * VROW + 8 * q);
                const long long o = at + (long long)f * P;
                dw_cp16(d, pa + o, lv);
                dw_cp16(d + 16, pa + o + down, l1);
                if (sloped) { dw_cp16(d + ARR, pb + o, lv); dw_cp16(d + ARR + 16, pb + o + down, l1); }
            }
        } else {
            const long long at = ((long long)n * g.F + f0) * P + (long long)oh * g.OW + ow;
            const bool r1 = live && oh + 1 < g.OH, c1 = ow + 1 < g.OW;
            const int down = r1 ? g.OW : 0, right = c1 ? 1 : 0;
            for (int f = warp; f < FC; f += 8) {
                const uint32_t d = v0 + 4u * (uint32_t)(f * VROW + 8 * (lane >> 1) + 2 * (lane & 1));
                const long long o = at + (long long)f * P;
                for (int k = 0; k < (sloped ? 2 : 1); k++) {
                    const float *p = (k ? pb : pa) + o;
                    const uint32_t dk = d + (k ? ARR : 0u);
                    if (run == 2) {
                        dw_cp8(dk, p, live);
                        dw_cp8(dk + 16, p + down, r1);
                    } else {
                        dw_cp4(dk, p, live);
                        dw_cp4(dk + 4, p + right, live && c1);
                        dw_cp4(dk + 16, p + down, r1);
                        dw_cp4(dk + 20, p + down + right, r1 && c1);
                    }
                }
            }
        }
    };

    const int groups = FL < 32 ? 1 : (FC + 31) / 32, grp = warp % groups, p_first = warp / groups, p_step = 8 / groups;
    const int sub = lane / FL, fl = grp * 32 + lane % FL;
    f32x2 acc[K], accb = 0ull;
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = 0ull;
    auto slope = [&](float v, float y) {
        switch (src.act) {
            case SEERA_ACT_RELU: return y > 0.f ? v : 0.f;
            case SEERA_ACT_SIGMOID: return v * (y * (1.f - y));
            case SEERA_ACT_TANH: return v * (1.f - y * y);
            default: return v;
        }
    };

    for (int s = 0; s < stages - 1; s++) {
        if ((int)(blockIdx.x + s * gridDim.x) < ntiles) request(blockIdx.x + s * gridDim.x, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int cur = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        if (stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncthreads();                         // this tile has landed for everyone, and the stage refilled next has been read out
        const int ahead = tile + (stages - 1) * (int)gridDim.x, slot = cur == 0 ? stages - 1 : cur - 1;
        if (ahead < ntiles) request(ahead, slot);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *stage = sm + cur * STAGE, *vrow = stage + (DW_UNITS / 2) * Sh::PAIR + fl * VROW;
        for (int i = p_first; i < DW_UNITS / 2 / SUB; i += p_step) {
            const int pr = i * SUB + sub;
            f32x2 v[4];                          // gradients of the four positions, of both units
            if (POOLED) {
                const float2 gq = *reinterpret_cast<const float2 *>(vrow + 2 * pr);
                const int2 m = *reinterpret_cast<const int2 *>(vrow + vf * VROW + 2 * pr);
                float a = gq.x, b = gq.y;
                if (sloped) {
                    const float2 y = *reinterpret_cast<const float2 *>(vrow + 2 * vf * VROW + 2 * pr);
                    a = slope(a, y.x); b = slope(b, y.y);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = pack2(m.x == q ? a : 0.f, m.y == q ? b : 0.f);
                accb = add2(accb, pack2((unsigned)m.x < 4u ? a : 0.f, (unsigned)m.y < 4u ? b : 0.f));
            } else {
                const float4 r0 = *reinterpret_cast<const float4 *>(vrow + 8 * pr), r1 = *reinterpret_cast<const float4 *>(vrow + 8 * pr + 4);
                float a[4] = {r0.x, r0.y, r1.x, r1.y}, b[4] = {r0.z, r0.w, r1.z, r1.w};
                if (sloped) {
                    const float4 y0 = *reinterpret_cast<const float4 *>(vrow + vf * VROW + 8 * pr);
                    const float4 y1 = *reinterpret_cast<const float4 *>(vrow + vf * VROW + 8 * pr + 4);
                    a[0] = slope(a[0], y0.x); a[1] = slope(a[1], y0.y); a[2] = slope(a[2], y1.x); a[3] = slope(a[3], y1.y);
                    b[0] = slope(b[0], y0.z); b[1] = slope(b[1], y0.w); b[2] = slope(b[2], y1.z); b[3] = slope(b[3], y1.w);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) { v[q] = pack2(a[q], b[q]); accb = add2(accb, v[q]); }
            }
            const float *in = stage + pr * Sh::PAIR;
#pragma unroll
            for (int c = 0; c < C; c++)
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    f32x2 row[COLS];
#pragma unroll
                    for (int j = 0; j < COLS; j += 2) {
                        const ulonglong2 x2 = *reinterpret_cast<const ulonglong2 *>(in + 2 * ((c * ROWS + r) * COLS + j));
                        row[j] = x2.x; row[j + 1] = x2.y;
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const int tr = r - (q >> 1) * ST;            // tap row of this input row at position q
                        if (tr < 0 || tr > 2) continue;
#pragma unroll
                        for (int ts = 0; ts < 3; ts++)
                            acc[c * 9 + tr * 3 + ts] = ffma2(row[ts + (q & 1) * ST], v[q], acc[c * 9 + tr * 3 + ts]);
                    }
                }
        }
        if (++cur == stages) cur = 0;
    }
    // both units of a pair, lanes of one filter, then the warps of one group, in a fixed order
    __syncthreads();
    float *red = sm + (size_t)warp * 32 * KP;
#pragma unroll
    for (int k = 0; k <= K; k++) {
        float lo, hi;
        unpack2(k < K ? acc[k] : accb, lo, hi);
        lo += hi;
#pragma unroll
        for (int o = FL; o < 32; o <<= 1) lo += __shfl_xor_sync(0xffffffffu, lo, o);
        red[k * 32 + lane] = lo;                   // [column][lane]
    }
    __syncthreads();
    float *out = partial + (((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) * (FIRST_FC * KP);
    for (int e = t; e < FC * KP; e += 256) {
        const int f = e / KP, k = e - f * KP;
        float s = 0.f;
        if (k <= K)
            for (int w = f >> 5; w < 8; w += groups) s += sm[((size_t)w * KP + k) * 32 + (f & 31)];
        out[f * KP + k] = s;
    }
}

bool first_dw_applies(const FirstGeom &g, const DzSource &src) {
    // a pooled gradient whose activation needs the layer output itself goes to the other kernels
    if (src.gp && ((src.act != SEERA_ACT_NONE && !src.yp) || (g.OH & 1) || (g.OW & 1))) return false;
    return g.R == 3 && g.S == 3 && g.C <= 4 && g.sh == g.sw && g.sh <= 2 && (long long)g.NB * (g.OH + 1) * (g.OW + 1) < (1ll << 31) - 64 &&
           (long long)g.C * g.H * g.W < (1ll << 30);
}

struct DwCall {
    const float *X; const DzSource *src; float *dW, *dbias; const FirstGeom *g; const char *name;
};
template <int C, int ST, int FL, bool POOLED>
static int dw_launch(const DwCall &a) {
    using Sh = DwShape<C, ST, FL, POOLED>;
    const FirstGeom &g = *a.g;
    const int ucols = (g.OW + 1) / 2, per_image = (g.OH + 1) / 2 * ucols, units = g.NB * per_image;
    const int ntiles = (units + DW_UNITS - 1) / DW_UNITS, chunks = (g.F + FIRST_FC - 1) / FIRST_FC;
    // stages: up to four, as many as leave room for two blocks on an SM, but at least two
    const int vf = FL < 32 ? FL : (g.F <= 32 ? 32 : FIRST_FC);
    const size_t stage_bytes = Sh::stage(vf) * sizeof(float), red_bytes = Sh::RED * sizeof(float);
    int stages = (int)(112 * 1024 / stage_bytes);
    if (stages > 4) stages = 4;
    if (stages < 2) stages = 2;
    const size_t smem = stages * stage_bytes > red_bytes ? stages * stage_bytes : red_bytes;
    const int per_sm = smem <= 112 * 1024 ? 2 : 1;
    const int cgroups = (g.C + C - 1) / C;
    int nblocks = rt().sm_count * per_sm / (chunks * cgroups);
    if (nblocks > (ntiles + 1) / 2) nblocks = (ntiles + 1) / 2;      // a block with one tile is all start and end
    if (nblocks < 1) nblocks = 1;
    float *partial = (float *)scratch_alloc((size_t)cgroups * chunks * nblocks * FIRST_FC * Sh::KP * sizeof(float));
    if (!partial) return SEERA_E_OOM;
    cudaStream_t st = rt().stream;
    profile_begin();
    auto kern = first_dw_kernel<C, ST, FL, POOLED>;
    cudaError_t e = allow_smem((const void *)kern, smem);
    if (e == cudaSuccess) {
        kern<<<dim3((unsigned)nblocks, (unsigned)chunks, (unsigned)cgroups), 256, smem, st>>>(a.X, *a.src, partial, g, units, ntiles, stages, vf, fast_div(per_image),
                                                                         fast_div(ucols));
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        first_wgrad_reduce(partial, a.dW, a.dbias, g.F, g.K, Sh::K, Sh::KP, nblocks, st);
        e = cudaGetLastError();
    }
    profile_end(2.0 * g.NB * g.OH * g.OW * (double)g.F * g.K, a.name);
    scratch_free(partial);
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, a.name);
}
template <int C, int ST>
static int dw_pick(const DwCall &a) {
    const int F = a.g->F;
    if (a.src->gp) return F <= 8 ? dw_launch<C, ST, 8, true>(a) : F <= 16 ? dw_launch<C, ST, 16, true>(a) : dw_launch<C, ST, 32, true>(a);
    return F <= 8 ? dw_launch<C, ST, 8, false>(a) : F <= 16 ? dw_launch<C, ST, 16, false>(a) : dw_launch<C, ST, 32, false>(a);
}

int first_dw(const float *X, const DzSource &src, float *dW, float *dbias, const FirstGeom &g, const char *name) {
    const DwCall a{X, &src, dW, dbias, &g, name};
    if (g.sh == 1) return g.C == 1 ? dw_pick<1, 1>(a) : g.C == 2 ? dw_pick<2, 1>(a) : g.C == 3 ? dw_pick<3, 1>(a) : dw_pick<4, 1>(a);        // more in groups of four
    return g.C == 1 ? dw_pick<1, 2>(a) : g.C == 2 ? dw_pick<2, 2>(a) : g.C == 3 ? dw_pick<3, 2>(a) : dw_pick<4, 2>(a);
}

}  // namespace seera
