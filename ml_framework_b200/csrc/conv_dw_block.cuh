// Weight and bias gradient of 3 x 3 layers on CUDA cores, the block of first_dw_kernel (conv_first_dw.cu says what it does), which the launch
// that forms both gradients of a small layer takes as well (conv_small.cu).
#pragma once
#include "conv_first.cuh"

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

// What a launch works on: units, tiles of 32 units, ring stages, filters whose gradient rows a stage holds; its blocks (tiles, chunks of 64
// filters, groups of C of the g.C input channels) and the shared memory of one.
struct DwArgs {
    const float *X; DzSource src; float *partial; FirstGeom g;
    int units, ntiles, stages, vf;
    FastDiv by_units, by_cols;
    int nblocks, chunks, cgroups;
    size_t smem;
};
// Block (bx, by, bz) of the launch, 256 threads; sm: a.smem bytes.
template <int C, int ST, int FL, bool POOLED>
__device__ __forceinline__ void first_dw_block(const DwArgs &a, int bx, int by, int bz, float *sm) {
    const float *__restrict__ X = a.X;
    float *__restrict__ partial = a.partial;
    const DzSource &src = a.src;
    const FirstGeom &g = a.g;
    const int units = a.units, ntiles = a.ntiles, stages = a.stages, vf = a.vf;
    const FastDiv &by_units = a.by_units, &by_cols = a.by_cols;
    using Sh = DwShape<C, ST, FL, POOLED>;
    constexpr int KP = Sh::KP, K = Sh::K, VROW = Sh::VROW, ROWS = Sh::ROWS, COLS = Sh::COLS, SUB = 32 / FL;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int c_first = bz * C, c_here = min(C, g.C - c_first);
    const int f0 = by * FIRST_FC, FC = min(vf, g.F - f0), STAGE = Sh::stage(vf);
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
        if (bx + s * a.nblocks < ntiles) request(bx + s * a.nblocks, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int cur = 0;
    for (int tile = bx; tile < ntiles; tile += a.nblocks) {
        if (stages == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncthreads();                         // this tile has landed for everyone, and the stage refilled next has been read out
        const int ahead = tile + (stages - 1) * a.nblocks, slot = cur == 0 ? stages - 1 : cur - 1;
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
    float *out = partial + (((long long)bz * a.chunks + by) * a.nblocks + bx) * (FIRST_FC * KP);
    for (int e = t; e < FC * KP; e += 256) {
        const int f = e / KP, k = e - f * KP;
        float s = 0.f;
        if (k <= K)
            for (int w = f >> 5; w < 8; w += groups) s += sm[((size_t)w * KP + k) * 32 + (f & 31)];
        out[f * KP + k] = s;
    }
}


// The launch's geometry, its partial sums not yet allocated.
template <int C, int ST, int FL, bool POOLED>
inline DwArgs dw_args(const float *X, const DzSource &src, const FirstGeom &g) {
    using Sh = DwShape<C, ST, FL, POOLED>;
    DwArgs a{X, src, nullptr, g};
    const int ucols = (g.OW + 1) / 2, per_image = (g.OH + 1) / 2 * ucols;
    a.units = g.NB * per_image;
    a.ntiles = (a.units + DW_UNITS - 1) / DW_UNITS;
    a.chunks = (g.F + FIRST_FC - 1) / FIRST_FC;
    a.by_units = fast_div(per_image); a.by_cols = fast_div(ucols);
    // stages: up to four, as many as leave room for two blocks on an SM, but at least two
    a.vf = FL < 32 ? FL : (g.F <= 32 ? 32 : FIRST_FC);
    const size_t stage_bytes = Sh::stage(a.vf) * sizeof(float), red_bytes = Sh::RED * sizeof(float);
    a.stages = (int)(112 * 1024 / stage_bytes);
    if (a.stages > 4) a.stages = 4;
    if (a.stages < 2) a.stages = 2;
    a.smem = a.stages * stage_bytes > red_bytes ? a.stages * stage_bytes : red_bytes;
    const int per_sm = a.smem <= 112 * 1024 ? 2 : 1;
    a.cgroups = (g.C + C - 1) / C;
    a.nblocks = rt().sm_count * per_sm / (a.chunks * a.cgroups);
    if (a.nblocks > (a.ntiles + 1) / 2) a.nblocks = (a.ntiles + 1) / 2;      // a block with one tile is all start and end
    if (a.nblocks < 1) a.nblocks = 1;
    return a;
}
template <int C>
inline size_t dw_partial_bytes(const DwArgs &a) { return (size_t)a.cgroups * a.chunks * a.nblocks * FIRST_FC * ((9 * C + 1 + 3) / 4 * 4) * sizeof(float); }

}  // namespace seera
