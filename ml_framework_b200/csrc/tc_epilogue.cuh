// Accumulator drain shared by the tensor-core kernels: one warp moves its 32 TMEM lanes (rows) x `ncols`
// columns to global memory through the output functor.
#pragma once
#include "tc_ptx.cuh"

namespace seera {

// Staging of one epilogue warp: a 32 x 32 tile of floats whose 16-byte pieces are permuted inside their row by the row number, so
// that lanes that hold rows and lanes that hold columns both move 16 bytes per access without bank conflicts and without padding
// (eight warps of it leave room for three 64 KB pipeline stages beside them; padded rows would leave two).
constexpr int EPI_WARP_SMEM = 32 * 32 * 4;
__device__ __forceinline__ float4 *epi_piece(float *stage, int row, int piece) {
    return reinterpret_cast<float4 *>(stage + row * 32 + ((piece ^ (row & 7)) << 2));
}
// lane = row: its 32 columns into the staging tile
__device__ __forceinline__ void epi_put_row(float *stage, int lane, const float *v) {
#pragma unroll
    for (int k = 0; k < 8; k++) *epi_piece(stage, lane, k) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
}

// taddr: TMEM address of (first lane of this warp's quarter, column c_begin); row_base: global row of lane 0.  The warp takes the
// 32-column chunks c_begin, c_begin + c_step, ... below c_end; `release` is called once, when the last of them has left TMEM.
// Outputs contiguous along m (NCHW pixels, transposed dense) are stored straight from registers: lanes hold
// consecutive rows, so each store instruction is one coalesced line.  Outputs contiguous along n (row-major
// C, split-K partials; nstride() is 1) go through the staging tile so that eight lanes store the 128 bytes of a row's chunk.
// Per-column bias and activation applied on the way out (bias == nullptr and act == 0: plain store).  Split-K partial
// sums are stored untouched; their reduction applies the same transform.
__device__ __forceinline__ float epilogue_act(float z, int act) {
    switch (act) {
        case 1: return z > 0.f ? z : 0.f;               // SEERA_ACT_RELU
        case 2: return 1.f / (1.f + expf(-z));          // SEERA_ACT_SIGMOID
        case 3: return tanhf(z);                        // SEERA_ACT_TANH
        default: return z;
    }
}

// Output functors that also keep 16-bit copies of what they store expose copy_out4(m, n, 4 values); the others do not.
template <class CS>
__device__ __forceinline__ auto maybe_copy_out4(const CS &cs, int m, int n, const float4 &v, int) -> decltype(cs.copy_out4(m, n, v), void()) {
    cs.copy_out4(m, n, v);
}
template <class CS>
__device__ __forceinline__ void maybe_copy_out4(const CS &, int, int, const float4 &, long) {}

// ... or copy_row(m, n0, 32 values) where lanes hold rows.
template <class CS>
__device__ __forceinline__ auto maybe_copy_row(const CS &cs, int m, int n0, const float *v, int) -> decltype(cs.copy_row(m, n0, v), void()) {
    cs.copy_row(m, n0, v);
}
template <class CS>
__device__ __forceinline__ void maybe_copy_row(const CS &, int, int, const float *, long) {}

struct NoRelease { __device__ void operator()() const {} };

template <class CS, class Release = NoRelease>
__device__ __forceinline__ void drain_accumulator(uint32_t taddr, int row_base, int col_base, int c_begin, int c_end, int c_step,
                                                  int M, int N, const CS &cs, float *partial, long long partial_off,
                                                  float *stage /* EPI_WARP_SMEM bytes, this warp's own */,
                                                  const float *bias = nullptr, int act = 0, float scale = 1.f,
                                                  int nacc = 1, uint32_t acc_stride = 0 /* partial accumulators to add up */,
                                                  const Release &release = Release()) {
    const int lane = threadIdx.x & 31;
    const bool transpose = partial != nullptr || !CS::kMContiguous;
    const bool fuse = !partial && (bias || act);
    if (partial) scale = 1.f;                      // the reduction of the partial sums applies it
    if (!transpose) {
        const long long sn = cs.nstride();
        const int m_own = row_base + lane;         // this lane owns row m; its address part is computed once, not per element
        float *own = m_own < M ? cs.row(m_own) : nullptr;
        for (int c = c_begin; c < c_end; c += c_step) {
            float v[32];
            tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
            if (c + c_step >= c_end) release();
            if (scale != 1.f) {            // operand copies carried power-of-two factors: take them out (exact)
#pragma unroll
                for (int j = 0; j < 32; j++) v[j] *= scale;
            }
            if (fuse) {            // lanes hold rows here: the 32 column biases go through this warp's staging buffer
                const int n = col_base + c + lane;
                __syncwarp();
                stage[lane] = (bias && n < N) ? __ldg(bias + n) : 0.f;
                __syncwarp();
                if (act == 1) {    // relu: the common case without a switch per value
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b4 = *reinterpret_cast<const float4 *>(stage + j);
                        float z;
                        z = v[j] + b4.x; v[j] = z > 0.f ? z : 0.f;
                        z = v[j + 1] + b4.y; v[j + 1] = z > 0.f ? z : 0.f;
                        z = v[j + 2] + b4.z; v[j + 2] = z > 0.f ? z : 0.f;
                        z = v[j + 3] + b4.w; v[j + 3] = z > 0.f ? z : 0.f;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 b4 = *reinterpret_cast<const float4 *>(stage + j);
                        v[j] = epilogue_act(v[j] + b4.x, act); v[j + 1] = epilogue_act(v[j + 1] + b4.y, act);
                        v[j + 2] = epilogue_act(v[j + 2] + b4.z, act); v[j + 3] = epilogue_act(v[j + 3] + b4.w, act);
                    }
                }
            }
            if (own) {
                float *q = own + (long long)(col_base + c) * sn;       // one pointer, advanced by the column stride
                const int nvalid = N - (col_base + c);
                if (nvalid >= 32) {
#pragma unroll
                    for (int j = 0; j < 32; j++) { *q = v[j]; q += sn; }
                } else {
#pragma unroll
                    for (int j = 0; j < 32; j++) {
                        if (j < nvalid) *q = v[j];
                        q += sn;
                    }
                }
                maybe_copy_row(cs, m_own, col_base + c, v, 0);
            }
        }
    } else {
        // Once through the staging tile a lane holds four consecutive columns (piece `k` of the chunk) of rows rs, rs + 4, ...
        const int k = lane & 7, rs = lane >> 3;
        const float *row0 = partial ? partial + partial_off + (long long)row_base * N : cs.row(row_base);
        const long long ld = partial ? (long long)N : cs.row(row_base + 1) - cs.row(row_base);
        const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(row0) & 15) == 0;
        const int rows = min(32, M - row_base);
        for (int c = c_begin; c < c_end; c += c_step) {
            float v[32];
            tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
            if (c + c_step >= c_end) release();
            __syncwarp();                          // the previous chunk has been read out
            epi_put_row(stage, lane, v);
            __syncwarp();
            const int n = col_base + c + 4 * k, nvalid = N - n;
            float b[4] = {0.f, 0.f, 0.f, 0.f};
            if (fuse && bias) {
#pragma unroll
                for (int j = 0; j < 4; j++) b[j] = j < nvalid ? __ldg(bias + n + j) : 0.f;
            }
            float *q = const_cast<float *>(row0) + (long long)rs * ld + n;
#pragma unroll
            for (int i = 0; i < 8; i++, q += 4 * ld) {
                const int r = 4 * i + rs;
                float4 x = *epi_piece(stage, r, k);
                x.x *= scale; x.y *= scale; x.z *= scale; x.w *= scale;
                if (fuse) {
                    x.x += b[0]; x.y += b[1]; x.z += b[2]; x.w += b[3];
                    if (act == 1) {
                        x.x = x.x > 0.f ? x.x : 0.f; x.y = x.y > 0.f ? x.y : 0.f; x.z = x.z > 0.f ? x.z : 0.f; x.w = x.w > 0.f ? x.w : 0.f;
                    } else {
                        x.x = epilogue_act(x.x, act); x.y = epilogue_act(x.y, act); x.z = epilogue_act(x.z, act); x.w = epilogue_act(x.w, act);
                    }
                }
                if (r < rows && nvalid > 0) {
                    if (vec && nvalid >= 4) {
                        *reinterpret_cast<float4 *>(q) = x;
                    } else {
                        q[0] = x.x;
                        if (nvalid > 1) q[1] = x.y;
                        if (nvalid > 2) q[2] = x.z;
                        if (nvalid > 3) q[3] = x.w;
                    }
                    if (!partial) {
                        if (nvalid < 4) { x.w = 0.f; if (nvalid < 3) x.z = 0.f; if (nvalid < 2) x.y = 0.f; }
                        maybe_copy_out4(cs, row_base + r, n, x, 0);
                    }
                }
            }
        }
    }
}

// ---- epilogue with a 2x2 / stride-2 max-pool folded in --------------------------------------------------------------
// The accumulator rows are output pixels of y = act(conv + bias); instead of storing y, each warp reduces the 2x2
// windows that lie inside its 32 rows with shuffles and stores only the pooled value, the window-local argmax (scan
// order (0,0), (0,1), (1,0), (1,1), strict comparison: the first maximum wins, as in cuda_maxpool_fwd) and the bf16
// channels-last copies of the pooled tensor for the next convolution.  y itself never reaches HBM.
// Row order: raster (row = pixel index; needs OW a power of two <= 16 so that a window's rows are lanes l, l^1, l^OW,
// l^(OW+1)) or window-major (row = 4 * window + position; partners are lanes l^1, l^2, l^3).
struct PoolOut {
    float *pooled;                 // [NB, F, OH/2, OW/2]
    int *mask;                     // same shape
    __nv_bfloat16 *copy[3];        // [NB, (OH/2)*(OW/2), Cp] or null
    int ns, Cp;
    Enc enc;                       // encoding of the copies
    int P, OW;                     // pixels per image and width of y
    int window_major;
    FastDiv by_P, by_OW, by_Pq;    // set by pool_out_geometry
};
inline void pool_out_geometry(PoolOut &po, int P, int OW, int window_major) {
    po.P = P; po.OW = OW; po.window_major = window_major;
    po.by_P = fast_div(P); po.by_OW = fast_div(OW); po.by_Pq = fast_div(P >> 2);
}

template <class Release = NoRelease>
__device__ __forceinline__ void drain_accumulator_pooled(uint32_t taddr, int row_base, int col_base, int c_begin, int c_end, int c_step,
                                                         int M, int N, const float *bias, int act, const PoolOut &po, float *stage,
                                                         float scale = 1.f, int nacc = 1, uint32_t acc_stride = 0,
                                                         const Release &release = Release()) {
    // The warp's 32 rows hold exactly 8 windows.  Each 32-column chunk goes through the staging tile so that a lane holds
    // EIGHT CHANNELS of ONE window: it reads the window's four rows as 16-byte pieces, applies bias and activation, takes the
    // maximum in registers, and writes the channels-last copies as one 16-byte store each (a lane per column would write them two
    // bytes at a time: with that epilogue a 128-column launch took twice the time of its main loop).
    const int lane = threadIdx.x & 31, w = lane >> 2, cg = lane & 3;
    const int Pq = po.P >> 2, d2 = po.window_major ? 2 : po.OW;
    // first row of the window inside the warp's rows, its image and its index inside the image
    int r0, img, wrem;
    if (po.window_major) {
        r0 = 4 * w;
        const int wi = (row_base >> 2) + w;
        img = po.by_Pq.div(wi); wrem = wi - img * Pq;
    } else {
        const int OWq = po.OW >> 1, wr = w / OWq, wc = w - wr * OWq;      // window row / column inside the warp's rows
        r0 = 2 * wr * po.OW + 2 * wc;
        const int m = row_base + r0, rem0 = po.by_P.div(m), rem = m - rem0 * po.P, oh = po.by_OW.div(rem), ow = rem - oh * po.OW;
        img = rem0; wrem = (oh >> 1) * OWq + (ow >> 1);
    }
    const bool live = row_base + r0 < M;
    const long long plane0 = (long long)img * N * Pq + wrem, pix0 = ((long long)img * Pq + wrem) * po.Cp;
    for (int c = c_begin; c < c_end; c += c_step) {
        float v[32];
        tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
        if (c + c_step >= c_end) release();
        __syncwarp();                                               // the previous chunk has been read out
        epi_put_row(stage, lane, v);
        __syncwarp();
        const int n0 = col_base + c + 8 * cg;
        float mx[8];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            // odd windows take their two pieces in the other order: the eight lanes of a phase then read eight different pieces
            const int hh = h ^ (w & 1), n = n0 + 4 * hh;
            float a[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 x = *epi_piece(stage, r0 + (i & 1) + (i >> 1) * d2, 2 * cg + hh);
                a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float b = (bias && n + j < N) ? __ldg(bias + n + j) : 0.f;
                float m = -3.402823466e+38f; int id = 0;           // -FLT_MAX, strict comparisons: the first maximum wins
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float z = a[i][j] * scale + b;
                    z = act == 1 ? (z > 0.f ? z : 0.f) : epilogue_act(z, act);
                    if (z > m) { m = z; id = i; }
                }
                if (live && n + j < N) {
                    const long long q = plane0 + (long long)(n + j) * Pq;
                    po.pooled[q] = m;
                    po.mask[q] = id;
                }
                mx[4 * h + j] = n + j < N ? m : 0.f;
            }
        }
        if (po.copy[0] && live && n0 < po.Cp) {                     // channels-last copies: four lanes write a window's 32 channels
            float o8[8];
#pragma unroll
            for (int j = 0; j < 4; j++) { o8[j] = (w & 1) ? mx[4 + j] : mx[j]; o8[4 + j] = (w & 1) ? mx[j] : mx[4 + j]; }
            const long long o = pix0 + n0;
            store_split8_n(o8, po.ns, po.enc, po.copy[0] + o, po.copy[1] + o, po.copy[2] + o);
        }
    }
}

}  // namespace seera
