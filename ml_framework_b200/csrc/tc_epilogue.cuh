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

// What bounds an epilogue is the fetch of its own instructions: a warp walks the code of a chunk once or twice per launch, and with every
// loop unrolled and both activation functions expanded per value that code was fetched from L2 for most of the time (ncu: 5 to 7
// warps per issue in the no_instruction stall; a 128 x 128 pooled tile took 3.8 us).  So the loops over a chunk's pieces are
// rolled, ReLU is a select, and the activations with a function call go through one rolled loop over the staging tile.  Dense products
// of a few tiles gain most (100 x 256 x 1024 in six products 10.5 -> 7.2 us, a 1024 x 256 x 512 weight gradient in one 12.5 -> 9.4).
__device__ __forceinline__ float epilogue_act(float z, int act) {
    switch (act) {
        case 1: return z > 0.f ? z : 0.f;               // SEERA_ACT_RELU
        case 2: return 1.f / (1.f + expf(-z));          // SEERA_ACT_SIGMOID
        case 3: return tanhf(z);                        // SEERA_ACT_TANH
        default: return z;
    }
}
// Sigmoid or tanh of a lane's row of the staging tile, in place, with the row's scale and column biases before it.
__device__ __forceinline__ void epi_act_row(float *stage, int lane, const float *bias, int n0, int N, int act, float scale) {
#pragma unroll 1
    for (int e = 0; e < 32; e++) {
        float *p = reinterpret_cast<float *>(epi_piece(stage, lane, e >> 2)) + (e & 3);
        const float b = (bias && n0 + e < N) ? __ldg(bias + n0 + e) : 0.f;
        *p = epilogue_act(*p * scale + b, act);
    }
}

// Output functors that also keep 16-bit copies of what they store expose copy_out4(m, n, 4 values); the others do not.
template <class CS>
__device__ __forceinline__ auto maybe_copy_out4(const CS &cs, int m, int n, const float4 &v, int) -> decltype(cs.copy_out4(m, n, v), void()) {
    cs.copy_out4(m, n, v);
}
template <class CS>
__device__ __forceinline__ void maybe_copy_out4(const CS &, int, int, const float4 &, long) {}

// ... or copies() and copy8(m, n, 8 values) where lanes hold rows.  The chunk goes through the staging tile for it: a lane that wrote its own
// row put 16 bytes into each of 32 lines per store (65536 x 64 x 288 with copies: 27.4 -> 25.3 us); so four lanes write the 64 bytes of a row.
template <class CS>
__device__ __forceinline__ auto maybe_copy_rows(const CS &cs, const float *v, int row_base, int M, int n0, float *stage, int)
    -> decltype(cs.copies(), void()) {
    if (!cs.copies()) return;
    const int lane = threadIdx.x & 31, cg = lane & 3;
    __syncwarp();
    epi_put_row(stage, lane, v);
    __syncwarp();
#pragma unroll 1
    for (int r = lane >> 2; r < 32; r += 8) {
        const float4 x = *epi_piece(stage, r, 2 * cg), y = *epi_piece(stage, r, 2 * cg + 1);
        float o8[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        if (row_base + r < M) cs.copy8(row_base + r, n0 + 8 * cg, o8);
    }
}
template <class CS>
__device__ __forceinline__ void maybe_copy_rows(const CS &, const float *, int, int, int, float *, long) {}

struct NoRelease { __device__ void operator()() const {} };

// ---- one 32 x 32 chunk, lane = row, v = its 32 columns -----------------------------------------------------------------------
// Outputs contiguous along m (NCHW pixels, transposed dense): lanes hold consecutive rows, so each store instruction is one
// coalesced line.  `own` is the address of (row, column 0) or null, `sn` the stride between columns.
template <class CS>
__device__ __forceinline__ void put_chunk_rows(float *v, float *own, long long sn, int row_base, int M, int n0, int N, const CS &cs,
                                               float *stage, const float *bias, int act, float scale) {
    const int lane = threadIdx.x & 31;
    if (act > 1) {
        __syncwarp();
        epi_put_row(stage, lane, v);
        epi_act_row(stage, lane, bias, n0, N, act, scale);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float4 x = *epi_piece(stage, lane, k);
            v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
        }
    } else {
        if (scale != 1.f) {                // operand copies carried power-of-two factors: take them out (exact)
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] *= scale;
        }
        if (bias) {                        // lanes hold rows here: the 32 column biases go through this warp's staging buffer
            __syncwarp();
            stage[lane] = n0 + lane < N ? __ldg(bias + n0 + lane) : 0.f;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const float4 b4 = *reinterpret_cast<const float4 *>(stage + j);
                v[j] += b4.x; v[j + 1] += b4.y; v[j + 2] += b4.z; v[j + 3] += b4.w;
            }
        }
        if (act == 1) {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = v[j] > 0.f ? v[j] : 0.f;
        }
    }
    if (own) {
        float *q = own + (long long)n0 * sn;                   // one pointer, advanced by the column stride
        const int nvalid = N - n0;
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
    }
    maybe_copy_rows(cs, v, row_base, M, n0, stage, 0);
}

// Outputs contiguous along n (row-major C, split-K partials): the chunk goes through the staging tile so that eight lanes store the
// 128 bytes of a row.  `row0` is the address of (first row, column 0), `ld` the pitch, `rows` how many rows are inside.  Partial sums
// are stored as they are (bias null, act 0, scale 1, no copies); their reduction applies the rest.
template <class CS>
__device__ __forceinline__ void put_chunk_columns(const float *v, float *row0, long long ld, int row_base, int rows, int n0, int N, const CS &cs,
                                                  bool copies, float *stage, const float *bias, int act, float scale) {
    const int lane = threadIdx.x & 31, k = lane & 7, rs = lane >> 3;
    const bool vec = (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(row0) & 15) == 0;
    const int n = n0 + 4 * k, nvalid = N - n;
    float b[4] = {0.f, 0.f, 0.f, 0.f};
    if (bias && act <= 1) {
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = j < nvalid ? __ldg(bias + n + j) : 0.f;
    }
    __syncwarp();                                  // the previous chunk has been read out
    epi_put_row(stage, lane, v);
    if (act > 1) { epi_act_row(stage, lane, bias, n0, N, act, scale); scale = 1.f; }
    __syncwarp();
    float *q = row0 + (long long)rs * ld + n;
    const bool relu = act == 1;
#pragma unroll 2
    for (int i = 0; i < 8; i++, q += 4 * ld) {
        const int r = 4 * i + rs;
        float4 x = *epi_piece(stage, r, k);
        x.x = x.x * scale + b[0]; x.y = x.y * scale + b[1]; x.z = x.z * scale + b[2]; x.w = x.w * scale + b[3];
        if (relu) { x.x = x.x > 0.f ? x.x : 0.f; x.y = x.y > 0.f ? x.y : 0.f; x.z = x.z > 0.f ? x.z : 0.f; x.w = x.w > 0.f ? x.w : 0.f; }
        if (r < rows && nvalid > 0) {
            if (vec && nvalid >= 4) {
                *reinterpret_cast<float4 *>(q) = x;
            } else {
                q[0] = x.x;
                if (nvalid > 1) q[1] = x.y;
                if (nvalid > 2) q[2] = x.z;
                if (nvalid > 3) q[3] = x.w;
            }
            if (copies) {
                if (nvalid < 4) { x.w = 0.f; if (nvalid < 3) x.z = 0.f; if (nvalid < 2) x.y = 0.f; }
                maybe_copy_out4(cs, row_base + r, n, x, 0);
            }
        }
    }
}

// A chunk whose row and column origin are known only now (the functor's address is formed per chunk).
template <class CS>
__device__ __forceinline__ void put_chunk(float *v, int row_base, int n0, int M, int N, const CS &cs, float *stage, const float *bias, int act,
                                          float scale) {
    if (CS::kMContiguous) {
        const int m = row_base + (threadIdx.x & 31);
        put_chunk_rows(v, m < M ? cs.row(m) : nullptr, cs.nstride(), row_base, M, n0, N, cs, stage, bias, act, scale);
    } else {
        float *row0 = cs.row(row_base);
        put_chunk_columns(v, row0, cs.row(row_base + 1) - row0, row_base, min(32, M - row_base), n0, N, cs, true, stage, bias, act, scale);
    }
}

// ---- epilogue with a 2x2 / stride-2 max-pool folded in --------------------------------------------------------------
// The accumulator rows are output pixels of y = act(conv + bias); instead of storing y, each warp reduces the 2x2
// windows that lie inside its 32 rows and stores only the pooled value, the window-local argmax (scan order (0,0), (0,1), (1,0),
// (1,1), strict comparison: the first maximum wins, as in cuda_maxpool_fwd) and the 16-bit
// channels-last copies of the pooled tensor for the next convolution.  y itself never reaches HBM.
// Row order: raster (row = pixel index; needs OW a power of two <= 16, so that 32 rows hold whole rows of windows) or window-major
// (row = 4 * window + position).  Either way the warp's eight windows follow one another in the pooled tensor.
struct PoolOut {
    float *pooled;                 // [NB, F, OH/2, OW/2]
    int *mask;                     // same shape
    __nv_bfloat16 *copy[3];        // [NB, (OH/2)*(OW/2), Cp] or null
    int ns, Cp;
    Enc enc;                       // encoding of the copies
    int P, OW;                     // pixels per image and width of y
    int window_major;
    FastDiv by_Pq;                 // set by pool_out_geometry
};
inline void pool_out_geometry(PoolOut &po, int P, int OW, int window_major) {
    po.P = P; po.OW = OW; po.window_major = window_major;
    po.by_Pq = fast_div(P >> 2);
}
__device__ __forceinline__ void put_chunk_pooled(const float *v, int row_base, int n0, int M, int N, const float *bias, int act, const PoolOut &po,
                                                 float *stage, float scale) {
    // Through the staging tile a lane holds FOUR CHANNELS of one window at a time: it reads the window's four rows as 16-byte pieces,
    // applies scale and bias, takes the maximum in registers (ReLU after it: the maximum of what it leaves, and position 0 where that
    // is nothing), and eight lanes write the 64 bytes of a window's channels-last copy.
    const int lane = threadIdx.x & 31, cg = lane & 7, n = n0 + 4 * cg;
    const int Pq = po.P >> 2, d2 = po.window_major ? 2 : po.OW;
    const int lq = po.window_major ? 0 : 30 - __clz(po.OW);            // log2 of a row of windows
    float b[4] = {0.f, 0.f, 0.f, 0.f};
    if (bias && act <= 1) {
#pragma unroll
        for (int j = 0; j < 4; j++) b[j] = n + j < N ? __ldg(bias + n + j) : 0.f;
    }
    __syncwarp();                                                   // the previous chunk has been read out
    epi_put_row(stage, lane, v);
    if (act > 1) { epi_act_row(stage, lane, bias, n0, N, act, scale); scale = 1.f; }
    __syncwarp();
    const bool relu = act == 1;
#pragma unroll 1
    for (int w = lane >> 3; w < 8; w += 4) {
        const int wr = w >> lq;
        const int r0 = po.window_major ? 4 * w : 2 * (wr * po.OW + (w - (wr << lq)));
        float mx[4];
        int id[4];
#pragma unroll
        for (int j = 0; j < 4; j++) { mx[j] = -3.402823466e+38f; id[j] = 0; }       // -FLT_MAX, strict comparisons: the first maximum wins
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 x = *epi_piece(stage, r0 + (i & 1) + (i >> 1) * d2, cg);
            const float z[4] = {x.x * scale + b[0], x.y * scale + b[1], x.z * scale + b[2], x.w * scale + b[3]};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (z[j] > mx[j]) { mx[j] = z[j]; id[j] = i; }
        }
        if (relu) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (!(mx[j] > 0.f)) { mx[j] = 0.f; id[j] = 0; }
        }
        if (row_base + r0 < M) {
            const int gw = (row_base >> 2) + w, img = po.by_Pq.div(gw);
            long long at = ((long long)img * N + n) * Pq + (gw - img * Pq);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (n + j < N) { po.pooled[at] = mx[j]; po.mask[at] = id[j]; }
                else mx[j] = 0.f;
                at += Pq;
            }
            if (po.copy[0] && n < po.Cp) {
                const long long o = (long long)gw * po.Cp + n;
                store_split4_n(mx, po.ns, po.enc, po.copy[0] + o, po.copy[1] + o, po.copy[2] + o);
            }
        }
    }
}

// ---- accumulator in TMEM -> chunks ----------------------------------------------------------------------------------------
// taddr: TMEM address of (first lane of this warp's quarter, column c_begin); row_base: global row of lane 0.  The warp takes the
// 32-column chunks c_begin, c_begin + c_step, ... below c_end; `release` is called once, when the last of them has left TMEM.
// Per-column bias and activation applied on the way out (bias == nullptr and act == 0: plain store).
template <class CS, class Release = NoRelease>
__device__ __forceinline__ void drain_accumulator(uint32_t taddr, int row_base, int col_base, int c_begin, int c_end, int c_step,
                                                  int M, int N, const CS &cs, float *partial, long long partial_off,
                                                  float *stage /* EPI_WARP_SMEM bytes, this warp's own */,
                                                  const float *bias = nullptr, int act = 0, float scale = 1.f,
                                                  int nacc = 1, uint32_t acc_stride = 0 /* partial accumulators to add up */,
                                                  const Release &release = Release()) {
    const int lane = threadIdx.x & 31;
    if (!partial && CS::kMContiguous) {
        const int m_own = row_base + lane;         // this lane owns row m; its address part is computed once, not per element
        float *own = m_own < M ? cs.row(m_own) : nullptr;
#pragma unroll 1
        for (int c = c_begin; c < c_end; c += c_step) {
            float v[32];
            tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
            if (c + c_step >= c_end) release();
            put_chunk_rows(v, own, cs.nstride(), row_base, M, col_base + c, N, cs, stage, bias, act, scale);
        }
    } else {
        float *row0 = partial ? partial + partial_off + (long long)row_base * N : cs.row(row_base);
        const long long ld = partial ? (long long)N : cs.row(row_base + 1) - cs.row(row_base);
        const int rows = min(32, M - row_base);
#pragma unroll 1
        for (int c = c_begin; c < c_end; c += c_step) {
            float v[32];
            tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
            if (c + c_step >= c_end) release();
            put_chunk_columns(v, row0, ld, row_base, rows, col_base + c, N, cs, !partial, stage, partial ? nullptr : bias, partial ? 0 : act,
                              partial ? 1.f : scale);
        }
    }
}

template <class Release = NoRelease>
__device__ __forceinline__ void drain_accumulator_pooled(uint32_t taddr, int row_base, int col_base, int c_begin, int c_end, int c_step,
                                                         int M, int N, const float *bias, int act, const PoolOut &po, float *stage,
                                                         float scale = 1.f, int nacc = 1, uint32_t acc_stride = 0,
                                                         const Release &release = Release()) {
#pragma unroll 1
    for (int c = c_begin; c < c_end; c += c_step) {
        float v[32];
        tmem_ld32_sum(taddr + (uint32_t)(c - c_begin), v, nacc, acc_stride);
        if (c + c_step >= c_end) release();
        put_chunk_pooled(v, row_base, col_base + c, M, N, bias, act, po, stage, scale);
    }
}

}  // namespace seera
