// Dense products with at most 16 output columns (classifier heads: 256 -> 10, 784 -> 10, 1024 -> 10), exact fp32 on the
// CUDA cores, used in every precision mode.
//
// Such a product is a few MFLOP: on the tensor-core path it costs two operand conversions, a TMA pipeline fill for a handful
// of k-steps into a 32-column tile that is two thirds padding, and a split-K reduce - about 15 us per launch, three launches per
// layer and step - for well under a microsecond of arithmetic.  Here each of the three products of a layer (reference:
// engine_cuda/src/GEMM.cu:95-103 forward, :164-225 backward) is one or two small launches that read the fp32 operands in place:
//   C  = act(A B + bias)   a warp per pair of rows (a block per pair where rows are few), lanes stride over k, N running sums
//                          per lane and row, shuffle reduction
//   dA = dC B^T            one thread per element of dA, N multiply-adds
//   dB = A^T dC (+ dbias)  one thread per row of dB walks its share of the M rows; the shares are summed in a fixed order by a
//                          second small kernel, so the result does not depend on scheduling
// All three are bound by how many reads they keep in flight and by what the two narrow operands cost on the way (a row of B per lane
// touches a line per lane, so B and dB pass through shared memory where that pays).  4096 x 1024 x 10: forward 11.1 -> 8.5 us,
// dA 6.1 -> 5.3, dB 10.2 -> 6.0; 1000 x 1024 x 10: 6.0 -> 5.2, 3.0, 8.2 -> 3.3.
#include "common.cuh"
#include "internal.h"
#include "tc_epilogue.cuh"

namespace seera {

constexpr int SK_MAXN = 16;

// k-extent of the slice of B a block keeps in shared memory, N rows of sk_pitch(N) floats, at most 48 KB; the pitch keeps the copies of
// one k (N of them, a pitch apart) in different banks
__host__ __device__ constexpr int sk_kc(int n) { return n <= 11 ? 1024 : 704; }
__host__ __device__ constexpr int sk_pitch(int n) { return sk_kc(n) + 4; }
constexpr int SK_ROWS = 64;          // most rows of dC a block stages at a time in the two backward kernels

// Softmax over the N values that the first N of 16 neighbouring lanes hold, for a head whose probabilities leave with its logits: the maximum
// and the sum go across the lanes as in softmax_fwd_kernel, so the bits are that kernel's.  All lanes of the warp take part.
// (A launch of its own behind the head's: a prediction of one image by the small CNN 48.5 us instead of 46.3, and 2.2 us of the 68.4 of a loss
// that follows a prediction of 64, which forms the softmax anyway.)
__device__ __forceinline__ float softmax_of_16(float v, bool in) {
    float mx = in ? v : -INFINITY;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = in ? expf(v - mx) : 0.f;
    float sum = e;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return e * (1.f / sum);
}

// C = act(A B + bias); P, where given, the softmax of C's rows (then there is no activation).  A block keeps B^T (slice by slice when K exceeds it) in shared memory as bt[n][k], so that lane = k reads
// it without bank conflicts; a warp forms two rows of C at a time: lanes stride over k (coalesced reads of A), 2 * N running
// sums per lane, shuffle reduction at the end.  With more than one slice the later slices add into C and the last applies
// bias and activation.
template <int N>
__global__ void __launch_bounds__(256) skinny_fwd_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias,
                                                         float *__restrict__ C, float *__restrict__ P, int rows, int K, int act) {
    constexpr int SK_KC = sk_kc(N), PITCH = sk_pitch(N);
    extern __shared__ float bt[];                                        // [N][PITCH]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k0 = 0; k0 < K; k0 += SK_KC) {
        const int kc = min(SK_KC, K - k0);
        __syncthreads();
        // e = k * N + n: consecutive floats of B, every copy in flight at once
        for (int e = threadIdx.x; e < kc * N; e += 256) {
            const int k = e / N, n = e - k * N;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(bt + n * PITCH + k)),
                         "l"(B + (long long)k0 * N + e) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const bool first = k0 == 0, last = k0 + kc == K;
        bool landed = false;
        for (int mb = blockIdx.x * 16; mb < rows; mb += gridDim.x * 16) {
            const int m = mb + warp * 2;
            const bool one = m < rows, two = m + 1 < rows;
            const float *a0 = A + (one ? (long long)m * K : 0) + k0, *a1 = a0 + (two ? K : 0);
            float acc0[N], acc1[N], x0[8], x1[8];
#pragma unroll
            for (int n = 0; n < N; n++) { acc0[n] = 0.f; acc1[n] = 0.f; }
            // eight steps of both rows are fetched while the eight before are used, the first of them while B lands
            auto fetch = [&](int kb, float (&u)[8], float (&v)[8]) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int k = kb + 32 * j + lane;
                    u[j] = k < kc ? __ldg(a0 + k) : 0.f;
                    v[j] = k < kc ? __ldg(a1 + k) : 0.f;
                }
            };
            fetch(0, x0, x1);
            if (!landed) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                __syncthreads();
                landed = true;
            }
            for (int kb = 0; kb < kc; kb += 256) {
                float y0[8], y1[8];
                fetch(kb + 256, y0, y1);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int k = kb + 32 * j + lane;
                    if (kb + 32 * j >= kc) break;
                    const float *b = bt + min(k, kc - 1);
#pragma unroll
                    for (int n = 0; n < N; n++) {
                        acc0[n] = fmaf(x0[j], b[n * PITCH], acc0[n]);
                        acc1[n] = fmaf(x1[j], b[n * PITCH], acc1[n]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; j++) { x0[j] = y0[j]; x1[j] = y1[j]; }
            }
            float v0 = 0.f, v1 = 0.f;
#pragma unroll
            for (int n = 0; n < N; n++) {
                float t0 = acc0[n], t1 = acc1[n];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    t0 += __shfl_xor_sync(0xffffffffu, t0, o);
                    t1 += __shfl_xor_sync(0xffffffffu, t1, o);
                }
                if (lane == n) { v0 = t0; v1 = t1; }
            }
            if (lane < N && one) {
                float *c0 = C + (long long)m * N + lane;
                if (!first) { v0 += *c0; if (two) v1 += c0[N]; }
                if (last) {
                    const float bv = bias ? __ldg(bias + lane) : 0.f;
                    v0 = epilogue_act(v0 + bv, act);
                    v1 = epilogue_act(v1 + bv, act);
                }
                *c0 = v0;
                if (two) c0[N] = v1;
            }
            if (P && last) {
                const float p0 = softmax_of_16(v0, lane < N), p1 = softmax_of_16(v1, lane < N);
                if (lane < N && one) {
                    P[(long long)m * N + lane] = p0;
                    if (two) P[(long long)(m + 1) * N + lane] = p1;
                }
            }
        }
    }
}

// The same for few rows (at most a few blocks' worth per SM): one block per ROWS rows (two, or four once that still leaves a block for
// every SM: what bounds it then is the reads of B), its eight warps take interleaved
// 32-wide pieces of k, B read in place (a warp's reads of B cover 32 * N consecutive floats over its n loop, served by L1), the
// warps' sums added in warp order through shared memory.  No staging of B, and a long contraction (a flattened feature map into
// ten classes) is spread over eight warps instead of walked by one.
template <int N, int ROWS>
__global__ void __launch_bounds__(256) skinny_fwd_small_kernel(const float *__restrict__ A, const float *__restrict__ B,
                                                               const float *__restrict__ bias, float *__restrict__ C, float *__restrict__ P,
                                                               int rows, int K, int act) {
    __shared__ float red[8][ROWS][N];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m = blockIdx.x * ROWS;
    const float *a[ROWS];
    float acc[ROWS][N];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        a[r] = A + (long long)min(m + r, rows - 1) * K;
#pragma unroll
        for (int n = 0; n < N; n++) acc[r][n] = 0.f;
    }
    constexpr int W = N % 2 == 0 ? 2 : 1;                 // floats of a row of B per read (its alignment: see skinny_fwd)
#pragma unroll 2
    for (int k = warp * 32 + lane; k < K; k += 256) {
        float x[ROWS], b[N];
#pragma unroll
        for (int r = 0; r < ROWS; r++) x[r] = __ldg(a[r] + k);
#pragma unroll
        for (int n = 0; n < N; n += W) {
            if (W == 2) {
                const float2 t = __ldg(reinterpret_cast<const float2 *>(B + (long long)k * N + n));
                b[n] = t.x; b[n + W - 1] = t.y;
            } else b[n] = __ldg(B + (long long)k * N + n);
        }
#pragma unroll
        for (int n = 0; n < N; n++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) acc[r][n] = fmaf(x[r], b[n], acc[r][n]);
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
        for (int n = 0; n < N; n++) {
            float t = acc[r][n];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) red[warp][r][n] = t;
        }
    __syncthreads();
    if (threadIdx.x < ROWS * 16) {                        // whole warps, 16 lanes a row
        const int r = threadIdx.x >> 4, n = threadIdx.x & 15;
        const bool in = n < N && m + r < rows;
        float v = 0.f;
        if (in) {
#pragma unroll
            for (int w = 0; w < 8; w++) v += red[w][r][n];
            if (bias) v += __ldg(bias + n);
            v = epilogue_act(v, act);
            C[(long long)(m + r) * N + n] = v;
        }
        if (P) {
            const float p = softmax_of_16(v, in);
            if (in) P[(long long)(m + r) * N + n] = p;
        }
    }
}

// Rows of dC staged in shared memory, padded to a multiple of four floats so that a row is read back with 128-bit broadcasts.
template <int N>
struct SkinnyRows {
    static constexpr int NP = (N + 3) / 4 * 4;
    float v[SK_ROWS][NP];
    __device__ void stage(const float *__restrict__ dC, int m0, int nrows) {
        for (int e = threadIdx.x; e < nrows * N; e += 256) {
            const int r = e / N, n = e - r * N;
            v[r][n] = __ldg(dC + (long long)m0 * N + e);
        }
    }
    __device__ void row(int r, float (&d)[NP]) const {
#pragma unroll
        for (int j = 0; j < NP; j += 4) {
            const float4 t = *reinterpret_cast<const float4 *>(&v[r][j]);
            d[j] = t.x; d[j + 1] = t.y; d[j + 2] = t.z; d[j + 3] = t.w;
        }
    }
};

// dA = dC B^T.  Grid (ceil(K / 256 V), row groups); thread = V neighbouring columns k of dA (V = 4 where K and the addresses allow) with
// their rows of B in registers, walking the rows of its group: V N multiply-adds against broadcast reads of a staged dC row, which one
// column per thread would be bound by; stores coalesced over k.
template <int N, int V>
__device__ __forceinline__ void skinny_dA_block(const float *__restrict__ dC, const float *__restrict__ B, float *__restrict__ dA, int rows, int K,
                                                int chunk_rows, int bx, int by, int groups, SkinnyRows<N> &sd, float *sb /* V = 4: 1024 rows of B */) {
    constexpr int NP = SkinnyRows<N>::NP;
    const int k = (bx * 256 + threadIdx.x) * V;
    float b[V][N];
    if (V == 4) {
        const int k0 = bx * 1024, n4 = min(1024, K - k0) * N / 4;
        for (int e = threadIdx.x; e < n4; e += 256)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(sb + 4 * e)),
                         "l"(B + (long long)k0 * N + 4 * e) : "memory");
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (k < K)
#pragma unroll
            for (int j = 0; j < V * N; j += 4) {
                const float4 t = *reinterpret_cast<const float4 *>(sb + threadIdx.x * (V * N) + j);
                b[j / N][j % N] = t.x; b[(j + 1) / N][(j + 1) % N] = t.y; b[(j + 2) / N][(j + 2) % N] = t.z; b[(j + 3) / N][(j + 3) % N] = t.w;
            }
    } else {
#pragma unroll
        for (int n = 0; n < N; n++) b[0][n] = k < K ? __ldg(B + (long long)k * N + n) : 0.f;
    }
    for (int m0 = by * chunk_rows; m0 < rows; m0 += groups * chunk_rows) {
        const int nrows = min(chunk_rows, rows - m0);
        __syncthreads();
        sd.stage(dC, m0, nrows);
        __syncthreads();
        if (k < K) {
#pragma unroll 4
            for (int r = 0; r < nrows; r++) {
                float d[NP], s[V];
                sd.row(r, d);
#pragma unroll
                for (int v = 0; v < V; v++) {
                    s[v] = 0.f;
#pragma unroll
                    for (int n = 0; n < N; n++) s[v] = fmaf(d[n], b[v][n], s[v]);
                }
                float *o = dA + (long long)(m0 + r) * K + k;
                if (V == 4) *reinterpret_cast<float4 *>(o) = make_float4(s[0], s[V > 1 ? 1 : 0], s[V > 2 ? 2 : 0], s[V > 3 ? 3 : 0]);
                else *o = s[0];
            }
        }
    }
}

template <int N, int V>
__global__ void __launch_bounds__(256) skinny_dA_kernel(const float *__restrict__ dC, const float *__restrict__ B, float *__restrict__ dA,
                                                        int rows, int K, int chunk_rows) {
    __shared__ __align__(16) SkinnyRows<N> sd;
    extern __shared__ __align__(16) float sb[];
    skinny_dA_block<N, V>(dC, B, dA, rows, K, chunk_rows, blockIdx.x, blockIdx.y, gridDim.y, sd, sb);
}

// dB = A^T dC, dbias = column sums of dC.  Grid (ceil(K / 256 V), splits); thread = V neighbouring rows k of dB (V = 2 where K and the
// address allow) walking its split's rows of A (coalesced over k, sixteen loads in flight, those past the end predicated off) against
// the staged dC rows.  The splits' sums are added up in index order by a second small kernel, so the result is the same on every run.
template <int N, int V>
__device__ __forceinline__ void skinny_dB_block(const float *__restrict__ A, const float *__restrict__ dC, float *__restrict__ dB,
                                                float *__restrict__ dbias, float *__restrict__ partial, int rows, int K, int chunk_rows, int bx, int s,
                                                int splits, SkinnyRows<N> &sd, float *so /* 256 V N floats */) {
    constexpr int NP = SkinnyRows<N>::NP;
    const int k = (bx * 256 + threadIdx.x) * V;
    const int chunks = (rows + chunk_rows - 1) / chunk_rows, per = (chunks + splits - 1) / splits;
    const int m_begin = (int)min((long long)rows, (long long)s * per * chunk_rows), m_end = (int)min((long long)rows, (long long)(s + 1) * per * chunk_rows);
    float acc[V][N], colsum = 0.f;
#pragma unroll
    for (int v = 0; v < V; v++)
#pragma unroll
        for (int n = 0; n < N; n++) acc[v][n] = 0.f;
    for (int m0 = m_begin; m0 < m_end; m0 += chunk_rows) {
        const int nrows = min(chunk_rows, m_end - m0);
        float x[16][V];
        auto fetch = [&](int r0) {
            const float *a = A + (long long)m0 * K + k;
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const bool in = k < K && r0 + j < nrows;
                if (V == 2) {
                    const float2 t = in ? __ldg(reinterpret_cast<const float2 *>(a + (long long)(r0 + j) * K)) : make_float2(0.f, 0.f);
                    x[j][0] = t.x; x[j][V - 1] = t.y;
                } else x[j][0] = in ? __ldg(a + (long long)(r0 + j) * K) : 0.f;
            }
        };
        fetch(0);                                         // on their way while the rows of dC are staged
        __syncthreads();
        sd.stage(dC, m0, nrows);
        __syncthreads();
        if (bx == 0 && threadIdx.x < N)
            for (int r = 0; r < nrows; r++) colsum += sd.v[r][threadIdx.x];
        for (int r = 0; r < nrows; r += 16) {
            if (r) fetch(r);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                if (r + j >= nrows) break;
                float d[NP];
                sd.row(r + j, d);
#pragma unroll
                for (int v = 0; v < V; v++)
#pragma unroll
                    for (int n = 0; n < N; n++) acc[v][n] = fmaf(x[j][v], d[n], acc[v][n]);
            }
        }
    }
    // one split: the sums are the result; several: partial[split][k][n] (row K = the column sums), added up in index order below.  They
    // leave through shared memory: N V floats per thread, side by side, would touch a line per lane and store.
#pragma unroll
    for (int v = 0; v < V; v++)
#pragma unroll
        for (int n = 0; n < N; n++) so[threadIdx.x * (V * N) + v * N + n] = acc[v][n];
    __syncthreads();
    const int k0 = bx * (256 * V), count = min(256 * V, K - k0) * N;
    float *p = (splits == 1 ? dB : partial + (long long)s * (K + 1) * N) + (long long)k0 * N;
    for (int e = threadIdx.x; e < count; e += 256) p[e] = so[e];
    if (bx == 0 && threadIdx.x < N) {
        if (splits > 1) partial[((long long)s * (K + 1) + K) * N + threadIdx.x] = colsum;
        else if (dbias) dbias[threadIdx.x] = colsum;
    }
}

template <int N, int V>
__global__ void __launch_bounds__(256) skinny_dB_kernel(const float *__restrict__ A, const float *__restrict__ dC, float *__restrict__ dB,
                                                        float *__restrict__ dbias, float *__restrict__ partial, int rows, int K, int chunk_rows) {
    __shared__ __align__(16) SkinnyRows<N> sd;
    __shared__ float so[256 * V * N];
    skinny_dB_block<N, V>(A, dC, dB, dbias, partial, rows, K, chunk_rows, blockIdx.x, blockIdx.y, gridDim.y, sd, so);
}
// Both in one launch, the blocks of dB first: neither needs anything of the other, and a launch of its own is half of what dA takes for a few
// hundred rows (64 x 784 x 10: 2.2 + 3.0 -> 3.1 us; 1024 rows 6.2 -> 4.3).  VA as V of dA, VB of dB.
struct SkinnyGrid { int kblocks, groups, chunk_rows; };
template <int N, int VA, int VB>
__global__ void __launch_bounds__(256) skinny_both_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ dC,
                                                          float *__restrict__ dA, float *__restrict__ dB, float *__restrict__ dbias,
                                                          float *__restrict__ partial, int rows, int K, SkinnyGrid ga, SkinnyGrid gb) {
    __shared__ __align__(16) SkinnyRows<N> sd;
    extern __shared__ __align__(16) float sb[];           // the larger of dB's outputs and dA's rows of B
    int b = blockIdx.x;
    if (b < gb.kblocks * gb.groups) {
        const int s = b / gb.kblocks;
        skinny_dB_block<N, VB>(A, dC, dB, dbias, partial, rows, K, gb.chunk_rows, b - s * gb.kblocks, s, gb.groups, sd, sb);
    } else {
        b -= gb.kblocks * gb.groups;
        const int y = b / ga.kblocks;
        skinny_dA_block<N, VA>(dC, B, dA, rows, K, ga.chunk_rows, b - y * ga.kblocks, y, ga.groups, sd, sb);
    }
}

bool skinny_applies(int M, int N, int K, int Nbatch) {
    return rt().precision != 0 && rt().skinny_gemm && N >= 1 && N <= SK_MAXN && K >= 1 && (long long)M * Nbatch < (1ll << 31) &&
           (long long)M * Nbatch * K < (1ll << 40);
}

#define SK_DISPATCH(N, CALL)                                                                          \
    switch (N) {                                                                                      \
        case 1: { constexpr int NN = 1; CALL; } break;   case 2: { constexpr int NN = 2; CALL; } break;   \
        case 3: { constexpr int NN = 3; CALL; } break;   case 4: { constexpr int NN = 4; CALL; } break;   \
        case 5: { constexpr int NN = 5; CALL; } break;   case 6: { constexpr int NN = 6; CALL; } break;   \
        case 7: { constexpr int NN = 7; CALL; } break;   case 8: { constexpr int NN = 8; CALL; } break;   \
        case 9: { constexpr int NN = 9; CALL; } break;   case 10: { constexpr int NN = 10; CALL; } break; \
        case 11: { constexpr int NN = 11; CALL; } break; case 12: { constexpr int NN = 12; CALL; } break; \
        case 13: { constexpr int NN = 13; CALL; } break; case 14: { constexpr int NN = 14; CALL; } break; \
        case 15: { constexpr int NN = 15; CALL; } break; default: { constexpr int NN = 16; CALL; } break; \
    }

int skinny_fwd(const float *A, const float *B, const float *bias, float *C, float *P, int rows, int N, int K, int act, const char *name) {
    cudaStream_t st = rt().stream;
    int grid = (rows + 15) / 16;
    if (grid > rt().sm_count * 2) grid = rt().sm_count * 2;
    const size_t smem = (size_t)N * sk_pitch(N) * sizeof(float);
    const bool small = (rows + 1) / 2 <= rt().sm_count * 4;             // a block per pair of rows still fits a wave or so
    profile_begin();
    if (small && (reinterpret_cast<uintptr_t>(B) & 7) == 0) {
        if ((rows + 3) / 4 >= rt().sm_count) { SK_DISPATCH(N, (skinny_fwd_small_kernel<NN, 4><<<(rows + 3) / 4, 256, 0, st>>>(A, B, bias, C, P, rows, K, act))) }
        else { SK_DISPATCH(N, (skinny_fwd_small_kernel<NN, 2><<<(rows + 1) / 2, 256, 0, st>>>(A, B, bias, C, P, rows, K, act))) }
    } else
    SK_DISPATCH(N, (skinny_fwd_kernel<NN><<<grid, 256, smem, st>>>(A, B, bias, C, P, rows, K, act)))
    count_launch();
    profile_end(2.0 * rows * N * (double)K, name);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, name);
}

int skinny_bwd(const float *A, const float *B, const float *dC, float *dA, float *dB, float *dbias, int rows, int N, int K) {
    cudaStream_t st = rt().stream;
    cudaError_t e = cudaSuccess;
    auto aligned = [&](const void *p, int v) { return K % v == 0 && (reinterpret_cast<uintptr_t>(p) & (4 * v - 1)) == 0; };
    // rows staged at a time and row groups for `kblocks` blocks of columns: about `per_sm` blocks per SM; few rows where the rows are few,
    // so that a small problem still spreads over many blocks (at least `least`, at most SK_ROWS)
    int chunk_rows = 0, groups = 0;
    auto split = [&](int kblocks, int per_sm, int least) {
        groups = (rt().sm_count * per_sm + kblocks - 1) / kblocks;
        chunk_rows = ((rows + groups - 1) / groups + least - 1) / least * least;
        if (chunk_rows > SK_ROWS) chunk_rows = SK_ROWS;
        const int chunks = (rows + chunk_rows - 1) / chunk_rows;
        if (groups > chunks) groups = chunks;
        if (groups > 65535) groups = 65535;
    };
    // (the copy of B per block pays from a few rows per block on)
    const bool four = aligned(dA, 4) && aligned(B, 4) && (long long)rows * K >= 1 << 19, two = aligned(A, 2);
    SkinnyGrid ga{}, gb{};
    split(four ? (K / 4 + 255) / 256 : (K + 255) / 256, four ? 2 : 4, 8);
    ga = SkinnyGrid{four ? (K / 4 + 255) / 256 : (K + 255) / 256, groups, chunk_rows};
    const int kb = ((two ? K / 2 : K) + 255) / 256;
    split(kb, 2, (long long)rows * K >= 1 << 19 ? 16 : 8);        // few splits: what each of them leaves is written and read again
    gb = SkinnyGrid{kb, groups, chunk_rows};
    const int splits = gb.groups;
    const bool want_b = dB || dbias, both = dA && want_b;
    float *partial = nullptr, *db_out = dB, *tmp = nullptr;
    if (want_b) {
        partial = (float *)scratch_alloc((size_t)splits * (K + 1) * N * sizeof(float));
        if (!partial) return SEERA_E_OOM;
        if (!dB) { tmp = (float *)scratch_alloc((size_t)K * N * sizeof(float)); if (!tmp) { scratch_free(partial); return SEERA_E_OOM; } db_out = tmp; }
    }
    profile_begin();
    if (both) {
        const size_t fa = four ? (size_t)1024 * N : 0, fb = (size_t)256 * (two ? 2 : 1) * N, smem = (fa > fb ? fa : fb) * sizeof(float);
        const unsigned grid = (unsigned)(ga.kblocks * ga.groups + gb.kblocks * gb.groups);
#define SK_BOTH(VA, VB)                                                                                                                      \
        SK_DISPATCH(N, e = allow_smem((const void *)skinny_both_kernel<NN, VA, VB>, smem))                                                   \
        if (e == cudaSuccess) SK_DISPATCH(N, (skinny_both_kernel<NN, VA, VB><<<grid, 256, smem, st>>>(A, B, dC, dA, db_out, dbias, partial, rows, K, ga, gb)))
        if (four && two) { SK_BOTH(4, 2) }
        else if (four) { SK_BOTH(4, 1) }
        else if (two) { SK_BOTH(1, 2) }
        else { SK_BOTH(1, 1) }
#undef SK_BOTH
        count_launch();
    } else if (dA) {
        const dim3 grid((unsigned)ga.kblocks, (unsigned)ga.groups);
        if (four) {
            const size_t smem = (size_t)1024 * N * sizeof(float);
            SK_DISPATCH(N, e = allow_smem((const void *)skinny_dA_kernel<NN, 4>, smem))
            if (e == cudaSuccess) SK_DISPATCH(N, (skinny_dA_kernel<NN, 4><<<grid, 256, smem, st>>>(dC, B, dA, rows, K, ga.chunk_rows)))
        } else {
            SK_DISPATCH(N, (skinny_dA_kernel<NN, 1><<<grid, 256, 0, st>>>(dC, B, dA, rows, K, ga.chunk_rows)))
        }
        count_launch();
    } else if (want_b) {
        const dim3 grid((unsigned)gb.kblocks, (unsigned)gb.groups);
        if (two) { SK_DISPATCH(N, (skinny_dB_kernel<NN, 2><<<grid, 256, 0, st>>>(A, dC, db_out, dbias, partial, rows, K, gb.chunk_rows))) }
        else { SK_DISPATCH(N, (skinny_dB_kernel<NN, 1><<<grid, 256, 0, st>>>(A, dC, db_out, dbias, partial, rows, K, gb.chunk_rows))) }
        count_launch();
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess && want_b && splits > 1) {
        launch_sum_splits(partial, db_out, (K + 1) * N, splits, st, dbias, K * N);
        e = cudaGetLastError();
    }
    profile_end((both ? 4.0 : 2.0) * rows * N * (double)K, both ? "cuda_matmul_bwd(dA+dB)" : (dA ? "cuda_matmul_bwd(dA)" : "cuda_matmul_bwd(dB)"));
    if (partial) scratch_free(partial);
    if (tmp) scratch_free(tmp);
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, "cuda_matmul_bwd");
}

}  // namespace seera
