// 3 x 3 unit-stride convolutions of little work (a few tens of million multiply-adds: the inner layers of a small network, or of any
// network at a small batch), exact fp32 on the CUDA cores.
//
// On the tensor-core path such a layer is all start-up: its filters are converted by one launch, the GEMM walks nine k-steps of 64
// channels of which it has eight or sixteen, and its gradient needs channels-last copies first - 12 us forward and 29 us backward for
// work of a microsecond (8 -> 16 channels, 64 images of 14 x 14; here 5 and 16 us).  Here a block takes a band of one image, stages it
// with its border of zeros, the filters as [input channel][tap][output channel], and a warp forms 32 blocks of 2 x 2 outputs for FW output channels:
// per input channel 8 reads of its own 4 x 4 patch and 9 broadcasts of FW weights for 36 FW / 2 packed multiply-adds.  The data
// gradient is the same convolution of dz with the taps reversed; dz - activation slope, and the routing through a 2x2 max-pool - is
// formed while the band is staged.  The weight gradient is first_dw's in groups of four input channels, in the same launch, and a
// layer with its pool goes to conv_pool_simt.
//
// The forward of a layer with up to four input channels (stride 1 or 2) takes the same kernel at any size: it is bound by its stores - the
// output and, for the convolution that reads it, the channels-last copies - of which a lane with 16 filters writes whole sectors, where
// the tensor-core form is bound by the warps that gather and split patches.  1 -> 32 channels, stride 2, 256 images of 64 x 64 with copies
// (67 MB): 35 -> 28 us, a third of it waiting for instructions (the straight-line code runs twice per warp); passing the outputs through
// shared memory to shorten it gave 26 there and cost 2 us where no copies are made.
#include "conv_dw_block.cuh"
#include "contraction_functors.cuh"
#include "internal.h"

namespace seera {

// Where the lines lie, forward with pool + backward, microseconds against the tensor-core path in fp16x3 / bf16x6 (which pads the
// channels of both operands to 64, so that its cost does not fall with C * F): 8 -> 16 channels 19 against 38 / 44 at 2 million
// multiply-adds, 38 against 101 / 132 at 64, 64 against 168 / 233 at 128; 16 -> 32 channels 34 against 35 / 43 at 2, 35 against 39 / 46
// at 32, 45 against 43 / 52 at 64; 32 -> 32 channels 42 against 33 / 40 at 2.
bool conv_small_applies(int NB, int C, int H, int W, int F, int R, int S, int sh, int sw, int ph, int pw) {
    // not in the modes of a single rounded product, whose results are those of rounded operands
    if (rt().precision < 2 || rt().precision > 4 || !rt().conv_tma) return false;
    if (R != 3 || S != 3 || sh != 1 || sw != 1 || ph < 0 || pw < 0 || ph > 2 || pw > 2 || NB < 1 || C * 9 <= 64 || C > 64 || F < 1 || F > 64 || C * F > 512)
        return false;
    const long long OH = (long long)H + 2 * ph - 2, OW = (long long)W + 2 * pw - 2, h = OH > H ? OH : H, w = OW > W ? OW : W;
    if (OH < 1 || OW < 1 || w * (C > F ? C : F) > 6144) return false;        // four rows of every channel fit a block's shared memory
    return NB * h * w < (1ll << 26) && NB * h * w * 9 * (C * F) * (C * F) <= 1ll << 35;
}

// What a band is made from: a tensor, its product with the slope of the activation whose output is y, or a pooled gradient.
struct SmallSource {
    const float *v, *y;        // y null: no slope
    const int *mask;           // v (and y) of a 2x2 / stride-2 max-pool; null: full resolution
    int act;
};
// Channels-last copies of the output ([pixel][Cp], Cp = O); p[0] null: none.
struct SmallCopies {
    __nv_bfloat16 *p[3];
    int Cp, ns;
    Enc enc;
};
struct SmallGeom {
    int I, IH, IW, O, OH, OW, ph, pw;        // input / output channels and planes, lower padding
    int window_rows, per_image, rows, pitch, OP, groups;
    FastDiv by_bands, by_pitch, by_rows, by_cols, by_groups;
};

// What a launch works on; `grid` blocks walk `total` bands.
struct SmallArgs {
    SmallSource src;
    const float *Wt, *bias;
    float *Y;
    SmallCopies cc;
    SmallGeom g;
    int total, reversed, act, grid;
    size_t smem;
};
template <int FW, int ST>
__device__ __forceinline__ void conv3x3_small_block(const SmallArgs &a, int block, float *sm) {
    const SmallSource &src = a.src;
    const float *__restrict__ Wt = a.Wt, *__restrict__ bias = a.bias;
    float *__restrict__ Y = a.Y;
    const SmallCopies &cc = a.cc;
    const SmallGeom &g = a.g;
    const int total = a.total, reversed = a.reversed, act = a.act;
    constexpr int PR = 3 + ST, PC = (PR + 1) / 2 * 2;     // rows of a patch, and columns read of it
    // sm: [I][9][OP] weights, [OP] biases, [8][4 FW][32] sums (data gradient), [I][rows][pitch] band
    float *bk = sm + g.I * 9 * g.OP, *red = bk + g.OP, *band = red + (reversed ? 8 * 4 * FW * 32 : 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = g.I * 9 * g.OP;
    // Wt[o][i][t], or for the data gradient Wt[i][o][8 - t]
    for (int e0 = threadIdx.x; e0 < nw; e0 += 8 * 256) {
        float w[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int e = e0 + j * 256, k = e / g.OP, o = e - k * g.OP, i = k / 9, t = k - i * 9;
            w[j] = e < nw && o < g.O ? __ldg(Wt + (reversed ? ((long long)i * g.O + o) * 9 + 8 - t : ((long long)o * g.I + i) * 9 + t)) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; j++)
            if (e0 + j * 256 < nw) sm[e0 + j * 256] = w[j];
    }
    for (int e = threadIdx.x; e < g.OP; e += 256) bk[e] = bias && e < g.O ? __ldg(bias + e) : 0.f;
    const int bplane = g.rows * g.pitch, bsize = g.I * bplane, cols = (g.OW + 1) >> 1;
    const long long iplane = (long long)g.IH * g.IW, oplane = (long long)g.OH * g.OW;
    const bool pairs = (g.OW & 1) == 0 && (reinterpret_cast<uintptr_t>(Y) & 7) == 0;

    for (int id = block; id < total; id += a.grid) {
        const int n = g.by_bands.div(id), q0 = (id - n * g.per_image) * g.window_rows, ih0 = 2 * ST * q0 - g.ph;
        if (src.mask) {                                   // every pixel from its window's gradient, index and output
            const int Wq = g.IW >> 1;
            const long long qplane = iplane >> 2, base = (long long)n * g.I * qplane;
            for (int e0 = threadIdx.x; e0 < bsize; e0 += 8 * 256) {
                float v[8], y[8];
                int m[8], pos[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int e = e0 + j * 256, rr = g.by_pitch.div(e), x = e - rr * g.pitch, i = g.by_rows.div(rr);
                    const int ih = ih0 + rr - i * g.rows, iw = x - g.pw;
                    const bool in = e < bsize && (unsigned)ih < (unsigned)g.IH && (unsigned)iw < (unsigned)g.IW;
                    const long long o = in ? base + i * qplane + (long long)(ih >> 1) * Wq + (iw >> 1) : 0;
                    pos[j] = in ? ((ih & 1) << 1) | (iw & 1) : -1;
                    v[j] = __ldg(src.v + o); m[j] = __ldg(src.mask + o); y[j] = src.y ? __ldg(src.y + o) : 0.f;
                }
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (e0 + j * 256 < bsize)
                        band[e0 + j * 256] = m[j] == pos[j] ? v[j] * (src.y ? first_slope(y[j], src.act) : 1.f) : 0.f;
            }
        } else {
            const long long base = (long long)n * g.I * iplane;
            for (int e0 = threadIdx.x; e0 < bsize; e0 += 8 * 256) {
                float v[8], y[8];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int e = e0 + j * 256, rr = g.by_pitch.div(e), x = e - rr * g.pitch, i = g.by_rows.div(rr);
                    const int ih = ih0 + rr - i * g.rows, iw = x - g.pw;
                    const bool in = e < bsize && (unsigned)ih < (unsigned)g.IH && (unsigned)iw < (unsigned)g.IW;
                    const long long o = base + i * iplane + (long long)ih * g.IW + iw;
                    v[j] = in ? __ldg(src.v + o) : 0.f;
                    y[j] = in && src.y ? __ldg(src.y + o) : 0.f;
                }
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (e0 + j * 256 < bsize) band[e0 + j * 256] = src.y ? v[j] * first_slope(y[j], src.act) : v[j];
            }
        }
        __syncthreads();
        const int windows = min(g.window_rows, ((g.OH + 1) >> 1) - q0) * cols, items = ((windows + 31) >> 5) * g.groups;
        // at most half as many items as warps: several warps share an item, each with its part of the input
        // channels (not in the forward, which gives the same bits as conv_pool_simt)
        const int lg = items > 4 || !reversed ? 0 : (items > 2 ? 1 : (items > 1 ? 2 : 3)), part = warp & ((1 << lg) - 1), ipart = (g.I + (1 << lg) - 1) >> lg;
        const int i0 = part * ipart, i1 = min(g.I, i0 + ipart);
        for (int base = 0; base < items; base += 8 >> lg) {
            const int at = base + (warp >> lg), item = min(at, items - 1);
            const bool mine = at < items;
            const int tile = g.by_groups.div(item), o0 = (item - tile * g.groups) * FW;
            const int w = tile * 32 + lane, wl = min(w, windows - 1), qr = g.by_cols.div(wl), qc = wl - qr * cols;
            const float *patch = band + i0 * bplane + 2 * ST * qr * g.pitch + 2 * ST * qc, *wc = sm + i0 * 9 * g.OP + o0;
            f32x2 acc[4][FW / 2];                         // [pixel of the 2 x 2 block][pair of output channels]
#pragma unroll
            for (int p = 0; p < 4; p++)
#pragma unroll
                for (int f = 0; f < FW / 2; f++) acc[p][f] = 0ull;
            for (int i = i0; i < i1; i++, wc += 9 * g.OP, patch += bplane) {
                f32x2 v[PR][PC];
#pragma unroll
                for (int r = 0; r < PR; r++)
#pragma unroll
                    for (int j = 0; j < PC; j += 2) {
                        const float2 u = *reinterpret_cast<const float2 *>(patch + r * g.pitch + j);
                        v[r][j] = pack2(u.x, u.x); v[r][j + 1] = pack2(u.y, u.y);
                    }
#pragma unroll
                for (int t = 0; t < 9; t++)
#pragma unroll
                    for (int f = 0; f < FW / 4; f++) {
                        const ulonglong2 w2 = *reinterpret_cast<const ulonglong2 *>(wc + t * g.OP + 4 * f);
#pragma unroll
                        for (int p = 0; p < 4; p++) {
                            acc[p][2 * f] = ffma2(v[(p >> 1) * ST + t / 3][(p & 1) * ST + t % 3], w2.x, acc[p][2 * f]);
                            acc[p][2 * f + 1] = ffma2(v[(p >> 1) * ST + t / 3][(p & 1) * ST + t % 3], w2.y, acc[p][2 * f + 1]);
                        }
                    }
            }
            if (lg) {                                     // the parts are added in order
                float *mine_at = red + warp * (4 * FW * 32) + lane;
                if (part)
#pragma unroll
                    for (int k = 0; k < 2 * FW; k++) {
                        float lo, hi;
                        unpack2(acc[k / (FW / 2)][k % (FW / 2)], lo, hi);
                        mine_at[(2 * k) * 32] = lo; mine_at[(2 * k + 1) * 32] = hi;
                    }
                __syncthreads();
                if (!part)
                    for (int q = 1; q < 1 << lg; q++)
#pragma unroll
                        for (int k = 0; k < 2 * FW; k++) {
                            const float *o = mine_at + q * (4 * FW * 32) + 2 * k * 32;
                            acc[k / (FW / 2)][k % (FW / 2)] = add2(acc[k / (FW / 2)][k % (FW / 2)], pack2(o[0], o[32]));
                        }
            }
            if (w < windows && mine && !part) {
                const int oh = 2 * (q0 + qr), ow = 2 * qc;
                float *yo = Y + ((long long)n * g.O + o0) * oplane + (long long)oh * g.OW + ow;
                float z[4][FW];
#pragma unroll
                for (int p = 0; p < 4; p++)
#pragma unroll
                    for (int f = 0; f < FW; f += 2) {
                        unpack2(acc[p][f >> 1], z[p][f], z[p][f + 1]);
                        z[p][f] = epilogue_act(z[p][f] + bk[o0 + f], act);
                        z[p][f + 1] = epilogue_act(z[p][f + 1] + bk[o0 + f + 1], act);
                    }
#pragma unroll
                for (int f = 0; f < FW; f++, yo += oplane) {
                    if (o0 + f >= g.O) break;
                    if (pairs) {
                        *reinterpret_cast<float2 *>(yo) = make_float2(z[0][f], z[1][f]);
                        if (oh + 1 < g.OH) *reinterpret_cast<float2 *>(yo + g.OW) = make_float2(z[2][f], z[3][f]);
                    } else {
                        yo[0] = z[0][f];
                        if (ow + 1 < g.OW) yo[1] = z[1][f];
                        if (oh + 1 < g.OH) { yo[g.OW] = z[2][f]; if (ow + 1 < g.OW) yo[g.OW + 1] = z[3][f]; }
                    }
                }
                if (FW >= 8 && cc.p[0]) {
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        if (oh + (p >> 1) >= g.OH || ow + (p & 1) >= g.OW) continue;
                        const long long c = ((long long)n * oplane + (long long)(oh + (p >> 1)) * g.OW + ow + (p & 1)) * cc.Cp + o0;
#pragma unroll
                        for (int h = 0; h + 8 <= FW; h += 8) store_split8_n(z[p] + h, cc.ns, cc.enc, cc.p[0] + c + h, cc.p[1] + c + h, cc.p[2] + c + h);
                    }
                }
            }
        }
        __syncthreads();                                  // the band has been read
    }
}

template <int FW, int ST>
__global__ void __launch_bounds__(256, FW >= 8 ? 2 : 1) conv3x3_small_kernel(const __grid_constant__ SmallArgs a) {
    extern __shared__ __align__(16) float sm[];
    conv3x3_small_block<FW, ST>(a, blockIdx.x, sm);
}
// Data and weight gradient of a layer in one launch: they depend on nothing of each other's, and one after the other each was a chain of
// start, staging and end of 6 us on a chip with room for both (8 -> 16 channels, 64 images of 14 x 14: 6.9 + 6.1 -> 9.2 us, 30 images 13.1 -> 8.3).
template <int FL, bool POOLED>
__global__ void __launch_bounds__(256, 2) conv3x3_small_bwd_kernel(const __grid_constant__ SmallArgs a, const __grid_constant__ DwArgs d) {
    extern __shared__ __align__(16) float sm[];
    const int b = blockIdx.x, per = d.nblocks * d.chunks, wblocks = per * d.cgroups;
    if (b < wblocks) {
        const int bz = b / per, rest = b - bz * per, by = rest / d.nblocks;
        first_dw_block<4, 1, FL, POOLED>(d, rest - by * d.nblocks, by, bz, sm);
    } else {
        conv3x3_small_block<4, 1>(a, b - wblocks, sm);
    }
}

template <int FW, int ST>
static SmallArgs small_args(const SmallSource &src, const float *Wt, const float *bias, float *Y, int NB, int I, int IH, int IW, int O, int OH, int OW,
                            int ph, int pw, int reversed, int act, const SmallCopies &cc, int blocks) {
    SmallArgs a{src, Wt, bias, Y, cc, {}, 0, reversed, act, 0, 0};
    SmallGeom &g = a.g;
    g.I = I; g.IH = IH; g.IW = IW; g.O = O; g.OH = OH; g.OW = OW; g.ph = ph; g.pw = pw;
    const int wrows = (OH + 1) / 2, cols = (OW + 1) / 2;
    g.OP = (O + FW - 1) / FW * FW; g.groups = g.OP / FW;
    g.pitch = 2 * ST * cols + 2;
    // bands of as many window rows as fit 24 KB (at least one), fewer while there would not be `blocks` of them
    const size_t row = (size_t)I * g.pitch * sizeof(float);
    auto rows = [](int wr) { return 2 * ST * wr + 3 - ST; };
    int wr = 1;
    while (wr < wrows && rows(wr + 1) * row <= 24 * 1024) wr++;
    while (wr > 1 && (long long)NB * ((wrows + wr - 1) / wr) < blocks) wr = (wr + 1) / 2;
    g.window_rows = wr; g.rows = rows(wr); g.per_image = (wrows + wr - 1) / wr;
    g.by_bands = fast_div(g.per_image); g.by_pitch = fast_div(g.pitch); g.by_rows = fast_div(g.rows);
    g.by_cols = fast_div(cols); g.by_groups = fast_div(g.groups);
    a.smem = ((size_t)(I * 9 + 1) * g.OP + (reversed ? 8 * 4 * FW * 32 : 0)) * sizeof(float) + g.rows * row;
    a.total = NB * g.per_image;
    a.grid = rt().sm_count * 4;
    if (a.grid > a.total) a.grid = a.total;
    return a;
}
template <int FW, int ST>
static int small_launch(const SmallSource &src, const float *Wt, const float *bias, float *Y, int NB, int I, int IH, int IW, int O, int OH, int OW,
                        int ph, int pw, int reversed, int act, const SmallCopies &cc, const char *name) {
    const SmallArgs a = small_args<FW, ST>(src, Wt, bias, Y, NB, I, IH, IW, O, OH, OW, ph, pw, reversed, act, cc, rt().sm_count);
    profile_begin();
    cudaError_t e = allow_smem((const void *)conv3x3_small_kernel<FW, ST>, a.smem);
    if (e == cudaSuccess) {
        conv3x3_small_kernel<FW, ST><<<a.grid, 256, a.smem, rt().stream>>>(a);
        count_launch();
        e = cudaGetLastError();
    }
    profile_end(2.0 * NB * OH * OW * (double)O * I * 9, name);
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, name);
}
// Both gradients in one launch; its blocks are the two launches' together.
template <int FL, bool POOLED>
static int small_bwd_launch(const SmallArgs &a, const float *X, const DzSource &dz, float *dW, float *dbias, const FirstGeom &g) {
    const char *name = "conv2d_small_bwd(dX+dW)";
    DwArgs d = dw_args<4, 1, FL, POOLED>(X, dz, g);
    d.partial = (float *)scratch_alloc(dw_partial_bytes<4>(d));
    if (!d.partial) return SEERA_E_OOM;
    const size_t smem = a.smem > d.smem ? a.smem : d.smem;
    profile_begin();
    cudaError_t e = allow_smem((const void *)conv3x3_small_bwd_kernel<FL, POOLED>, smem);
    if (e == cudaSuccess) {
        conv3x3_small_bwd_kernel<FL, POOLED><<<d.nblocks * d.chunks * d.cgroups + a.grid, 256, smem, rt().stream>>>(a, d);
        count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        using Sh = DwShape<4, 1, FL, POOLED>;
        first_wgrad_reduce(d.partial, dW, dbias, g.F, g.K, Sh::K, Sh::KP, d.nblocks, rt().stream);
        e = cudaGetLastError();
    }
    profile_end(4.0 * g.NB * g.OH * g.OW * (double)g.F * g.K, name);
    scratch_free(d.partial);
    return e == cudaSuccess ? SEERA_OK : check_cuda(e, name);
}
// four output channels per warp: a small layer has too few 32-window tiles to fill the chip with more
static int small_run(const SmallSource &src, const float *Wt, const float *bias, float *Y, int NB, int I, int IH, int IW, int O, int OH, int OW,
                     int ph, int pw, int reversed, int act, const char *name) {
    return small_launch<4, 1>(src, Wt, bias, Y, NB, I, IH, IW, O, OH, OW, ph, pw, reversed, act, SmallCopies{}, name);
}

bool conv_direct_applies(int NB, int C, int H, int W, int F, int R, int S, int sh, int sw, int ph, int pw, bool copies) {
    // Not in the mode of a single bf16 product, whose results are those of rounded operands.  Not in mode 3 either, the default, with whose
    // results runs are compared: a new order of the sums there moves ReLU and pool decisions of the layers behind (up to 4e-2 of a gradient two
    // steps into a batch-norm network, in four of eight seeds), and is taken where it pays - conv_small and first_dw take a half to a
    // fourth of what they replaced.  Here it is 16.3 -> 12.7 us of a step of 300 (3 -> 32 channels, 128 images of 32 x 32; 64 images of 4 x 20 x 20
    // into 48: 10.6 -> 14.7), although against 64 bits this kernel is off by 1.0e-7 where the tensor-core form's six products are by 3.3e-7.
    if (rt().precision < 2 || rt().precision == 3 || !rt().conv_tma || R != 3 || S != 3 || sh != sw || sh < 1 || sh > 2 || ph < 0 || pw < 0 || ph > 2 || pw > 2) return false;
    const long long OH = ((long long)H + 2 * ph - 3) / sh + 1, OW = ((long long)W + 2 * pw - 3) / sw + 1;
    return NB >= 1 && C >= 1 && C <= 4 && F >= 1 && (size_t)(C * 9 + 1) * (F + 15) * sizeof(float) <= 64 * 1024 && (!copies || F % 8 == 0) &&
           H + 2 * ph >= 3 && W + 2 * pw >= 3 && (long long)W * C <= 4096 && NB * OH * OW < (1ll << 31) - 64 && (long long)C * H * W < (1ll << 30);
}
int conv_direct_fwd(const float *X, const float *Wt, const float *bias, float *Y, int NB, int C, int H, int W, int F, int st, int ph, int pw, int act,
                    const StorePixelRows *copies, const char *name) {
    const int OH = (H + 2 * ph - 3) / st + 1, OW = (W + 2 * pw - 3) / st + 1;
    SmallCopies cc{};
    if (copies) {
        for (int i = 0; i < 3; i++) cc.p[i] = copies->cp[i];
        cc.Cp = copies->Cp; cc.ns = copies->ns; cc.enc = copies->enc;
    }
    const SmallSource src{X, nullptr, nullptr, 0};
    // 16 filters per warp (one read of a value per 16 of them, whole sectors of the copies) where that leaves every scheduler a warp
    const long long tiles = (long long)NB * ((OH + 1) / 2) * ((OW + 1) / 2) / 32;
#define SEERA_DIRECT(FW) \
    (st == 1 ? small_launch<FW, 1>(src, Wt, bias, Y, NB, C, H, W, F, OH, OW, ph, pw, 0, act, cc, name) \
             : small_launch<FW, 2>(src, Wt, bias, Y, NB, C, H, W, F, OH, OW, ph, pw, 0, act, cc, name))
    if (F > 8 && (!copies || F % 16 == 0) && tiles * ((F + 15) / 16) >= 4ll * rt().sm_count) return SEERA_DIRECT(16);
    if (F > 4) return SEERA_DIRECT(8);
    return SEERA_DIRECT(4);
#undef SEERA_DIRECT
}

int conv_small_fwd(const float *X, const float *Wt, const float *bias, float *Y, int NB, int C, int H, int W, int F, int ph, int pw, int act,
                   const char *name) {
    return small_run(SmallSource{X, nullptr, nullptr, 0}, Wt, bias, Y, NB, C, H, W, F, H + 2 * ph - 2, W + 2 * pw - 2, ph, pw, 0, act, name);
}
bool conv_small_bwd_applies(const float *y, const float *gp, const float *y_pooled, int act) {
    return !gp || act == SEERA_ACT_NONE || y_pooled;       // with the layer output alone a pooled gradient's slope would need a gather
}
int conv_small_bwd(const float *Wt, const float *X, const float *y, const float *g, const float *gp, const int *mask, const float *y_pooled,
                   float *dX, float *dW, float *dbias, int NB, int C, int H, int W, int F, int ph, int pw, int act) {
    const int OH = H + 2 * ph - 2, OW = W + 2 * pw - 2;
    const bool sloped = act != SEERA_ACT_NONE;
    int s = SEERA_OK;
    if (dX && dW && C > 3) {                // (fewer channels have their own weight-gradient kernels)
        const SmallSource src{gp ? gp : g, sloped ? (gp ? y_pooled : y) : nullptr, gp ? mask : nullptr, act};
        // two thirds of a block per SM: the weight gradient's blocks fill the rest, and 354 blocks for 296 places took a second round
        const SmallArgs a = small_args<4, 1>(src, Wt, nullptr, dX, NB, F, OH, OW, C, H, W, 2 - ph, 2 - pw, 1, SEERA_ACT_NONE, SmallCopies{},
                                             rt().sm_count * 2 / 3);
        const FirstGeom geo{NB, C, H, W, F, 3, 3, 1, 1, ph, pw, OH, OW, C * 9};
        const DzSource dz{nullptr, g, gp, mask, y, act, y_pooled};
        if (gp) return F <= 8 ? small_bwd_launch<8, true>(a, X, dz, dW, dbias, geo) : F <= 16 ? small_bwd_launch<16, true>(a, X, dz, dW, dbias, geo)
                                                                                                   : small_bwd_launch<32, true>(a, X, dz, dW, dbias, geo);
        return F <= 8 ? small_bwd_launch<8, false>(a, X, dz, dW, dbias, geo) : F <= 16 ? small_bwd_launch<16, false>(a, X, dz, dW, dbias, geo)
                                                                                          : small_bwd_launch<32, false>(a, X, dz, dW, dbias, geo);
    }
    if (dX) {
        const SmallSource src{gp ? gp : g, sloped ? (gp ? y_pooled : y) : nullptr, gp ? mask : nullptr, act};
        s = small_run(src, Wt, nullptr, dX, NB, F, OH, OW, C, H, W, 2 - ph, 2 - pw, 1, SEERA_ACT_NONE, "conv2d_small_bwd(dX)");
    }
    if (!s && dW) {
        FirstGeom geo{NB, C, H, W, F, 3, 3, 1, 1, ph, pw, OH, OW, C * 9};
        s = first_dw(X, DzSource{nullptr, g, gp, mask, y, act, y_pooled}, dW, dbias, geo, "conv2d_small_bwd(dW)");
    }
    return s;
}

}  // namespace seera
