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
#include "conv_dw_block.cuh"
#include "internal.h"

namespace seera {

template <int C, int ST, int FL, bool POOLED>
__global__ void __launch_bounds__(256, 2) first_dw_kernel(const __grid_constant__ DwArgs a) {
    extern __shared__ __align__(16) float sm[];
    first_dw_block<C, ST, FL, POOLED>(a, blockIdx.x, blockIdx.y, blockIdx.z, sm);
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
    DwArgs d = dw_args<C, ST, FL, POOLED>(a.X, *a.src, g);
    float *partial = d.partial = (float *)scratch_alloc(dw_partial_bytes<C>(d));
    if (!partial) return SEERA_E_OOM;
    const int nblocks = d.nblocks;
    cudaStream_t st = rt().stream;
    profile_begin();
    auto kern = first_dw_kernel<C, ST, FL, POOLED>;
    cudaError_t e = allow_smem((const void *)kern, d.smem);
    if (e == cudaSuccess) {
        kern<<<dim3((unsigned)nblocks, (unsigned)d.chunks, (unsigned)d.cgroups), 256, d.smem, st>>>(d);
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
