// Shared by the kernels for convolutions with a short patch, C*R*S <= 64 (conv_first.cu, conv_first_dw.cu).
#pragma once
#include "common.cuh"
#include "tc_ptx.cuh"

namespace seera {

struct FirstGeom {
    int NB, C, H, W, F, R, S, sh, sw, ph, pw, OH, OW, K;
    FastDiv by_P, by_OW, by_Pq, by_OWq;      // pixels per image, output width, and the same counted in 2x2 windows
};

// Where the weight gradient takes the output gradient dz[img][f][pixel] from: a stored fp32 tensor, or computed on the
// fly as dy * act'(y) with dy either a full-resolution gradient g or the gradient gp of a 2x2 / stride-2 max-pool of
// y routed through the pool's window-local argmax indices.
struct DzSource {
    const float *dz;            // stored gradient, or null
    const float *g, *gp;        // exactly one of these when dz is null
    const int *mask;
    const float *y;
    int act;
    const float *yp;            // with gp: the pool's output (y at each window's argmax), or null
};
__device__ __forceinline__ float first_slope(float y, int act) {
    switch (act) {
        case SEERA_ACT_RELU: return y > 0.f ? 1.f : 0.f;
        case SEERA_ACT_SIGMOID: return y * (1.f - y);
        case SEERA_ACT_TANH: return 1.f - y * y;
        default: return 1.f;
    }
}

constexpr int FIRST_FC = 64;        // filters per block pass

// dW (and dbias, if not null) of a 3 x 3 layer on CUDA cores in exact fp32 (conv_first_dw.cu)
bool first_dw_applies(const FirstGeom &g, const DzSource &src);
int first_dw(const float *X, const DzSource &src, float *dW, float *dbias, const FirstGeom &g, const char *name);
// Adds the blocks' partial sums [group of Kg taps][chunk of 64 filters][block][64][KP] in block order; column Kg holds the bias gradient.
void first_wgrad_reduce(const float *partial, float *dW, float *dbias, int F, int K, int Kg, int KP, int nblocks, cudaStream_t st);

}  // namespace seera
