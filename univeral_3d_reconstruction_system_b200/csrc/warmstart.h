// warmstart.h - learned warm-start network: sizes and launch interface (see warmstart.cu).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/u3dg.h"

namespace u3dg {

constexpr int kWarmInputs = 134;
constexpr int kWarmHidden = 128;
constexpr int kWarmOutputs = 11;
constexpr int kWarmNeighbours = 16;
constexpr int kWarmViews = 7;
// Layer l maps kWarmIn[l] -> kWarmOut[l]; parameters are W (out x in) then b, layer after layer.
constexpr int kWarmLayers = 4;
constexpr int kWarmIn[kWarmLayers] = {kWarmInputs, kWarmHidden, kWarmHidden, kWarmHidden};
constexpr int kWarmOut[kWarmLayers] = {kWarmHidden, kWarmHidden, kWarmHidden, kWarmOutputs};
constexpr int kWarmParams = kWarmInputs * kWarmHidden + kWarmHidden + 2 * (kWarmHidden * kWarmHidden + kWarmHidden) +
                            kWarmHidden * kWarmOutputs + kWarmOutputs; // 51,723

void launchKnn(const float *queries, int nq, const float *points, int np, int k, int excludeSelf, int *idx, float *d2,
               cudaStream_t s);
size_t warmViewRefBytes();
void fillWarmViewRef(void *dst, const u3dg_camera &cam, const uint8_t *rgbDev);
void launchWarmFeatures(const float *xyz, const float *rgb, int n, const int *nbr, const float *nd2,
                        const float *baseScale, const void *views, int nViews, float *feat, cudaStream_t s);
// y (n x out) = x (n x in) W^T + b, then ReLU (relu).
void launchLayer(const float *x, int in, const float *W, const float *b, float *y, int out, int n, bool relu,
                 cudaStream_t s);
// dIn (n x in) = dOut (n x out) W, zero where the layer's input activation act is not positive.
void launchLayerInputGrad(const float *dOut, int out, const float *W, int in, const float *act, float *dIn, int n,
                          cudaStream_t s);
// One partial gradient per row chunk of a layer's weights and biases, at offsets w and b of
// parameter-sized arrays (partial: gradPartialEntries(n) floats); launchReduceGrad adds the chunks of
// every parameter in chunk order once all layers are done.
constexpr int kGradChunks = 64;
void launchLayerParamGrad(const float *dOut, int out, const float *act, int in, int n, float *partial, size_t w,
                          size_t b, cudaStream_t s);
void launchReduceGrad(const float *partial, int n, float *grad, cudaStream_t s);
size_t gradPartialEntries(int n);
int mseBlocks();
void launchMse(const float *y, const float *t, const float *w, int n, float *dy, double *partial, float *lossOut,
               cudaStream_t s);
void launchAdamFlat(float *p, const float *g, float *m, float *v, int n, float stepSize, float invSqrtBc2, float eps,
                    cudaStream_t s);
void launchGatherRows(const float *src, int width, const int *rows, int n, float *dst, cudaStream_t s);
void launchWarmCombine(const float *pred, int n, float *scales, float *quats, float *opac, float *colors,
                       cudaStream_t s);

} // namespace u3dg
