// The surrogate's tensor-core kernels (C = 24), as surrogate.cu calls them.
// dims: nx, ny, nz, batch; ghosted buffers: tc_ghost_bytes each.
#ifndef LGD_CONV_TC_H
#define LGD_CONV_TC_H

#include <cuda_runtime.h>
#include <stddef.h>

namespace lgd {
namespace sur {

// packed weights: forward per layer, input gradient of layers 2 .. 4 (training)
struct TcWeights {
    void *base;
    void *fwd[4];
    void *grad[4];
};

bool tc_applicable(int nx, int ny, int channels);
size_t tc_ghost_bytes(int nx, int ny, int nz, int batch);
TcWeights tc_alloc_weights(bool training);
void tc_free_weights(TcWeights& w);
void tc_pack_weights(const float *const layer[4], const TcWeights& w, cudaStream_t stream);

// layer 1 (u, kappa -> 24), layers 2 and 3 (24 -> 24): ghosted BF16 output;
// gelu_grad (or null) receives GELU' of the pre-activations for the backward
// pass
void tc_layer1(const float *u, const float *k, const void *w, const float *bias, void *out, float *gelu_grad, const int dims[4],
               int *err, cudaStream_t stream);
void tc_layer_mid(const void *in, const void *w, const float *bias, void *out, float *gelu_grad, const int dims[4], int *err,
                  cudaStream_t stream);
// layer 4 (24 -> 1): out = conv + bias, or out += that; copy (or null)
// receives conv + bias
void tc_layer_last(const void *in, const void *w, const float *bias, float *out, bool add, float *copy, const int dims[4],
                   int *err, cudaStream_t stream);

// input gradients: dz of the layer below = conv_t(dz) * gelu_grad, ghosted, and
// its sum over the voxels added to db.  The last layer's takes the loss
// gradient scale * (du - target) itself
void tc_grad_mid(const void *dz, const void *w, const float *gelu_grad, void *out, float *db, const int dims[4], int *err,
                 cudaStream_t stream);
void tc_grad_last(const float *du, const float *target, float scale, const void *w, const float *gelu_grad, void *out, float *db,
                  const int dims[4], int *err, cudaStream_t stream);

// weight gradients of layer 0 (x0: BF16 pairs u, kappa; dz), 1 and 2 (h the
// layer's input, dz), 3 (h, du, target, scale): each CTA's share into its
// slice of partials (tc_partial_floats); returns the CTAs.  tc_wgrad_reduce
// sums all layers' shares into grads.  Layer 3 also adds the sum of (du -
// target)^2 to loss and the output bias' gradient to db.
size_t tc_partial_floats();
int tc_wgrad(int layer, const void *h, const void *x0, const void *dz, const float *du, const float *target, float scale,
             double *loss, float *db, float *partials, const int dims[4], int *err, cudaStream_t stream);
void tc_wgrad_reduce(const float *partials, const int ctas[4], const long long w_off[4], float *grads,
                     cudaStream_t stream);

// floats of a layer's gelu_grad
inline size_t tc_gelu_grad_floats(int nx, int ny, int nz, int batch) { return (size_t)nx * ny * nz * batch * 24; }

}  // namespace sur
}  // namespace lgd

#endif
