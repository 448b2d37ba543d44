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
int tc_pack_weights(const float *const layer[4], const TcWeights& w, cudaStream_t stream);   // launches made

// layer 1 (u, kappa -> 24), layers 2 and 3 (24 -> 24): ghosted BF16 output;
// z (or null) receives the pre-activations for the backward pass
void tc_layer1(const float *u, const float *k, const void *w, const float *bias, void *out, float *z, const int dims[4],
               int *err, cudaStream_t stream);
void tc_layer_mid(const void *in, const void *w, const float *bias, void *out, float *z, const int dims[4], int *err,
                  cudaStream_t stream);
// layer 4 (24 -> 1): out = conv + bias, or out += that
void tc_layer_last(const void *in, const void *w, const float *bias, float *out, bool add, const int dims[4], int *err,
                   cudaStream_t stream);

}  // namespace sur
}  // namespace lgd

#endif
