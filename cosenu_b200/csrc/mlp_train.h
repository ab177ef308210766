// Launch interface of the fused training kernels (mlp_train.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstddef>

#include "mlp_math.cuh"

namespace mlptrain {

constexpr int MAXL = 8;

// One minibatch step.  Layer l has weights [dout][din] at woff and biases at
// boff of the flat parameter vectors.
struct Args {
    int nl, rows;
    int din[MAXL], dout[MAXL];
    size_t woff[MAXL], boff[MAXL];
    float *w, *m1, *m2;      // FP32 master parameters and AdamW moments
    __nv_bfloat16 *wb;       // BF16 copy of w
    const __nv_bfloat16 *x;  // [rows][din[0]]
    const float *t;          // [rows][dout[nl - 1]]
    float *z[MAXL];          // pre-activations of the hidden layers
    __nv_bfloat16 *h[MAXL];  // their activations
    __nv_bfloat16 *dz[MAXL]; // loss gradients with respect to the pre-activations
    float *loss;             // [loss_tiles()] partial sums of (y - t)^2
    float scale;             // 1 / (rows * n_out)
    mlpmath::AdamW opt;
    int *err;
};

// Whether the kernels take this network and batch.
bool fits(int nl, const int *din, const int *dout, int rows);
int loss_tiles(int n_out);
// Sets the kernels' shared-memory limit on the current device (before step).
cudaError_t prepare();
// Queues one training step on s; chained: the previous operation there is a step
// of the same call.
cudaError_t step(const Args &a, cudaStream_t s, bool chained);

}  // namespace mlptrain
