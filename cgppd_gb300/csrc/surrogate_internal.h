// surrogate_internal.h -- declarations shared by the surrogate's kernels and host code.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "surrogate.cuh"

struct cgppd_surrogate;

namespace cgppd {

constexpr int kNetRows = 64;                       // batch rows of one tile
constexpr int kNetTileElems = kSurH * kNetRows;    // a 256 x 64 bf16 tile image (tc05.cuh)

// Tile images of a batch, [kind][tile][256 x 64]: activations of layers 1..4 and
// pre-activation gradients of layers 1..4.
enum NetAct { kActH1 = 0, kActZ1 = 4, kActKinds = 8 };

struct NetRowsArgs {
    const float *X;                // [..][8] features
    const float *y;                // targets (backward; forward: or null)
    const int *perm;               // row -> row of X and y (targets then clipped to +-clip), or null
    float clip;
    int rows;
    const float *P;                // FP32 master parameters
    const __nv_bfloat16 *wtiles;   // [6][4][256 x 64]: W2 W3 W4, then their transposes W4 W3 W2
    float *o;                      // [rows] predictions, or null
    __nv_bfloat16 *act;            // [kActKinds][tiles][256 x 64] (backward)
    float *xb;                     // (backward) the batch's features, [8][rows]
    float *dO, *r2;                // (with targets) 2 (o - y) / rows; (o - y)^2
    unsigned *err;
};

struct NetWgradArgs {
    const __nv_bfloat16 *act;
    int tiles, splits, split_tiles;  // tiles = splits * split_tiles
    float *part;                     // [3][splits][256][256]
    unsigned *err;
};

struct NetUpdateArgs {
    const float *wpart;   // of k_net_wgrad
    int splits;
    const __nv_bfloat16 *act;  // of k_net_rows, and its xb, dO, r2
    const float *xb, *dO, *r2;
    int rows;
    int first;            // first block of the work (set by the launcher)
    float *G;             // gradient (no Adam step)
    float *loss_sum;      // sum of squared residuals
    float *P, *m, *v;     // Adam
    float lr, b1, b2, eps, c1, c2;
    __nv_bfloat16 *Wf, *wtiles;
};

// What k_net_update does with the sums: end the loss alone, store the gradient, or take
// an Adam step.
enum NetUpdateMode { kNetLossOnly = 0, kNetGradient, kNetAdam };

cudaError_t net_set_limits();
cudaError_t launch_net_rows(const NetRowsArgs &a, bool backward, int max_ctas, cudaStream_t st);
cudaError_t launch_net_wgrad(const NetWgradArgs &a, cudaStream_t st);
cudaError_t launch_net_update(const NetUpdateArgs &a, NetUpdateMode mode, cudaStream_t st);
cudaError_t launch_net_copies(const float *P, __nv_bfloat16 *Wf, __nv_bfloat16 *wtiles, cudaStream_t st);

// perm[0 .. n): the shuffle of 0 .. n - 1 that splitmix64 from `state` gives (permutation.cu;
// n - 1 words are used).  partner, place: n words each; left: 3 words.
cudaError_t launch_permutation(int n, uint64_t state, int *perm, int *partner, unsigned long long *place,
                               unsigned *left, int max_ctas, cudaStream_t st);

// The engine reads a trained surrogate's FP32 parameters and BF16 forward weights.
const float *surrogate_device_params(const cgppd_surrogate *s);
const __nv_bfloat16 *surrogate_device_wf(const cgppd_surrogate *s);
// Append n samples held in device memory (features [n][8], energies [n]).
int surrogate_append_device_samples(cgppd_surrogate *s, const float *dX, const float *dY, int n);

}  // namespace cgppd
