// tcgen05 (sm_100a) inference kernels of the surrogate denoiser.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace cpb {

struct TcNetArgs {
    int n, h, w;               // frames and their size
    int strips;                // columns are walked in this many strips (set by tc_net)
    int bands, band_rows;      // narrow frames: bands of rows side by side, and a band's rows (set by tc_net)
    const void* rgba;          // dense RGBA frames [n][h][w][4]: the network's input and the residual's base
    void* out;                 // back half: the denoised frames (may be rgba)
    const float* ab;           // front half: n (a, b) noise-model pairs
    float sigma_scale;         // front half: scale of the noise map
    __nv_bfloat16* act;        // the fourth layer's output, bf16 planes [n][4][h][w][8]
    const __nv_bfloat16* weights[4];  // the half's packed forward weights, [cout][9 * cin padded to 16]
    const float* bias[4];
    int* err;                  // device int: nonzero when a pipeline wait ran out
};

// One half of the network: layers 0-3 (RGBA -> act) or 4-7 (act and RGBA ->
// out); binary16 frames when f16, else float32.
cudaError_t tc_net(bool front, bool f16, TcNetArgs a, cudaStream_t stream);

}  // namespace cpb
