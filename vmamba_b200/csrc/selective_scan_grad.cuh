// The selective-scan gradients for 1 .. 16 states (selective_scan_grad.cu), as the entry point in selective_scan_bwd.cu calls them.
#pragma once
#include "common.cuh"

namespace ss2d {

// Where the partial sums of a backward pass lie, for the kernel that folds them.
struct BwdFold {
    const float *rowred, *bcpart;
    int64_t images;      // partials per row: images, times segments
    int64_t Lp;          // floats per row of bcpart
    int parts;
};

bool selective_scan_grad_takes(const ss2d_scan_bwd_params* p);
long long selective_scan_grad_workspace_bytes(const ss2d_scan_bwd_params* p);
int selective_scan_grad(const ss2d_scan_bwd_params* p, BwdFold& fold, cudaStream_t st);

}  // namespace ss2d
