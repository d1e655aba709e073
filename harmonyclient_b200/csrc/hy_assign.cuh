// Nearest-centroid assignment of many rows (k-means and add) on the tensor
// cores, with the exact FP32 rule's answer (see hy_assign.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "hy_device.cuh"

namespace hy {

// Largest d the kernel's resident row tile takes.
constexpr int ASSIGN_DMAX = 256;

struct AssignWork {
    const void* cimg;      // split centroid image (launch_centroid_image)
    const float* cxn;      // [nlist] squared norms
    float* cmax;           // [4] maxima over the centroids (launch_centroid_image)
    int32_t* second;       // [n] the other candidate of a row with two, else -1
    int32_t* hard;         // [n] rows whose candidates did not fit
    int32_t* hard_count;   // [1]
    int* err;              // DEV_ERR_TIMEOUT when a wait gave up: rows are then left unwritten
    uint32_t wait_limit = WAIT_LIMIT;
};

// Tensor-core pass: per row its best centroid by score (labels), a second
// candidate where the bound leaves two, and the list of rows it leaves to the
// exact scores of every centroid.
cudaError_t launch_assign(const float* x, int n, int d, int nlist, int metric, const AssignWork& w, int nsm,
                          int64_t* labels, cudaStream_t s);
// Rows with two candidates get the better by exact score; score (may be
// null) gets every row's exact score against its label.
cudaError_t launch_assign_exact(const float* x, int n, int d, const float* cent, int metric, const AssignWork& w,
                                int64_t* labels, float* score, cudaStream_t s);

}  // namespace hy
