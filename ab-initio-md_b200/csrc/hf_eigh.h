// Launcher of the small symmetric eigensolver (hf_eigh.cu).
#pragma once
#include <cuda_runtime.h>

namespace hf {
cudaError_t launch_eigh(int n, const double* A, double* V, double* w, int warm, cudaStream_t st);
}
