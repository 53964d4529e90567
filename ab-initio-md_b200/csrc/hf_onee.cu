// Launchers of the one-electron kernels (one launch per shell-pair class).
#include "hf_launch.h"

namespace hf {

namespace {
// CTAs of a launch over n shell pairs, one warp each: as many as are
// resident at once; their warps walk the pairs with that stride.
int onee_grid(const void* kernel, size_t smem, int nsm, int n) {
    const int need = (n + ONEE_THREADS / 32 - 1) / (ONEE_THREADS / 32), fit = persistent_grid(kernel, ONEE_THREADS, smem, nsm);
    return need < fit ? need : fit;
}
template <int CL>
cudaError_t onee_class(const LaunchEnv& e, const ShellView& sv, int b0, int b1, const double* o, double* S, double* T,
                       double* M, double* V, cudaStream_t st) {
    const auto kernel = onee_kernel<cls_la(CL), cls_lb(CL)>;
    const size_t smem = sizeof(double) * BoysOf<cls_la(CL) + cls_lb(CL), double, true>::elems;
    const cudaError_t r = set_smem_limit((const void*)kernel, smem);
    if (r != cudaSuccess) return r;
    kernel<<<onee_grid((const void*)kernel, smem, e.nsm, b1 - b0), ONEE_THREADS, smem, st>>>(sv, b0, b1, o[0], o[1], o[2], S,
                                                                                             T, M, V);
    return cudaGetLastError();
}
template <int CL>
cudaError_t onee_grad_class(const LaunchEnv& e, const ShellView& sv, int b0, int b1, const double* W, const double* D,
                            facc* grad, cudaStream_t st) {
    const size_t acc = sizeof(facc) * 3 * e.natm;
    if (acc > 48 * 1024) return cudaErrorInvalidConfiguration;
    const auto kernel = onee_grad_kernel<cls_la(CL), cls_lb(CL)>;
    const size_t smem = acc + sizeof(double) * BoysOf<cls_la(CL) + cls_lb(CL) + 1, double, true>::elems;
    const cudaError_t r = set_smem_limit((const void*)kernel, smem);
    if (r != cudaSuccess) return r;
    kernel<<<onee_grid((const void*)kernel, smem, e.nsm, b1 - b0), ONEE_THREADS, smem, st>>>(sv, b0, b1, W, D, grad);
    return cudaGetLastError();
}
}  // namespace

#define AIMD_BY_CLASS(F, ...)                  \
    switch (cl) {                              \
        case 0: return F<0>(__VA_ARGS__);      \
        case 1: return F<1>(__VA_ARGS__);      \
        case 2: return F<2>(__VA_ARGS__);      \
        case 3: return F<3>(__VA_ARGS__);      \
        case 4: return F<4>(__VA_ARGS__);      \
        default: return F<5>(__VA_ARGS__);     \
    }

cudaError_t launch_onee(const LaunchEnv& e, const ShellView& sv, int cl, const int* sp_cls_start, const double* origin,
                        double* S, double* T, double* M, double* V, cudaStream_t st) {
    const int b0 = sp_cls_start[cl], b1 = sp_cls_start[cl + 1];
    if (b1 == b0) return cudaSuccess;
    const double o[3] = {origin ? origin[0] : 0.0, origin ? origin[1] : 0.0, origin ? origin[2] : 0.0};
    AIMD_BY_CLASS(onee_class, e, sv, b0, b1, o, S, T, M, V, st)
}

cudaError_t launch_onee_grad(const LaunchEnv& e, const ShellView& sv, int cl, const int* sp_cls_start, const double* W,
                             const double* D, facc* grad, cudaStream_t st) {
    const int b0 = sp_cls_start[cl], b1 = sp_cls_start[cl + 1];
    if (b1 == b0) return cudaSuccess;
    AIMD_BY_CLASS(onee_grad_class, e, sv, b0, b1, W, D, grad, st)
}
#undef AIMD_BY_CLASS

}  // namespace hf
