// Gradient launcher of one (bra class, ket class) pair (AIMD_CLASS = 0..5: ss, ps, pp, ds, dp, dd;
// AIMD_KET = 0..AIMD_CLASS) and one arithmetic type (AIMD_REAL = 0: FP64; 1: FP32 quartets of the
// mixed-precision path).
#include "hf_launch.h"

#ifndef AIMD_CLASS
#error "compile with -DAIMD_CLASS=<0..5>"
#endif
#ifndef AIMD_KET
#error "compile with -DAIMD_KET=<0..AIMD_CLASS>"
#endif
#ifndef AIMD_REAL
#define AIMD_REAL 0
#endif
#define AIMD_CAT2(a, b) a##b
#define AIMD_CAT(a, b) AIMD_CAT2(a, b)

namespace hf {

constexpr int CX = AIMD_CLASS;
constexpr int CY = AIMD_KET;
static_assert(CY <= CX, "ket class above bra class");

#if AIMD_REAL == 0
using RT = double;
#define AIMD_GRAD_NAME AIMD_CAT(AIMD_CAT(AIMD_CAT(launch_grad_c, AIMD_CLASS), _), AIMD_KET)
#else
using RT = float;
#define AIMD_GRAD_NAME AIMD_CAT(AIMD_CAT(AIMD_CAT(launch_grad32_c, AIMD_CLASS), _), AIMD_KET)
#endif

template <int X, int Y, typename T>
size_t grad_bytes(const LaunchEnv& e, const LaunchSlot& s) {
    return grad_smem_bytes<X, Y, T>(e.natm, s.nx, e.nao, e.maxbp[X],
                                    grad_rbuf_elems<X, Y, T>(s.threads, e.maxbp[X], e.maxbp[Y]), s.dglobal != 0);
}

cudaError_t AIMD_GRAD_NAME(const LaunchEnv& e, const GradArgs& a0) {
    const int cnt = e.cls_count[CX];
    if (cnt == 0 || e.cls_count[CY] == 0) return cudaSuccess;
    constexpr int rt = sizeof(RT) == sizeof(double) ? 0 : 1;
    GradArgs a = a0;
    const void* kernel = (const void*)grad2e_bra_kernel<CX, CY, RT>;
    LaunchSlot& slot = e.slot(1, rt, CX, CY);
    if (slot.grid == 0 || slot.nx != a.nx) {
        slot.nx = a.nx;
        const cudaError_t r = class_shape(kernel, e, 1, CX, slot, grad_bytes<CX, CY, RT>);
        if (r != cudaSuccess) {
            slot.grid = 0;
            return r;
        }
    }
    a.rbuf = grad_rbuf_elems<CX, CY, RT>(slot.threads, e.maxbp[CX], e.maxbp[CY]);
    a.dglobal = slot.dglobal;
    a.plan = e.plan_of(CX, CY, rt);
    grad2e_bra_kernel<CX, CY, RT><<<slot.grid, slot.threads, slot.smem, e.stream_of(CX, CY)>>>(a);
    return cudaGetLastError();
}

}  // namespace hf
