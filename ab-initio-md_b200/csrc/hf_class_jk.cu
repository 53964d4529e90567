// J/K and Schwarz launchers of one bra pair class (AIMD_CLASS = 0..5: ss, ps, pp, ds, dp, dd) and one
// arithmetic type (AIMD_REAL = 0: FP64 J/K + Schwarz; 1: FP32 J/K quartets of the mixed-precision path).
#include "hf_launch.h"

#ifndef AIMD_CLASS
#error "compile with -DAIMD_CLASS=<0..5>"
#endif
#ifndef AIMD_REAL
#define AIMD_REAL 0
#endif
#define AIMD_CAT2(a, b) a##b
#define AIMD_CAT(a, b) AIMD_CAT2(a, b)

namespace hf {

constexpr int CX = AIMD_CLASS;
using Q0 = QClass<CX, 0>;

#if AIMD_REAL == 0
using RT = double;
#define AIMD_JK_NAME AIMD_CAT(launch_jk_c, AIMD_CLASS)

cudaError_t AIMD_CAT(launch_schwarz_c, AIMD_CLASS)(const LaunchEnv& e, const QuartetArgs& q, cudaStream_t st) {
    const int cnt = e.cls_count[CX];
    if (cnt == 0) return cudaSuccess;
    const size_t smem = sizeof(double) * (size_t)e.maxbp[CX] * (bra_e_size<Q0::LA, Q0::LB>() + SBW);
    cudaError_t r = set_smem_limit((const void*)schwarz_kernel<CX>, smem);
    if (r != cudaSuccess) return r;
    schwarz_kernel<CX><<<cnt, SCHWARZ_THREADS, smem, st>>>(q, e.by_class + e.cls_start[CX], e.Q);
    return cudaGetLastError();
}
#else
using RT = float;
#define AIMD_JK_NAME AIMD_CAT(launch_jk32_c, AIMD_CLASS)
#endif

// One (class, ket class, type) launch. Every class unit instantiates it for its
// own class, so class and type are template arguments: an internal name alone
// does not keep the units' copies apart (the compiler makes it from a hash of
// the unit, which two units of one source compiled at once can share).
template <int X, int YK, typename T>
size_t jk_bytes(const LaunchEnv& e, const LaunchSlot& s) {
    constexpr int Y = YK < 0 ? 0 : YK;
    return jk_smem_bytes<X, Y, T>(s.threads, e.nao, e.maxbp[X], jk_rbuf_elems<X, YK, T>(e.maxbp[X], e.maxbp[Y]),
                                     s.kglobal != 0, s.dglobal != 0);
}
template <int X, int YK, typename T>
cudaError_t launch_one(const LaunchEnv& e, const JKArgs& a0) {
    constexpr int Y = YK < 0 ? 0 : YK;
    constexpr int rt = sizeof(T) == sizeof(double) ? 0 : 1;
    JKArgs a = a0;
    a.rbuf = jk_rbuf_elems<X, YK, T>(e.maxbp[X], e.maxbp[Y]);
    const void* kernel = (const void*)jk_bra_kernel<X, T, YK>;
    LaunchSlot& slot = e.slot(0, rt, X, Y);
    if (slot.grid == 0) {
        slot.kglobal = a.kglobal;
        const cudaError_t r = class_shape(kernel, e, 0, X, slot, jk_bytes<X, YK, T>);
        if (r != cudaSuccess) return r;
    }
    a.kglobal = slot.kglobal;
    a.dglobal = slot.dglobal;
    a.plan = e.plan_of(X, Y, rt);
    jk_bra_kernel<X, T, YK><<<slot.grid, slot.threads, slot.smem, e.stream_of(X, Y)>>>(a);
    return cudaGetLastError();
}

// split bra classes: one launch per non-empty ket class (largest first); ss: one
// launch, whose only ket class is ss
cudaError_t AIMD_JK_NAME(const LaunchEnv& e, const JKArgs& a) {
    const int cnt = e.cls_count[CX];
    if (cnt == 0) return cudaSuccess;
    if constexpr (!JKKernel<CX>::SPLIT) {
        return launch_one<CX, -1, RT>(e, a);
    } else {
        cudaError_t r = cudaSuccess;
        if constexpr (CX >= 5) if (r == cudaSuccess && e.cls_count[5]) r = launch_one<CX, 5, RT>(e, a);
        if constexpr (CX >= 4) if (r == cudaSuccess && e.cls_count[4]) r = launch_one<CX, 4, RT>(e, a);
        if constexpr (CX >= 3) if (r == cudaSuccess && e.cls_count[3]) r = launch_one<CX, 3, RT>(e, a);
        if constexpr (CX >= 2) if (r == cudaSuccess && e.cls_count[2]) r = launch_one<CX, 2, RT>(e, a);
        if (r == cudaSuccess && e.cls_count[1]) r = launch_one<CX, 1, RT>(e, a);
        if (r == cudaSuccess && e.cls_count[0]) r = launch_one<CX, 0, RT>(e, a);
        return r;
    }
}

}  // namespace hf
