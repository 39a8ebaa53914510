// mps_lanes.cuh -- launches of the kernels with G lanes per particle.
//
// Each precision and each G is a translation unit of its own (mps_lanes.cu): a device module is
// loaded whole at the first launch from it, and these kernels are two thirds of the code. In one
// module with the rest the first handle of a precision took 24 to 28 ms to create, 4 to 5 before
// there were several lanes; a program now loads the lanes that its scenes use.
#pragma once
#include "mps_kernels.cuh"

namespace mps {

template <class R, class RN, int G> struct Lanes {
    using Args = PassArgs<R, RN>;
    static void pass_a(const Args& a, bool diag, bool tape, cudaStream_t st);
    static void pass_b(const Args& a, bool diag, cudaStream_t st);
    static void pass_c(const Args& a, bool diag, bool tape, bool corr, cudaStream_t st);
    static void gen(const Args& a, bool diag, bool tape, bool cls, const V4<R>* pos, const R* prs,
                    const int8_t* typ, cudaStream_t st);
    // VscTrm, ChkCol, MkPrs and PrsGrdTrm by themselves
    static void vsc(const Args& a, cudaStream_t st);
    static void col(const Args& a, cudaStream_t st);
    static void prs(const Args& a, cudaStream_t st);
    static void grd(const Args& a, bool corr, cudaStream_t st);
};

}  // namespace mps
