// mps_lanes.cu -- the kernels with MPS_LANES lanes per particle, for state in MPS_REAL and number
// density in MPS_DENSITY. Compiled once for each.
#include <algorithm>

#include "mps_lanes.cuh"

namespace mps {

template <class R, class RN, int G> static unsigned lanes_grid(const PassArgs<R, RN>& a) {
    return std::max(1, (a.nF + 128 / G - 1) / (128 / G));
}

template <class R, class RN, int G>
void Lanes<R, RN, G>::pass_a(const Args& a, bool diag, bool tape, cudaStream_t st) {
    const unsigned n = lanes_grid<R, RN, G>(a);
    if (tape) k_pass_a_g<R, RN, false, true, G><<<n, 128, 0, st>>>(a);
    else if (diag) k_pass_a_g<R, RN, true, false, G><<<n, 128, 0, st>>>(a);
    else k_pass_a_g<R, RN, false, false, G><<<n, 128, 0, st>>>(a);
}

template <class R, class RN, int G>
void Lanes<R, RN, G>::pass_b(const Args& a, bool diag, cudaStream_t st) {
    const unsigned n = lanes_grid<R, RN, G>(a);
    if (diag) k_pass_b_g<R, RN, true, G><<<n, 128, 0, st>>>(a);
    else k_pass_b_g<R, RN, false, G><<<n, 128, 0, st>>>(a);
}

template <class R, class RN, int G>
void Lanes<R, RN, G>::pass_c(const Args& a, bool diag, bool tape, bool corr, cudaStream_t st) {
    const unsigned n = lanes_grid<R, RN, G>(a);
    if (tape) k_pass_c_g<R, RN, false, true, false, G><<<n, 128, 0, st>>>(a);
    else if (corr && diag) k_pass_c_g<R, RN, true, false, true, G><<<n, 128, 0, st>>>(a);
    else if (corr) k_pass_c_g<R, RN, false, false, true, G><<<n, 128, 0, st>>>(a);
    else if (diag) k_pass_c_g<R, RN, true, false, false, G><<<n, 128, 0, st>>>(a);
    else k_pass_c_g<R, RN, false, false, false, G><<<n, 128, 0, st>>>(a);
}

template <class R, class RN, int G>
void Lanes<R, RN, G>::gen(const Args& a, bool diag, bool tape, bool cls, const V4<R>* pos, const R* prs,
                          const int8_t* typ, cudaStream_t st) {
    const unsigned n = lanes_grid<R, RN, G>(a);
    if (tape && cls) k_gen_cull_g<R, RN, false, true, true, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
    else if (tape) k_gen_cull_g<R, RN, false, true, false, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
    else if (diag && cls) k_gen_cull_g<R, RN, true, false, true, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
    else if (diag) k_gen_cull_g<R, RN, true, false, false, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
    else if (cls) k_gen_cull_g<R, RN, false, false, true, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
    else k_gen_cull_g<R, RN, false, false, false, G><<<n, 128, 0, st>>>(a, pos, prs, typ);
}

template <class R, class RN, int G> void Lanes<R, RN, G>::vsc(const Args& a, cudaStream_t st) {
    k_pass_a_g<R, RN, false, false, G, true><<<lanes_grid<R, RN, G>(a), 128, 0, st>>>(a);
}
template <class R, class RN, int G> void Lanes<R, RN, G>::col(const Args& a, cudaStream_t st) {
    k_pass_b_g<R, RN, false, G, PASS_COL><<<lanes_grid<R, RN, G>(a), 128, 0, st>>>(a);
}
template <class R, class RN, int G> void Lanes<R, RN, G>::prs(const Args& a, cudaStream_t st) {
    k_pass_b_g<R, RN, false, G, PASS_PRS><<<lanes_grid<R, RN, G>(a), 128, 0, st>>>(a);
}
template <class R, class RN, int G> void Lanes<R, RN, G>::grd(const Args& a, bool corr, cudaStream_t st) {
    const unsigned n = lanes_grid<R, RN, G>(a);
    if (corr) k_pass_c_g<R, RN, false, false, true, G, true><<<n, 128, 0, st>>>(a);
    else k_pass_c_g<R, RN, false, false, false, G, true><<<n, 128, 0, st>>>(a);
}

template struct Lanes<MPS_REAL, MPS_DENSITY, MPS_LANES>;

}  // namespace mps
