// generic_launch.cuh -- launches of the generic passes (passes.cuh) by the
// largest radix their line plan needs.
//
// Each generic pass is compiled three times: with compile-time butterflies up
// to radix 5, up to 13 and up to 31.  A kernel that holds a radix-31 butterfly
// needs its registers on every length (an FP64 one 200 and more, one CTA per
// SM instead of two or three), while a radix the kernel does not hold runs the
// run-time butterfly, whose inputs live in local memory.  So a length takes the
// smallest variant that holds all its radices.  Measured: FP64 thermal 65^3
// (65 = 5 x 13) 6.81 -> 3.12 ms a solve (1.8 with fewer stages and the stage
// constants of fft_smem.cuh), 28^3 (radix 7) batch homogenization 17.7 -> 11.9 ms.
// Lengths of the factors 2, 3 and 5 run the radix-5 variant.
// The radix-13 and radix-31 variants are instantiated in generic_r13.cu and
// generic_r31.cu, compiled beside solver.cu.
#pragma once
#include "inelastic.cuh"
#include "passes.cuh"
#include "physics.cuh"
#include "smem_limit.cuh"

namespace m3d {

// The variant of a plan: the smallest that holds its odd radices (primes up to 31).
inline int max_radix(const LinePlan& p) {
    int r = 5;
    for (int s = 0; s < p.nstages; ++s)
        if (p.radix[s] % 2 && p.radix[s] % 3 && p.radix[s] % 5 && p.radix[s] > r) r = p.radix[s];  // a prime above 5
    return r <= 5 ? 5 : (r <= 13 ? 13 : 31);
}
template <int R> struct RadixC { static constexpr int value = R; };
template <class F> void with_radix(const LinePlan& p, F&& f) {
    switch (max_radix(p)) {
        case 5: f(RadixC<5>{}); break;
        case 13: f(RadixC<13>{}); break;
        default: f(RadixC<31>{}); break;
    }
}

template <int MaxR, typename T, int C, class Pro>
void gen_zfwd(dim3 grid, int nt, size_t smem, cudaStream_t st, const GridDims& g, const LinePlan& p,
              const typename Cx<T>::t* tw, typename Cx<T>::t* sp, const Pro& pro, const Ctl* ctl, int G, double* part) {
    allow_smem(k_zfwd<T, C, Pro, MaxR>);
    k_zfwd<T, C, Pro, MaxR><<<grid, nt, smem, st>>>(g, p, tw, sp, pro, ctl, G, part);
}
template <int MaxR, typename T>
void gen_y(dim3 grid, int nt, size_t smem, cudaStream_t st, const GridDims& g, const LinePlan& p,
           const typename Cx<T>::t* tw, typename Cx<T>::t* sp, FastDiv tz, FastDiv ntz, int CC, int sign, const Ctl* ctl) {
    allow_smem(k_ypass<T, MaxR>);
    k_ypass<T, MaxR><<<grid, nt, smem, st>>>(g, p, tw, sp, tz, ntz, CC, sign, ctl);
}
template <int MaxR, typename T, int C, class Spec>
void gen_x(dim3 grid, int nt, size_t smem, cudaStream_t st, const GridDims& g, const LinePlan& p,
           const typename Cx<T>::t* tw, typename Cx<T>::t* sp, FastDiv tz, FastDiv ntz, const Spec& op, const Ctl* ctl, double* part) {
    allow_smem(k_xturn<T, C, Spec, MaxR>);
    k_xturn<T, C, Spec, MaxR><<<grid, nt, smem, st>>>(g, p, tw, sp, tz, ntz, op, ctl, part);
}
template <int MaxR, typename T, int C, class Epi, class Fin>
void gen_zinv(dim3 grid, int nt, size_t smem, cudaStream_t st, const GridDims& g, const LinePlan& p,
              const typename Cx<T>::t* tw, const typename Cx<T>::t* sp, const Epi& epi, Ctl* ctl, int G, double* part,
              const Fin& fin) {
    allow_smem(k_zinv<T, C, Epi, Fin, MaxR>);
    k_zinv<T, C, Epi, Fin, MaxR><<<grid, nt, smem, st>>>(g, p, tw, sp, epi, ctl, G, part, fin);
}

// every generic launch the solver makes, for one MaxR (explicit instantiation
// declarations and definitions)
#define M3D_GEN_ZFWD(EXT, R, T, C, PRO)                                                                              \
    EXT template void gen_zfwd<R, T, C, PRO>(dim3, int, size_t, cudaStream_t, const GridDims&, const LinePlan&,           \
                                             const Cx<T>::t*, Cx<T>::t*, const PRO&, const Ctl*, int, double*);
#define M3D_GEN_Y(EXT, R, T)                                                                                         \
    EXT template void gen_y<R, T>(dim3, int, size_t, cudaStream_t, const GridDims&, const LinePlan&, const Cx<T>::t*,     \
                                  Cx<T>::t*, FastDiv, FastDiv, int, int, const Ctl*);
#define M3D_GEN_X(EXT, R, T, C, SPEC)                                                                                \
    EXT template void gen_x<R, T, C, SPEC>(dim3, int, size_t, cudaStream_t, const GridDims&, const LinePlan&,             \
                                           const Cx<T>::t*, Cx<T>::t*, FastDiv, FastDiv, const SPEC&, const Ctl*, double*);
#define M3D_GEN_ZINV(EXT, R, T, C, EPI, FIN)                                                                         \
    EXT template void gen_zinv<R, T, C, EPI, FIN>(dim3, int, size_t, cudaStream_t, const GridDims&, const LinePlan&,      \
                                                  const Cx<T>::t*, const Cx<T>::t*, const EPI&, Ctl*, int, double*,  \
                                                  const FIN&);
typedef ProMat<float, 3> GPm3f; typedef ProMat<float, 6> GPm6f; typedef ProMat<double, 3> GPm3d; typedef ProMat<double, 6> GPm6d;
typedef SpecGreen<float, 3> GSg3f; typedef SpecGreen<float, 6> GSg6f; typedef SpecGreen<double, 3> GSg3d; typedef SpecGreen<double, 6> GSg6d;
typedef SpecEqVar<float, 3> GSe3f; typedef SpecEqVar<float, 6> GSe6f; typedef SpecEqVar<double, 3> GSe3d; typedef SpecEqVar<double, 6> GSe6d;
typedef EpiEM<float, 3> GEe3f; typedef EpiEM<float, 6> GEe6f; typedef EpiEM<double, 3> GEe3d; typedef EpiEM<double, 6> GEe6d;
#define M3D_GEN_ALL(EXT, R)                                                                   \
    M3D_GEN_ZFWD(EXT, R, float, 3, GPm3f) M3D_GEN_ZFWD(EXT, R, float, 6, GPm6f)               \
    M3D_GEN_ZFWD(EXT, R, double, 3, GPm3d) M3D_GEN_ZFWD(EXT, R, double, 6, GPm6d)             \
    M3D_GEN_ZFWD(EXT, R, double, 3, ProRefine64<3>) M3D_GEN_ZFWD(EXT, R, double, 6, ProRefine64<6>) \
    M3D_GEN_ZFWD(EXT, R, float, 6, ProStress<float>) M3D_GEN_ZFWD(EXT, R, double, 6, ProStress<double>) \
    M3D_GEN_Y(EXT, R, float) M3D_GEN_Y(EXT, R, double)                                        \
    M3D_GEN_X(EXT, R, float, 3, GSg3f) M3D_GEN_X(EXT, R, float, 6, GSg6f)                     \
    M3D_GEN_X(EXT, R, double, 3, GSg3d) M3D_GEN_X(EXT, R, double, 6, GSg6d)                   \
    M3D_GEN_X(EXT, R, float, 3, GSe3f) M3D_GEN_X(EXT, R, float, 6, GSe6f)                     \
    M3D_GEN_X(EXT, R, double, 3, GSe3d) M3D_GEN_X(EXT, R, double, 6, GSe6d)                   \
    M3D_GEN_X(EXT, R, float, 6, SpecBasic<float>) M3D_GEN_X(EXT, R, double, 6, SpecBasic<double>) \
    M3D_GEN_ZINV(EXT, R, float, 3, GEe3f, FinLinear) M3D_GEN_ZINV(EXT, R, float, 6, GEe6f, FinLinear) \
    M3D_GEN_ZINV(EXT, R, double, 3, GEe3d, FinLinear) M3D_GEN_ZINV(EXT, R, double, 6, GEe6d, FinLinear) \
    M3D_GEN_ZINV(EXT, R, double, 3, EpiDefect<3>, FinLinear) M3D_GEN_ZINV(EXT, R, double, 6, EpiDefect<6>, FinLinear) \
    M3D_GEN_ZINV(EXT, R, float, 6, EpiBasic<float>, FinJ2) M3D_GEN_ZINV(EXT, R, double, 6, EpiBasic<double>, FinJ2)

}  // namespace m3d
