// zmid_launch.cuh -- launches of the fused z pass on the row layout
// (passes_zmid.cuh; instantiated in zmid.cu and, for lines with prime factors
// above 5, in generic_r13.cu and generic_r31.cu, compiled beside solver.cu).
#pragma once
#include <algorithm>

#include "generic_launch.cuh"
#include "passes_zmid.cuh"

namespace m3d {

// compile-time line lengths: a length with a kernel, and whole tiles of lines
// (NL = Nx Ny)
template <typename T>
bool zmid_rows_ok(int N, int C, long long NL);
// J2 (j2) or damage; the transforms in T
template <typename T>
cudaError_t zmid_rows_inelastic(int N, bool j2, int entries, cudaStream_t st, const GridDims& g,
                                const typename Cx<T>::t* tw, typename Cx<T>::t* sp, const MidJ2Args& op, Ctl* ctl,
                                double* part, const FinJ2& fin);
// the EM update of C components
template <typename T>
cudaError_t zmid_rows_em(int N, int C, int entries, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                         typename Cx<T>::t* sp, const MidEMArgs<T>& op, Ctl* ctl, double* part, const FinLinear& fin);

// any other length
template <int MaxR, typename T, int C, class Op, class Fin>
cudaError_t gen_zmid(int entries, cudaStream_t st, const GridDims& g, const LinePlan& p, const typename Cx<T>::t* tw,
                     typename Cx<T>::t* sp, const typename Op::Args& op, Ctl* ctl, int G, double* part, const Fin& fin) {
    auto kern = k_zmid_gen<T, C, Op, Fin, MaxR>;
    allow_smem(kern);
    const int nl = G / 2 * C;
    const size_t smem = (size_t)p.n * (1 + 2 * nl) * 2 * sizeof(T) + 16 + 32 * Op::NSUM * sizeof(double) + Op::smem_bytes(op.nph);
    const int grid = (int)std::min<long long>((g.NL + G - 1) / G, kZGenGrid);
    // at least two warps more than the butterflies need: the pointwise step has G Nz items
    kern<<<dim3(grid, entries), p.n * G > 2 * 256 ? 256 : 128, smem, st>>>(g, p, tw, sp, op, ctl, G, part, fin);
    return cudaGetLastError();
}

typedef MidEM<float, 1, 3> GMe3f; typedef MidEM<float, 1, 6> GMe6f; typedef MidEM<double, 1, 3> GMe3d; typedef MidEM<double, 1, 6> GMe6d;
typedef MidJ2<float, true> GMj2f; typedef MidJ2<double, true> GMj2d; typedef MidJ2<float, false> GMdf; typedef MidJ2<double, false> GMdd;
#define M3D_GEN_ZMID(EXT, R, T, C, OP, FIN)                                                                          \
    EXT template cudaError_t gen_zmid<R, T, C, OP, FIN>(int, cudaStream_t, const GridDims&, const LinePlan&,         \
                                                        const Cx<T>::t*, Cx<T>::t*, const OP::Args&, Ctl*, int,      \
                                                        double*, const FIN&);
#define M3D_GEN_ZMID_ALL(EXT, R)                                                                    \
    M3D_GEN_ZMID(EXT, R, float, 3, GMe3f, FinLinear) M3D_GEN_ZMID(EXT, R, float, 6, GMe6f, FinLinear) \
    M3D_GEN_ZMID(EXT, R, double, 3, GMe3d, FinLinear) M3D_GEN_ZMID(EXT, R, double, 6, GMe6d, FinLinear) \
    M3D_GEN_ZMID(EXT, R, float, 6, GMj2f, FinJ2) M3D_GEN_ZMID(EXT, R, double, 6, GMj2d, FinJ2)     \
    M3D_GEN_ZMID(EXT, R, float, 6, GMdf, FinJ2) M3D_GEN_ZMID(EXT, R, double, 6, GMdd, FinJ2)

}  // namespace m3d
