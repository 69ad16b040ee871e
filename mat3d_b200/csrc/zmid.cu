// zmid.cu -- the fused z pass on the row layout: kernels and launches.
#include "zmid_launch.cuh"

namespace m3d {

namespace {
template <int NN> struct IntC { static constexpr int value = NN; };
template <class F> void with_n(int n, F&& f) {
    switch (n) {
        case 32: f(IntC<32>{}); break;
        case 48: f(IntC<48>{}); break;
        case 64: f(IntC<64>{}); break;
        case 96: f(IntC<96>{}); break;
        case 128: f(IntC<128>{}); break;
        case 256: f(IntC<256>{}); break;
        default: break;
    }
}
template <typename T, int NN, int C, class Op, class Fin>
cudaError_t go(int entries, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw, typename Cx<T>::t* sp,
               const typename Op::Args& op, Ctl* ctl, double* part, const Fin& fin) {
    typedef ZRowsGeom<T, NN, C> Z;
    auto kern = k_zmid_rows<T, NN, C, Op, Fin>;
    allow_smem(kern);
    kern<<<dim3((unsigned)std::min<long long>(g.NL / Z::G, kZRowsGrid), entries), Z::NT, Z::template smem<Op>(op.nph), st>>>(g, tw, sp, op, ctl, part, fin);
    return cudaGetLastError();
}
}  // namespace

// The EM kernels are for the shapes that the two-pass sweeps (passes_plane.cuh,
// passes_slab.cuh) do not cover.  Of those, five passes remain for lines of 32, 48
// and 64 points, of 96 in FP32, and of 128 in FP32 thermal solves: grids whose other
// lengths keep them from two passes.
template <typename T, int C, class F> void with_em_n(int n, F&& f) {
    switch (n) {
        case 96: if constexpr (sizeof(T) == 8) f(IntC<96>{}); break;
        case 128: if constexpr (sizeof(T) == 8 || C == 6) f(IntC<128>{}); break;
        case 256: f(IntC<256>{}); break;
        default: break;
    }
}
template <typename T>
bool zmid_rows_ok(int N, int C, long long NL) {
    bool ok = false;
    if (C == 6) with_n(N, [&](auto nc) { ok = NL % ZRowsGeom<T, decltype(nc)::value, 6>::G == 0; });
    else with_em_n<T, 3>(N, [&](auto nc) { ok = NL % ZRowsGeom<T, decltype(nc)::value, 3>::G == 0; });
    return ok;
}
template bool zmid_rows_ok<float>(int, int, long long);
template bool zmid_rows_ok<double>(int, int, long long);

template <typename T>
cudaError_t zmid_rows_em(int N, int C, int entries, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                         typename Cx<T>::t* sp, const MidEMArgs<T>& op, Ctl* ctl, double* part, const FinLinear& fin) {
    cudaError_t e = cudaErrorInvalidValue;
    constexpr int W = sizeof(T) == 4 ? 2 : 1;
    if (C == 6)
        with_em_n<T, 6>(N, [&](auto nc) {
            e = go<T, decltype(nc)::value, 6, MidEM<T, W, 6>, FinLinear>(entries, st, g, tw, sp, op, ctl, part, fin);
        });
    else
        with_em_n<T, 3>(N, [&](auto nc) {
            e = go<T, decltype(nc)::value, 3, MidEM<T, W, 3>, FinLinear>(entries, st, g, tw, sp, op, ctl, part, fin);
        });
    return e;
}
template cudaError_t zmid_rows_em<float>(int, int, int, cudaStream_t, const GridDims&, const float2*, float2*,
                                         const MidEMArgs<float>&, Ctl*, double*, const FinLinear&);
template cudaError_t zmid_rows_em<double>(int, int, int, cudaStream_t, const GridDims&, const double2*, double2*,
                                          const MidEMArgs<double>&, Ctl*, double*, const FinLinear&);

M3D_GEN_ZMID_ALL(, 5)

template <typename T>
cudaError_t zmid_rows_inelastic(int N, bool j2, int entries, cudaStream_t st, const GridDims& g,
                                const typename Cx<T>::t* tw, typename Cx<T>::t* sp, const MidJ2Args& op, Ctl* ctl,
                                double* part, const FinJ2& fin) {
    cudaError_t e = cudaErrorInvalidValue;
    with_n(N, [&](auto nc) {
        constexpr int NN = decltype(nc)::value;
        e = j2 ? go<T, NN, 6, MidJ2<T, true>, FinJ2>(entries, st, g, tw, sp, op, ctl, part, fin)
               : go<T, NN, 6, MidJ2<T, false>, FinJ2>(entries, st, g, tw, sp, op, ctl, part, fin);
    });
    return e;
}
template cudaError_t zmid_rows_inelastic<float>(int, bool, int, cudaStream_t, const GridDims&, const float2*, float2*,
                                                const MidJ2Args&, Ctl*, double*, const FinJ2&);
template cudaError_t zmid_rows_inelastic<double>(int, bool, int, cudaStream_t, const GridDims&, const double2*, double2*,
                                                 const MidJ2Args&, Ctl*, double*, const FinJ2&);

}  // namespace m3d
