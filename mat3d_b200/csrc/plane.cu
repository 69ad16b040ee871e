// plane.cu -- kernels and launches of the two-pass elastic sweep.
#include "plane_launch.cuh"
#include "smem_limit.cuh"

namespace m3d {

namespace {
template <int NN> struct IntC { static constexpr int value = NN; };
template <typename T, class F> bool with_plane_n(int n, F&& f) {
    switch (n) {
        case 32: if constexpr (PlaneGeom<T, 32>::ok) { f(IntC<32>{}); return true; } return false;
        case 48: if constexpr (PlaneGeom<T, 48>::ok) { f(IntC<48>{}); return true; } return false;
        case 64: if constexpr (PlaneGeom<T, 64>::ok) { f(IntC<64>{}); return true; } return false;
        case 96: if constexpr (PlaneGeom<T, 96>::ok) { f(IntC<96>{}); return true; } return false;
        default: return false;
    }
}
}  // namespace

template <typename T> bool plane_size(int N) {
    return with_plane_n<T>(N, [](auto) {});
}

template <typename T>
cudaError_t plane_pass(int N, int entries, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                       typename Cx<T>::t* sp, const SpecGreen<T, 6>& op, const Ctl* ctl) {
    cudaError_t e = cudaErrorInvalidValue;
    with_plane_n<T>(N, [&](auto nc) {
        constexpr int NN = decltype(nc)::value;
        typedef PlaneGeom<T, NN> P;
        auto kern = k_plane<T, NN>;
        allow_smem(kern);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((NN / 2 + 1) * P::CS, entries);
        cfg.blockDim = dim3(P::NT);
        cfg.dynamicSmemBytes = P::smem();
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = P::CS;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = P::CS > 1 ? 1 : 0;
        e = cudaLaunchKernelEx(&cfg, kern, g, tw, sp, op, ctl);
    });
    return e;
}

template <typename T>
cudaError_t zmid_pass(int N, int entries, bool mix, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                      typename Cx<T>::t* sp, const MidEMArgs<T>& op, Ctl* ctl, double* part, const FinLinear& fin) {
    cudaError_t e = cudaErrorInvalidValue;
    with_plane_n<T>(N, [&](auto nc) {
        constexpr int NN = decltype(nc)::value;
        typedef ZMidGeom<T, NN> Z;
        const dim3 grid(NN * (NN / Z::G), entries);
        if (mix) {
            auto kern = k_zmid<T, NN, MidEM<T, Z::W>, true, FinLinear>;
            allow_smem(kern);
            kern<<<grid, Z::NT, Z::smem(), st>>>(g, tw, sp, op, ctl, part, fin);
        } else {
            auto kern = k_zmid<T, NN, MidEM<T, Z::W>, false, FinLinear>;
            allow_smem(kern);
            kern<<<grid, Z::NT, Z::smem(), st>>>(g, tw, sp, op, ctl, part, fin);
        }
        e = cudaGetLastError();
    });
    return e;
}

#define M3D_PLANE_INST(T)                                                                                             \
    template bool plane_size<T>(int);                                                                                 \
    template cudaError_t plane_pass<T>(int, int, cudaStream_t, const GridDims&, const Cx<T>::t*, Cx<T>::t*,           \
                                       const SpecGreen<T, 6>&, const Ctl*);                                           \
    template cudaError_t zmid_pass<T>(int, int, bool, cudaStream_t, const GridDims&, const Cx<T>::t*, Cx<T>::t*,      \
                                      const MidEMArgs<T>&, Ctl*, double*, const FinLinear&);
M3D_PLANE_INST(float)
M3D_PLANE_INST(double)

}  // namespace m3d
