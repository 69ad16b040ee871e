// plane_launch.cuh -- launches of the two-pass elastic sweep (passes_plane.cuh,
// instantiated in plane.cu, compiled beside solver.cu).
#pragma once
#include "passes_plane.cuh"

namespace m3d {

// cubic grids of length N with a plane kernel in T
template <typename T> bool plane_size(int N);
template <typename T>
cudaError_t plane_pass(int N, int entries, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                       typename Cx<T>::t* sp, const SpecGreen<T, 6>& op, const Ctl* ctl);
// mix = false: only the forward half (the first sweep of a solve)
template <typename T>
cudaError_t zmid_pass(int N, int entries, bool mix, cudaStream_t st, const GridDims& g, const typename Cx<T>::t* tw,
                      typename Cx<T>::t* sp, const MidEMArgs<T>& op, Ctl* ctl, double* part, const FinLinear& fin);

}  // namespace m3d
