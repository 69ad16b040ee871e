// zmid_launch.cuh -- launches of the fused z pass on the row layout
// (passes_zmid.cuh, instantiated in zmid.cu, compiled beside solver.cu).
#pragma once
#include "passes_zmid.cuh"

namespace m3d {

// a line length with a kernel, and whole tiles of lines (NL = Nx Ny)
template <typename T>
bool zmid_rows_ok(int N, long long NL);
// J2 (j2) or damage; the transforms in T
template <typename T>
cudaError_t zmid_rows_inelastic(int N, bool j2, int entries, cudaStream_t st, const GridDims& g,
                                const typename Cx<T>::t* tw, typename Cx<T>::t* sp, const MidJ2Args& op, Ctl* ctl,
                                double* part, const FinJ2& fin);

}  // namespace m3d
