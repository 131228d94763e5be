// Binary32 steps of configurations with several materials outside the fused
// kernels (tj_multi32_path.cuh).
#pragma once

#include "tj_fp64.cuh"

namespace tj {
namespace multi32 {

// One direction of one RK stage: k_recon, k_flux, k_update; the CFL pass. One
// instance per (material count, direction), 0 and -1 the generic one
// (tj_multi32.cu). Return the number of launches.
template <class PT, int DC>
int path_dir(const PT& P, const PathBufs<float>& b, const float* X, float* Y, int d, int first, int last, int finish,
             cudaStream_t st, Prof* pr);
template <class PT>
int path_cfl(const PT& P, const PathBufs<float>& b, const float* X, cudaStream_t st, Prof* pr);

inline int stage(const DevParams32& P, const PathBufs<float>& b, const float* X, float* Y, int finish, cudaStream_t st,
                 Prof* pr)
{
    using P2 = WithM<DevParams32, 2>;
    int n = 0;
    for (int d = 0; d < P.dim; ++d) {
        const int first = d == 0, last = d == P.dim - 1;
        if (P.M != 2) n += path_dir<DevParams32, -1>(P, b, X, Y, d, first, last, finish, st, pr);
        else if (d == 0) n += path_dir<P2, 0>(P2(P), b, X, Y, d, first, last, finish, st, pr);
        else if (d == 1) n += path_dir<P2, 1>(P2(P), b, X, Y, d, first, last, finish, st, pr);
        else n += path_dir<P2, 2>(P2(P), b, X, Y, d, first, last, finish, st, pr);
    }
    return n;
}
inline int cfl(const DevParams32& P, const PathBufs<float>& b, const float* X, cudaStream_t st, Prof* pr)
{
    if (P.M == 2) return path_cfl<WithM<DevParams32, 2>>(WithM<DevParams32, 2>(P), b, X, st, pr);
    return path_cfl<DevParams32>(P, b, X, st, pr);
}

}  // namespace multi32
}  // namespace tj
