// Launchers of the per-direction kernels (tj_path.cuh) for one working type.
// Each (material count, direction) pair with M = 1 or 2 has its own instance,
// in which both are compile-time constants: the per-material loops unroll,
// the cell structures stay in registers and every direction-indexed access
// is static. M = 3 and 4 use the generic instance (runtime M and direction).
// In binary64 the fluids and the plastic solids have instances of their own
// (ParamKind), without the code and the registers of the rest.
// The instances are compiled in separate translation units
// (tj_path_inst.cu, once per type, M and direction) so that they build in
// parallel.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "tj_fp64.cuh"

namespace tj {

// One direction of one RK stage: k_recon, k_flux, k_update. Returns the
// number of launches.
template <class PT, int DC>
int path_dir(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, typename PT::real* Y,
             int d, int first, int last, int finish, cudaStream_t st, Prof* pr);
// The fluxes of one direction alone (k_thinc, k_recon, k_flux), into b.FX.
template <class PT, int DC>
int path_faces(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, int d, cudaStream_t st,
               Prof* pr);
// The update of a stage from the fluxes of every direction (k_update_all):
// direction d's follow those of d - 1 in b.FX.
template <class PT>
int path_update(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, typename PT::real* Y,
                int finish, cudaStream_t st, Prof* pr);
// The CFL pass (k_cfl) over the state X.
template <class PT>
int path_cfl(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, cudaStream_t st,
             Prof* pr);

// Whether a working type has instances of its own for a kind: binary64 for
// both, binary32 for the plastic solids (its fluids have the fused kernels),
// the tangent for none.
template <class Base, int K>
constexpr bool kHasKind = K == KIND_FLUID ? std::is_same<Base, DevParams>::value
                                          : std::is_same<Base, DevParams>::value ||
                                                std::is_same<Base, DevParams32>::value;

// Whether it serves several materials: those of binary32 have kernels of their
// own (tj_multi32.cuh).
template <class Base>
constexpr bool kSeveral = !std::is_same<Base, DevParams32>::value;

template <class Base, int K>
inline int path_dir_kind(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                         typename Base::real* Y, int d, int first, int last, int finish, cudaStream_t st, Prof* pr)
{
#define TJ_DIR(MC, DC) path_dir<WithM<Base, MC, K>, DC>(WithM<Base, MC, K>(P), b, X, Y, d, first, last, finish, st, pr)
    if (P.M == 1) return d == 0 ? TJ_DIR(1, 0) : d == 1 ? TJ_DIR(1, 1) : TJ_DIR(1, 2);
    if constexpr (kSeveral<Base>) {
        if (P.M == 2) return d == 0 ? TJ_DIR(2, 0) : d == 1 ? TJ_DIR(2, 1) : TJ_DIR(2, 2);
        return path_dir<Base, -1>(P, b, X, Y, d, first, last, finish, st, pr);
    }
    return 0;  // not reached: several materials in binary32 have kernels of their own (tj_multi32.cuh)
#undef TJ_DIR
}

template <class Base>
inline int path_dir_any(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                        typename Base::real* Y, int d, int first, int last, int finish, cudaStream_t st, Prof* pr)
{
    if constexpr (kHasKind<Base, KIND_FLUID>)
        if (param_kind(P) == KIND_FLUID) return path_dir_kind<Base, KIND_FLUID>(P, b, X, Y, d, first, last, finish, st, pr);
    if constexpr (kHasKind<Base, KIND_PLASTIC>)
        if (param_kind(P) == KIND_PLASTIC) return path_dir_kind<Base, KIND_PLASTIC>(P, b, X, Y, d, first, last, finish, st, pr);
    return path_dir_kind<Base, KIND_ANY>(P, b, X, Y, d, first, last, finish, st, pr);
}

template <class Base, int K>
inline int path_faces_kind(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X, int d,
                           cudaStream_t st, Prof* pr)
{
#define TJ_FACES(MC, DC) path_faces<WithM<Base, MC, K>, DC>(WithM<Base, MC, K>(P), b, X, d, st, pr)
    if (P.M == 1) return d == 0 ? TJ_FACES(1, 0) : d == 1 ? TJ_FACES(1, 1) : TJ_FACES(1, 2);
    if constexpr (kSeveral<Base>) {
        if (P.M == 2) return d == 0 ? TJ_FACES(2, 0) : d == 1 ? TJ_FACES(2, 1) : TJ_FACES(2, 2);
        return path_faces<Base, -1>(P, b, X, d, st, pr);
    }
    return 0;  // not reached, as above
#undef TJ_FACES
}

template <class Base>
inline int path_faces_any(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X, int d,
                          cudaStream_t st, Prof* pr)
{
    if constexpr (kHasKind<Base, KIND_FLUID>)
        if (param_kind(P) == KIND_FLUID) return path_faces_kind<Base, KIND_FLUID>(P, b, X, d, st, pr);
    if constexpr (kHasKind<Base, KIND_PLASTIC>)
        if (param_kind(P) == KIND_PLASTIC) return path_faces_kind<Base, KIND_PLASTIC>(P, b, X, d, st, pr);
    return path_faces_kind<Base, KIND_ANY>(P, b, X, d, st, pr);
}

template <class Base, int K>
inline int path_stage_kind(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                           typename Base::real* Y, int finish, cudaStream_t st, Prof* pr)
{
    int n = 0;
    if (!b.all_dirs) {
        for (int d = 0; d < P.dim; ++d)
            n += path_dir_kind<Base, K>(P, b, X, Y, d, d == 0, d == P.dim - 1, finish, st, pr);
        return n;
    }
    PathBufs<typename Base::real> bd = b;
    for (int d = 0; d < P.dim; ++d) {
        n += path_faces_kind<Base, K>(P, bd, X, d, st, pr);
        bd.FX += P.NX * b.nftot[d];
    }
    if (P.M == 1) return n + path_update(WithM<Base, 1, K>(P), b, X, Y, finish, st, pr);
    if constexpr (kSeveral<Base>) {
        if (P.M == 2) return n + path_update(WithM<Base, 2, K>(P), b, X, Y, finish, st, pr);
        return n + path_update(P, b, X, Y, finish, st, pr);
    }
    return n;
}

// One RK stage: every direction's fluxes from the stage input X, then one
// update into Y, or with finish into b.A; direction by direction where b.FX holds
// one direction's fluxes (flux_words).
template <class Base>
inline int path_stage_any(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                          typename Base::real* Y, int finish, cudaStream_t st, Prof* pr)
{
    if constexpr (kHasKind<Base, KIND_FLUID>)
        if (param_kind(P) == KIND_FLUID) return path_stage_kind<Base, KIND_FLUID>(P, b, X, Y, finish, st, pr);
    if constexpr (kHasKind<Base, KIND_PLASTIC>)
        if (param_kind(P) == KIND_PLASTIC) return path_stage_kind<Base, KIND_PLASTIC>(P, b, X, Y, finish, st, pr);
    return path_stage_kind<Base, KIND_ANY>(P, b, X, Y, finish, st, pr);
}

template <class Base, int K>
inline int path_cfl_kind(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                         cudaStream_t st, Prof* pr)
{
    if (P.M == 1) return path_cfl<WithM<Base, 1, K>>(WithM<Base, 1, K>(P), b, X, st, pr);
    if constexpr (kSeveral<Base>) {
        if (P.M == 2) return path_cfl<WithM<Base, 2, K>>(WithM<Base, 2, K>(P), b, X, st, pr);
        return path_cfl<Base>(P, b, X, st, pr);
    }
    return 0;  // not reached, as above
}

template <class Base>
inline int path_cfl_any(const Base& P, const PathBufs<typename Base::real>& b, const typename Base::real* X,
                        cudaStream_t st, Prof* pr)
{
    if constexpr (kHasKind<Base, KIND_FLUID>)
        if (param_kind(P) == KIND_FLUID) return path_cfl_kind<Base, KIND_FLUID>(P, b, X, st, pr);
    if constexpr (kHasKind<Base, KIND_PLASTIC>)
        if (param_kind(P) == KIND_PLASTIC) return path_cfl_kind<Base, KIND_PLASTIC>(P, b, X, st, pr);
    return path_cfl_kind<Base, KIND_ANY>(P, b, X, st, pr);
}

}  // namespace tj
