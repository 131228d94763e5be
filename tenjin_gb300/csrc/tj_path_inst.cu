// One instance of the per-direction launchers (tj_path_launch.cuh), selected
// at compile time: TJ_INST_R = 64 (binary64, DevParams) or 32 (binary32,
// DevParams32); TJ_INST_M = material count, 0 for the generic instance;
// TJ_INST_K = its ParamKind (0 if not given);
// TJ_INST_D = direction, -1 for the generic instance; TJ_INST_R = 128 is the
// tangent instance (DevParamsT, tj_dual.cuh), which has no CFL pass. The CFL
// pass and the whole-stage update are instantiated with the first direction of
// each material count.
#if defined(TJ_INST_R) && TJ_INST_R == 32
#define TJ_QUOT_EXPR
#endif
#if defined(TJ_INST_R) && TJ_INST_R == 128
#include "tj_dual.cuh"
#elif defined(TJ_INST_K) && TJ_INST_K > 0
#define TJ_DEV __device__ __forceinline__
#endif
#include "tj_path.cuh"
#include "tj_path_launch.cuh"
#if defined(TJ_INST_R) && TJ_INST_R == 128
#include "tj_dual_path.cuh"
#endif

#if !defined(TJ_INST_R) || !defined(TJ_INST_M) || !defined(TJ_INST_D)
#error "TJ_INST_R, TJ_INST_M and TJ_INST_D select the instance"
#endif

namespace tj {

namespace {
template <class PT>
inline LaunchShape path_shape(long long n)
{
    return launch_shape(n, kPathThreads<PT>);
}

// kernel(P, b, args...), overlapping the launch before it (tj_launch.cuh) where
// the grid leaves each SM room: up to the four blocks an SM that launch_shape
// halves the blocks for (64^2 cells driven operator by operator 1.70 -> 1.62
// ms). With more, the blocks of the next kernel take the SMs that drain first
// and are dealt unevenly (copper 40^3 in binary64, 1000 blocks, 10 steps: 14.05
// ms, overlapped 14.5). Not while the stream is captured, where plain edges are
// the faster ones (Sod, 1000 cells, 100 steps in binary64: 6.8 ms, overlapped
// 7.8), nor around single kernels' events (pr).
template <class PT, class... Params, class... Args>
inline void path_launch(void (*kernel)(PT, PathBufs<typename PT::real>, Params...), LaunchShape s, cudaStream_t st,
                        Prof* pr, const PT& P, PathBufs<typename PT::real> b, const Args&... args)
{
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    b.overlap = !pr && s.blocks <= 152 * 4 && cudaStreamIsCapturing(st, &capture) == cudaSuccess &&
                capture == cudaStreamCaptureStatusNone;
    launch(kernel, dim3(s.blocks), s.threads, 0, st, b.overlap, P, b, args...);
}
}  // namespace

template <class PT, int DC>
int path_faces(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, int d, cudaStream_t st,
               Prof* pr)
{
    constexpr bool f64 = sizeof(typename PT::real) == 8;
    const char* nr = f64 ? "tj_recon_fp64" : "tj_recon_fp32";
    const char* nf = f64 ? "tj_flux_fp64" : "tj_flux_fp32";
    const LaunchShape cells = path_shape<PT>(b.ntot), faces = path_shape<PT>(b.nftot[d]);
    if (pr) pr->begin(nr, st);
    if (P.thinc) {
        const LaunchShape sh = path_shape<PT>(b.ntot * P.M);
        path_launch(k_thinc<PT, DC>, sh, st, pr, P, b, X, reinterpret_cast<int*>(b.FX), d);
    }
    path_launch(k_recon<PT, DC>, cells, st, pr, P, b, X, d);
    if (pr) pr->end(nr, st);
    if (pr) pr->begin(nf, st);
    path_launch(k_flux<PT, DC>, faces, st, pr, P, b, d);
    if (pr) pr->end(nf, st);
    return P.thinc ? 3 : 2;
}

template <class PT, int DC>
int path_dir(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, typename PT::real* Y,
             int d, int first, int last, int finish, cudaStream_t st, Prof* pr)
{
    const char* nu = sizeof(typename PT::real) == 8 ? "tj_update_fp64" : "tj_update_fp32";
    const LaunchShape cells = path_shape<PT>(b.ntot);
    const int n = path_faces<PT, DC>(P, b, X, d, st, pr);
    if (pr) pr->begin(nu, st);
    path_launch(k_update<PT, DC>, cells, st, pr, P, b, X, Y, d, first, last, finish);
    if (pr) pr->end(nu, st);
    return n + 1;
}

template <class PT>
int path_update(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, typename PT::real* Y,
                int finish, cudaStream_t st, Prof* pr)
{
    const char* nu = sizeof(typename PT::real) == 8 ? "tj_update_fp64" : "tj_update_fp32";
    const LaunchShape cells = path_shape<PT>(b.ntot);
    if (pr) pr->begin(nu, st);
    if (finish) path_launch(k_update_all<PT, true>, cells, st, pr, P, b, X, Y, finish);
    else path_launch(k_update_all<PT, false>, cells, st, pr, P, b, X, Y, 0);
    if (pr) pr->end(nu, st);
    return 1;
}

template <class PT>
int path_cfl(const PT& P, const PathBufs<typename PT::real>& b, const typename PT::real* X, cudaStream_t st, Prof* pr)
{
    const char* nc = sizeof(typename PT::real) == 8 ? "tj_cfl_fp64" : "tj_cfl_fp32";
    if (pr) pr->begin(nc, st);
    const LaunchShape s = path_shape<PT>(b.ntot);
    path_launch(k_cfl<PT>, s, st, pr, P, b, X);
    if (pr) pr->end(nc, st);
    return 1;
}

#if TJ_INST_R == 64
using InstBase = DevParams;
#elif TJ_INST_R == 128
using InstBase = DevParamsT;
#else
using InstBase = DevParams32;
#endif
#if TJ_INST_M > 0
#ifndef TJ_INST_K
#define TJ_INST_K 0
#endif
using InstPT = WithM<InstBase, TJ_INST_M, TJ_INST_K>;
#else
using InstPT = InstBase;
#endif

template int path_dir<InstPT, TJ_INST_D>(const InstPT&, const PathBufs<InstPT::real>&, const InstPT::real*,
                                         InstPT::real*, int, int, int, int, cudaStream_t, Prof*);
#if TJ_INST_R != 128
template int path_faces<InstPT, TJ_INST_D>(const InstPT&, const PathBufs<InstPT::real>&, const InstPT::real*, int,
                                           cudaStream_t, Prof*);
#endif
#if TJ_INST_D <= 0 && TJ_INST_R != 128
template int path_update<InstPT>(const InstPT&, const PathBufs<InstPT::real>&, const InstPT::real*, InstPT::real*, int,
                                 cudaStream_t, Prof*);
template int path_cfl<InstPT>(const InstPT&, const PathBufs<InstPT::real>&, const InstPT::real*, cudaStream_t, Prof*);
#endif

}  // namespace tj
