// One instance of the binary32 kernels of several materials (tj_multi32.cuh):
// TJ_INST_M = 2, or 0 for the generic one; TJ_INST_D = direction, -1 for the
// generic one.
#define TJ_QUOT_EXPR
#include "tj_multi32_path.cuh"
#include "tj_multi32.cuh"

namespace tj {
namespace multi32 {

// Blocks of 256 on grids of any size for THINC: its candidates are formed by the
// reconstruction, each cell's three times, and the spread-out blocks of
// launch_shape lose there (two domains of 128^2, 10 steps: 2.91 ms with 256, 3.60
// with 32; 96^2 with RADIAL 2.73 / 3.22 ms). Without THINC they win (1-D, 4000
// cells, 40 steps: 1.94 / 1.82 ms; 48^3 solid and gas, 6 steps: 3.98 / 3.58 ms),
// and with a mixture, whose root find outweighs the candidates (128^2, 10 steps:
// 15.5 / 14.4 ms).
template <class PT>
static LaunchShape multi_shape(const PT& P, long long n)
{
    if (!P.thinc || P.nmix) return launch_shape(n, 256);
    const long long b = (n + 255) / 256, most = 152 * 16;
    return {(int)(b < 1 ? 1 : b > most ? most : b), 256};
}

template <class PT, int DC>
int path_dir(const PT& P, const PathBufs<float>& b, const float* X, float* Y, int d, int first, int last, int finish,
             cudaStream_t st, Prof* pr)
{
    const LaunchShape cells = multi_shape(P, b.ntot), faces = multi_shape(P, b.nftot[d]);
    if (pr) pr->begin("tj_recon_fp32", st);
    k_recon<PT, DC><<<cells.blocks, cells.threads, 0, st>>>(P, b, X, d);
    if (pr) pr->end("tj_recon_fp32", st);
    if (pr) pr->begin("tj_flux_fp32", st);
    k_flux<PT, DC><<<faces.blocks, faces.threads, 0, st>>>(P, b, d);
    if (pr) pr->end("tj_flux_fp32", st);
    if (pr) pr->begin("tj_update_fp32", st);
    k_update<PT, DC><<<cells.blocks, cells.threads, 0, st>>>(P, b, X, Y, d, first, last, finish);
    if (pr) pr->end("tj_update_fp32", st);
    return 3;
}

template <class PT>
int path_cfl(const PT& P, const PathBufs<float>& b, const float* X, cudaStream_t st, Prof* pr)
{
    const LaunchShape s = multi_shape(P, b.ntot);
    if (pr) pr->begin("tj_cfl_fp32", st);
    k_cfl<<<s.blocks, s.threads, 0, st>>>(P, b, X);
    if (pr) pr->end("tj_cfl_fp32", st);
    return 1;
}

#if TJ_INST_M > 0
using InstPT = WithM<DevParams32, TJ_INST_M>;
#else
using InstPT = DevParams32;
#endif
template int path_dir<InstPT, TJ_INST_D>(const InstPT&, const PathBufs<float>&, const float*, float*, int, int, int, int,
                                         cudaStream_t, Prof*);
#if TJ_INST_D <= 0
template int path_cfl<InstPT>(const InstPT&, const PathBufs<float>&, const float*, cudaStream_t, Prof*);
#endif

}  // namespace multi32
}  // namespace tj
