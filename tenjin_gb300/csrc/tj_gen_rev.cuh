// Reverse kernels of the general reverse mode (tj_adjoint_gen.cu) that run the
// FP64 path's own device functions in forward mode, one direction a thread.
#pragma once

#include "tj_dual.cuh"
#include "tj_dual_path.cuh"
#include "tj_path.cuh"

namespace tj {

constexpr int kGT = 128;  // threads per block of the reverse kernels
// Blocks an SM is to hold of the two kernels here: they wait for instructions and
// for the binary64 pipe's latency, and 24 warps of 80 registers hide more of it
// than 16 of 128 or 8 of 255, spills included (copper 16^3, 4 steps, forward and
// backward: 48.9 / 54.4 / 63 ms).
constexpr int kGBlocks = 6;
constexpr int kNS = 48;   // carried words (39 at most: 4 solid plastic materials)
constexpr int kNX = 32;   // flux words (29 at most)
constexpr int kNF = 32;   // face-state words (31 at most)

// A cell's or a face's words as the reverse kernels pass them to the forward
// path's functions (tj_path.cuh load_state and others): read in place, the word
// `seed` carrying direction 1. Nothing is copied into per-thread arrays, whose
// indexing by word would put them into local memory.
struct SeedWords {
    const double* X;
    long long n, at;
    int seed;
    __device__ __forceinline__ SeedWords operator+(long long) const { return *this; }  // at the cell already
    __device__ __forceinline__ Dual operator[](long long w) const
    {
        return Dual(X[w * n + at], w == seed ? 1.0 : 0.0);
    }
};
// Where results go: each word's direction times its adjoint, summed (a zero
// adjoint takes no part).
template <class Lam>
struct DotWords {
    const Lam& lam;
    double& sum;
    struct Word {
        double lo;
        double& sum;
        __device__ __forceinline__ void operator=(Dual x) const
        {
            if (lo != 0.0) sum += lo * x.d;
        }
    };
    __device__ __forceinline__ DotWords operator+(long long) const { return *this; }
    __device__ __forceinline__ Word operator[](long long w) const { return {lam((int)w), sum}; }
};
// The second stage's end reads U^n from the words it then replaces.
template <class Lam>
struct SeedDotWords {
    SeedWords in;
    const Lam& lam;
    double& sum;
    struct Word {
        Dual x;
        double lo;
        double& sum;
        __device__ __forceinline__ operator Dual() const { return x; }
        __device__ __forceinline__ void operator=(Dual y) const
        {
            if (lo != 0.0) sum += lo * y.d;
        }
    };
    __device__ __forceinline__ SeedDotWords operator+(long long) const { return *this; }
    __device__ __forceinline__ Word operator[](long long w) const { return {in[w], lam((int)w), sum}; }
};
// Flux words of a cell's two faces; the seed is on face 0.
struct FacePairSeed {
    const double* FX;
    long long nf, f0, f1;
    int seed;
    __device__ __forceinline__ Dual operator()(int w, int s) const
    {
        return Dual(FX[(long long)w * nf + (s ? f1 : f0)], (!s && w == seed) ? 1.0 : 0.0);
    }
};

// The inputs of a cell's update whose derivatives are formed, one pass each
// (the others have none: conservativeToPrimitive and the radial return
// overwrite the words they would come from, and a face flux enters as the
// difference of the two faces, so face 1's adjoint is the negative of face
// 0's). kind 0: accumulator, 1: stage input, 2: flux of face 0, 3: U^n,
// 4: EOS parameter (word = material * npar + parameter).
struct UpdPass {
    short kind, word;
};
constexpr int kMaxPass = 3 * kNS + kNX + TJ_MAX_MAT * TJ_MAX_EOS_PARAMS;
struct UpdPasses {
    int n;
    UpdPass p[kMaxPass];
};

// ---------------------------------------------------------------------------
// Update of one direction, reversed per cell. Inputs: the accumulator Yin
// (not read by the first direction, whose accumulator is U), the stage input
// U, the two face fluxes F0 / F1 and, with the finish, U^n (A0). The output
// adjoint lamOut is that of the direction's output (the next accumulator, or
// U^{n+1} for the finish). Writes the adjoints of Yin and of the two fluxes
// (per cell: F0 of the face below, F1 of the face above; the words without a
// pass are zeroed by the host), adds those of U and A0, and adds each EOS
// parameter's part into geos (per cell).
//
// One thread per cell and pass, cells fastest: the passes are independent
// forward-mode evaluations of the cell's update whose values are the same and
// whose direction is one input's. (One thread per cell running its ~110
// passes in turn left 32 blocks for the 16^3 copper plate and spent its time in
// the latency of one serial chain: backward 580 ms for 4 steps.) A warp's
// lanes share the pass, so zero directions are skipped together.
// ---------------------------------------------------------------------------
template <class PT>
__global__ void __launch_bounds__(kGT, kGBlocks) k_gen_upd_rev(const __grid_constant__ PT P, Fp64Bufs fb,
                                                     const UpdPasses* __restrict__ passes, const double* Yin,
                                                     const double* U, const double* A0, const double* lamOut,
                                                     double* lamYin, double* lamU, double* lamA0, double* lamF0,
                                                     double* lamF1, double* geos, int d, int first, int finish,
                                                     int npar)
{
    const long long nt = fb.ntot, all = nt * passes->n;
    const DevDomain D = fb.doms[0];
    const Dual dtv(fb.scal->dt);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < all; e += (long long)gridDim.x * blockDim.x) {
        const int pass = (int)(e / nt);
        const long long g = e - (long long)pass * nt;
        const int kind = passes->p[pass].kind, word = passes->p[pass].word;
        int i, j, k;
        split3(g - D.off, D.n[0], D.n[1], i, j, k);
        const FacePairSeed fx{fb.FX, fb.nftot[d], face_index(D, d, i, j, k),
                              face_index(D, d, i + (d == 0), j + (d == 1), k + (d == 2)), kind == 2 ? word : -1};
        const auto lam = [&](int w) { return lamOut[w * nt + g]; };
        double s = 0.0;
        const SeedWords X{U, nt, g, kind == 1 ? word : -1}, Y0{Yin, nt, g, kind == 0 ? word : -1};
        const DotWords<decltype(lam)> out{lam, s};
        const SeedDotWords<decltype(lam)> A{{A0, nt, g, kind == 3 ? word : -1}, lam, s};
        const bool last_box = fb.cell_box[g] == D.nbox - 1;
        const auto run = [&](const PT& Q) {
            CellT<Dual> Uc, Yc;
            load_state(Q, X, 1LL, 0LL, nullptr, Uc);
            if (first) Yc = Uc;
            else load_state(Q, Y0, 1LL, 0LL, nullptr, Yc);
            add_fluxes(Q, Uc, Yc, quot(dtv, Dual(D.dx[d])), fx);
            finish_cell(Q, fb.scal, last_box, Yc, out, A, 1LL, 0LL, D, i, finish, dtv);
        };
        PT Q;
        const PT* par = &P;
        if (kind == 4) {  // an EOS parameter's direction: a copy of the block with it
            Q = P;
            Q.prm[word / npar][word % npar].d = 1.0;
            par = &Q;
        }
        run(*par);
        const long long at = (long long)word * nt + g;
        if (kind == 0) lamYin[at] = s;
        else if (kind == 1) lamU[at] += s;
        else if (kind == 2) {
            lamF0[at] = s;
            lamF1[at] = -s;
        } else if (kind == 3) lamA0[at] += s;
        else geos[at] += s;
    }
}

// ---------------------------------------------------------------------------
// Riemann problem of one face, reversed: the face's flux adjoint is gathered
// from the cell above (its F0) and the cell below (its F1); one pass per
// word of the two stored face states (UR of the cell below, UL of the cell
// above, boundary images as k_flux maps them) gives their adjoints, per face,
// one per EOS parameter in use those of the parameters: one thread per face
// and pass, faces fastest, as in k_gen_upd_rev.
// ---------------------------------------------------------------------------
template <class PT, int DC>
__global__ void __launch_bounds__(kGT, kGBlocks) k_gen_flux_rev(const __grid_constant__ PT P, Fp64Bufs fb,
                                                      const UpdPasses* __restrict__ passes, const double* lamF0,
                                                      const double* lamF1, double* lamLf, double* lamRf,
                                                      double* geos_f, int dyn_d, int npar)
{
    const int d = DC >= 0 ? DC : dyn_d;
    const long long nt = fb.ntot, nf = fb.nftot[d], all = nf * passes->n;
    const DevDomain D = fb.doms[0];
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < all; e += (long long)gridDim.x * blockDim.x) {
        const int pass = (int)(e / nf);
        const long long f = e - (long long)pass * nf;
        const int kind = passes->p[pass].kind, word = passes->p[pass].word;
        int i, j, k;
        split3(f - D.foff[d], D.n[0] + (d == 0), D.n[1] + (d == 1), i, j, k);
        int rl[3], rr[3];
        const long long gl = map_cell(P, D, i - (d == 0), j - (d == 1), k - (d == 2), rl);
        const long long gr = map_cell(P, D, i, j, k, rr);
        // the adjoint of a flux word: from the cell above (its face 0) and the one below (its face 1)
        const int at_d = d == 0 ? i : d == 1 ? j : k;
        const long long up_cell = D.off + i + (long long)D.n[0] * (j + (long long)D.n[1] * k);
        const long long lo_cell = up_cell - (d == 0 ? 1 : d == 1 ? D.n[0] : (long long)D.n[0] * D.n[1]);
        const auto lam = [&](int w) {
            double l = 0.0;
            if (at_d >= 1) l += lamF1[w * nt + lo_cell];
            if (at_d < D.n[d]) l += lamF0[w * nt + up_cell];
            return l;
        };
        double s = 0.0;
        const auto run = [&](const PT& Q) {
            CellT<Dual> L, R;
            FluxV<Dual> F;
            Dual Ss, vstar[3] = {Dual(0.0), Dual(0.0), Dual(0.0)};
            load_prim_face(Q, SeedWords{fb.UR, nt, gl, kind == 0 ? word : -1}, 1LL, 0LL, rl[d] ? d : -1, L);
            load_prim_face(Q, SeedWords{fb.UL, nt, gr, kind == 1 ? word : -1}, 1LL, 0LL, rr[d] ? d : -1, R);
            face_flux(Q, L, R, d, F, Ss, vstar, fb.scal);
            store_flux(Q, DotWords<decltype(lam)>{lam, s}, 1LL, 0LL, F, Ss, vstar);
        };
        PT Q;
        const PT* par = &P;
        if (kind == 4) {  // an EOS parameter's direction: a copy of the block with it
            Q = P;
            Q.prm[word / npar][word % npar].d = 1.0;
            par = &Q;
        }
        run(*par);
        if (kind == 0) lamLf[word * nf + f] = s;
        else if (kind == 1) lamRf[word * nf + f] = s;
        else geos_f[(long long)word * nf + f] += s;
    }
}

// Launchers, one instance each (tj_gen_inst.cu): the n passes of the list `pl`.
struct GenUpd {
    const double *Yin, *U, *A0, *lamOut;
    double *lamYin, *lamU, *lamA0, *lamF0, *lamF1, *geos;
    int d, first, finish, npar;
};
struct GenFlux {
    const double *lamF0, *lamF1;
    double *lamLf, *lamRf, *geos_f;
    int d, npar;
};
template <class PT>
void gen_upd_rev(const PT& P, const Fp64Bufs& fb, const UpdPasses* pl, int n, const GenUpd& a, cudaStream_t st)
{
    const LaunchShape s = launch_shape(fb.ntot * n, kGT);
    k_gen_upd_rev<PT><<<s.blocks, s.threads, 0, st>>>(P, fb, pl, a.Yin, a.U, a.A0, a.lamOut, a.lamYin, a.lamU, a.lamA0,
                                                      a.lamF0, a.lamF1, a.geos, a.d, a.first, a.finish, a.npar);
}
template <class PT, int DC>
void gen_flux_rev(const PT& P, const Fp64Bufs& fb, const UpdPasses* pl, int n, const GenFlux& a, cudaStream_t st)
{
    const LaunchShape s = launch_shape(fb.nftot[a.d] * n, kGT);
    k_gen_flux_rev<PT, DC><<<s.blocks, s.threads, 0, st>>>(P, fb, pl, a.lamF0, a.lamF1, a.lamLf, a.lamRf, a.geos_f, a.d,
                                                           a.npar);
}

}  // namespace tj
