// The per-direction kernels of the per-timestep update (reconstruction, face
// flux, update), one source for two working types: PT = DevParams (binary64,
// the reference's evaluation order: bit-exact parity, compiled with
// -fmad=false in tj_fp64.cu) and PT = DevParams32 (binary32 bulk, tj_fp32.cu).
// The binary32 instance keeps the total energy as a compensated pair (E, Elo),
// closes the pressure in binary64 (in c2p) and runs the plastic return map in
// binary64 (plastic_cell_proj64); everything else is the same code.
//
// One RK stage (HLLCadvance, hllc.cpp:579-695) is, per direction d:
//   k_thinc   per cell and material: the cell's THINC candidates (thinc.cpp:67-147)
//   k_recon   per cell : MUSCL (hllc.cpp:541-575), the BVD choice (thinc.cpp:148-208),
//                        cleanUpAlpha of the reconstructed states (hllc.cpp:628-629),
//                        primitiveToConservative + getSoundSpeed (634-638)
//   k_flux    per face : HLLC (hllc.cpp:384-487) or 5-wave (133-380)
// and, with every direction's fluxes, once:
//   k_update_all per cell : update (hllc.cpp:493-523) in the order x, y, z;
//                        conservativeToPrimitive (689), and at the end of the
//                        second stage the RK2 average (705), plasticUpdate,
//                        cleanUpV, cleanUpAlpha and the NaN check
//                        (main.cpp:145-187).
// The adjoint's and the tangent's runs update direction by direction (k_update).
// Ghost cells are never stored: a read outside a domain maps the index back
// (foextrap: nearest cell; reflect: mirror, negating the normal velocity and
// momentum), which is what the reference's FillDomainBoundary and
// FillBoundary calls leave in the ghost cells (main.cpp:124-126,
// hllc.cpp:642-646,690-691).
#pragma once

#include <cuda_runtime.h>

#include "tj_device.cuh"
#include "tj_fp64.cuh"
#include "tj_launch.cuh"

namespace tj {

// Registers of the binary64 instances: 128 a thread, so that 16 warps share an
// SM. With the divisions on the integer units the kernels wait for their own
// serial chains, and two warps a scheduler (255 registers) hide less of them
// than four, spills included: bubble 256^2, 20 steps 21.6 / 17.2 / 18.0 ms and
// copper 40^3, 10 steps 24.6 / 19.5 / 20.3 ms with 4 / 8 / 12 blocks of 64.
constexpr int kBlocks64 = 8;

// Blocks of the per-direction kernels and how many an SM is to hold. binary32:
// blocks of 128 (finer waves than 256) with 128 registers; the one-material
// plastic solids' reconstruction and fluxes fit in 102, a fifth block (copper
// 128^3, 5 steps: 15.46 ms with two blocks of 256, 14.97 with three and 80
// registers, 14.83 so). The instance for every other one-material configuration
// does not (its flux spills 490 bytes there): 2 / 3 / 4 / 5 blocks take 1.27 / 1.28 /
// 1.36 / 1.49 ms for a gas of 4000 cells in 1-D, 40 steps, and 8.01 / 5.59 / 5.48 /
// 5.77 ms for 1000^2 with RADIAL, 10 steps.
template <class PT>
constexpr bool kPath32 = sizeof(typename PT::real) == 4;
template <class PT>
constexpr int kPathThreads = kPath32<PT> ? 128 : 64;
template <class PT>
constexpr int kUpdateBlocks = kPath32<PT> ? 4 : kBlocks64;
template <class PT>
constexpr int kFaceBlocks = kPath32<PT> ? 3 : kBlocks64;
template <>
constexpr int kFaceBlocks<WithM<DevParams32, 1, KIND_PLASTIC>> = 5;

// The first statement of every per-direction kernel (tj_launch.cuh).
template <typename R>
__device__ __forceinline__ void overlap_start(const PathBufs<R>& b)
{
    if (b.overlap) {
        grid_wait();
        grid_go();
    }
}

// Error-free accumulation of b into the pair (hi, lo) (binary32 energy).
__device__ __forceinline__ void dd_add32(float& hi, float& lo, float b)
{
    const float s = __fadd_rn(hi, b);
    const float bb = __fsub_rn(s, hi);
    const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    lo = __fadd_rn(lo, e);
    const float t = __fadd_rn(s, lo);
    lo = __fsub_rn(lo, __fsub_rn(t, s));
    hi = t;
}

// (ah + al) / 2 + (bh + bl) / 2 into (bh, bl) (the RK2 average of the energy).
__device__ __forceinline__ void avg_pair32(float ah, float al, float& bh, float& bl)
{
    float hs = 0.5f * ah, ls = 0.5f * al;
    dd_add32(hs, ls, 0.5f * bh);
    ls = __fadd_rn(ls, 0.5f * bl);
    const float t = __fadd_rn(hs, ls);
    bl = __fsub_rn(ls, __fsub_rn(t, hs));
    bh = t;
}

// a / 2 + b / 2, the RK2 average of one word (hllc.cpp:705). The products are
// exact, so in binary64 one is left to the fused multiply-add and the other to
// the exponent: one operation of that pipe instead of three, the same bits.
template <typename R>
__device__ __forceinline__ R mean(R a, R b)
{
    return (a * (R(1.0) / R(2.0))) + (b * (R(1.0) / R(2.0)));
}
__device__ __forceinline__ double mean(double a, double b)
{
    const int h = __double2hiint(b), eb = (h >> 20) & 0x7ff, ea = (__double2hiint(a) >> 20) & 0x7ff;
    if (eb - 2u < 0x7fdu && ea - 2u < 0x7fdu) return fma(0.5, a, __hiloint2double(h - 0x100000, __double2loint(b)));
    return (a * (1.0 / 2.0)) + (b * (1.0 / 2.0));  // zero, next to subnormal, infinite or no number
}

__device__ __forceinline__ int find_dom(const DevDomain* doms, int ndom, long long g)
{
    int lo = 0, hi = ndom - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (doms[mid].off <= g) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// (i, j, k) of entry l of an n0 x n1 x n2 block (i fastest). One domain's
// cells and faces number below 2^32 at any size that fits the device, so the
// division runs in 32-bit unsigned arithmetic (a 64-bit division is a long
// software sequence); the 64-bit form remains for larger blocks.
__device__ __forceinline__ void split3(long long l, int n0, int n1, int& i, int& j, int& k)
{
    if ((unsigned long long)l < 4294967296ULL) {
        const unsigned u = (unsigned)l, q = u / (unsigned)n0;
        i = (int)(u - q * (unsigned)n0);
        const unsigned k2 = q / (unsigned)n1;
        j = (int)(q - k2 * (unsigned)n1);
        k = (int)k2;
    } else {
        i = (int)(l % n0);
        j = (int)((l / n0) % n1);
        k = (int)(l / ((long long)n0 * n1));
    }
}

__device__ __forceinline__ int find_dom_face(const DevDomain* doms, int ndom, int d, long long f)
{
    int lo = 0, hi = ndom - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (doms[mid].foff[d] <= f) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ void set_status(DevScalars* s, int code)
{
    atomicCAS(&s->status, 0, code);
}

// Map (i,j,k), possibly outside the domain, to a valid cell; refl[d] = 1 when
// direction d reflected.
template <typename PT, typename R = typename PT::real>
__device__ __forceinline__ long long map_cell(const PT& P, const DevDomain& D, int i, int j, int k, int* refl)
{
    int ijk[3] = {i, j, k};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        refl[d] = 0;
        if (d >= P.dim) continue;
        int n = D.n[d];
        if (ijk[d] < 0) {
            if (P.lo_bc[d] == TJ_BC_REFLECTIVE) { ijk[d] = -1 - ijk[d]; refl[d] = 1; }
            else ijk[d] = 0;
        } else if (ijk[d] > n - 1) {
            if (P.hi_bc[d] == TJ_BC_REFLECTIVE) { ijk[d] = 2 * n - 1 - ijk[d]; refl[d] = 1; }
            else ijk[d] = n - 1;
        }
    }
    return D.off + ijk[0] + (long long)D.n[0] * (ijk[1] + (long long)D.n[1] * ijk[2]);
}

__device__ __forceinline__ long long face_index(const DevDomain& D, int d, int i, int j, int k)
{
    int nf0 = D.n[0] + (d == 0), nf1 = D.n[1] + (d == 1);
    return D.foff[d] + i + (long long)nf0 * (j + (long long)nf1 * k);
}

// The words of a cell are addressed from a pointer to its first one: a word's
// offset from there is the same for every thread, so less is computed and held
// per thread (spills of the binary32 stage's end 300 -> 4 bytes; copper 128^3,
// 5 steps 14.9 -> 13.5 ms).
// Carried-state load with the reflect_odd sign applied. X here and the arrays of
// the other accessors below are pointers to the state's words, or what reads
// (takes) a word by its index in place of one.
template <typename PT, typename XP, typename R = typename PT::real>
TJ_DEV void load_state(const PT& P, const XP& X, long long nt, long long g, const int* refl,
                                  CellT<R>& c)
{
    const auto Xg = X + g;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        c.alpha[m] = Xg[(P.S_ALPHA + m) * nt];
        c.arho[m] = Xg[(P.S_ARHO + m) * nt];
        c.rhok[m] = Xg[(P.S_RHOK + m) * nt];
    }
    c.rho = Xg[P.S_RHO * nt];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        R u = Xg[(P.S_VEL + r) * nt], ru = Xg[(P.S_RHOU + r) * nt];
        if (refl && refl[r]) { u = -u; ru = -ru; }
        c.vel[r] = u;
        c.rhou[r] = ru;
    }
    c.E = Xg[P.S_E * nt];
    if constexpr (sizeof(R) == 4) c.Elo = Xg[P.S_ELO * nt];
    c.p = Xg[P.S_P * nt];
    c.hj2 = R(0.0);
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) c.V[q] = Xg[(P.S_V + q) * nt];
        c.hj2 = Xg[P.S_HJ2 * nt];
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) {
            c.eps[m] = Xg[(P.S_EPS + m) * nt];
            c.are[m] = Xg[(P.S_ARE + m) * nt];
        }
    if (P.nmix) {
        c.rm0 = Xg[P.S_RMIX * nt];
        c.rm1 = Xg[(P.S_RMIX + 1) * nt];
        c.lam = Xg[P.S_LAM * nt];
        c.arl = Xg[P.S_ARL * nt];
    }
}

// The fields of a carried cell that reconstruction reads (load_state without
// the conservative variables, which primitiveToConservative recomputes on
// each face state): the primitives with the reflect_odd sign, the cell's own
// HJ2 (SOLID) and alphaRhoEps (PLASTIC), and lambda (mixtures).
template <typename PT, typename R = typename PT::real>
TJ_DEV void load_prims(const PT& P, const R* X, long long nt, long long g, const int* refl, CellT<R>& c)
{
    const auto Xg = X + g;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        c.alpha[m] = Xg[(P.S_ALPHA + m) * nt];
        c.rhok[m] = Xg[(P.S_RHOK + m) * nt];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        R u = Xg[(P.S_VEL + r) * nt];
        if (refl && refl[r]) u = -u;
        c.vel[r] = u;
    }
    c.p = Xg[P.S_P * nt];
    c.hj2 = R(0.0);
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) c.V[q] = Xg[(P.S_V + q) * nt];
        c.hj2 = Xg[P.S_HJ2 * nt];
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) {
            c.eps[m] = Xg[(P.S_EPS + m) * nt];
            c.are[m] = Xg[(P.S_ARE + m) * nt];
        }
    if (P.nmix) c.lam = Xg[P.S_LAM * nt];
}

template <typename PT, typename XP, typename R = typename PT::real>
TJ_DEV void store_state(const PT& P, const XP& X, long long nt, long long g, const CellT<R>& c)
{
    const auto Xg = X + g;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        Xg[(P.S_ALPHA + m) * nt] = c.alpha[m];
        Xg[(P.S_ARHO + m) * nt] = c.arho[m];
        Xg[(P.S_RHOK + m) * nt] = c.rhok[m];
    }
    Xg[P.S_RHO * nt] = c.rho;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        Xg[(P.S_VEL + r) * nt] = c.vel[r];
        Xg[(P.S_RHOU + r) * nt] = c.rhou[r];
    }
    Xg[P.S_E * nt] = c.E;
    if constexpr (sizeof(R) == 4) Xg[P.S_ELO * nt] = c.Elo;
    Xg[P.S_P * nt] = c.p;
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) Xg[(P.S_V + q) * nt] = c.V[q];
        Xg[P.S_HJ2 * nt] = c.hj2;
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) {
            Xg[(P.S_EPS + m) * nt] = c.eps[m];
            Xg[(P.S_ARE + m) * nt] = c.are[m];
        }
    if (P.nmix) {
        Xg[P.S_RMIX * nt] = c.rm0;
        Xg[(P.S_RMIX + 1) * nt] = c.rm1;
        Xg[P.S_LAM * nt] = c.lam;
        Xg[P.S_ARL * nt] = c.arl;
    }
}

template <typename PT, typename R = typename PT::real>
TJ_DEV void store_face(const PT& P, R* F, long long nt, long long g, const CellT<R>& c)
{
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        F[(P.F_ALPHA + m) * nt + g] = c.alpha[m];
        F[(P.F_ARHO + m) * nt + g] = c.arho[m];
    }
    F[P.F_RHO * nt + g] = c.rho;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        F[(P.F_RHOU + r) * nt + g] = c.rhou[r];
        F[(P.F_VEL + r) * nt + g] = c.vel[r];
    }
    F[P.F_E * nt + g] = c.E;
    F[P.F_P * nt + g] = c.p;
    F[P.F_A * nt + g] = c.a;
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            F[(P.F_SIGMA + q) * nt + g] = c.sigma[q];
            F[(P.F_V + q) * nt + g] = c.V[q];
        }
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) F[(P.F_ARE + m) * nt + g] = c.are[m];
    if (P.nmix) F[P.F_ARL * nt + g] = c.arl;
}

template <typename PT, typename R = typename PT::real>
TJ_DEV void load_face(const PT& P, const R* F, long long nt, long long g, int oddir, CellT<R>& c)
{
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        c.alpha[m] = F[(P.F_ALPHA + m) * nt + g];
        c.arho[m] = F[(P.F_ARHO + m) * nt + g];
        c.rhok[m] = R(0.0);
    }
    c.rho = F[P.F_RHO * nt + g];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        R u = F[(P.F_VEL + r) * nt + g], ru = F[(P.F_RHOU + r) * nt + g];
        if (r == oddir) { u = -u; ru = -ru; }
        c.vel[r] = u;
        c.rhou[r] = ru;
    }
    c.E = F[P.F_E * nt + g];
    c.p = F[P.F_P * nt + g];
    c.a = F[P.F_A * nt + g];
    c.hj2 = R(0.0);
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            c.sigma[q] = F[(P.F_SIGMA + q) * nt + g];
            c.V[q] = F[(P.F_V + q) * nt + g];
        }
    } else {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 3; ++q) c.sigma[3 * r + q] = -c.p * (R)(r == q);  // stressTensor, fluid
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) c.are[m] = F[(P.F_ARE + m) * nt + g];
    if (P.nmix) c.arl = F[P.F_ARL * nt + g];
}

// Without BVD-THINC (whose repeated cleanUpAlpha feeds the closures one
// alpha and the flux another) and without mixtures, the reconstruction
// stores the primitives of each face state -- alpha[M], rho_k[M], u[3], p,
// V[9] (solids), epsilon[M] (plastic): 16 words for the copper plate instead
// of the 31 of a closed state -- and the flux kernel closes them
// (primitiveToConservative, getSoundSpeed) where it reads them: the same
// calls on the same values, so the same bits reach the Riemann solver.
template <typename PT>
__device__ __forceinline__ bool compact_faces(const PT& P)
{
    return !P.thinc && !P.nmix;
}

template <typename PT, typename R = typename PT::real>
TJ_DEV void store_prim_face(const PT& P, R* F, long long nt, long long g, const CellT<R>& c)
{
    const auto Fg = F + g;
    int w = 0;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) Fg[(long long)(w++) * nt] = c.alpha[m];
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) Fg[(long long)(w++) * nt] = c.rhok[m];
#pragma unroll
    for (int r = 0; r < 3; ++r) Fg[(long long)(w++) * nt] = c.vel[r];
    Fg[(long long)(w++) * nt] = c.p;
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) Fg[(long long)(w++) * nt] = c.V[q];
        if (!P.any_solid) Fg[(long long)(w++) * nt] = c.hj2;  // getHenckyJ2 does not run: the cell's own
    }
    if (P.plastic)  // epsilon of a solid closes alphaRhoEps; a fluid's alphaRhoEps is the cell's own
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) Fg[(long long)(w++) * nt] = phase_of(P, m) == TJ_PHASE_SOLID ? c.eps[m] : c.are[m];
}

// The closed face state of load_face from stored primitives: the closures
// of the reconstruction, then the fields load_face leaves at zero, then the
// reflect_odd sign of a boundary image.
template <typename PT, typename FP, typename R = typename PT::real>
TJ_DEV void load_prim_face(const PT& P, const FP& F, long long nt, long long g, int oddir, CellT<R>& c)
{
    const auto Fg = F + g;
    int w = 0;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) c.alpha[m] = Fg[(long long)(w++) * nt];
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) c.rhok[m] = Fg[(long long)(w++) * nt];
#pragma unroll
    for (int r = 0; r < 3; ++r) c.vel[r] = Fg[(long long)(w++) * nt];
    c.p = Fg[(long long)(w++) * nt];
    c.hj2 = R(0.0);
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) c.V[q] = Fg[(long long)(w++) * nt];
        if (!P.any_solid) c.hj2 = Fg[(long long)(w++) * nt];
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) {
            const R v = Fg[(long long)(w++) * nt];
            if (phase_of(P, m) == TJ_PHASE_SOLID) c.eps[m] = v;
            else c.are[m] = v;
        }
    p2c(P, c);
    c.a = sound_speed(P, c);
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) c.rhok[m] = R(0.0);
    c.hj2 = R(0.0);
    if (!P.solid)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int q = 0; q < 3; ++q) c.sigma[3 * r + q] = -c.p * (R)(r == q);  // stressTensor, fluid
    if (oddir >= 0) {
        c.vel[oddir] = -c.vel[oddir];
        c.rhou[oddir] = -c.rhou[oddir];
    }
}

template <typename R>
__device__ __forceinline__ R vanleer(R r)  // hllc.cpp:527-537
{
    if (r <= R(0.0)) return R(0.0);
    R a = quot(R(2.0), R(1.0) + r), b = quot(R(2.0) * r, R(1.0) + r);
    return (b < a) ? b : a;
}

template <typename R>
__device__ __forceinline__ void muscl1(R um, R u0, R up, R& l, R& r)  // hllc.cpp:557-568
{
    R rr = quot(u0 - um, up - u0);
    if (isinf(rr) || isnan(rr)) rr = R(0.0);
    R grad = vanleer(rr) * R(0.5) * (up - um);
    l = u0 - R(0.5) * grad;
    r = u0 + R(0.5) * grad;
}

// The limited extrapolation in the order of the reference, out of line: for the
// values at which the form below would round otherwise.
static __device__ __noinline__ double2 muscl_rare(double um, double u0, double up)
{
    double rr = (u0 - um) / (up - u0);
    if (isinf(rr) || isnan(rr)) rr = 0.0;
    const double grad = vanleer(rr) * 0.5 * (up - um);
    return make_double2(u0 - 0.5 * grad, u0 + 0.5 * grad);
}

// The same in binary64 with the same bits and fewer operations of that pipe:
// a ratio that is not positive and finite gives slope 0 without a division;
// of the limiter's two quotients 2 / (1 + r) and 2 r / (1 + r) the smaller is
// the one with the smaller numerator (rounding is monotonic), so one is formed;
// and the factors of one half go into that quotient and into the fused
// multiply-adds (7 binary64 operations instead of about 45). They are exact where
// the limiter's value and half the slope, about the smaller difference, are normal
// numbers: a ratio of 2^1022 or more and a difference below 2^-1019 are left to the
// general form.
__device__ __forceinline__ void muscl1(double um, double u0, double up, double& l, double& r)
{
    const double num = u0 - um, den = up - u0;
    const int hn = __double2hiint(num), hd = __double2hiint(den);
    const unsigned an = (unsigned)hn & 0x7fffffffu, ad = (unsigned)hd & 0x7fffffffu;
    double half = 0.0;
    bool rare = false;
    if ((hn ^ hd) >= 0) {
        if (min(an, ad) >= 0x00400000u) {
            const double rr = quot(num, den);
            const unsigned hr = (unsigned)__double2hiint(rr);
            if (hr < 0x7fd00000u) half = quot(hr < 0x3ff00000u ? rr : 1.0, 1.0 + rr);
            else rare = hr < 0x7ff00000u;
        } else {
            rare = (an | (unsigned)__double2loint(num)) != 0 && (ad | (unsigned)__double2loint(den)) != 0;
        }
    }
    const double grad = half * (up - um);
    l = fma(-0.5, grad, u0);
    r = fma(0.5, grad, u0);
    if (rare) {
        const double2 x = muscl_rare(um, u0, up);
        l = x.x;
        r = x.y;
    }
}

// One carried word at a possibly-ghost cell.
template <typename PT, typename R = typename PT::real>
__device__ __forceinline__ R gv(const PT& P, const DevDomain& D, const R* X, long long nt, int word,
                                     int i, int j, int k)
{
    int refl[3];
    long long g = map_cell(P, D, i, j, k, refl);
    R v = X[word * nt + g];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        if (d < P.dim && refl[d] && (word == P.S_VEL + d || word == P.S_RHOU + d)) v = -v;
    return v;
}

// ---------------------------------------------------------------------------
// BVD-THINC candidate of one material in one cell (thinc.cpp:67-147).
// ---------------------------------------------------------------------------
template <typename PT, typename R = typename PT::real>
TJ_DEV R youngs(const PT& P, const DevDomain& D, const R* X, long long nt, int m, int i,
                                int j, int k, int d)  // thinc.cpp:28-53
{
    int a = P.S_ALPHA + m;
#define NB(di, dj) gv(P, D, X, nt, a, i + (di), j + (dj), k)
    R nx = quot(-R(1.0), R(8.0) * (R)D.dx[0]) * (NB(1, 1) + R(2.0) * NB(1, 0) + NB(1, -1) - NB(-1, 1) - R(2.0) * NB(-1, 0) - NB(-1, -1));
    R ny = quot(-R(1.0), R(8.0) * (R)D.dx[1]) * (NB(1, 1) + R(2.0) * NB(0, 1) + NB(-1, 1) - NB(-1, -1) - R(2.0) * NB(0, -1) - NB(1, -1));
#undef NB
    R norm = root(nx * nx + ny * ny);
    if (norm < R(1E-20)) return 0;
    return d == 0 ? fabs(nx / norm) : fabs(ny / norm);
}

template <typename PT, typename R = typename PT::real>
TJ_DEV bool thinc_cand(const PT& P, const DevDomain& D, const R* X, long long nt, int m, int i, int j, int k, int d,
                       R& L, R& Rv)
{
    const R eps = R(1E-20), beta0 = P.beta;
    int o[3] = {0, 0, 0};
    o[d] = 1;
    int a = P.S_ALPHA + m;
    R aL = gv(P, D, X, nt, a, i - o[0], j - o[1], k - o[2]);
    R aR = gv(P, D, X, nt, a, i + o[0], j + o[1], k + o[2]);
    R a0 = gv(P, D, X, nt, a, i, j, k);
    R mn = (aR < aL) ? aR : aL;
    R mx = ((aL < aR) ? aR : aL) - mn;
    R theta = (R)((R(0.0) < aR - aL) - (aR - aL < R(0.0)));
    R C = (mx < eps) ? R(0.0) : quot(a0 - mn + eps, mx + eps);
    R delta = R(1E-4);
    if (!((C > delta) && (C < (R(0.999999) - delta)) && ((aR - a0) * (a0 - aL) >= R(0.0)))) return false;
    R nvc = (P.dim == 2) ? youngs(P, D, X, nt, m, i, j, k, d) : R(1.0);
    R beta = nvc * beta0 + R(0.01);
    R coshB = tjm_cosh(beta), tanhB = tjm_tanh(beta);
    R B = tjm_exp(theta * beta * ((R(2.0) * C) - R(1.0)));
    R A = quot((quot(B, coshB)) - R(1.0), tanhB);
    Rv = mn + (mx * R(0.5)) * (R(1.0) + theta * (quot(tanhB + A, R(1.0) + A * tanhB)));
    L = mn + (mx * R(0.5)) * (R(1.0) + theta * A);
    return true;
}

// The candidates of every cell and material (thinc.cpp:67-147, the first
// pass), one thread each: those of mixed cells into the persistent scratch
// (the reference's ULStar / URStar), and which they are into mixed[m nt + g]
// (the flux array's memory, which the reconstruction of a direction does not
// use otherwise). The scratch of a mixed cell is read in this pass as its
// candidate and never as the older value, so writing it before the
// reconstruction reads any changes nothing. A cell's reconstruction needs its
// own and both neighbours' candidates: formed there, each was formed three
// times, in one thread's serial chain (adjoint 96^2, every cell mixed: k_recon
// 205 us a direction).
template <typename PT, int DC = -1, typename R = typename PT::real>
__global__ void __launch_bounds__(kPathThreads<PT>, kFaceBlocks<PT>)
    k_thinc(PT P, PathBufs<typename PT::real> b, const R* __restrict__ X, int* __restrict__ mixed, int dyn_d)
{
    const int d = DC >= 0 ? DC : dyn_d;
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot, all = nt * P.M;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < all; e += (long long)gridDim.x * blockDim.x) {
        int m = 0;
        long long g = e;
        for (; g >= nt; g -= nt) ++m;
        const DevDomain D = b.doms[find_dom(b.doms, b.ndom, g)];
        int i, j, k;
        split3(g - D.off, D.n[0], D.n[1], i, j, k);
        R L, Rv;
        const bool mix = thinc_cand(P, D, X, nt, m, i, j, k, d, L, Rv);
        mixed[e] = mix;
        if (mix) {
            b.ulstar[e] = L;
            b.urstar[e] = Rv;
        }
    }
}

// ---------------------------------------------------------------------------
// Reconstruction of one direction.
// ---------------------------------------------------------------------------
// DC >= 0: the direction as a compile-time constant (d is then ignored).
template <typename PT, int DC = -1, typename R = typename PT::real>
__global__ void __launch_bounds__(kPathThreads<PT>, kFaceBlocks<PT>)
    k_recon(PT P, PathBufs<typename PT::real> b, const R* __restrict__ X, int dyn_d)
{
    const int d = DC >= 0 ? DC : dyn_d;
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nt; g += (long long)gridDim.x * blockDim.x) {
        const int q = find_dom(b.doms, b.ndom, g);
        const DevDomain D = b.doms[q];
        long long l = g - D.off;
        int i, j, k;
        split3(l, D.n[0], D.n[1], i, j, k);
        int o[3] = {0, 0, 0};
        o[d] = 1;
        int rm[3], rp[3];
        long long gm = map_cell(P, D, i - o[0], j - o[1], k - o[2], rm);
        long long gp = map_cell(P, D, i + o[0], j + o[1], k + o[2], rp);
        CellT<R> um, u0, up, L, Rc;
        load_prims(P, X, nt, gm, rm, um);
        load_prims(P, X, nt, g, nullptr, u0);
        load_prims(P, X, nt, gp, rp, up);
        L = u0;
        Rc = u0;
        if (P.muscl) {  // MUSCLextrapolate over the primitive list
            #pragma unroll UnrollM<PT>::n
            for (int m = 0; m < P.M; ++m) {
                muscl1(um.alpha[m], u0.alpha[m], up.alpha[m], L.alpha[m], Rc.alpha[m]);
                muscl1(um.rhok[m], u0.rhok[m], up.rhok[m], L.rhok[m], Rc.rhok[m]);
            }
#pragma unroll
            for (int r = 0; r < 3; ++r) muscl1(um.vel[r], u0.vel[r], up.vel[r], L.vel[r], Rc.vel[r]);
            muscl1(um.p, u0.p, up.p, L.p, Rc.p);
            if (P.solid)
#pragma unroll
                for (int qq = 0; qq < 9; ++qq) muscl1(um.V[qq], u0.V[qq], up.V[qq], L.V[qq], Rc.V[qq]);
            if (P.plastic)
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m) muscl1(um.eps[m], u0.eps[m], up.eps[m], L.eps[m], Rc.eps[m]);
            if (P.nmix) muscl1(um.lam, u0.lam, up.lam, L.lam, Rc.lam);
        }
        int reps = 0;
        if (P.thinc) {
            const int* bx = b.boxes + 6 * (D.box_off + b.cell_box[g]);
            int idx[3] = {i, j, k};
            const int in_m = idx[d] - 1 >= bx[d], in_p = idx[d] + 1 <= bx[3 + d];
            reps = D.nbox - b.cell_box[g];
            const long long gmm = D.off + (i - o[0]) + (long long)D.n[0] * ((j - o[1]) + (long long)D.n[1] * (k - o[2]));
            const long long gpp = D.off + (i + o[0]) + (long long)D.n[0] * ((j + o[1]) + (long long)D.n[1] * (k + o[2]));
            // the candidates of mixed cells are in the scratch (k_thinc)
            const int* mixed = reinterpret_cast<const int*>(b.FX);
            const bool flag = mixed[(long long)(P.M - 1) * nt + g] != 0;  // the last material wins (thinc.cpp:110-114)
            int code = 0;
            if (flag) {
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m) {
                    const int a = P.S_ALPHA + m;
                    R urm, ulp, trm, tlp;
                    // UR.left / UL.right: MUSCL value inside the box, stage input in a ghost.
                    if (in_m) {
                        R l_, r_;
                        muscl1(gv(P, D, X, nt, a, i - 2 * o[0], j - 2 * o[1], k - 2 * o[2]), um.alpha[m], u0.alpha[m], l_, r_);
                        urm = r_;
                        trm = b.urstar[(long long)m * nt + gmm];
                    } else {
                        urm = um.alpha[m];
                        trm = R(0.0);  // URStar ghosts are never written
                    }
                    if (in_p) {
                        R l_, r_;
                        muscl1(u0.alpha[m], up.alpha[m], gv(P, D, X, nt, a, i + 2 * o[0], j + 2 * o[1], k + 2 * o[2]), l_, r_);
                        ulp = l_;
                        tlp = b.ulstar[(long long)m * nt + gpp];
                    } else {
                        ulp = up.alpha[m];
                        // ULStar's ghost at the box's hi+1 face: star alpha of the last flux pass along d
                        tlp = b.gstar[d][(long long)m * b.nftot[d] + face_index(D, d, i + o[0], j + o[1], k + o[2])];
                    }
                    R tpl = b.ulstar[(long long)m * nt + g];
                    R tpr = b.urstar[(long long)m * nt + g];
                    R upl = L.alpha[m], upr = Rc.alpha[m];
#define MN(x, y) (((y) < (x)) ? (y) : (x))
#define TBV(PL, PR)                                                                                          \
        MN(MN(fabs(urm - (PL)) + fabs((PR)-ulp), fabs(trm - (PL)) + fabs((PR)-tlp)),                            \
           MN(fabs(urm - (PL)) + fabs((PR)-tlp), fabs(trm - (PL)) + fabs((PR)-ulp)))
                    R tbvm = TBV(upl, upr);
                    R tbvt = TBV(tpl, tpr);
#undef TBV
#undef MN
                    if (tbvt < tbvm) {
                        L.alpha[m] = tpl;
                        Rc.alpha[m] = tpr;
                        code |= (mixed[(long long)m * nt + g] ? 1 : 2) << (2 * m);
                    }
                }
            }
            if (b.rec) {
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m) {
                    b.rec[((long long)(d * 2) * P.M + m) * nt + g] = L.alpha[m];
                    b.rec[((long long)(d * 2 + 1) * P.M + m) * nt + g] = Rc.alpha[m];
                }
                b.rec_code[(long long)d * nt + g] = code;
            }
        }
        if (compact_faces(P)) {  // closed by the flux kernel
            store_prim_face(P, b.UL, nt, g, L);
            store_prim_face(P, b.UR, nt, g, Rc);
            continue;
        }
        // cleanUpAlpha of UL and UR: nbox-b times for box b, the closures see
        // the first (hllc.cpp:628-638).
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            CellT<R>& S = side ? Rc : L;
            if (reps > 0) {
                int e = cleanup_alpha(P, S.alpha);
                if (e) set_status(b.scal, e);
            }
            p2c(P, S);
            S.a = sound_speed(P, S);
            for (int r = 1; r < reps; ++r) {
                R before[TJ_MAX_MAT];
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m) before[m] = S.alpha[m];
                int e = cleanup_alpha(P, S.alpha);
                if (e) set_status(b.scal, e);
                bool same = true;
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m)
                    same &= same_bits(before[m], S.alpha[m]);
                if (same) break;
            }
        }
        store_face(P, b.UL, nt, g, L);
        store_face(P, b.UR, nt, g, Rc);
    }
}

// ---------------------------------------------------------------------------
// Riemann solvers (hllc.cpp:1-487, flux.cpp:5-47).
// ---------------------------------------------------------------------------
template <typename PT, typename R = typename PT::real>
TJ_DEV void star_state(const PT& P, const CellT<R>& U, CellT<R>& Us, R SK, R Ss, int d)  // :12-73
{
    R ud = U.vel[d];
    // |(Ss - ud) / Ss| < 1e-20: the difference of two binary64 numbers that
    // differ is not smaller than 2^-54 of either, so the quotient is that small
    // only when they are equal (and not zero)
    bool contact;
    if constexpr (sizeof(R) == 4) contact = fabs((Ss - ud) / Ss) < R(1E-20);
    else contact = Ss - ud == R(0.0) && Ss != R(0.0);
    R mult = contact ? R(1.0) : quot(SK - ud, SK - Ss);
    Us.rho = R(0.0);
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        Us.alpha[m] = U.alpha[m];
        Us.arho[m] = mult * U.arho[m];
        Us.rhok[m] = quot(Us.arho[m], Us.alpha[m]);
        if (P.nmix && m == 0) Us.arl = mult * U.arl;
        // a fluid carries no plastic strain: its alphaRhoEps star value is 0
        // (the reference writes only the plastic materials' and resets the
        // fluids' after every step, so no result depends on it)
        if (P.plastic) Us.are[m] = phase_of(P, m) == TJ_PHASE_SOLID ? mult * U.are[m] : R(0.0);
        Us.rho += Us.arho[m];
    }
#pragma unroll
    for (int row = 0; row < 3; ++row) {
        if (row == d) Us.rhou[row] = mult * U.rho * Ss;
        else Us.rhou[row] = mult * U.rhou[row];
        Us.vel[row] = quot(Us.rhou[row], Us.rho);
        if (P.solid)
#pragma unroll
            for (int col = 0; col < 3; ++col)
                Us.V[3 * row + col] = (row == d) ? U.V[3 * row + col] : mult * U.V[3 * row + col];
    }
    Us.E = mult * U.rho * (quot(U.E, U.rho) + (Ss - ud) * (Ss - quot(U.sigma[4 * d], U.rho * (SK - ud))));
}

// The conservative variables of one state, or their fluxes, by name: kept in
// registers; the flux-word layout is applied only where a face is stored.
template <typename R>
struct FluxV {
    R alpha[TJ_MAX_MAT], arho[TJ_MAX_MAT], rhou[3], E, V[9], are[TJ_MAX_MAT], arl;
};

// Physical flux of the conservative variables (flux.cpp:33-47).
template <typename PT, typename R = typename PT::real>
TJ_DEV void phys_flux(const PT& P, const CellT<R>& U, int d, FluxV<R>& F)
{
    R ud = U.vel[d];
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        F.alpha[m] = U.alpha[m] * ud;
        F.arho[m] = U.arho[m] * ud;
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) F.rhou[r] = U.rhou[r] * ud - U.sigma[3 * r + d];
    R vs = R(0.0);
#pragma unroll
    for (int i = 0; i < 3; ++i) vs += U.vel[i] * U.sigma[3 * i + d];
    F.E = U.E * ud - vs;
    if (P.solid)
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            int row = q / 3, col = q % 3;
            F.V[q] = U.V[q] * ud - U.V[3 * d + col] * U.vel[row];
        }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) F.are[m] = U.are[m] * ud;
    if (P.nmix) F.arl = U.arl * ud;
}

// Conservative values of a state.
template <typename PT, typename R = typename PT::real>
TJ_DEV void cons_vals(const PT& P, const CellT<R>& U, FluxV<R>& Q)
{
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        Q.alpha[m] = U.alpha[m];
        Q.arho[m] = U.arho[m];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) Q.rhou[r] = U.rhou[r];
    Q.E = U.E;
    if (P.solid)
#pragma unroll
        for (int q = 0; q < 9; ++q) Q.V[q] = U.V[q];
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) Q.are[m] = U.are[m];
    if (P.nmix) Q.arl = U.arl;
}

// The face flux of every conservative variable but alpha, in the reference's
// evaluation order (hllc.cpp:416-476, 287-371):
//   NT = 0: FK
//   NT = 1: FK + S1 (Q1 - Q0)
//   NT = 2: FK + S1 (Q1 - Q0) + S2 (Q2 - Q1)
// alpha takes the flux of the star state FA.
template <int NT, typename PT, typename R = typename PT::real>
TJ_DEV void flux_combine(const PT& P, FluxV<R>& F, const FluxV<R>& FA, const FluxV<R>& FK,
                                    const FluxV<R>& Q0, const FluxV<R>& Q1, const FluxV<R>& Q2, R S1, R S2)
{
    auto one = [&](R fk, R q0, R q1, R q2) -> R {
        if constexpr (NT == 0) return fk;
        else if constexpr (NT == 1) return fk + S1 * (q1 - q0);
        else return fk + S1 * (q1 - q0) + S2 * (q2 - q1);
    };
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        F.alpha[m] = FA.alpha[m];
        F.arho[m] = one(FK.arho[m], Q0.arho[m], Q1.arho[m], Q2.arho[m]);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) F.rhou[r] = one(FK.rhou[r], Q0.rhou[r], Q1.rhou[r], Q2.rhou[r]);
    F.E = one(FK.E, Q0.E, Q1.E, Q2.E);
    if (P.solid)
#pragma unroll
        for (int q = 0; q < 9; ++q) F.V[q] = one(FK.V[q], Q0.V[q], Q1.V[q], Q2.V[q]);
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) F.are[m] = one(FK.are[m], Q0.are[m], Q1.are[m], Q2.are[m]);
    if (P.nmix) F.arl = one(FK.arl, Q0.arl, Q1.arl, Q2.arl);
}

// One face into the flux-word layout (nf faces per word).
template <typename PT, typename FP, typename R = typename PT::real>
TJ_DEV void store_flux(const PT& P, const FP& FX, long long nf, long long f, const FluxV<R>& F, R Ss,
                                  const R* vstar)
{
    const auto FXf = FX + f;
#define FXS(w) FXf[(long long)(w) * nf]
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        FXS(P.X_ALPHA + m) = F.alpha[m];
        FXS(P.X_ARHO + m) = F.arho[m];
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) FXS(P.X_RHOU + r) = F.rhou[r];
    FXS(P.X_E) = F.E;
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) FXS(P.X_V + q) = F.V[q];
#pragma unroll
        for (int col = 0; col < 3; ++col) FXS(P.X_VSTAR + col) = vstar[col];
    }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) FXS(P.X_ARE + m) = F.are[m];
    if (P.nmix) FXS(P.X_ARL) = F.arl;
    FXS(P.X_SSTAR) = Ss;
#undef FXS
}

// K = first ? A : B over the words the Riemann solvers read.
template <typename PT, typename R = typename PT::real>
TJ_DEV void select_cell(const PT& P, bool first, const CellT<R>& A, const CellT<R>& B, CellT<R>& K)
{
#define TJ_PICK(w) K.w = first ? A.w : B.w
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        TJ_PICK(alpha[m]);
        TJ_PICK(arho[m]);
        if (P.plastic) TJ_PICK(are[m]);
    }
    TJ_PICK(rho);
    TJ_PICK(E);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        TJ_PICK(rhou[r]);
        TJ_PICK(vel[r]);
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        TJ_PICK(sigma[q]);
        if (P.solid) TJ_PICK(V[q]);
    }
    if (P.nmix) TJ_PICK(arl);
#undef TJ_PICK
}

// HLLC (hllc.cpp:384-487) or the 5-wave solver (133-380) at one face. F gets
// the conservative fluxes, Ss the contact speed, vstar the VSTAR(d, col)
// values (solids). Returns the side whose star alpha the face carries: 0
// left, 1 right.
template <typename PT, typename R = typename PT::real>
TJ_DEV int face_flux(const PT& P, const CellT<R>& L, const CellT<R>& Rc, int d, FluxV<R>& F, R& Ss,
                                R* vstar, DevScalars* scal)
{
    R x1 = fabs(L.vel[d]) + L.a, x2 = fabs(Rc.vel[d]) + Rc.a;
    R SR = (x1 < x2) ? x2 : x1;
    R SL = -SR;
    Ss = quot(-Rc.sigma[4 * d] + L.sigma[4 * d] + L.rhou[d] * (SL - L.vel[d]) - Rc.rhou[d] * (SR - Rc.vel[d]), L.rho * (SL - L.vel[d]) - Rc.rho * (SR - Rc.vel[d]));  // getSstar, hllc.cpp:5-8
    // 5-wave solver for solids (hllc.cpp:133-380)
    if (P.solid && (isnan(SL) || isnan(SR) || isnan(Ss))) { set_status(scal, TJ_ERR_WAVESPEED); return 0; }
    // The two sides run one code path on the upwind state K (and, for the inner
    // wave, the other state O), picked word by word: a warp whose faces blow
    // both ways would run a path of each side, one after the other (copper
    // plate with 1 % noise: 21 of 32 threads active).
    const bool left = SL >= R(0.0) || Ss >= R(0.0);
    const bool plain = left ? SL >= R(0.0) : !(SR >= R(0.0));  // supersonic: the flux of K itself
    CellT<R> K, Ks;
    select_cell(P, left, L, Rc, K);
    const R SK = left ? SL : SR;
    star_state(P, K, Ks, SK, Ss, d);
    FluxV<R> FK, FAs, QK, QKs;
    phys_flux(P, K, d, FK);
    phys_flux(P, Ks, d, FAs);
    auto vstar_of = [&](const CellT<R>& U) {  // VSTAR(d, col), read by update
        if (P.solid)
#pragma unroll
            for (int col = 0; col < 3; ++col) vstar[col] = U.V[3 * d + col];
    };
    if (plain) {
        flux_combine<0>(P, F, FAs, FK, FK, FK, FK, R(0.0), R(0.0));
        vstar_of(K);
        return left ? 0 : 1;
    }
    cons_vals(P, K, QK);
    cons_vals(P, Ks, QKs);
    if (!P.solid) {
        flux_combine<1>(P, F, FAs, FK, QK, QKs, QKs, SK, R(0.0));
        return left ? 0 : 1;
    }
    const R cK = transverse_speed(P, Ks);
    const R SKT = left ? Ss - cK : Ss + cK;
    if (left ? SKT >= R(0.0) : !(SKT >= R(0.0))) {
        flux_combine<1>(P, F, FAs, FK, QK, QKs, QKs, SK, R(0.0));
        vstar_of(Ks);
        if (isnan(SKT)) set_status(scal, TJ_ERR_WAVESPEED);
        return left ? 0 : 1;
    }
    CellT<R> O, Os;
    select_cell(P, left, Rc, L, O);
    star_state(P, O, Os, left ? SR : SL, Ss, d);
    const R cO = transverse_speed(P, Os);
    const R SOT = left ? Ss + cO : Ss - cO;
    const R lr = left ? Ks.rho : Os.rho, rr = left ? Os.rho : Ks.rho;
    const R SLT = left ? SKT : SOT, SRT = left ? SOT : SKT;
    // getStarStarState, hllc.cpp:87-129
    CellT<R> Uss = Ks;
#pragma unroll
    for (int i = 0; i < 3; ++i)  // getSigmaStar, hllc.cpp:75-83
        Ks.sigma[3 * i + d] = quot(lr * (Ss - SLT) * rr * (Ss - SRT) * (L.vel[i] - Rc.vel[i]) +
                                       lr * (Ss - SLT) * Rc.sigma[3 * i + d] - rr * (Ss - SRT) * L.sigma[3 * i + d],
                                   lr * (Ss - SLT) - rr * (Ss - SRT));
#pragma unroll
    for (int row = 0; row < 3; ++row) {
        if (row == d) continue;
        Uss.rhou[row] += quot(Ks.sigma[3 * row + d] - K.sigma[3 * row + d], Ss - SKT);
        Uss.vel[row] = quot(Uss.rhou[row], Uss.rho);
    }
#pragma unroll
    for (int row = 0; row < 3; ++row) {
        if (row == d) continue;
        Uss.E += quot(Uss.vel[row] * Ks.sigma[3 * row + d] - K.vel[row] * K.sigma[3 * row + d], Ss - SKT);
#pragma unroll
        for (int col = 0; col < 3; ++col)
            Uss.V[3 * row + col] += quot(Uss.V[3 * d + col] * (Uss.vel[row] - K.vel[row]), Ss - SKT);
    }
    FluxV<R> QSS;
    cons_vals(P, Uss, QSS);
    flux_combine<2>(P, F, FAs, FK, QK, QKs, QSS, SK, SKT);
    vstar_of(Uss);
    if (isnan(SKT) || isnan(SOT)) set_status(scal, TJ_ERR_WAVESPEED);
    return left ? 0 : 1;
}

template <typename PT, int DC = -1, typename R = typename PT::real>
__global__ void __launch_bounds__(kPathThreads<PT>, kFaceBlocks<PT>)
    k_flux(PT P, PathBufs<typename PT::real> b, int dyn_d)
{
    const int d = DC >= 0 ? DC : dyn_d;
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot, nf = b.nftot[d];
    for (long long f = blockIdx.x * (long long)blockDim.x + threadIdx.x; f < nf; f += (long long)gridDim.x * blockDim.x) {
        const int q = find_dom_face(b.doms, b.ndom, d, f);
        const DevDomain D = b.doms[q];
        int nfv[3] = {D.n[0], D.n[1], D.n[2]};
        nfv[d] += 1;
        long long l = f - D.foff[d];
        int i, j, k;
        split3(l, nfv[0], nfv[1], i, j, k);
        int o[3] = {0, 0, 0};
        o[d] = 1;
        int rl[3], rr[3];
        long long gl = map_cell(P, D, i - o[0], j - o[1], k - o[2], rl);
        long long gr = map_cell(P, D, i, j, k, rr);
        CellT<R> L, Rc;
        if (compact_faces(P)) {
            load_prim_face(P, b.UR, nt, gl, rl[d] ? d : -1, L);
            load_prim_face(P, b.UL, nt, gr, rr[d] ? d : -1, Rc);
        } else {
            load_face(P, b.UR, nt, gl, rl[d] ? d : -1, L);
            load_face(P, b.UL, nt, gr, rr[d] ? d : -1, Rc);
        }
        FluxV<R> F;
        R Ss, vstar[3] = {R(0.0), R(0.0), R(0.0)};
        int side = face_flux(P, L, Rc, d, F, Ss, vstar, b.scal);
        store_flux(P, b.FX, nf, f, F, Ss, vstar);
        if (P.thinc) {
            int idx[3] = {i, j, k};
            if (idx[d] < D.n[d]) {  // ULStar alpha at the valid cell of this face
                long long g = D.off + i + (long long)D.n[0] * (j + (long long)D.n[1] * k);
                #pragma unroll UnrollM<PT>::n
                for (int m = 0; m < P.M; ++m) b.ulstar[(long long)m * nt + g] = (side ? Rc.alpha[m] : L.alpha[m]);
            }
            if (idx[d] >= 1) {  // the ghost hi+1 of the box to the left, if this is its hi face
                long long gL = D.off + (i - o[0]) + (long long)D.n[0] * ((j - o[1]) + (long long)D.n[1] * (k - o[2]));
                const int* bx = b.boxes + 6 * (D.box_off + b.cell_box[gL]);
                if (bx[3 + d] == idx[d] - 1)
                    #pragma unroll UnrollM<PT>::n
                    for (int m = 0; m < P.M; ++m) b.gstar[d][(long long)m * nf + f] = (side ? Rc.alpha[m] : L.alpha[m]);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Plastic radial return (plastic.cpp:83-223) and cleanUpV (:476-528).
// ---------------------------------------------------------------------------
template <typename PT, typename R = typename PT::real>
TJ_DEV int plastic_cell(const PT& P, CellT<R>& c)
{
    R tsolid = R(0.0);
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m)
        if (phase_of(P, m) == TJ_PHASE_SOLID) tsolid += c.alpha[m];
    if (tsolid <= R(0.5)) {  // cellIsMostlyFluid
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) { c.eps[m] = R(0.0); c.are[m] = R(0.0); }
        return 0;
    }
    hencky(P, c);
    R JT = R(0.0), JB = R(0.0), norm = R(0.0), J, Jn;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        ECellT<R> e = ecell_of(c, m);
        if (phase_of(P, m) == TJ_PHASE_SOLID) {
            J = root(c.hj2);
            R G = eos_G(P, m, e);
            if (G * J * sqrt(R(3.0)) > P.yield[m]) Jn = quot(P.yield[m], sqrt(R(3.0)) * G);
            else Jn = J;
            c.eps[m] += sqrt(R(2.0) / R(3.0)) * (J - Jn);
            c.are[m] = c.eps[m] * c.arho[m];
        } else {
            J = R(0.0);
            Jn = R(0.0);
            c.eps[m] = R(0.0);
            c.are[m] = R(0.0);
        }
        JB += (eos_invG(P, m, e)) * J;
        JT += (eos_invG(P, m, e)) * Jn;
        norm += (eos_invG(P, m, e));
    }
    JB *= quot(R(1.0), norm);
    JT *= quot(R(1.0), norm);
    if (JB == R(0.0) && JT == R(0.0)) { JB = R(1.0); JT = R(1.0); }
    R t1[9], t2[9], t2i[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            R& dv = c.devH[3 * r + q];
            if (dv != R(0.0) && JB == R(0.0) && JT != R(0.0)) return TJ_ERR_PLASTIC;
            dv *= quot(JT, JB);
            t1[3 * r + q] = (R)(r == q) + R(0.5) * dv;
            t2[3 * r + q] = (R)(r == q) - R(0.5) * dv;
        }
    invert3(t2, t2i);
    mm3(t2i, t1, c.V);
    return 0;
}

// The radial return of a binary32 cell with its return map in binary64
// (plastic.cpp:83-223): the Hencky strain of V is binary32; J = sqrt(HJ2),
// the projection J -> J_new onto the yield surface, the plastic strain and
// alphaRhoEpsilon, the mixture-weighted scale JTotal / JBefore and the
// scaled devH are binary64 from the binary64 EOS parameters, rounded back
// once; the reconstruction of V from devH and the conservativeToPrimitive
// that follows are binary32 (pressure closure in binary64).
template <typename PT, typename R = typename PT::real>
TJ_DEV int plastic_cell_proj64(const PT& P, CellT<R>& c)
{
    const DevParams& PD = P.d;
    R tsolid = R(0.0);
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m)
        if (phase_of(P, m) == TJ_PHASE_SOLID) tsolid += c.alpha[m];
    if (tsolid <= R(0.5)) {  // cellIsMostlyFluid
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) { c.eps[m] = R(0.0); c.are[m] = R(0.0); }
        return 0;
    }
    hencky(P, c);
    const double hj2 = c.hj2;
    double JT = 0.0, JB = 0.0, norm = 0.0;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        ECellT<double> e;
        e.alpha = c.alpha[m];
        e.arho = c.arho[m];
        e.rhok = c.rhok[m];
        e.p = c.p;
        e.hj2 = hj2;
        e.lam = c.lam;
        e.rm0 = c.rm0;
        e.rm1 = c.rm1;
        double J, Jn;
        if (phase_of(P, m) == TJ_PHASE_SOLID) {
            J = root(hj2);
            const double G = eos_G(PD, m, e);
            Jn = (G * J * sqrt(3.0) > PD.yield[m]) ? quot(PD.yield[m], sqrt(3.0) * G) : J;
            const double eps = (double)c.eps[m] + sqrt(2.0 / 3.0) * (J - Jn);
            c.eps[m] = (R)eps;
            c.are[m] = (R)(eps * (double)c.arho[m]);
        } else {
            J = 0.0;
            Jn = 0.0;
            c.eps[m] = R(0.0);
            c.are[m] = R(0.0);
        }
        const double ig = eos_invG(PD, m, e);
        JB += ig * J;
        JT += ig * Jn;
        norm += ig;
    }
    JB *= quot(1.0, norm);
    JT *= quot(1.0, norm);
    if (JB == 0.0 && JT == 0.0) { JB = 1.0; JT = 1.0; }
    R t1[9], t2[9], t2i[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            R& dv = c.devH[3 * r + q];
            if (dv != R(0.0) && JB == 0.0 && JT != 0.0) return TJ_ERR_PLASTIC;
            dv = (R)((double)dv * (quot(JT, JB)));
            t1[3 * r + q] = (R)(r == q) + R(0.5) * dv;
            t2[3 * r + q] = (R)(r == q) - R(0.5) * dv;
        }
    invert3(t2, t2i);
    mm3(t2i, t1, c.V);
    return 0;
}

template <typename PT, typename R = typename PT::real>
TJ_DEV void cleanup_v_cell(const PT& P, CellT<R>& c)
{
    R ta = R(0.0), ts = R(0.0);
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        ta += c.alpha[m];
        if (phase_of(P, m) == TJ_PHASE_SOLID) ts += c.alpha[m];
    }
    R B[9], Sq[9];
    mmT3(c.V, c.V, B);
    sqrtm3(B, Sq);
    R norm = tjm_pow(det3(Sq), -R(1.0) / R(3.0));
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int q = 0; q < 3; ++q) c.V[3 * r + q] = quot((Sq[3 * r + q] * norm * ts) + (R)(r == q) * (ta - ts), ta);
}

// contains_nan over the conservative and primitive lists of one cell.
template <typename PT, typename R = typename PT::real>
TJ_DEV bool cell_has_nan(const PT& P, const CellT<R>& c)
{
    bool n = false;
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) n |= isnan(c.alpha[m]) || isnan(c.arho[m]) || isnan(c.rhok[m]);
#pragma unroll
    for (int r = 0; r < 3; ++r) n |= isnan(c.rhou[r]) || isnan(c.vel[r]);
    n |= isnan(c.E) || isnan(c.p);
    if (P.solid)
#pragma unroll
        for (int q = 0; q < 9; ++q) n |= isnan(c.V[q]);
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) n |= isnan(c.eps[m]) || isnan(c.are[m]);
    if (P.nmix) n |= isnan(c.lam) || isnan(c.arl);
    return n;
}

// pressureBased_UpdateMassFraction (reactive.cpp:3-26) for the mixture
// (material 0): alphaRhoLambda after one Euler step of the pressure-based burn
// d(alpha rho lambda)/dt = -20 (alpha rho)^0.5 (alpha rho lambda)^0.5 (p/1e6)^1.2,
// clipped at 0; cells with alpha < 0.5 keep their value.
template <typename R>
__device__ __forceinline__ R reactive_euler(R arl, R arho, R p, R alpha, R dt)
{
    const R sigma = R(20.0), nu = R(0.5), n = R(1.2);
    if (alpha < R(0.5)) return arl;
    R r = arl - (dt) * (sigma * tjm_pow(arho, R(1.0) - nu) * tjm_pow(arl, nu) * tjm_pow((quot(p, R(1E6))), n));
    if (r < R(0.0)) r = R(0.0);
    return r;
}

// reactiveUpdate (reactive.cpp:60-103) on one cell: two Euler steps from the
// same alphaRho, pressure and alpha, averaged with the start value, then
// conservativeToPrimitive. Returns the c2p status.
template <typename PT, typename R = typename PT::real>
TJ_DEV int reactive_cell(const PT& P, CellT<R>& c, R dt)
{
    const R a0 = c.arl;
    const R a1 = reactive_euler(a0, c.arho[0], c.p, c.alpha[0], dt);
    const R a2 = reactive_euler(a1, c.arho[0], c.p, c.alpha[0], dt);
    c.arl = (a0 * (R(1.0) / R(2.0))) + (a2 * (R(1.0) / R(2.0)));
    return c2p(P, c);
}

// addGeometricSourceTerm (radial.cpp:5-31) on one cell: every conservative
// variable gains dt * (multiplier / r) * geometricFlux (flux.cpp:51-77), with
// r = (i + 0.5) dx[0] and multiplier -2 in 1-D (spherical symmetry), -1 in 2-D
// and 3-D (cylindrical). `sg` is the stress the reference's state holds at that
// point and the velocity is the cell's; neither changes while the conservative
// variables are updated, so the per-cell order is the reference's.
template <typename PT, typename R = typename PT::real>
TJ_DEV void radial_source(const PT& P, CellT<R>& c, const R* sg, int i, double dx0, R dt)
{
    const R inv_r = quot(R(P.dim == 1 ? -2.0 : -1.0), ((R)i + R(0.5)) * (R)dx0);
    const R s = dt * inv_r;
    const R u = c.vel[0];
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        c.alpha[m] += s * R(0.0);
        c.arho[m] += s * (c.arho[m] * u);
    }
    c.rhou[0] += s * (((c.rhou[0] * u) - sg[0]) + sg[8]);
    c.rhou[1] += s * ((c.rhou[1] * u) - sg[1]);
    c.rhou[2] += s * (R(-2.0) * sg[2]);
    R vds = R(0.0);  // vdotsigma (flux.cpp:19-29) along x
#pragma unroll
    for (int r = 0; r < 3; ++r) vds += c.vel[r] * sg[3 * r];
    if constexpr (sizeof(R) == 4) dd_add32(c.E, c.Elo, s * ((c.E * u) - vds));
    else c.E += s * ((c.E * u) - vds);
    if (P.nmix) c.arl += s * (c.arl * u);
    if (P.solid) {
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const R g = (q < 6) ? (R(1.0) / R(3.0)) * c.V[q] * u : -(R(2.0) / R(3.0)) * c.V[q] * u;
            c.V[q] += s * g;
        }
        if (P.plastic)
            #pragma unroll UnrollM<PT>::n
            for (int m = 0; m < P.M; ++m) c.are[m] += s * (c.are[m] * u);
    }
}

// ---------------------------------------------------------------------------
// Update of one direction; last direction: c2p; second stage: average and
// the post-advance operators of main.cpp:145-187.
// ---------------------------------------------------------------------------
// Flux words of the two faces of a cell in the face arrays (side 0: the
// face below the cell along d, 1: the face above).
template <typename R>
struct FacePairGlobal {
    const R *F0, *F1;  // at the faces
    long long nf;
    __device__ __forceinline__ R operator()(int w, int s) const { return (s ? F1 : F0)[(long long)w * nf]; }
};

// Adds the update along d of one cell from the fluxes of its two faces
// (FXW(w, side)) to its accumulator Yc (hllc.cpp:493-523); U is the cell's
// stage input.
template <typename PT, typename FA, typename R = typename PT::real>
__device__ __forceinline__ void add_fluxes(const PT& P, const CellT<R>& U, CellT<R>& Yc, R dtdx, const FA& FXW)
{
    #pragma unroll UnrollM<PT>::n
    for (int m = 0; m < P.M; ++m) {
        Yc.alpha[m] += dtdx * (FXW(P.X_ALPHA + m, 0) - FXW(P.X_ALPHA + m, 1) - U.alpha[m] * (FXW(P.X_SSTAR, 0) - FXW(P.X_SSTAR, 1)));
        Yc.arho[m] += dtdx * (FXW(P.X_ARHO + m, 0) - FXW(P.X_ARHO + m, 1));
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) Yc.rhou[r] += dtdx * (FXW(P.X_RHOU + r, 0) - FXW(P.X_RHOU + r, 1));
    if constexpr (sizeof(R) == 4) dd_add32(Yc.E, Yc.Elo, dtdx * (FXW(P.X_E, 0) - FXW(P.X_E, 1)));
    else Yc.E += dtdx * (FXW(P.X_E, 0) - FXW(P.X_E, 1));
    if (P.solid)
#pragma unroll
        for (int qq = 0; qq < 9; ++qq) {
            int row = qq / 3, col = qq % 3;
            Yc.V[qq] += dtdx * (FXW(P.X_V + qq, 0) - FXW(P.X_V + qq, 1) -
                                (R(2.0) / R(3.0)) * U.V[qq] * (FXW(P.X_SSTAR, 0) - FXW(P.X_SSTAR, 1)) +
                                U.vel[row] * (FXW(P.X_VSTAR + col, 0) - FXW(P.X_VSTAR + col, 1)));
        }
    if (P.plastic)
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) Yc.are[m] += dtdx * (FXW(P.X_ARE + m, 0) - FXW(P.X_ARE + m, 1));
    if (P.nmix) Yc.arl += dtdx * (FXW(P.X_ARL, 0) - FXW(P.X_ARL, 1));
}

// The end of a stage of one cell whose accumulator holds every direction's
// update: conservativeToPrimitive; second stage: the average and the
// post-advance operators of main.cpp:145-187.
template <typename PT, typename YP, typename AP, typename R = typename PT::real>
__device__ __forceinline__ void finish_cell(const PT& P, DevScalars* scal, bool last_box, CellT<R>& Yc, const YP& Y,
                                            const AP& A, long long nt, long long g, const DevDomain& D, int i,
                                            int finish, R dtdx_num)
{
    const int ce = c2p(P, Yc);
    if (ce) set_status(scal, ce);
    if (finish) {
        const R p_stage = Yc.p;  // U2's pressure, before the average
        // U1 = U*0.5 + U2*0.5 over every carried component (hllc.cpp:705)
        CellT<R> A0;
        load_state(P, A, nt, g, nullptr, A0);
        #pragma unroll UnrollM<PT>::n
        for (int m = 0; m < P.M; ++m) {
            Yc.alpha[m] = mean(A0.alpha[m], Yc.alpha[m]);
            Yc.arho[m] = mean(A0.arho[m], Yc.arho[m]);
            Yc.rhok[m] = mean(A0.rhok[m], Yc.rhok[m]);
            if (P.plastic) {
                Yc.eps[m] = mean(A0.eps[m], Yc.eps[m]);
                Yc.are[m] = mean(A0.are[m], Yc.are[m]);
            }
        }
        Yc.rho = mean(A0.rho, Yc.rho);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            Yc.rhou[r] = mean(A0.rhou[r], Yc.rhou[r]);
            Yc.vel[r] = mean(A0.vel[r], Yc.vel[r]);
        }
        if constexpr (sizeof(R) == 4) avg_pair32(A0.E, A0.Elo, Yc.E, Yc.Elo);
        else Yc.E = mean(A0.E, Yc.E);
        Yc.p = mean(A0.p, Yc.p);
        if (P.solid) {
#pragma unroll
            for (int qq = 0; qq < 9; ++qq) Yc.V[qq] = mean(A0.V[qq], Yc.V[qq]);
            Yc.hj2 = mean(A0.hj2, Yc.hj2);
        }
        if (P.nmix) {
            Yc.rm0 = mean(A0.rm0, Yc.rm0);
            Yc.rm1 = mean(A0.rm1, Yc.rm1);
            Yc.lam = mean(A0.lam, Yc.lam);
            Yc.arl = mean(A0.arl, Yc.arl);
        }
        if (finish == 2) {  // advance() alone: the average only
            store_state(P, A, nt, g, Yc);
            return;
        }
        if (P.reactive && P.nmix) {  // main.cpp:149-152
            const int re = reactive_cell(P, Yc, dtdx_num);
            if (re) set_status(scal, re);
        }
        if (P.plastic) {
            int e;
            if constexpr (sizeof(R) == 4) e = plastic_cell_proj64(P, Yc);
            else e = plastic_cell(P, Yc);
            c2p(P, Yc);
            if (e) set_status(scal, e);
        }
        if (P.radial) {
            // the stress the reference's U1 holds here: fresh from the
            // c2p of the plastic or the reactive update, else the
            // average of U's and U2's (fluids only: -p I each,
            // boxaccesscellarray.cpp:204-212)
            const bool fresh = P.plastic || (P.reactive && P.nmix);
            R sg[9];
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int qq = 0; qq < 3; ++qq) {
                    const R dl = (R)(r == qq);
                    sg[3 * r + qq] = fresh ? Yc.sigma[3 * r + qq]
                                               : ((-A0.p * dl) * (R(1.0) / R(2.0))) +
                                                     ((-p_stage * dl) * (R(1.0) / R(2.0)));
                }
            radial_source(P, Yc, sg, i, D.dx[0], dtdx_num);
            const int rc = c2p(P, Yc);  // geometricSourceTerm (radial.cpp:50)
            if (rc) set_status(scal, rc);
        }
        if (P.solid) cleanup_v_cell(P, Yc);
        int e = cleanup_alpha(P, Yc.alpha);
        if (e) set_status(scal, e);
        if (last_box && cell_has_nan(P, Yc)) atomicOr(&scal->nan_flag, 1);
        store_state(P, A, nt, g, Yc);
        return;
    }
    store_state(P, Y, nt, g, Yc);
}

// Update of cell g along d alone, from the accumulator in Y (the stage input
// for the first direction), with the stage's end after the last direction.
template <typename PT, typename XP, typename YP, typename AP, typename FA, typename R = typename PT::real>
__device__ __forceinline__ void update_cell(const PT& P, DevScalars* scal, bool last_box, const XP& X, const YP& Y,
                                            const AP& A, long long nt, long long g, const DevDomain& D, int i, int d,
                                            int first, int last, int finish, R dtdx_num, const FA& FXW)
{
    CellT<R> U, Yc;
    load_state(P, X, nt, g, nullptr, U);
    if (first) Yc = U;
    else load_state(P, Y, nt, g, nullptr, Yc);
    add_fluxes(P, U, Yc, quot(dtdx_num, (R)D.dx[d]), FXW);
    if (last) finish_cell(P, scal, last_box, Yc, Y, A, nt, g, D, i, finish, dtdx_num);
    else store_state(P, Y, nt, g, Yc);
}

// Update of a whole stage: every direction's fluxes (the update is unsplit:
// they all come from the same stage input) in the order x, y, z, then the
// stage's end. One pass over the state instead of one per direction that
// carries the accumulator through memory: the words a copper cell moves a
// stage fall from about 200 to 103, the same arithmetic in the same order.
// Two instances: the first stage's has no code for the second's end (FIN).
template <typename PT, bool FIN, typename R = typename PT::real>
__global__ void __launch_bounds__(kPathThreads<PT>, kUpdateBlocks<PT>)
    k_update_all(PT P, PathBufs<typename PT::real> b, const R* __restrict__ X, R* Y, int finish)
{
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot;
    const R dtdx_num = b.scal->dt;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nt; g += (long long)gridDim.x * blockDim.x) {
        const int q = find_dom(b.doms, b.ndom, g);
        const DevDomain D = b.doms[q];
        int i, j, k;
        split3(g - D.off, D.n[0], D.n[1], i, j, k);
        CellT<R> U, Yc;
        load_state(P, X, nt, g, nullptr, U);
        Yc = U;
        const R* FX = b.FX;
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d < P.dim) {
                const FacePairGlobal<R> fx{FX + face_index(D, d, i, j, k),
                                           FX + face_index(D, d, i + (d == 0), j + (d == 1), k + (d == 2)), b.nftot[d]};
                add_fluxes(P, U, Yc, quot(dtdx_num, (R)D.dx[d]), fx);
                FX += P.NX * b.nftot[d];
            }
        finish_cell(P, b.scal, b.cell_box[g] == D.nbox - 1, Yc, Y, b.A, nt, g, D, i, FIN ? finish : 0, dtdx_num);
    }
}

template <typename PT, int DC = -1, typename R = typename PT::real>
__global__ void __launch_bounds__(kPathThreads<PT>, kUpdateBlocks<PT>)
    k_update(PT P, PathBufs<typename PT::real> b, const R* __restrict__ X, R* Y, int dyn_d, int first, int last,
             int finish)
{
    const int d = DC >= 0 ? DC : dyn_d;
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot, nf = b.nftot[d];
    const R dtdx_num = b.scal->dt;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nt; g += (long long)gridDim.x * blockDim.x) {
        const int q = find_dom(b.doms, b.ndom, g);
        const DevDomain D = b.doms[q];
        long long l = g - D.off;
        int i, j, k;
        split3(l, D.n[0], D.n[1], i, j, k);
        int o[3] = {0, 0, 0};
        o[d] = 1;
        const FacePairGlobal<R> fx{b.FX + face_index(D, d, i, j, k), b.FX + face_index(D, d, i + o[0], j + o[1], k + o[2]), nf};
        update_cell(P, b.scal, b.cell_box[g] == D.nbox - 1, X, Y, b.A, nt, g, D, i, d, first, last, finish, dtdx_num, fx);
    }
}

// ---------------------------------------------------------------------------
// CFL (timestep.cpp:7-70) and device-side time bookkeeping (main.cpp:121-143).
// ---------------------------------------------------------------------------
template <typename PT, typename R = typename PT::real>
__global__ void k_cfl(PT P, PathBufs<typename PT::real> b, const R* __restrict__ X)
{
    overlap_start(b);
    if (b.scal->done) return;
    const long long nt = b.ntot;
    R mn = R(sizeof(R) == 4 ? 3.0e38 : 1.79769313486231570815e+308);
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < nt; g += (long long)gridDim.x * blockDim.x) {
        const int q = find_dom(b.doms, b.ndom, g);
        const DevDomain D = b.doms[q];
        CellT<R> c;
        load_state(P, X, nt, g, nullptr, c);
        R a = sound_speed(P, c);
#pragma unroll
        for (int n = 0; n < 3; ++n)
            if (n < P.dim) {
                R v = quot((R)D.dx[n], a + fabs(c.vel[n]));
                if (v < mn) mn = v;
            }
    }
    for (int s = 16; s > 0; s >>= 1) {
        R o = __shfl_down_sync(0xffffffffu, mn, s);
        if (o < mn) mn = o;
    }
    __shared__ R red[32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) red[w] = mn;
    __syncthreads();
    if (w == 0) {
        mn = (lane < (int)(blockDim.x >> 5)) ? red[lane] : R(sizeof(R) == 4 ? 3.0e38 : 1.79769313486231570815e+308);
        for (int s = 16; s > 0; s >>= 1) {
            R o = __shfl_down_sync(0xffffffffu, mn, s);
            if (o < mn) mn = o;
        }
        if (lane == 0) atomicMin(&b.scal->dtmin_bits, (unsigned long long)__double_as_longlong((double)mn));
    }
}

}  // namespace tj
