// hype_stage_tile.cuh -- the tile function of the fused FP64 stage kernel,
// shared by the primitive-variable kernels (hype_stage.cu: grid and persistent
// forms) and the conservative-variable kernels (hype_stage_cons.cu).
//
// One launch of a stage kernel evaluates HyPE-2D's right-hand side L(S)
// (RHSFunctionPrim, rhs_function_prim.c:12-626, or RHSFunction,
// rhs_function.c:12-625) on the stage input S and writes one SSP-RK stage
// combination of it, folding the CFL wave-speed maximum
// (rhs_function_prim.c:617-623) into a device scalar.
//
// Tiling.  A tile is a strip of up to CELLS-2 columns and a run of rows of one
// grid, processed by a block of 2*CELLS threads, two per column.  The block
// marches up its rows; at row r the thread pair m reconstructs the cell in
// column x0-1+m (the strip plus one ring column each side), so only two of
// CELLS reconstructions per row are repeated by the neighbouring strip.  Rows
// of the conserved state arrive by one TMA 3-D box load per row (all fields,
// columns x0-4 .. x0+CELLS+1) into a ring of STAGE_SLOTS shared-memory rows,
// are patched at domain edges with the boundary-condition copies, and are
// converted to primitive variables in place (primitive path).  Reconstruction
// coefficients go to shared memory, the x-face Riemann problem at the left of
// each column is solved by that column's pair from its own and its left
// neighbour's coefficients, the y-face problem below each cell by the cell's
// pair from its coefficients and the top-face values it kept from the row
// below.  Row r-1 is completed (y-flux difference, volume non-conservative
// term, RK combination) while row r is processed.
//
// One pass over a cell's coefficients gives every point value the row needs:
// the values at the four faces' Gauss point q = h, which are also the nodes of
// the admissibility check, and at the half's volume Gauss points.  The points
// differ by signs only, so the pass forms each product coefficient x |basis
// value| once and adds or subtracts it (a product changes only its sign with
// its factor's: same bits).  The left and right values then replace the
// coefficients in shared memory, the top values stay for the row above, the
// bottom and volume values in registers.
//
// What bounds the tile is FP64 issue: dependent FP64 chains at 8 or 16 warps per SM.
// Point values come from one pass, the admissibility divisions are left to the few cells
// that need them, products that are zero take no sums or shuffles, and divisions are
// branch-free chains that interleave (hype_div.cuh).  Right-hand sides from and to device
// memory: Kapila N = 2 2048^2 1.46 ms, Euler 1531x897 0.287, BN 1024^2 0.642, Kapila N = 3 500^2
// 0.166; with a pass per use of the point values, the compiler's divisions and a conversion
// to planes 2.09, 0.414, 0.945 and 0.278.
//
// Two block barriers a row (where the fluxes share the coefficients' memory, also a count
// of the warps that have read their neighbours', which a warp waits for before its first
// coefficient replaces them): after the first, the neighbours' face values are
// there, and row r+3 (loaded in the previous iteration) is converted beside
// the x-face problems; the second makes the x fluxes and that row visible.
//
// Compiled with --fmad=false: arithmetic rounds exactly as the reference's C does.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include "hype_internal.h"
#include "hype_physics_fast.cuh"
#include "hype_tma.cuh"

namespace hype {

// The stage parameters a persistent kernel's tile reads, copied to shared memory for each
// work item.  What a batch instance never has (slab and block offsets, interleaved output,
// a run range, the test hook) is a constant: the tile drops its code, and the struct leaves
// room for two blocks per SM.
template <int MODE>
struct BatchParamsOf {
    static constexpr int mode = MODE;
    int nx, ny, pitch, strips, runs, reduce_smax;
    int bc[4];
    long long plane;
    EosBase eos;
    double r1_h, ka, kb, kc, mu1, mu2;
    const double *in, *xn, *inlet;
    double *out, *out2;
    DevScalars *sc;
    static constexpr int out_aos = 0, row_off = 0, col_off = 0, skip_loads = 0, skip_loads_from = 0;
    static constexpr int push_shift_lo = 0, push_shift_hi = 0;
    static constexpr long long push_plane_lo = 0, push_plane_hi = 0;
    static constexpr double *push_lo = nullptr, *push_hi = nullptr;
    __device__ __forceinline__ void load(const StageParams &p, int refine)
    {
        nx = p.nx; ny = p.ny; pitch = p.pitch; strips = p.strips; runs = p.runs * refine;
        reduce_smax = p.reduce_smax;
        for (int k = 0; k < 4; ++k) bc[k] = p.bc[k];
        plane = p.plane;
        eos = p.eos;
        r1_h = p.r1_h; ka = p.ka; kb = p.kb; kc = p.kc; mu1 = p.mu1; mu2 = p.mu2;
        in = p.in; xn = p.xn; inlet = p.inlet; out = p.out; out2 = p.out2; sc = p.sc;
    }
};

struct BatchParams : BatchParamsOf<OUT_AXPY> {   // the mode at run time (conservative and viscous kinds)
    int mode;
    __device__ __forceinline__ void load(const StageParams &p, int refine)
    {
        BatchParamsOf<OUT_AXPY>::load(p, refine);
        mode = p.mode;
    }
};

// The parameters of a right-hand side from and to cell-major arrays: what it never needs of the
// stage combinations, slabs and blocks is a constant.
struct RhsParams : StageParams {
    static constexpr int mode = OUT_RHS, out_aos = 1, row_off = 0, col_off = 0;
    static constexpr double kb = 1.0;
    static constexpr double *push_lo = nullptr, *push_hi = nullptr;
};

// The parameters of a stage combination of a whole grid (no slab, block or interleaved output).
// The kernels of the time loop know their mode: 10 steps of 256^2 Kapila 2.56 -> 2.42 ms, a
// 2048^2 stage 1.50 -> 1.45.
template <int MODE>
struct ModeParams : StageParams {
    static constexpr int mode = MODE, out_aos = 0, row_off = 0, col_off = 0;
    static constexpr double *push_lo = nullptr, *push_hi = nullptr;
};

// The SSP plans (ssp_plan) add OUT_AXPY stages, one that mixes in u^n, and for N = 3 a fifth one
// of its own
template <int N> constexpr int MIX_MODE = N == 2 ? OUT_ZXS : OUT_ZSX;

template <int SYS, int N, int CELLS_>
struct StageKernel {
    using S = System<SYS>;
    using QD = Quad<N>;
    static constexpr int NV = S::NV;
    static constexpr int CELLS = CELLS_;         // reconstruction columns per tile
    static constexpr int NT = 2 * CELLS;         // two threads per cell
    static constexpr int BW = stage_box_width(CELLS, NV);   // TMA box width
    static constexpr int SLOTS = STAGE_SLOTS;
    static constexpr int NDOF = QD::NDOF;
    static constexpr int NC = NDOF - 1;                    // stored coefficients (k >= 1)
    static constexpr int ROW_ELEMS = BW * NV;
    // cell-major input: a row's elements (those the stencils read, rounded to 128 bytes) in
    // boxes of at most 256, each at a 128-byte offset; the last one ends with the row, over part
    // of the one before
    static constexpr int AOS_ELEMS = ROW_ELEMS / 16 * 16, AOS_PARTS = (AOS_ELEMS + 255) / 256;
    static constexpr int AOS_BOX = (AOS_ELEMS / AOS_PARTS + 15) / 16 * 16;
    static constexpr int aos_at(int k) { return k + 1 < AOS_PARTS ? k * AOS_BOX : AOS_ELEMS - AOS_BOX; }
    static_assert(AOS_ELEMS >= (CELLS + 5) * NV && AOS_BOX <= 256 && AOS_PARTS * AOS_BOX >= AOS_ELEMS, "cell-major boxes cover the stencils");
    static constexpr int ROW_BYTES = ROW_ELEMS * 8;
    static constexpr int SLOT_STRIDE = ((ROW_BYTES + 127) / 128) * 128 / 8;   // doubles
    // components with a non-conservative product (the same ones on the conservative path)
    static constexpr int nz(int c)   // its index among them, -1 where there is none
    {
        if (!S::ncp_nonzero(c)) return -1;
        int z = 0;
        for (int k = 0; k < c; ++k) z += S::ncp_nonzero(k) ? 1 : 0;
        return z;
    }
    static constexpr int count_nz() { int z = 0; for (int c = 0; c < S::NV; ++c) z += S::ncp_nonzero(c) ? 1 : 0; return z; }
    static constexpr int NZ = count_nz();
    // per-cell arrays, [k][c][cell] so consecutive cells hit consecutive banks.  Coefficients
    // k >= 1; later, by slot, the left and right face values at each Gauss point (2 q, 2 q + 1)
    // and, without FX_OWN, the x-face fluxes (slot 0) and fluctuations (slot 2)
    static constexpr int COEF_ELEMS = (NC > 3 ? NC : 3) * NV * CELLS;
    static constexpr int YT_ELEMS = 2 * QD::NFGP * NV * CELLS;                 // top-face values of rows r-1 and r, by Gauss point
    static constexpr int CARRY_ELEMS = (2 * NV + 2 * NZ) * CELLS;              // t1, G below; ncp, E below
    // the ring, the per-cell arrays and one more row slot: the conserved input of the row
    // being finished (row r-1), for the RK combination
    static constexpr size_t SMEM_BASE = (size_t)(SLOTS + 1) * SLOT_STRIDE * 8 +
                                        (size_t)(COEF_ELEMS + YT_ELEMS + CARRY_ELEMS) * 8 + 64 /* barriers */;
    // blocks the 228 KB of an SM's shared memory holds (1 KB reserved per block, and the
    // persistent form's 256 bytes); the launch bound asks for no more than that, so no register
    // limit is paid for blocks that could not be resident anyway (Kapila N = 3 at 128-column
    // tiles: 1)
    static constexpr int REG_TARGET = (NV <= 6 ? 2 : 1) * (128 / CELLS);
    static constexpr int fit(size_t smem) { return (int)(233472 / (smem + 1024 + 256)); }
    static constexpr int blocks(size_t smem) { return fit(smem) < 1 ? 1 : (fit(smem) < REG_TARGET ? fit(smem) : REG_TARGET); }
    // x-face fluxes and fluctuations, exchanged with the neighbours: an array of their own where
    // that costs no resident block, else coefficient slots, whose reuse has to be waited for (the
    // wait measured 3 % in the Baer-Nunziato and N = 3 tiles, nothing in Kapila N = 2)
    static constexpr int FX_ELEMS = (NV + NZ) * CELLS;
    static constexpr size_t SMEM_MOST = 232448 - 512;   // of one block
    static constexpr bool FX_OWN = SMEM_BASE + FX_ELEMS * 8 <= SMEM_MOST && blocks(SMEM_BASE + FX_ELEMS * 8) == blocks(SMEM_BASE);
    static constexpr size_t SMEM = SMEM_BASE + (FX_OWN ? FX_ELEMS * 8 : 0);
    static constexpr int MIN_BLOCKS = blocks(SMEM);
    static_assert((SLOTS + 2) * 8 <= 64, "the barriers fit their space");
    static constexpr size_t smem_bytes() { return SMEM; }
};

// x with its sign flipped where mask = 0x80000000 (0: unchanged)
__device__ __forceinline__ double flip_sign(double x, unsigned mask)
{
    return __hiloint2double((int)((unsigned)__double2hiint(x) ^ mask), __double2loint(x));
}

// v + ck * p, where p is P0 for half 0 of the pair and P1 for half 1 and |P0| = |P1|.
// `mask` flips half 0's sign.  The product is formed with |p| and added or subtracted,
// so that points whose basis values differ in sign share it; FAST fuses each term instead.
template <bool FAST, class P>
__device__ __forceinline__ double add_term(double v, double ck, unsigned mask)
{
    constexpr double p0 = P::p0(), p1 = P::p1(), a = p1 < 0.0 ? -p1 : p1;
    static_assert(p0 == p1 || p0 == -p1, "the halves' points mirror each other");
    if constexpr (a == 0.0) {
        return v;   // the reference adds ck * 0 to a sum that is never -0
    } else if constexpr (p0 == p1) {
        const double t = a == 1.0 ? ck : ck * a;
        return p1 > 0.0 ? v + t : v - t;
    } else if constexpr (FAST) {
        const double cs = flip_sign(ck, mask);
        return p1 > 0.0 ? v + cs * a : v - cs * a;
    } else {
        const double t = flip_sign(ck * a, mask);
        return p1 > 0.0 ? v + t : v - t;
    }
}
// the basis values of coefficient K at the points of halves 0 and 1: face F's Gauss point
// q = half; the half's volume Gauss point A, values and derivatives
template <int N, int F, int K> struct FacePt {
    static constexpr double p0() { return Quad<N>::phi_face(F, 0, K); }
    static constexpr double p1() { return Quad<N>::phi_face(F, Quad<N>::NFGP > 1 ? 1 : 0, K); }
};
template <int N, int A, int K> struct VolPt {
    static constexpr int q1 = Quad<N>::NVGP > 1 ? Quad<N>::NVGP / 2 + A : A;
    static constexpr double p0() { return Quad<N>::phi_vol(A, K); }
    static constexpr double p1() { return Quad<N>::phi_vol(q1, K); }
};
template <int N, int A, int D, int K> struct VolGrad {
    static constexpr int q1 = VolPt<N, A, K>::q1;
    static constexpr double p0() { return D == 0 ? Quad<N>::dphi_vol_x(A, K) : Quad<N>::dphi_vol_y(A, K); }
    static constexpr double p1() { return D == 0 ? Quad<N>::dphi_vol_x(q1, K) : Quad<N>::dphi_vol_y(q1, K); }
};
// One variable's polynomial at face F's Gauss point of the half, terms in ascending k as the
// reference's loops.  The reference starts from 0.0: 0.0 + c0 differs from c0 for c0 = -0 only,
// and a zero's sign reaches no result (every flux and product sum starts from +0).
template <int N, int F, bool FAST>
__device__ __forceinline__ double face_pt(const double *cf, unsigned mask)
{
    double v = cf[0];
    static_for<Quad<N>::NDOF - 1>([&](auto kk) { constexpr int k = decltype(kk)::value + 1; v = add_term<FAST, FacePt<N, F, k>>(v, cf[k], mask); });
    return v;
}
template <int N, int A, bool FAST>
__device__ __forceinline__ double vol_pt(const double *cf, unsigned mask)
{
    double v = cf[0];
    static_for<Quad<N>::NDOF - 1>([&](auto kk) { constexpr int k = decltype(kk)::value + 1; v = add_term<FAST, VolPt<N, A, k>>(v, cf[k], mask); });
    return v;
}
template <int N, int A, int D, bool FAST>
__device__ __forceinline__ double vol_grad(const double *cf, unsigned mask)
{
    if constexpr (N == 0) {
        return 0.0;
    } else {
        constexpr int first = 1 + D;   // the linear coefficient along D, basis derivative 1
        double v = cf[first];
        static_for<Quad<N>::NDOF - 1 - first>([&](auto kk) {
            constexpr int k = decltype(kk)::value + 1 + first;
            v = add_term<FAST, VolGrad<N, A, D, k>>(v, cf[k], mask);
        });
        return v;
    }
}

// Gradient component D (0: x, 1: y) of one variable at Gauss point q of face
// F from its unlimited coefficients uc: sum_k uc[k] gradphiFace_D(F, q, k) from
// 0.0 in ascending k (rhs_function_prim.c:362-369), before the 1/h factor.
// Terms of zero basis gradients are dropped (add_term).
template <int N, int F, int D>
__device__ __forceinline__ double face_grad(const double *uc, int q)
{
    using QD = Quad<N>;
    double v = 0.0;
    static_for<QD::NDOF>([&](auto kk) {
        constexpr int k = decltype(kk)::value;
        constexpr double p0 = QD::dphi_face(F, 0, D, k);
        constexpr double p1 = QD::dphi_face(F, QD::NFGP > 1 ? 1 : 0, D, k);
        if constexpr (p0 == p1) {
            if constexpr (p0 != 0.0) {
                if constexpr (p0 == 1.0) v = v + uc[k];
                else v = v + uc[k] * p0;
            }
        } else {
            const double p = q ? p1 : p0;
            v = v + uc[k] * p;
        }
    });
    return v;
}

// riemann.c:112-140 (RiemannSolverPrim) at one face Gauss point, n = e_x (DIR 0) or e_y
// (DIR 1), dividing by dv; S is the system's physics (System<SYS>, or FastSystem<SYS> for the
// FP64 performance form)
template <class S, int DIR, class E, class Dv>
__device__ __forceinline__ double riemann_prim(const E &eos, Dv &dv, const double *VL, const double *VR, double *F, double *D, bool &bad)
{
    constexpr int NV = S::NV;
    constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
    double QL[NV], QR[NV], FL[NV], FR[NV];
    S::prim2cons(eos, dv, VL, QL);
    S::prim2cons(eos, dv, VR, QR);
    const double sl = S::template flux<DIR>(eos, dv, VL, FL, bad);
    const double sr = S::template flux<DIR>(eos, dv, VR, FR, bad);
    const double s = (sl < sr) ? sr : sl;
    double Vav[NV], gx[NV], gy[NV];
#pragma unroll
    for (int c = 0; c < NV; ++c) {
        Vav[c] = 0.5 * (VR[c] + VL[c]);
        gx[c] = nx * (VR[c] - VL[c]);
        gy[c] = ny * (VR[c] - VL[c]);
        F[c] = 0.5 * (FR[c] + FL[c] - s * (QR[c] - QL[c]));
    }
    S::ncp(eos, dv, Vav, gx, gy, D);
    return s;
}

// one face Gauss point: RiemannSolverPrim (VL/VR primitive) or, for the conservative path,
// riemann.c:52-105 (RiemannSolver, VL/VR conserved).  CR: the branch-free divisions, and the
// compiler's for the few points outside their range.  Measured: BN 1024^2 right-hand side
// 0.780 -> 0.736 ms, Kapila N = 3 500^2 0.256 -> 0.246, Kapila N = 2 64^2 113.7 -> 110.2 us,
// 2048^2 and Euler even
template <class S, int DIR, bool CONS, bool CR, class E>
__device__ __forceinline__ double riemann_gp(const E &eos, const double *VL, const double *VR, double *F, double *D, bool &bad)
{
    constexpr int NV = S::NV;
    constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
    if constexpr (CONS) {
        double FL[NV], FR[NV];
        const double sl = S::template flux_cons<DIR>(eos, VL, FL, bad);
        const double sr = S::template flux_cons<DIR>(eos, VR, FR, bad);
        const double s = (sl < sr) ? sr : sl;
        double Qav[NV], gx[NV], gy[NV];
#pragma unroll
        for (int c = 0; c < NV; ++c) {
            Qav[c] = 0.5 * (VR[c] + VL[c]);
            gx[c] = nx * (VR[c] - VL[c]);
            gy[c] = ny * (VR[c] - VL[c]);
            F[c] = 0.5 * (FR[c] + FL[c] - s * (VR[c] - VL[c]));
        }
        S::ncp_cons(eos, Qav, gx, gy, D);
        return s;
    }
    if constexpr (CR) {
        CrDiv dv;
        bool b = false;
        const double s = riemann_prim<S, DIR>(eos, dv, VL, VR, F, D, b);
        if (eos.cr && !dv.special()) {
            bad |= b;
            return s;
        }
    }
    IeeeDiv dv;
    return riemann_prim<S, DIR>(eos, dv, VL, VR, F, D, bad);
}

// One tile of one grid: columns of strip `strip` (of p.strips) and rows of run
// `run` (of p.runs).  Called by every thread of a block of K::NT threads.
// CONS: the conservative-variable RHS (RHSFunction, rhs_function.c:12-625):
// no conversion of the staged rows, PDECheckPAD / PDEFlux / PDENCP on
// conserved values, and a PAD fallback that keeps only the cell mean.
// VISC: the reference's VISCOUS build (Kapila, N >= 1): walls also negate the
// tangential velocity, every face Gauss point adds the mean of the two sides'
// viscous fluxes (riemann.c:146-186) with gradients taken from the unlimited
// coefficients (rhs_function_prim.c:356-374), and the viscous eigenvalue
// maximum goes to DevScalars.smax_v for the dt (rhs_function_prim.c:617).
// FAST: the FP64 performance form (primitive path only): FastSystem / ReconFast
// of hype_physics_fast.cuh, in a translation unit built with FMA contraction;
// reads the derived constants of p.eos (Eos::derive, filled by the host).
// AOS: the input is the caller's cell-major array (p.in, 16-byte aligned rows) instead of
// planes: a row is loaded as it is and laid out by component when it is converted.
template <int SYS, int N, int CELLS_, bool CONS, bool VISC = false, bool FAST = false, bool AOS = false, class P>
__device__ __forceinline__ void stage_tile(const P &p, const CUtensorMap *tmap, int strip, int run, unsigned char *smem_raw)
{
    static_assert(!(FAST && (CONS || VISC)), "the FP64 performance form covers the primitive inviscid path");
    using K = StageKernel<SYS, N, CELLS_>;
    using S = std::conditional_t<FAST, FastSystem<SYS>, typename K::S>;
    using QD = typename K::QD;
    constexpr int NV = K::NV, CELLS = K::CELLS, BW = K::BW, SLOTS = K::SLOTS, NDOF = K::NDOF, NZ = K::NZ;
    constexpr int NFGP = QD::NFGP, NVGP = QD::NVGP;
    constexpr int NVH = (NV + 1) / 2;          // variables per half in the reconstruction
    constexpr unsigned FULL = 0xffffffffu;
    constexpr bool HAS_PAD = CONS ? N >= 1 : N >= 2;   // orders whose coefficients the admissibility check can replace

    if (p.sc->idle) return;   // finished or held run (set by begin_step; 0 outside a time loop)

    double *rows_s = reinterpret_cast<double *>(smem_raw);
    // conserved input of row r-1 (the row the RK combination finishes), [c][BW], its own mbarrier
    double *orow_s = rows_s + (size_t)SLOTS * K::SLOT_STRIDE;
    double *coef_s = orow_s + K::SLOT_STRIDE;                   // [slot][c][cell]
    double *yt_s = coef_s + K::COEF_ELEMS;                      // [row parity][q][c][cell]
    double *carry_s = yt_s + K::YT_ELEMS;                       // t1, G below [c][cell]; ncp, E below [z][cell]
    uint64_t *bars = reinterpret_cast<uint64_t *>(carry_s + K::CARRY_ELEMS);
    // one arrival per warp and row, once it has read its neighbours' x-face fluxes: the next row's
    // coefficients may replace them
    uint64_t *fluxes_read = bars + SLOTS + 1;
    // VISC: gradients of the variables the viscous flux reads (primitive u, v;
    // conserved a1r1, a2r2, ru, rv) at the top face, kept for the row above:
    // [q][g][d][cell], at the end
    constexpr int NG = CONS ? 4 : 2, G0 = CONS ? 0 : 2;
    double *fx_s = carry_s + K::CARRY_ELEMS + 8;                // FX_OWN: F [c][cell], D [z][cell]
    double *ygt_s = fx_s + (K::FX_OWN ? K::FX_ELEMS : 0);
    double *red_s = carry_s;                                    // block reductions at the tile's end

    const int t = threadIdx.x;
    const int m = t >> 1;            // cell of this thread's pair
    const int h = t & 1;             // which half of the pair
    const unsigned mask0 = h ? 0u : 0x80000000u;   // half 0's sign (add_term)
    // strips split the columns evenly on even boundaries (TMA x origin alignment);
    // row runs split the rows evenly
    const int x0 = 2 * (int)(((long long)strip * p.nx) / (2LL * p.strips));
    const int x1 = (strip + 1 == p.strips) ? p.nx : 2 * (int)(((long long)(strip + 1) * p.nx) / (2LL * p.strips));
    const int owc = x1 - x0;
    const int y0 = (int)(((long long)run * p.ny) / p.runs);
    const int H = (int)(((long long)(run + 1) * p.ny) / p.runs) - y0;
    if (owc > CELLS - 2 || owc < 1 || H < 1) {   // launch geometry outside what the tiling covers
        if (threadIdx.x == 0) raise_error(p.sc, ERR_BAD_LAUNCH, 0u);
        return;
    }
    const int xs = x0 - 4;                    // TMA box origin (even: x0 is even)
    const int i = x0 - 1 + m;                 // this pair's reconstruction column
    const bool active = m <= owc + 1;
    const bool owned = m >= 1 && m <= owc;
    const bool xface = m >= 1 && m <= owc + 1;
    const bool warp_active = ((t & ~31) >> 1) <= owc + 1;   // some cell of this warp is in the strip
    const bool touches_x = (x0 == 0) || (x0 + owc >= p.nx);
    const int bcL = p.bc[0], bcR = p.bc[1], bcB = p.bc[2], bcT = p.bc[3];
    const bool py = (bcB == BC_PERIODIC || bcT == BC_PERIODIC);
    const double dt = (p.mode == OUT_RHS) ? 0.0 : p.sc->dt;
    const double b = dt / p.kb;   // the RK combination's dt/kb, the same for every row
    const auto &eos = p.eos;
    const double r1_h = p.r1_h;
    const bool quick_eos = S::quick_eos(eos);   // pad_quick's accept holds for these constants

    __syncthreads();   // the previous tile of this block is done with every buffer
    if (t == 0) {
        for (int s = 0; s <= SLOTS; ++s) mbar_init(&bars[s], 1);
        mbar_init(fluxes_read, K::NT / 32);
        fence_mbar_init();
    }
    __syncthreads();

    const int row_lo = y0 - 3, row_hi = y0 + H + 2;   // rows of state this block reads
    int next_issue = row_lo, next_conv = row_lo;
    auto slot_of = [&](int row) { return (row - row_lo) % SLOTS; };
    auto row_ptr = [&](int row) { return rows_s + (size_t)slot_of(row) * K::SLOT_STRIDE; };   // [c][BW]
    auto cidx = [&](int slot, int c, int cell) { return (slot * NV + c) * CELLS + cell; };     // coef_s index
    auto flux_s = [&](int c, int cell) -> double & { return K::FX_OWN ? fx_s[c * CELLS + cell] : coef_s[cidx(0, c, cell)]; };
    auto fluct_s = [&](int c, int z, int cell) -> double & { return K::FX_OWN ? fx_s[(NV + z) * CELLS + cell] : coef_s[cidx(2, c, cell)]; };
    auto t1_s = [&](int c) -> double & { return carry_s[c * CELLS + m]; };
    auto g_s = [&](int c) -> double & { return carry_s[(NV + c) * CELLS + m]; };
    auto ncp_s = [&](int z) -> double & { return carry_s[(2 * NV + z) * CELLS + m]; };
    auto e_s = [&](int z) -> double & { return carry_s[(2 * NV + NZ + z) * CELLS + m]; };
    // Component c = 2 j + h of the half, j compile time: a per-component register array's
    // element, and whether and where the component has a non-conservative product
    auto own = [&](auto jj, const double *a) {
        constexpr int c0 = 2 * decltype(jj)::value, c1 = c0 + 1 < NV ? c0 + 1 : c0;
        return h ? a[c1] : a[c0];
    };
    // the other half's component 2 j + 1 - h of the array, 0 where there is none
    auto other = [&](auto jj, const double *a) {
        constexpr int c0 = 2 * decltype(jj)::value, c1 = c0 + 1 < NV ? c0 + 1 : c0;
        return h ? a[c0] : a[c1];
    };

    // A face's flux of component 2 j + h from its two Gauss points' weighted values, one per half:
    // Flux = 0.0; Flux += w F(q0); Flux += w F(q1)   (rhs_function_prim.c:548-577),
    // VISC: Flux += w Fv(q) after each Gauss point's convective part.  Each half sends the
    // other the component it needs; two terms add up alike in either order
    auto face_sum = [&](auto jj, const double *Fq, const double *Vq) {
        if constexpr (NFGP > 1) {
            const double f = own(jj, Fq), fo = __shfl_xor_sync(FULL, other(jj, Fq), 1);
            if constexpr (VISC) {
                const double v = own(jj, Vq), vo = __shfl_xor_sync(FULL, other(jj, Vq), 1);
                return (((0.0 + (h ? fo : f)) + (h ? vo : v)) + (h ? f : fo)) + (h ? v : vo);
            } else {
                return f + fo;   // (0.0 + f) + fo but for a zero's sign, which the right-hand side's own sums lose
            }
        } else {
            if constexpr (VISC) return (0.0 + own(jj, Fq)) + own(jj, Vq);
            else return 0.0 + own(jj, Fq);
        }
    };
    auto fluct_sum = [&](auto jj, const double *Dq) {
        if constexpr (NFGP > 1) {
            const double d = own(jj, Dq), d_o = __shfl_xor_sync(FULL, other(jj, Dq), 1);
            return d + d_o;
        } else {
            return 0.0 + own(jj, Dq);
        }
    };

    double smax_loc = 0.0, smaxv_loc = 0.0;
    bool bad = false;
    unsigned bad_cell = 0xffffffffu;
    // A bounded wait ran out (ERR_TMA_TIMEOUT): thread 0 waits for the loads still in
    // flight -- ring rows issued but not yet converted, and the finish-row slot while
    // its load is outstanding -- then invalidates the barriers; the block returns.
    auto give_up = [&](bool orow_pending, unsigned orow_parity) {
        if (t != 0) return;
        raise_error(p.sc, ERR_TMA_TIMEOUT, 0u);
        const unsigned long long deadline = global_ns() + TMA_WAIT_NS;
        bool drained = true;
        for (int row = next_conv; row < next_issue; ++row)
            drained = drained && mbar_wait_until(&bars[slot_of(row)], (unsigned)(((row - row_lo) / SLOTS) & 1), deadline);
        if (orow_pending) drained = drained && mbar_wait_until(&bars[SLOTS], orow_parity, deadline);
        if (drained)
            for (int k = 0; k <= SLOTS + 1; ++k) mbar_inval(&bars[k]);
    };
    // thread 0: issue the ring rows up to `last`.  AOS: the prologue's rows land in the memory
    // that the coefficients take later, the others in their ring slots
    double *land_s = coef_s;
    static_assert(!AOS || 5 * K::SLOT_STRIDE <= K::COEF_ELEMS + K::YT_ELEMS + K::CARRY_ELEMS, "the prologue's rows fit");
    auto issue_rows = [&](int last) {
        for (; next_issue <= min(last, row_hi) && (!p.skip_loads || next_issue < p.skip_loads_from); ++next_issue) {
            const int row = next_issue;
            const int src = map_axis(row, p.ny, bcB, bcT);
            uint64_t *bar = &bars[slot_of(row)];
            mbar_expect_tx(bar, AOS ? K::AOS_PARTS * K::AOS_BOX * 8 : K::ROW_BYTES);
            if constexpr (AOS) {
                double *to = row <= y0 + 1 ? land_s + (row - row_lo) * K::SLOT_STRIDE : row_ptr(row);
#pragma unroll
                for (int k = 0; k < K::AOS_PARTS; ++k) tma_load_2d(to + K::aos_at(k), tmap, xs * NV + K::aos_at(k), src, bar);
            } else {
                tma_load_3d(row_ptr(row), tmap, xs + p.col_off, src + p.row_off, 0, bar);   // the map starts col_off columns left of column 0, row_off rows below row 0
            }
        }
    };
    auto wait_row = [&](int row) { return mbar_wait_bounded(&bars[slot_of(row)], (unsigned)(((row - row_lo) / SLOTS) & 1)); };
    // Conserved values of column cc (1 .. owc+6, the ones the stencils read) of a loaded row;
    // ghost columns take their source's
    auto conserved = [&](int row, const double *raw, int cc, double *Q) {
        const int g = xs + cc;
        int col = cc;
        if (g < 0 || g >= p.nx) {
            const int gm = map_axis(g, p.nx, bcL, bcR);
            col = gm - xs;
            if (col < 0 || col >= (AOS ? K::AOS_ELEMS / NV : BW)) {   // the far side of a periodic axis
                const int src = map_axis(row, p.ny, bcB, bcT);
#pragma unroll
                for (int c = 0; c < NV; ++c)
                    Q[c] = AOS ? p.in[((long long)src * p.nx + gm) * NV + c] : p.in[(long long)c * p.plane + (long long)src * p.pitch + gm];
                return;
            }
        }
#pragma unroll
        for (int c = 0; c < NV; ++c) Q[c] = AOS ? raw[col * NV + c] : raw[c * BW + col];
    };
    // Primitive values of a column's conserved ones, reflections and inlet values applied, into
    // its ring row
    auto put_primitive = [&](int row, int cc, const double *Q) {
        double *rp = row_ptr(row);
        const bool yg = row < 0 || row >= p.ny;
        const bool yrefl = yg && ((row < 0 ? bcB : bcT) == BC_REFLECTIVE);
        const int g = xs + cc;
        const bool isg = g < 0 || g >= p.nx;
        double V[NV];
        if constexpr (CONS) {
#pragma unroll
            for (int c = 0; c < NV; ++c) V[c] = Q[c];
        } else if constexpr (!FAST && ((SYS == SYS_BN && (N == 1 || N == 2)) || (SYS == SYS_KAPILA && N <= 1))) {
            // branch-free divisions: the cell's independent ones overlap.  Only in the tiles where
            // it measured faster (BN 1024^2 0.738 -> 0.731 ms; Kapila N = 2 -0.7 % at 128 columns,
            // +1.4 % at 64, N = 3 +0.6 %)
            CrDiv dv;
            S::cons2prim_dv(eos, Q, V, dv);
            if (!eos.cr || dv.special()) S::cons2prim(eos, Q, V);
        } else {
            S::cons2prim(eos, Q, V);
        }
        if (isg) {
            const int side_bc = g < 0 ? bcL : bcR;
            if (side_bc == BC_INLET && p.inlet) {
                const int jr = py ? row : map_axis(row, p.ny, bcB, bcT);
#pragma unroll
                for (int c = 0; c < NV; ++c) V[c] = p.inlet[((size_t)(g + 3) * (p.ny + 6) + (jr + 3)) * NV + c];
            } else if (side_bc == BC_REFLECTIVE) {
                if (S::RX0 >= 0) V[S::RX0] = -V[S::RX0];
                if (S::RX1 >= 0) V[S::RX1] = -V[S::RX1];
                if constexpr (VISC) V[S::RXV] = -V[S::RXV];
            }
        }
        if (yrefl) {
            if (S::RY0 >= 0) V[S::RY0] = -V[S::RY0];
            if (S::RY1 >= 0) V[S::RY1] = -V[S::RY1];
            if constexpr (VISC) V[S::RYV] = -V[S::RYV];
        }
#pragma unroll
        for (int c = 0; c < NV; ++c) rp[c * BW + cc] = V[c];
    };

    // ---------------- prologue: rows y0-3 .. y0+1, row y0+2 in flight --------------
    if (t == 0) {
        fence_proxy_async();   // earlier generic accesses to the slots precede the TMA writes
        issue_rows(y0 + 2);
    }
    {
        const int width = owc + 6;   // converted columns of a row
        bool here = true;
        for (int row = row_lo; row <= y0 + 1; ++row) here = here && wait_row(row);
        if (!AOS && touches_x && here) {   // ghost columns first: the conversion is in place
            for (int k = t; k < 5 * width; k += K::NT) {
                const int row = row_lo + k / width, cc = 1 + k % width, g = xs + cc;
                if (g >= 0 && g < p.nx) continue;
                double Q[NV], *rp = row_ptr(row);
                conserved(row, rp, cc, Q);
#pragma unroll
                for (int c = 0; c < NV; ++c) rp[c * BW + cc] = Q[c];
            }
        }
        if (__syncthreads_or(!here)) {
            give_up(false, 0u);
            return;   // block-uniform exit; the caller's next barrier is block-uniform too
        }
#pragma unroll 1
        for (int k = t; k < 5 * width; k += K::NT) {
            const int row = row_lo + k / width, cc = 1 + k % width;
            double Q[NV];
            if constexpr (AOS) {
                conserved(row, land_s + (row - row_lo) * K::SLOT_STRIDE, cc, Q);
            } else {
                const double *rp = row_ptr(row);
#pragma unroll
                for (int c = 0; c < NV; ++c) Q[c] = rp[c * BW + cc];
            }
            put_primitive(row, cc, Q);
        }
        next_conv = y0 + 2;
    }
    __syncthreads();

    for (int r = y0 - 1; r <= y0 + H; ++r) {
        const bool in_rows = r >= y0;
        const bool full_row = r >= y0 && r < y0 + H;
        const int q = NFGP > 1 ? h : 0;
        const int ccm = m + 3;                                    // column of i in the ring rows
        const double *w_m2 = row_ptr(r - 2), *w_m1 = row_ptr(r - 1), *w_0 = row_ptr(r), *w_p1 = row_ptr(r + 1), *w_p2 = row_ptr(r + 2);
        const bool finish_row = r > y0 && p.mode != OUT_RHS;   // this iteration's RK combination reads row r-1's input
        // VISC: unlimited coefficients of variable c of the cell `cell` of row r, from the ring rows
        auto load_uc = [&](int c, int cell, double *uc) {
            if constexpr (VISC) {
                const int col = cell + 3;
                Stencil st;
                const double *a0 = w_0 + c * BW + col;
                st.c = a0[0];
                st.xm2 = a0[-2]; st.xm1 = a0[-1]; st.xp1 = a0[1]; st.xp2 = a0[2];
                st.ym2 = w_m2[c * BW + col]; st.ym1 = w_m1[c * BW + col]; st.yp1 = w_p1[c * BW + col]; st.yp2 = w_p2[c * BW + col];
                st.pp = w_p1[c * BW + col + 1]; st.pm = w_m1[c * BW + col + 1]; st.mp = w_p1[c * BW + col - 1]; st.mm = w_m1[c * BW + col - 1];
                UCoef<N>::run(st, uc);
            }
        };
        // finish_row: row r-1's conserved input, issued in the previous iteration
        bool here = !finish_row || mbar_wait_bounded(&bars[SLOTS], (unsigned)((r - y0 - 1) & 1));

        if (warp_active) {
        // ---------------- A. reconstruction of cell (r, i), split by variable ---
#pragma unroll 1
        for (int kv = 0; kv < NVH; ++kv) {
            const int c = h * NVH + kv;
            if (c >= NV) break;
            auto stencil = [&] {
                Stencil st;
                const double *a0 = w_0 + c * BW + ccm;
                st.c = a0[0];
                st.xm2 = a0[-2]; st.xm1 = a0[-1]; st.xp1 = a0[1]; st.xp2 = a0[2];
                st.ym2 = w_m2[c * BW + ccm]; st.ym1 = w_m1[c * BW + ccm]; st.yp1 = w_p1[c * BW + ccm]; st.yp2 = w_p2[c * BW + ccm];
                st.pp = w_p1[c * BW + ccm + 1]; st.pm = w_m1[c * BW + ccm + 1]; st.mp = w_p1[c * BW + ccm - 1]; st.mm = w_m1[c * BW + ccm - 1];
                return st;
            };
            auto keep = [&](const double *cf) {
                // the row's first store over the fluxes: most of a reconstruction after they were
                // read, so the wait is over before it begins
                if (!K::FX_OWN && kv == 0 && r >= y0) here = mbar_wait_bounded(fluxes_read, (unsigned)((r - y0) & 1)) && here;
#pragma unroll
                for (int k = 1; k < NDOF; ++k) coef_s[cidx(k - 1, c, m)] = cf[k];
            };
            double cf[NDOF];
            if constexpr (FAST) {
                ReconFast<N>::run(stencil(), cf);
                keep(cf);
            } else if constexpr (N >= 2) {
                // branch-free correctly rounded reciprocals and quotients let the weights' chains
                // overlap; the compiler's division where an operand is outside their range
                // (from the ring again, so that the stencil is not held for it)
                bool special;
                ReconCr<N>::run(stencil(), cf, special);
                keep(cf);
                if (special && active) {
                    Recon<N>::run(stencil(), cf);
                    keep(cf);
                }
            } else {
                Recon<N>::run(stencil(), cf);
                keep(cf);
            }
        }
        __syncwarp();

        // ---------------- B. point values of the cell, all variables ----------------
        // bottom and (old) top values at the y-face's Gauss point, values and gradients at
        // the half's volume Gauss points in registers; left, right and (new) top in shared memory
        constexpr int QH = NVGP > 1 ? NVGP / 2 : 1;
        double VR[NV];                              // bottom values
        const double *yt_lo = yt_s + ((((r - y0) & 1) * NFGP + q) * NV) * CELLS + m;     // top values of row r-1,
        double *yt_up = yt_s + ((((r - y0 + 1) & 1) * NFGP + q) * NV) * CELLS + m;       // and of row r
        double tq[QH][NV] = {};                          // weighted volume products
        bool ok = quick_eos;                        // every node in the plainly admissible range
        // the point values from the coefficients that coef(c, cf) gives
        auto points = [&](auto coef) {
            [[maybe_unused]] double Vv[QH][NV], gx[QH][NV], gy[QH][NV];
            static_for<NV>([&](auto sc_) {
                constexpr int c = S::order(decltype(sc_)::value);   // the product's velocity part first: fewer values wait for it
                double cf[NDOF];
                cf[0] = w_0[c * BW + ccm];
                coef(c, cf);
                const double vl = face_pt<N, 0, FAST>(cf, mask0), vr = face_pt<N, 1, FAST>(cf, mask0);
                const double vt = face_pt<N, 3, FAST>(cf, mask0);
                VR[c] = face_pt<N, 2, FAST>(cf, mask0);
                coef_s[cidx(2 * q, c, m)] = vl;
                coef_s[cidx(2 * q + 1, c, m)] = vr;
                yt_up[c * CELLS] = vt;
                if constexpr (HAS_PAD && !CONS)
                    ok = ok && S::template pad_quick<c>(vl) && S::template pad_quick<c>(vr) && S::template pad_quick<c>(VR[c]) &&
                         S::template pad_quick<c>(vt);
                if constexpr (NZ > 0) {
                    static_for<QH>([&](auto sa) {
                        constexpr int a = decltype(sa)::value;
                        Vv[a][c] = vol_pt<N, a, FAST>(cf, mask0);
                        gx[a][c] = r1_h * vol_grad<N, a, 0, FAST>(cf, mask0);
                        gy[a][c] = r1_h * vol_grad<N, a, 1, FAST>(cf, mask0);
                    });
                }
            });
            // the volume non-conservative products (rhs_function_prim.c:459-479).  CONS, N > 0: of the run's own
            // rows (many divisions a point: Kapila N = 2 64^2 69.5 -> 61.5 us, 1024^2 0.752 -> 0.740 ms)
            if constexpr (NZ > 0) {
                if (!CONS || N == 0 || full_row) static_for<QH>([&](auto sa) {
                    constexpr int a = decltype(sa)::value;
                    double B[NV];
                    if constexpr (CONS) S::ncp_cons(eos, Vv[a], gx[a], gy[a], B);
                    else {
                        IeeeDiv dv;   // the branch-free divisions measured slower here (2048^2 +0.6 %: registers)
                        S::ncp(eos, dv, Vv[a], gx[a], gy[a], B);
                    }
#pragma unroll
                    for (int c = 0; c < NV; ++c) tq[a][c] = -QD::wv(0) * B[c];
                });
            }
        };
        // CONS (rhs_function.c:380-420): a refused cell keeps its mean alone, so what refuses it cheaply
        // is looked at before its pass: the node values of a variable that can do so by itself (for
        // Kapila nearly every time), and for N = 1 the whole check (a half's two of the four nodes
        // are two terms each).  The other cells are checked on the pass's values, and refused ones
        // take a second pass.  1024^2 right-hand sides, all cells checked after -> this way (and the
        // volume products of own rows only): Kapila N = 1 0.515 -> 0.456 ms, N = 2 0.850 -> 0.738, N = 3
        // 1.224 -> 1.082, BN N = 1 0.800 -> 0.715; checked before for every N: BN N = 2 1.195 -> 1.218,
        // N = 3 1.279 -> 1.401, Euler N = 2 0.267 -> 0.287
        bool whole = true;
        if constexpr (CONS && HAS_PAD && (N == 1 || S::CONS_SCREEN >= 0)) {
            constexpr int NODES = NFGP > 1 ? 4 : 2;   // of this half: the four faces at q = h, or two of the four faces
            auto node = [&](auto ff, int c) {
                constexpr int f = decltype(ff)::value;
                double cf[NDOF];
                cf[0] = w_0[c * BW + ccm];
#pragma unroll
                for (int k = 1; k < NDOF; ++k) cf[k] = coef_s[cidx(k - 1, c, m)];
                if constexpr (NFGP > 1) return face_pt<N, f, FAST>(cf, mask0);
                double v = cf[0];
                static_for<NDOF - 1>([&](auto kk) {
                    constexpr int k = decltype(kk)::value + 1;
                    v = v + cf[k] * (h ? FacePt<N, 2 + f % 2, k>::p0() : FacePt<N, f % 2, k>::p0());
                });
                return v;
            };
            if constexpr (S::CONS_SCREEN >= 0)
                static_for<NODES>([&](auto ff) { whole = whole && S::cons_screen(node(ff, S::CONS_SCREEN)); });
            if constexpr (N == 1)
                static_for<NODES>([&](auto ff) {
                    if (!whole || !active) return;
                    double V[NV];
#pragma unroll
                    for (int c = 0; c < NV; ++c) V[c] = node(ff, c);
                    whole = S::pad_cons(eos, V);
                });
            // every lane takes part in the shuffle (no short-circuit around it)
            const int pair = __shfl_xor_sync(FULL, (int)whole, 1);
            whole = whole && pair;
        }
        points([&](int c, double *cf) {
#pragma unroll
            for (int k = 1; k < NDOF; ++k) cf[k] = whole ? coef_s[cidx(k - 1, c, m)] : 0.0;
            __syncwarp();   // both halves have the variable's coefficients: its face values may replace them
        });
        if constexpr (HAS_PAD && !(CONS && N == 1)) {
            // admissibility at the nodes (rhs_function_prim.c:382-404): the four faces' values at
            // this half's Gauss point
            if (active && whole && (CONS || !ok)) {
                ok = true;
#pragma unroll 1
                for (int f = 0; f < 4 && ok; ++f) {
                    double V[NV];
#pragma unroll
                    for (int c = 0; c < NV; ++c) V[c] = f == 0 ? VR[c] : f < 3 ? coef_s[cidx(2 * q + f - 1, c, m)] : yt_up[c * CELLS];
                    if constexpr (SYS == SYS_KAPILA && !CONS && !FAST) {   // whole regions of a liquid under tension come here
                        CrDiv dv;
                        ok = S::pad_dv(eos, dv, V);
                        if (!eos.cr || dv.special()) ok = S::pad(eos, V);
                    } else {
                        ok = CONS ? S::pad_cons(eos, V) : S::pad(eos, V);
                    }
                }
            }
            // every lane takes part in the shuffle (no short-circuit around it)
            const int ok_pair = __shfl_xor_sync(FULL, (int)ok, 1);
            if (active && whole && !(ok && ok_pair)) {
                // the fallback's coefficients: [w, minmod_x, minmod_y, 0 ...] (rhs_function_prim.c:407-421);
                // conservative path: the mean alone (rhs_function.c:410-420)
                points([&](int c, double *cf) {
#pragma unroll
                    for (int k = 1; k < NDOF; ++k) cf[k] = 0.0;
                    if constexpr (!CONS && N >= 2) {
                        const double *a0 = w_0 + c * BW + ccm;
                        cf[1] = minmod(a0[1] - cf[0], cf[0] - a0[-1]);
                        cf[2] = minmod(w_p1[c * BW + ccm] - cf[0], cf[0] - w_m1[c * BW + ccm]);
                    }
                });
            }
        }
        __syncwarp();

        // ---------------- C. volume non-conservative term: the pair's sum
        double vol[(NV + 1) / 2] = {};   // of components 2 j + h; kept once row r-1 has read its own
        if constexpr (NZ > 0) {
            // rhs = 0.0; rhs += -w_q B_q for q = 0..NVGP-1; the pair holds q = 2h, 2h+1
            static_for<(NV + 1) / 2>([&](auto jj) {
                constexpr int j = decltype(jj)::value, z0 = K::nz(2 * j), z1 = 2 * j + 1 < NV ? K::nz(2 * j + 1) : -1;
                if constexpr (z0 >= 0 || z1 >= 0) {
                    double acc = 0.0;
                    if constexpr (NVGP > 1) {
                        double parts[NVGP];
#pragma unroll
                        for (int a = 0; a < QH; ++a) {
                            const double mine = own(jj, tq[a]), got = __shfl_xor_sync(FULL, other(jj, tq[a]), 1);
                            parts[a] = h ? got : mine;
                            parts[QH + a] = h ? mine : got;
                        }
#pragma unroll
                        for (int a = 0; a < NVGP; ++a) acc += parts[a];
                    } else {
                        acc = 0.0 + own(jj, tq[0]);
                    }
                    vol[j] = acc;
                }
            });
        }

        // ---------------- D. y-face below (r, i): Gauss point q = h ----------------
        {
            const bool doit = owned && in_rows;
            double Fq[NV], Dq[NV], Vq[NV];
            if (doit) {
                double VL[NV];
#pragma unroll
                for (int c = 0; c < NV; ++c) VL[c] = yt_lo[c * CELLS];
                const double s = riemann_gp<S, 1, CONS, !FAST>(eos, VL, VR, Fq, Dq, bad);
                smax_loc = fmax(smax_loc, s);
#pragma unroll
                for (int c = 0; c < NV; ++c) { Fq[c] = QD::wf(0) * Fq[c]; Dq[c] = QD::wf(0) * Dq[c]; }
                if constexpr (VISC) {
                    double gL[NV][2], gR[NV][2];
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        const int c = G0 + g;
                        double uc[NDOF];
                        load_uc(c, m, uc);
                        gR[c][0] = r1_h * face_grad<N, 2, 0>(uc, q);
                        gR[c][1] = r1_h * face_grad<N, 2, 1>(uc, q);
                        gL[c][0] = ygt_s[((q * NG + g) * 2 + 0) * CELLS + m];
                        gL[c][1] = ygt_s[((q * NG + g) * 2 + 1) * CELLS + m];
                    }
                    double FvL[NV], FvR[NV];
                    double svl, svr;
                    if constexpr (CONS) {
                        svl = S::template visc_cons<1>(VL, gL, p.mu1, p.mu2, FvL);
                        svr = S::template visc_cons<1>(VR, gR, p.mu1, p.mu2, FvR);
                    } else {
                        svl = S::template visc_prim<1>(VL, gL, p.mu1, p.mu2, FvL);
                        svr = S::template visc_prim<1>(VR, gR, p.mu1, p.mu2, FvR);
                    }
                    smaxv_loc = fmax(smaxv_loc, (svl < svr) ? svr : svl);
#pragma unroll
                    for (int c = 0; c < NV; ++c) Vq[c] = QD::wf(0) * (0.5 * (FvR[c] + FvL[c]));
                }
                if (bad && bad_cell == 0xffffffffu) bad_cell = (unsigned)(r * p.nx + i);
            } else {
#pragma unroll
                for (int c = 0; c < NV; ++c) { Fq[c] = 0.0; Dq[c] = 0.0; Vq[c] = 0.0; }
            }
            static_for<(NV + 1) / 2>([&](auto jj) {
                constexpr int j = decltype(jj)::value, z0 = K::nz(2 * j), z1 = 2 * j + 1 < NV ? K::nz(2 * j + 1) : -1;
                const double Gc = face_sum(jj, Fq, Vq);
                double Ec = 0.0;
                if constexpr (z0 >= 0 || z1 >= 0) Ec = fluct_sum(jj, Dq);
                if (!doit || (2 * j + 1 >= NV && h)) return;   // odd NV: the last variable is half 0's alone
                const int c = 2 * j + h;
                const int z = h ? z1 : z0;
                if (r > y0) {
                    // row r-1: rhs = ncp + ((-1/h) X - (1/h) Y)  (rhs_function_prim.c:589-602), then the RK combination
                    const int jo = r - 1;
                    const size_t gidx = (size_t)jo * p.pitch + i;
                    double Y = Gc - g_s(c);
                    double ncp = 0.0;
                    if constexpr (z0 >= 0 || z1 >= 0) {   // a component without a product adds 0.5 (0 + 0)
                        if (z >= 0) {
                            Y = Y + 0.5 * (Ec + e_s(z));
                            ncp = ncp_s(z);
                        }
                    }
                    const double ty = r1_h * Y;
                    const double rhs = ncp + (t1_s(c) - ty);
                    if (p.mode == OUT_RHS) {
                        if (p.out_aos) p.out[((size_t)jo * p.nx + i) * NV + c] = rhs;
                        else p.out[(size_t)c * p.plane + gidx] = rhs;
                    } else {
                        const double Sv = orow_s[c * BW + ccm];   // = p.in[c * plane + gidx], staged by TMA
                        const double bF = b * rhs;
                        double o;
                        if (p.mode == OUT_AXPY) {
                            o = Sv + bF;
                        } else if (p.mode == OUT_ZXS) {
                            const double Xv = p.xn[(size_t)c * p.plane + gidx];
                            const double s0 = p.ka * Xv + bF;
                            o = s0 + p.kc * Sv;
                        } else if (p.mode == OUT_ZSX) {
                            const double Xv = p.xn[(size_t)c * p.plane + gidx];
                            const double s0 = p.ka * Sv + bF;
                            o = s0 + p.kc * Xv;
                        } else {   // OUT_RK104_5
                            const double Xv = p.xn[(size_t)c * p.plane + gidx];
                            const double w = Sv + bF;
                            const double w1 = (1. / 25) * Xv + (9. / 25) * w;
                            p.out2[(size_t)c * p.plane + gidx] = w1;
                            o = 15.0 * w1 + (-5.0) * w;
                        }
                        p.out[(size_t)c * p.plane + gidx] = o;
                        // a y-slab's edge rows are the neighbours' halo rows: store them there too
                        if (p.push_lo && jo < 3)
                            p.push_lo[(long long)c * p.push_plane_lo + (long long)(jo + p.push_shift_lo) * p.pitch + i] = o;
                        if (p.push_hi && jo >= p.ny - 3)
                            p.push_hi[(long long)c * p.push_plane_hi + (long long)(jo + p.push_shift_hi) * p.pitch + i] = o;
                    }
                }
                g_s(c) = Gc;
                if constexpr (z0 >= 0 || z1 >= 0) {
                    if (z >= 0) {
                        e_s(z) = Ec;
                        ncp_s(z) = vol[j];
                    }
                }
            });
            if constexpr (VISC) {   // the top face's gradients for the row above
                if (owned && r < y0 + H && (NFGP > 1 || h == 0)) {
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        double uc[NDOF];
                        load_uc(G0 + g, m, uc);
                        ygt_s[((q * NG + g) * 2 + 0) * CELLS + m] = r1_h * face_grad<N, 3, 0>(uc, q);
                        ygt_s[((q * NG + g) * 2 + 1) * CELLS + m] = r1_h * face_grad<N, 3, 1>(uc, q);
                    }
                }
            }
        }
        }   // warp_active

        const bool conv = r + 3 <= row_hi;   // row r+3 is converted in this iteration
        const int cc = 1 + t;
        const bool conv_me = conv && cc <= owc + 6;
        [[maybe_unused]] double Qn[NV];   // AOS: held across S1, after which the row changes its layout in place
        if (conv_me) {
            here = wait_row(r + 3) && here;
            if constexpr (AOS) {
                if (here) conserved(r + 3, row_ptr(r + 3), cc, Qn);
            } else {
                const int g = xs + cc;
                if (here && (g < 0 || g >= p.nx)) {   // ghost columns before their sources are converted
                    double Q[NV], *rp = row_ptr(r + 3);
                    conserved(r + 3, rp, cc, Q);
#pragma unroll
                    for (int c = 0; c < NV; ++c) rp[c * BW + cc] = Q[c];
                }
            }
        }
        // the loads of the next iteration: row r's input, and row r+4 into the slot of row r-2
        const bool load_orow = full_row && p.mode != OUT_RHS && (!p.skip_loads || r < p.skip_loads_from);
        auto issue_next = [&] {
            if (t != 0) return;
            fence_proxy_async();   // the block's accesses to the slots precede the TMA writes
            issue_rows(r + 4);
            if (load_orow) {
                mbar_expect_tx(&bars[SLOTS], K::ROW_BYTES);
                tma_load_3d(orow_s, tmap, xs + p.col_off, r + p.row_off, 0, &bars[SLOTS]);
            }
        };
        // S1: every column's face values of row r visible, row r+3's ghost columns fetched
        if (__syncthreads_or(!here)) {
            give_up(finish_row && (!p.skip_loads || r - 1 < p.skip_loads_from), (unsigned)((r - y0 - 1) & 1));
            return;   // block-uniform exit
        }
        if constexpr (!VISC) issue_next();
        if (AOS && conv_me) put_primitive(r + 3, cc, Qn);
        if (conv) ++next_conv;

        // ---------------- E. x-face at the left of column i: Gauss point q ----------
        double Fown[(NV + 1) / 2], Down[(NV + 1) / 2];   // components 2 j + h
        if (warp_active && full_row) {
            double Fq[NV], Dq[NV], Vq[NV];
            if (xface) {
                double VL[NV], VR[NV];
#pragma unroll
                for (int c = 0; c < NV; ++c) {
                    VL[c] = coef_s[cidx(2 * q + 1, c, m - 1)];
                    VR[c] = coef_s[cidx(2 * q, c, m)];
                }
                const double s = riemann_gp<S, 0, CONS, !FAST>(eos, VL, VR, Fq, Dq, bad);
                smax_loc = fmax(smax_loc, s);
#pragma unroll
                for (int c = 0; c < NV; ++c) { Fq[c] = QD::wf(0) * Fq[c]; Dq[c] = QD::wf(0) * Dq[c]; }
                if constexpr (VISC) {
                    double gL[NV][2], gR[NV][2];
#pragma unroll
                    for (int g = 0; g < NG; ++g) {
                        const int c = G0 + g;
                        double ul[NDOF], ur[NDOF];
                        load_uc(c, m - 1, ul);
                        load_uc(c, m, ur);
                        gL[c][0] = r1_h * face_grad<N, 1, 0>(ul, q);
                        gL[c][1] = r1_h * face_grad<N, 1, 1>(ul, q);
                        gR[c][0] = r1_h * face_grad<N, 0, 0>(ur, q);
                        gR[c][1] = r1_h * face_grad<N, 0, 1>(ur, q);
                    }
                    double FvL[NV], FvR[NV];
                    double svl, svr;
                    if constexpr (CONS) {
                        svl = S::template visc_cons<0>(VL, gL, p.mu1, p.mu2, FvL);
                        svr = S::template visc_cons<0>(VR, gR, p.mu1, p.mu2, FvR);
                    } else {
                        svl = S::template visc_prim<0>(VL, gL, p.mu1, p.mu2, FvL);
                        svr = S::template visc_prim<0>(VR, gR, p.mu1, p.mu2, FvR);
                    }
                    smaxv_loc = fmax(smaxv_loc, (svl < svr) ? svr : svl);
#pragma unroll
                    for (int c = 0; c < NV; ++c) Vq[c] = QD::wf(0) * (0.5 * (FvR[c] + FvL[c]));
                }
                if (bad && bad_cell == 0xffffffffu) bad_cell = (unsigned)(r * p.nx + i);
            } else {
#pragma unroll
                for (int c = 0; c < NV; ++c) { Fq[c] = 0.0; Dq[c] = 0.0; Vq[c] = 0.0; }
            }
            if constexpr (!K::FX_OWN) __syncwarp();   // both halves have their left values: the fluxes may replace them
            static_for<(NV + 1) / 2>([&](auto jj) {
                constexpr int j = decltype(jj)::value, z0 = K::nz(2 * j), z1 = 2 * j + 1 < NV ? K::nz(2 * j + 1) : -1;
                Fown[j] = face_sum(jj, Fq, Vq);
                Down[j] = 0.0;
                if constexpr (z0 >= 0 || z1 >= 0) Down[j] = fluct_sum(jj, Dq);
                if (!xface || (2 * j + 1 >= NV && h)) return;
                flux_s(2 * j + h, m) = Fown[j];
                if constexpr (z0 >= 0 || z1 >= 0) {
                    if ((h ? z1 : z0) >= 0) fluct_s(2 * j + h, h ? z1 : z0, m) = Down[j];
                }
            });
        }
        if (!AOS && conv_me) {   // beside the x-face problems: 2 % of a 256^2 step against right after S1
            double Q[NV];
            const double *rp = row_ptr(r + 3);
#pragma unroll
            for (int c = 0; c < NV; ++c) Q[c] = rp[c * BW + cc];
            put_primitive(r + 3, cc, Q);
        }
        __syncthreads();   // S2: the x-face fluxes and prim rows r-1 .. r+3 ready
        if constexpr (VISC) issue_next();
        if (owned && full_row) {
            static_for<(NV + 1) / 2>([&](auto jj) {
                constexpr int j = decltype(jj)::value, z0 = K::nz(2 * j), z1 = 2 * j + 1 < NV ? K::nz(2 * j + 1) : -1;
                if (2 * j + 1 >= NV && h) return;
                const int c = 2 * j + h;
                double X = flux_s(c, m + 1) - Fown[j];
                if constexpr (z0 >= 0 || z1 >= 0) {
                    if ((h ? z1 : z0) >= 0) X = X + 0.5 * (fluct_s(c, h ? z1 : z0, m + 1) + Down[j]);
                }
                t1_s(c) = -r1_h * X;
            });
        }
        if constexpr (!K::FX_OWN) {
            __syncwarp();
            if ((t & 31) == 0) mbar_arrive(fluxes_read);
        }
    }

    // ---------------- CFL maximum: warp shuffle, block, one atomic ------------
    if (bad) raise_error(p.sc, ERR_INADMISSIBLE_FACE, bad_cell);
    __syncthreads();   // the carries are done with: red_s takes their place
    if (p.reduce_smax) {
        double mx = smax_loc;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
        if ((t & 31) == 0) red_s[t >> 5] = mx;
        __syncthreads();
        if (t == 0) {
            double b = red_s[0];
#pragma unroll
            for (int w = 1; w < K::NT / 32; ++w) b = fmax(b, red_s[w]);
            if (b > 0.0) atomicMax(&p.sc->smax, (unsigned long long)__double_as_longlong(b));
        }
        if constexpr (VISC) {   // the same for the viscous eigenvalue
            __syncthreads();
            double mv = smaxv_loc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mv = fmax(mv, __shfl_xor_sync(FULL, mv, o));
            if ((t & 31) == 0) red_s[t >> 5] = mv;
            __syncthreads();
            if (t == 0) {
                double b = red_s[0];
#pragma unroll
                for (int w = 1; w < K::NT / 32; ++w) b = fmax(b, red_s[w]);
                if (b > 0.0) atomicMax(&p.sc->smax_v, (unsigned long long)__double_as_longlong(b));
            }
        }
    }
    for (int k = t; k <= SLOTS + 1; k += K::NT) mbar_inval(&bars[k]);
}

}  // namespace hype
