// Fused per-direction line sweep of the zone_FD right-hand side.
//
// Replaces SpDistributor::rhsSolve (zone_FD/src/src/sp_distributor.cpp:3-79)
// for one direction together with Equation::consToPrim (equation.cpp:8-93)
// and OneDBnd::update (oneDBnd.cpp:31-114) for the lines it touches, and
// optionally the RK3 stage combination of BlockSolver::RK3_SSP
// (blockSolver.cpp:58-86) plus the reductions for the log value and the next
// CFL step.
//
// Work decomposition. A CTA owns W neighbouring lines along the sweep axis AX
// and one segment [s_begin, s_end) of them. It marches through the segment in
// chunks of S cells. Per chunk it
//   1. loads the S new cells (cons -> prim on the fly, ghost cells from the
//      line's boundary wiring) into a shared-memory ring of S+8 positions
//      (S+10 with the TRAD6 difference),
//   2. computes the S new face fluxes (one face per thread) into a ring of
//      S+3 faces (S+5); the faces shared with the previous chunk are reused,
//   3. applies the MND6 difference (node fluxes recomputed from the prim ring)
//      or the TRAD6 one, and the epilogue for S cells.
// Face values and face fluxes never leave shared memory, and every cell is
// read from HBM once per sweep plus 8 (10) halo cells per line segment.
//
// Thread layout: along x (AX = 0) consecutive threads take consecutive cells
// of a line; along y/z consecutive threads take neighbouring lines (adjacent
// x), so every global access is coalesced along x in all three sweeps.
#pragma once
#include <cuda_pipeline.h>

#include "euler_math.cuh"
#include "mixed.cuh"
#include "sweep_params.h"

namespace cfd {
namespace CFD_NS {

template <int NV, class O>
__device__ __forceinline__ void load_cons_prim(const double *__restrict__ u, long long ncell, long long cell,
                                               double *pr, O &o)
{
    double c[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) c[v] = __ldg(u + v * ncell + cell);
    cons_to_prim<NV>(c, pr, o);
}

// Ghost cell k (0 = nearest the boundary) of a line end, as OneDBnd::update
// leaves it after Bnds::update (oneDBnd.cpp:31-114).
template <int NV, int NG, class O>
__device__ __forceinline__ void ghost_prim(const SweepParams &p, const BcLine &bl, int k, double tstage, double *pr,
                                           O &o)
{
    switch (bl.type) {
    case BND_PERIODIC1D:
        load_cons_prim<NV>(p.u, p.ncell, bl.i0 + (long long)k * bl.offset, pr, o);
        return;
    case BND_SUPERSONICOUTLET:
        load_cons_prim<NV>(p.u, p.ncell, bl.i0, pr, o);
        return;
    case BND_SYMMETRYX:
    case BND_SYMMETRYY:
    case BND_SYMMETRYZ:
    case BND_SYMMETRY1D: {
        load_cons_prim<NV>(p.u, p.ncell, bl.i0 + (long long)k * bl.offset, pr, o);
        int neg = (bl.type == BND_SYMMETRYY) ? 2 : (bl.type == BND_SYMMETRYZ) ? 3 : 1;
        if (neg < NV - 1) pr[neg] = -pr[neg];
        if (bl.type == BND_SYMMETRY1D) {
            // SYMMETRY1D writes only the first three values of each ghost cell.
            for (int v = 3; v < NV; v++) pr[v] = (bl.slot >= 0) ? p.bc_vals[((long long)bl.slot * NG + k) * NV + v] : 0.0;
        }
        return;
    }
    case BND_DOUBLEMACHUP: {
        // oneDBnd.cpp:87-108: exact post- or pre-shock state at the stage time.
        // As in the reference, ghost k is placed at y = -dh/2 + k*dh (measured
        // from 0, not from the line end) and x is the edge cell's centre.
        double x = bl.coor_x;
        double y = -bl.dh_y / 2 + k * bl.dh_y;
        double gt = 1.0 / 6.0 + sqrt(3.0) / 3.0 * (1.0 + 20 * tstage);
        if (y > sqrt(3.0) * (x - gt)) {
            pr[0] = 8.0; pr[1] = p.dm_u; pr[2] = p.dm_v; pr[NV - 1] = 116.5;
        } else {
            pr[0] = 1.4; pr[1] = 0; pr[2] = 0; pr[NV - 1] = 1.0;
        }
        if (NV == 5) pr[3] = 0.0;
        return;
    }
    case BND_HALO: {
        // rows of the neighbouring slab, ascending: the low side's nearest
        // ghost is the neighbour's last row, the high side's its first
        const int kk = k > 3 ? 3 : k;  // four halo rows (MND6 only)
        const int r = (bl.offset == 0) ? 3 - kk : kk;
        const double *hb = (bl.offset == 0) ? p.halo_lo : p.halo_hi;
        double c[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) c[v] = hb[((long long)v * 4 + r) * p.halo_nl + bl.i0];
        cons_to_prim<NV>(c, pr, o);
        return;
    }
    default:
        // DIRICLET and every type whose update() is a no-op keep their static data.
        for (int v = 0; v < NV; v++) pr[v] = (bl.slot >= 0) ? p.bc_vals[((long long)bl.slot * NG + k) * NV + v] : 0.0;
        return;
    }
}

template <int NV>
struct PrimVals {
    double v[NV];
};

// The same out of line, returned by value: boundary ghosts are a few cells
// per line end, and one copy of this code instead of one per cell-loader call
// site keeps the sweep's instruction footprint small.
template <int NV, int NG>
__device__ __noinline__ PrimVals<NV> ghost_prim_ool(const SweepParams &p, const BcLine &bl, int k, double tstage)
{
    PrimVals<NV> r;
    OpsIeee o;
    ghost_prim<NV, NG>(p, bl, k, tstage, r.v, o);
    return r;
}

// What the FP64 sweeps keep of a cell: prim, the cons the reference re-derives
// from it (primToChar's prologue) and its Roe weights.
template <int NV>
struct CellVals {
    double pr[NV], cs[NV], kw[NV];
};

template <int NV, int AX, bool RW, class O>
__device__ __forceinline__ void cell_from_cons(const double *u, CellVals<NV> &c, O &o)
{
    const double ir = cons_to_prim<NV>(u, c.pr, o);
    prim_to_cons<NV>(c.pr, c.cs, o);
    if constexpr (RW && NV >= 4) EigenBase<NV, AX>::roe_weights(c.pr, c.kw, ir, o);
}

// Out of line with IEEE operations: operands outside OpsSpec's range.
template <int NV, int AX, bool RW>
__device__ __noinline__ CellVals<NV> cell_ieee(PrimVals<NV> u)
{
    CellVals<NV> c;
    OpsIeee o;
    cell_from_cons<NV, AX, RW>(u.v, c, o);
    return c;
}

// A boundary ghost, out of line (a few cells per line end). On a small grid the
// CTAs at the line ends are the ones the sweep waits for: without the IEEE
// operations' branches 24 strict steps of 64^2 took 1.19 instead of 1.22 ms, 3
// of 128^3 8.06 instead of 8.19 ms.
template <int NV, int AX, int NG, bool RW>
__device__ __noinline__ CellVals<NV> ghost_cell(const SweepParams &p, bool low, int lid, long long base, int k,
                                                double tstage)
{
    BcLine bl;
    if (p.bc_lo) {
        bl = low ? p.bc_lo[lid] : p.bc_hi[lid];
    } else {
        // a whole side of one type, wired by the rules of the tables: the low
        // end reads from the first cell on, the high end from the last cell
        // back, a true wrap from the far end
        const long long last = base + (long long)(p.n[AX] - 1) * p.stride[AX];
        const int type = p.bc_type[low ? 0 : 1];
        const bool wrap = type == BND_PERIODIC_WRAP;
        bl.type = wrap ? BND_PERIODIC1D : type;
        bl.i0 = low != wrap ? base : last;
        bl.offset = low != wrap ? (int)p.stride[AX] : -(int)p.stride[AX];
        bl.slot = -1;
        bl.coor_x = bl.dh_y = 0.0;
    }
    CellVals<NV> c;
    auto fill = [&](auto &o) {
        ghost_prim<NV, NG>(p, bl, k, tstage, c.pr, o);
        prim_to_cons<NV>(c.pr, c.cs, o);
        if constexpr (RW && NV >= 4) EigenBase<NV, AX>::roe_weights(c.pr, c.kw, o.rcp(c.pr[0]), o);
    };
    OpsSpec s;
    fill(s);
    if (!s.ok) {
        OpsIeee o;
        fill(o);
    }
    return c;
}

// max wave speed terms of a new state, out of line (IEEE operations): u_d + c
// over h_d and the two values of the sign test
template <int NV>
__device__ __noinline__ PrimVals<5> wave_terms_ieee(PrimVals<NV> u, double h0, double h1, double h2)
{
    PrimVals<5> r;
    double pr[NV];
    const double hd[3] = {h0, h1, h2};
    cons_to_prim<NV>(u.v, pr);
    const double cs = sqrt(kGamma * pr[NV - 1] / pr[0]);
    for (int d = 0; d < 3; d++) r.v[d] = (d < NV - 2) ? (cs + fabs(pr[1 + d])) / hd[d] : 0.0;
    r.v[3] = pr[0];
    r.v[4] = pr[NV - 1];
    return r;
}

// The flux of one FP64 face from its stencil in shared memory (sp, sc, kw:
// the line's prim, cons and Roe weights, PITCH doubles per variable, cell m of
// the stencil at ring position (s0 + m) & MASK).
template <int NV, int AX, int FAM, int FLUX, int PITCH, int MASK, bool RW, class O>
__device__ __forceinline__ void face_flux(const double *sp, const double *sc, const double *kw, int s0, double icst,
                                          double kap, int posl, double *fx, O &o)
{
    int slot[6];
#pragma unroll
    for (int m = 0; m < 6; m++) slot[m] = (s0 + m) & MASK;
    double fl[NV], fr[NV], ir[2] = {0.0, 0.0};
    if constexpr (NV == 3) {
        double pr6[6][NV], cs6[6][NV];
#pragma unroll
        for (int m = 0; m < 6; m++) {
#pragma unroll
            for (int v = 0; v < NV; v++) {
                pr6[m][v] = sp[v * PITCH + slot[m]];
                cs6[m][v] = sc[v * PITCH + slot[m]];
            }
        }
        reconstruct_face<NV, AX, FAM>(pr6, cs6, icst, kap, fl, fr, o, ir);
    } else {
        auto csacc = [&](int m, int v) { return sc[v * PITCH + slot[m]]; };
        auto pracc = [&](int m, int v) { return sp[v * PITCH + slot[m]]; };
        double kl[NV], kr[NV];
        if constexpr (RW) {
#pragma unroll
            for (int v = 0; v < NV; v++) {
                kl[v] = kw[v * PITCH + slot[2]];
                kr[v] = kw[v * PITCH + slot[3]];
            }
        } else {
            double pl[NV], pr[NV];
#pragma unroll
            for (int v = 0; v < NV; v++) {
                pl[v] = pracc(2, v);
                pr[v] = pracc(3, v);
            }
            EigenBase<NV, AX>::roe_weights(pl, kl, o.rcp(pl[0]), o);
            EigenBase<NV, AX>::roe_weights(pr, kr, o.rcp(pr[0]), o);
        }
        const EigenBase<NV, AX> eb(kl, kr, o);
        reconstruct_face_stream<NV, AX, FAM>(eb, csacc, pracc, icst, kap, fl, fr, posl, o, ir);
    }
    riemann<NV, AX, FLUX>(fl, fr, fx, o, ir);
}

// The same out of line with IEEE operations, the positivity fallback and
// limiters: faces whose operands or states OpsSpec's version does not cover.
template <int NV, int AX, int FAM, int FLUX, int PITCH, int MASK, bool RW>
__device__ __noinline__ PrimVals<NV> face_flux_ieee(const double *sp, const double *sc, const double *kw, int s0,
                                                    double icst, double kap, int posl)
{
    PrimVals<NV> r;
    OpsIeee o;
    face_flux<NV, AX, FAM, FLUX, PITCH, MASK, RW>(sp, sc, kw, s0, icst, kap, posl, r.v, o);
    return r;
}

#ifndef CFD_SWEEP_MINB
#define CFD_SWEEP_MINB 2
#endif
#ifndef CFD_SWEEP_MINB128
#define CFD_SWEEP_MINB128 4  // resident 128-thread CTAs per SM (2D/3D)
#endif

#if defined(CFD_FAST)
constexpr bool kStrictFlavour = false;
#else
constexpr bool kStrictFlavour = true;
#endif

constexpr int pow2_ceil(int x)
{
    int r = 1;
    while (r < x) r <<= 1;
    return r;
}

template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC = 0, int DIFF = 0>
struct SweepShape {
    static constexpr int NT = S * W;
    // Halo cells per side: MND6 differences faces x_{i-3/2}..x_{i+3/2} (cells
    // i-4..i+4), TRAD6 faces x_{i-5/2}..x_{i+5/2} (cells i-5..i+5). A chunk
    // shares FC = 2 HG - 5 faces with the previous one.
    static constexpr int HG = DIFF ? 5 : 4;
    static constexpr int FC = 2 * HG - 5;
    // ring sizes are powers of two so that ring positions are bit masks
    static constexpr int R = pow2_ceil(S + 2 * HG);  // prim ring positions (S + 2 HG used)
    static constexpr int RF = pow2_ceil(S + FC);     // face ring positions (S + FC used)
    static constexpr int LSP = R | 1;         // odd line strides avoid bank conflicts
    static constexpr int LSF = RF | 1;
    // The 3D mixed y/z sweeps keep no FP64 cons ring: they read the cons as
    // hi + lo from the FP32 split (within 2^-48 of the cons), which leaves room
    // for the cp.async staging below (the x sweep stages less and has room).
    static constexpr bool HL_CS = (PREC == 1 && NV == 5 && AX != 0 && FAM != FAM_RESEARCH);
    static constexpr int SMEM_DOUBLES0 = (HL_CS ? 1 : 2) * NV * W * LSP + NV * W * LSF;
    // mixed form: FP32 hi/lo split of the cons ring (exact FP32 increments)
    static constexpr int SMEM_FLOATS = PREC ? 2 * NV * W * LSP : 0;
    // Resident CTAs per SM the launch bounds ask for: 512 threads per SM in
    // 2D/3D (two CTAs of 256 threads or four of 128), 128 registers a thread;
    // or three 128-thread CTAs (168 registers, fewer spills). Timed again on
    // the branch-free arithmetic, four against three: 2D WCNS5 x 256 against
    // 261 us fast and 379 against 400 strict, y 334 against 287 fast; 2D TENO
    // strict x 356 against 346, y 468 against 378 (2048^2); 3D WCNS5 fast x 166
    // against 173, y 176 against 171, z 210 against 197 (128^3), strict x 260
    // against 266, y 275 against 276, z 303 against 308 at two (255
    // registers). So four for WCNS5 along x and for the strict 3D WCNS5
    // sweeps, and three, as before, for 2D y, 3D and the FP64 TENO-Z x sweep,
    // and the 3D mixed TENO-Z sweeps; two for the other families' strict z.
    static constexpr bool FOUR = PREC == 0 && NV == 5 && FAM == FAM_WCNS5 && (AX == 0 || kStrictFlavour);
    static constexpr bool THREE = !FOUR && (((FAM == FAM_TENOZ) && (PREC == 0 ? AX == 0 : NV == 5)) ||
                                            (PREC == 0 && NV == 5) || (PREC == 0 && NV == 4 && AX == 1));
    static constexpr bool TWO = !FOUR && kStrictFlavour && PREC == 0 && NV == 5 && AX == 2;
    static constexpr int MINB128 = TWO ? 2 : THREE ? 3 : CFD_SWEEP_MINB128;
    static constexpr int MINB = (NT <= 256) ? (NV >= 4 ? (NT == 128 ? MINB128 : CFD_SWEEP_MINB * (256 / NT))
                                                       : CFD_SWEEP_MINB)
                                            : 1;
    // Asynchronous staging (cp.async) of each thread's global operands: the next
    // chunk's cell and the epilogue's rhs / U^0 / U^k, so that their latency
    // hides behind the face phase. Only where MINB CTAs per SM still fit in the
    // 228 KB of an SM (1 KB of it reserved per CTA).
    // The x sweep of a 2D/3D step is always the first direction (no epilogue
    // operands to stage), so it stages only the next chunk's cells.
    static constexpr int NSTG = (AX == 0 && NV >= 4) ? 1 : 4;
    static constexpr size_t SMEM_STAGE = sizeof(double) * NSTG * NV * NT;
    static constexpr size_t SMEM_LIMIT = (size_t)(MINB > 2 ? 224 / MINB : 112) * 1024;
    // FP64 multi-dimensional sweeps keep each cell's Roe weights (sqrt(rho),
    // sqrt(rho) v, sqrt(rho) H) beside its prim: formed once per cell instead
    // of once for each of the cell's two faces; where the ring fits beside the
    // staging buffers
    static constexpr bool RW = (PREC == 0 && NV >= 4) &&
                               sizeof(double) * (SMEM_DOUBLES0 + NV * W * LSP) + SMEM_STAGE <= SMEM_LIMIT;
    static constexpr int SMEM_DOUBLES = SMEM_DOUBLES0 + (RW ? NV * W * LSP : 0);
    static constexpr size_t SMEM_RINGS = sizeof(double) * SMEM_DOUBLES + sizeof(float) * SMEM_FLOATS;
    static constexpr bool PF = SMEM_RINGS + SMEM_STAGE <= SMEM_LIMIT;
    static constexpr bool PF_EPI = PF && NSTG == 4;
    static constexpr size_t SMEM_BYTES = SMEM_RINGS + (PF ? SMEM_STAGE : 0);
};

// ONE: every segment has at most S - FC cells. Its faces are one pass of the
// threads: the prologue loads HG + 2 - FO cells and the chunk S, and the cells
// are finished by the threads from FC on. Otherwise a segment's first chunk
// takes the FC faces ahead of it in a second pass, nearly another face's
// latency, which long segments spread over their chunks. (One kernel for both
// lengths cost the long ones 5 to 14%: the offsets became variables.)
template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC, int DIFF, bool ONE = false>
__device__ __forceinline__ void sweep_tile(const SweepParams &p, int block_id)
{
    using SH = SweepShape<NV, AX, FAM, FLUX, S, W, PREC, DIFF>;
    constexpr int NT = SH::NT, R = SH::R, RF = SH::RF, LSP = SH::LSP, LSF = SH::LSF;
    constexpr int HG = SH::HG, FC = SH::FC, FO = HG - 3;  // face j sits at face-ring position j - s_begin + FO
    // device-resident loop: the whole launch is a no-op once the loop is done
    if (p.ctl && p.ctl->done) return;
    const double tstage = p.ctl ? p.ctl->tst[p.rk_stage] : p.t;
    const double inv_h = 1.0 / p.h;
    // RN(1/h_d) for the correctly rounded wave-speed quotients of the epilogue
    double inv_hdir[3] = {0.0, 0.0, 0.0};
    if (p.mode == MODE_RK && p.want_reduce)
        for (int d = 0; d < NV - 2; d++) inv_hdir[d] = 1.0 / p.hdir[d];
    // ring positions (R and RF are powers of two; arguments are never negative)
    auto ring = [](int x) { return (int)((unsigned)x & (unsigned)(R - 1)); };
    auto fring = [](int x) { return (int)((unsigned)x & (unsigned)(RF - 1)); };
    const double rkBdt = p.ctl ? p.ctl->bdt[p.rk_stage] : p.rkBdt;
    extern __shared__ double smem[];
    double *sp = smem;                   // [NV][W][LSP] prim
    double *sc = sp + NV * W * LSP;      // [NV][W][LSP] cons re-derived from prim (primToChar prologue); absent with HL_CS
    double *sf = SH::HL_CS ? sc : sc + NV * W * LSP;  // [NV][W][LSF] face flux
    // mixed form: [NV][W][LSP] (hi, lo) = ((float)cons, (float)(cons - hi))
    float2 *shl = reinterpret_cast<float2 *>(sf + NV * W * LSF);
    // FP64 form: [NV][W][LSP] Roe weights of each cell (in place of the mixed form's split)
    double *skw = sf + NV * W * LSF;
    // staging: [0] next chunk's cons, [1] rhs, [2] U^0, [3] U^k; [NV][NT] each
    double *stg = reinterpret_cast<double *>(reinterpret_cast<char *>(smem) + SH::SMEM_RINGS);
    constexpr bool PF = SH::PF, PF_EPI = SH::PF_EPI;

    constexpr int T0 = (AX == 0) ? 1 : 0;  // transverse axis with neighbouring lines in a CTA
    constexpr int T1 = (AX == 2) ? 1 : 2;
    const int nd = p.n[AX];
    const int nt0 = p.n[T0];
    const int nseg = (nd + p.seg_len - 1) / p.seg_len;
    const int nblk0 = (nt0 + W - 1) / W;
    int bid = block_id;
    int seg;
    if (p.seg_outer) {  // segments outermost (partial sweeps along the last dimension)
        const int per = nblk0 * p.n[T1];
        seg = bid / per;
        bid -= seg * per;
    } else {
        seg = bid % nseg;
        bid /= nseg;
    }
    const int a0 = (bid % nblk0) * W;
    const int bb = bid / nblk0;
    const int s_begin = seg * p.seg_len;
    const int s_end = min(s_begin + p.seg_len, nd);

    const int tid = threadIdx.x;
    const int tl = (AX == 0) ? tid / S : tid % W;   // line within the CTA
    const int tp = (AX == 0) ? tid % S : tid / W;   // position within the chunk
    const long long sAX = p.stride[AX];

    auto line_of = [&](int l, bool &ok, long long &base, int &lid) {
        int a = a0 + l;
        ok = a < nt0;
        base = (long long)a * p.stride[T0] + (long long)bb * p.stride[T1];
        lid = a + nt0 * bb;
    };
    // the thread's own line, fixed for the whole tile: held in registers by
    // the mixed form, recomputed where needed by the FP64 form (whose kernels
    // have no registers to spare)
    bool my_ok = false; long long my_base = 0; int my_lid = 0;
    if constexpr (PREC == 1) line_of(tl, my_ok, my_base, my_lid);
    auto own_line = [&](bool &ok, long long &base, int &lid) {
        if constexpr (PREC == 1) {
            ok = my_ok; base = my_base; lid = my_lid;
        } else {
            line_of(tl, ok, base, lid);
        }
    };

    // Stage cell P (global index along AX, may be a ghost) of line l; staged:
    // its cons already sit in stg[0] (interior cells of the thread's own line).
    auto load_pos = [&](int l, int P, bool staged = false) {
        bool ok; long long base; int lid;
        if (PREC == 1 && l == tl) own_line(ok, base, lid);
        else line_of(l, ok, base, lid);
        int slot = ring(P - s_begin + HG);
        if constexpr (PREC == 0) {
            CellVals<NV> c;
            if (!ok) {  // past the last line: any admissible state, never read back
#pragma unroll
                for (int v = 0; v < NV; v++) c.pr[v] = c.cs[v] = c.kw[v] = (v == 0 || v == NV - 1) ? 1.0 : 0.0;
                c.cs[NV - 1] = 2.5;
                c.kw[NV - 1] = 3.5;
            } else if (P >= 0 && P < nd) {
                PrimVals<NV> u;
#pragma unroll
                for (int v = 0; v < NV; v++)
                    u.v[v] = staged ? stg[v * NT + threadIdx.x] : __ldg(p.u + v * p.ncell + base + (long long)P * sAX);
                OpsSpec o;
                cell_from_cons<NV, AX, SH::RW>(u.v, c, o);
                if (!o.ok) c = cell_ieee<NV, AX, SH::RW>(u);
            } else {
                const bool lo = P < 0;
                const int k = lo ? -P - 1 : P - nd;
                c = ghost_cell<NV, AX, HG, SH::RW>(p, lo, lid, base, k > HG - 1 ? HG - 1 : k, tstage);
            }
#pragma unroll
            for (int v = 0; v < NV; v++) {
                sp[(v * W + l) * LSP + slot] = c.pr[v];
                sc[(v * W + l) * LSP + slot] = c.cs[v];
                if constexpr (SH::RW) skw[(v * W + l) * LSP + slot] = c.kw[v];
            }
            return;
        }
        double pr[NV];
        double cs[NV];
        bool have_cs = false;  // the mixed form takes interior cells' cons as loaded
        if (!ok) {
            pr[0] = 1.0;
            for (int v = 1; v < NV - 1; v++) pr[v] = 0.0;
            pr[NV - 1] = 1.0;
        } else if (P >= 0 && P < nd) {
            if (staged) {
#pragma unroll
                for (int v = 0; v < NV; v++) cs[v] = stg[v * NT + threadIdx.x];
            } else {
#pragma unroll
                for (int v = 0; v < NV; v++) cs[v] = __ldg(p.u + v * p.ncell + base + (long long)P * sAX);
            }
            cons_to_prim<NV>(cs, pr);
            have_cs = (PREC == 1);
        } else if (P < 0) {
            int k = -P - 1;
            const PrimVals<NV> g = ghost_prim_ool<NV, HG>(p, p.bc_lo[lid], k > HG - 1 ? HG - 1 : k, tstage);
#pragma unroll
            for (int v = 0; v < NV; v++) pr[v] = g.v[v];
        } else {
            int k = P - nd;
            const PrimVals<NV> g = ghost_prim_ool<NV, HG>(p, p.bc_hi[lid], k > HG - 1 ? HG - 1 : k, tstage);
#pragma unroll
            for (int v = 0; v < NV; v++) pr[v] = g.v[v];
        }
        if (!have_cs) prim_to_cons<NV>(pr, cs);  // as the reference's primToChar re-derives them
#pragma unroll
        for (int v = 0; v < NV; v++) {
            sp[(v * W + l) * LSP + slot] = pr[v];
            if constexpr (!SH::HL_CS) sc[(v * W + l) * LSP + slot] = cs[v];
            if constexpr (PREC == 1) {
                const float hi = (float)cs[v];
                shl[(v * W + l) * LSP + slot] = make_float2(hi, (float)(cs[v] - (double)hi));
            }
        }
    };

    // Face j lies between cells j-1 and j (x_{j-1/2}); stencil cells j-3..j+2.
    auto face = [&](int l, int j) {
        double fx[NV];
        const double *spl = sp + l * LSP, *scl = sc + l * LSP;
        if constexpr (PREC == 0) {
            const int s0 = j - 3 - s_begin + HG;
            OpsSpec o;
            face_flux<NV, AX, FAM, FLUX, W * LSP, R - 1, SH::RW>(spl, scl, skw + l * LSP, s0, p.icst, p.icst_k, p.posl, fx,
                                                                 o);
            if (!o.ok) {
                const PrimVals<NV> r = face_flux_ieee<NV, AX, FAM, FLUX, W * LSP, R - 1, SH::RW>(
                    spl, scl, skw + l * LSP, s0, p.icst, p.icst_k, p.posl);
#pragma unroll
                for (int v = 0; v < NV; v++) fx[v] = r.v[v];
            }
        } else {
            int slot[6];
#pragma unroll
            for (int m = 0; m < 6; m++) slot[m] = ring(j - 3 + m - s_begin + HG);
            double fl[NV], fr[NV];
            auto csacc = [&](int m, int v) { return scl[v * W * LSP + slot[m]]; };
            auto pracc = [&](int m, int v) { return spl[v * W * LSP + slot[m]]; };
            const float2 *hll = shl + l * LSP;
            // the FP32 hi/lo split of each stencil cell's cons
            auto hlacc = [&](int m, int v) {
                return hll[v * W * LSP + slot[m]];
            };
            if constexpr (SH::HL_CS) {
                auto hlcs = [&](int m, int v) {
                    const float2 t = hlacc(m, v);
                    return (double)t.x + (double)t.y;
                };
                reconstruct_face_mixed<NV, AX, FAM>(hlcs, pracc, hlacc, p.icst, p.icst_k, fl, fr);
            } else {
                reconstruct_face_mixed<NV, AX, FAM>(csacc, pracc, hlacc, p.icst, p.icst_k, fl, fr);
            }
            if constexpr (FLUX == FLUX_ROE) roe_md_mixed<NV, AX>(fl, fr, fx);
            else hllc_md_mixed<NV, AX>(fl, fr, fx);
        }
        int fslot = fring(j - s_begin + FO);
#pragma unroll
        for (int v = 0; v < NV; v++) sf[(v * W + l) * LSF + fslot] = fx[v];
    };

    // prologue: cells s_begin-HG .. s_begin+HC-1, HC of the chunks' offset
    constexpr int HC = ONE ? 2 - FO : HG;
    for (int idx = tid; idx < (HG + HC) * W; idx += NT) {
        int l = (AX == 0) ? idx / (HG + HC) : idx % W;
        int q = (AX == 0) ? idx % (HG + HC) : idx / W;
        load_pos(l, s_begin - HG + q);
    }

    double red_rho = 0.0, red_lam[3] = {0.0, 0.0, 0.0};
    unsigned err = 0;

    // cp.async of this thread's interior cell at position P into stg[0]
    auto prefetch_cell = [&](int P) {
        bool ok; long long base; int lid;
        own_line(ok, base, lid);
        if (ok && P >= 0 && P < nd) {
            const long long cell = base + (long long)P * sAX;
#pragma unroll
            for (int v = 0; v < NV; v++) __pipeline_memcpy_async(stg + v * NT + tid, p.u + v * p.ncell + cell, 8);
        }
        __pipeline_commit();
    };
    // cp.async of the epilogue operands of this thread's cell i
    const bool need_rhs = PF_EPI && !p.first, need_u0 = PF_EPI && p.mode == MODE_RK,
               need_u = PF_EPI && p.mode == MODE_RK && p.rk_stage != 1;
    auto prefetch_epilogue = [&](int i) {
        bool ok; long long base; int lid;
        own_line(ok, base, lid);
        if (ok && i < s_end && (!ONE || i >= s_begin)) {
            const long long cell = base + (long long)i * sAX;
#pragma unroll
            for (int v = 0; v < NV; v++) {
                const long long gi = v * p.ncell + cell;
                if (need_rhs) __pipeline_memcpy_async(stg + (1 * NV + v) * NT + tid, p.rhs + gi, 8);
                if (need_u0) __pipeline_memcpy_async(stg + (2 * NV + v) * NT + tid, p.u0 + gi, 8);
                if (need_u) __pipeline_memcpy_async(stg + (3 * NV + v) * NT + tid, p.u + gi, 8);
            }
        }
        __pipeline_commit();
    };
    if constexpr (ONE) {
        // the epilogue's operands fly while the faces are computed
        if constexpr (PF) prefetch_epilogue(s_begin - FC + tp);
    } else if constexpr (PF) {
        prefetch_cell(s_begin + HG + tp);
    }

    for (int c0 = s_begin; ONE ? c0 == s_begin : c0 < s_end; c0 += S) {
        if constexpr (ONE) {
            if (tp < s_end - s_begin + FC) load_pos(tl, c0 + HC + tp);
        } else if constexpr (PF) {
            __pipeline_wait_prior(0);
            load_pos(tl, c0 + HG + tp, true);
            prefetch_epilogue(c0 + tp);
            prefetch_cell(c0 + S + HG + tp);  // an empty group past the segment
        } else {
            load_pos(tl, c0 + HG + tp);
        }
        __syncthreads();
        {
            // the chunk's S new faces per line, and before the segment's first
            // chunk also the FC faces ahead of them, from one call site (the
            // face code is emitted once)
            const int nface = (c0 == s_begin && !ONE) ? NT + FC * W : NT;
            for (int idx = (ONE && tp >= s_end - s_begin + FC) ? NT : tid; idx < nface; idx += NT) {
                int l, j;
                if (ONE || idx < NT) {
                    l = tl;
                    j = c0 + tp + (ONE ? -FO : HG - 2);
                } else {
                    const int e = idx - NT;
                    l = (AX == 0) ? e / FC : e % W;
                    j = s_begin - FO + ((AX == 0) ? e % FC : e / W);
                }
                face(l, j);
            }
        }
        __syncthreads();

        const int i = c0 + tp - (ONE ? FC : 0);
        bool ok; long long base; int lid;
        own_line(ok, base, lid);
        if constexpr (PF) __pipeline_wait_prior(ONE ? 0 : 1);  // the epilogue operands; the next cell may still fly
        if (ok && i < s_end && (!ONE || i >= s_begin)) {
            double fnm[NV], fnp[NV];
            if constexpr (DIFF == 0) {  // node fluxes of cells i-1 and i+1 (SolvePointSolver, nl = nr = 1)
                double pm[NV], pp[NV];
                int sm = ring(i - 1 - s_begin + HG), spp = ring(i + 1 - s_begin + HG);
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    pm[v] = sp[(v * W + tl) * LSP + sm];
                    pp[v] = sp[(v * W + tl) * LSP + spp];
                }
                node_flux<NV, AX>(pm, fnm);
                node_flux<NV, AX>(pp, fnp);
            }
            // faces j = i-(FC-1)/2 .. i+(FC+1)/2, face j being x_{j-1/2}
            int fs[FC + 1];
#pragma unroll
            for (int m = 0; m <= FC; m++) fs[m] = fring(i - (FC - 1) / 2 + m - s_begin + FO);
            const long long cell = base + (long long)i * sAX;
            // MND6 differences of the NV variables (strict: the NV quotients by
            // h formed together, one branch for the group)
            double dd[NV];
            if constexpr (DIFF == 0) {
#if defined(CFD_FAST)
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const double *fv = sf + (v * W + tl) * LSF;
                    dd[v] = mnd6(fnm[v], fnp[v], fv[fs[0]], fv[fs[1]], fv[fs[2]], fv[fs[3]], p.h, inv_h);
                }
#else
                DivN<NV> num;
                OpsSpec o;
                o.need(OpsSpec::in_range(p.h));
#pragma unroll
                for (int v = 0; v < NV; v++) {
                    const double *fv = sf + (v * W + tl) * LSF;
                    num.v[v] = mnd6_num(fnm[v], fnp[v], fv[fs[0]], fv[fs[1]], fv[fs[2]], fv[fs[3]]);
                    dd[v] = o.div_y(num.v[v], p.h, inv_h);
                }
                if (!o.ok) {
                    DivN<NV> hh;
#pragma unroll
                    for (int v = 0; v < NV; v++) hh.v[v] = p.h;
                    const DivN<NV> q = divs_ieee<NV>(num, hh);
#pragma unroll
                    for (int v = 0; v < NV; v++) dd[v] = q.v[v];
                }
#endif
            }
            double uo[NV];
#pragma unroll
            for (int v = 0; v < NV; v++) {
                const double *fv = sf + (v * W + tl) * LSF;
                double d;
                if constexpr (DIFF == 0) d = dd[v];
                else d = trad6(fv[fs[0]], fv[fs[1]], fv[fs[2]], fv[fs[3]], fv[fs[4]], fv[fs[5]], p.h, inv_h);
                const long long gi = v * p.ncell + cell;
                const double *sv = stg + v * NT + tid;
                double r = p.first ? (0.0 + d) : ((PF_EPI ? sv[1 * NV * NT] : p.rhs[gi]) + d);
                if constexpr (NV == 4) {
                    // SourceTerm::calGravitySource (sourceTerm.cpp:3-20) on the
                    // stage's prim: rhs(rho v) -= rho, rhs(rho E) -= rho v
                    if (p.gravity) {
                        const int sc0 = ring(i - s_begin + HG);
                        const double rho = sp[(0 * W + tl) * LSP + sc0];
                        if (v == 2) r -= rho;
                        if (v == 3) r -= rho * sp[(2 * W + tl) * LSP + sc0];
                    }
                }
                if (p.mode != MODE_RK) {
                    p.rhs[gi] = r;
                } else {
                    if (v == 0 && p.want_reduce) red_rho = fmax(red_rho, fabs(r));
                    double o;
                    const double u0v = PF_EPI ? sv[2 * NV * NT] : p.u0[gi];
                    if (p.rk_stage == 1) {
                        o = u0v - rkBdt * r;
                    } else {
                        o = p.rkA * u0v - rkBdt * r + p.rkC * (PF_EPI ? sv[3 * NV * NT] : p.u[gi]);
                    }
                    uo[v] = o;
                    p.u_out[gi] = o;
                }
            }
            if (p.mode == MODE_RK) {
                bool fin = true;
#pragma unroll
                for (int v = 0; v < NV; v++) fin = fin && isfinite(uo[v]);
                if (!fin) err |= ERR_NONFINITE;
                if constexpr (PREC == 0) {
                    if (p.want_reduce) {
                        double pr[NV], lam[3] = {0.0, 0.0, 0.0};
                        OpsSpec o;
                        const double ir = cons_to_prim<NV>(uo, pr, o);
                        (void)ir;
#if defined(CFD_FAST)
                        const double cs = o.sqrt(o.div(kGamma * pr[NV - 1], pr[0]));
#else
                        const double cs = o.sqrt(o.div_y(kGamma * pr[NV - 1], pr[0], ir));
#endif
#pragma unroll
                        for (int d = 0; d < NV - 2; d++) {
                            const double a = cs + fabs(pr[1 + d]);
                            o.need(OpsSpec::in_range(a) & OpsSpec::in_range(p.hdir[d]));
                            lam[d] = OpsSpec::quot(a, p.hdir[d], inv_hdir[d]);
                        }
                        if (!o.ok) {
                            PrimVals<NV> u;
#pragma unroll
                            for (int v = 0; v < NV; v++) u.v[v] = uo[v];
                            const PrimVals<5> w = wave_terms_ieee<NV>(u, p.hdir[0], p.hdir[1], p.hdir[2]);
#pragma unroll
                            for (int d = 0; d < NV - 2; d++) lam[d] = w.v[d];
                            pr[0] = w.v[3];
                            pr[NV - 1] = w.v[4];
                        }
                        if (!(pr[0] > 0.0) || !(pr[NV - 1] > 0.0)) err |= ERR_NEGATIVE;
#pragma unroll
                        for (int d = 0; d < NV - 2; d++) red_lam[d] = fmax(red_lam[d], lam[d]);
                    }
                } else if (p.want_reduce) {
                    double pr[NV];
                    cons_to_prim<NV>(uo, pr);
                    if (!(pr[0] > 0.0) || !(pr[NV - 1] > 0.0)) err |= ERR_NEGATIVE;
                    double cs = sqrt(kGamma * pr[NV - 1] / pr[0]);
#pragma unroll
                    for (int d = 0; d < NV - 2; d++)
                        red_lam[d] = fmax(red_lam[d], div_rn(cs + fabs(pr[1 + d]), p.hdir[d], inv_hdir[d]));
                }
            }
        }
        if constexpr (!ONE) __syncthreads();
    }

    if (p.mode == MODE_RK) {
        if (err) atomicOr(p.err, err);
        if (p.want_reduce) block_max_reduce<NT, 4>(red_rho, red_lam, p.red);
    }
}

template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC, int DIFF, bool ONE>
__global__ void __launch_bounds__(S *W, (SweepShape<NV, AX, FAM, FLUX, S, W, PREC, DIFF>::MINB))
    sweep_kernel(const __grid_constant__ SweepParams p)
{
    sweep_tile<NV, AX, FAM, FLUX, S, W, PREC, DIFF, ONE>(p, (int)(p.tile0 + blockIdx.x));
    if constexpr (AX == NV - 3) {
        if (p.ctl_step) {
            __threadfence();  // this CTA's maxima before its ticket
            __syncthreads();
            if (threadIdx.x == 0 && atomicAdd(p.ticket, 1u) == gridDim.x - 1) {
                __threadfence();
                *p.ticket = 0u;
                step_end(p.ctl_step, p.red, p.linf);
                step_begin(p.ctl_step, p.red, NV - 2, p.dts);
            }
        }
    }
}

// Number of CTA tiles one case's sweep along AX needs.
template <int AX, int W>
__host__ __device__ inline long long sweep_tiles(const SweepParams &p)
{
    constexpr int T0 = (AX == 0) ? 1 : 0;
    constexpr int T1 = (AX == 2) ? 1 : 2;
    long long nseg = (p.n[AX] + p.seg_len - 1) / p.seg_len;
    return (long long)((p.n[T0] + W - 1) / W) * p.n[T1] * nseg;
}

// Persistent sweep over many independent cases: the tiles of all cases form
// one work list (tile_start[c] = first tile of case c, prefix sums); each CTA
// walks the list with a grid stride, copies its case's parameter block to
// shared memory and runs the same tile code as sweep_kernel. Cases whose
// device loop is done are skipped tile by tile.
template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC>
__global__ void __launch_bounds__(S *W, (SweepShape<NV, AX, FAM, FLUX, S, W, PREC>::MINB))
    sweep_batched_kernel(const SweepParams *__restrict__ cases, const long long *__restrict__ tile_start, int ncases)
{
    __shared__ SweepParams sp;
    __shared__ int s_case;
    const long long total = tile_start[ncases];
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        __syncthreads();  // the previous tile is done with sp
        if (threadIdx.x == 0) {
            int lo = 0, hi = ncases - 1;  // last case with tile_start <= item
            while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (tile_start[mid] <= item) lo = mid; else hi = mid - 1;
            }
            s_case = lo;
        }
        __syncthreads();
        const int c = s_case;
        {
            const int words = (int)(sizeof(SweepParams) / sizeof(int));
            const int *src = reinterpret_cast<const int *>(cases + c);
            int *dst = reinterpret_cast<int *>(&sp);
            for (int k = threadIdx.x; k < words; k += blockDim.x) dst[k] = src[k];
        }
        __syncthreads();
        sweep_tile<NV, AX, FAM, FLUX, S, W, PREC, 0>(sp, (int)(item - tile_start[c]));
    }
}

template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC, int DIFF, bool ONE>
static cudaError_t launch_sweep_kernel(const SweepParams &p, cudaStream_t st)
{
    using SH = SweepShape<NV, AX, FAM, FLUX, S, W, PREC, DIFF>;
    auto kern = sweep_kernel<NV, AX, FAM, FLUX, S, W, PREC, DIFF, ONE>;
    // the dynamic shared-memory opt-in is per device
    static bool attr_set[64] = {};
    int dev = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 != cudaSuccess) return e0;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        attr_set[dev] = true;
    }
    constexpr int T0 = (AX == 0) ? 1 : 0;
    constexpr int T1 = (AX == 2) ? 1 : 2;
    long long nseg = (p.n[AX] + p.seg_len - 1) / p.seg_len;
    const long long nblk0 = (p.n[T0] + W - 1) / W;
    long long nblk = nblk0 * p.n[T1] * nseg;
    if (nblk > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    SweepParams q = p;
    q.tile0 = 0;
    if (p.part_lo < p.part_hi) {
        // the tiles covering [part_lo, part_hi) of the last dimension L
        const int L = (p.n[2] > 1) ? 2 : 1;
        if (AX == L) {  // whole segments, segments outermost
            if (!p.seg_outer) return cudaErrorInvalidValue;
            const long long s0 = p.part_lo / p.seg_len, s1 = (p.part_hi + p.seg_len - 1) / p.seg_len;
            q.tile0 = s0 * nblk0 * p.n[T1];
            nblk = (s1 - s0) * nblk0 * p.n[T1];
        } else if (T0 == L) {  // lines of L in blocks of W (2D)
            if (p.part_lo % W) return cudaErrorInvalidValue;
            const long long b0 = p.part_lo / W, b1 = (p.part_hi + W - 1) / W;
            q.tile0 = b0 * nseg;
            nblk = (b1 - b0) * nseg;
        } else {  // planes of L (3D)
            q.tile0 = (long long)p.part_lo * nblk0 * nseg;
            nblk = (long long)(p.part_hi - p.part_lo) * nblk0 * nseg;
        }
    } else if (p.seg_outer) {
        return cudaErrorInvalidValue;
    }
    if (nblk <= 0) return cudaSuccess;
    kern<<<(unsigned)nblk, SH::NT, SH::SMEM_BYTES, st>>>(q);
    return cudaGetLastError();
}

template <int NV, int AX, int FAM, int S, int W, int PREC, int DIFF>
static cudaError_t launch_sweep_shape(int flux, const SweepParams &p, cudaStream_t st)
{
    // The strict flavour only: there both kernels round alike, while contraction
    // may differ between two kernels of the fast flavour, whose results must not
    // depend on how lines are cut.
    if constexpr (DIFF == 0 && kStrictFlavour) {
        if (p.seg_len <= S - SweepShape<NV, AX, FAM, FLUX_ROE, S, W, PREC, DIFF>::FC)
            return flux == FLUX_HLLC ? launch_sweep_kernel<NV, AX, FAM, FLUX_HLLC, S, W, PREC, DIFF, true>(p, st)
                                     : launch_sweep_kernel<NV, AX, FAM, FLUX_ROE, S, W, PREC, DIFF, true>(p, st);
    }
    return flux == FLUX_HLLC ? launch_sweep_kernel<NV, AX, FAM, FLUX_HLLC, S, W, PREC, DIFF, false>(p, st)
                             : launch_sweep_kernel<NV, AX, FAM, FLUX_ROE, S, W, PREC, DIFF, false>(p, st);
}

template <int NV, int AX, int FAM, int FLUX, int S, int W, int PREC>
static cudaError_t launch_batched_shape_p(const BatchSweep &b, cudaStream_t st)
{
    using SH = SweepShape<NV, AX, FAM, FLUX, S, W, PREC>;
    auto kern = sweep_batched_kernel<NV, AX, FAM, FLUX, S, W, PREC>;
    static bool attr_set[64] = {};
    static int blocks_per_sm[64] = {};
    int dev = 0;
    cudaError_t e0 = cudaGetDevice(&dev);
    if (e0 != cudaSuccess) return e0;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm[dev], kern, SH::NT, SH::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        if (blocks_per_sm[dev] < 1) blocks_per_sm[dev] = 1;
        attr_set[dev] = true;
    }
    long long grid = (long long)b.num_sms * (b.one_cta ? 1 : blocks_per_sm[dev]);
    if (b.total_tiles < grid) grid = b.total_tiles;
    if (grid <= 0) return cudaSuccess;
    sweep_batched_kernel<NV, AX, FAM, FLUX, S, W, PREC>
        <<<(unsigned)grid, SH::NT, SH::SMEM_BYTES, st>>>(b.cases, b.tile_start, b.ncases);
    return cudaGetLastError();
}

// Tile shapes (sweep_params.h): kXSn x kXWn along x in 3D and for 2D FP64,
// kXS x kXW along x for the 2D mixed form; kYSm x kYWm along y and z;
// kXS x kXW and kYS x kYW for the TRAD6 difference (FP64 only); k1S x k1W in
// 1D. The mixed form exists in the fast flavour of the multi-dimensional
// kernels.
template <int NV, int AX, int FAM>
static cudaError_t launch_sweep_ax(int flux, const SweepParams &p, cudaStream_t st)
{
    if (p.diff == DIFF_TRAD6) {
        if (p.prec != 0) return cudaErrorInvalidValue;
        if constexpr (NV == 3) return launch_sweep_shape<NV, AX, FAM, k1S, k1W, 0, 1>(flux, p, st);
        else if constexpr (AX == 0) return launch_sweep_shape<NV, AX, FAM, kXS, kXW, 0, 1>(flux, p, st);
        else return launch_sweep_shape<NV, AX, FAM, kYS, kYW, 0, 1>(flux, p, st);
    }
    if (p.prec != 0) {
#if defined(CFD_FAST)
        if constexpr (NV >= 4 && FAM != FAM_RESEARCH) {
            if constexpr (AX == 0 && NV == 4) return launch_sweep_shape<NV, AX, FAM, kXS, kXW, 1, 0>(flux, p, st);
            else if constexpr (AX == 0) return launch_sweep_shape<NV, AX, FAM, kXSn, kXWn, 1, 0>(flux, p, st);
            else return launch_sweep_shape<NV, AX, FAM, kYSm, kYWm, 1, 0>(flux, p, st);
        }
#endif
        return cudaErrorInvalidValue;
    }
    if constexpr (NV == 3) return launch_sweep_shape<NV, AX, FAM, k1S, k1W, 0, 0>(flux, p, st);
    else if constexpr (AX == 0) return launch_sweep_shape<NV, AX, FAM, kXSn, kXWn, 0, 0>(flux, p, st);
    else return launch_sweep_shape<NV, AX, FAM, kYSm, kYWm, 0, 0>(flux, p, st);
}

template <int NV, int FAM>
cudaError_t launch_sweep(int ax, int flux, const SweepParams &p, cudaStream_t st)
{
    if (ax == 0) return launch_sweep_ax<NV, 0, FAM>(flux, p, st);
    if constexpr (NV >= 4) {
        if (ax == 1) return launch_sweep_ax<NV, 1, FAM>(flux, p, st);
    }
    if constexpr (NV == 5) {
        if (ax == 2) return launch_sweep_ax<NV, 2, FAM>(flux, p, st);
    }
    return cudaErrorInvalidValue;
}

// Persistent batched sweep (1D, 2D and 3D): the single-grid tile shapes, which
// 2D/3D FP64 has as b.shape = 1 beside the longer tiles of b.shape = 0.
template <int NV, int AX, int FAM, int S, int W, int PREC>
static cudaError_t launch_batched_flux(int flux, const BatchSweep &b, cudaStream_t st)
{
    return flux == FLUX_HLLC ? launch_batched_shape_p<NV, AX, FAM, FLUX_HLLC, S, W, PREC>(b, st)
                             : launch_batched_shape_p<NV, AX, FAM, FLUX_ROE, S, W, PREC>(b, st);
}

template <int NV, int AX, int FAM>
static cudaError_t launch_batched_ax(int flux, const BatchSweep &b, cudaStream_t st)
{
    if (b.prec == 1) {
#if defined(CFD_FAST)
        if constexpr (FAM != FAM_RESEARCH) {
            if (b.shape) return cudaErrorInvalidValue;
            if constexpr (AX == 0 && NV == 4) return launch_batched_flux<NV, AX, FAM, kXS, kXW, 1>(flux, b, st);
            else if constexpr (AX == 0) return launch_batched_flux<NV, AX, FAM, kXSn, kXWn, 1>(flux, b, st);
            else return launch_batched_flux<NV, AX, FAM, kYSm, kYWm, 1>(flux, b, st);
        }
#endif
        return cudaErrorInvalidValue;
    }
    if constexpr (AX == 0)
        return b.shape ? launch_batched_flux<NV, AX, FAM, kXSn, kXWn, 0>(flux, b, st)
                       : launch_batched_flux<NV, AX, FAM, kXS, kXW, 0>(flux, b, st);
    else
        return b.shape ? launch_batched_flux<NV, AX, FAM, kYSm, kYWm, 0>(flux, b, st)
                       : launch_batched_flux<NV, AX, FAM, kYS, kYW, 0>(flux, b, st);
}

template <int NV, int FAM>
cudaError_t launch_sweep_batched(int ax, int flux, const BatchSweep &b, cudaStream_t st)
{
    if constexpr (NV == 3) {
        if (ax != 0 || b.prec != 0) return cudaErrorInvalidValue;
        return launch_batched_flux<3, 0, FAM, k1S, k1W, 0>(flux, b, st);
    } else {
        if (ax == 0) return launch_batched_ax<NV, 0, FAM>(flux, b, st);
        if (ax == 1) return launch_batched_ax<NV, 1, FAM>(flux, b, st);
        if constexpr (NV == 5) {
            if (ax == 2) return launch_batched_ax<NV, 2, FAM>(flux, b, st);
        }
        return cudaErrorInvalidValue;
    }
}

} // namespace CFD_NS
} // namespace cfd

namespace cfd {
namespace CFD_NS {

// The RK stage combination of the last sweep's epilogue, applied by itself to
// a complete RHS in p.rhs (the last sweep having run with MODE_WRITE):
// U_out = (A U0 - Bdt R) + C U_k (stage 1: U0 - dt R) with the epilogue's
// non-finite check. Compiled in the flavour's own unit, so it rounds the
// expression as the fused epilogue does. No reductions: it serves stage 1.
template <int NV>
__global__ void __launch_bounds__(256) rk_combine_kernel(const __grid_constant__ SweepParams p)
{
    if (p.ctl && p.ctl->done) return;
    const double rkBdt = p.ctl ? p.ctl->bdt[p.rk_stage] : p.rkBdt;
    unsigned err = 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < p.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        bool fin = true;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const long long gi = v * p.ncell + c;
            const double r = p.rhs[gi];
            double o;
            if (p.rk_stage == 1) o = p.u0[gi] - rkBdt * r;
            else o = p.rkA * p.u0[gi] - rkBdt * r + p.rkC * p.u[gi];
            p.u_out[gi] = o;
            fin = fin && isfinite(o);
        }
        if (!fin) err |= ERR_NONFINITE;
    }
    if (err) atomicOr(p.err, err);
}

template <int NV>
cudaError_t launch_rk_combine(const SweepParams &p, cudaStream_t st)
{
    long long g = (p.ncell + 255) / 256;
    if (g > 148LL * 16) g = 148LL * 16;
    if (g < 1) g = 1;
    rk_combine_kernel<NV><<<(unsigned)g, 256, 0, st>>>(p);
    return cudaGetLastError();
}

} // namespace CFD_NS
} // namespace cfd
