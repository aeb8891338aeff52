// stage.cuh -- one fused stage of the MHD step on a Cartesian grid, plain FP64 or mixed precision:
// the kernels and their launchers, instantiated per form by stage_plain.cu, stage_mixed.cu and
// stage_delta.cu (separate files only so they compile in parallel).
//
// Replaces the reference's face kernel + cell kernel pair (CUF_MGD_grans_RK2 /
// CUF_MGD_cell_RK2, SET_Fortran_Cuda_MHD/cuf_solvers.cuf:243-440 and :561-794; Euler variants
// :62-241, :443-558), which exchange fluxes through a 9 x N_gran array in HBM, with a single
// kernel per stage:
//   * a CTA owns a 32 x TY column of cells and marches along z over lz planes;
//   * each plane (cells + 2-cell x/y halo) is read from the SoA conserved state once, turned into
//     primitives once (FP64 pressure recovery) and kept in a 4-plane shared-memory ring
//     (planes k-1 .. k+2), which is all the z-stencil of the minmod reconstruction needs;
//   * every face of the plane (x, y and the z face k-1/2) is computed once, by one thread, from
//     shared memory, and its flux is applied to both neighbouring cells; a warp owns a tile row, so
//     z and x fluxes stay in its registers and only y fluxes are exchanged (run_tile);
//   * the conservative update, p floor, source re-imposition and the dt candidate reduction
//     (warp shuffle -> one atomicMin per CTA) are fused; the last CTA rolls the lagged-dt clock.
//
// P = 0, plain form: everything in FP64; the ring holds the field as b = B / sqrt(4 pi), the units
//   the Riemann solver works in, and the primitives are recovered exactly as the oracle does
//   wherever the kinetic and magnetic energies exceed 64 p, within a few ulps elsewhere
//   (prim_from_cons_guarded).
// P = 1, mixed form: the ring holds FP32 primitives (recovered from the FP64 state in FP64),
//   reconstruction and the Riemann solver run in FP32, fluxes are stored in FP32; a face whose
//   selected FP32 state has rho <= 0 or p <= 0 (or a non-finite flux) is recomputed in FP64 from
//   the FP64 state; the flux divergence and the update are FP64, and the second Heun stage (or
//   the Euler step) is a compensated sum with the compensation kept in FP32; dt is reduced in
//   FP64.
// P = 2, delta form: FP64 ring and fluxes, the Riemann solver's small differences in FP32.
#pragma once
#include <atomic>
#include <cfloat>
#include <type_traits>
#include "riemann_f32x2.cuh"
#include "riemann_fp64.cuh"
#include "setb_internal.cuh"

namespace sb {
namespace {

// Storage and arithmetic types of the two forms: ring (primitives), flux buffer, Riemann math.
template <int P> struct Types {
    using Ring = double;
    using Flux = double;
    using Math = double;
};
template <> struct Types<2> {   // delta form: FP64 states and fluxes, FP32 inside the solver
    using Ring = double;
    using Flux = double;
    using Math = double;
};
template <> struct Types<1> {
    using Ring = float;
    using Flux = float;
    using Math = float;
};
constexpr int RING = 4;

// Column tile of each form (tile_shape): TX = 32 cells per tile row, one lane per column.  The
// 3 TY + 2 warp jobs of a plane's faces (see run_tile) take three rounds of the CTA's warps
// (32 x 7 cells: 23 jobs over 8 warps; 32 x 11: 35 jobs over 12 warps).  Threads 0..NC-1 own
// one cell each in the update.
template <int P, int SK> struct Tile {   // SK: the shape of tile_shape
    static constexpr int TX = kTileX, TY = tile_shape(P, SK).ty, NT = tile_shape(P, SK).threads;
    static constexpr int MINB = tile_shape(P, SK).ctas_per_sm;
    static constexpr int NC = TX * TY;
    static constexpr int HX = TX + 4, HY = TY + 4, PLANE = HX * HY;
    static constexpr int NYF = TX * (TY + 1);        // y faces
    using RG = typename Types<P>::Ring;
    using FT = typename Types<P>::Flux;
    // dynamic shared memory: alignment slack, staged box (FP64), primitive ring, and the exchanged y
    // and east x fluxes (two buffers each)
    static constexpr int kSmem = 128 + 8 * PLANE * (int)sizeof(double) + RING * 8 * PLANE * (int)sizeof(RG) +
                                 2 * 8 * (NYF + TY) * (int)sizeof(FT);
    static_assert(TX == 32, "one lane per tile column");
    static_assert(NT == 32 * (TY + 1), "one warp per tile row and one for the edges");
    static_assert(TY <= 32, "one lane per row for the east faces");
};

__device__ __forceinline__ int ring_slot(int k) { return (k + 4 * RING) & (RING - 1); }

// The inflow ghost state beyond x = hi as a primitive ring entry: stored B, or with SB the
// solver's b = B / sqrt(4 pi) (correctly rounded, as prim_from_cons<true, true> forms it).
template <bool SB>
__device__ __forceinline__ void inflow_prim(const GridGeom& g, double* q) {
#pragma unroll
    for (int v = 0; v < 8; v++) q[v] = (SB && v >= 5) ? div_rn(g.inflow[v], kSpi4, kInvSpi4) : g.inflow[v];
}

// FP64 primitive state of global cell (i,j,k) with the boundary rules: inflow beyond x = hi,
// zero-gradient (clamped index) elsewhere.  SB: the field as b (see prim_from_cons).
template <bool EXACT, bool SB = false>
__device__ __forceinline__ void fetch_prim64(const StageArgs& A, int i, int j, int k, double* q) {
    const GridGeom& g = A.g;
    if (i >= g.nx) {
        inflow_prim<SB>(g, q);
        return;
    }
    i = max(i, 0);
    j = min(max(j, 0), g.ny - 1);
    k = min(max(k, 0), g.nz - 1);
    const long long off = (long long)k * g.ps + (long long)j * g.px + i;
    double U[8];
#pragma unroll
    for (int v = 0; v < 8; v++) U[v] = __ldcg(A.Uin + v * g.vs + off);   // not by the read-only path: launch_chained
    if constexpr (EXACT) {
        prim_from_cons_guarded<SB>(U, q);
    } else {
        double ke, me;
        prim_from_cons<false, SB>(U, q, ke, me);
    }
}

// Loads cells n0, n0 + step, ... < n1 of the planes from kk on (with halo; cell n is cell n % PLANE of
// plane kk + n / PLANE) of the tile starting at (i0, j0) as primitives into their ring slots.
template <int P, int SK, typename RT>
__device__ __forceinline__ void load_planes(const StageArgs& A, RT* ring, int i0, int j0, int kk, int n1, int n0,
                                            int step) {
    constexpr int HX = Tile<P, SK>::HX, PLANE = Tile<P, SK>::PLANE;
#pragma unroll 2
    for (int n = n0; n < n1; n += step) {
        const int k = kk + n / PLANE, c = n % PLANE;
        const int cx = c % HX, cy = c / HX;
        RT* dst = ring + ring_slot(k) * 8 * PLANE;
        double q[8];
        fetch_prim64<P != 1, P == 0>(A, i0 - 2 + cx, j0 - 2 + cy, k, q);
#pragma unroll
        for (int v = 0; v < 8; v++) dst[v * PLANE + c] = (RT)q[v];
    }
}

// ---- plane copies by the tensor-memory accelerator
// One copy per plane: the (kTileX + 4) x (TY + 4) x 1 x 8 box of the state at (i0-2, j0-2, k, 0)
// lands in the staging buffer as [variable][y][x]; its completion is counted on an mbarrier.
// Coordinates outside the grid read zeros (the boundary rules are applied when the plane is
// converted); x = i0 - 2 is even, so the copy starts on a 16-byte boundary.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Non-blocking probe of phase `parity` of the barrier.
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Waits for phase `parity` of the barrier for at most `limit` SM cycles (0: kCopyWaitCycles,
// < 0: one non-blocking check); false when it gave up.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity, long long limit) {
    if (limit < 0) return mbar_test_wait(bar, parity);
    if (limit == 0) limit = kCopyWaitCycles;
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > limit) return false;
    return true;
}

// Issued by one thread: expects `bytes` on the barrier and starts the copy.  The caller has
// ordered earlier generic-proxy reads of `dst` before this (barrier + proxy fence).
__device__ __forceinline__ void tma_plane(void* dst, const CUtensorMap* tm, int x, int y, int z, unsigned bytes,
                                          unsigned long long* bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(tm), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_u32(bar))
        : "memory");
}

// A tensor map in global memory that the host wrote, possibly where an earlier map lay: the thread that
// issues the copies acquires it before its first use (the SM's descriptor cache may hold the earlier one).
__device__ __forceinline__ void acquire_tmap(const CUtensorMap* tm) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(tm) : "memory");
}

// Cells c0, c0 + step, ... < c1 of a primitive plane with the boundary rules from a staged box
// (conserved, [v][y][x] with row HX): inflow beyond x = hi, zero-gradient (clamped index, always
// inside the box) elsewhere.
template <int P, int SK, typename RT>
__device__ __forceinline__ void convert_plane(const StageArgs& A, const double* stg, RT* dst, int i0, int j0, int c0,
                                              int step, int c1) {
    constexpr int HX = Tile<P, SK>::HX, PLANE = Tile<P, SK>::PLANE;
    const GridGeom& g = A.g;
    for (int c = c0; c < c1; c += step) {
        const int cx = c % HX, cy = c / HX;
        const int i = i0 - 2 + cx, j = j0 - 2 + cy;
        double q[8];
        if (i >= g.nx) {
            inflow_prim<P == 0>(g, q);
        } else {
            const int sx = max(i, 0) - (i0 - 2), sy = min(max(j, 0), g.ny - 1) - (j0 - 2);
            const double* src = stg + sy * HX + sx;
            double U[8];
#pragma unroll
            for (int v = 0; v < 8; v++) U[v] = src[v * PLANE];
            if constexpr (P == 1) {
                double ke, me;
                prim_from_cons<false, false>(U, q, ke, me);
            } else {
                prim_from_cons_guarded<P == 0>(U, q);
            }
        }
#pragma unroll
        for (int v = 0; v < 8; v++) dst[v * PLANE + c] = (RT)q[v];
    }
}

// Face-frame order (normal, t1, t2) of the components of a face normal to axis AX: entry v of
// the face-frame state is natural component face_perm<AX>(v) of (rho, u, v, w, p, Bx, By, Bz).
template <int AX> __host__ __device__ constexpr int face_perm(int v) {
    return (v == 0 || v == 4) ? v
           : (v < 4 ? 0 : 4) + ((v & 3) == 1 ? 1 + AX : ((v & 3) == 2 ? (AX == 0 ? 2 : 1) : (AX == 2 ? 2 : 3)));
}

// face_perm<AX>(v) for an axis known only at run time (the rare FP64 recompute path).
__device__ __forceinline__ int face_perm_dyn(int axis, int v) {
    return axis == 0 ? face_perm<0>(v) : (axis == 1 ? face_perm<1>(v) : face_perm<2>(v));
}

// Face-frame states at a face normal to AX from its 4-cell stencil of ring cells (component planes
// PLANE apart).  B is first order, so only the inner pair carries it.
template <int AX, int PLANE, int P, int ORDER, typename RG, typename RT>
__device__ __forceinline__ void face_states(const RG* pLL, const RG* pL, const RG* pR, const RG* pRR, RT* q1, RT* q2) {
    RT qLL[8], qL[8], qR[8], qRR[8];
#pragma unroll
    for (int v = 0; v < 8; v++) {
        const int o = face_perm<AX>(v) * PLANE;
        qL[v] = (RT)pL[o];
        qR[v] = (RT)pR[o];
        qLL[v] = (ORDER == 2 && v < 5) ? (RT)pLL[o] : RT(0);
        qRR[v] = (ORDER == 2 && v < 5) ? (RT)pRR[o] : RT(0);
    }
    if constexpr (P == 1 && ORDER == 2) reconstruct_f32x2(qLL, qL, qR, qRR, q1, q2);
    else if constexpr (P == 0)
        reconstruct_fp64<ORDER>(qLL, qL, qR, qRR, q1, q2,
                                [&](int s, int v) { return (s ? pR : pL)[face_perm<AX>(v) * PLANE]; });
    else reconstruct<RT, ORDER>(qLL, qL, qR, qRR, q1, q2);
}

// What the out-of-line FP64 recompute of a face needs, passed by value: a reference or pointer to
// the kernel's arguments would make the compiler copy them to local memory and read every field
// from there on the hot path.
struct FetchArgs {
    const double* Uin;
    long long vs, ps, px;
    int nx, ny, nz, n_disc;
    double inflow[8];
};
struct FaceFlux {
    double F[8];   // natural component order
    double sl, sr;
    int fl;
};

__device__ __forceinline__ FetchArgs fetch_args(const StageArgs& A) {
    FetchArgs f;
    f.Uin = A.Uin;
    f.vs = A.g.vs;
    f.ps = A.g.ps;
    f.px = A.g.px;
    f.nx = A.g.nx;
    f.ny = A.g.ny;
    f.nz = A.g.nz;
    f.n_disc = A.n_disc;
#pragma unroll
    for (int v = 0; v < 8; v++) f.inflow[v] = A.g.inflow[v];
    return f;
}

// FP64 primitive state of global cell (i,j,k), boundary rules as fetch_prim64.
__device__ __forceinline__ void fetch_prim64_f(const FetchArgs& f, int i, int j, int k, double* q) {
    if (i >= f.nx) {
#pragma unroll
        for (int v = 0; v < 8; v++) q[v] = f.inflow[v];
        return;
    }
    i = max(i, 0);
    j = min(max(j, 0), f.ny - 1);
    k = min(max(k, 0), f.nz - 1);
    const long long off = (long long)k * f.ps + (long long)j * f.px + i;
    double U[8];
#pragma unroll
    for (int v = 0; v < 8; v++) U[v] = __ldcg(f.Uin + v * f.vs + off);
    double ke, me;
    prim_from_cons(U, q, ke, me);
}

// The FP64 recompute of one face of the mixed and delta forms from the FP64 state (rare path;
// kept out of line so the main path keeps its registers), with the library special functions.
// (i, j, k) is the cell on the high side of the face.
template <int NSTATE, int ORDER>
__device__ __noinline__ FaceFlux face_fp64(const FetchArgs fa, int axis, int i, int j, int k) {
    const int di = axis == 0, dj = axis == 1, dk = axis == 2;
    double c[4][8];
    fetch_prim64_f(fa, i - 2 * di, j - 2 * dj, k - 2 * dk, c[0]);
    fetch_prim64_f(fa, i - di, j - dj, k - dk, c[1]);
    fetch_prim64_f(fa, i, j, k, c[2]);
    fetch_prim64_f(fa, i + di, j + dj, k + dk, c[3]);
    const int pn = 1 + axis, pt1 = axis == 0 ? 2 : 1, pt2 = axis == 2 ? 2 : 3;
    const int perm[8] = {0, pn, pt1, pt2, 4, 4 + pn, 4 + pt1, 4 + pt2};
    double f[4][8];
    for (int s = 0; s < 4; s++)
        for (int v = 0; v < 8; v++) f[s][v] = c[s][perm[v]];
    double q1[8], q2[8], G[8], SM;
    reconstruct<double, ORDER>(f[0], f[1], f[2], f[3], q1, q2);
    FaceFlux r;
    r.fl = riemann<double, NSTATE, false, false, false, false, false>(q1, q2, 0.0, fa.n_disc, G, r.sl, r.sr, SM);
    for (int v = 0; v < 8; v++) r.F[perm[v]] = G[v];
    return r;
}

// What the update of a cell reads from HBM / L2: the stage input, Heun stage 2's base state and the
// mixed forms' compensation.
template <int P, int KIND> struct CellState {
    double u[8], base[KIND ? 8 : 1];
    float comp[P ? 8 : 1];
};
template <int P, int KIND>
__device__ __forceinline__ void load_cell(const StageArgs& A, long long off, CellState<P, KIND>& c) {
#pragma unroll
    for (int v = 0; v < 8; v++) {
        c.u[v] = A.Uin[v * A.g.vs + off];
        if (KIND) c.base[KIND * v] = A.Ubase[v * A.g.vs + off];
        if (P != 0) c.comp[P == 0 ? 0 : v] = A.comp ? A.comp[v * A.g.vs + off] : 0.0f;
    }
}

// The update of one cell (offset `off`, indices gi, gj, k) from its flux divergence times the
// volume, pot: Euler step / Heun stage 1 (KIND 0) or Heun stage 2 (KIND 1), p floor, source
// re-imposition, negative-density check.  cnt[0], cnt[1]: the CTA's negative-density and p-floor
// counters.
template <int P, int KIND>
__device__ __forceinline__ void update_cell(const StageArgs& A, const CellState<P, KIND>& in, long long off, int gi,
                                            int gj, int k, bool col_src, double dt_vol, const double* pot,
                                            unsigned long long* cnt) {
    const GridGeom& g = A.g;
    double un[8], qs[8];
    bool reset_comp = false;
    bool is_src = false;
    if (col_src) is_src = source_prim(g, gi, gj, k + g.koff, qs);
    if (is_src) {
        cons_from_prim_exact(qs, un);
        reset_comp = true;
    } else {
        double cmp[8];
        const double* uin = in.u;
#pragma unroll
        for (int v = 0; v < 8; v++) {
            const double inc = pot[v] * dt_vol;
            if (P != 0 && A.comp) {
                // compensated sum U_new = base + delta (cuf_solvers.cuf:741-770 as an
                // increment); the FP32 compensation carries the rounding of the add
                const double base = KIND == 0 ? uin[v] : in.base[KIND * v];
                const double delta = KIND == 0 ? -inc : 0.5 * ((uin[v] - base) - inc);
                const double y = delta - (double)in.comp[P == 0 ? 0 : v];
                const double s = base + y;
                cmp[v] = (s - base) - y;
                un[v] = s;
            } else if (KIND == 0) {
                un[v] = uin[v] - inc;
            } else {
                un[v] = 0.5 * ((in.base[KIND * v] + uin[v]) - inc);
            }
        }
        if (!(un[0] > 0.0)) {                    // cuf_solvers.cuf:708-711
            atomicAdd(&cnt[0], 1ull);
            atomicMin(&A.st->first_bad,
                      (unsigned long long)(gi + (long long)g.nx * (gj + (long long)g.ny * (k + g.koff))));
#pragma unroll
            for (int v = 0; v < 8; v++) un[v] = uin[v];
            reset_comp = true;
        } else if (P == 1 || !pressure_surely_positive(un)) {
            // the exact recovery (P != 1) only where the quick test cannot clear p > 0
            double q[8], ke, me;
            prim_from_cons<P != 1>(un, q, ke, me);
            if (q[4] <= 0.0) {                    // cuf_solvers.cuf:777-779
                atomicAdd(&cnt[1], 1ull);
                un[4] = floor_energy(ke, me);
                cmp[4] = 0.0;
            }
        }
        if (P != 0 && A.comp && !reset_comp) {
#pragma unroll
            for (int v = 0; v < 8; v++) A.comp[v * g.vs + off] = (float)cmp[v];
        }
    }
    if (P != 0 && A.comp && reset_comp) {
#pragma unroll
        for (int v = 0; v < 8; v++) A.comp[v * g.vs + off] = 0.0f;
    }
#pragma unroll
    for (int v = 0; v < 8; v++) A.Uout[v * g.vs + off] = un[v];
}

// One tile of one stage: the column (bx, by) of TX x TY cells, planes [bz*lz, min(nz, (bz+1)*lz)).
// `total_tiles` is the number of tiles of this solve in the launch; the last one to finish rolls
// the solve's clock.  Called by the single-solve kernel (one tile per CTA) and by the batch
// kernel (tiles of many solves drawn from a work queue); every CTA-wide barrier is reached by all
// threads, and the function ends with one so a CTA may run the next tile immediately.
// `tm` is the tensor map of a single solve's A.Uin, a kernel parameter; a batch's lies at A.tm_in, acquired
// by the caller (A.tm_in is null where planes are read with plain loads).
// `phase` is the parity of the next wait on the staging box's barrier and `tma_dead` is set once a plane copy did not
// land within both bounded waits (the thread then reads its planes with plain loads); both are
// per thread and carried across the tiles a CTA runs.
//
// Work split: warp w < TY owns tile row w, one lane per column, and computes that row's z faces
// (k-1/2), its x faces (i-1/2) and its y faces (j-1/2); the last warp computes what the rows leave
// over, the east x faces of all rows (row = lane) and the y faces above the last row.  A row's z
// and x fluxes therefore never leave its warp: they are summed in registers (the x neighbour's by a
// shuffle), and only the y fluxes and the east x fluxes pass through shared memory.
//
// One barrier per plane.  Interval k (between two barriers) runs
//   1. z faces k-1/2, which complete plane k-1: its update is written;
//   2. x and y faces of plane k, summed into the next update's flux divergence;
//   3. the conversion of staged plane k+2 into the ring slot of plane k-2.
// Faces of plane k read the ring planes k-1, k, k+1 only: the left state of z face k-1/2 comes
// from the slope of cell k-1, formed one plane earlier with the right state of face k-3/2 (one
// minmod per z face and variable instead of two) and carried in registers.  The exchanged y / east
// fluxes are double buffered.  Warps drift apart by up to an interval, so one warp's conversion
// and update overlap the others' faces.  Handing the faces of a plane out as warp jobs behind two
// barriers took 2.31 / 2.44 ms a stage at 256^3 (plain form), this split 2.14 / 2.25 ms with one
// solver body in a loop over the three axes and 2.04 / 2.15 ms with the loop unrolled (a third of
// the register moves and no axis dispatch; the code still streams: 4 % of stalls are
// instruction fetch), the solver unchanged.
template <int P, int NSTATE, int ORDER, int KIND, int SK, int ND>
__device__ __forceinline__ void run_tile(const StageArgs& A, const CUtensorMap* tm, int bx, int by, int bz,
                                         unsigned total_tiles, unsigned long long* bar, unsigned& phase, bool& tma_dead) {
    using RG = typename Types<P>::Ring;
    using FT = typename Types<P>::Flux;
    using RT = typename Types<P>::Math;
    using C = Tile<P, SK>;
    constexpr bool WANT_DT = KIND == 0;   // the first stage's faces give the next step's dt
    constexpr int TX = C::TX, TY = C::TY, NC = C::NC, NT = C::NT, HX = C::HX, PLANE = C::PLANE;
    constexpr int NYF = C::NYF;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // [8][PLANE] staged conserved box; tensor copies land on a 128-byte aligned address.  The
    // alignment pad is an offset from the shared array itself, so every pointer below stays in
    // the shared address space (shared loads and stores with 32-bit addresses, not generic ones).
    const unsigned pad = (128u - (smem_u32(smem_raw) & 127u)) & 127u;
    double* stg = reinterpret_cast<double*>(smem_raw + pad);
    RG* ring = reinterpret_cast<RG*>(stg + 8 * PLANE);
    FT* fy = reinterpret_cast<FT*>(ring + RING * 8 * PLANE);   // [2][8][NYF]: y fluxes of plane k at k & 1
    FT* fe = fy + 2 * 8 * NYF;                                  // [2][8][TY]: east x fluxes
    __shared__ double red[NT / 32];
    __shared__ unsigned long long cnt[6];
    __shared__ bool last_cta;

    const GridGeom& g = A.g;
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const bool rows = warp < TY;   // owns a tile row
    const int i0 = bx * TX, j0 = by * TY;
    const int gi = i0 + lane, gj = j0 + warp;
    const bool own = rows && gi < g.nx && gj < g.ny;
    const int kb = plane_begin(g), ke = plane_end(g);
    const int k0 = kb + bz * g.lz;
    const int k1 = min(ke, k0 + g.lz);
    const double dt = A.clk->dt_cur;
    const double dt_vol = dt * g.inv_vol;   // dt / cell volume
    if (t < 6) cnt[t] = 0;

    double rate = 0.0;   // max over this thread's real faces of max(|SL|,|SR|)/dist
    unsigned n_recon = 0, n_wave = 0, n_redo = 0, n_tmo = 0;

    // ---- plane staging.  Plane kk enters ring slot kk & 3.  With a tensor map, the copy of the
    // next plane is in flight while the faces and the update of an interval run; the last copy
    // issued is plane k1+1.
    const bool use_tma = A.tm_in != nullptr && !tma_dead;
    const bool late = A.copy_wait < 0;   // each copy issued right before its waits, which run out
    constexpr unsigned kPlaneBytes = 8u * PLANE * sizeof(double);
    const int kz_last = k1 + 1;
    auto issue_copy = [&](int kk) {
        tma_plane(stg, ND == 2 ? A.tm_in : tm, i0 - 2, j0 - 2, min(max(kk, 0), g.nz - 1), kPlaneBytes, bar);
    };
    // Converts plane kk for the cells c0, c0 + step, ... < c1 of this thread.
    auto take_plane = [&](int kk, int c0, int step, int c1) {
        RG* slot = ring + ring_slot(kk) * 8 * PLANE;
        if (use_tma && !tma_dead) {
            if (late && t == 0) issue_copy(kk);
            // A wait that runs out is counted (SETB_ETIMEOUT), then the copy gets a second bounded
            // wait to land before the box is read; a copy that never lands switches this thread to
            // plain loads (and thread 0 stops issuing copies), so no read races a late copy.
            bool ok = mbar_wait_bounded(bar, phase, A.copy_wait);
            if (!ok) {
                n_tmo++;
                ok = mbar_wait_bounded(bar, phase, kCopyWaitCycles);
            }
            phase ^= 1u;
            if (ok) convert_plane<P, SK, RG>(A, stg, slot, i0, j0, c0, step, c1);
            else tma_dead = true;
        }
        if (!use_tma || tma_dead) load_planes<P, SK, RG>(A, ring, i0, j0, kk, c1, c0, step);
        __syncthreads();
        if (use_tma && !tma_dead && !late && t == 0 && kk < kz_last) issue_copy(kk + 1);
    };
    // The first four planes come by plain loads, all in flight together, while the first copy (plane
    // k0+2) runs: the values are the same, and four copies one after the other through the staging
    // box would take four latencies (32^3 a stage: 22 -> 20 us).
    if (use_tma && !late && t == 0) issue_copy(k0 + 2);
    load_planes<P, SK, RG>(A, ring, i0, j0, k0 - 2, 4 * PLANE, t, NT);
    __syncthreads();

    // whether this thread's column crosses the source sphere (x^2 + y^2 < r_src^2)
    bool col_src;
    {
        const double x = cell_coord(g.lo[0], gi, g.h[0]), y = cell_coord(g.lo[1], gj, g.h[1]);
        col_src = g.r_src > 0.0 && dadd(dmul(x, x), dmul(y, y)) < dmul(g.r_src, g.r_src);
    }

    const int cc = (warp + 2) * HX + lane + 2;   // this thread's cell in a ring plane
    // left state of the next z face (ORDER 2): t_c + 0.5*minmod of cell k-1, face-frame order
    RT zl[5] = {};
    if (ORDER == 2 && rows) {
        const RG* pm = ring + ring_slot(k0 - 2) * 8 * PLANE + cc;
        const RG* pc = ring + ring_slot(k0 - 1) * 8 * PLANE + cc;
        const RG* pp = ring + ring_slot(k0) * 8 * PLANE + cc;
#pragma unroll
        for (int v = 0; v < 5; v++) {
            const int o = face_perm<2>(v) * PLANE;
            zl[v] = muscl((RT)pm[o], (RT)pc[o], (RT)pp[o]);
        }
        if (sb_neg(zl[0])) zl[0] = (RT)pc[face_perm<2>(0) * PLANE];
        if (sb_neg(zl[4])) zl[4] = (RT)pc[face_perm<2>(4) * PLANE];
    }
    __syncthreads();   // the first interval converts into the slot of plane k0-2

    // A face that another tile computes too (where the grid goes on: the z face below the chunk, the east x
    // faces and the y faces above the last row) enters dt candidates and diagnostics in one of the two only.
    // Plain and delta forms: bit r, this thread's z, x or y face is one that this tile counts (256^3 Heun
    // 20.82 ms for six steps; with the conditions formed at each face 21.1-21.2, behind warp votes 21.46,
    // with every face counted 20.95; delta 160x131x192 6.77 / 6.9 / 7.09 / 6.73).  The mixed form has no
    // register for the bits: it asks behind a vote, where there is something to count (count_face; six-grid
    // ensemble 227 ms, with the bits 232, with every face counted 228; 384^3 32.3 / 32.2 / 32.5).
    unsigned faces = 0;
    if constexpr (P != 1) {
        faces = own ? 1u : 0u;
        if (rows ? gi <= g.nx && gj < g.ny : lane < TY && i0 + TX == g.nx && j0 + lane < g.ny) faces |= 2u;
        if (gi < g.nx && (rows ? gj <= g.ny : gj == g.ny)) faces |= 4u;
    }

    // Flux sums of the plane in progress, natural component order.  FP64 fluxes: acc is the
    // area-weighted sum so far (starting with minus the z flux below); FP32 fluxes: the x
    // difference and the z flux below are kept apart, so the sum keeps its written order.
    double acc[P == 1 ? 1 : 8] = {};
    float ax[P == 1 ? 8 : 1] = {}, fzl[P == 1 ? 8 : 1] = {};
#pragma unroll 1
    for (int k = k0; k <= k1; k++) {
#pragma unroll
        for (int r = 0; r < 3; r++) {   // z face k-1/2, x faces, y faces
            if (r == 0 ? !rows : k == k1) continue;
            int axis, fxx, fyy;
            bool real;   // counted by this tile (mixed form: a face of the grid)
            double sq, idist;   // face area and 1/dist of the axis
            RT q1[8], q2[8];
            if (r == 0) {
                axis = 2;
                sq = g.square[2];
                idist = g.inv_dist[2];
                fxx = lane;
                fyy = warp;
                const RG* pL = ring + ring_slot(k - 1) * 8 * PLANE + cc;
                const RG* pR = ring + ring_slot(k) * 8 * PLANE + cc;
                const RG* pRR = ring + ring_slot(k + 1) * 8 * PLANE + cc;
#pragma unroll
                for (int v = 0; v < 8; v++) {
                    const int o = face_perm<2>(v) * PLANE;
                    q1[v] = (RT)pL[o];
                    q2[v] = (RT)pR[o];
                    if (ORDER == 2 && v < 5) {
                        const RT c = q2[v];
                        // minmod() and not slope(): either far cell may be invalid here, this
                        // face's or the next one's
                        const RT m = minmod(c - q1[v], (RT)pRR[o] - c);
                        q1[v] = zl[v];
                        q2[v] = c - RT(0.5) * m;
                        zl[v] = c + RT(0.5) * m;
                        if (v == 0 || v == 4) {
                            if (sb_neg(q2[v])) q2[v] = c;
                            if (sb_neg(zl[v])) zl[v] = c;
                        }
                    }
                }
                real = P == 1 ? own : (faces & 1u) && (k > k0 || k0 == kb);
            } else if (r == 1) {
                axis = 0;
                sq = g.square[0];
                idist = g.inv_dist[0];
                fxx = rows ? lane : TX;
                fyy = rows ? warp : min(lane, TY - 1);
                const RG* b = ring + ring_slot(k) * 8 * PLANE + (fyy + 2) * HX + fxx;
                face_states<0, PLANE, P, ORDER>(b, b + 1, b + 2, b + 3, q1, q2);
                real = P == 1 ? (rows || lane < TY) && i0 + fxx <= g.nx && j0 + fyy < g.ny : (faces & 2u) != 0;
            } else {
                axis = 1;
                sq = g.square[1];
                idist = g.inv_dist[1];
                fxx = lane;
                fyy = warp;
                const RG* b = ring + ring_slot(k) * 8 * PLANE + cc - 2 * HX;
                face_states<1, PLANE, P, ORDER>(b, b + HX, b + 2 * HX, b + 3 * HX, q1, q2);
                real = P == 1 ? gi < g.nx && gj <= g.ny : (faces & 4u) != 0;
            }
            auto count_face = [&](int which) {   // mixed form
                if (real && (r == 0 ? k > k0 || k0 == kb : rows || (r == 1 ? i0 + TX == g.nx : gj == g.ny)))
                    atomicAdd(&cnt[which], 1ull);
            };
            const bool recon = sb_neg(q1[0]) || sb_neg(q2[0]);
            if constexpr (P == 1) {
                if (__any_sync(0xffffffffu, recon) && recon) count_face(2);
            } else {
                if (real && recon) n_recon++;
            }
            int fl;
            double sl, sr;
            RT F[8];
            bool redone = false;
            if constexpr (P == 2) {
                float SLf, SRf, SMf;
                fl = riemann_delta<NSTATE>(q1, q2, F, SLf, SRf, SMf);
                sl = (double)SLf;
                sr = (double)SRf;
                redone = fl & kFlagStar;
            } else {
                RT SL, SR, SM;
                if constexpr (P == 1 && NSTATE >= 2) {
                    if (A.n_disc == 0)
                        fl = riemann_f32x2<NSTATE, ND != 2>(q1, q2, F, SL, SR, SM);
                    else
                        fl = riemann<RT, NSTATE, false, true, true, false, false>(q1, q2, RT(0), A.n_disc, F, SL, SR, SM);
                } else if constexpr (P == 0) {
                    // the plain form's ring holds b = B / sqrt(4 pi) (BS), and its flux sums hold
                    // the field's fluxes in those units
                    bool general = true;
                    if constexpr (NSTATE >= 2 && ND != 1) {
                        if (ND == 0 || A.n_disc == 0) {
                            general = false;
                            fl = flux_fp64<NSTATE>(q1, q2, F, SL, SR) ? kFlagWave : 0;
                        }
                    }
                    if (general) {
                        fl = riemann<RT, NSTATE, false, false, true, true>(q1, q2, RT(0), A.n_disc, F, SL, SR, SM);
#pragma unroll
                        for (int v = 5; v < 8; v++) F[v] = F[v] * (RT)kInvSpi4;
                    }
                } else {
                    fl = riemann<RT, NSTATE, false, true, true, false>(q1, q2, RT(0), A.n_disc, F, SL, SR, SM);
                }
                sl = (double)SL;
                sr = (double)SR;
                redone = P == 1 && real && (fl & kFlagStar);
            }
            if (P == 1) {
#pragma unroll
                for (int v = 0; v < 8; v++) F[v] = __fmul_rn((float)F[v], (float)sq);   // rounded before it is summed
            }
            // the same face states, refetched: FP64 throughout
            if constexpr (P == 2) {
                if (redone) {
                    const FaceFlux f = face_fp64<NSTATE, ORDER>(fetch_args(A), axis, i0 + fxx, j0 + fyy, k);
                    fl = f.fl;
                    sl = f.sl;
                    sr = f.sr;
#pragma unroll
                    for (int v = 0; v < 8; v++) F[v] = f.F[face_perm_dyn(axis, v)];
                    if (real) n_redo++;
                }
            }
            if constexpr (P == 1) {
                // What is live here is parked in local memory around the call by hand: left to the
                // compiler, the call's register convention spills it on the common path (stage 1 /
                // 2 at 384^3: 4.81 / 5.58 against 5.04 / 5.67 ms).
                if (__any_sync(0xffffffffu, redone)) {
                    volatile float park[30];
                    volatile double park_rate = rate;
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        park[v] = F[v];
                        park[8 + v] = ax[v];
                        park[16 + v] = fzl[v];
                        if (ORDER == 2 && v < 5) park[24 + v] = zl[v];
                    }
                    const FaceFlux f = face_fp64<NSTATE, ORDER>(fetch_args(A), axis, i0 + fxx, j0 + fyy, k);
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        F[v] = park[v];
                        ax[v] = park[8 + v];
                        fzl[v] = park[16 + v];
                        if (ORDER == 2 && v < 5) zl[v] = park[24 + v];
                    }
                    rate = park_rate;
                    if (redone) {
                        fl = f.fl;
                        sl = f.sl;
                        sr = f.sr;
#pragma unroll
                        for (int v = 0; v < 8; v++) F[v] = (RT)(f.F[face_perm_dyn(axis, v)] * sq);
                        count_face(4);
                    }
                }
            }
            // a face no wave-fan region matched gets a zero flux; the warp vote keeps the (never
            // taken in a valid state) zeroing out of the common path
            if (__any_sync(0xffffffffu, fl & kFlagWave) && (fl & kFlagWave)) {
                if (!(P == 1 && redone)) {
#pragma unroll
                    for (int v = 0; v < 8; v++) F[v] = RT(0);
                }
                if (P == 1) count_face(3);
            }
            if (P != 1 && (fl & kFlagWave) && real) n_wave++;
            // compare-and-select maxima (the library fmax of doubles is a far longer sequence); a NaN
            // speed is skipped, as fmax would skip it
            if (WANT_DT && real) rate = sb_max(rate, sb_max(fabs(sl), fabs(sr)) * idist);

            if (r == 1) {
                FT* e = fe + (k & 1) * 8 * TY;
                if (!rows) {
                    if (lane < TY) {
#pragma unroll
                        for (int v = 0; v < 8; v++) e[face_perm<0>(v) * TY + lane] = F[v];
                    }
                } else {   // F(i+1/2) - F(i-1/2); lane 31's F(i+1/2) is the east flux, added later
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        const RT hi = __shfl_down_sync(0xffffffffu, F[v], 1);
                        if constexpr (P == 1) ax[face_perm<0>(v)] = lane < 31 ? hi - F[v] : F[v];
                        else acc[face_perm<0>(v)] = fma(sq, (lane < 31 ? hi : 0.0) - F[v], acc[face_perm<0>(v)]);
                    }
                }
            } else if (r == 2) {
                FT* y = fy + (k & 1) * 8 * NYF + warp * TX + lane;
#pragma unroll
                for (int v = 0; v < 8; v++) {
                    y[face_perm<1>(v) * NYF] = F[v];
                    if constexpr (P != 1) {
                        if (rows) acc[face_perm<1>(v)] = fma(-sq, F[v], acc[face_perm<1>(v)]);
                    }
                }
            } else {
                if (k > k0) {   // plane k-1 is complete: update it
                    const int kf = k - 1;
                    const FT* yl = fy + (kf & 1) * 8 * NYF + warp * TX + lane;
                    const FT* e = fe + (kf & 1) * 8 * TY + warp;
                    const long long off = (long long)kf * g.ps + (long long)gj * g.px + gi;
                    // The plain form's Heun stage 2 streams its base state U^n from HBM, which no
                    // plane copy has touched: ask L2 for the next plane's cells now, so their
                    // loads one interval later hit L2 instead of waiting on DRAM (stage 2 at
                    // 256^3: 2.78 -> 2.74 ms; the same hint in the mixed form, for U^n and its
                    // compensation, measured 1-2 % slower).
                    if (P == 0 && KIND == 1 && own && k < k1) {
#pragma unroll
                        for (int v = 0; v < 8; v++)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(A.Ubase + v * g.vs + off + g.ps));
                    }
                    double pot[8];   // flux divergence times the volume
#pragma unroll
                    for (int w = 0; w < 8; w++) {
                        const int v = face_perm<2>(w);
                        if constexpr (P == 1) {
                            // FP32 fluxes: each opposite-face difference is exact when the two
                            // fluxes are within a factor 2 (Sterbenz) and otherwise rounds
                            // relative to the difference, far below the fluxes' own FP32
                            // rounding; one conversion per variable instead of six
                            const float dx = lane < 31 ? ax[v] : e[v * TY] - ax[v];
                            const float dy = yl[v * NYF + TX] - yl[v * NYF];
                            pot[v] = (double)((dx + dy) + (F[w] - fzl[v]));
                        } else {
                            double s = fma(g.square[1], (double)yl[v * NYF + TX], acc[v]);
                            if (lane == 31) s = fma(g.square[0], (double)e[v * TY], s);
                            pot[v] = fma(sq, (double)F[w], s);
                            if (P == 0 && v >= 5) pot[v] *= kSpi4;
                        }
                    }
                    if (own) {
                        CellState<P, KIND> in;
                        load_cell<P, KIND>(A, off, in);
                        update_cell<P, KIND>(A, in, off, gi, gj, kf, col_src, dt_vol, pot, cnt);
                    }
                }
#pragma unroll
                for (int w = 0; w < 8; w++) {
                    const int v = face_perm<2>(w);
                    if constexpr (P == 1) fzl[v] = F[w];
                    else acc[v] = -(sq * F[w]);
                }
            }
        }
        if (k == k1) break;
        // rows take their own columns' share of the staged plane, the last warp the halo's rest
        take_plane(k + 2, rows ? t : NC + lane, 32, rows ? t + 1 : PLANE);
    }

    // ---- reductions: counters and the dt candidate
    if (n_recon) atomicAdd(&cnt[2], (unsigned long long)n_recon);
    if (n_wave) atomicAdd(&cnt[3], (unsigned long long)n_wave);
    if (n_redo) atomicAdd(&cnt[4], (unsigned long long)n_redo);
    if (n_tmo) atomicAdd(&cnt[5], (unsigned long long)n_tmo);
    if (WANT_DT) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) rate = fmax(rate, __shfl_xor_sync(0xffffffffu, rate, o));
        if ((t & 31) == 0) red[t >> 5] = rate;
    }
    __syncthreads();
    if (t == 0) {
        if (WANT_DT) {
            double r = red[0];
#pragma unroll
            for (int w = 1; w < NT / 32; w++) r = fmax(r, red[w]);
            const double cand = fmin(kDtFaceCap, A.cfl / r);   // r == 0 -> +inf -> cap
            atomicMin(&A.clk->dt_next, (unsigned long long)__double_as_longlong(cand));
        }
        if (cnt[0]) atomicAdd(&A.st->n_negdens, cnt[0]);
        if (cnt[1]) atomicAdd(&A.st->n_pfloor, cnt[1]);
        if (cnt[2]) atomicAdd(&A.st->n_recon, cnt[2]);
        if (cnt[3]) atomicAdd(&A.st->n_wave, cnt[3]);
        if (cnt[4]) atomicAdd(&A.st->n_redo, cnt[4]);
        if (cnt[5]) atomicAdd(&A.st->n_timeout, cnt[5]);
        __threadfence();
        const unsigned ticket = atomicAdd(&A.clk->counter, 1u);
        last_cta = (ticket == total_tiles - 1);
    }
    __syncthreads();
    if (last_cta && t == 0) {
        __threadfence();
        DevClock* c = A.clk;
        c->counter = 0;
        if (A.finalize) {
            const unsigned long long nb = atomicExch(&c->dt_next, (unsigned long long)__double_as_longlong(kDtReset));
            c->time_all += c->dt_cur;
            c->dt_last = c->dt_cur;
            c->dt_cur = __longlong_as_double((long long)nb);
            c->steps += 1;
        }
        __threadfence();
    }
    __syncthreads();
}

template <int P, int NSTATE, int ORDER, int KIND, int ND, int SK>
__global__ void __launch_bounds__(Tile<P, SK>::NT, Tile<P, SK>::MINB)
    stage_kernel(const StageArgs A, const __grid_constant__ CUtensorMap tm) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) mbar_init(&bar);
    __syncthreads();
    allow_successor();
    wait_for_predecessor();
    unsigned phase = 0;
    bool tma_dead = false;
    run_tile<P, NSTATE, ORDER, KIND, SK, ND>(A, &tm, blockIdx.x, blockIdx.y, blockIdx.z,
                                             gridDim.x * gridDim.y * gridDim.z, &bar, phase, tma_dead);
}

// Persistent batch kernel: each CTA takes tiles from the work queue until it is empty; the
// tile's solve selects the arguments (copied to shared memory).  One launch covers the solves of
// one Riemann solver (NSTATE), so the kernel holds one solver body.  The items of one solve are
// counted by its own clock, so every solve keeps its own lagged dt.
template <int P, int NSTATE, int ORDER, int KIND>
__global__ void __launch_bounds__(Tile<P, kBatchShape>::NT, Tile<P, kBatchShape>::MINB) batch_stage_kernel(const BatchArgs B) {
    __shared__ __align__(16) StageArgs As;
    __shared__ int4 it;
    __shared__ __align__(8) unsigned long long bar;
    constexpr int WORDS = sizeof(StageArgs) / sizeof(unsigned long long);
    static_assert(sizeof(StageArgs) % sizeof(unsigned long long) == 0, "StageArgs must be 8-byte granular");
    __shared__ int acquired;   // the solve whose tensor map this CTA has acquired
    if (threadIdx.x == 0) {
        mbar_init(&bar);
        acquired = -1;
    }
    unsigned phase = 0;   // the same in every thread
    bool tma_dead = false;
    for (;;) {
        if (threadIdx.x == 0) {
            const unsigned i = atomicAdd(B.queue, 1u);
            it = i < (unsigned)B.n_items ? B.items[i] : make_int4(-1, 0, 0, 0);
        }
        __syncthreads();
        const int4 w = it;
        if (w.x < 0) break;
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(B.inst + w.x);
        unsigned long long* dst = reinterpret_cast<unsigned long long*>(&As);
        for (int q = threadIdx.x; q < WORDS; q += Tile<P, kBatchShape>::NT) dst[q] = src[q];
        __syncthreads();
        if (threadIdx.x == 0 && acquired != w.x) {
            if (As.tm_in) acquire_tmap(As.tm_in);
            acquired = w.x;
        }
        run_tile<P, NSTATE, ORDER, KIND, kBatchShape, 2>(As, nullptr, w.y, w.z, w.w, As.total_tiles, &bar, phase,
                                                         tma_dead);
    }
}

template <int P, int NSTATE, int ORDER, int KIND, int ND, int SK>
cudaError_t launch_shape(const StageArgs& a, cudaStream_t s) {
    auto kern = stage_kernel<P, NSTATE, ORDER, KIND, ND, SK>;
    const int smem = Tile<P, SK>::kSmem;
    // The dynamic shared-memory opt-in is a per-device attribute of the kernel: set it once per
    // device ordinal (a bit per device, atomically; two threads that both set it set the same
    // value), and on every launch for ordinals beyond the mask.
    static std::atomic<unsigned long long> attr_set{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
    if (!bit || !(attr_set.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
        attr_set.fetch_or(bit, std::memory_order_release);
    }
    constexpr int TX = Tile<P, SK>::TX, TY = Tile<P, SK>::TY;
    const int nzu = plane_end(a.g) - plane_begin(a.g);
    dim3 grid((a.g.nx + TX - 1) / TX, (a.g.ny + TY - 1) / TY, (nzu + a.g.lz - 1) / a.g.lz);
    return launch_chained(kern, grid, Tile<P, SK>::NT, smem, s, a, a.tm_in ? *a.tm_in : CUtensorMap{});
}

template <int P, int NSTATE, int ORDER, int KIND, int ND>
cudaError_t launch_nd(const StageArgs& a, cudaStream_t s) {
    if constexpr (num_shapes(P) > 1)
        if (a.shape == 1) return launch_shape<P, NSTATE, ORDER, KIND, ND, 1>(a, s);
    return launch_shape<P, NSTATE, ORDER, KIND, ND, 0>(a, s);
}

// n_disc selects the wave-speed estimate.  The plain form's HLLC / HLLD for n_disc 0 have a solver
// of their own (flux_fp64); every other combination reads n_disc at run time (ND = 1).
template <int P, int NSTATE, int ORDER, int KIND>
cudaError_t launch_t(const StageArgs& a, cudaStream_t s) {
    if constexpr (P == 0 && NSTATE >= 2)
        if (a.n_disc == 0) return launch_nd<P, NSTATE, ORDER, KIND, 0>(a, s);
    return launch_nd<P, NSTATE, ORDER, KIND, 1>(a, s);
}

template <int P, int NSTATE>
cudaError_t launch_n(const StageArgs& a, int order, int kind, cudaStream_t s) {
    if (order == 2) return kind == 0 ? launch_t<P, NSTATE, 2, 0>(a, s) : launch_t<P, NSTATE, 2, 1>(a, s);
    return kind == 0 ? launch_t<P, NSTATE, 1, 0>(a, s) : launch_t<P, NSTATE, 1, 1>(a, s);
}

template <int P, int NSTATE>
cudaError_t batch_attr() {
    cudaError_t e = cudaFuncSetAttribute(batch_stage_kernel<P, NSTATE, 2, 0>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<P, kBatchShape>::kSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(batch_stage_kernel<P, NSTATE, 2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                Tile<P, kBatchShape>::kSmem);
}

template <int P, int NSTATE>
void launch_batch_n(const BatchArgs& b, int kind, int grid, cudaStream_t s) {
    constexpr int NT = Tile<P, kBatchShape>::NT;
    if (kind == 0) batch_stage_kernel<P, NSTATE, 2, 0><<<grid, NT, Tile<P, kBatchShape>::kSmem, s>>>(b);
    else batch_stage_kernel<P, NSTATE, 2, 1><<<grid, NT, Tile<P, kBatchShape>::kSmem, s>>>(b);
}

}  // namespace

template <int P>
cudaError_t launch_stage_form(const StageArgs& a, int n_state, int order, int kind, cudaStream_t s) {
    if constexpr (P != 2) {   // the delta form covers HLLC (n_state 2) and HLLD (n_state 3)
        if (n_state == 0) return launch_n<P, 0>(a, order, kind, s);
        if (n_state == 1) return launch_n<P, 1>(a, order, kind, s);
    }
    return n_state == 2 ? launch_n<P, 2>(a, order, kind, s) : launch_n<P, 3>(a, order, kind, s);
}

template <int P>
cudaError_t launch_batch_form(const BatchArgs& b, int n_state, int kind, int grid, cudaStream_t s) {
    if (n_state == 3) launch_batch_n<P, 3>(b, kind, grid, s);
    else launch_batch_n<P, 2>(b, kind, grid, s);
    return cudaGetLastError();
}

template <int P>
cudaError_t prepare_batch_form() {
    const cudaError_t e = batch_attr<P, 3>();
    return e != cudaSuccess ? e : batch_attr<P, 2>();
}

}  // namespace sb
