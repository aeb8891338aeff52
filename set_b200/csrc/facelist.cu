// facelist.cu -- the MHD step on the reference's own geometry: an explicit face list.
//
// The reference's GPU solver (SET_Fortran_Cuda_MHD/cuf_solvers.cuf) runs on an unstructured grid
// of cells and faces read from the grid file (Storage_module.f90:20-37): a face kernel
// (CUF_MGD_grans_RK2, :243-440) computes each face's flux once into Gran_POTOK and a cell kernel
// (CUF_MGD_cell_RK2, :561-794) sums the fluxes of its faces with the owner sign.  This file keeps
// that structure, B200-side:
//   * the cell state is conserved SoA FP64 (coalesced in the cell kernel); the primitive state is
//     kept beside it cell-major (8 doubles = 64 B per cell), so a face gathers a cell with four
//     16-byte loads; a pass of its own forms it for the first stage of a call, the cell kernel
//     leaves it for every later one;
//   * per-face geometry the face kernel needs (the slope weights of the TVD distances, the
//     reference's "skip" rule, the owner sign) is derived once at set-up in FP64, so the stage
//     kernels read it instead of recomputing it from cell centres;
//   * the face kernel reduces the dt candidate with warp shuffles and one atomicMin per block;
//     the cell kernel's last block rolls the lagged-dt clock on the device, so a run of steps
//     needs no host round trip;
//   * the face flux array persists between stages: a skipped face keeps its previous flux, as
//     Gran_POTOK does in the reference.
// Physics 0 is the conservative ideal-MHD update of all 8 variables used by the Cartesian path,
// optionally with the div-B terms the reference carries commented out (face flux Gran_POTOK(9),
// sources proportional to its owner-signed sum); physics 1 is the reference's live cell kernel,
// a 2D axisymmetric hydro update with charge exchange.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <utility>
#include <vector>

#include "setb200.h"
#include "setb_internal.cuh"
#include "riemann_fp64.cuh"

namespace sb {

// What the kernels read (passed by value).
struct FlView {
    int64_t n_cell = 0, n_gran = 0;
    // cells
    double* cell_center = nullptr;   // [N][3]
    double* inv_volume = nullptr;    // [N] 1 / volume
    int32_t* cell_gran = nullptr;    // [N][6]: +-(face + 1), + where the cell is the face's first
                                     // neighbour; 0 = none
    unsigned char* cell_flag = nullptr;   // kFrozen, kSource
    // faces
    double* normal = nullptr;        // [G][4]: normal, area
    double* geo = nullptr;           // [G][4]: dist = |c_face - c_s1|, and the weights of the face
                                     // values' slopes (fl_face_kernel)
    int32_t* nb = nullptr;           // [G][4]: neighbours 1, 2 (a ghost face: 1 again) and the TVD cells
                                     // (both -1 where the face is first order), 0-based
    int32_t* type = nullptr;         // [G]: 0 = skipped, else the reference's face type 1..5
                                     // (kInner: an interior type-2 face), plus kLaxFace on the
                                     // near-axis faces of physics 1
    // work
    double* prim = nullptr;          // [N][8] primitive state of the stage input, field as b = B / sqrt(4 pi)
    double* flux = nullptr;          // [G+1][8] face flux * area (persistent), field fluxes in units of b;
                                     // the last row stays zero (a cell's missing faces)
    GridGeom src{};                  // source-sphere parameters (r_src 0 = none)
    double* hatom = nullptr;         // physics 1: [N][8] H-atom fluids (Cell_par columns 9..16)
    int powell = 0;                  // physics 0: div-B terms (0 off, 1 momentum + induction, 2 + energy)
    double* divb = nullptr;          // powell: [G+1] div-B face flux * area, Gran_POTOK(9) (persistent)
};

struct FaceListDev {
    FlView v;
    int physics = 0;                 // 0: 3D MHD; 1: the reference's axisymmetric hydro update
    // locality order: device cell d holds the caller's cell perm[d] (both 0-based)
    std::vector<int32_t> perm;
};

namespace {

constexpr int kFaceThreads = 64, kCellThreads = 256, kPrimThreads = 256;
constexpr int kInner = 6;     // face type: a type-2 face with a second neighbour
constexpr int kLaxFace = 8;   // face-type bit: the reference's Lax flux on near-axis faces
constexpr int kFrozen = 1, kSource = 2;   // cell flags: not updated; inside the source sphere

double norm3(const double* x) {
    return std::sqrt((x[0] * x[0] + x[1] * x[1]) + x[2] * x[2]);
}

template <typename T>
cudaError_t upload(T** dst, const T* src, size_t n, cudaStream_t s) {
    cudaError_t e = cudaMalloc(dst, sizeof(T) * std::max<size_t>(n, 1));
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(*dst, src, sizeof(T) * n, cudaMemcpyHostToDevice, s);
}

// ------------------------------------------------------------------------------ kernels
__device__ __forceinline__ void store_prim(double* P, int64_t c, const double* q) {
    double2* p2 = reinterpret_cast<double2*>(P + 8 * c);
#pragma unroll
    for (int v = 0; v < 4; v++) p2[v] = make_double2(q[2 * v], q[2 * v + 1]);
}

// Primitive state of the first stage of a call (later stages get theirs from the cell kernel).
__global__ void fl_prim_kernel(int64_t n, const double* U, int64_t vs, double* P) {
    allow_successor();
    wait_for_predecessor();
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += (int64_t)gridDim.x * blockDim.x) {
        double u8[8], q[8], ke, me;
#pragma unroll
        for (int v = 0; v < 8; v++) u8[v] = U[v * vs + c];
        prim_from_cons<true, true>(u8, q, ke, me);
        store_prim(P, c, q);
    }
}

// The first NV (even) components of a cell's primitive state.
template <int NV = 8>
__device__ __forceinline__ void load_prim(const double* P, int64_t c, double* q) {
    const double2* p2 = reinterpret_cast<const double2*>(P + 8 * c);
#pragma unroll
    for (int v = 0; v < NV / 2; v++) {
        const double2 d = p2[v];
        q[2 * v] = d.x;
        q[2 * v + 1] = d.y;
    }
}

// Source_MK (SET_Fortran_Cuda_MHD/cuf_kernel.cuf:215-288): charge-exchange momentum (x, y) and
// energy sources against two H-atom fluids (rho, u, v, T per fluid in h[0..3], h[4..7]).  The
// reference's default-real literals enter as their single-precision values.  Common denominators are
// reciprocals (rounding only): the cell kernel is a chain of dependent FP64 operations.
__device__ __forceinline__ void source_mk(const double* q, const double* h, double* out) {
    const double pi = 3.141592653589793;
    const double rho = q[0], u = q[1], v = q[2], p = q[4];
    const double small = (double)0.0000001f;
    const double c_m = 64.0 / (9.0 * pi), c_u = 4.0 / pi;
    const double c_s = (double)0.1307345665f;
    const double c_n = (double)(3.0f / 0.4326569f);
    const double tp = p * rs_rcp(rho);   // p / rho
    double s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        double rH = h[4 * k], tH = h[4 * k + 3];   // 2 pH / rH = T
        const double uH = h[4 * k + 1], vH = h[4 * k + 2];
        if (rH < small) {
            rH = small;
            tH = 0.0;
        }
        const double du = u - uH, dv = v - vH;
        const double th = tp + tH;
        const double d2 = fma(dv, dv, du * du);
        const double um2 = fma(c_m, th, d2), uh2 = fma(c_u, th, d2);
        const double iUM = rs_rsqrt(um2), UM = um2 * iUM, UH = over_sqrt(uh2, uh2);
        const double lg = fma(-0.5 * c_s, log(um2), 1.0);
        const double cn = c_n * ((rho * rH * UM) * (lg * lg));
        s1 = fma(cn, uH - u, s1);
        s2 = fma(cn, vH - v, s2);
        const double ke = 0.5 * (fma(vH, vH, uH * uH) - fma(v, v, u * u));
        s3 = fma(cn, fma(UH * iUM, tH - tp, ke), s3);
    }
    out[0] = s1;
    out[1] = s2;
    out[2] = s3;
}

// The reference's live cell update (cuf_solvers.cuf:561-794): 2D axisymmetric hydro about the x
// axis with radius rr(2) = y, w = B = 0, charge exchange, p floor and the near-axis v clamp.  q: the
// stage input's primitive state; writes the conserved result to un; returns 1 for a non-positive
// density (un = the stage input), 2 when the p floor applied.
template <int KIND>
__device__ __forceinline__ int axisym_update(const double* Uin, const double* Ubase, int64_t vs, int64_t c,
                                             const double* q, const double* pot, double ivol, double x, double y,
                                             const double* h, double t, double* un) {
    double u8[8], source[3];
#pragma unroll
    for (int v = 0; v < 8; v++) u8[v] = Uin[v * vs + c];
    double b8[8];   // the base state of the sum: itself, or Heun stage 2's U^n (energies without field)
    if (KIND == 1) {
#pragma unroll
        for (int v = 0; v < 8; v++) b8[v] = Ubase[v * vs + c];
        b8[4] -= (0.5 * kInvSpi4 * kInvSpi4) * fma(b8[7], b8[7], fma(b8[6], b8[6], b8[5] * b8[5]));
    }
    source_mk(q, h, source);
    const double iy = rs_rcp(y);
    const double uv2 = fma(q[2], q[2], q[1] * q[1]);
    const double e1 = fma(0.5 * q[0], fma(q[3], q[3], uv2), kInvG1 * q[4]);
    const double X = fma(0.5 * q[0], uv2, (kGamma * kInvG1) * q[4]);
    const double rv = q[0] * q[2] * iy;   // rho v / y
    const double d0 = fma(pot[0], ivol, rv), d1 = fma(pot[1], ivol, fma(rv, q[1], -source[0]));
    const double d2 = fma(pot[2], ivol, fma(rv, q[2], -source[1]));
    const double d4 = fma(pot[4], ivol, fma(q[2] * iy, X, -source[2]));
    double ro3, mx, my, e3;
    if (KIND == 0) {
        ro3 = fma(-t, d0, u8[0]);
        mx = fma(-t, d1, u8[1]);
        my = fma(-t, d2, u8[2]);
        e3 = fma(-t, d4, e1);
    } else {
        ro3 = 0.5 * fma(-t, d0, b8[0] + u8[0]);
        mx = 0.5 * fma(-t, d1, b8[1] + u8[1]);
        my = 0.5 * fma(-t, d2, b8[2] + u8[2]);
        e3 = 0.5 * fma(-t, d4, b8[4] + e1);
    }
    if (!(ro3 > 0.0)) {
#pragma unroll
        for (int v = 0; v < 8; v++) un[v] = u8[v];
        return 1;
    }
    const double i3 = rs_rcp(ro3);
    const double u3 = mx * i3;
    double v3 = my * i3;
    double p3 = fma(-0.5 * ro3, fma(v3, v3, u3 * u3), e3) * kG1;
    int rc = 0;
    if (p3 <= 0.0) {
        p3 = kPFloor;
        rc = 2;
    }
    if (x > (double)0.28f && y < (double)0.07f && v3 < 0.0) v3 = (double)0.01f;
    un[0] = ro3;
    un[1] = ro3 * u3;
    un[2] = ro3 * v3;
    un[4] = fma(0.5 * ro3, fma(v3, v3, u3 * u3), kInvG1 * p3);
    un[3] = un[5] = un[6] = un[7] = 0.0;
    return rc;
}

// The primitive rows of a warp's 32 faces in shared memory: 64-byte rows of the two near cells 80 bytes
// apart, 48-byte rows (rho, u, v, w, p and one more) of the two far ones 48 apart, so eight lanes
// reading 16 bytes of their own rows hit different banks.  Every member is called by the whole warp.
struct FaceRows {
    static constexpr int kNear1 = 0, kNear2 = 32 * 80, kFar1 = 2 * 32 * 80, kFar2 = kFar1 + 32 * 48;
    static constexpr int kBytes = kFar2 + 32 * 48;
    unsigned char* base;
    int lane;
    __device__ __forceinline__ explicit FaceRows(unsigned char* b) : base(b), lane(threadIdx.x & 31) {}
    template <int NV> static __device__ __forceinline__ constexpr int pitch() { return NV == 8 ? 80 : 48; }
    // Starts the copies of cell `c` of every lane (c < 0: none), NV components each, four lanes a row.
    template <int NV> __device__ __forceinline__ void fetch(int at, const double* prim, int c) const {
        const int q = lane & 3;
#pragma unroll
        for (int r = 0; r < 32; r += 8) {
            const int f = r + (lane >> 2);
            const int64_t cell = __shfl_sync(0xffffffffu, c, f);
            const unsigned dst = (unsigned)__cvta_generic_to_shared(base + at + pitch<NV>() * f + 16 * q);
            if (cell >= 0 && 2 * q < NV)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(prim + 8 * cell + 2 * q)
                             : "memory");
        }
    }
    __device__ __forceinline__ void arrived() const {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }
    template <int NV> __device__ __forceinline__ void own(int at, double* q) const {
        const double2* p = reinterpret_cast<const double2*>(base + at + pitch<NV>() * lane);
#pragma unroll
        for (int v = 0; v < NV / 2; v++) {
            const double2 d = p[v];
            q[2 * v] = d.x;
            q[2 * v + 1] = d.y;
        }
    }
    // Flux rows of the warp's faces (lane's face gr), of those with `keep`.
    __device__ __forceinline__ void store_flux(double* flux, int64_t gr, const double* F, bool keep) const {
        const unsigned mask = __ballot_sync(0xffffffffu, keep);   // also: every lane has read its rows
        double2* own = reinterpret_cast<double2*>(base + kNear1 + 80 * lane);
#pragma unroll
        for (int v = 0; v < 4; v++) own[v] = make_double2(F[2 * v], F[2 * v + 1]);
        __syncwarp();
        const int q = lane & 3;
        double2* out = reinterpret_cast<double2*>(flux) + 4 * (gr - lane) + q;
#pragma unroll
        for (int r = 0; r < 32; r += 8) {
            const int f = r + (lane >> 2);
            if (mask >> f & 1u) out[4 * f] = *reinterpret_cast<const double2*>(base + kNear1 + 80 * f + 16 * q);
        }
    }
};

// One face per thread, cuf_solvers.cuf:243-440 (face speed 0).  Bound by the latency of its gathers
// and of dependent FP64 operations at 16 warps per SM (128 registers, no spills).  A face's four
// cells are one 16-byte index load; the solver is the Cartesian path's (riemann_fp64.cuh) on any
// tangents.  With the cell kernel below, a stage on a 96x80x64 box took 0.235 / 0.225 ms with the
// library-division solver on the reference's field-aligned basis, a primitive pass before every
// stage and three index arrays, 0.169 / 0.167 ms with each thread reading its own rows, and 0.138 /
// 0.144 ms so.
// The distance-weighted face value of cell 1, linear(-dff1, q11, -df1, q1, df2, q2) at 0
// (Solvers.f90:141-150), is q1 + minmod((q1 - q11) df1/(dff1 - df1), (q2 - q1) df1/(df1 + df2)): the
// weights are geometry, formed at set-up (geo = df1, df1/(df1 + df2), df1/(dff1 - df1),
// df2/(dff2 - df2); the second weight of side 2 is one minus that of side 1).
// The rows pass through shared memory, four lanes a row on the way in (cp.async) and out, as in
// sum_fluxes: a warp has all its 128 rows in flight at once, and the kernel was bound by the L1's
// throughput (70 %) when each thread read its own rows (96^3: 158 us, so 150 us; blocks of two warps instead of four, 148 us).
// FAST: n_disc is 0 (HLLC / HLLD by the FP64 solvers).  LAX: the grid may have Lax faces (physics 1).
template <int NSTATE, int ORDER, bool WANT_DT, bool FAST, bool LAX>
__global__ void __launch_bounds__(kFaceThreads, 8) fl_face_kernel(const FlView m, double cfl, int n_disc,
                                                               DevClock* clk, DevStatus* st) {
    __shared__ __align__(16) unsigned char rows[kFaceThreads / 32][FaceRows::kBytes];
    __shared__ double red[kFaceThreads / 32];
    __shared__ unsigned long long cnt[2];
    if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
    __syncthreads();
    const FaceRows fr(rows[threadIdx.x >> 5]);
    const int64_t gr = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double cand = kDtReset;
    unsigned n_recon = 0, n_wave = 0;
    allow_successor();
    const int64_t gc = gr < m.n_gran ? gr : m.n_gran - 1;   // geometry: no kernel writes it
    const int tword = gr < m.n_gran ? __ldg(m.type + gc) : 0;
    const int type = tword & 7;
    const int4 nb = __ldg(reinterpret_cast<const int4*>(m.nb) + gc);
    const double2* n2 = reinterpret_cast<const double2*>(m.normal + 4 * gc);
    const double2 na = __ldg(n2);
    const double n[3] = {na.x, na.y, __ldg(m.normal + 4 * gc + 2)};
    const double2* g2 = reinterpret_cast<const double2*>(m.geo + 4 * gc);
    const double2 ga = __ldg(g2);
    wait_for_predecessor();
    fr.fetch<8>(FaceRows::kNear1, m.prim, nb.x);
    fr.fetch<8>(FaceRows::kNear2, m.prim, nb.y);   // a ghost face: cell 1 again
    if (ORDER == 2) {
        fr.fetch<6>(FaceRows::kFar1, m.prim, nb.z);
        fr.fetch<6>(FaceRows::kFar2, m.prim, nb.w);
    }
    fr.arrived();
    double F[8] = {};
    if (type != 0) {
        double q1[8], q2[8];
        fr.own<8>(FaceRows::kNear1, q1);
        fr.own<8>(FaceRows::kNear2, q2);
        if (type == 4) {                          // :318-324 outer boundary
            if (q2[1] > -0.1) q2[1] = -0.1;
        } else if (type == 5) {                   // :325-329 axis
            q2[2] = -q2[2];
        } else if (type == 2) {                   // :330-345 reflecting wall
            const double vel = dadd(dadd(dmul(n[0], q1[1]), dmul(n[1], q1[2])), dmul(n[2], q1[3]));
#pragma unroll
            for (int a = 0; a < 3; a++) q2[1 + a] = dsub(dsub(q1[1 + a], dmul(vel, n[a])), dmul(vel, n[a]));
        } else if (ORDER == 2 && nb.z >= 0) {     // :358-412
            const double2 gb = __ldg(g2 + 1);
            double q11[6], q22[6];
            fr.own<6>(FaceRows::kFar1, q11);
            fr.own<6>(FaceRows::kFar2, q22);
            const double b1 = ga.y, b2 = 1.0 - ga.y;
            double t1[5], t2[5];
#pragma unroll
            for (int v = 0; v < 5; v++) {
                const double dq = q2[v] - q1[v];
                double h;
                const double m1 = slope((q1[v] - q11[v]) * gb.x, dq * b1, h);
                t1[v] = fma(h + h, m1, q1[v]);
                const double m2 = slope((q22[v] - q2[v]) * gb.y, dq * b2, h);
                t2[v] = fma(-(h + h), m2, q2[v]);
            }
            if (face_values_bad(t1[0], t1[4], t2[0], t2[4])) {
                fr.own<8>(FaceRows::kNear1, q1);   // type 2 and ghost faces are first order: the cells' own rows
                fr.own<8>(FaceRows::kNear2, q2);
#pragma unroll
                for (int v = 0; v < 5; v++) {
                    t1[v] = mend_face_value(v, t1[v], q1[v]);
                    t2[v] = mend_face_value(v, t2[v], q2[v]);
                }
            }
#pragma unroll
            for (int v = 0; v < 5; v++) {
                q1[v] = t1[v];
                q2[v] = t2[v];
            }
        }
        if (sb_neg(q1[0]) || sb_neg(q2[0])) n_recon++;
        if (m.powell) {   // :433 as commented there: 0.5 * n.(B1 + B2) * square, B of the chlld states
            const double nbs = dadd(dadd(dmul(n[0], dadd(q1[5], q2[5])), dmul(n[1], dadd(q1[6], q2[6]))),
                                    dmul(n[2], dadd(q1[7], q2[7])));
            m.divb[gr] = dmul(dmul(0.5 * kSpi4, nbs), __ldg(m.normal + 4 * gc + 3));
        }
        double SL, SR;
        bool none;
        auto reload = [&](double* m3) {
            asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(m3[0]), "=d"(m3[1]) : "l"(n2));
            asm volatile("ld.global.f64 %0, [%1];" : "=d"(m3[2]) : "l"(n2 + 1));
        };
        // the faces do not move (w = 0): no face-speed terms
        if (LAX && (tword & kLaxFace)) none = flux_normal_fp64<0, false>(n, reload, q1, q2, n_disc, F, SL, SR);   // :293-295
        else none = flux_normal_fp64<NSTATE, FAST>(n, reload, q1, q2, n_disc, F, SL, SR);
        if (none) {
            n_wave++;
#pragma unroll
            for (int v = 0; v < 8; v++) F[v] = 0.0;
        }
        const double sq = __ldg(m.normal + 4 * gc + 3);
#pragma unroll
        for (int v = 0; v < 8; v++) F[v] *= sq;
        // compare-and-select min / max (the library fmin / fmax of doubles are far longer sequences)
        if (WANT_DT) cand = sb_min(kDtFaceCap, cfl * ga.x * rs_rcp(sb_max(fabs(SL), fabs(SR))));
    }
    fr.store_flux(m.flux, gr, F, type != 0);   // a skipped face keeps its flux
    if (n_recon) atomicAdd(&cnt[0], (unsigned long long)n_recon);
    if (n_wave) atomicAdd(&cnt[1], (unsigned long long)n_wave);
    if (WANT_DT) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cand = sb_min(cand, __shfl_xor_sync(0xffffffffu, cand, o));
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = cand;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (WANT_DT) {
            double r = red[0];
#pragma unroll
            for (int w = 1; w < kFaceThreads / 32; w++) r = sb_min(r, red[w]);
            atomicMin(&clk->dt_next, (unsigned long long)__double_as_longlong(r));
        }
        if (cnt[0]) atomicAdd(&st->n_recon, cnt[0]);
        if (cnt[1]) atomicAdd(&st->n_wave, cnt[1]);
    }
}

// Owner-signed sums of the face fluxes of a warp's 32 cells (:691-703), each in the order of its face
// list: lane's cell in pot (and the div-B sum in sks).  Four lanes read one 64-byte flux row together
// (a thread reading its own rows 16 bytes at a time touches 32 rows an instruction and is bound by
// the L1's throughput: 96^3 cell update 98 us, so 79 us), eight rows an instruction, twelve
// instructions in flight; the sums pass through shared memory (`tile`, 32 x 10 doubles of the warp) to
// the lane that owns the cell.  A missing face reads the zero row.  All lanes take part.
template <bool POWELL>
__device__ __forceinline__ void sum_fluxes(const FlView& m, int64_t c, double* tile, double* pot, double& sks) {
    const int lane = threadIdx.x & 31, q = lane & 3, quad = lane >> 2;
    const int64_t cc = min(c, m.n_cell - 1);
    const int2* j2 = reinterpret_cast<const int2*>(m.cell_gran + 6 * cc);
    int j[6];
#pragma unroll
    for (int f = 0; f < 3; f++) {
        const int2 p = __ldg(j2 + f);
        j[2 * f] = p.x;
        j[2 * f + 1] = p.y;
    }
    const double2* flux = reinterpret_cast<const double2*>(m.flux) + q;
#pragma unroll
    for (int h = 0; h < 4; h += 2) {   // cells 8 h + quad, 8 (h + 1) + quad of the warp
        double2 d[2][6];
        int jc[2][6];
#pragma unroll
        for (int i = 0; i < 2; i++) {
#pragma unroll
            for (int f = 0; f < 6; f++) {
                const int x = __shfl_sync(0xffffffffu, j[f], 8 * (h + i) + quad);
                jc[i][f] = x;
                d[i][f] = flux[4 * (x ? (int64_t)abs(x) - 1 : m.n_gran)];
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++) {
            double2 t = make_double2(0.0, 0.0);
#pragma unroll
            for (int f = 0; f < 6; f++) {
                const double s = jc[i][f] < 0 ? -1.0 : 1.0;
                t.x = fma(s, d[i][f].x, t.x);
                t.y = fma(s, d[i][f].y, t.y);
            }
            *reinterpret_cast<double2*>(tile + 10 * (8 * (h + i) + quad) + 2 * q) = t;
        }
    }
    sks = 0.0;
    if (POWELL) {
#pragma unroll
        for (int f = 0; f < 6; f++) {
            const double db = m.divb[j[f] ? (int64_t)abs(j[f]) - 1 : m.n_gran];
            sks = j[f] < 0 ? sks - db : sks + db;
        }
    }
    __syncwarp();
    const double2* own = reinterpret_cast<const double2*>(tile + 10 * lane);
#pragma unroll
    for (int v = 0; v < 4; v++) {
        const double2 t = own[v];
        pot[2 * v] = t.x;
        pot[2 * v + 1] = t.y;
    }
}

// One cell per thread, cuf_solvers.cuf:561-794 as the conservative MHD update: flux sum, Euler / Heun
// stage (:705-770), negative-density check, p floor (:777-779), frozen cells (:611) and the re-imposed
// source sphere.  The new state's primitives go to m.prim where a next stage of the call reads them
// (`more`), so no pass of its own re-reads the state.  The last block of a finalizing launch rolls the
// clock.
// PHYS: the physics option; POWELL: the div-B terms are on (their energy term by m.powell ==
// 2).  Compile-time, so a launch carries only its own code (registers set the occupancy of this
// gather-bound kernel).
template <int KIND, int PHYS, bool POWELL>
__global__ void __launch_bounds__(kCellThreads) fl_cell_kernel(const FlView m, const double* Uin,
                                                               const double* Ubase, double* Uout, int64_t vs,
                                                               DevClock* clk, DevStatus* st, int finalize, int more) {
    __shared__ __align__(16) double tiles[kCellThreads / 32][320];
    __shared__ unsigned long long cnt[2];
    __shared__ bool last;
    if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    allow_successor();
    const int flag = c < m.n_cell ? __ldg(m.cell_flag + c) : 0;
    wait_for_predecessor();
    const double dt = clk->dt_cur;
    double pot[8], sks;
    sum_fluxes<POWELL>(m, c, tiles[threadIdx.x >> 5], pot, sks);
    if (c < m.n_cell) {
        double un[8], q[8];
        bool have_q = false;
        if (flag & kFrozen) {
#pragma unroll
            for (int v = 0; v < 8; v++) un[v] = KIND == 0 ? Uin[v * vs + c] : Ubase[v * vs + c];
        } else if (PHYS == 0 && (flag & kSource)) {
            const double x = m.cell_center[3 * c], y = m.cell_center[3 * c + 1], z = m.cell_center[3 * c + 2];
            source_state(m.src, x, y, z, dadd(dadd(dmul(x, x), dmul(y, y)), dmul(z, z)), q);
            cons_from_prim_exact(q, un);
        } else if (PHYS == 1) {
            load_prim(m.prim, c, q);
            const int rc = axisym_update<KIND>(Uin, Ubase, vs, c, q, pot, m.inv_volume[c], m.cell_center[3 * c],
                                               m.cell_center[3 * c + 1], m.hatom + 8 * c, dt, un);
            if (rc == 1) {
                atomicAdd(&cnt[0], 1ull);
                atomicMin(&st->first_bad, (unsigned long long)c);
            } else if (rc == 2) {
                atomicAdd(&cnt[1], 1ull);
            }
        } else {
            if (POWELL) {
                // div-B sources inside the flux sum (cuf_solvers.cuf:529-533 / 729-733, commented
                // there): momentum + (B/4pi) sks, B + u sks, powell 2 energy + (u.B/4pi) sks, with
                // u and B of the stage input (its primitive state); b = B / sqrt(4 pi), and the field
                // sums are in units of b
                load_prim(m.prim, c, q);
                const double sb = sks * kInvSpi4;
#pragma unroll
                for (int a = 0; a < 3; a++) {
                    pot[1 + a] = dadd(pot[1 + a], dmul(q[5 + a], sb));
                    pot[5 + a] = dadd(pot[5 + a], dmul(q[1 + a], sb));
                }
                if (m.powell == 2) {
                    const double ub = dadd(dadd(dmul(q[1], q[5]), dmul(q[2], q[6])), dmul(q[3], q[7]));
                    pot[4] = dadd(pot[4], dmul(ub, sb));
                }
            }
            const double ivol = m.inv_volume[c];
            const double ivb = ivol * kSpi4;   // field fluxes are in units of b
            double uin[8];
#pragma unroll
            for (int v = 0; v < 8; v++) {
                uin[v] = Uin[v * vs + c];
                const double d = pot[v] * (v < 5 ? ivol : ivb);
                if (KIND == 0) un[v] = uin[v] - dt * d;
                else un[v] = 0.5 * ((Ubase[v * vs + c] + uin[v]) - dt * d);
            }
            if (!(un[0] > 0.0)) {
                atomicAdd(&cnt[0], 1ull);
                atomicMin(&st->first_bad, (unsigned long long)c);
#pragma unroll
                for (int v = 0; v < 8; v++) un[v] = uin[v];
            } else {
                double ke, me;
                prim_from_cons<true, true>(un, q, ke, me);
                have_q = true;
                if (q[4] <= 0.0) {
                    atomicAdd(&cnt[1], 1ull);
                    un[4] = floor_energy(ke, me);
                    have_q = false;
                }
            }
        }
#pragma unroll
        for (int v = 0; v < 8; v++) Uout[v * vs + c] = un[v];
        if (more) {
            if (!have_q) {
                double ke, me;
                prim_from_cons<true, true>(un, q, ke, me);
            }
            store_prim(m.prim, c, q);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (cnt[0]) atomicAdd(&st->n_negdens, cnt[0]);
        if (cnt[1]) atomicAdd(&st->n_pfloor, cnt[1]);
        __threadfence();
        last = atomicAdd(&clk->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        clk->counter = 0;
        if (finalize) {
            const unsigned long long nb = atomicExch(&clk->dt_next, (unsigned long long)__double_as_longlong(kDtReset));
            clk->time_all += clk->dt_cur;
            clk->dt_last = clk->dt_cur;
            clk->dt_cur = __longlong_as_double((long long)nb);
            clk->steps += 1;
        }
        __threadfence();
    }
}

template <int NSTATE, int ORDER, bool WANT_DT>
void launch_face_o(const FlView& m, bool lax, double cfl, int n_disc, DevClock* clk, DevStatus* st, cudaStream_t s) {
    const unsigned grid = (unsigned)((m.n_gran + kFaceThreads - 1) / kFaceThreads);
#define SB_FACE(F, L) \
    launch_chained(fl_face_kernel<NSTATE, ORDER, WANT_DT, F, L>, grid, kFaceThreads, 0, s, m, cfl, n_disc, clk, st)
    if constexpr (NSTATE >= 2) {
        if (n_disc == 0) {
            if (lax) SB_FACE(true, true);
            else SB_FACE(true, false);
            return;
        }
    }
    SB_FACE(false, true);
#undef SB_FACE
}

template <int NSTATE>
void launch_face_n(const FlView& m, bool lax, int order, bool want_dt, double cfl, int n_disc, DevClock* clk,
                   DevStatus* st, cudaStream_t s) {
    if (order == 2) {
        if (want_dt) launch_face_o<NSTATE, 2, true>(m, lax, cfl, n_disc, clk, st, s);
        else launch_face_o<NSTATE, 2, false>(m, lax, cfl, n_disc, clk, st, s);
    } else {
        if (want_dt) launch_face_o<NSTATE, 1, true>(m, lax, cfl, n_disc, clk, st, s);
        else launch_face_o<NSTATE, 1, false>(m, lax, cfl, n_disc, clk, st, s);
    }
}

}  // namespace

// ------------------------------------------------------------------------------ host side
void fl_destroy(FaceListDev* f) {
    if (!f) return;
    const FlView& m = f->v;
    void* ptrs[] = {m.cell_center, m.inv_volume, m.cell_gran, m.cell_flag, m.normal, m.geo, m.nb,
                    m.type,        m.prim,       m.flux,      m.hatom,     m.divb};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    delete f;
}

// Host-side check that every index the kernels follow stays inside its array: cell faces in
// 0..G, neighbours in 1..N (neighbour 2 may be -1 only on a ghost face: type 4, 5, or a type-2
// wall), TVD cells in 1..N or -1, face types 1..5, volumes positive.
int fl_validate(int64_t N, int64_t G, const double* cell_center, const double* cell_volume, const int32_t* cell_gran,
                const double* gran_normal, const double* gran_square, const double* gran_center,
                const int32_t* gran_neighbour, const int32_t* gran_neighbour_tvd, const int32_t* gran_type) {
    if (N < 1 || G < 1 || !cell_center || !cell_volume || !cell_gran || !gran_normal || !gran_square || !gran_center ||
        !gran_neighbour || !gran_neighbour_tvd || !gran_type)
        return SETB_EINVAL;
    if (N > INT32_MAX - 1 || G > INT32_MAX - 1) return SETB_ESIZE;
    for (int64_t c = 0; c < N; c++) {
        if (!(cell_volume[c] > 0.0)) return SETB_EINVAL;
        for (int f = 0; f < 6; f++) {
            const int32_t j = cell_gran[6 * c + f];
            if (j < 0 || j > G) return SETB_EINVAL;
        }
    }
    for (int64_t g = 0; g < G; g++) {
        const int32_t s1 = gran_neighbour[2 * g], s2 = gran_neighbour[2 * g + 1], t = gran_type[g];
        const int32_t ss1 = gran_neighbour_tvd[2 * g], ss2 = gran_neighbour_tvd[2 * g + 1];
        if (s1 < 1 || s1 > N || t < 1 || t > 5) return SETB_EINVAL;
        const bool ghost = t == 4 || t == 5 || (t == 2 && s2 == -1);
        if (!ghost && (s2 < 1 || s2 > N)) return SETB_EINVAL;
        if ((ss1 != -1 && (ss1 < 1 || ss1 > N)) || (ss2 != -1 && (ss2 < 1 || ss2 > N))) return SETB_EINVAL;
    }
    return SETB_OK;
}

namespace {
// 21-bit spread for a 63-bit Morton code
uint64_t spread3(uint64_t x) {
    x &= 0x1fffffull;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}
}  // namespace

int fl_create(FaceListDev** out, int64_t N, int64_t G, const double* cell_center_in, const double* cell_volume_in,
              const int32_t* cell_gran_in, const double* gran_normal_in, const double* gran_square_in,
              const double* gran_center_in, const int32_t* gran_neighbour_in, const int32_t* gran_neighbour_tvd_in,
              const int32_t* gran_type_in, const setb_fl_params* p, cudaStream_t s) {
    *out = nullptr;
    if (!p) return SETB_EINVAL;
    int rc = fl_validate(N, G, cell_center_in, cell_volume_in, cell_gran_in, gran_normal_in, gran_square_in,
                         gran_center_in, gran_neighbour_in, gran_neighbour_tvd_in, gran_type_in);
    if (rc) return rc;
    // Locality order: cells along the Morton curve of their centres, faces by their first cell, so
    // the cells a face gathers and the faces a cell gathers sit close in memory whatever the
    // caller's numbering (ties by the caller's order).  cperm[d] = caller's cell of device cell d; fperm
    // likewise for faces, which are counted into place: sorts that compare through the caller's random
    // numbering were half of the set-up.
    std::vector<int32_t> cperm((size_t)N), fperm((size_t)G), cnew((size_t)N), fnew((size_t)G);
    {
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int64_t c = 0; c < N; c++)
            for (int a = 0; a < 3; a++) {
                lo[a] = std::min(lo[a], cell_center_in[3 * c + a]);
                hi[a] = std::max(hi[a], cell_center_in[3 * c + a]);
            }
        std::vector<std::pair<uint64_t, int32_t>> key((size_t)N);
        for (int64_t c = 0; c < N; c++) {
            uint64_t code = 0;
            for (int a = 0; a < 3; a++) {
                const double span = hi[a] > lo[a] ? hi[a] - lo[a] : 1.0;
                const double u = (cell_center_in[3 * c + a] - lo[a]) / span;
                code |= spread3((uint64_t)std::min(2097151.0, std::max(0.0, u * 2097151.0))) << a;
            }
            key[c] = {code, (int32_t)c};
        }
        std::sort(key.begin(), key.end());
        for (int64_t d = 0; d < N; d++) {
            cperm[d] = key[d].second;
            cnew[cperm[d]] = (int32_t)d;
        }
        std::vector<int32_t> at((size_t)N + 1, 0);   // first face of each cell, then its next free place
        for (int64_t g = 0; g < G; g++) at[cnew[gran_neighbour_in[2 * g] - 1] + 1]++;
        for (int64_t d = 0; d < N; d++) at[d + 1] += at[d];
        for (int64_t g = 0; g < G; g++) {
            fnew[g] = at[cnew[gran_neighbour_in[2 * g] - 1]]++;
            fperm[fnew[g]] = (int32_t)g;
        }
    }
    // Cells, then faces, then the cells' face lists: what a face needs of its cells, and a cell of its
    // faces, is read from the arrays already in locality order (a renumbered 96x80x64 box: this function
    // on the host 390 ms; 760 with every array read through the caller's numbering and the sorts above by
    // comparison, 690 with such sorts alone).
    auto cell_ref = [&](int32_t c1) { return cnew[c1 - 1]; };   // caller's 1-based -> device 0-based
    std::vector<double> cell_center((size_t)N * 3), inv_volume((size_t)N), geo((size_t)G * 4), normal4((size_t)G * 4);
    std::vector<int32_t> cell_gran((size_t)N * 6), type((size_t)G), nb((size_t)G * 4);
    std::vector<unsigned char> flag((size_t)N);
    for (int64_t d = 0; d < N; d++) {
        const int64_t c = cperm[d];
        const double* x = cell_center_in + 3 * c;
        for (int a = 0; a < 3; a++) cell_center[3 * d + a] = x[a];
        const double r2 = (x[0] * x[0] + x[1] * x[1]) + x[2] * x[2];
        flag[d] = ((p->cell_freeze_radius > 0.0 && norm3(x) < p->cell_freeze_radius) ? kFrozen : 0) |
                  ((p->r_src > 0.0 && r2 < p->r_src * p->r_src) ? kSource : 0);
        inv_volume[d] = 1.0 / cell_volume_in[c];
    }
    for (int64_t d = 0; d < G; d++) {
        const int64_t g = fperm[d];
        const int32_t s1 = gran_neighbour_in[2 * g], s2 = gran_neighbour_in[2 * g + 1], t = gran_type_in[g];
        const int32_t ss1 = gran_neighbour_tvd_in[2 * g], ss2 = gran_neighbour_tvd_in[2 * g + 1];
        const bool ghost = t == 4 || t == 5 || (t == 2 && s2 == -1);
        const bool tvd = !ghost && ss1 >= 1 && ss2 >= 1;
        int32_t* cells = nb.data() + 4 * d;
        cells[0] = cell_ref(s1);
        cells[1] = ghost ? cells[0] : cell_ref(s2);
        cells[2] = tvd ? cell_ref(ss1) : -1;
        cells[3] = tvd ? cell_ref(ss2) : -1;
        // distances as the reference forms them each step (cuf_solvers.cuf:290-292, 362-372)
        const double* gc = gran_center_in + 3 * g;
        auto distance = [&](int32_t c) {
            const double* x = cell_center.data() + 3 * (int64_t)c;
            const double r[3] = {gc[0] - x[0], gc[1] - x[1], gc[2] - x[2]};
            return norm3(r);
        };
        const double df1 = distance(cells[0]);
        geo[4 * d] = df1;
        if (tvd) {
            const double df2 = distance(cells[1]), dff1 = distance(cells[2]), dff2 = distance(cells[3]);
            geo[4 * d + 1] = df1 / (df1 + df2);
            geo[4 * d + 2] = df1 / (dff1 - df1);
            geo[4 * d + 3] = df2 / (dff2 - df2);
        }
        const double* n = gran_normal_in + 3 * g;
        for (int a = 0; a < 3; a++) normal4[4 * d + a] = n[a];
        normal4[4 * d + 3] = gran_square_in[g];
        // the reference skips faces whose first cell lies inside its frozen core (:284)
        const double* c1 = cell_center.data() + 3 * (int64_t)cells[0];
        type[d] = (p->face_skip_radius > 0.0 && norm3(c1) < p->face_skip_radius) ? 0 : (t == 2 && !ghost ? kInner : t);
        // physics 1: the reference's Lax flux on faces near the axis (cuf_solvers.cuf:293-295)
        if (type[d] && p->physics == 1 && gc[0] > (double)0.22f && gc[1] < (double)0.1f &&
            std::fabs(n[0]) < (double)0.1f)
            type[d] |= kLaxFace;
    }
    for (int64_t d = 0; d < N; d++)
        for (int f = 0; f < 6; f++) {   // the face, positive where this cell is its first neighbour
            const int32_t j = cell_gran_in[6 * (int64_t)cperm[d] + f];
            if (j < 1) continue;
            const int32_t jd = fnew[j - 1];
            cell_gran[6 * d + f] = nb[4 * (int64_t)jd] == (int32_t)d ? jd + 1 : -(jd + 1);
        }

    FaceListDev* f = new (std::nothrow) FaceListDev();
    if (!f) return SETB_ENOMEM;
    FlView& m = f->v;
    m.n_cell = N;
    m.n_gran = G;
    m.src.r_src = p->r_src;
    m.src.rho_src = p->rho_src;
    m.src.v_src = p->v_src;
    m.src.p_over_rho_src = p->p_over_rho_src;
    m.src.r_floor = p->r_floor;
    m.powell = p->powell;
    f->perm = cperm;
    f->physics = p->physics;
    const size_t rows = (size_t)G + 1;
    bool ok = upload(&m.cell_center, cell_center.data(), 3 * (size_t)N, s) == cudaSuccess &&
              upload(&m.inv_volume, inv_volume.data(), (size_t)N, s) == cudaSuccess &&
              upload(&m.cell_gran, cell_gran.data(), 6 * (size_t)N, s) == cudaSuccess &&
              upload(&m.cell_flag, flag.data(), (size_t)N, s) == cudaSuccess &&
              upload(&m.normal, normal4.data(), 4 * (size_t)G, s) == cudaSuccess &&
              upload(&m.geo, geo.data(), 4 * (size_t)G, s) == cudaSuccess &&
              upload(&m.nb, nb.data(), 4 * (size_t)G, s) == cudaSuccess &&
              upload(&m.type, type.data(), (size_t)G, s) == cudaSuccess &&
              cudaMalloc(&m.prim, sizeof(double) * 8 * (size_t)N) == cudaSuccess &&
              cudaMalloc(&m.flux, sizeof(double) * 8 * rows) == cudaSuccess &&
              (p->physics != 1 || cudaMalloc(&m.hatom, sizeof(double) * 8 * (size_t)N) == cudaSuccess) &&
              cudaMemsetAsync(m.flux, 0, sizeof(double) * 8 * rows, s) == cudaSuccess &&
              (p->powell == 0 || (cudaMalloc(&m.divb, sizeof(double) * rows) == cudaSuccess &&
                                  cudaMemsetAsync(m.divb, 0, sizeof(double) * rows, s) == cudaSuccess)) &&
              cudaStreamSynchronize(s) == cudaSuccess;   // host vectors are released on return
    if (!ok) {
        cudaGetLastError();
        fl_destroy(f);
        return SETB_ENOMEM;
    }
    *out = f;
    return SETB_OK;
}

cudaError_t fl_launch_stage(const FaceListDev* f, const double* Uin, const double* Ubase, double* Uout, int64_t vs,
                            DevClock* clk, DevStatus* st, const setb_step_opts* o, int kind, bool want_dt,
                            bool finalize, bool first, bool more, cudaStream_t s) {
    const FlView& m = f->v;
    if (first) {
        const unsigned pgrid = (unsigned)std::min<int64_t>((m.n_cell + kPrimThreads - 1) / kPrimThreads, 148 * 16);
        launch_chained(fl_prim_kernel, pgrid, kPrimThreads, 0, s, m.n_cell, Uin, vs, m.prim);
    }
    switch (o->n_state) {
        case 0: launch_face_n<0>(m, f->physics == 1, o->order, want_dt, o->cfl, o->n_disc, clk, st, s); break;
        case 1: launch_face_n<1>(m, f->physics == 1, o->order, want_dt, o->cfl, o->n_disc, clk, st, s); break;
        case 2: launch_face_n<2>(m, f->physics == 1, o->order, want_dt, o->cfl, o->n_disc, clk, st, s); break;
        default: launch_face_n<3>(m, f->physics == 1, o->order, want_dt, o->cfl, o->n_disc, clk, st, s); break;
    }
    const unsigned cgrid = (unsigned)((m.n_cell + kCellThreads - 1) / kCellThreads);
#define SB_CELL(K, PH, PW) \
    launch_chained(fl_cell_kernel<K, PH, PW>, cgrid, kCellThreads, 0, s, m, Uin, Ubase, Uout, vs, clk, st, finalize, more)
    if (f->physics == 1) {
        if (kind == 0) SB_CELL(0, 1, false);
        else SB_CELL(1, 1, false);
    } else if (m.powell) {
        if (kind == 0) SB_CELL(0, 0, true);
        else SB_CELL(1, 0, true);
    } else {
        if (kind == 0) SB_CELL(0, 0, false);
        else SB_CELL(1, 0, false);
    }
#undef SB_CELL
    return cudaGetLastError();
}

}  // namespace sb

namespace sb {
const int32_t* fl_perm(const FaceListDev* f) { return f ? f->perm.data() : nullptr; }
}  // namespace sb

namespace sb {
// Uploads the H-atom fluids (Cell_par columns 9..16, caller numbering) of a physics-1 face list.
int fl_set_hatom(FaceListDev* f, const double* cell_par, cudaStream_t s) {
    if (!f || !f->v.hatom) return SETB_OK;
    if (copy_rows_to_device(f->v.hatom, cell_par + 8, 16 * sizeof(double), 8 * sizeof(double), (size_t)f->v.n_cell,
                            f->perm.data(), s) != cudaSuccess)
        return SETB_ECUDA;
    return SETB_OK;
}
}  // namespace sb
