// Explicit right-hand side of the RK3 substep and the wall ghost refresh.
//
// k_ghosts:  apply_bc_u{2,4} / apply_bc_w{2,4} of chanfast.c:404-418 for
//            every column, plus the in-place wall rewrite that
//            massflux{x,y,z}4 performs before the advection (advect.c:100-131).
// k_rhs:     fused massflux{x,y,z} + advect{u,v,w} + add_laplacexy_operator
//            + flux_quick + advect_scalar + add_buoyancy
//            (chanfast.c:420-452 / 1344-1376) for every interior point; mass
//            fluxes are formed on the fly and never stored.  Expressions keep
//            the reference's evaluation order; this file is compiled with FMA
//            contraction (its kernels are FP64-throughput bound), so results
//            agree with the reference to rounding.
#include "engine.cuh"
#include "host_band.h"
#include "wall.cuh"
#include "batch.cuh"
#include "rounding.cuh"

#include <algorithm>
#include <type_traits>

namespace cf {

// ------------------------------------------------------------------ ghosts

// One thread per column and field (blockIdx.y: 0 u, 1 v, 2 c, 3 w): wall ghost
// rows of u, v, c (apply_bc_u) and w (apply_bc_w, then with EXTRAP the
// massflux4 extrapolation of advect.c:100-131).  Bound: latency, of one
// column's few dependent reads and divisions; a thread per column doing the
// four fields one after another took 8 us at 64 x 64 x 64, this 6.7.
template <int ORDER, bool EXTRAP>
__device__ __forceinline__ void ghosts_body(const Geo& G, const GhostArgs& A, uint3 bid)
{
    long long col = (long long) bid.x * blockDim.x + threadIdx.x;
    if (col >= G.plane) return;
    const long long P = G.plane;
    const int n2 = G.n2, kb = GZ - 1, kt = n2 - GZ, q = bid.y;
    if (q < 3) {
        double* f = (q == 0 ? A.F.u : q == 1 ? A.F.v : A.F.c) + col;
        auto at = [&](int k) -> double& { return f[k * P]; };
        const double bcb = q == 0 ? A.bc_u : q == 1 ? A.bc_v : A.bc_c_bot;
        const double bct = q == 0 ? A.bc_u : q == 1 ? A.bc_v : A.bc_c_top;
        double b1, b2, b3, t1, t2, t3;
        bc_u_bot<ORDER>(A.ub, bcb, at(kb + 1), at(kb + 2), at(kb + 3), b1, b2, b3);
        bc_u_top<ORDER>(A.ut, bct, at(kt - 1), at(kt - 2), at(kt - 3), t1, t2, t3);
        at(kb) = b1;
        at(kt) = t1;
        if (ORDER == 4) {
            at(kb - 1) = b2;
            at(kb - 2) = b3;
            at(kt + 1) = t2;
            at(kt + 2) = t3;
        }
        return;
    }
    double* w = A.F.w + col;
    auto at = [&](int k) -> double& { return w[k * P]; };
    const int wt = n2 - GZ - 1;
    const double x0 = at(kb + 1), x1 = at(kb + 2), y0 = at(wt - 1), y1 = at(wt - 2);
    double b1, b2, b3, t1, t2, t3;
    bc_w_bot<ORDER>(A.wb, A.bc_w, x0, x1, b1, b2, b3);
    bc_w_top<ORDER>(A.wt, A.bc_w, y0, y1, t1, t2, t3);
    at(kb) = b1;
    at(wt) = t1;
    if (ORDER == 4) {
        // EXTRAP: massflux4 wall extrapolation (advect.c:108-109, 124-125)
        at(kb - 1) = EXTRAP ? mad(2.0, b1, -x0) : b2;
        at(kb - 2) = EXTRAP ? mad(2.0, b1, -x1) : b3;
        at(wt + 1) = EXTRAP ? mad(2.0, t1, -y0) : t2;
        at(wt + 2) = EXTRAP ? mad(2.0, t1, -y1) : t3;
    }
}

template <int ORDER, bool EXTRAP>
__global__ void k_ghosts(Geo G, GhostArgs A)
{
    ghosts_body<ORDER, EXTRAP>(G, A, blockIdx);
}

template <int ORDER, bool EXTRAP>
__global__ void k_ghosts_batch(const BatchRec<GhostArgs>* r, int n)
{
    uint3 b;
    const BatchRec<GhostArgs>& R = batch_locate(r, n, b);
    ghosts_body<ORDER, EXTRAP>(R.G, R.A, b);
}

// --------------------------------------------------------------------- RHS
//
// One block owns an 8 (x) by 32 (y) column tile and marches up A.chunk rows.
// Sixteen warps: four for each of u, v, w, c, a thread taking two
// neighbouring points in y of its field.  A thread keeps its own column's next
// values, the z fluxes carried up the column and the forward sweep; its
// field's plane k with a periodic halo of 3 rows in x and 4 columns in y comes
// from a ring of shared-memory planes, filled by cp.async one plane ahead, two
// values per load.
//
// What one field's equation needs of another's are velocities interpolated
// to its faces.  Each is formed once, by the thread that holds the values it
// interpolates, and handed over through shared memory:
//   u threads: u interpolated in y (for v's x flux) and in z (for w's)
//   v threads: v interpolated in x (for u's y flux) and in z (for w's)
//   w threads: w interpolated in x and y one row up (u's and v's z flux)
// The faces of the tile's rim that no thread of the tile holds are formed by
// the scalar's threads.  A row is: own differences and faces; a barrier; the
// fluxes with the others' faces.  The face buffers alternate, so that one
// block-wide barrier per row is enough.
//
// Bound: instruction issue and shared-memory bandwidth (order 4, ncu at
// 256 x 256 x 192: LSU wavefronts 70 %, FP64 42 %, issue 52 %).  One thread
// per point doing all four equations (256 threads, 253 registers) formed each
// interpolated velocity four times and had two warps per scheduler to hide
// latency with.  us, before and now: order 4 512 x 512 x 384 5161 -> 4174,
// 256 x 256 x 192 748 -> 621, 128 x 128 x 96 (row blocks) 99 -> 89; order 2
// 256 x 256 x 192 507 -> 480, 128 x 128 x 96 (row blocks) 66.
// The four equations' loops have to fit the SM's instruction cache together
// (about 27 KB at order 4): with two rows of points a thread, fewer
// instructions but 42 KB of code, the warps waited for instructions (1105 us at
// 256 x 256 x 192), and so they did with a test for odd ny and the wall
// closures inside the loop (850).  Hence EVEN is a template parameter, the
// interior rows have a loop of their own, and a scheduler's four warps all
// work on the same field.
//
// Divisions by the grid metrics are multiplications by their reciprocals (host
// tables), the 0.5 of a face average is folded into the interpolation weights
// and a direction's metric is factored out of its flux sum, so results agree
// with the reference to rounding, not bit for bit.  Which product of a sum is
// fused is written down (rounding.cuh): the same flow in another instantiation
// of the body, or in other row blocks, gives the same bits.
//
// After a row's explicit right-hand side the thread forms the right-hand side
// h of its implicit solve (chanfast.c:459-480), which overwrites g.
// MODE RHS_SWEEP: and runs the solve's forward sweep, leaving s (the back
//   sweep follows in k_line); the block takes the whole column.
// MODE RHS_H: leaves h (both sweeps follow in k_line, partitioned).
// MODE RHS_CHANNEL (the fully implicit scheme of channel.c): f has no x-y
//   diffusion (channel.c:419-438) and h = x + nuadt (Lxy + Lz) x + gamdt f +
//   zetdt g - hbc (channel.c:455-467, 531-543, 560-572, 636-648); A.nu and
//   A.kappa then carry nuadt and nuadt / prandtl.  The spectral solves follow
//   (kernels_pressure.cu).

constexpr int RT_I = 8, RT_J = 32;
constexpr int RT_FIELD = RT_I * RT_J / 2;   // threads of one field
constexpr int RT_THREADS = 4 * RT_FIELD;
enum RhsMode { RHS_SWEEP, RHS_H, RHS_CHANNEL };

// Ring geometry per order: the x-y halo of the stencils (order 4: 3, the
// fourth-order fluxes and Laplacian; order 2: 2, the QUICK scalar fluxes),
// and a ring holding the ZH planes below and above a row and the one in
// flight.  The y halo is rounded up to an even width (XL) so that, for even
// ny, every haloed row segment starts on a 16-byte boundary in global and
// shared memory.
template <int ORDER>
struct RhsTile {
    static constexpr int H = ORDER == 2 ? 2 : 3;
    static constexpr int ZH = H;
    static constexpr int XL = (H + 1) & ~1;                      // y halo columns: 4 / 2
    static constexpr int SLOTS = 2 * ZH + 2;
    static constexpr int PI = RT_I + 2 * H, PJ = RT_J + 2 * XL;  // 14 x 40 / 12 x 36
    static constexpr int PLANE = PI * PJ;
    static constexpr int FIELD = SLOTS * PLANE;                  // one field's ring
    // plane kk >= 0 (every plane a row reads lies in 0 .. n2-1): an unsigned
    // remainder, a single AND for the 8-slot ring
    __host__ __device__ static constexpr int slot(int kk) { return (int) ((unsigned) kk % (unsigned) SLOTS); }
};
constexpr double B1h = 0.5 * B1, B2h = 0.5 * B2;   // halved interpolation weights (exact)
// 7-point form of the fourth-order staggered second difference:
// A1 (d+1/2 - d-1/2) + A2 (d+3/2 - d-3/2) = L1 (F1+F-1-2F0) + L2 (F2+F-2-2F0) + L3 (F3+F-3-2F0),
// evaluated as L1 (F1+F-1) + L2 (F2+F-2) + L3 (F3+F-3) - 2 (L1+L2+L3) F0.  Mathematically the
// same; the centre term no longer cancels exactly, an error of a few ulps of |u| (1/dx^2 + 1/dy^2) nu.
constexpr double L1 = A1 * A1 - 2.0 * A1 * A2, L2 = 2.0 * A1 * A2, L3 = A2 * A2;

constexpr int RT_FWMAX = 14;  // widest fused row (order 4: 13), padded to 16-byte pairs
// per-row grid metrics: dydz[k-1..k+2], dxdz[k-1..k+2], ivol[k], ivolw[k], and with RCS a field's scalars
template <bool RCS>
constexpr int RT_MROW = RCS ? 16 : 12;
constexpr int RM_DXDY = 10, RM_DIFF = 11, RM_SHIFT = 12, RM_IDX2 = 13, RM_IDY2 = 14;
// face buffers: u's with rows i0-2 .. i0+8, v's with columns j0-2 .. j0+33, w's on the tile
constexpr int RF_U = (RT_I + 3) * RT_J, RF_V = RT_I * (RT_J + 4), RF_W = RT_I * RT_J;
constexpr int RF_UY = 0, RF_UZ = RF_U, RF_VX = 2 * RF_U, RF_VZ = 2 * RF_U + RF_V, RF_WX = 2 * RF_U + 2 * RF_V,
              RF_WY = RF_WX + RF_W, RF_ALL = RF_WY + RF_W;
// ring of haloed planes + two rows of faces + per field two rows of its fused
// coefficients and of the grid metrics + plane offsets of the copies
template <int ORDER>
__host__ __device__ constexpr int rhs_faces() { return 4 * RhsTile<ORDER>::FIELD; }
template <int ORDER>
__host__ __device__ constexpr int rhs_rows() { return rhs_faces<ORDER>() + 2 * RF_ALL; }
template <int ORDER, bool RCS>
__host__ __device__ constexpr int rhs_queue() { return rhs_rows<ORDER>() + 4 * 2 * (RT_FWMAX + RT_MROW<RCS>); }
template <int ORDER, bool RCS>
__host__ __device__ constexpr int rhs_offs() { return rhs_queue<ORDER, RCS>() + (ORDER == 4 ? 4 * 2 * RT_THREADS : 0); }
template <int ORDER, bool RCS = false>
constexpr size_t rhs_smem_bytes()
{
    return (size_t) rhs_offs<ORDER, RCS>() * sizeof(double) + RhsTile<ORDER>::PLANE * sizeof(int);
}

extern __shared__ __align__(16) double rhs_sm[];

__device__ __forceinline__ void cp_async8(double* dst, const double* src)
{
    unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(double* dst, const double* src)   // L2 only
{
    unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// pairs of points
__device__ __forceinline__ double2 ld2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ void st2(double* p, double2 v) { *reinterpret_cast<double2*>(p) = v; }

// Halved interpolation to the face between a0 and a1 (massflux{x,y,z}{2,4},
// advect.c:6-283, with the 0.5 of the advected face value).
template <int ORDER>
__device__ __forceinline__ double2 face(double2 am, double2 a0, double2 a1, double2 a2)
{
    if (ORDER == 2) return 0.25 * (a0 + a1);
    return B1h * (a0 + a1) + B2h * (am + a2);
}

// Flux difference over a cell (advect{u,v,w}{2,4}, advect.c:286-734) from the
// halved face velocities m[-2..1] and the advected values q[-3..3].
template <int ORDER>
__device__ __forceinline__ double2 flux(double2 mm2, double2 mm1, double2 m0, double2 m1, double2 qm3, double2 qm1,
                                        double2 q0, double2 q1, double2 q3)
{
    const double2 d = m0 * (q0 + q1) - mm1 * (q0 + qm1);
    if (ORDER == 2) return d;
    return A1 * d + A2 * (m1 * (q0 + q3) - mm2 * (q0 + qm3));
}

struct RhsBlock {
    int i0, j0, kb, ke, q, ty, jl;   // tile, rows, thread of the field, its row and first column
    bool v0, v1;                     // this thread's points lie in the plane
    long long plane, gij;            // gij: plane offset of the first point
};

// The march of field F's threads: 0 u, 1 v, 2 w, 3 c.  RCS: the scalars that
// every row needs wait behind its metrics in shared memory instead of in
// registers or the constant bank (k_rhs_batch).
template <int ORDER, int MODE, int F, bool EVEN, bool RCS>
__device__ __forceinline__ void rhs_field(const Geo& G, const RhsArgs& A, const RhsBlock& T)
{
    using RT = RhsTile<ORDER>;
    constexpr int PJ = RT::PJ, NZ = ORDER == 2 ? 2 : 3, HH = ORDER == 2 ? 1 : 3;   // z reach of the window, of the solve
    constexpr int FWR = 2 * HH + 7;                               // fused row: cu[-HH..HH], cf, cg, c0, f1, f2, f3
    const int n2 = G.n2, top = n2 - GZ - 1;                       // last interior row
    const double* __restrict__ src = F == 0 ? A.u : F == 1 ? A.v : F == 2 ? A.w : A.c;
    double* __restrict__ fout = (F == 0 ? A.fu : F == 1 ? A.fv : F == 2 ? A.fw : A.fc) + T.gij + T.kb * T.plane;   // row k
    double* gio = A.sw[F].g + T.gij + T.kb * T.plane;                                                             // row k
    double* const mine = rhs_sm + F * RT::FIELD;
    const int* const goff = reinterpret_cast<const int*>(rhs_sm + rhs_offs<ORDER, RCS>());   // plane offsets of the copies
    const int at = (T.ty + RT::H) * PJ + T.jl + RT::XL;           // own point within a plane
    const double2 z2 = make_double2(0.0, 0.0);

    // ---- copies: this field's planes, coefficients and metrics
    const double* b = src + (T.kb - RT::ZH) * T.plane;   // the next plane to copy
    auto load_plane = [&](int kk) {
        double* d = mine + RT::slot(kk) * RT::PLANE;
        if (EVEN) {   // pairs
#pragma unroll
            for (int e = 0; e < RT::PLANE / 2; e += RT_FIELD)
                if (e + RT_FIELD <= RT::PLANE / 2 || e + T.q < RT::PLANE / 2)
                    cp_async16(d + 2 * (e + T.q), b + goff[e + T.q]);
        } else {
#pragma unroll
            for (int e = 0; e < RT::PLANE; e += RT_FIELD)
                if (e + RT_FIELD <= RT::PLANE || e + T.q < RT::PLANE) cp_async8(d + e + T.q, b + goff[e + T.q]);
        }
        b += T.plane;
    };
    double* const cst = rhs_sm + rhs_rows<ORDER>() + F * 2 * (RT_FWMAX + RT_MROW<RCS>);   // [2][RT_FWMAX] fused coefficients
    double* const mst = cst + 2 * RT_FWMAX;                      // [2][RT_MROW<RCS>] grid metrics
    // thread e copies value e of a row: its coefficients, then the metrics
    // (rows kk-1 .. kk+2 lie within 0 .. n2-1)
    const double* xsrc = nullptr;
    int xstep = 0, xdst = 0;
    if (T.q < FWR) {
        xsrc = A.sw[F].rows + (T.kb - GZ) * FWR + T.q;
        xstep = FWR;
        xdst = T.q;
    } else if (T.q >= 32 && T.q < 42) {
        const int m = T.q - 32;
        xsrc = m < 4 ? G.dydz + T.kb - 1 + m : m < 8 ? G.dxdz + T.kb - 5 + m : m == 8 ? G.ivol + T.kb : G.ivolw + T.kb;
        xstep = 1;
        xdst = 2 * RT_FWMAX + m;
    }
    const int xodd = T.q < FWR ? RT_FWMAX : RT_MROW<RCS>;
    auto load_extras = [&](int kk) {   // (the w solve has nz - 1 rows)
        if (xsrc && !(F == 2 && T.q < FWR && kk >= top)) cp_async8(cst + xdst + (kk & 1) * xodd, xsrc);
        xsrc = xsrc ? xsrc + xstep : xsrc;
    };
    auto load_g = [&](int kk, const double* p) {
        if (F == 2 && kk >= top) return z2;
        if (EVEN) return T.v0 ? ld2(p) : z2;
        return make_double2(T.v0 ? p[0] : 0.0, T.v1 ? p[1] : 0.0);
    };
    if (RCS && T.q < 2) {
        double* c = mst + T.q * RT_MROW<RCS>;
        c[RM_DXDY] = G.dxdy;
        c[RM_DIFF] = F == 3 ? A.kappa : A.nu;
        c[RM_SHIFT] = A.sw[F].gshift ? *A.sw[F].gshift : 0.0;
        c[RM_IDX2] = G.idx * G.idx;
        c[RM_IDY2] = G.idy * G.idy;
    }
    load_extras(T.kb);
    for (int kk = T.kb - RT::ZH; kk <= T.kb + RT::ZH; kk++) load_plane(kk);
    double2 gnext = load_g(T.kb, gio);
    cp_async_wait_all();
    __syncthreads();

    auto ringat = [&](int f, int kk) { return rhs_sm + f * RT::FIELD + RT::slot(kk) * RT::PLANE + at; };
    const double dxdy = G.dxdy, idx2 = G.idx * G.idx, idy2 = G.idy * G.idy;
    const double diff = F == 3 ? A.kappa : A.nu;
    const bool buoyancy = A.betg_x != 0.0 || A.betg_y != 0.0 || A.betg_z != 0.0;
    const double shift = A.sw[F].gshift ? *A.sw[F].gshift : 0.0;

    // w interpolated to this point's u (v) face in plane kk, from the ring
    auto wface = [&](int kk) {
        const double* w = ringat(2, kk);
        if (F == 0) return face<ORDER>(ORDER == 4 ? ld2(w - PJ) : z2, ld2(w), ld2(w + PJ), ORDER == 4 ? ld2(w + 2 * PJ) : z2);
        const double2 a = ld2(w - 2), b = ld2(w), c = ld2(w + 2);
        return face<ORDER>(make_double2(a.y, b.x), b, make_double2(b.y, c.x), c);
    };

    // ---- state carried up the column, as if row kb - 1 had just been done
    // own values of rows k-LO .. k+NZ.  At order 4 the rows below k are read back
    // from the ring: kept, they cost 12 registers (spills with the sweep) and as
    // many moves a row, 4517 against 4390 us at 512 x 512 x 384; at order 2,
    // with registers to spare, keeping them is the faster way, 478 against 496
    // us at 256 x 256 x 192.
    constexpr int LO = ORDER == 2 ? NZ : 0;
    double2 zw[LO + NZ + 1];
#pragma unroll
    for (int d = 0; d < LO + NZ; d++) zw[d + 1] = ld2(ringat(F, T.kb - LO + d));
    zw[0] = z2;
    // z fluxes with the halved face velocity m(k): F1(k) = m(k) (q(k) + q(k+1)),
    // F3(k) = m(k+1) (q(k) + q(k+3)); row k needs F1(k), F1(k-1), F3(k), F3(k-3)
    double2 f1 = z2, mz = z2;   // F1(k-1), m(k); F3 of the last rows in this thread's own slots f3q[k & 3]
    double* const f3q = rhs_sm + rhs_queue<ORDER, RCS>() + 2 * threadIdx.x;
    double2 kz = z2, fz = z2;                                 // scalar: z curvature of row k, flux of face k-1
    if (F < 3) {
        auto own = [&](int d) { return ld2(ringat(F, T.kb + d)); };
        double2 mm1, mm2 = z2;
        if (F == 2) {
            mm1 = face<ORDER>(ORDER == 4 ? own(-2) : z2, own(-1), own(0), ORDER == 4 ? own(1) : z2);
            if (ORDER == 4) {
                mz = face<ORDER>(own(-1), own(0), own(1), own(2));
                mm2 = face<ORDER>(own(-3), own(-2), own(-1), own(0));
            }
        } else {
            mm1 = wface(T.kb - 1);
            if (ORDER == 4) {
                mz = wface(T.kb);
                mm2 = wface(T.kb - 2);
            }
        }
        f1 = mm1 * (own(-1) + own(0));
        if (ORDER == 4) {
            st2(f3q + ((T.kb - 3) & 3) * 2 * RT_THREADS, mm2 * (own(-3) + own(0)));
            st2(f3q + ((T.kb - 2) & 3) * 2 * RT_THREADS, mm1 * (own(-2) + own(1)));
            st2(f3q + ((T.kb - 1) & 3) * 2 * RT_THREADS, mz * (own(-1) + own(2)));
        }
    }
    auto curv = [](double2 x, double2 y, double2 z) { return x - 2.0 * y + z; };
    // QUICK (scalar.c:79-162): the face value between c0 and c1 takes the
    // curvature centred on the upwind cell
    auto quick = [](double2 m, double2 c0, double2 c1, double2 kup, double2 kdn) {
        const double2 k = make_double2(m.x > 0.0 ? kup.x : kdn.x, m.y > 0.0 ? kup.y : kdn.y);
        return m * (0.5 * (c0 + c1) + -0.125 * k);
    };
    if (F == 3) {
        const double2 cm2 = ld2(ringat(F, T.kb - 2)), cm1 = ld2(ringat(F, T.kb - 1)), c0 = zw[LO + 1], c1 = zw[LO + 2];
        kz = curv(c1, c0, cm1);
        fz = quick(dxdy * ld2(ringat(2, T.kb - 1)), cm1, c0, curv(c0, cm1, cm2), kz);
    }
    double2 s1 = z2, s2 = z2, s3 = z2;   // forward sweep: s of rows k-1, k-2, k-3

    auto row = [&](int k, auto wall_tag) {
        constexpr bool WALL = decltype(wall_tag)::value;   // rows within two of a wall
        const bool live = F != 2 || !WALL || k < top;      // w has no point on the top wall
        double* const fb = rhs_sm + rhs_faces<ORDER>() + (k & 1) * RF_ALL;
        const double* mrow = mst + (k & 1) * RT_MROW<RCS>;
        auto DYDZ = [&](int d) { return mrow[1 + d]; };
        auto DXDZ = [&](int d) { return mrow[5 + d]; };
        auto scalar_of = [&](int m, double v) { return RCS ? mrow[m] : v; };
        // the window moves up one row
#pragma unroll
        for (int d = 0; d < LO + NZ; d++) zw[d] = zw[d + 1];
        zw[LO + NZ] = ld2(ringat(F, k + NZ));
        auto Z = [&](int d) { return LO + d >= 0 ? zw[LO + d >= 0 ? LO + d : 0] : ld2(ringat(F, k + d)); };
        const double2 q0 = Z(0);
        const double2 gk = gnext + make_double2(scalar_of(RM_SHIFT, shift), scalar_of(RM_SHIFT, shift));
        if (k + 1 < T.ke) gnext = load_g(k + 1, gio + T.plane);

        // ---- plane k: x neighbours, y neighbours (columns j-4 .. j+5)
        const double* p = ringat(F, k);
        double2 x[7], y[5];
#pragma unroll
        for (int d = -3; d <= 3; d++) x[d + 3] = d == 0 ? q0 : (ORDER == 4 || (d >= -2 && d <= 2)) ? ld2(p + d * PJ) : z2;
#pragma unroll
        for (int d = -2; d <= 2; d++) y[d + 2] = d == 0 ? q0 : (ORDER == 4 || (d >= -1 && d <= 1)) ? ld2(p + 2 * d) : z2;
        auto X = [&](int d) { return x[d + 3]; };
        // (q(j + d), q(j + 1 + d))
        auto Y = [&](int d) {
            const int e = d + 4;
            return (e & 1) == 0 ? y[e / 2] : make_double2(y[(e - 1) / 2].y, y[(e + 1) / 2].x);
        };
        // add_laplacexy_operator_{u,w}{2,4} (diffuseu.c:286-359, diffusew.c:290-363)
        const double rx = scalar_of(RM_IDX2, idx2), ry = scalar_of(RM_IDY2, idy2);
        double2 lap;
        if (ORDER == 2) {
            lap = rx * (X(1) - 2.0 * q0 + X(-1)) + ry * (Y(1) - 2.0 * q0 + Y(-1));
        } else {
            const double lapc = -2.0 * (L1 + L2 + L3) * (rx + ry);
            const double2 lx = L3 * (X(3) + X(-3)) + L2 * (X(2) + X(-2)) + L1 * (X(1) + X(-1));
            const double2 ly = L3 * (Y(3) + Y(-3)) + L2 * (Y(2) + Y(-2)) + L1 * (Y(1) + Y(-1));
            lap = (rx * lx + ry * ly) + lapc * q0;
        }
        // the explicit diffusion enters first at order 2 and last at order 4, by measurement (64 x 64 x 384
        // 413 -> 399 us, 256 x 256 x 192 at order 4 the other way round 619 -> 626)
        if (MODE == RHS_CHANNEL) lap = scalar_of(RM_DIFF, diff) * lap;
        auto onto_lap = [&](Product2 advection) -> double2 {
            if (MODE == RHS_CHANNEL || ORDER == 4) return advection;
            return advection + scalar_of(RM_DIFF, diff) * lap;
        };

        // ---- faces for the other fields, and the flux of the field's own direction
        const int wat = T.ty * RT_J + T.jl, uat = (T.ty + 2) * RT_J + T.jl, vat = T.ty * (RT_J + 4) + T.jl + 2;
        double2 own = z2;
        if (F == 0) {
            st2(fb + RF_UY + uat, face<ORDER>(Y(-1), q0, Y(1), Y(2)));
            if (ORDER == 2) st2(fb + RF_UZ + uat, 0.25 * (DYDZ(0) * q0 + DYDZ(1) * Z(1)));
            else st2(fb + RF_UZ + uat, (B1h * DYDZ(0)) * q0 + (B1h * DYDZ(1)) * Z(1) + ((B2h * DYDZ(-1)) * Z(-1) + (B2h * DYDZ(2)) * Z(2)));
            own = flux<ORDER>(ORDER == 4 ? face<ORDER>(X(-3), X(-2), X(-1), q0) : z2, face<ORDER>(X(-2), X(-1), q0, X(1)),
                              face<ORDER>(X(-1), q0, X(1), X(2)), ORDER == 4 ? face<ORDER>(q0, X(1), X(2), X(3)) : z2,
                              X(-3), X(-1), q0, X(1), X(3));
        } else if (F == 1) {
            st2(fb + RF_VX + vat, face<ORDER>(X(-1), q0, X(1), X(2)));
            if (ORDER == 2) st2(fb + RF_VZ + vat, 0.25 * (DXDZ(0) * q0 + DXDZ(1) * Z(1)));
            else st2(fb + RF_VZ + vat, (B1h * DXDZ(0)) * q0 + (B1h * DXDZ(1)) * Z(1) + ((B2h * DXDZ(-1)) * Z(-1) + (B2h * DXDZ(2)) * Z(2)));
            // faces j-2 .. j+2, each once for both points
            const double2 e0 = face<ORDER>(Y(-3), Y(-2), Y(-1), q0);                     // faces -2, -1
            const double2 e2 = face<ORDER>(Y(-1), q0, Y(1), Y(2));                       // faces 0, 1
            const double e4 = ORDER == 4 ? dot(B2h, add(Y(1).x, Y(3).y), B1h, add(Y(2).x, Y(3).x)) : 0.0;   // face 2
            own = flux<ORDER>(e0, make_double2(e0.y, e2.x), e2, make_double2(e2.y, e4), Y(-3), Y(-1), q0, Y(1), Y(3));
        } else if (F == 2) {
            if (ORDER == 2) {   // plane k: the z fluxes use m(k)
                st2(fb + RF_WX + wat, 0.25 * (q0 + X(1)));
                st2(fb + RF_WY + wat, 0.25 * (q0 + Y(1)));
            } else {            // plane k + 1: they use m(k + 1)
                const double* w = ringat(2, k + 1);
                const double2 w0 = Z(1), a = ld2(w - 2), c = ld2(w + 2);
                st2(fb + RF_WX + wat, face<ORDER>(ld2(w - PJ), w0, ld2(w + PJ), ld2(w + 2 * PJ)));
                st2(fb + RF_WY + wat, face<ORDER>(make_double2(a.y, w0.x), w0, make_double2(w0.y, c.x), c));
            }
        } else {
            // the rim: u's faces of rows i0-2, i0-1, i0+8 (order 2: i0-1), v's of the
            // column pairs j0-2 and j0+32 (order 2: j0-2)
            if (ORDER == 4 ? T.q < 48 : T.q < 16) {
                const int r = ORDER == 2 ? -1 : T.q < 16 ? -2 : T.q < 32 ? -1 : RT_I, j = 2 * (T.q & 15);
                const int o = (r + RT::H) * PJ + j + RT::XL;
                auto U = [&](int kk) { return rhs_sm + RT::slot(kk) * RT::PLANE + o; };
                const double* u = U(k);
                const double2 a = ld2(u - 2), b = ld2(u), c = ld2(u + 2);
                double* d = fb + RF_UY + (r + 2) * RT_J + j;
                st2(d, face<ORDER>(make_double2(a.y, b.x), b, make_double2(b.y, c.x), c));
                const double2 b1 = ld2(U(k + 1));
                if (ORDER == 2) st2(d + RF_UZ - RF_UY, 0.25 * (DYDZ(0) * b + DYDZ(1) * b1));
                else st2(d + RF_UZ - RF_UY, (B1h * DYDZ(0)) * b + (B1h * DYDZ(1)) * b1
                                            + ((B2h * DYDZ(-1)) * ld2(U(k - 1)) + (B2h * DYDZ(2)) * ld2(U(k + 2))));
            } else if (ORDER == 4 ? T.q < 64 : T.q >= 32 && T.q < 40) {
                const int e = T.q - (ORDER == 4 ? 48 : 32);
                const int r = ORDER == 4 ? e >> 1 : e, j = ORDER == 4 && (e & 1) ? RT_J : -2;
                const int o = RT::FIELD + (r + RT::H) * PJ + j + RT::XL;
                auto V = [&](int kk) { return rhs_sm + RT::slot(kk) * RT::PLANE + o; };
                const double* v = V(k);
                const double2 b = ld2(v), b1 = ld2(V(k + 1));
                double* d = fb + RF_VX + r * (RT_J + 4) + j + 2;
                st2(d, face<ORDER>(ORDER == 4 ? ld2(v - PJ) : z2, b, ld2(v + PJ), ORDER == 4 ? ld2(v + 2 * PJ) : z2));
                if (ORDER == 2) st2(d + RF_VZ - RF_VX, 0.25 * (DXDZ(0) * b + DXDZ(1) * b1));
                else st2(d + RF_VZ - RF_VX, (B1h * DXDZ(0)) * b + (B1h * DXDZ(1)) * b1
                                            + ((B2h * DXDZ(-1)) * ld2(V(k - 1)) + (B2h * DXDZ(2)) * ld2(V(k + 2))));
            }
        }

        double2 f;
        // flux_quick + advect_scalar (scalar.c:79-162): no faces of others.  At order 2
        // the longest work of a row, done while the other fields form their fluxes
        // (64 x 64 x 384 449 -> 413 us); at order 4 before the barrier, beside the
        // velocities' own longer halves (after it 256 x 256 x 192 619 -> 687 us).
        auto scalar = [&]() {
            const double* u = ringat(0, k);
            const double* v = ringat(1, k);
            const double2 va = ld2(v - 2), vb = ld2(v);
            const double2 kx0 = curv(X(1), q0, X(-1)), ky0 = curv(Y(1), q0, Y(-1)), kzp = curv(Z(2), Z(1), q0);
            const Product2 fxp = quick(DYDZ(0) * ld2(u), q0, X(1), kx0, curv(X(2), X(1), q0));
            const Product2 fxm = quick(DYDZ(0) * ld2(u - PJ), X(-1), q0, curv(q0, X(-1), X(-2)), kx0);
            const Product2 fyp = quick(DXDZ(0) * vb, q0, Y(1), ky0, curv(Y(2), Y(1), q0));
            const Product2 fym = quick(DXDZ(0) * make_double2(va.y, vb.x), Y(-1), q0, curv(q0, Y(-1), Y(-2)), ky0);
            const double2 fzp = quick(scalar_of(RM_DXDY, dxdy) * ld2(ringat(2, k)), q0, Z(1), kz, kzp);
            f = onto_lap((-mrow[8]) * ((fxp - fxm) + (fyp - fym) + (fzp - fz)));
            kz = kzp;
            fz = fzp;
        };
        if (F == 3 && ORDER == 4) scalar();
        __syncthreads();   // the row's faces are in place
        if (F == 3 && ORDER == 2) scalar();

        if (F < 3) {
            double2 other;   // the flux (for w: both) of the directions whose faces others hold
            if (F == 0 || F == 2) {   // y flux with v's faces, columns j-2 .. j+3
                const double* m = fb + (F == 0 ? RF_VX : RF_VZ) + vat;
                const double2 a = ld2(m - 2), b = ld2(m), c = ORDER == 4 ? ld2(m + 2) : z2;
                other = flux<ORDER>(a, make_double2(a.y, b.x), b, make_double2(b.y, c.x), Y(-3), Y(-1), q0, Y(1), Y(3));
            }
            if (F == 1 || F == 2) {   // x flux with u's faces, rows i-2 .. i+1
                const double* m = fb + (F == 1 ? RF_UY : RF_UZ) + uat;
                const double2 t = flux<ORDER>(ORDER == 4 ? ld2(m - 2 * RT_J) : z2, ld2(m - RT_J), ld2(m),
                                              ORDER == 4 ? ld2(m + RT_J) : z2, X(-3), X(-1), q0, X(1), X(3));
                other = F == 1 ? t : other + t;
            }
            // z fluxes
            double2 zph, zmh = f1, zp3 = z2, zm3 = ORDER == 4 ? ld2(f3q + ((k - 3) & 3) * 2 * RT_THREADS) : z2, mup;   // mup: m(k) at order 2, m(k+1) at order 4
            if (F == 2) mup = ORDER == 2 ? 0.25 * (q0 + Z(1)) : face<ORDER>(q0, Z(1), Z(2), Z(NZ));
            else mup = ld2(fb + (F == 0 ? RF_WX : RF_WY) + wat);
            if (ORDER == 2) {
                zph = mup * (q0 + Z(1));
                f1 = zph;
            } else {
                zph = mz * (q0 + Z(1));
                zp3 = mup * (q0 + Z(NZ));
                f1 = zph;
                st2(f3q + (k & 3) * 2 * RT_THREADS, zp3);
                if (WALL && F < 2) {   // wall closures of the cell-centred fields: the wall value qbot / qtop
                    auto wallq = [&](double2 a, double2 b, double2 c, double2 d) {   // ghost 2, ghost 1, first, second
                        return (0.5 * A2) * (a + d) + (0.5 * (A1 + 2.0 * A2)) * (b + c);
                    };
                    if (k == top) {
                        const double2 qt = wallq(Z(2), Z(1), q0, Z(-1));
                        zph = (2.0 * mz) * qt;
                        zp3 = (4.0 * mz) * qt - wface(k - 1) * (Z(-2) + Z(1));
                    }
                    if (k == top - 1) zp3 = (2.0 * mup) * wallq(Z(NZ), Z(2), Z(1), q0);
                    if (k == GZ) {
                        const double2 qb = wallq(Z(-2), Z(-1), q0, Z(1)), mb = wface(k - 1);
                        zmh = (2.0 * mb) * qb;
                        zm3 = (4.0 * mb) * qb - mz * (Z(2) + Z(-1));
                    }
                    if (k == GZ + 1) zm3 = (2.0 * wface(k - 2)) * wallq(Z(-NZ), Z(-2), Z(-1), q0);
                }
                mz = mup;
            }
            const double2 zs = ORDER == 2 ? zph - zmh : A1 * (zph - zmh) + A2 * (zp3 - zm3);
            if (F == 0) f = onto_lap((-mrow[8]) * ((DYDZ(0) * own + DXDZ(0) * other) + scalar_of(RM_DXDY, dxdy) * zs));
            if (F == 1) f = onto_lap((-mrow[8]) * ((DYDZ(0) * other + DXDZ(0) * own) + scalar_of(RM_DXDY, dxdy) * zs));
            if (F == 2) f = onto_lap((-mrow[9]) * (other + scalar_of(RM_DXDY, dxdy) * zs));
            // add_buoyancy{2,4} (scalar.c:6-76); skipped when every betg is zero
            if (buoyancy) {
                const double* c = ringat(3, k);
                const double2 c0 = ld2(c);
                if (F == 0) {
                    const double2 t = ORDER == 2 ? 0.5 * (c0 + ld2(c + PJ))
                                                 : B1 * (c0 + ld2(c + PJ)) + B2 * (ld2(c - PJ) + ld2(c + 2 * PJ));
                    f = f + A.betg_x * t;
                } else if (F == 1) {
                    const double2 a = ld2(c - 2), b = ld2(c + 2), n = make_double2(c0.y, b.x);
                    const double2 t = ORDER == 2 ? 0.5 * (c0 + n) : B1 * (c0 + n) + B2 * (make_double2(a.y, c0.x) + b);
                    f = f + A.betg_y * t;
                } else {
                    const double2 n = ld2(ringat(3, k + 1));
                    const double2 t = ORDER == 2 ? 0.5 * (c0 + n)
                                                 : B1 * (c0 + n) + B2 * (ld2(ringat(3, k - 1)) + ld2(ringat(3, k + 2)));
                    f = f + A.betg_z * t;
                }
            }
        }
        if (MODE != RHS_CHANNEL && ORDER == 4) f = f + scalar_of(RM_DIFF, diff) * lap;

        // ---- right-hand side of the implicit solve, rows GZ .. (u, v, c: nz rows; w: nz - 1 faces)
        const double2* r2 = reinterpret_cast<const double2*>(cst + (k & 1) * RT_FWMAX);
        double r[RT_FWMAX];
#pragma unroll
        for (int e = 0; e < (FWR + 1) / 2; e++) {
            if (2 * e < 2 * HH + 4 || MODE == RHS_SWEEP) {
                const double2 t = r2[e];
                r[2 * e] = t.x;
                r[2 * e + 1] = t.y;
            }
        }
        double2 h = r[2 * HH + 1] * f + r[2 * HH + 2] * gk;
        h = h + make_double2(r[2 * HH + 3], r[2 * HH + 3]);
        // the old w beyond its wall faces is apply_bc_w's (the ring holds the massflux4 extrapolation)
        double2 b1 = z2, b2 = z2;
        if (WALL && F == 2 && ORDER == 4) {
            double u;
            if (k <= GZ + 1) {
                const double2 w0 = k == GZ ? q0 : Z(-1), w1 = k == GZ ? Z(1) : q0;
                bc_w_bot<4>(A.wbot, A.wbc_bot, w0.x, w1.x, u, b1.x, b2.x);
                bc_w_bot<4>(A.wbot, A.wbc_bot, w0.y, w1.y, u, b1.y, b2.y);
            } else {
                const double2 w0 = k == top - 2 ? Z(1) : q0, w1 = k == top - 2 ? q0 : Z(-1);
                bc_w_top<4>(A.wtop, A.wbc_top, w0.x, w1.x, u, b1.x, b2.x);
                bc_w_top<4>(A.wtop, A.wbc_top, w0.y, w1.y, u, b1.y, b2.y);
            }
        }
#pragma unroll
        for (int d = -HH; d <= HH; d++) {
            double2 v = Z(d);
            if (WALL && F == 2 && ORDER == 4) {
                const int kk = k + d;
                if (kk < GZ - 1) v = kk == GZ - 2 ? b1 : b2;
                if (kk > top) v = kk == top + 1 ? b1 : b2;
            }
            h = h + r[d + HH] * v;
        }
        if (MODE == RHS_CHANNEL) h = h + lap;
        if (MODE == RHS_SWEEP) {
            if (ORDER == 4) {
                h = (h - r[2 * HH + 6] * s3) - r[2 * HH + 5] * s2;
                s3 = s2;
                s2 = s1;
            }
            h = h - r[2 * HH + 4] * s1;   // the previous row's s enters last
            s1 = h;
        }
        if (live) {
            if (EVEN) {
                if (T.v0) {
                    st2(fout, f);
                    st2(gio, h);
                }
            } else {
                if (T.v0) { fout[0] = f.x; gio[0] = h.x; }
                if (T.v1) { fout[1] = f.y; gio[1] = h.y; }
            }
        }
        fout += T.plane;
        gio += T.plane;
    };

    auto begin = [&](int k) {
        if (k + 1 < T.ke) {
            load_extras(k + 1);
            load_plane(k + RT::ZH + 1);   // row k + 1 reads up to k + 1 + ZH
        }
    };
    auto end = [&]() {
        // This field's threads alone: a field reads its own newest plane and its
        // own coefficients; of the others' planes rows up to k + 2 (order 2: k + 1),
        // which landed a row or more before the last block-wide barrier.  That
        // barrier also keeps a field within one row of the others: a ring slot
        // or a face buffer is rewritten only after every reader has passed it.
        cp_async_wait_all();
        asm volatile("bar.sync %0, %1;\n" ::"n"(F + 1), "n"(RT_FIELD) : "memory");
    };
    for (int k = T.kb; k < T.ke;) {
        const int inner = min(T.ke, top - 2);
        if (k > GZ + 1 && k < inner) {
            for (; k < inner; k++) {
                begin(k);
                row(k, std::false_type{});
                end();
            }
        } else {
            begin(k);
            row(k, std::true_type{});
            end();
            k++;
        }
    }
}

template <int ORDER, int MODE, bool EVEN, bool RCS>
__device__ __forceinline__ void rhs_body(const Geo& G, const RhsArgs& A, uint3 bid)
{
    using RT = RhsTile<ORDER>;
    RhsBlock T;
    int* goff = reinterpret_cast<int*>(rhs_sm + rhs_offs<ORDER, RCS>());
    const int nx = G.nx, ny = G.ny, tid = threadIdx.x;
    T.i0 = bid.y * RT_I;
    T.j0 = bid.x * RT_J;
    T.kb = GZ + (int) bid.z * A.chunk;
    T.ke = min(T.kb + A.chunk, GZ + G.nz);
    T.q = (tid >> 7) * 32 + (tid & 31);
    T.ty = T.q >> 4;
    T.jl = 2 * (T.q & 15);
    T.plane = G.plane;
    const int i = T.i0 + T.ty, j = T.j0 + T.jl;
    T.v0 = i < nx && j < ny;
    T.v1 = i < nx && j + 1 < ny;
    T.gij = T.v0 ? (long long) i * ny + j : 0;
    // The points (even ny: pairs) of a haloed plane, the same in every plane and
    // field: their offsets within a plane.  For even ny a pair starts at an
    // even y index (j0 and XL are even), so it never straddles the periodic
    // wrap and its global and shared addresses are 16-byte aligned.
    for (int e = tid; e < (EVEN ? RT::PLANE / 2 : RT::PLANE); e += RT_THREADS) {
        const int w = EVEN ? RT::PJ / 2 : RT::PJ, ii = e / w, jj = (e - ii * w) * (EVEN ? 2 : 1);
        int gi = (T.i0 + ii - RT::H) % nx; if (gi < 0) gi += nx;
        int gj = (T.j0 + jj - RT::XL) % ny; if (gj < 0) gj += ny;
        goff[e] = gi * ny + gj;
    }
    __syncthreads();
    // Warp w works on field w mod 4, so that the warps of one of the SM's four
    // schedulers run the same code.  Every field takes the same barriers.
    switch ((tid >> 5) & 3) {
    case 0: rhs_field<ORDER, MODE, 0, EVEN, RCS>(G, A, T); break;
    case 1: rhs_field<ORDER, MODE, 1, EVEN, RCS>(G, A, T); break;
    case 2: rhs_field<ORDER, MODE, 2, EVEN, RCS>(G, A, T); break;
    default: rhs_field<ORDER, MODE, 3, EVEN, RCS>(G, A, T); break;
    }
}

template <int ORDER, int MODE, bool EVEN>
__global__ void __launch_bounds__(RT_THREADS, 1) k_rhs(Geo G, RhsArgs A)
{
    rhs_body<ORDER, MODE, EVEN, false>(G, A, blockIdx);
}

// Members with partitioned line solves and those without: at order 2 in one
// launch, FORM_EITHER (of two, the first's last wave runs out before the second
// begins: 6 flows of 90 x 75 x 53, 100 x 120 x 64 and 240 x 250 x 64, a substep
// 1372 against 1260 us); at order 4 in launches of their own, since both bodies
// in one kernel cost more registers than there are (6 x 192 x 192 x 128 a
// substep 3356 against 3519 us; the mixed sizes above 1683 against 1644).
// A record's scalars are no constants and cost registers too.  Without the
// sweep they go to shared memory (RCS), 8 x 128 x 128 x 96 at order 4 a substep 1872 -> 1584
// us; with it the spills are cheaper, 6 x 192 x 192 x 128 3356 against 3510.
enum RhsForm { FORM_EITHER, FORM_SWEEP, FORM_H };
template <int ORDER, int FORM, bool EVEN>
__global__ void __launch_bounds__(RT_THREADS, 1) k_rhs_batch(const BatchRec<RhsArgs>* r, int n)
{
    uint3 b;
    const BatchRec<RhsArgs>& R = batch_locate(r, n, b);
    if (FORM == FORM_H || (FORM == FORM_EITHER && R.G.partitioned)) rhs_body<ORDER, RHS_H, EVEN, true>(R.G, R.A, b);
    else rhs_body<ORDER, RHS_SWEEP, EVEN, false>(R.G, R.A, b);
}

// ------------------------------------------------------------- launchers

constexpr int GHOST_THREADS = 128;

dim3 grid_ghosts(const Geo& G) { return dim3((unsigned) ((G.plane + GHOST_THREADS - 1) / GHOST_THREADS), 4); }

void launch_ghosts(const Geo& G, const GhostArgs& A, cudaStream_t st, bool extrap)
{
    const int th = GHOST_THREADS;
    const dim3 nb = grid_ghosts(G);
    if (extrap) {
        if (G.order == 2) k_ghosts<2, true><<<nb, th, 0, st>>>(G, A);
        else k_ghosts<4, true><<<nb, th, 0, st>>>(G, A);
    } else {
        if (G.order == 2) k_ghosts<2, false><<<nb, th, 0, st>>>(G, A);
        else k_ghosts<4, false><<<nb, th, 0, st>>>(G, A);
    }
}

dim3 grid_rhs(const Geo& G, int chunk)
{
    return dim3((G.ny + RT_J - 1) / RT_J, (G.nx + RT_I - 1) / RT_I, (G.nz + chunk - 1) / chunk);
}

long long rhs_tiles(const Geo& G) { return (long long) ((G.ny + RT_J - 1) / RT_J) * ((G.nx + RT_I - 1) / RT_I); }

// Rows per k_rhs block of an instance that has `sms` SMs to itself (in a batch,
// its share of them by tiles).  One block fills an SM, so the time is the
// number of waves times a block's rows plus its start (the ring's first planes
// and the primed fluxes, about RHS_START rows); the chunk count with the least
// of it is taken.  Whole columns with the forward sweep in the kernel (sweep),
// and where the tiles alone give three quarters of the SMs a block (as
// line_partitioned).  Results do not depend on it: a block primes the fluxes
// and curvatures that it would have carried up, in the same operations
// (rounding.cuh).
int rhs_chunk(const Geo& G, int sms, bool sweep)
{
    constexpr int RHS_START = 4;
    const long long tiles = rhs_tiles(G);
    if (sweep || 4 * tiles > 3 * sms) return G.nz;
    long long best = -1;
    int chunk = G.nz;
    for (int c = 1; c <= std::max(1, G.nz / RHS_MIN_ROWS); c++) {
        const int rows = (G.nz + c - 1) / c;
        const long long n = (G.nz + rows - 1) / rows, waves = (tiles * n + sms - 1) / sms;
        const long long cost = waves * (rows + RHS_START);
        if (best < 0 || cost < best) {
            best = cost;
            chunk = rows;
        }
    }
    return chunk;
}

void launch_ghosts_batch(const BatchLaunch& L, int order, cudaStream_t st)
{
    auto r = static_cast<const BatchRec<GhostArgs>*>(L.recs);
    if (order == 2) k_ghosts_batch<2, true><<<L.blocks, GHOST_THREADS, 0, st>>>(r, L.n);
    else k_ghosts_batch<4, true><<<L.blocks, GHOST_THREADS, 0, st>>>(r, L.n);
}

void launch_rhs_batch(const BatchLaunch& L, int key, cudaStream_t st)
{
    auto r = static_cast<const BatchRec<RhsArgs>*>(L.recs);
    const dim3 blk(RT_THREADS);
#define CASE_(key_, o_, form_) \
    case key_: k_rhs_batch<o_, form_, true><<<L.blocks, blk, rhs_smem_bytes<o_, true>(), st>>>(r, L.n); break; \
    case key_ + 8: k_rhs_batch<o_, form_, false><<<L.blocks, blk, rhs_smem_bytes<o_, true>(), st>>>(r, L.n); break;
    switch (key) {
    CASE_(2, 2, FORM_EITHER) CASE_(4, 4, FORM_SWEEP) CASE_(20, 4, FORM_H)
    default: break;
    }
#undef CASE_
}

void launch_rhs(const Geo& G, const RhsArgs& A, bool implicit3d, cudaStream_t st)
{
    const dim3 blk(RT_THREADS), grd = grid_rhs(G, A.chunk);
    const int mode = implicit3d ? RHS_CHANNEL : G.partitioned ? RHS_H : RHS_SWEEP;
#define CASE_(o_, m_) \
    if (G.order == o_ && mode == m_) { \
        if (G.ny % 2 == 0) k_rhs<o_, m_, true><<<grd, blk, rhs_smem_bytes<o_>(), st>>>(G, A); \
        else k_rhs<o_, m_, false><<<grd, blk, rhs_smem_bytes<o_>(), st>>>(G, A); \
    }
    CASE_(2, RHS_SWEEP) CASE_(2, RHS_H) CASE_(2, RHS_CHANNEL)
    CASE_(4, RHS_SWEEP) CASE_(4, RHS_H) CASE_(4, RHS_CHANNEL)
#undef CASE_
}

cudaError_t rhs_set_smem_limits()
{
    const int v2 = (int) rhs_smem_bytes<2, true>(), v4 = (int) rhs_smem_bytes<4, true>();
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* f, int v) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
    };
    set((const void*) k_rhs<2, RHS_SWEEP, true>, v2);
    set((const void*) k_rhs<2, RHS_SWEEP, false>, v2);
    set((const void*) k_rhs<2, RHS_H, true>, v2);
    set((const void*) k_rhs<2, RHS_H, false>, v2);
    set((const void*) k_rhs<2, RHS_CHANNEL, true>, v2);
    set((const void*) k_rhs<2, RHS_CHANNEL, false>, v2);
    set((const void*) k_rhs<4, RHS_SWEEP, true>, v4);
    set((const void*) k_rhs<4, RHS_SWEEP, false>, v4);
    set((const void*) k_rhs<4, RHS_H, true>, v4);
    set((const void*) k_rhs<4, RHS_H, false>, v4);
    set((const void*) k_rhs<4, RHS_CHANNEL, true>, v4);
    set((const void*) k_rhs<4, RHS_CHANNEL, false>, v4);
    set((const void*) k_rhs_batch<2, FORM_EITHER, true>, v2);
    set((const void*) k_rhs_batch<2, FORM_EITHER, false>, v2);
    set((const void*) k_rhs_batch<4, FORM_SWEEP, true>, v4);
    set((const void*) k_rhs_batch<4, FORM_SWEEP, false>, v4);
    set((const void*) k_rhs_batch<4, FORM_H, true>, v4);
    set((const void*) k_rhs_batch<4, FORM_H, false>, v4);
    return e;
}

}  // namespace cf
