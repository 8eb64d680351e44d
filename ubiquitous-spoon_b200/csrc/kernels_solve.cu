// Implicit wall-normal diffusion: the line solves of u, v, c and w.
//
// Per column the substep does what chanfast.c:459-482 does for one field
// (order 2; :1383-1406 order 4):
//   h  = helmholtz1d_operator(x, nuadt) + gamdt*f + zetdt*g - hbc
//   x  = solve_helmholtz1d(h, -nubdt)       (tridag.c / heptdag.c)
//   apply_bc(x)
// The band matrix is the same for every column, so its factorisation comes
// precomputed from host_band.cpp.  k_rhs (kernels_rhs.cu) leaves h, scaled
// by cell volume and pivot (fused_rows), in the g buffer, or already swept
// forward (line_partitioned decides); k_line does the rest of the four fields'
// solves and apply_bc in one launch, and the bulk and wall statistics of u
// and c that the controls need.
#include <algorithm>

#include "engine.cuh"
#include "host_band.h"
#include "wall.cuh"
#include "batch.cuh"
#include "rounding.cuh"

namespace cf {

__device__ __forceinline__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over 8 lanes (one chunk of 16 columns, two per lane); every lane gets it.
__device__ __forceinline__ double oct_sum(double v)
{
    const unsigned mask = 0xffu << (threadIdx.x & 24);
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o, 8);
    return v;
}

// apply_bc after the solve (chanfast.c:481-482): the ghost rows of one column
// from its last solved values next to each wall, stored for valid columns.
template <int ORDER, bool IS_W>
__device__ __forceinline__ void ghosts_bot(const SolveArgs& A, double* x, long long P, bool valid, double x0, double x1,
                                           double x2, double& g1, double& g2)
{
    double g3;
    if (IS_W) bc_w_bot<ORDER>(A.bcb, A.bc_bot, x0, x1, g1, g2, g3);
    else bc_u_bot<ORDER>(A.bcb, A.bc_bot, x0, x1, x2, g1, g2, g3);
    if (!valid) return;
    const int kb = GZ - 1;
    x[kb * P] = g1;
    if (ORDER == 4) {
        x[(kb - 1) * P] = g2;
        x[(kb - 2) * P] = g3;
    }
}

template <int ORDER, bool IS_W>
__device__ __forceinline__ void ghosts_top(const SolveArgs& A, double* x, long long P, int n2, bool valid, double x0,
                                           double x1, double x2, double& g1, double& g2)
{
    double g3;
    if (IS_W) bc_w_top<ORDER>(A.bct, A.bc_top, x0, x1, g1, g2, g3);
    else bc_u_top<ORDER>(A.bct, A.bc_top, x0, x1, x2, g1, g2, g3);
    if (!valid) return;
    const int kt = IS_W ? n2 - GZ - 1 : n2 - GZ;
    x[kt * P] = g1;
    if (ORDER == 4) {
        x[(kt + 1) * P] = g2;
        x[(kt + 2) * P] = g3;
    }
}

// One line solve, partitioned: a column's n rows are cut into C chunks of
// LINE_R rows (the last one may be shorter), one thread per chunk and pair of
// columns, its right-hand sides in registers.  Both sweeps are linear
// recurrences whose coefficients do not depend on the column.  Each thread
// first sweeps its chunk as if the values before it were zero and keeps only
// the last H; one thread per pair then carries the true boundary values
// through the chunks,
//   b_{c+1} = e_c + M_c b_c     (M_c: H x H, line_rows in host_band.h)
// and every thread sweeps its chunk again from its true boundary values, in
// the serial solve's own operations.  The same for the back sweep.
// Eight lanes of two columns make a 128-byte row segment; the recurrence rows
// are staged in shared memory.
//
// Bound: latency, of four sweeps over 16 rows and two carries over C chunks,
// where a thread per column walks all rows twice: 10 against 22 us for the four
// fields' back sweeps alone at 64 x 64 x 64, order 2 (and k_rhs no longer
// sweeps).  Also tried: one column a thread (fewer chains in flight), blocks
// that walk over column groups with the next group prefetched (the carries
// then wait for one another), whole columns staged in shared memory and swept
// serially (two warps per SM at 384 rows show every latency): all slower.
template <int ORDER, bool IS_W>
__device__ __forceinline__ void line_chunks(const Geo& G, const SolveArgs& A, uint3 bid, double* sm)
{
    constexpr int H = ORDER == 2 ? 1 : 3, R = LINE_R, CS = line_chunk_stride(ORDER), MS = line_mat_stride(ORDER);
    const int C = line_chunk_count(G.nz), n = A.n;
    const int lanes = line_lanes(blockDim.x, C);
    const int c = threadIdx.x / lanes, lc = threadIdx.x - c * lanes;   // chunk, column pair
    const bool work = c < C;
    const long long P = G.plane, col = (long long) bid.x * 2 * lanes + 2 * lc;
    const bool v0 = work && col < P, v1 = work && col + 1 < P;
    const bool pairs = (P & 1) == 0;           // 16-byte accesses: every row starts on an even offset
    const int n2 = G.n2, lo = c * R, size = work ? min(R, n - lo) : 0;   // size <= 0: a chunk of padding
    const double* __restrict__ t = A.s + (long long) (GZ + lo) * P + (v0 ? col : 0);
    double* x = A.x + (v0 ? col : 0);
    double* tab = sm;                              // [C][CS] recurrence rows
    double* mat = tab + C * CS;                    // [2][C][MS] boundary matrices
    double2* ends = reinterpret_cast<double2*>(mat + 2 * C * MS);   // [C][H][lanes]: values at a chunk's end, swept from zero
    double2* hist = ends + max(C * H, 3) * lanes;  // [C][H][lanes]: true values beyond its boundary

    for (int e = threadIdx.x; e < C * (CS + 2 * MS) / 2; e += blockDim.x) {
        const unsigned d = (unsigned) __cvta_generic_to_shared(sm + 2 * e);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(A.rows + 2 * e) : "memory");
    }
    double2 h[R];
    if (pairs) {
#pragma unroll
        for (int r = 0; r < R; r++, t += P)
            h[r] = v0 && r < size ? __ldg(reinterpret_cast<const double2*>(t)) : make_double2(0.0, 0.0);
    } else {
#pragma unroll
        for (int r = 0; r < R; r++, t += P) {
            h[r].x = v0 && r < size ? __ldg(t) : 0.0;
            h[r].y = v1 && r < size ? __ldg(t + 1) : 0.0;
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    const double2* F = reinterpret_cast<const double2*>(tab + (work ? c : 0) * CS);   // f_1..f_H of rows 0 .. R-1
    const double2* B = F + R * H / 2;                                                // P, Q, R of rows 0 .. R-1

    // one row: the newest value enters last
    auto step = [](double2 v, double k1, double k2, double k3, double2& a1, double2& a2, double2& a3) {
        if (ORDER == 4) {
            v = (v - k3 * a3) - k2 * a2;
            a3 = a2;
            a2 = a1;
        }
        return a1 = v - k1 * a1;
    };
    // coefficients of rows r and r + 1 (r even)
    auto rows2 = [&](const double2* T, int r, double (&k)[6]) {
        if (ORDER == 2) {
            const double2 q = T[r / 2];
            k[0] = q.x;
            k[3] = q.y;
            k[1] = k[2] = k[4] = k[5] = 0.0;
        } else {
            const double2 q0 = T[3 * r / 2], q1 = T[3 * r / 2 + 1], q2 = T[3 * r / 2 + 2];
            k[0] = q0.x; k[1] = q0.y; k[2] = q1.x; k[3] = q1.y; k[4] = q2.x; k[5] = q2.y;
        }
    };
    auto put_ends = [&](double2 e1, double2 e2, double2 e3) {
        if (!work) return;
        ends[(c * H + 0) * lanes + lc] = e1;
        if (ORDER == 4) {
            ends[(c * H + 1) * lanes + lc] = e2;
            ends[(c * H + 2) * lanes + lc] = e3;
        }
    };
    auto get_hist = [&](double2& b1, double2& b2, double2& b3) {
        b1 = hist[(c * H + 0) * lanes + lc];
        if (ORDER == 4) {
            b2 = hist[(c * H + 1) * lanes + lc];
            b3 = hist[(c * H + 2) * lanes + lc];
        }
    };
    // the boundary values through all chunks, from chunk q in direction dir
    auto carry = [&](const double* M, int q, int dir) {
        double2 b1 = make_double2(0.0, 0.0), b2 = b1, b3 = b1;
        for (int i = 0; i + 1 < C; i++, q += dir) {
            const double2 e1 = ends[(q * H + 0) * lanes + lc];
            double2* to = hist + (q + dir) * H * lanes + lc;
            if (ORDER == 2) {
                b1 = e1 + M[q] * b1;
            } else {
                const double2 e2 = ends[(q * H + 1) * lanes + lc], e3 = ends[(q * H + 2) * lanes + lc];
                const double2* m = reinterpret_cast<const double2*>(M + q * MS);
                const double2 m01 = m[0], m23 = m[1], m45 = m[2], m67 = m[3];
                const double m8 = m[4].x;
                const double2 c1 = (e1 + m01.x * b1) + (m01.y * b2 + m23.x * b3);
                const double2 c2 = (e2 + m23.y * b1) + (m45.x * b2 + m45.y * b3);
                b3 = (e3 + m67.x * b1) + (m67.y * b2 + m8 * b3);
                b1 = c1;
                b2 = c2;
                to[1 * lanes] = b2;
                to[2 * lanes] = b3;
            }
            to[0] = b1;
        }
    };
    const double2 z = make_double2(0.0, 0.0);
    double2 a1 = z, a2 = z, a3 = z;
    double k[6];

    if (C > 1) {
#pragma unroll
        for (int r = 0; r < R; r += 2) {
            rows2(F, r, k);
            step(h[r], k[0], k[1], k[2], a1, a2, a3);
            step(h[r + 1], k[3], k[4], k[5], a1, a2, a3);
        }
        put_ends(a1, a2, a3);
        __syncthreads();
        if (c == 0) carry(mat, 0, 1);
        __syncthreads();
        a1 = a2 = a3 = z;
        if (work && c > 0) get_hist(a1, a2, a3);
    }
    // (padding rows of the last chunk have zero coefficients: they stay zero)
#pragma unroll
    for (int r = 0; r < R; r += 2) {
        rows2(F, r, k);
        h[r] = step(h[r], k[0], k[1], k[2], a1, a2, a3);
        h[r + 1] = step(h[r + 1], k[3], k[4], k[5], a1, a2, a3);
    }
    a1 = a2 = a3 = z;
    if (C > 1) {
#pragma unroll
        for (int r = R - 2; r >= 0; r -= 2) {
            rows2(B, r, k);
            step(h[r + 1], k[3], k[4], k[5], a1, a2, a3);
            step(h[r], k[0], k[1], k[2], a1, a2, a3);
        }
        put_ends(a1, a2, a3);
        __syncthreads();
        if (c == 0) carry(mat + C * MS, C - 1, -1);
        __syncthreads();
        a1 = a2 = a3 = z;
        if (work && c < C - 1) get_hist(a1, a2, a3);
    }
#pragma unroll
    for (int r = R - 2; r >= 0; r -= 2) {
        rows2(B, r, k);
        h[r + 1] = step(h[r + 1], k[3], k[4], k[5], a1, a2, a3);
        h[r] = step(h[r], k[0], k[1], k[2], a1, a2, a3);
    }

    if (pairs) {
        if (v0) {
#pragma unroll
            for (int r = 0; r < R; r++)
                if (r < size) *reinterpret_cast<double2*>(x + (GZ + lo + r) * P) = h[r];
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (v0 && r < size) x[(GZ + lo + r) * P] = h[r].x;
            if (v1 && r < size) x[(GZ + lo + r) * P + 1] = h[r].y;
        }
    }
    // the last three rows, which may lie in the last two chunks, by way of
    // `ends` (last read before the last barrier)
    if (work && c >= C - 2) {
        const int top = n - 1 - lo;
#pragma unroll
        for (int r = 0; r < R; r++)
            if (r <= top && r > top - 3) ends[(top - r) * lanes + lc] = h[r];
    }
    __syncthreads();
    double2 top0 = z, top1 = z, top2 = z, gb1 = z, gb2 = z, gt1 = z, gt2 = z;
    if (work && c == C - 1) {
        top0 = ends[0 * lanes + lc];
        top1 = ends[1 * lanes + lc];
        top2 = ends[2 * lanes + lc];
        ghosts_top<ORDER, IS_W>(A, x, P, n2, v0, top0.x, top1.x, top2.x, gt1.x, gt2.x);
        ghosts_top<ORDER, IS_W>(A, x + 1, P, n2, v1, top0.y, top1.y, top2.y, gt1.y, gt2.y);
    }
    if (work && c == 0) {
        ghosts_bot<ORDER, IS_W>(A, x, P, v0, h[0].x, h[1].x, h[2].x, gb1.x, gb2.x);
        ghosts_bot<ORDER, IS_W>(A, x + 1, P, v1, h[0].y, h[1].y, h[2].y, gb1.y, gb2.y);
    }
    if (A.partial == nullptr) return;

    // column sums over each group of 16 columns: slot 0 sum of x dz, 1-4
    // rows g-2 .. g+1, 5-8 rows n2-g-2 .. n2-g+1, 9 and 10 the centre rows
    const long long grp = col / 16, ng = A.ngroups;
    const bool lead = (threadIdx.x & 7) == 0 && work && grp < ng;
    auto put = [&](int q, double2 v) {
        const double s = oct_sum((v0 ? v.x : 0.0) + (v1 ? v.y : 0.0));
        if (lead) A.partial[q * ng + grp] = s;
    };
    if (work && c == 0) {
        put(1, gb2);
        put(2, gb1);
        put(3, h[0]);
        put(4, h[1]);
    }
    if (work && c == C - 1) {
        put(5, top1);
        put(6, top0);
        put(7, gt1);
        put(8, gt2);
    }
    const int m0 = (G.nz - 1) / 2 - lo, m1 = G.nz / 2 - lo;   // centre rows, as rows of this chunk
    if (work && m1 >= 0 && m0 < R) {
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (r == m0) put(9, h[r]);
            if (r == m1) put(10, h[r]);
        }
    }
    double2 bulk = z;
    const double* dz = G.dz + GZ + lo;
#pragma unroll
    for (int r = 0; r < R; r++)
        if (r < size) {
            bulk = bulk + __ldg(dz + r) * h[r];
        }
    const double sum = oct_sum((v0 ? bulk.x : 0.0) + (v1 ? bulk.y : 0.0));
    double* sums = reinterpret_cast<double*>(hist);   // last read before the last barrier
    if ((threadIdx.x & 7) == 0 && work) sums[(lc / 8) * C + c] = sum;
    __syncthreads();
    if (c == 0 && lead) {
        double b = 0.0;
        for (int q = 0; q < C; q++) b += sums[(lc / 8) * C + q];
        A.partial[grp] = b;
    }
}

// The back sweep with one thread per column, of rows whose forward sweep k_rhs
// has done (its SWEEP variant); s of row i - PD is loaded while row i is
// computed.
// Bound: HBM, 16 bytes per point and field; 1.08 ms for four fields at
// 512 x 512 x 384, order 4 (6.0 TB/s).  That takes about 70 KB of loads in flight
// on an SM: PD = 8 at 9 or 10 blocks.  With PD = 4, us for the four fields,
// 512 x 512 x 384 order 4 1480, 300 x 320 x 200 order 2 312 (now 226).
template <int ORDER, bool IS_W, bool STATS>
__device__ __forceinline__ void back_column(const Geo& G, const SolveArgs& A, uint3 bid)
{
    constexpr int H = ORDER == 2 ? 1 : 3, PD = 8;
    const long long P = G.plane, col = (long long) bid.x * blockDim.x + threadIdx.x;
    const bool valid = col < P;
    const int n = A.n, n2 = G.n2;
    const double* __restrict__ s = A.s + GZ * P + (valid ? col : 0);
    double* x = A.x + (valid ? col : 0);
    const double* __restrict__ rows = A.back;
    const double* __restrict__ dz = G.dz + GZ;
    double y1 = 0.0, y2 = 0.0, y3 = 0.0, bulk = 0.0, p[PD];
#pragma unroll
    for (int u = 0; u < PD; u++) p[u] = n - 1 - u >= 0 ? s[(n - 1 - u) * P] : 0.0;
    for (int i0 = n - 1; i0 >= 0; i0 -= PD) {
#pragma unroll
        for (int u = 0; u < PD; u++) {
            const int i = i0 - u;
            if (i >= 0) {
                double y = p[u];
                if (i - PD >= 0) p[u] = s[(i - PD) * P];
                if (ORDER == 4) y = msub(__ldg(rows + i * H + 1), y2, msub(__ldg(rows + i * H + 2), y3, y));
                y = msub(__ldg(rows + i * H), y1, y);   // y1 last
                y3 = y2; y2 = y1; y1 = y;
                if (valid) x[(GZ + i) * P] = y;
                if (STATS) bulk = mad(y, __ldg(dz + i), bulk);
            }
        }
    }
    // rows by the top wall and at the centre, read back (kept in registers
    // they would cost resident blocks)
    auto again = [&](int i) { return valid && i >= 0 ? x[(GZ + i) * P] : 0.0; };
    const double top0 = again(n - 1), top1 = again(n - 2), top2 = again(n - 3);
    const double mid0 = STATS ? again((G.nz - 1) / 2) : 0.0, mid1 = STATS ? again(G.nz / 2) : 0.0;
    double gb1, gb2, gt1, gt2;
    ghosts_bot<ORDER, IS_W>(A, x, P, valid, y1, y2, y3, gb1, gb2);
    ghosts_top<ORDER, IS_W>(A, x, P, n2, valid, top0, top1, top2, gt1, gt2);
    if (!STATS) return;
    const long long grp = col / 32;
    auto put = [&](int q, double v) {
        v = warp_sum(valid ? v : 0.0);
        if ((threadIdx.x & 31) == 0 && grp < A.ngroups) A.partial[q * A.ngroups + grp] = v;
    };
    put(0, bulk);
    put(1, gb2);
    put(2, gb1);
    put(3, y1);
    put(4, y2);
    put(5, top1);
    put(6, top0);
    put(7, gt1);
    put(8, gt2);
    put(9, mid0);
    put(10, mid1);
}

// The control and its log row from the bulk mean, the averages of rows
// g-2 .. g+1 (bot), n2-g-2 .. n2-g+1 (top) and the centreline.
__device__ __forceinline__ void control_finish(const MassArgs& A, long long cnt, double mean, const double* bot,
                                               const double* top, double centre)
{
    const int g = GZ, n2 = A.n2;
    const double* dz = A.dz;
    double s[4];
    s[0] = mean;
    if (A.order == 4) {
        s[1] = mul(A.kappa, dot(A1, bot[2] - bot[1], A2, bot[3] - bot[0])) / (0.5 * (dz[g] + dz[g - 1]));
        s[2] = mul(A.kappa, dot(A1, top[2] - top[1], A2, top[3] - top[0])) / (0.5 * (dz[n2 - g] + dz[n2 - g - 1]));
    } else {
        s[1] = A.kappa * (bot[2] - bot[1]) / (0.5 * (dz[g] + dz[g - 1]));
        s[2] = A.kappa * (top[2] - top[1]) / (0.5 * (dz[n2 - g] + dz[n2 - g - 1]));
    }
    s[3] = centre;
    double m = A.mode == 1 ? (A.target - s[0]) / A.green[0] : A.fixed;
    // The bulk mean sums every interior point of the field, so a NaN or Inf
    // anywhere in it (or in the control) shows here; the flag stays set
    // until the host resets it with new fields.
    if (A.nonfinite && !isfinite(s[0] + m)) *A.nonfinite = 1.0;
    for (int t = 0; t < 4; t++) s[t] = mad(A.green[t], m, s[t]);
    *A.m_out = m;
    if (A.log_base) {
        double* row = A.log_base + (cnt % A.log_cap) * LOG_COLS + A.col;
        row[0] = m;
        row[1] = s[1];
        row[2] = s[2];
        row[3] = s[0];
        row[4] = s[3];
    }
}

// Bulk-mean control of chanfast.c:485-529 (u) / 572-616 (c).  The warp
// stages the profile and the cell heights in shared memory (rows up to
// MASS_MAX_N2, else read in place); one thread then sums them in the
// reference's order.
constexpr int MASS_MAX_N2 = 2048;   // 32 KB of static shared memory
__device__ __forceinline__ void mass_control_body(const MassArgs& A)
{
    __shared__ double s_avg[MASS_MAX_N2], s_dz[MASS_MAX_N2];
    const int g = GZ, n2 = A.n2, nz = A.nz;
    const bool staged = n2 <= MASS_MAX_N2;
    if (staged) {
        for (int k = threadIdx.x; k < n2; k += blockDim.x) {
            s_avg[k] = A.avg[k];
            s_dz[k] = A.dz[k];
        }
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    const double* avg = staged ? s_avg : A.avg;
    const double* dz = staged ? s_dz : A.dz;
    double a = 0.0, l = 0.0;  // get_z_avg (get.c:490-502)
    for (int k = g; k < nz + g; k++) {
        a += avg[k] * dz[k];
        l += dz[k];
    }
    const long long cnt = *A.counter;
    control_finish(A, cnt, a / l, avg + g - 2, avg + n2 - g - 2, 0.5 * (avg[g + (nz - 1) / 2] + avg[g + nz / 2]));
    if (A.log_base && A.advance) *A.counter = cnt + 1;
}
__global__ void k_mass_control(MassArgs A)
{
    if (blockIdx.x == 0) mass_control_body(A);
}

// Mass-flux (u) and scalar-mean (c) control of the z-implicit scheme from the
// column sums of k_line: one block per field and slot adds its groups in a
// fixed order, and the last block to finish does both controls.  One launch
// of 2 x LINE_STATS blocks in place of four (two row averages over n2 rows of
// every 32 columns, two single-block controls): 7 against 17 us at
// 64 x 64 x 64, 10 against 56 us at 512 x 512 x 384, where it reads 1.4 MB of
// sums instead of 51 MB.
__device__ __forceinline__ void control_body(const ControlArgs& A, uint3 bid)
{
    __shared__ double red[CONTROL_THREADS / 32];
    const int f = bid.x / LINE_STATS, slot = bid.x - f * LINE_STATS;
    const double* __restrict__ p = A.partial[f] + slot * A.ngroups;
    double v = 0.0;
    for (long long q = threadIdx.x; q < A.ngroups; q += CONTROL_THREADS) v += p[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x / 32] = v;
    __syncthreads();
    if (threadIdx.x >= 32) return;
    unsigned done = 0;
    if (threadIdx.x == 0) {
        v = 0.0;
        for (int q = 0; q < CONTROL_THREADS / 32; q++) v += red[q];
        A.sums[bid.x] = v * A.scale;
        __threadfence();
        done = atomicAdd(A.ticket, 1u);
    }
    if (__shfl_sync(0xffffffffu, done, 0) != 2 * LINE_STATS - 1) return;
    __threadfence();
    const long long cnt = *A.m[1].counter;   // both rows before the count moves on
    __syncwarp();
    if (threadIdx.x < 2) {
        const int q = threadIdx.x;
        double s[LINE_STATS];
#pragma unroll
        for (int e = 0; e < LINE_STATS; e++) s[e] = __ldcg(A.sums + q * LINE_STATS + e);
        control_finish(A.m[q], cnt, mul(s[0], A.ilz), s + 1, s + 5, 0.5 * (s[9] + s[10]));
    }
    if (threadIdx.x == 0) {
        *A.m[1].counter = cnt + 1;
        *A.ticket = 0;   // for the next substep's launch
    }
}

__global__ void __launch_bounds__(CONTROL_THREADS) k_control(ControlArgs A) { control_body(A, blockIdx); }

__global__ void __launch_bounds__(CONTROL_THREADS) k_control_batch(const BatchRec<ControlArgs>* r, int n)
{
    uint3 b;
    const BatchRec<ControlArgs>& R = batch_locate(r, n, b);
    control_body(R.A, b);
}

// The line solves of the four fields in one launch; blockIdx.y selects the
// field: 0 u, 1 v, 2 c, 3 w (u and c with column sums).  CHUNKS: both sweeps, partitioned; else the back
// sweep alone (line_partitioned decides).
template <int ORDER, bool CHUNKS>
__device__ __forceinline__ void line_body(const Geo& G, const SolveBatch& B, uint3 bid)
{
    extern __shared__ __align__(16) double line_sm[];
    if constexpr (CHUNKS) {
        if (bid.y < 3) line_chunks<ORDER, false>(G, B.a[bid.y], bid, line_sm);
        else line_chunks<ORDER, true>(G, B.a[3], bid, line_sm);
    } else {
        if (bid.y == 3) back_column<ORDER, true, false>(G, B.a[3], bid);
        else if (bid.y == 1) back_column<ORDER, false, false>(G, B.a[1], bid);
        else back_column<ORDER, false, true>(G, B.a[bid.y], bid);
    }
}

// Blocks of 128 threads per SM of the back sweep.  Order 4: 56 registers, one block
// fewer measured 45 % slower at 512 x 512 x 384; order 2: 48 registers, 512 x 512
// x 256 665 us, with 9 blocks 946, with 12 (40 registers) 849.  The batched form
// of order 4 takes 10 (3 x 256 x 256 x 192, a substep 4167 us, with 9 4246).
template <int ORDER>
constexpr int BACK_BLOCKS = ORDER == 2 ? 10 : 9;

template <int ORDER, bool CHUNKS>
__global__ void __launch_bounds__(CHUNKS ? 256 : 128, CHUNKS ? 2 : BACK_BLOCKS<ORDER>) k_line(Geo G, SolveBatch B)
{
    line_body<ORDER, CHUNKS>(G, B, blockIdx);
}

template <int ORDER, bool CHUNKS>
__global__ void __launch_bounds__(CHUNKS ? 256 : 128, CHUNKS ? 2 : 10) k_line_batch(const BatchRec<SolveBatch>* r, int n)
{
    uint3 b;
    const BatchRec<SolveBatch>& R = batch_locate(r, n, b);
    line_body<ORDER, CHUNKS>(R.G, R.A, b);
}

// Threads of a block, from the tuned solve_threads: at C chunks, the groups of
// 16 columns (8 C threads each) that fit 192 (128) or 96 (64) threads, at
// least one; for the back sweep the number of columns.
int line_threads(const Geo& G)
{
    if (!G.partitioned) return G.shape.solve_threads;
    const int C = line_chunk_count(G.nz);
    return std::max(1, line_batch_threads(G) / (8 * C)) * 8 * C;
}

// Threads of a batched launch's blocks, the same for every member's C; those
// beyond a member's line_threads have no chunk.
int line_batch_threads(const Geo& G)
{
    if (!G.partitioned) return G.shape.solve_threads;
    static_assert(8 * line_chunk_count(LINE_MAX_ROWS) <= 96, "a group of columns of the tallest member fits");
    return G.shape.solve_threads == 64 ? 96 : 192;
}

dim3 grid_line(const Geo& G)
{
    const int nt = line_threads(G);
    const int cols = G.partitioned ? 2 * line_lanes(nt, line_chunk_count(G.nz)) : nt;
    return dim3((unsigned) ((G.plane + cols - 1) / cols), 4);
}

// groups of columns with a column sum each, whatever the block size
long long line_groups(const Geo& G)
{
    const int cols = G.partitioned ? 16 : 32;
    return (G.plane + cols - 1) / cols;
}

size_t line_smem(const Geo& G)
{
    if (!G.partitioned) return 0;
    const int C = line_chunk_count(G.nz), H = G.order == 2 ? 1 : 3, lanes = line_lanes(line_threads(G), C);
    // two sets of boundary values; the first holds three rows at the top
    return (size_t) C * (line_chunk_stride(G.order) + 2 * line_mat_stride(G.order)) * sizeof(double)
         + (size_t) (std::max(C * H, 3) + C * H) * lanes * sizeof(double2);
}

void launch_line(const Geo& G, const SolveBatch& B, cudaStream_t st)
{
    const dim3 grd = grid_line(G);
    const int nt = line_threads(G);
    const size_t sm = line_smem(G);
    if (G.order == 2) {
        if (sm) k_line<2, true><<<grd, nt, sm, st>>>(G, B);
        else k_line<2, false><<<grd, nt, 0, st>>>(G, B);
    } else {
        if (sm) k_line<4, true><<<grd, nt, sm, st>>>(G, B);
        else k_line<4, false><<<grd, nt, 0, st>>>(G, B);
    }
}

void launch_control(const ControlArgs& A, cudaStream_t st)
{
    k_control<<<2 * LINE_STATS, CONTROL_THREADS, 0, st>>>(A);
}

void launch_mass_control(const MassArgs& M, cudaStream_t st)
{
    k_mass_control<<<1, 32, 0, st>>>(M);
}

void launch_line_batch(const BatchLaunch& L, int key, cudaStream_t st)
{
    auto r = static_cast<const BatchRec<SolveBatch>*>(L.recs);
    switch (key) {
    case 2: k_line_batch<2, false><<<L.blocks, L.block, 0, st>>>(r, L.n); break;
    case 4: k_line_batch<4, false><<<L.blocks, L.block, 0, st>>>(r, L.n); break;
    case 18: k_line_batch<2, true><<<L.blocks, L.block, L.smem, st>>>(r, L.n); break;
    default: k_line_batch<4, true><<<L.blocks, L.block, L.smem, st>>>(r, L.n); break;
    }
}

void launch_control_batch(const BatchLaunch& L, cudaStream_t st)
{
    k_control_batch<<<L.blocks, CONTROL_THREADS, 0, st>>>(static_cast<const BatchRec<ControlArgs>*>(L.recs), L.n);
}

}  // namespace cf
