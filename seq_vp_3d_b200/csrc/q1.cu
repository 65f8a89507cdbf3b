// Fused per-cell Q1 kernels of the certified-registration energy (FP64 plain form):
//   warp_kernel          cubic B-spline value (+ gradient) at X + u, image and proximity energy sums
//   cell_soft_kernel     JD/curl penalties against u_ref and their stable changes, from the closed27 J
//   cell_barrier_kernel  localized barrier, its change and violations of the cells near the activation
//   cell_grad_kernel     per-cell vertex gradients of the soft penalties -> SoA locals; cell_grad_barrier_kernel adds
//                        the barrier's
//   gather_kernel        atomic-free node gather in fixed vertex order, plus the node terms
//   ggn kernels, node JD measure, global closed27 cubic root; the mixed form's float32 cell kernels
// Reference: jd_curl/three_d/{residuals.py, linearization.py, energy_comparison.py, interpolation.py,
// solvers/jd_affine.py, solvers/global_jd_step.py}.
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "pair.cuh"
#include "q1_closed.cuh"

namespace svp {
namespace {

constexpr int CT = 128;      // threads per block of the cell kernels
constexpr int CELL_PER_SM = 8;

// ============================================================================================== spline sampler
struct SplineRef {
    const double *c;
    const double *t[3];    // x, y, z knots
    const double *rcp[3];  // per span, the reciprocals of the knot differences cubic_basis divides by (6 per span)
    long long n[3];        // nx, ny, nz coefficients per axis
    double x0[3], ih[3];
};

// The span s with t[s] <= x < t[s+1] (clamped to [3, n-1]): a first guess from the uniform node spacing, then the
// knot comparisons decide (so the guess's rounding never matters).
__device__ __forceinline__ int find_span(const double *__restrict__ t, long long n, double x, double x0, double ih) {
    long long i = (long long)floor((x - x0) * ih);
    long long s = i + 2;
    s = s < 3 ? 3 : (s > n - 1 ? n - 1 : s);
    while (s < n - 1 && __ldg(t + s + 1) <= x) s++;
    while (s > 3 && __ldg(t + s) > x) s--;
    return (int)s;
}

// backends/spline.py:12 cubic_basis: Cox-de Boor values and derivatives of the 4 B-splines on the span.  The
// denominators are knot differences (right + left = t[s+r+1] - t[s+1-d+r] up to rounding), so their reciprocals are
// tabled per span and the divisions become multiplies (a relative change of one rounding, inside the float64
// contract's 1e-12).  The derivative's denominators are those of degree 3, so 6 reciprocals do, read as 3 pairs: a
// warp's lanes stand on 32 x spans, and each load of the x row touches every line of the 32 rows.
__device__ __forceinline__ void cubic_basis(const double *__restrict__ t, const double *__restrict__ rcp, int s,
                                            double x, double B[4], double dB[4]) {
    const double2 *R2 = reinterpret_cast<const double2 *>(rcp + 6 * (long long)s);
    const double2 r01 = __ldg(R2), r23 = __ldg(R2 + 1), r45 = __ldg(R2 + 2);
    const double R[6] = {r01.x, r01.y, r23.x, r23.y, r45.x, r45.y};
    double b[4] = {1., 0., 0., 0.}, q[3];
#pragma unroll
    for (int degree = 1; degree <= 3; degree++) {
        double nb[4];
        double saved = 0.;
#pragma unroll
        for (int r = 0; r < degree; r++) {
            double right = __ldg(t + s + r + 1) - x;
            double left = x - __ldg(t + s + 1 - degree + r);
            double temp = b[r] * R[(degree - 1) * degree / 2 + r];
            nb[r] = saved + right * temp;
            saved = left * temp;
        }
        nb[degree] = saved;
#pragma unroll
        for (int r = 0; r <= degree; r++) b[r] = nb[r];
        if (degree == 2) { q[0] = b[0]; q[1] = b[1]; q[2] = b[2]; }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) B[k] = b[k];
    // 3 q_(k-1) R - 3 q_k R, the first product fused: the mixed form rounds the image gradient to float32, where a
    // change of the last float64 bit can show as one of the last float32 bit
    const double d0 = 3. * q[0] * R[3], d1 = 3. * q[1] * R[4], d2 = 3. * q[2] * R[5];
    dB[0] = -d0;
    dB[1] = fma(3. * q[0], R[3], -d1);
    dB[2] = fma(3. * q[1], R[4], -d2);
    dB[3] = d2;
}

__device__ __forceinline__ void prefetch_l1(const void *p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// value and (optionally) xyz gradient at physical point (x, y, z)
template <bool GRAD>
__device__ __forceinline__ double spline_eval(const SplineRef &S, double px, double py, double pz, double g[3]) {
    int sx = find_span(S.t[0], S.n[0], px, S.x0[0], S.ih[0]);
    int sy = find_span(S.t[1], S.n[1], py, S.x0[1], S.ih[1]);
    int sz = find_span(S.t[2], S.n[2], pz, S.x0[2], S.ih[2]);
    const long long nx = S.n[0], plane = S.n[1] * nx;
    const double *c = S.c + (long long)(sz - 3) * plane + (long long)(sy - 3) * nx + (sx - 3);
    // the first plane's 16 coefficients are on their way while the bases are formed, then a plane ahead
    double f[16];
    auto fetch = [&](const double *p) {
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int k = 0; k < 4; k++) f[4 * j + k] = __ldg(p + j * nx + k);
    };
    fetch(c);
    double bx[4], dx[4], by[4], dy[4], bz[4], dz[4];
    cubic_basis(S.t[0], S.rcp[0], sx, px, bx, dx);
    cubic_basis(S.t[1], S.rcp[1], sy, py, by, dy);
    cubic_basis(S.t[2], S.rcp[2], sz, pz, bz, dz);
    double val = 0., gx = 0., gy = 0., gz = 0.;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        double pv = 0., px_ = 0., py_ = 0.;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const double c0 = f[4 * j], c1 = f[4 * j + 1], c2 = f[4 * j + 2], c3 = f[4 * j + 3];
            double rv = c0 * bx[0] + c1 * bx[1] + c2 * bx[2] + c3 * bx[3];
            pv += by[j] * rv;
            if (GRAD) {
                double rd = c0 * dx[0] + c1 * dx[1] + c2 * dx[2] + c3 * dx[3];
                px_ += by[j] * rd;
                py_ += dy[j] * rv;
            }
        }
        if (i < 3) fetch(c + (i + 1) * plane);
        val += bz[i] * pv;
        if (GRAD) {
            gx += bz[i] * px_;
            gy += bz[i] * py_;
            gz += dz[i] * pv;
        }
    }
    if (GRAD) { g[0] = gx; g[1] = gy; g[2] = gz; }
    return val;
}

__device__ __forceinline__ double node_weight(long long x, long long y, long long z, const Q1Const &q) {
    double tx = (x == 0 || x == q.nx - 1) ? .5 : 1.;
    double ty = (y == 0 || y == q.ny - 1) ? .5 : 1.;
    double tz = (z == 0 || z == q.nz - 1) ? .5 : 1.;
    return ((q.omega * tz) * ty) * tx;
}

// warped image at X + u (+ gradient), and the image / proximity energy sums (before the 1/2, lambda/2 factors)
template <bool GRAD>
__global__ void __launch_bounds__(256) warp_kernel(Q1Const q, SplineRef S, const double *__restrict__ u,
                                                   const double *__restrict__ fixed, const double *__restrict__ uref,
                                                   double *__restrict__ warped, double *__restrict__ image_grad,
                                                   dd *partial) {
    dd acc[2] = {{0., 0.}, {0., 0.}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nnode;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.nx, q.ny, x, y, z);
        double ux = u[3 * i], uy = u[3 * i + 1], uz = u[3 * i + 2];
        double px = (q.x0[0] + q.h[0] * (double)x) + ux;
        double py = (q.x0[1] + q.h[1] * (double)y) + uy;
        double pz = (q.x0[2] + q.h[2] * (double)z) + uz;
        double g[3];
        double w = spline_eval<GRAD>(S, px, py, pz, g);
        warped[i] = w;
        if (GRAD) {
            image_grad[3 * i] = g[0];
            image_grad[3 * i + 1] = g[1];
            image_grad[3 * i + 2] = g[2];
        }
        if (partial) {
            double qw = node_weight(x, y, z, q);
            double d = w - fixed[i];
            double e0 = ux - uref[3 * i], e1 = uy - uref[3 * i + 1], e2 = uz - uref[3 * i + 2];
            acc[0] = dd_add_d(acc[0], qw * d * d);
            acc[1] = dd_add_d(acc[1], qw * (e0 * e0 + e1 * e1 + e2 * e2));
        }
    }
    if (partial) block_reduce_dd<2>(acc, partial);
}

__global__ void __launch_bounds__(256) node_energy_kernel(Q1Const q, const double *__restrict__ u,
                                                          const double *__restrict__ warped,
                                                          const double *__restrict__ fixed,
                                                          const double *__restrict__ uref, dd *partial) {
    dd acc[2] = {{0., 0.}, {0., 0.}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nnode;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.nx, q.ny, x, y, z);
        double qw = node_weight(x, y, z, q);
        double d = warped[i] - fixed[i];
        double e0 = u[3 * i] - uref[3 * i], e1 = u[3 * i + 1] - uref[3 * i + 1], e2 = u[3 * i + 2] - uref[3 * i + 2];
        acc[0] = dd_add_d(acc[0], qw * d * d);
        acc[1] = dd_add_d(acc[1], qw * (e0 * e0 + e1 * e1 + e2 * e2));
    }
    block_reduce_dd<2>(acc, partial);
}

__global__ void __launch_bounds__(256) sample_points_kernel(SplineRef S, const double *__restrict__ pts, long long n,
                                                            double *__restrict__ value, double *__restrict__ grad) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        double g[3];
        if (grad) {
            value[i] = spline_eval<true>(S, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], g);
            grad[3 * i] = g[0]; grad[3 * i + 1] = g[1]; grad[3 * i + 2] = g[2];
        } else {
            value[i] = spline_eval<false>(S, pts[3 * i], pts[3 * i + 1], pts[3 * i + 2], g);
        }
    }
}

// ============================================================================================== cell helpers
// Kernels with 27-point tables keep them in a per-thread slice of dynamic shared memory (slice k at
// smem[k * blockDim.x + threadIdx.x]: bank-conflict free); the edges of the fields stay in registers.  Local memory
// is touched by cell_grad_kernel (64 bytes of spills) and cell_ggn_hvp_kernel (148).
constexpr int CS = 64;     // threads per block of the shared-memory cell kernels

__device__ __forceinline__ void load_edges(const double *__restrict__ u, long long n0, const Q1Const &q,
                                           double E[3][4][3]) {
    double v[8][3];
    load_cell(u, n0, q, v);
    cell_edges(v, E);
}
template <class R>
__device__ __forceinline__ void zero_slice(R *sl, int T, int n) {
    for (int k = 0; k < n; k++) sl[k * T] = R(0);
}
// S[j][s][t][r] += f[r][j] at point (ix, iy, iz): j = 0 -> (iy, iz), j = 1 -> (ix, iz), j = 2 -> (ix, iy)
template <class R>
__device__ __forceinline__ void add_flux(R *sl, int T, int ix, int iy, int iz, const R f[3][3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
        sl[((iy * 3 + iz) * 3 + r) * T] += f[r][0];
        sl[(27 + (ix * 3 + iz) * 3 + r) * T] += f[r][1];
        sl[(54 + (ix * 3 + iy) * 3 + r) * T] += f[r][2];
    }
}
// adjoint of the edge interpolation: adds the fluxes S (add_flux) from the slice to the vertex values L
template <class R, class C>
__device__ __forceinline__ void scatter_slice(const R *sl, int T, const C n[3], const C m[3], const C ih[3],
                                              R L[8][3]) {
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
            R e[4] = {R(0), R(0), R(0), R(0)};
#pragma unroll
            for (int s = 0; s < 3; s++) {
                R t0 = R(0), t1 = R(0);
#pragma unroll
                for (int t = 0; t < 3; t++) {
                    R v = sl[(27 * j + (s * 3 + t) * 3 + r) * T] * (R)ih[j];
                    t0 += (R)m[t] * v;
                    t1 += (R)n[t] * v;
                }
                e[0] += (R)m[s] * t0;
                e[1] += (R)n[s] * t0;
                e[2] += (R)m[s] * t1;
                e[3] += (R)n[s] * t1;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                int lo = k & 1, hi = k >> 1;
                int a = j == 0 ? 2 * lo + 4 * hi : (j == 1 ? lo + 4 * hi : lo + 2 * hi);
                L[a | (1 << j)][r] += e[k];
                L[a][r] -= e[k];
            }
        }
}

// ============================================================================================== cell energies
// The JD and curl penalties of a state against u_ref (ENERGY) and their stable changes from a base (DIFF), one cell
// per thread on its closed27 J (q1_closed.cuh): per cell sum w (J - Jr)^2 and sum w |C - Cr|^2, and the changes
// d (2 r - d) in Legendre and Hadamard coefficients (r the state's residual, d the change from the base; the
// difference of the squares without cancelling them).  Block sums in double-double; a cell's values do not depend on
// which of the two parts is compiled in.
//
// Bound: FP64 issue.  About 2,000 FP64 instructions per cell with both parts (J of three fields at 27 points each 11
// operations, edges and averages 162, two Legendre transforms 108); the Gauss27 form took 6,200.  The 27 J - 1, the
// residual's coefficients and its curl's wait in the thread's shared slice (72 doubles: one access costs as much as four
// FP64 instructions, so tables that are used at once stay in registers).  Trial on 256^3: 11.20 -> 3.04 ms per launch,
// 2.96 with the curl taken from differences of the fields; FP64 pipe 64% busy; two warps per scheduler (255 registers) leave its dependency stalls.  Three warps
// (168 registers, 800 bytes of spills) took 5.0 ms, loads of the next field before this field's points 3.36 ms.
//
// flags[c]: bit 0, some closed27 J of the state may be below the activation; bit 1, some of the base may be.
// cell_barrier_kernel evaluates the barrier of those cells; elsewhere it and its change are zero.  A cell with a
// column that is not finite is flagged too.
constexpr int kEnergySlots = 27, kDiffSlots = 72;
template <bool ENERGY, bool DIFF>
__global__ void __launch_bounds__(CS) cell_soft_kernel(Q1Const q, const double *__restrict__ ua,
                                                       const double *__restrict__ ub,
                                                       const double *__restrict__ uref, dd *pe, dd *pd,
                                                       uint8_t *__restrict__ flags,
                                                       uint8_t *__restrict__ trial_act) {
    extern __shared__ double smem[];
    double *sJ = smem + threadIdx.x;
    const int T = blockDim.x;
    double *sR = sJ + 27 * T, *sX = sJ + 54 * T;
    dd acc[2] = {{0., 0.}, {0., 0.}}, dif[2] = {{0., 0.}, {0., 0.}};
    const double wj = .5 * q.mu * q.omega, wc = .5 * q.nu * q.omega, low = near_bound(q.act);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const long long n0 = cell_node0(c, q);
        Columns C;
        {
            double v[8][3], w[8][3], k[18];
            load_cell(ub, n0, q, v);
            load_cell(uref, n0, q, w);
            curl_difference(v, w, q, k);
            if (ENERGY)
                acc[1] = dd_add_d(acc[1], __dmul_rn(q.omega, curl_sum([&](int i, double &a) {
                                                        a = __fma_rn(k[i], k[i], a);
                                                    })));
            if (DIFF)
#pragma unroll
                for (int i = 0; i < 18; i++) sX[i * T] = k[i];
            vertex_columns(w, q, C);
            closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3],
                                 const double (&Z)[3]) { sJ[p * T] = det_minus_one(X, Y, Z); });
        }
        unsigned char flag = 0;
        {
            load_columns(ub, n0, q, C);
            double r[27];
            bool near = false;
            closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3],
                                 const double (&Z)[3]) {
                const double J = det_minus_one(X, Y, Z);
                near |= !(J >= low);
                r[p] = __dsub_rn(J, sJ[p * T]);
                if (DIFF) sJ[p * T] = J;
            });
            if (near) flag = 1;
            legendre27(r);
            if (ENERGY)
                acc[0] = dd_add_d(acc[0], __dmul_rn(q.omega, legendre_sum([&](int i, double &a) {
                                                        a = __fma_rn(r[i], r[i], a);
                                                    })));
            if (DIFF)
#pragma unroll
                for (int i = 0; i < 27; i++) sR[i * T] = r[i];
        }
        if (DIFF) {
            double v[8][3], w[8][3], k[18], d[27];
            load_cell(ub, n0, q, v);
            load_cell(ua, n0, q, w);
            curl_difference(v, w, q, k);
            dif[1] = dd_add_d(dif[1], __dmul_rn(wc, curl_sum([&](int i, double &a) {
                                                    a = __fma_rn(k[i], __fma_rn(2., sX[i * T], -k[i]), a);
                                                })));
            vertex_columns(w, q, C);
            bool near = false;
            closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3],
                                 const double (&Z)[3]) {
                const double J = det_minus_one(X, Y, Z);
                near |= !(J >= low);
                d[p] = __dsub_rn(sJ[p * T], J);
            });
            if (near) flag |= 2;
            legendre27(d);
            dif[0] = dd_add_d(dif[0], __dmul_rn(wj, legendre_sum([&](int i, double &a) {
                                                    a = __fma_rn(d[i], __fma_rn(2., sR[i * T], -d[i]), a);
                                                })));
        }
        flags[c] = flag;
        if (trial_act) trial_act[c] = 0;
    }
    // a J that is not finite need not lie below the bound, but leaves no finite sum: then flag the cells it came from
    // (checked per cell in the loop above, the trial on 256^3 took 3.11 in place of 3.06 ms)
    if (!finite64(DIFF ? dif[0].hi : acc[0].hi))
        for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
             c += (long long)gridDim.x * blockDim.x) {
            Columns C;
            load_columns(ub, cell_node0(c, q), q, C);
            bool finite = finite_columns(C);
            if (DIFF && finite) {
                load_columns(ua, cell_node0(c, q), q, C);
                finite = finite_columns(C);
            }
            if (!finite) flags[c] = 3;
        }
    if (ENERGY) block_reduce_dd<2>(acc, pe);
    if (ENERGY && DIFF) __syncthreads();     // the two reductions share block_reduce_dd's shared array
    if (DIFF) block_reduce_dd<2>(dif, pd);
}

// Per-cell vertex values -> SoA locals L[(a * 3 + r) * ncell + c].
template <class R>
__device__ __forceinline__ void store_locals(R *__restrict__ L, long long c, long long ncell, const R v[8][3]) {
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int r = 0; r < 3; r++) L[(long long)(a * 3 + r) * ncell + c] = v[a][r];
}

// ============================================================================================== flagged cells
// The plain form's barrier kernels: a block scans the flags of its cells (kScan groups of blockDim cells at a time,
// groups dealt out over the grid), queues the flagged ones in cell order and hands up to blockDim of them to
// body(n, queue).  Inside, the J of a cell belong to one thread and the n x 27 points are spread over the block: a
// barrier point is a long dependency chain (a logarithm and a division), so a thread that walks the 27 points of
// its cell leaves the SM idle (the trial's barrier on 48^3, 3.4% of its cells flagged: 37 us, spread 16 us; on 256^3
// 606 -> 496 us).  The assignment is the same on every run, so the threads' sums are deterministic.
constexpr int BT = 128;               // threads per block of these kernels
constexpr int kScan = 4;
template <class Body>
__device__ __forceinline__ void for_flagged_blocks(const Q1Const &q, const uint8_t *__restrict__ flags,
                                                   long long *queue, Body &&body) {
    __shared__ int counts[kScan][BT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ngroup = (int)((q.ncell + BT - 1) / BT);
    int n = 0;                         // queued cells, the same in every thread
    for (int k = blockIdx.x; k < ngroup || n > 0;) {
        while (n < BT && k < ngroup) {
            unsigned m[kScan];
#pragma unroll
            for (int j = 0; j < kScan; j++) {
                const long long c = (long long)(k + j * (int)gridDim.x) * BT + threadIdx.x;
                m[j] = __ballot_sync(0xFFFFFFFFu, c < q.ncell && flags[c] != 0);
                if (lane == 0) counts[j][warp] = __popc(m[j]);
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kScan; j++) {
                int at = n;
                for (int w = 0; w < BT / 32; w++) {
                    if (w == warp && ((m[j] >> lane) & 1u))
                        queue[at + __popc(m[j] & ((1u << lane) - 1u))] =
                            (long long)(k + j * (int)gridDim.x) * BT + threadIdx.x;
                    at += counts[j][w];
                    if (w == BT / 32 - 1) n = at;
                }
            }
            k += kScan * (int)gridDim.x;
            __syncthreads();
        }
        const int take = n < BT ? n : BT;
        if (take) body(take);
        __syncthreads();
        // at most kScan blocks of leftovers: move them to the front, one block at a time
        for (int i = take; i < n; i += BT) {
            const int at = i + threadIdx.x;
            const long long c = at < n ? queue[at] : 0;
            __syncthreads();
            if (at < n) queue[at - take] = c;
            __syncthreads();
        }
        n -= take;
    }
}
constexpr int kBlockQueue = (kScan + 1) * BT;
// Calls f(p, l) for the points p < 27 of the n queued cells, spread over the block (the cells rounded up to a power of
// two, so a point's indices are a shift and a mask).
template <class F>
__device__ __forceinline__ void for_block_points(int n, F &&f) {
    const int shift = 32 - __clz(n - 1), l = threadIdx.x & ((1 << shift) - 1);
    if (l >= n) return;
    for (int p = threadIdx.x >> shift; p < 27; p += BT >> shift) f(p, l);
}
unsigned flagged_blocks(const Q1Const &q) { return blocks_for(q.ncell, BT, 4); }
// cell_barrier_kernel's 168 registers let three blocks stand on an SM; a fourth ran alone in a second wave (0.54 -> 0.37
// ms on 256^3, 17 -> 13 us on 48^3).  One grid for its three forms: a sum's order depends on it.
unsigned cell_barrier_blocks(const Q1Const &q) { return blocks_for(q.ncell, BT, 3); }

// ============================================================================================== cell gradients
// Vertex values of the soft penalties' gradient (mu_scale, nu_scale: 1 or 0), one cell per thread on its closed27 J
// (q1_closed.cuh): the JD part's derivative by J at the 27 points is the 1D mass matrices applied to J - Jr, and one
// adjoint pass of J carries it to the edge columns, where the curl part's Hadamard adjoint joins.  flags (when the
// state has no mask): 1 for the cells with some closed27 J that may be below the activation, for cell_grad_barrier_kernel.
//
// Bound: FP64 issue (about 2,100 FP64 instructions per cell, the adjoint pass 27 x 24 of them; the Gauss27 form took
// 4,500 and kept 81 flux sums in shared memory).  160x192x224: 3.06 -> 1.36 ms per launch.  The barrier's slopes stay
// in their own kernel: evaluated here, on points packed over the warp, they cost 0.50 ms where that kernel takes 0.18
// (a few warps per scheduler cannot hide their latency).
__global__ void __launch_bounds__(CS) cell_grad_kernel(Q1Const q, const double *__restrict__ u,
                                                       const double *__restrict__ uref, double mu_scale,
                                                       double nu_scale, double *__restrict__ L1,
                                                       uint8_t *__restrict__ flags) {
    extern __shared__ double smem[];
    double *sJ = smem + threadIdx.x;
    const int T = blockDim.x;
    double *sC = sJ + 27 * T;
    // the mass matrices' 30 per axis and the quadrature's volume
    const double wj = q.mu * mu_scale * q.omega * (1. / 27000.), wc = q.nu * nu_scale * q.omega;
    const double low = near_bound(q.act);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const long long n0 = cell_node0(c, q);
        Columns C, G;
        {
            double v[8][3], w[8][3], k[18];
            load_cell(u, n0, q, v);
            load_cell(uref, n0, q, w);
            curl_difference(v, w, q, k);
#pragma unroll
            for (int i = 0; i < 18; i++) sC[i * T] = k[i];
            vertex_columns(w, q, C);
            closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3],
                                 const double (&Z)[3]) { sJ[p * T] = det_minus_one(X, Y, Z); });
        }
        load_columns(u, n0, q, C);
        {
            double r[27];
            bool near = false;
            closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3],
                                 const double (&Z)[3]) {
                const double J = det_minus_one(X, Y, Z);
                near |= !(J >= low);
                r[p] = __dsub_rn(J, sJ[p * T]);
            });
            mass27(r);
            if (flags) flags[c] = near || !finite64(r[0]) ? 1 : 0;     // r[0] has a share of all 27
#pragma unroll
            for (int p = 0; p < 27; p++) sJ[p * T] = wj * r[p];
        }
        add_identity(C);
        closed_adjoint(C, G, [&](int p) { return sJ[p * T]; });
        {
            double k[18];
#pragma unroll
            for (int i = 0; i < 18; i++) k[i] = sC[i * T];
            curl_adjoint(k, wc, G);
        }
        double L[8][3];
        columns_to_vertices(G, q, L);
        store_locals(L1, c, q.ncell, L);
    }
}

// The flags alone, for a gradient without soft penalties.
__global__ void __launch_bounds__(CS) cell_flag_kernel(Q1Const q, const double *__restrict__ u,
                                                       uint8_t *__restrict__ flags) {
    const double low = near_bound(q.act);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        Columns C;
        load_columns(u, cell_node0(c, q), q, C);
        bool near = !finite_columns(C);
        closed_points(C, [&](int, int, int, int, const double (&X)[3], const double (&Y)[3], const double (&Z)[3]) {
            near |= !(det_minus_one(X, Y, Z) >= low);
        });
        flags[c] = near ? 1 : 0;
    }
}

// The barrier's vertex values of the flagged cells (the state's mask, or the cells cell_grad_kernel flags): b'(J) at
// the 27 points (zero above the activation) and the same adjoint pass; added to L1 and, with split, stored in L2 for
// every flagged cell.
__global__ void __launch_bounds__(BT) cell_grad_barrier_kernel(Q1Const q, const double *__restrict__ u,
                                                               const uint8_t *__restrict__ flags, bool split,
                                                               double *__restrict__ L1, double *__restrict__ L2) {
    extern __shared__ double smem[];
    __shared__ long long queue[kBlockQueue];
    const BarrierRule rule = barrier_rule(q);
    for_flagged_blocks(q, flags, queue, [&](int n) {
        const bool mine = (int)threadIdx.x < n;
        double *sl = smem + threadIdx.x;
        const long long c = mine ? queue[threadIdx.x] : 0;
        Columns C, G;
        bool some = false;
        if (mine) some = closed_jacobians(u, cell_node0(c, q), q, C, sl, BT);
        __syncthreads();
        for_block_points(n, [&](int p, int l) {
            const double J = smem[p * BT + l];
            smem[p * BT + l] = J < q.act ? barrier_slope(J, rule) : 0.;
        });
        __syncthreads();
        if (mine) {
            // a cell that is not finite has a gradient only where some point has a slope
            if (!some)
                for (int p = 0; p < 27; p++) some |= sl[p * BT] != 0.;
            load_columns<true>(u, cell_node0(c, q), q, C);     // again: 36 columns do not wait in registers
            closed_adjoint(C, G, [&](int p) { return sl[p * BT]; });
            double Lb[8][3];
            columns_to_vertices(G, q, Lb);
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) Lb[a][r] = some ? Lb[a][r] : 0.;
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) L1[(size_t)(3 * a + r) * q.ncell + c] += Lb[a][r];
            if (split) store_locals(L2, c, q.ncell, Lb);
        }
    });
}

// ============================================================================================== gather
struct GatherSpec {
    int nout;
    double ci[3], cp[3], c1[3], c2[3];  // coefficients of image, proximity, L1, L2 per output
    double *out[3];
};

// Free node (z, y, x): sum of the 8 cells' vertex values in fixed order a = 0..7, plus node terms.  With TWO,
// has2 marks the cells whose L2 values were written; the others' are zero (most cells have no barrier term: one byte
// is read for 24).
// Last nodes first: the cell kernel has just written the last cells' values, up to 126 MB of them are still in L2 (two
// float64 sets of 2.7 M cells 145 -> 136 us, two float32 ones of 6.7 M 344 -> 281 us; one float64 set of 6.7 M, 1.3 GB:
// no change at 315 us).
template <bool TWO, class LT>
__global__ void __launch_bounds__(256) gather_kernel(Q1Const q, GatherSpec g, const LT *__restrict__ L1,
                                                     const LT *__restrict__ L2,
                                                     const uint8_t *__restrict__ has2, const double *__restrict__ u,
                                                     const double *__restrict__ uref,
                                                     const double *__restrict__ warped,
                                                     const double *__restrict__ fixed,
                                                     const double *__restrict__ image_grad) {
    for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < q.nfree;
         j += (long long)gridDim.x * blockDim.x) {
        const long long i = q.nfree - 1 - j;
        long long x, y, z;
        unflatten3(i, q.fx, q.fy, x, y, z);
        x++; y++; z++;
        long long node = (z * q.ny + y) * q.nx + x;
        double qw = node_weight(x, y, z, q);
        double dimg = warped ? qw * (warped[node] - fixed[node]) : 0.;
        // the 8 cells' vertex values summed in the locals' type (float locals: one conversion per sum, not per term)
        LT t1[3] = {LT(0), LT(0), LT(0)}, t2[3] = {LT(0), LT(0), LT(0)};
        long long cell[8];
        uint8_t two[8], some = 0;
#pragma unroll
        for (int a = 0; a < 8; a++) {
            cell[a] = ((z - (a >> 2)) * q.cy + (y - ((a >> 1) & 1))) * q.cx + (x - (a & 1));
            if (TWO) {
                two[a] = has2[cell[a]];
                some |= two[a];
            }
        }
        if (L1)
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) t1[r] += L1[(long long)(a * 3 + r) * q.ncell + cell[a]];
        if (TWO && some)
#pragma unroll
            for (int a = 0; a < 8; a++)
                if (two[a])
#pragma unroll
                    for (int r = 0; r < 3; r++) t2[r] += L2[(long long)(a * 3 + r) * q.ncell + cell[a]];
        const double s1[3] = {(double)t1[0], (double)t1[1], (double)t1[2]};
        const double s2[3] = {(double)t2[0], (double)t2[1], (double)t2[2]};
#pragma unroll
        for (int r = 0; r < 3; r++) {
            double img = image_grad ? dimg * image_grad[3 * node + r] : 0.;
            double prox = uref ? q.lam * qw * (u[3 * node + r] - uref[3 * node + r]) : 0.;
#pragma unroll
            for (int k = 0; k < 3; k++)     // constant indices keep the spec in the parameter bank
                if (k < g.nout)
                    g.out[k][r * q.nfree + i] = ((g.ci[k] * img + g.cp[k] * prox) + g.c1[k] * s1[r]) + g.c2[k] * s2[r];
        }
    }
}

// ============================================================================================== GGN
// Per-cell diagonal contributions sum_p w_p l_a,r(p)^2 with l = sum_j A_rj D_j(p, a), A the cofactors of F.  D_j is
// +-1/h_j times the two other coordinates' linear shape values f, so with P, Q, R = the weighted A_r0, A_r1, A_r2 the
// eight vertices' l are +-f_y f_z P + f_x (+-f_z Q +- f_y R): 28 operations per point and row for all eight, where
// forming each vertex's D and dot product took 100.  The rule's columns are linear interpolations per plane and row.
// weight(p, ix, iy, iz): the factor of l (SQUARED: of l^2).
template <bool CLOSED, bool SQUARED, class Weight>
__device__ __forceinline__ void ggn_points(const Columns &C, const Q1Const &q, Weight &&weight, double (&out)[8][3]) {
    const double n[3] = {rule_n<CLOSED>(q, 0), rule_n<CLOSED>(q, 1), rule_n<CLOSED>(q, 2)};
    const double m[3] = {rule_m<CLOSED>(q, 0), rule_m<CLOSED>(q, 1), rule_m<CLOSED>(q, 2)};
#pragma unroll 1
    for (int iz = 0; iz < 3; iz++) {
        const double nz = rule_n<CLOSED>(q, iz), mz = rule_m<CLOSED>(q, iz);
        double X[3][3], Y[3][3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const double x0 = fma(nz, C.X[2][r] - C.X[0][r], C.X[0][r]), x1 = fma(nz, C.X[3][r] - C.X[1][r], C.X[1][r]);
            const double y0 = fma(nz, C.Y[2][r] - C.Y[0][r], C.Y[0][r]), y1 = fma(nz, C.Y[3][r] - C.Y[1][r], C.Y[1][r]);
            const double dx = x1 - x0, dy = y1 - y0;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                X[i][r] = fma(n[i], dx, x0);
                Y[i][r] = fma(n[i], dy, y0);
            }
        }
#pragma unroll
        for (int iy = 0; iy < 3; iy++) {
            double z0[3], dz[3];
#pragma unroll
            for (int r = 0; r < 3; r++) {
                z0[r] = fma(n[iy], C.Z[2][r] - C.Z[0][r], C.Z[0][r]);
                dz[r] = fma(n[iy], C.Z[3][r] - C.Z[1][r], C.Z[1][r]) - z0[r];
            }
#pragma unroll
            for (int ix = 0; ix < 3; ix++) {
                const double s = weight(9 * iz + 3 * iy + ix, ix, iy, iz);
                double F[3][3];      // rows of F
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    F[r][0] = X[iy][r];
                    F[r][1] = Y[ix][r];
                    F[r][2] = fma(n[ix], dz[r], z0[r]);
                }
                const double k0 = SQUARED ? q.ih[0] : s * q.ih[0], k1 = SQUARED ? q.ih[1] : s * q.ih[1],
                             k2 = SQUARED ? q.ih[2] : s * q.ih[2];
                const double fy[2] = {m[iy], n[iy]}, fz[2] = {mz, nz};
                const double fyz[2][2] = {{fy[0] * fz[0], fy[0] * fz[1]}, {fy[1] * fz[0], fy[1] * fz[1]}};
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    const int j = (r + 1) % 3, k = (r + 2) % 3;
                    const double P = k0 * (F[j][1] * F[k][2] - F[j][2] * F[k][1]);
                    const double Q = k1 * (F[j][2] * F[k][0] - F[j][0] * F[k][2]);
                    const double R = k2 * (F[j][0] * F[k][1] - F[j][1] * F[k][0]);
                    const double Qz[2] = {fz[0] * Q, fz[1] * Q}, Ry[2] = {fy[0] * R, fy[1] * R};
#pragma unroll
                    for (int bz = 0; bz < 2; bz++)
#pragma unroll
                        for (int by = 0; by < 2; by++) {
                            const double t1 = fyz[by][bz] * P;
                            const double t2 = (by ? Qz[bz] : -Qz[bz]) + (bz ? Ry[by] : -Ry[by]);
                            const double l0 = fma(m[ix], t2, -t1), l1 = fma(n[ix], t2, t1);
                            double &o0 = out[2 * by + 4 * bz][r], &o1 = out[1 + 2 * by + 4 * bz][r];
                            o0 = fma(SQUARED ? s * l0 : l0, l0, o0);
                            o1 = fma(SQUARED ? s * l1 : l1, l1, o1);
                        }
                }
            }
        }
    }
}

// The JD part at the Gauss points (weights w mu) plus the state-independent curl part q.ggn_curl.  flags (when the
// state has no mask): 1 for the cells with some closed27 J that may be below the activation.
// Bound: FP64 issue, about 3,300 FP64 instructions per cell (5,600 with a D per vertex): 128x144x128 0.78 -> 0.47
// ms per launch.
__global__ void __launch_bounds__(CS) cell_ggn_diag_kernel(Q1Const q, const double *__restrict__ u,
                                                           double *__restrict__ L, uint8_t *__restrict__ flags) {
    const double root = sqrt(q.mu * q.omega), low = near_bound(q.act);
    constexpr double side = 0.52704627669472988, centre = 2. / 3.;     // sqrt(5 / 18), sqrt(4 / 9)
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        Columns C;
        load_columns(u, cell_node0(c, q), q, C);
        bool near = false;
        if (flags)
            closed_points(C, [&](int, int, int, int, const double (&X)[3], const double (&Y)[3], const double (&Z)[3]) {
                near |= !(det_minus_one(X, Y, Z) >= low);
            });
        add_identity(C);
        double out[8][3];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) out[a][r] = q.ggn_curl[3 * a + r];
        ggn_points<false, false>(C, q, [&](int, int ix, int iy, int iz) {
            return root * (iz == 1 ? centre : side) * ((iy == 1 ? centre : side) * (ix == 1 ? centre : side));
        }, out);
        // a column that is not finite shows in two components of any vertex
        if (flags) flags[c] = near || !finite64(out[0][0] + out[0][1]) ? 1 : 0;
        store_locals(L, c, q.ncell, out);
    }
}

// GGN action on a node field vv (zero faces): Gauss JD/curl linearization + closed27 barrier curvature.
__global__ void __launch_bounds__(CS) cell_ggn_hvp_kernel(Q1Const q, const double *__restrict__ u,
                                                          const double *__restrict__ vv, double *__restrict__ L) {
    extern __shared__ double smem[];
    double *sl = smem + threadIdx.x;
    const int T = blockDim.x;
    const double cn[3] = {0., .5, 1.}, cm[3] = {1., .5, 0.};
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        long long n0 = cell_node0(c, q);
        double E[3][4][3], Ev[3][4][3], out[8][3];
        load_edges(u, n0, q, E);
        load_edges(vv, n0, q, Ev);
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) out[a][r] = 0.;
        zero_slice(sl, T, 81);
        sweep2<false>(E, Ev, q, [&](int p, int ix, int iy, int iz, const double (&V)[3][3],
                                    const double (&W)[3][3]) {
            double A[3][3], J, K[3];
            cofactor_det(V, A, J);
            double jd = 0.;
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int jj = 0; jj < 3; jj++) jd += A[r][jj] * W[r][jj];
            curl_of(W, K);
            const double gw = q.gw[p];
            jd *= q.mu * gw;
            double k0 = q.nu * gw * K[0], k1 = q.nu * gw * K[1], k2 = q.nu * gw * K[2];
            double f[3][3];
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int jj = 0; jj < 3; jj++) f[r][jj] = A[r][jj] * jd;
            f[2][1] += k0; f[1][2] -= k0;
            f[0][2] += k1; f[2][0] -= k1;
            f[1][0] += k2; f[0][1] -= k2;
            add_flux(sl, T, ix, iy, iz, f);
        });
        scatter_slice(sl, T, q.gn, q.gm, q.ih, out);
        zero_slice(sl, T, 81);
        bool any = false;
        sweep2<true>(E, Ev, q, [&](int, int ix, int iy, int iz, const double (&V)[3][3], const double (&W)[3][3]) {
            if (!(det_only(V) < q.act)) return;
            double A[3][3], J, b, b1, b2;
            cofactor_det(V, A, J);
            barrier_eval(J, q.act, q.delta, q.bw, b, b1, b2);
            double lj = 0.;
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int jj = 0; jj < 3; jj++) lj += A[r][jj] * W[r][jj];
            lj *= b2;
            double f[3][3];
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int jj = 0; jj < 3; jj++) f[r][jj] = A[r][jj] * lj;
            add_flux(sl, T, ix, iy, iz, f);
            any = true;
        });
        if (any) scatter_slice(sl, T, cn, cm, q.ih, out);
        store_locals(L, c, q.ncell, out);
    }
}

// node part of the GGN: q |b|^2 + lambda q (diagonal) or q b (b . v) + lambda q v (action)
template <class LT>
__global__ void __launch_bounds__(256) ggn_node_kernel(Q1Const q, const LT *__restrict__ L,
                                                       const double *__restrict__ image_grad,
                                                       const double *__restrict__ vv, double *__restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nfree;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.fx, q.fy, x, y, z);
        x++; y++; z++;
        long long node = (z * q.ny + y) * q.nx + x;
        double qw = node_weight(x, y, z, q);
        double s[3] = {0., 0., 0.};
#pragma unroll
        for (int a = 0; a < 8; a++) {
            long long c = ((z - (a >> 2)) * q.cy + (y - ((a >> 1) & 1))) * q.cx + (x - (a & 1));
#pragma unroll
            for (int r = 0; r < 3; r++) s[r] += (double)L[(long long)(a * 3 + r) * q.ncell + c];
        }
        const double *b = image_grad + 3 * node;
        if (vv) {
            const double *v = vv + 3 * node;
            double bv = b[0] * v[0] + b[1] * v[1] + b[2] * v[2];
#pragma unroll
            for (int r = 0; r < 3; r++) out[r * q.nfree + i] = (qw * b[r] * bv + q.lam * qw * v[r]) + s[r];
        } else {
#pragma unroll
            for (int r = 0; r < 3; r++) out[r * q.nfree + i] = (qw * b[r] * b[r] + q.lam * qw) + s[r];
        }
    }
}

// ============================================================================================== mixed form
// The direction pipeline in float32 (gradient, GGN diagonal): edge differences formed in float64 from the float64
// state and rounded once, grad u, cofactors, fluxes and the separable adjoint in float32, float32 locals gathered in
// float64.  The localized barrier stays float64, in separate kernels that visit only the flagged cells: cells active
// in the state's mask, or (without a mask) cells with some float32 closed27 J within kBarrierGuard of the
// activation.  There the whole closed27 sweep is redone in float64 from the float64 state (the plain form's J,
// cofactors and barrier values) and added to the cell's float32 locals, so the float32 kernels carry neither the
// float64 sweep nor its registers.
constexpr float kBarrierGuard = 1e-3f;
constexpr int CB = 128;               // threads per block of the float64 barrier kernels
constexpr int kFlagChunk = 256;       // consecutive cells a warp scans at a time for flagged cells

// Calls f(c, flags[c]) for the flagged cells (flags[c] != 0).  Warp w of the grid scans the chunks of kFlagChunk
// cells w, w + warps, ...; the flagged cells are queued in the warp's shared queue (64 entries) in cell order and
// handed to the lanes 32 at a time, so the float64 work runs on full warps whatever the flags' pattern, and every cell
// goes to the same lane on every run (the lanes' sums are deterministic).
template <class F>
__device__ __forceinline__ void for_flagged_cells(const Q1Const &q, const uint8_t *__restrict__ flags,
                                                  long long *queue, F &&f) {
    const int lane = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long nchunk = (q.ncell + kFlagChunk - 1) / kFlagChunk;
    long long k = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    long long b = k * kFlagChunk;
    int qn = 0;
    // a chunk's 256 flags are read once, 8 per lane (one 64-bit load where the chunk is whole and aligned), and the
    // flag of cell chunk + 32 j + l is byte l % 8 of lane 4 j + l / 8's word; cells past the end read as zero
    const bool wide = (reinterpret_cast<uintptr_t>(flags) & 7) == 0;
    unsigned long long word = 0;
    for (;;) {
        // fill the queue to a full warp's worth, or until the warp's chunks are exhausted
        while (qn < 32 && k < nchunk) {
            const long long c0 = k * kFlagChunk, hi = min(c0 + kFlagChunk, q.ncell), c = b + lane;
            if (b == c0) {
                const long long f0 = c0 + 8 * lane;
                if (wide && c0 + kFlagChunk <= q.ncell) {
                    word = *reinterpret_cast<const unsigned long long *>(flags + f0);
                } else {
                    word = 0;
#pragma unroll
                    for (int t = 0; t < 8; t++)
                        if (f0 + t < q.ncell) word |= (unsigned long long)flags[f0 + t] << (8 * t);
                }
            }
            const int j = (int)((b - c0) >> 5);
            const unsigned long long v = __shfl_sync(0xFFFFFFFFu, word, 4 * j + (lane >> 3));
            const bool on = c < hi && ((v >> (8 * (lane & 7))) & 0xFFull) != 0;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, on);
            if (on) queue[qn + __popc(m & ((1u << lane) - 1u))] = c;
            qn += __popc(m);
            b += 32;
            if (b >= hi) {
                k += warps;
                b = k * kFlagChunk;
            }
        }
        __syncwarp();
        if (qn == 0) break;
        const int take = qn < 32 ? qn : 32;
        const long long c = lane < take ? queue[lane] : -1;
        __syncwarp();
        if (lane + 32 < qn) queue[lane] = queue[lane + 32];
        __syncwarp();
        qn -= take;
        if (c >= 0) f(c, flags[c]);
    }
}
unsigned barrier_blocks(const Q1Const &q) {
    const long long nchunk = (q.ncell + kFlagChunk - 1) / kFlagChunk;
    return blocks_for(nchunk * 32, CB, 4);
}

__device__ __forceinline__ void load_edges_f32(const double *__restrict__ u, long long n0, const Q1Const &q,
                                               float E[3][4][3]) {
    double v[8][3];
    load_cell(u, n0, q, v);
    double E64[3][4][3];
    cell_edges(v, E64);
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
        for (int e = 0; e < 4; e++)
#pragma unroll
            for (int r = 0; r < 3; r++) E[j][e][r] = (float)E64[j][e][r];
}
// Float columns at the Gauss points from the interpolants along the lower other axis, which depend on one index each:
// lo[s], hi[s] are column<J>'s l0, l1 at node s, and P(s, t) = (m_t lo_s + n_t hi_s) / h.  The operations are column's,
// evaluated once per distinct value (513 per field for the 27 points, where column at every point takes 1,323).
template <int J>
__device__ __forceinline__ void lower_interpolants(const float (&E)[3][4][3], const Q1Const &q, float (&lo)[3][3],
                                                   float (&hi)[3][3]) {
#pragma unroll
    for (int s = 0; s < 3; s++) {
        const float ms = q.gmf[s], ns = q.gnf[s];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            lo[s][r] = ms * E[J][0][r] + ns * E[J][1][r];
            hi[s][r] = ms * E[J][2][r] + ns * E[J][3][r];
        }
    }
}
__device__ __forceinline__ void upper_value(const float (&lo)[3], const float (&hi)[3], float mt, float nt, float ih,
                                            float (&pre)[3], float (&out)[3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
        pre[r] = mt * lo[r] + nt * hi[r];
        out[r] = pre[r] * ih;
    }
}
// Visits the Gauss points in sweep's order with grad u and curl u in float: body(p, ix, iy, iz, V, C).  A curl
// component is one fused operation on its first term's value before that term's division by h.
template <class Row, class Body, class Plane>
__device__ __forceinline__ void gauss_points32(const float (&E)[3][4][3], const Q1Const &q, Row &&row, Body &&body,
                                               Plane &&plane) {
    float xl[3][3], xh[3][3], yl[3][3], yh[3][3], zl[3][3], zh[3][3];
    lower_interpolants<0>(E, q, xl, xh);
    lower_interpolants<1>(E, q, yl, yh);
    lower_interpolants<2>(E, q, zl, zh);
#pragma unroll 1
    for (int iz = 0; iz < 3; iz++) {
        const float nz = q.gnf[iz], mz = q.gmf[iz];
        float Y[3][3], yp[3][3];
#pragma unroll
        for (int ix = 0; ix < 3; ix++) upper_value(yl[ix], yh[ix], mz, nz, q.ihf[1], yp[ix], Y[ix]);
#pragma unroll
        for (int iy = 0; iy < 3; iy++) {
            float X[3], xp[3];
            upper_value(xl[iy], xh[iy], mz, nz, q.ihf[0], xp, X);
#pragma unroll
            for (int ix = 0; ix < 3; ix++) {
                float Z[3], zp[3];
                upper_value(zl[ix], zh[ix], q.gmf[iy], q.gnf[iy], q.ihf[2], zp, Z);
                const float V[3][3] = {{X[0], Y[ix][0], Z[0]}, {X[1], Y[ix][1], Z[1]}, {X[2], Y[ix][2], Z[2]}};
                const float C[3] = {__fmaf_rn(yp[ix][2], q.ihf[1], -Z[1]), __fmaf_rn(zp[0], q.ihf[2], -X[2]),
                                    __fmaf_rn(xp[1], q.ihf[0], -Y[ix][0])};
                body(9 * iz + 3 * iy + ix, ix, iy, iz, V, C);
            }
            row(iy, iz);
        }
        plane(iz);
    }
}

// The soft part (JD, curl penalties) of the gradient locals.  flags (when the state has no mask): 1 for the cells with
// some float32 closed27 J within the guard.
// Bound: FP32 issue.  The reference's J and curl wait in the thread's slice (108 floats); the flux sums along x and y
// complete within a row and a plane and are stored once, those along z stay in registers (81 sums read, added to and
// written back at every point took 486 shared accesses).  Every sum adds the same terms in the same order as before,
// so the values are bitwise those of the kernel that swept both fields together.  160x192x224: 1.63 -> 1.18 ms
// (254 registers; 168 took 1.37 ms, 128 with spills 1.60).
constexpr int kGrad32Slots = 108 + 54;
__global__ void __launch_bounds__(CS, 4) cell_grad32_kernel(Q1Const q, const double *__restrict__ u,
                                                            const double *__restrict__ uref, double mu_scale,
                                                            double nu_scale, float *__restrict__ L1,
                                                            uint8_t *__restrict__ flags) {
    extern __shared__ float smemf[];
    float *ref = smemf + threadIdx.x;
    const int T = blockDim.x;
    float *sl = ref + 108 * T;
    const float mu = (float)(q.mu * mu_scale), nu = (float)(q.nu * nu_scale);
    const float guard = (float)q.act + kBarrierGuard;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const long long n0 = cell_node0(c, q);
        float L[8][3];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) L[a][r] = 0.f;
        if (mu != 0.f || nu != 0.f) {
            float E[3][4][3];
            load_edges_f32(uref, n0, q, E);
            gauss_points32(E, q, [](int, int) {}, [&](int p, int, int, int, const float (&V)[3][3], const float (&C)[3]) {
                ref[(4 * p) * T] = det_only(V);
                ref[(4 * p + 1) * T] = C[0];
                ref[(4 * p + 2) * T] = C[1];
                ref[(4 * p + 3) * T] = C[2];
            }, [](int) {});
            load_edges_f32(u, n0, q, E);
            float SX[3] = {0.f, 0.f, 0.f}, SY[3][3], SZ[3][3][3];      // SZ[ix][iy][r]
#pragma unroll
            for (int i = 0; i < 9; i++)
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    SZ[i / 3][i % 3][r] = 0.f;
                    SY[i / 3][i % 3] = 0.f;
                }
            gauss_points32(E, q,
                [&](int iy, int iz) {
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        sl[((iy * 3 + iz) * 3 + r) * T] = SX[r];
                        SX[r] = 0.f;
                    }
                },
                [&](int p, int ix, int iy, int, const float (&V)[3][3], const float (&C)[3]) {
                    float A[3][3], J;
                    cofactor_det(V, A, J);
                    const float Jr = ref[(4 * p) * T];
                    const float gw = q.gwf[p];
                    const float jd = mu * gw * (J - Jr);
                    const float k0 = nu * gw * (C[0] - ref[(4 * p + 1) * T]), k1 = nu * gw * (C[1] - ref[(4 * p + 2) * T]),
                                k2 = nu * gw * (C[2] - ref[(4 * p + 3) * T]);
                    float f[3][3];
#pragma unroll
                    for (int r = 0; r < 3; r++)
#pragma unroll
                        for (int jj = 0; jj < 3; jj++) f[r][jj] = A[r][jj] * jd;
                    f[2][1] += k0; f[1][2] -= k0;
                    f[0][2] += k1; f[2][0] -= k1;
                    f[1][0] += k2; f[0][1] -= k2;
#pragma unroll
                    for (int r = 0; r < 3; r++) {
                        SX[r] += f[r][0];
                        SY[ix][r] += f[r][1];
                        SZ[ix][iy][r] += f[r][2];
                    }
                },
                [&](int iz) {
#pragma unroll
                    for (int ix = 0; ix < 3; ix++)
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            sl[(27 + (ix * 3 + iz) * 3 + r) * T] = SY[ix][r];
                            SY[ix][r] = 0.f;
                        }
                });
            // the adjoint of the edge interpolation, as scatter_slice
#pragma unroll
            for (int j = 0; j < 3; j++)
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int s = 0; s < 3; s++) {
                        float t0 = 0.f, t1 = 0.f;
#pragma unroll
                        for (int t = 0; t < 3; t++) {
                            const float v = (j < 2 ? sl[(27 * j + (s * 3 + t) * 3 + r) * T] : SZ[s][t][r]) * q.ihf[j];
                            t0 += q.gmf[t] * v;
                            t1 += q.gnf[t] * v;
                        }
                        e[0] += q.gmf[s] * t0;
                        e[1] += q.gnf[s] * t0;
                        e[2] += q.gmf[s] * t1;
                        e[3] += q.gnf[s] * t1;
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int lo = k & 1, hi = k >> 1;
                        const int a = j == 0 ? 2 * lo + 4 * hi : (j == 1 ? lo + 4 * hi : lo + 2 * hi);
                        L[a | (1 << j)][r] += e[k];
                        L[a][r] -= e[k];
                    }
                }
        }
        // without a mask, the cells with some float32 closed27 J within the guard are flagged for the barrier kernel
        if (flags) {
            float E[3][4][3];
            load_edges_f32(u, n0, q, E);
            bool near = false;
            sweep<true, float>(E, q, [&](int, int, int, int, const float (&V)[3][3]) {
                near |= det_only(V) < guard;
            });
            flags[c] = near ? 1 : 0;
        }
        store_locals(L1, c, q.ncell, L);
    }
}

// The barrier's locals of the flagged cells in float64: the closed27 sweep from the float64 state, J, b' and the
// cofactors in float64, the flux rounded to float32 and scattered as the soft kernel scatters its own; then added to
// the cell's locals (L1 += Lb) and, for the outer triple, stored apart (L2, for every flagged cell).
__global__ void __launch_bounds__(CB) cell_grad_barrier32_kernel(Q1Const q, const double *__restrict__ u,
                                                               const uint8_t *__restrict__ flags, bool split,
                                                               float *__restrict__ L1, float *__restrict__ L2) {
    extern __shared__ float smemf[];
    __shared__ long long queue[CB / 32][64];
    float *sl = smemf + threadIdx.x;
    const int T = blockDim.x;
    const float cn[3] = {0.f, .5f, 1.f}, cm[3] = {1.f, .5f, 0.f};
    const float ih[3] = {(float)q.ih[0], (float)q.ih[1], (float)q.ih[2]};
    for_flagged_cells(q, flags, queue[threadIdx.x >> 5], [&](long long c, uint8_t) {
        double E64[3][4][3];
        load_edges(u, cell_node0(c, q), q, E64);
        zero_slice(sl, T, 81);
        bool any = false;
        sweep<true>(E64, q, [&](int, int ix, int iy, int iz, const double (&V)[3][3]) {
            if (!(det_only(V) < q.act)) return;
            double A[3][3], J, b, b1, b2;
            cofactor_det(V, A, J);
            barrier_eval(J, q.act, q.delta, q.bw, b, b1, b2);
            float f[3][3];
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int jj = 0; jj < 3; jj++) f[r][jj] = (float)(A[r][jj] * b1);
            add_flux(sl, T, ix, iy, iz, f);
            any = true;
        });
        if (!any && !split) return;
        float Lb[8][3];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) Lb[a][r] = 0.f;
        scatter_slice(sl, T, cn, cm, ih, Lb);
        if (any)
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) L1[(size_t)(3 * a + r) * q.ncell + c] += Lb[a][r];
        if (split) store_locals(L2, c, q.ncell, Lb);
    });
}

// GGN diagonal contributions in float32 (Gauss JD/curl part); flags (when the state has no mask) as the gradient's.
__global__ void __launch_bounds__(CT, 4) cell_ggn_diag32_kernel(Q1Const q, const double *__restrict__ u,
                                                             float *__restrict__ L, uint8_t *__restrict__ flags) {
    const float guard = (float)q.act + kBarrierGuard;
    const float mu = (float)q.mu;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        const long long n0 = cell_node0(c, q);
        float E[3][4][3], out[8][3];
        load_edges_f32(u, n0, q, E);
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) out[a][r] = 0.f;
        sweep<false, float>(E, q, [&](int p, int ix, int iy, int iz, const float (&V)[3][3]) {
            float A[3][3], J;
            cofactor_det(V, A, J);
            const float gmu = q.gwf[p] * mu;
#pragma unroll
            for (int a = 0; a < 8; a++) {
                const int bx = a & 1, by = (a >> 1) & 1, bz = (a >> 2) & 1;
                const float fx = bx ? q.gnf[ix] : q.gmf[ix];
                const float fy = by ? q.gnf[iy] : q.gmf[iy];
                const float fz = bz ? q.gnf[iz] : q.gmf[iz];
                float D[3];
                D[0] = (bx ? q.ihf[0] : -q.ihf[0]) * fy * fz;
                D[1] = (by ? q.ihf[1] : -q.ihf[1]) * fx * fz;
                D[2] = (bz ? q.ihf[2] : -q.ihf[2]) * fx * fy;
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    float lj = A[r][0] * D[0] + A[r][1] * D[1] + A[r][2] * D[2];
                    out[a][r] += gmu * (lj * lj);
                }
            }
        });
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) out[a][r] += q.ggn_curlf[3 * a + r];
        if (flags) {
            bool near = false;
            sweep<true, float>(E, q, [&](int, int, int, int, const float (&V)[3][3]) { near |= det_only(V) < guard; });
            flags[c] = near ? 1 : 0;
        }
        store_locals(L, c, q.ncell, out);
    }
}

template <bool CLOSED>
__device__ __forceinline__ void point_D(const Q1Const &q, int ix, int iy, int iz, int a, double D[3]) {
    const int bx = a & 1, by = (a >> 1) & 1, bz = (a >> 2) & 1;
    const double fx = bx ? rule_n<CLOSED>(q, ix) : rule_m<CLOSED>(q, ix);
    const double fy = by ? rule_n<CLOSED>(q, iy) : rule_m<CLOSED>(q, iy);
    const double fz = bz ? rule_n<CLOSED>(q, iz) : rule_m<CLOSED>(q, iz);
    D[0] = (bx ? q.ih[0] : -q.ih[0]) * fy * fz;
    D[1] = (by ? q.ih[1] : -q.ih[1]) * fx * fz;
    D[2] = (bz ? q.ih[2] : -q.ih[2]) * fx * fy;
}

// The barrier curvature b'' lc^2 of the flagged cells in float64 (J, b'' and the cofactors lc from the float64
// state), rounded to float32 and added point by point in sweep order to the cell's locals.
__global__ void __launch_bounds__(CB) cell_ggn_barrier32_kernel(Q1Const q, const double *__restrict__ u,
                                                              const uint8_t *__restrict__ flags,
                                                              float *__restrict__ L) {
    __shared__ long long queue[CB / 32][64];
    for_flagged_cells(q, flags, queue[threadIdx.x >> 5], [&](long long c, uint8_t) {
        double E64[3][4][3];
        load_edges(u, cell_node0(c, q), q, E64);
        float out[8][3];
#pragma unroll
        for (int a = 0; a < 8; a++)
#pragma unroll
            for (int r = 0; r < 3; r++) out[a][r] = L[(size_t)(3 * a + r) * q.ncell + c];
        bool any = false;
        sweep<true>(E64, q, [&](int, int ix, int iy, int iz, const double (&V64)[3][3]) {
            if (!(det_only(V64) < q.act)) return;
            any = true;
            double A[3][3], J, b, b1, b2;
            cofactor_det(V64, A, J);
            barrier_eval(J, q.act, q.delta, q.bw, b, b1, b2);
#pragma unroll
            for (int a = 0; a < 8; a++) {
                double D[3];
                point_D<true>(q, ix, iy, iz, a, D);
#pragma unroll
                for (int r = 0; r < 3; r++) {
                    double lc = A[r][0] * D[0] + A[r][1] * D[1] + A[r][2] * D[2];
                    out[a][r] += (float)(b2 * lc * lc);
                }
            }
        });
        if (any) store_locals(L, c, q.ncell, out);
    });
}

// The plain form's barrier curvature of the flagged cells: b'' at the 27 points spread over the block, then each
// cell's squares by its own thread, added to its locals.
__global__ void __launch_bounds__(BT) cell_ggn_barrier_kernel(Q1Const q, const double *__restrict__ u,
                                                              const uint8_t *__restrict__ flags,
                                                              double *__restrict__ L) {
    extern __shared__ double smem[];
    __shared__ long long queue[kBlockQueue];
    for_flagged_blocks(q, flags, queue, [&](int n) {
        const bool mine = (int)threadIdx.x < n;
        const long long c = mine ? queue[threadIdx.x] : 0;
        Columns C;
        if (mine) closed_jacobians(u, cell_node0(c, q), q, C, smem + threadIdx.x, BT);
        __syncthreads();
        for_block_points(n, [&](int p, int l) {
            const double J = smem[p * BT + l];
            double b, b1, b2 = 0.;
            if (J < q.act) barrier_eval(J, q.act, q.delta, q.bw, b, b1, b2);
            smem[p * BT + l] = b2;
        });
        __syncthreads();
        if (mine) {
            double out[8][3];
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) out[a][r] = 0.;
            ggn_points<true, true>(C, q, [&](int p, int, int, int) { return smem[p * BT + threadIdx.x]; }, out);
#pragma unroll
            for (int a = 0; a < 8; a++)
#pragma unroll
                for (int r = 0; r < 3; r++) L[(size_t)(3 * a + r) * q.ncell + c] += out[a][r];
        }
    });
}

// ============================================================================================== stable differences
// One residual pair: (b - a)(b + a) / 2 accumulated exactly enough in double-double.
__device__ __forceinline__ dd sq_change(double a, double b) {
    dd d = two_sum(b, -a), s = two_sum(b, a);
    dd p = two_prod(d.hi, s.hi);
    p.lo += d.hi * s.lo + d.lo * s.hi;
    return {p.hi * .5, p.lo * .5};
}

// node_weight halves omega once per face that the node lies on: four values, whose roots the stable differences scale
// by.  A block forms them once: two roots per node were 75 of warp_trial_kernel's 1211 us at 256^3.
struct NodeScale {
    double w[4], sq[4], sl[4];    // weight, sqrt(weight), sqrt(lambda weight) on 0..3 faces
};
__device__ __forceinline__ void node_scale(const Q1Const &q, NodeScale &t) {
    if (threadIdx.x < 4) {
        double w = q.omega;
        for (int m = 0; m < (int)threadIdx.x; m++) w *= .5;
        t.w[threadIdx.x] = w;
        t.sq[threadIdx.x] = sqrt(w);
        t.sl[threadIdx.x] = sqrt(q.lam * w);
    }
    __syncthreads();
}
__device__ __forceinline__ int node_faces(long long x, long long y, long long z, const Q1Const &q) {
    return (x == 0 || x == q.nx - 1) + (y == 0 || y == q.ny - 1) + (z == 0 || z == q.nz - 1);
}

// compensated (hi, lo) accumulation of t
__device__ __forceinline__ void acc_add(dd &acc, dd t) {
    dd s = two_sum(acc.hi, t.hi);
    acc.hi = s.hi;
    acc.lo += s.lo + t.lo;
}

__global__ void __launch_bounds__(256) node_diff_kernel(Q1Const q, const double *__restrict__ ua,
                                                        const double *__restrict__ wa,
                                                        const double *__restrict__ ub,
                                                        const double *__restrict__ wb,
                                                        const double *__restrict__ fixed,
                                                        const double *__restrict__ uref, dd *partial) {
    __shared__ NodeScale scale;
    node_scale(q, scale);
    dd acc[2] = {{0., 0.}, {0., 0.}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nnode;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.nx, q.ny, x, y, z);
        const int m = node_faces(x, y, z, q);
        const double sq = scale.sq[m], sl = scale.sl[m];
        acc_add(acc[0], sq_change(sq * (wa[i] - fixed[i]), sq * (wb[i] - fixed[i])));
#pragma unroll
        for (int r = 0; r < 3; r++)
            acc_add(acc[1], sq_change(sl * (ua[3 * i + r] - uref[3 * i + r]),
                                  sl * (ub[3 * i + r] - uref[3 * i + r])));
    }
#pragma unroll
    for (int k = 0; k < 2; k++) acc[k] = two_sum(acc[k].hi, acc[k].lo);
    block_reduce_dd<2>(acc, partial);
}

// ============================================================================================== line-search trial
// A trial evaluated against its base in one node pass and one cell pass (cell_soft_kernel, cell_barrier_kernel): the
// trial's warped image (and image gradient), its energy sums exactly as node_energy_kernel and the energy-only cell
// kernels form them, and the stable base -> trial changes exactly as node_diff_kernel and the difference-only cell
// kernels form them (same grids, same per-thread order, so the results are bitwise those of the separate passes).
// Bound by the latency of its scattered loads (16 warps per SM at 128 registers; 85 registers spill and lose) and the
// float64 work between them.  At 256^3: 1441 us; 1401 with a plane of coefficients fetched ahead, 1329 with the L1
// prefetches, 1240 with 6 reciprocals per axis read as pairs in place of 14 single ones, 1211 with the differences
// accumulated in 8 operations for 26, 1136 with the weights' roots from a table.  Its 16 doubles a node at 6.55 TB/s
// would take 328 us.
template <bool GRAD>
__global__ void __launch_bounds__(256) warp_trial_kernel(Q1Const q, SplineRef S, const double *__restrict__ ua,
                                                         const double *__restrict__ wa,
                                                         const double *__restrict__ ub,
                                                         const double *__restrict__ fixed,
                                                         const double *__restrict__ uref, double *__restrict__ wb,
                                                         double *__restrict__ image_grad, dd *pe, dd *pd) {
    __shared__ NodeScale scale;
    node_scale(q, scale);
    dd acc[2] = {{0., 0.}, {0., 0.}}, dif[2] = {{0., 0.}, {0., 0.}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nnode;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.nx, q.ny, x, y, z);
        // the operands read after the spline, and the next node's displacement, on their way to L1 meanwhile: no register
        const long long next = i + (long long)gridDim.x * blockDim.x;
        prefetch_l1(wa + i);
        prefetch_l1(fixed + i);
        prefetch_l1(uref + 3 * i);
        prefetch_l1(ua + 3 * i);
        if (next < q.nnode) prefetch_l1(ub + 3 * next);
        double ux = ub[3 * i], uy = ub[3 * i + 1], uz = ub[3 * i + 2];
        double px = (q.x0[0] + q.h[0] * (double)x) + ux;
        double py = (q.x0[1] + q.h[1] * (double)y) + uy;
        double pz = (q.x0[2] + q.h[2] * (double)z) + uz;
        double g[3];
        double w = spline_eval<GRAD>(S, px, py, pz, g);
        wb[i] = w;
        if (GRAD) {
            image_grad[3 * i] = g[0];
            image_grad[3 * i + 1] = g[1];
            image_grad[3 * i + 2] = g[2];
        }
        const int m = node_faces(x, y, z, q);
        const double qw = scale.w[m];
        double f = fixed[i];
        double d = w - f;
        double r0 = uref[3 * i], r1 = uref[3 * i + 1], r2 = uref[3 * i + 2];
        double e0 = ux - r0, e1 = uy - r1, e2 = uz - r2;
        acc[0] = dd_add_d(acc[0], qw * d * d);
        acc[1] = dd_add_d(acc[1], qw * (e0 * e0 + e1 * e1 + e2 * e2));
        const double sq = scale.sq[m], sl = scale.sl[m];
        acc_add(dif[0], sq_change(sq * (wa[i] - f), sq * d));
        acc_add(dif[1], sq_change(sl * (ua[3 * i] - r0), sl * e0));
        acc_add(dif[1], sq_change(sl * (ua[3 * i + 1] - r1), sl * e1));
        acc_add(dif[1], sq_change(sl * (ua[3 * i + 2] - r2), sl * e2));
    }
#pragma unroll
    for (int k = 0; k < 2; k++) dif[k] = two_sum(dif[k].hi, dif[k].lo);
    block_reduce_dd<2>(acc, pe);
    __syncthreads();     // the two reductions share block_reduce_dd's shared array
    block_reduce_dd<2>(dif, pd);
}

// The barrier of the flagged cells (cell_soft_kernel's flags): the state's barrier sum, violations (J <= delta) and
// activity mask (trial_act[c] = 1 when some closed27 J is below the activation), and with DIFF its stable change from
// the base.  pe: per block, the barrier sum and the count of violations (an exact sum of whole numbers, so that nothing
// is carried from one evaluation to the next); pd: the change.
template <bool ENERGY, bool DIFF>
__global__ void __launch_bounds__(BT, 3) cell_barrier_kernel(Q1Const q, const double *__restrict__ ua,
                                                          const double *__restrict__ ub,
                                                          const uint8_t *__restrict__ flags, dd *pe, dd *pd,
                                                          uint8_t *__restrict__ trial_act) {
    extern __shared__ double smem[];
    __shared__ long long queue[kBlockQueue];
    __shared__ dd total[ENERGY ? BT : 1];     // barrier sum of the cells of each place in a group
    double *sb = smem, *sa = smem + 27 * BT;
    if (ENERGY) total[threadIdx.x] = {0., 0.};
    dd dif[1] = {{0., 0.}};
    unsigned nbad = 0;
    const BarrierRule rule = barrier_rule(q);
    for_flagged_blocks(q, flags, queue, [&](int n) {
        if ((int)threadIdx.x < n) {
            const long long n0 = cell_node0(queue[threadIdx.x], q);
            Columns C;
            closed_jacobians(ub, n0, q, C, sb + threadIdx.x, BT);
            if (DIFF) closed_jacobians(ua, n0, q, C, sa + threadIdx.x, BT);
        }
        __syncthreads();
        double change = 0.;
        bool active = false;
        int cell = 0;
        for_block_points(n, [&](int p, int l) {
            const double jb = sb[p * BT + l];
            if (DIFF) {
                const double ja = sa[p * BT + l];
                if (ja < q.act || jb < q.act) change += barrier_change(ja, jb, rule);
            }
            if (ENERGY) {
                active |= jb < q.act;
                cell = l;
                double b = 0.;
                if (!(jb > q.delta)) nbad++;
                else if (jb < q.act) b = barrier_value(jb, rule);
                sb[p * BT + l] = b;
            }
        });
        if (DIFF) dif[0] = dd_add_d(dif[0], q.bw * change);
        if (ENERGY) {
            // The sum does not depend on what else is queued (a trial's queue has the base's cells too): each cell's
            // points in order, then the cells of one place in their groups of BT in the queue's order, warp after warp
            // and, where a warp has several of one place, lane after lane (0.50 -> 0.54 ms on 256^3).
            if (trial_act && active) trial_act[queue[cell]] = 1;
            __syncthreads();
            const bool mine = (int)threadIdx.x < n;
            const int lane = threadIdx.x & 31, place = mine ? (int)queue[threadIdx.x] & (BT - 1) : -1;
            double s[3] = {0., 0., 0.};
            if (mine)
#pragma unroll
                for (int p = 0; p < 27; p++) s[p / 9] += sb[p * BT + threadIdx.x];
            const double sum = (s[0] + s[1]) + s[2];
            const int before = __popc(__match_any_sync(0xFFFFFFFFu, place) & ((1u << lane) - 1u));
            for (int w = 0; 32 * w < n; w++) {
                if ((int)threadIdx.x >> 5 == w)
                    for (int r = 0; __any_sync(0xFFFFFFFFu, mine && before >= r); r++) {
                        if (mine && before == r) total[place] = dd_add_d(total[place], sum);
                        __syncwarp();
                    }
                __syncthreads();
            }
        }
    });
    if (ENERGY) {
        dd acc[2] = {total[threadIdx.x], {(double)nbad, 0.}};
        block_reduce_dd<2>(acc, pe);
    }
    if (ENERGY && DIFF) __syncthreads();     // the two reductions share block_reduce_dd's shared array
    if (DIFF) block_reduce_dd<1>(dif, pd);
}

// ============================================================================================== screened trial
// A trial for hosts that screen energies: the JD and curl penalties at the Gauss points in float32 (reference J and curl
// in a float slice, both fields' float edges), their per-cell sums in float and the block sums in double-double; the
// localized barrier and its difference in float64 by cell_barrier_kernel over the cells with some float32 closed27 J
// within kBarrierGuard of the activation (elsewhere every J is above the activation in both arithmetics, where the
// barrier and its difference vanish).  So the violation count and the activity mask are the float64 trial's and the
// barrier sum and difference its sums, and only the JD/curl sums carry float32 error, which the host screens against a
// band (the reference's float32 energy screen, backends/accelerated.py:66-77).
__device__ __forceinline__ void reference_points32(const double *__restrict__ uref, long long n0, const Q1Const &q,
                                                   float *sl, int T) {
    float Er[3][4][3];
    load_edges_f32(uref, n0, q, Er);
    sweep<false, float>(Er, q, [&](int p, int, int, int, const float (&Vr)[3][3]) {
        float Cr[3];
        curl_of(Vr, Cr);
        sl[(4 * p) * T] = det_only(Vr);
        sl[(4 * p + 1) * T] = Cr[0];
        sl[(4 * p + 2) * T] = Cr[1];
        sl[(4 * p + 3) * T] = Cr[2];
    });
}
// The soft part of the screened trial (JD and curl penalty sums and differences) in float32; the barrier part runs in
// cell_barrier_kernel over the cells this kernel flags.  pe, pd: per block, the two soft sums and their two
// differences; pb (the screen's error-bound sums): sum w (|ra| + |rb|) of the JD residuals, the same of the curl
// residual components, sum w ra^2 and sum w |xa|^2 (the base's soft sums), all from the float32 residuals.
__global__ void __launch_bounds__(CS) cell_trial32_kernel(Q1Const q, const double *__restrict__ ua,
                                                          const double *__restrict__ ub,
                                                          const double *__restrict__ uref, dd *pe, dd *pd, dd *pb,
                                                          uint8_t *__restrict__ flags,
                                                          uint8_t *__restrict__ trial_act,
                                                          const uint8_t *__restrict__ base_act) {
    extern __shared__ float smemf[];
    const int T = blockDim.x;
    // per thread: 108 floats (reference J and curl at the Gauss points), strided by the block size
    float *fsl = smemf + threadIdx.x;
    const float guard = (float)q.act + kBarrierGuard;
    dd acc[2] = {{0., 0.}, {0., 0.}}, dif[2] = {{0., 0.}, {0., 0.}};
    dd bnd[4] = {{0., 0.}, {0., 0.}, {0., 0.}, {0., 0.}};
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        long long n0 = cell_node0(c, q);
        reference_points32(uref, n0, q, fsl, T);
        float Ea[3][4][3], Eb[3][4][3];
        load_edges_f32(ua, n0, q, Ea);
        load_edges_f32(ub, n0, q, Eb);
        float sj = 0.f, sc = 0.f, dj = 0.f, dc = 0.f, mj = 0.f, mc = 0.f, aj = 0.f, ac = 0.f;
        sweep2<false, float>(Ea, Eb, q, [&](int p, int, int, int, const float (&Va)[3][3], const float (&Vb)[3][3]) {
            float Ca[3], Cb[3];
            const float jr = fsl[(4 * p) * T];
            const float ja = det_only(Va) - jr, jb = det_only(Vb) - jr;
            curl_of(Va, Ca);
            curl_of(Vb, Cb);
            const float w = q.gwf[p];
            float cb2 = 0.f, ca2 = 0.f, cd = 0.f, cm = 0.f;
#pragma unroll
            for (int r = 0; r < 3; r++) {
                const float cr = fsl[(4 * p + 1 + r) * T];
                const float xa = Ca[r] - cr, xb = Cb[r] - cr;
                cb2 += xb * xb;
                ca2 += xa * xa;
                cd += (xb - xa) * (xb + xa);
                cm += fabsf(xa) + fabsf(xb);
            }
            sj += w * jb * jb;
            sc += w * cb2;
            dj += w * ((jb - ja) * (jb + ja));
            dc += w * cd;
            mj += w * (fabsf(ja) + fabsf(jb));
            mc += w * cm;
            aj += w * ja * ja;
            ac += w * ca2;
        });
        // the closed27 J in float32: a cell with some trial point within the guard or not finite (bit 0), or some base
        // point within the guard where the base may be active (bit 1), is flagged for the float64 barrier kernel;
        // elsewhere every J is above the activation in both arithmetics (no barrier, no difference, no violation)
        bool near_b = false, near_a = false;
        sweep<true, float>(Eb, q, [&](int, int, int, int, const float (&Vb)[3][3]) {
            const float J = det_only(Vb);
            near_b |= !(J >= guard && J <= 3.402823466e38f);
        });
        if (near_b || !base_act || base_act[c])
            sweep<true, float>(Ea, q, [&](int, int, int, int, const float (&Va)[3][3]) {
                near_a |= det_only(Va) < guard;
            });
        flags[c] = (near_b ? 1 : 0) | (near_a ? 2 : 0);
        if (trial_act) trial_act[c] = 0;
        acc[0] = dd_add_d(acc[0], (double)sj);
        acc[1] = dd_add_d(acc[1], (double)sc);
        acc_add(dif[0], dd{.5 * q.mu * (double)dj, 0.});
        acc_add(dif[1], dd{.5 * q.nu * (double)dc, 0.});
        bnd[0] = dd_add_d(bnd[0], (double)mj);
        bnd[1] = dd_add_d(bnd[1], (double)mc);
        bnd[2] = dd_add_d(bnd[2], (double)aj);
        bnd[3] = dd_add_d(bnd[3], (double)ac);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) dif[k] = two_sum(dif[k].hi, dif[k].lo);
    block_reduce_dd<2>(acc, pe);
    __syncthreads();     // the reductions share block_reduce_dd's shared array
    block_reduce_dd<2>(dif, pd);
    __syncthreads();
    block_reduce_dd<4>(bnd, pb);
}

// ============================================================================================== node JD measure
// ext_act > 0 (T69/T73): cells whose closed27 Bernstein coefficients allow a value below min(m_c, ext_act) are
// appended to cand (order of arrival; each is then estimated independently, so the order does not matter).
// Bound: FP64 issue, about 560 FP64 instructions per cell (closed27 J 243 and their columns 204, 12 edge quadratics);
// 160x192x224: 1.00 -> 0.49 ms per launch (the edge and Bernstein loops unrolled on registers: 0.86 -> 0.49).  Six
// blocks per SM: the compiler's 190 registers allow five (metric call on 128x144x128 1050 against 1025 us).
__global__ void __launch_bounds__(CS, 6) cell_min_jd_kernel(Q1Const q, const double *__restrict__ u,
                                                         double *__restrict__ m, double ext_act,
                                                         unsigned long long *__restrict__ ncand,
                                                         long long *__restrict__ cand) {
    extern __shared__ double smem[];
    double *J = smem + threadIdx.x;
    const int T = blockDim.x;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        Columns C;
        closed_jacobians(u, cell_node0(c, q), q, C, J, T);
        double j[27], mn = __longlong_as_double(0x7FF0000000000000LL);
#pragma unroll
        for (int p = 0; p < 27; p++) {
            j[p] = J[p * T];
            mn = fmin(mn, j[p]);
        }
        // exact interior minima of the edge quadratics through t = 0, 1/2, 1 (solvers/jd_affine.py:24)
#pragma unroll
        for (int e = 0; e < 12; e++) {
            // x edges: iz, iy in {0, 2}; y edges: iz, ix; z edges: iy, ix
            const int k = e & 3, st = e < 4 ? 1 : (e < 8 ? 3 : 9);
            const int f0 = e < 4 ? 9 * ((k >> 1) * 2) + 3 * ((k & 1) * 2)
                                 : (e < 8 ? 9 * ((k >> 1) * 2) + (k & 1) * 2 : 3 * ((k >> 1) * 2) + (k & 1) * 2);
            const double j0 = j[f0], j1 = j[f0 + st], j2 = j[f0 + 2 * st];
            const double a = 2 * (j0 - 2 * j1 + j2);
            const double b = -3 * j0 + 4 * j1 - j2;
            if (a > 0 && b < 0 && -b < 2 * a) mn = fmin(mn, j0 - b * b / (4 * a));
        }
        m[c] = mn;
        if (ext_act > 0.) {
            // closed27 values -> Bernstein coefficients: per axis x, y, z the middle entry becomes 2 b - (a + c) / 2
            // (bernstein_barrier.py:26 to_bernstein)
#pragma unroll
            for (int axis = 0; axis < 3; axis++) {
                const int st = axis == 0 ? 1 : (axis == 1 ? 3 : 9);
#pragma unroll
                for (int l = 0; l < 9; l++) {
                    const int o = axis == 0 ? 3 * l : (axis == 1 ? (l / 3) * 9 + (l % 3) : l);
                    j[o + st] = 2. * j[o + st] - .5 * (j[o] + j[o + 2 * st]);
                }
            }
            double bmin = j[0];
#pragma unroll
            for (int k = 1; k < 27; k++) bmin = fmin(bmin, j[k]);
            if (bmin < fmin(mn, ext_act)) cand[atomicAdd(ncand, 1ull)] = c;
        }
    }
}

// ---- T69/T73 face/interior estimate mu_c on candidate cells (solvers/jd_affine.py:45-150) ----
// J on a cell is triquadratic; mu_c = min of its values on the 9^3 grid {0, 1/8, .., 1}^3 and of a bounded Newton
// descent (30 iterations, halving backtracking <= 40, strict decrease only) from the 4 lowest grid points (stable
// order).  A value J attains, so an estimate for the metric, never a bound.  One warp per candidate cell.
struct Tri {
    double c[27];    // monomial coefficients C[k][j][i] of z^k y^j x^i
};
// NumPy's add-reduce order for a contiguous length-27 axis (eight accumulators; jd_affine_compiled.py:_sum27)
__device__ __forceinline__ double sum27(const double *a) {
    double r[8];
#pragma unroll
    for (int i = 0; i < 8; i++) r[i] = a[i];
#pragma unroll
    for (int b = 8; b < 24; b += 8)
#pragma unroll
        for (int i = 0; i < 8; i++) r[i] += a[b + i];
    double res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
    res += a[24];
    res += a[25];
    res += a[26];
    return 0.0 + res;
}
// sum C[k][j][i] (Z_k Y_j) X_i
__device__ __forceinline__ double tri_e(const Tri &T, const double Z[3], const double Y[3], const double X[3]) {
    double tmp[27];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const double zy = Z[k] * Y[j];
#pragma unroll
            for (int i = 0; i < 3; i++) tmp[9 * k + 3 * j + i] = T.c[9 * k + 3 * j + i] * (zy * X[i]);
        }
    return sum27(tmp);
}
__device__ __forceinline__ void tri_powers(double t, double P[3][3]) {
    P[0][0] = 1.; P[0][1] = t; P[0][2] = t * t;
    P[1][0] = 0.; P[1][1] = 1.; P[1][2] = 2. * t;
    P[2][0] = 0.; P[2][1] = 0.; P[2][2] = 2.;
}
__device__ __forceinline__ double tri_value(const Tri &T, const double x[3]) {
    double px[3][3], py[3][3], pz[3][3];
    tri_powers(x[0], px); tri_powers(x[1], py); tri_powers(x[2], pz);
    return tri_e(T, pz[0], py[0], px[0]);
}
__device__ __forceinline__ double clip01(double v) {
    if (v != v) return v;
    const double w = v > 0. ? v : 0.;
    return w < 1. ? w : 1.;
}
// Symmetric 3x3 eigen-decomposition by cyclic Jacobi rotations: A = Q diag(w) Q^T (columns of Q).
__device__ void sym3_eigen(double A[3][3], double w[3], double Q[3][3]) {
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) Q[i][j] = i == j ? 1. : 0.;
#pragma unroll 1
    for (int sweep = 0; sweep < 64; sweep++) {
        const double off = fabs(A[0][1]) + fabs(A[0][2]) + fabs(A[1][2]);
        const double dia = fabs(A[0][0]) + fabs(A[1][1]) + fabs(A[2][2]);
        if (off == 0. || off <= 1e-300 + 1e-18 * dia) break;
#pragma unroll 1
        for (int pq = 0; pq < 3; pq++) {
            const int p = pq == 2 ? 1 : 0, qq = pq == 0 ? 1 : 2;
            const double apq = A[p][qq];
            if (apq == 0.) continue;
            // rotation zeroing A[p][q] (symmetric Schur decomposition of the 2x2 block)
            const double tau = (A[qq][qq] - A[p][p]) / (2. * apq);
            const double t = (tau >= 0. ? 1. : -1.) / (fabs(tau) + sqrt(1. + tau * tau));
            const double cs = 1. / sqrt(1. + t * t), sn = t * cs;
#pragma unroll
            for (int k = 0; k < 3; k++) {     // A <- A J
                const double akp = A[k][p], akq = A[k][qq];
                A[k][p] = cs * akp - sn * akq;
                A[k][qq] = sn * akp + cs * akq;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {     // A <- J^T A
                const double apk = A[p][k], aqk = A[qq][k];
                A[p][k] = cs * apk - sn * aqk;
                A[qq][k] = sn * apk + cs * aqk;
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {     // Q <- Q J
                const double qkp = Q[k][p], qkq = Q[k][qq];
                Q[k][p] = cs * qkp - sn * qkq;
                Q[k][qq] = sn * qkp + cs * qkq;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 3; i++) w[i] = A[i][i];
}
// jd_affine.py:_bounded_newton for one start; returns the lowest value reached
__device__ double bounded_newton(const Tri &T, double x[3], double best) {
#pragma unroll 1
    for (int it = 0; it < 30; it++) {
        double px[3][3], py[3][3], pz[3][3];
        tri_powers(x[0], px); tri_powers(x[1], py); tri_powers(x[2], pz);
        double g[3], H[3][3];
        g[0] = tri_e(T, pz[0], py[0], px[1]);
        g[1] = tri_e(T, pz[0], py[1], px[0]);
        g[2] = tri_e(T, pz[1], py[0], px[0]);
        H[0][0] = tri_e(T, pz[0], py[0], px[2]);
        H[1][1] = tri_e(T, pz[0], py[2], px[0]);
        H[2][2] = tri_e(T, pz[2], py[0], px[0]);
        H[0][1] = H[1][0] = tri_e(T, pz[0], py[1], px[1]);
        H[0][2] = H[2][0] = tri_e(T, pz[1], py[0], px[1]);
        H[1][2] = H[2][1] = tri_e(T, pz[1], py[1], px[0]);
        bool free_[3];
        double gf[3], Hf[3][3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            free_[a] = !((x[a] <= 0. && g[a] > 0.) || (x[a] >= 1. && g[a] < 0.));
            gf[a] = free_[a] ? g[a] : 0.;
        }
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
                Hf[a][b] = (free_[a] && free_[b]) ? H[a][b] : (a == b && !free_[a] ? 1. : 0.);
        double w[3], Q[3][3];
        sym3_eigen(Hf, w, Q);
        const double scale = fmax(1., fmax(fabs(w[0]), fmax(fabs(w[1]), fabs(w[2]))));
        const bool ok = w[0] > 1e-12 * scale && w[1] > 1e-12 * scale && w[2] > 1e-12 * scale;
        double d[3];
        if (ok) {
            double proj[3];
#pragma unroll
            for (int j = 0; j < 3; j++) proj[j] = (Q[0][j] * gf[0] + Q[1][j] * gf[1] + Q[2][j] * gf[2]) / w[j];
#pragma unroll
            for (int i = 0; i < 3; i++) d[i] = -(Q[i][0] * proj[0] + Q[i][1] * proj[1] + Q[i][2] * proj[2]);
        } else {
#pragma unroll
            for (int i = 0; i < 3; i++) d[i] = -gf[i] / scale;
        }
        double step = 1.;
        bool done = false;
#pragma unroll 1
        for (int bt = 0; bt < 40; bt++) {
            double xt[3];
#pragma unroll
            for (int a = 0; a < 3; a++) xt[a] = clip01(x[a] + step * d[a]);
            const double ft = tri_value(T, xt);
            if (ft < best) {
                x[0] = xt[0]; x[1] = xt[1]; x[2] = xt[2];
                best = ft;
                done = true;
                break;
            }
            step = .5 * step;
        }
        if (!done) break;       // no strict decrease: converged to rounding (or stuck)
    }
    return best;
}

__device__ __forceinline__ double lagrange3(int a, double t) {
    return a == 0 ? 2. * (t - .5) * (t - 1.) : (a == 1 ? -4. * t * (t - 1.) : 2. * t * (t - .5));
}
// (value, index) lexicographic order: the stable ascending sort of the grid values (NaN last)
__device__ __forceinline__ bool vi_less(double v, int i, double w, int j) {
    if (v < w) return true;
    if (w != w && v == v) return true;
    if (v == w || (v != v && w != w)) return i < j;
    return false;
}

__global__ void __launch_bounds__(128) jd_extension_kernel(Q1Const q, const double *__restrict__ u,
                                                           const unsigned long long *__restrict__ ncand,
                                                           const long long *__restrict__ cand,
                                                           double *__restrict__ m) {
    __shared__ double sJ[4][27];
    __shared__ Tri sT[4];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const long long n = (long long)*ncand;
    for (long long w = blockIdx.x * 4LL + wib; w < n; w += (long long)gridDim.x * 4) {
        const long long c = cand[w];
        double E[3][4][3];
        load_edges(u, cell_node0(c, q), q, E);
        if (lane == 0)
            sweep<true>(E, q, [&](int p, int, int, int, const double (&V)[3][3]) { sJ[wib][p] = det_only(V); });
        __syncwarp();
        // monomial coefficients C[k][j][i] = sum_cba J[c][b][a] M[c][k] M[b][j] M[a][i], M the Lagrange-to-power map
        if (lane < 27) {
            const double M[3][3] = {{1., -3., 2.}, {0., 4., -4.}, {0., -1., 2.}};
            const int k = lane / 9, j = (lane / 3) % 3, i = lane % 3;
            double acc = 0.;
#pragma unroll
            for (int cc = 0; cc < 3; cc++)
#pragma unroll
                for (int b = 0; b < 3; b++)
#pragma unroll
                    for (int a = 0; a < 3; a++)
                        acc += sJ[wib][9 * cc + 3 * b + a] * (M[cc][k] * (M[b][j] * M[a][i]));
            sT[wib].c[lane] = acc;
        }
        __syncwarp();
        // 9^3 grid values (z-major, x fastest), each lane keeping its 4 lowest in stable order
        double tv[4];
        int ti[4];
#pragma unroll
        for (int r = 0; r < 4; r++) { tv[r] = __longlong_as_double(0x7FF8000000000000LL); ti[r] = 0x7FFFFFFF; }
        for (int pnt = lane; pnt < 729; pnt += 32) {
            const int ix = pnt % 9, iy = (pnt / 9) % 9, iz = pnt / 81;
            const double tx = .125 * ix, ty = .125 * iy, tz = .125 * iz;
            double val = 0.;
#pragma unroll
            for (int cc = 0; cc < 3; cc++)
#pragma unroll
                for (int b = 0; b < 3; b++)
#pragma unroll
                    for (int a = 0; a < 3; a++)
                        val += sJ[wib][9 * cc + 3 * b + a] * (lagrange3(cc, tz) * (lagrange3(b, ty) * lagrange3(a, tx)));
            if (vi_less(val, pnt, tv[3], ti[3])) {
                int pos = 3;
                while (pos > 0 && vi_less(val, pnt, tv[pos - 1], ti[pos - 1])) {
                    tv[pos] = tv[pos - 1]; ti[pos] = ti[pos - 1];
                    pos--;
                }
                tv[pos] = val; ti[pos] = pnt;
            }
        }
        // butterfly merge of the lanes' sorted lists
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            double ov[4];
            int oi[4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                ov[r] = __shfl_xor_sync(0xFFFFFFFFu, tv[r], o);
                oi[r] = __shfl_xor_sync(0xFFFFFFFFu, ti[r], o);
            }
            double nv[4];
            int ni[4];
            int a = 0, b = 0;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                if (vi_less(tv[a], ti[a], ov[b], oi[b])) { nv[r] = tv[a]; ni[r] = ti[a]; a++; }
                else { nv[r] = ov[b]; ni[r] = oi[b]; b++; }
            }
#pragma unroll
            for (int r = 0; r < 4; r++) { tv[r] = nv[r]; ti[r] = ni[r]; }
        }
        // bounded Newton from the 4 lowest grid points, lanes 0..3
        double found = __longlong_as_double(0x7FF0000000000000LL);
        if (lane < 4) {
            const int s0 = lane == 0 ? ti[0] : (lane == 1 ? ti[1] : (lane == 2 ? ti[2] : ti[3]));
            double x[3] = {.125 * (s0 % 9), .125 * ((s0 / 9) % 9), .125 * (s0 / 81)};
            found = bounded_newton(sT[wib], x, tri_value(sT[wib], x));
        }
#pragma unroll
        for (int o = 2; o; o >>= 1) found = fmin(found, __shfl_xor_sync(0xFFFFFFFFu, found, o));
        if (lane == 0) {
            const double mu = fmin(tv[0], found);       // grid minimum and the Newton descents
            const double mc = m[c];
            m[c] = (mu < mc || mu != mu) ? mu : mc;     // np.minimum
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256) node_min_kernel(Q1Const q, const double *__restrict__ m,
                                                       double *__restrict__ node) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nnode;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.nx, q.ny, x, y, z);
        double mn = __longlong_as_double(0x7FF0000000000000LL);
#pragma unroll
        for (int a = 0; a < 8; a++) {
            long long cz = z - (a >> 2), cy = y - ((a >> 1) & 1), cx = x - (a & 1);
            if (cz < 0 || cy < 0 || cx < 0 || cz >= q.cz || cy >= q.cy || cx >= q.cx) continue;
            mn = fmin(mn, m[(cz * q.cy + cy) * q.cx + cx]);
        }
        node[i] = mn;
    }
}

// ============================================================================================== global JD root
// solvers/global_jd_step.py:52 first_roots for one point (b0 > 0), normalized s in (0, 1]; +inf if none
__device__ double first_root(double b0, double b1, double b2, double b3) {
    const double INF = __longlong_as_double(0x7FF0000000000000LL);
    if (b0 > fabs(b1) + fabs(b2) + fabs(b3)) return INF;
    const double nan = __longlong_as_double(0x7FF8000000000000LL);
    double a = 3 * b3, b = 2 * b2, c = b1;
    bool linear = a == 0;
    double r_lin = (linear && b != 0) ? -c / b : nan;
    double disc = b * b - 4 * a * c;
    double sq = sqrt(disc >= 0 ? disc : 0.);
    double qq = -(b + (b >= 0 ? sq : -sq)) / 2;
    double r1 = (!linear && disc >= 0 && a != 0) ? qq / a : nan;
    double r2 = (!linear && disc >= 0 && qq != 0) ? c / qq : nan;
    if (linear) { r1 = r_lin; r2 = nan; }
    r1 = (r1 > 0 && r1 < 1) ? r1 : 1.;
    r2 = (r2 > 0 && r2 < 1) ? r2 : 1.;
    double t1 = fmin(r1, r2), t2 = fmax(r1, r2);
    auto qv = [&](double s) { return b0 + s * (b1 + s * (b2 + s * b3)); };
    const double eps4 = 4 * 2.220446049250313e-16;
    auto touch = [&](double s) { return eps4 * (fabs(b0) + s * (fabs(b1) + s * (fabs(b2) + s * fabs(b3)))); };
    double lo, hi;
    if (qv(t1) <= touch(t1)) { lo = 0.; hi = t1; }
    else if (qv(t2) <= touch(t2)) { lo = t1; hi = t2; }
    else if (qv(1.) <= 0) { lo = t2; hi = 1.; }
    else return INF;
    for (int k = 0; k < 50; k++) {
        double mid = .5 * (lo + hi);
        if (qv(mid) <= 0) hi = mid;
        else lo = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(CT) jd_root_kernel(Q1Const q, const double *__restrict__ u,
                                                     const double *__restrict__ pv, double limit,
                                                     long long *__restrict__ best_key,
                                                     unsigned long long *__restrict__ invalid) {
    long long key = kKeyPosInf;
    unsigned long long nbad = 0;
    const double L2 = limit * limit, L3 = limit * limit * limit;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < q.ncell;
         c += (long long)gridDim.x * blockDim.x) {
        long long n0 = cell_node0(c, q);
        double E[3][4][3], Ep[3][4][3];
        load_edges(u, n0, q, E);
        load_edges(pv, n0, q, Ep);
        sweep2<true>(E, Ep, q, [&](int, int, int, int, const double (&V)[3][3], const double (&W)[3][3]) {
            double AF[3][3], AV[3][3], J, JV;
            cofactor_det(V, AF, J);
#pragma unroll
            for (int r = 0; r < 3; r++) {
                int j = (r + 1) % 3, k = (r + 2) % 3;
#pragma unroll
                for (int cc = 0; cc < 3; cc++) {
                    int l = (cc + 1) % 3, mm = (cc + 2) % 3;
                    AV[r][cc] = W[j][l] * W[k][mm] - W[j][mm] * W[k][l];
                }
            }
            JV = (W[0][0] * AV[0][0] + W[0][1] * AV[0][1]) + W[0][2] * AV[0][2];
            double c0 = J - q.delta, c1 = 0., c2 = 0.;
#pragma unroll
            for (int r = 0; r < 3; r++)
#pragma unroll
                for (int cc = 0; cc < 3; cc++) {
                    c1 += AF[r][cc] * W[r][cc];
                    c2 += (V[r][cc] + (r == cc ? 1. : 0.)) * AV[r][cc];
                }
            if (!(c0 > 0)) { nbad++; return; }
            double s = first_root(c0, c1 * limit, c2 * L2, JV * L3);
            long long k = order_key(s);
            key = k < key ? k : key;
        });
    }
    for (int o = 16; o; o >>= 1) {
        long long y = __shfl_xor_sync(0xFFFFFFFFu, key, o);
        key = y < key ? y : key;
        nbad += __shfl_xor_sync(0xFFFFFFFFu, nbad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(best_key, key);
        if (nbad) atomicAdd(invalid, nbad);
    }
}

// ============================================================================================== PG metric pieces
__global__ void __launch_bounds__(256) shift_kernel(Q1Const q, const double *__restrict__ image_grad, dd *partial) {
    dd acc[1] = {{0., 0.}};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nfree;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.fx, q.fy, x, y, z);
        x++; y++; z++;
        const double *b = image_grad + 3 * ((z * q.ny + y) * q.nx + x);
        double qo = node_weight(x, y, z, q) / q.omega;
        acc[0] = dd_add_d(acc[0], qo * ((b[0] * b[0] + b[1] * b[1]) + b[2] * b[2]));
    }
    block_reduce_dd<1>(acc, partial);
}

__global__ void __launch_bounds__(256) pg_scale_kernel(Q1Const q, const double *__restrict__ diag,
                                                       const double *__restrict__ node, double sm, double act,
                                                       double floor_, double *__restrict__ scale,
                                                       unsigned long long *bad) {
    unsigned long long nb = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < q.nfree;
         i += (long long)gridDim.x * blockDim.x) {
        long long x, y, z;
        unflatten3(i, q.fx, q.fy, x, y, z);
        x++; y++; z++;
        double ja = node[(z * q.ny + y) * q.nx + x];
        double r = fmin(1., fmax(ja, floor_) / act);
        if (!(ja == ja) || !(ja < INFINITY) || !(ja > -INFINITY)) nb++;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            double d = diag[c * q.nfree + i];
            double s = (sm / sqrt(d)) * r;
            if (!(d > 0) || !(s > 0) || !(s < INFINITY)) nb++;
            scale[c * q.nfree + i] = s;
        }
    }
    for (int o = 16; o; o >>= 1) nb += __shfl_xor_sync(0xFFFFFFFFu, nb, o);
    if ((threadIdx.x & 31) == 0 && nb) atomicAdd(bad, nb);
}

// ============================================================================================== final reduction
// All block sums of one evaluation in one launch, one block per sum: thread t adds blocks t, t + 256, ... in order, then
// a fixed tree.  The results go straight to the pair's pinned host buffer, so the evaluation ends with a wait and no copy.  A trial took six of these launches, a
// memset and two copies to pageable memory: on 48^3 about 60 of its 161 us.
struct ReduceSpec {
    static constexpr int kMost = 8;
    const dd *src[kMost];
    long long blocks[kMost];
    int K[kMost], out[kMost], n = 0, sums = 0;
    void add(const dd *partial, long long count, int k, int at) {
        src[n] = partial; blocks[n] = count; K[n] = k; out[n] = at;
        n++;
        sums += k;
    }
};
__global__ void __launch_bounds__(256) reduce_results_kernel(const __grid_constant__ ReduceSpec r, double *out) {
    int i = 0, k = blockIdx.x;
    while (k >= r.K[i]) k -= r.K[i++];
    const dd *partial = r.src[i];
    const int K = r.K[i];
    const dd sum = sum_partials(partial, r.blocks[i], K, k);
    if (threadIdx.x == 0) {
        out[r.out[i] + 2 * k] = sum.hi;
        out[r.out[i] + 2 * k + 1] = sum.lo;
    }
}

SplineRef spline_ref(const svp_pair *p) {
    SplineRef S;
    S.c = p->coeff;
    for (int k = 0; k < 3; k++) {
        S.t[k] = p->knots[k];
        S.rcp[k] = p->spline_rcp[k];
        S.x0[k] = p->q.x0[k];
        S.ih[k] = 1. / p->q.h[k];
    }
    S.n[0] = p->q.nx; S.n[1] = p->q.ny; S.n[2] = p->q.nz;
    return S;
}

unsigned cell_blocks(const svp_pair *p) { return blocks_for(p->q.ncell, CT, CELL_PER_SM); }
unsigned slice_blocks(const Q1Const &q) { return blocks_for(q.ncell, CS, 2 * CELL_PER_SM); }
unsigned slice_blocks(const svp_pair *p) { return slice_blocks(p->q); }
// dynamic shared memory of the slice kernels: k doubles per thread
constexpr size_t slice_bytes(int k) { return sizeof(double) * (size_t)k * CS; }
// the cell kernels' slices, beside block_reduce_dd's 1 KB, fit the default
static_assert(slice_bytes(kDiffSlots) + 1024 <= 48 * 1024, "a cell kernel's slice is above the default shared memory");
int allow_slices() {
    // the two-field barrier kernels' J (54 KB) are above the 48 KB default.  The attribute belongs to the device's context (the primary
    // context torch and this library share), so it is set on the first call per device, not on every launch: a
    // cudaFuncSetAttribute costs host time that the GPU then spends idle.
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    SVP_CUDA(cudaGetDevice(&dev));
    SVP_REQUIRE(dev >= 0 && dev < 64, "allow_slices: device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return SVP_OK;
    SVP_CUDA(cudaFuncSetAttribute(cell_barrier_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * 54 * BT)));
    SVP_CUDA(cudaFuncSetAttribute(cell_barrier_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(double) * 54 * BT)));
    done[dev] = true;
    return SVP_OK;
}
unsigned node_blocks(long long n) { return blocks_for(n, 256, 8); }

int reduce_results(svp_pair *p, const ReduceSpec &r, cudaStream_t s) {
    SVP_LAUNCH(reduce_results_kernel<<<(unsigned)r.sums, 256, 0, s>>>(r, p->host));
    SVP_CUDA(cudaStreamSynchronize(s));
    return SVP_OK;
}

}  // namespace

long long pair_partial_count(const Q1Const &q) {
    const long long nb = node_blocks(q.nnode), cb = slice_blocks(q);
    return nb * 4 + cb * 10 + cell_barrier_blocks(q) * 3LL;       // the screened trial's sums
}

int pair_locals(svp_pair *p, int n) {
    size_t bytes = sizeof(double) * 24 * (size_t)p->q.ncell;
    if (n >= 1 && !p->loc1) SVP_CUDA(cudaMalloc((void **)&p->loc1, bytes));
    if (n >= 2 && !p->loc2) SVP_CUDA(cudaMalloc((void **)&p->loc2, bytes));
    return SVP_OK;
}

}  // namespace svp

using namespace svp;

extern "C" int svp_pair_set_precision(svp_pair *p, int32_t precision) {
    SVP_REQUIRE(p && (precision == SVP_PRECISION_PLAIN || precision == SVP_PRECISION_MIXED),
                "svp_pair_set_precision: SVP_PRECISION_PLAIN or SVP_PRECISION_MIXED");
    p->precision = precision;
    return SVP_OK;
}

extern "C" int svp_warp(const svp_pair *p, const double *u, double *warped, double *image_grad, void *stream) {
    SVP_REQUIRE(p && u && warped, "svp_warp: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    SplineRef S = spline_ref(p);
    unsigned nb = node_blocks(p->q.nnode);
    if (image_grad)
        { svp::KernelTimer _t("warp_kernel_grad", s); SVP_LAUNCH(warp_kernel<true><<<nb, 256, 0, s>>>(p->q, S, u, p->fixed, p->u_ref, warped, image_grad, nullptr)); }
    else
        { svp::KernelTimer _t("warp_kernel", s); SVP_LAUNCH(warp_kernel<false><<<nb, 256, 0, s>>>(p->q, S, u, p->fixed, p->u_ref, warped, nullptr, nullptr)); }
    SVP_LAUNCH_CHECK("warp_kernel");
    return SVP_OK;
}

extern "C" int svp_sample_points(const svp_pair *p, const double *points, int64_t n, double *value,
                                 double *gradient, void *stream) {
    SVP_REQUIRE(p && n >= 0, "svp_sample_points: invalid arguments");
    if (!n) return SVP_OK;
    SVP_REQUIRE(points && value, "svp_sample_points: null pointer");
    SVP_LAUNCH(sample_points_kernel<<<node_blocks(n), 256, 0, (cudaStream_t)stream>>>(spline_ref(p), points, n, value,
                                                                           gradient));
    SVP_LAUNCH_CHECK("sample_points_kernel");
    return SVP_OK;
}

extern "C" int svp_energy(svp_pair *p, const double *u, const double *warped, double *terms5,
                          int64_t *barrier_violations, void *stream) {
    SVP_REQUIRE(p && u && warped && terms5, "svp_energy: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned nb = node_blocks(p->q.nnode), cb = slice_blocks(p), bb = cell_barrier_blocks(p->q);
    { svp::KernelTimer _t("node_energy_kernel", s); SVP_LAUNCH(node_energy_kernel<<<nb, 256, 0, s>>>(p->q, u, warped, p->fixed, p->u_ref, p->partial)); }
    SVP_LAUNCH_CHECK("node_energy_kernel");
    dd *pc = p->partial + (long long)nb * 2, *pb = pc + (long long)cb * 2;
    {
        svp::KernelTimer _t("cell_energy_kernel", s);
        SVP_LAUNCH(cell_soft_kernel<true, false><<<cb, CS, slice_bytes(kEnergySlots), s>>>(
            p->q, nullptr, u, p->u_ref, pc, nullptr, p->flags, nullptr));
    }
    {
        svp::KernelTimer _t("cell_barrier_kernel", s);
        SVP_LAUNCH(cell_barrier_kernel<true, false><<<bb, BT, sizeof(double) * 27 * BT, s>>>(
            p->q, nullptr, u, p->flags, pb, nullptr, nullptr));
    }
    SVP_LAUNCH_CHECK("cell_energy_kernel");
    double node2[2], cell3[3];
    ReduceSpec red;
    red.add(p->partial, nb, 2, 0);
    red.add(pc, cb, 2, 4);
    red.add(pb, bb, 2, 8);
    const int rc = reduce_results(p, red, s);
    if (rc) return rc;
    const double *tmp = p->host;
    for (int k = 0; k < 2; k++) node2[k] = tmp[2 * k] + tmp[2 * k + 1];
    for (int k = 0; k < 3; k++) cell3[k] = tmp[4 + 2 * k] + tmp[4 + 2 * k + 1];
    terms5[0] = .5 * node2[0];
    terms5[1] = .5 * p->q.lam * node2[1];
    terms5[2] = .5 * p->q.mu * cell3[0];
    terms5[3] = .5 * p->q.nu * cell3[1];
    terms5[4] = cell3[2];
    if (barrier_violations) *barrier_violations = (int64_t)(tmp[10] + tmp[11]);
    return SVP_OK;
}

extern "C" int svp_energy_difference_masked(svp_pair *p, const double *base_u, const double *base_warped,
                                            const double *trial_u, const double *trial_warped,
                                            const uint8_t *base_active, const uint8_t *trial_active, double *diff2,
                                            void *stream) {
    SVP_REQUIRE(p && base_u && base_warped && trial_u && trial_warped && diff2, "svp_energy_difference: null");
    cudaStream_t s = (cudaStream_t)stream;
    // the cell kernels find the cells near the activation from the J they evaluate, so the masks save nothing here
    (void)base_active;
    (void)trial_active;
    unsigned nb = node_blocks(p->q.nnode), cb = slice_blocks(p), bb = cell_barrier_blocks(p->q);
    int rc = allow_slices();
    if (rc) return rc;
    { svp::KernelTimer _t("node_diff_kernel", s); SVP_LAUNCH(node_diff_kernel<<<nb, 256, 0, s>>>(p->q, base_u, base_warped, trial_u, trial_warped, p->fixed, p->u_ref,
                                        p->partial)); }
    dd *pc = p->partial + (long long)nb * 2, *pb = pc + (long long)cb * 2;
    {
        svp::KernelTimer _t("cell_diff_kernel", s);
        SVP_LAUNCH(cell_soft_kernel<false, true><<<cb, CS, slice_bytes(kDiffSlots), s>>>(
            p->q, base_u, trial_u, p->u_ref, nullptr, pc, p->flags, nullptr));
    }
    {
        svp::KernelTimer _t("cell_barrier_kernel", s);
        SVP_LAUNCH(cell_barrier_kernel<false, true><<<bb, BT, sizeof(double) * 54 * BT, s>>>(
            p->q, base_u, trial_u, p->flags, nullptr, pb, nullptr));
    }
    SVP_LAUNCH_CHECK("difference kernels");
    ReduceSpec red;
    red.add(p->partial, nb, 2, 0);
    red.add(pc, cb, 2, 4);
    red.add(pb, bb, 1, 8);
    if ((rc = reduce_results(p, red, s))) return rc;
    const double *tmp = p->host;
    // E = image + proximity + jd + curl + barrier; F = image + barrier (sums of double-double pieces)
    double img = tmp[0] + tmp[1], prox = tmp[2] + tmp[3];
    double jd = tmp[4] + tmp[5], curl = tmp[6] + tmp[7], bar = tmp[8] + tmp[9];
    diff2[0] = (((img + prox) + jd) + curl) + bar;
    diff2[1] = img + bar;
    return SVP_OK;
}

extern "C" int svp_energy_difference(svp_pair *p, const double *base_u, const double *base_warped,
                                     const double *trial_u, const double *trial_warped, double *diff2,
                                     void *stream) {
    return svp_energy_difference_masked(p, base_u, base_warped, trial_u, trial_warped, nullptr, nullptr, diff2,
                                        stream);
}

// Absolute error estimates of float32 quantities in the screened trial, in units of the float32 unit roundoff
// 2^-24: a Gauss-point J of I + V and its reference J (cofactor products and a 3-term dot product of entries of size
// up to ~2, both rounded), a curl component (one rounded difference of each field's derivatives); and the relative
// rounding of the squared-residual sums.
constexpr double kScreenJ = 256., kScreenCurl = 32., kScreenSum = 64.;

// |error of the E difference| <= mu dJ sum w (|ra| + |rb|) + nu dC sum w (|xa| + |xb|) + 2 dS (soft_a + soft_b): the
// residuals' absolute errors times the summed residual magnitudes, plus the rounding of the squares.  sums: the
// trial's JD and curl sums (unweighted by mu/2, nu/2), then the four pb sums of cell_trial32_kernel.
static double screen_band(const svp_pair *p, const double sums[6]) {
    const double u32 = std::ldexp(1., -24);
    const double soft = .5 * p->q.mu * (sums[0] + sums[4]) + .5 * p->q.nu * (sums[1] + sums[5]);
    return p->q.mu * kScreenJ * u32 * sums[2] + p->q.nu * kScreenCurl * u32 * sums[3] + 2. * kScreenSum * u32 * soft;
}

// The mixed form's screened E/F difference of two evaluated states: node terms float64 (node_diff_kernel), the JD and
// curl penalty differences float32 (cell_trial32_kernel, with the error band), the barrier differences float64 over
// the flagged cells; F (image + barrier) is float64 throughout.
extern "C" int svp_energy_difference_screened(svp_pair *p, const double *base_u, const double *base_warped,
                                              const double *trial_u, const double *trial_warped,
                                              const uint8_t *base_active, double *diff2, double *band,
                                              void *stream) {
    SVP_REQUIRE(p && base_u && base_warped && trial_u && trial_warped && diff2 && band,
                "svp_energy_difference_screened: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned nb = node_blocks(p->q.nnode), cb = slice_blocks(p), bb = cell_barrier_blocks(p->q);
    int rc = allow_slices();
    if (rc) return rc;
    dd *pn = p->partial, *pce = pn + (long long)nb * 2, *pcd = pce + (long long)cb * 2, *pcb = pcd + (long long)cb * 2;
    dd *pbd = pcb + (long long)cb * 4;
    {
        svp::KernelTimer _t("node_diff_kernel", s);
        SVP_LAUNCH(node_diff_kernel<<<nb, 256, 0, s>>>(p->q, base_u, base_warped, trial_u, trial_warped, p->fixed,
                                                       p->u_ref, pn));
    }
    {
        svp::KernelTimer _t("cell_trial32_kernel", s);
        SVP_LAUNCH(cell_trial32_kernel<<<cb, CS, sizeof(float) * 108 * CS, s>>>(
            p->q, base_u, trial_u, p->u_ref, pce, pcd, pcb, p->flags, nullptr, base_active));
    }
    {
        svp::KernelTimer _t("cell_barrier_kernel", s);
        SVP_LAUNCH(cell_barrier_kernel<false, true><<<bb, BT, sizeof(double) * 54 * BT, s>>>(
            p->q, base_u, trial_u, p->flags, nullptr, pbd, nullptr));
    }
    SVP_LAUNCH_CHECK("screened difference kernels");
    ReduceSpec red;
    red.add(pn, nb, 2, 0);
    red.add(pcd, cb, 2, 4);
    red.add(pbd, bb, 1, 8);
    red.add(pce, cb, 2, 10);
    red.add(pcb, cb, 4, 14);
    if ((rc = reduce_results(p, red, s))) return rc;
    const double *tmp = p->host;
    // E = image + proximity + jd + curl + barrier; F = image + barrier, as svp_energy_difference combines them
    double img = tmp[0] + tmp[1], prox = tmp[2] + tmp[3];
    double jd = tmp[4] + tmp[5], curl = tmp[6] + tmp[7], bar = tmp[8] + tmp[9];
    diff2[0] = (((img + prox) + jd) + curl) + bar;
    diff2[1] = img + bar;
    double sums[6];
    for (int k = 0; k < 6; k++) sums[k] = tmp[10 + 2 * k] + tmp[11 + 2 * k];
    *band = screen_band(p, sums);
    return SVP_OK;
}

static int trial_energy(svp_pair *p, const double *base_u, const double *base_warped, const double *trial_u,
                        double *trial_warped, double *trial_image_grad, const uint8_t *base_active,
                        uint8_t *trial_active, double *terms5, double *diff2, int64_t *barrier_violations,
                        bool screened, double *band, void *stream) {
    SVP_REQUIRE(p && base_u && base_warped && trial_u && trial_warped && terms5 && diff2,
                "svp_trial_energy: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned nb = node_blocks(p->q.nnode), cb = slice_blocks(p), bb = cell_barrier_blocks(p->q);
    int rc = allow_slices();
    if (rc) return rc;
    dd *pne = p->partial, *pnd = pne + (long long)nb * 2, *pce = pnd + (long long)nb * 2, *pcd = pce + (long long)cb * 3;
    dd *pcb = pcd + (long long)cb * 3, *pbe = pcb + (long long)cb * 4, *pbd = pbe + (long long)bb * 2;
    SplineRef S = spline_ref(p);
    if (trial_image_grad) {
        svp::KernelTimer _t("warp_trial_kernel_grad", s);
        SVP_LAUNCH(warp_trial_kernel<true><<<nb, 256, 0, s>>>(p->q, S, base_u, base_warped, trial_u, p->fixed,
                                                                p->u_ref, trial_warped, trial_image_grad, pne, pnd));
    } else {
        svp::KernelTimer _t("warp_trial_kernel", s);
        SVP_LAUNCH(warp_trial_kernel<false><<<nb, 256, 0, s>>>(p->q, S, base_u, base_warped, trial_u, p->fixed,
                                                                 p->u_ref, trial_warped, nullptr, pne, pnd));
    }
    SVP_LAUNCH_CHECK("warp_trial_kernel");
    if (screened) {
        svp::KernelTimer _t("cell_trial32_kernel", s);
        SVP_LAUNCH(cell_trial32_kernel<<<cb, CS, sizeof(float) * 108 * CS, s>>>(
            p->q, base_u, trial_u, p->u_ref, pce, pcd, pcb, p->flags, trial_active, base_active));
    } else {
        svp::KernelTimer _t("cell_trial_kernel", s);
        SVP_LAUNCH(cell_soft_kernel<true, true><<<cb, CS, slice_bytes(kDiffSlots), s>>>(
            p->q, base_u, trial_u, p->u_ref, pce, pcd, p->flags, trial_active));
    }
    {
        svp::KernelTimer _t("cell_barrier_kernel", s);
        SVP_LAUNCH(cell_barrier_kernel<true, true><<<bb, BT, sizeof(double) * 54 * BT, s>>>(
            p->q, base_u, trial_u, p->flags, pbe, pbd, trial_active));
    }
    SVP_LAUNCH_CHECK("cell_trial_kernel");
    // soft sums and differences from the soft kernel, the barrier's from the barrier kernel
    ReduceSpec red;
    red.add(pne, nb, 2, 0);
    red.add(pce, cb, 2, 4);
    red.add(pbe, bb, 2, 8);
    red.add(pnd, nb, 2, 12);
    red.add(pcd, cb, 2, 16);
    red.add(pbd, bb, 1, 20);
    if (screened) red.add(pcb, cb, 4, 22);
    if ((rc = reduce_results(p, red, s))) return rc;
    const double *tmp = p->host;
    // energy terms exactly as svp_energy
    double node2[2], cell3[3];
    for (int k = 0; k < 2; k++) node2[k] = tmp[2 * k] + tmp[2 * k + 1];
    for (int k = 0; k < 3; k++) cell3[k] = tmp[4 + 2 * k] + tmp[4 + 2 * k + 1];
    terms5[0] = .5 * node2[0];
    terms5[1] = .5 * p->q.lam * node2[1];
    terms5[2] = .5 * p->q.mu * cell3[0];
    terms5[3] = .5 * p->q.nu * cell3[1];
    terms5[4] = cell3[2];
    if (barrier_violations) *barrier_violations = (int64_t)(tmp[10] + tmp[11]);
    // differences exactly as svp_energy_difference
    double img = tmp[12] + tmp[13], prox = tmp[14] + tmp[15];
    double jd = tmp[16] + tmp[17], curl = tmp[18] + tmp[19], bar = tmp[20] + tmp[21];
    diff2[0] = (((img + prox) + jd) + curl) + bar;
    diff2[1] = img + bar;
    if (band) {
        *band = 0.;
        if (screened) {
            const double sums[6] = {cell3[0], cell3[1], tmp[22] + tmp[23], tmp[24] + tmp[25], tmp[26] + tmp[27],
                                    tmp[28] + tmp[29]};
            *band = screen_band(p, sums);
        }
    }
    return SVP_OK;
}

extern "C" int svp_trial_energy_active(svp_pair *p, const double *base_u, const double *base_warped,
                                       const double *trial_u, double *trial_warped, double *trial_image_grad,
                                       const uint8_t *base_active, uint8_t *trial_active, double *terms5,
                                       double *diff2, int64_t *barrier_violations, void *stream) {
    return trial_energy(p, base_u, base_warped, trial_u, trial_warped, trial_image_grad, base_active, trial_active,
                        terms5, diff2, barrier_violations, false, nullptr, stream);
}

extern "C" int svp_trial_energy_screened(svp_pair *p, const double *base_u, const double *base_warped,
                                         const double *trial_u, double *trial_warped, double *trial_image_grad,
                                         const uint8_t *base_active, uint8_t *trial_active, double *terms5,
                                         double *diff2, double *band, int64_t *barrier_violations, void *stream) {
    return trial_energy(p, base_u, base_warped, trial_u, trial_warped, trial_image_grad, base_active, trial_active,
                        terms5, diff2, barrier_violations, true, band, stream);
}

extern "C" int svp_trial_energy_masked(svp_pair *p, const double *base_u, const double *base_warped,
                                       const double *trial_u, double *trial_warped, double *trial_image_grad,
                                       uint8_t *trial_active, double *terms5, double *diff2,
                                       int64_t *barrier_violations, void *stream) {
    return svp_trial_energy_active(p, base_u, base_warped, trial_u, trial_warped, trial_image_grad, nullptr,
                                   trial_active, terms5, diff2, barrier_violations, stream);
}

extern "C" int svp_trial_energy(svp_pair *p, const double *base_u, const double *base_warped,
                                const double *trial_u, double *trial_warped, double *trial_image_grad,
                                double *terms5, double *diff2, int64_t *barrier_violations, void *stream) {
    return svp_trial_energy_masked(p, base_u, base_warped, trial_u, trial_warped, trial_image_grad, nullptr, terms5,
                                   diff2, barrier_violations, stream);
}

template <class LT>
static int run_gather(svp_pair *p, const GatherSpec &g, const LT *L1, const LT *L2, const uint8_t *has2,
                      const double *u, const double *uref, const double *warped, const double *image_grad,
                      cudaStream_t s) {
    svp::KernelTimer _t("gather_kernel", s);
    const unsigned nb = node_blocks(p->q.nfree);
    if (L2)
        SVP_LAUNCH((gather_kernel<true, LT><<<nb, 256, 0, s>>>(p->q, g, L1, L2, has2, u, uref, warped, p->fixed,
                                                              image_grad)));
    else
        SVP_LAUNCH((gather_kernel<false, LT><<<nb, 256, 0, s>>>(p->q, g, L1, nullptr, nullptr, u, uref, warped,
                                                               p->fixed, image_grad)));
    return SVP_OK;
}

// The plain form's gradient locals: the soft kernel, then the barrier kernel over the flagged cells (the state's mask,
// or without one the cells the soft kernel flags).  Without a soft penalty its values are zeros, also where the field is
// not finite, and no cell is evaluated for them.  *has2: the cells whose L2 values were written.
static int grad64(svp_pair *p, const double *u, double mu_scale, double nu_scale, bool barrier, bool split,
                  const uint8_t *active, const uint8_t **has2, cudaStream_t s) {
    uint8_t *flags = barrier && !active ? p->flags : nullptr;
    const uint8_t *marked = active ? active : flags;
    if (p->q.mu * mu_scale == 0. && p->q.nu * nu_scale == 0.) {
        SVP_CUDA(cudaMemsetAsync(p->loc1, 0, sizeof(double) * 24 * (size_t)p->q.ncell, s));
        if (flags) SVP_LAUNCH(cell_flag_kernel<<<slice_blocks(p), CS, 0, s>>>(p->q, u, flags));
    } else {
        svp::KernelTimer _t("cell_grad_kernel", s);
        SVP_LAUNCH(cell_grad_kernel<<<slice_blocks(p), CS, slice_bytes(45), s>>>(p->q, u, p->u_ref, mu_scale,
                                                                                nu_scale, p->loc1, flags));
    }
    if (barrier) {
        svp::KernelTimer _t("cell_grad_barrier_kernel", s);
        SVP_LAUNCH(cell_grad_barrier_kernel<<<flagged_blocks(p->q), BT, sizeof(double) * 27 * BT, s>>>(
            p->q, u, marked, split, p->loc1, split ? p->loc2 : nullptr));
    }
    *has2 = split ? marked : nullptr;
    return SVP_OK;
}

// The mixed form's gradient locals: the float32 soft kernel, then the float64 barrier kernel over the flagged cells
// (the state's mask, or without one the cells the soft kernel flags from its float32 closed27 J).
static int grad32(svp_pair *p, const double *u, double mu_scale, double nu_scale, bool barrier, bool split,
                  const uint8_t *active, const uint8_t **has2, cudaStream_t s) {
    uint8_t *flags = barrier && !active ? p->flags : nullptr;
    {
        svp::KernelTimer _t("cell_grad32_kernel", s);
        SVP_LAUNCH(cell_grad32_kernel<<<slice_blocks(p), CS, sizeof(float) * kGrad32Slots * CS, s>>>(
            p->q, u, p->u_ref, mu_scale, nu_scale, (float *)p->loc1, flags));
    }
    if (barrier) {
        svp::KernelTimer _t("cell_grad_barrier32_kernel", s);
        SVP_LAUNCH(cell_grad_barrier32_kernel<<<barrier_blocks(p->q), CB, sizeof(float) * 81 * CB, s>>>(
            p->q, u, active ? active : flags, split, (float *)p->loc1, (float *)p->loc2));
    }
    *has2 = split ? (active ? active : flags) : nullptr;
    return SVP_OK;
}

extern "C" int svp_gradient_masked(svp_pair *p, const double *u, const double *warped, const double *image_grad,
                                   int32_t terms, const uint8_t *active, double *out, void *stream) {
    SVP_REQUIRE(p && u && out, "svp_gradient: null argument");
    SVP_REQUIRE((terms & ~SVP_TERM_TOTAL) == 0 && terms, "svp_gradient: invalid term mask");
    bool img = terms & SVP_TERM_IMAGE;
    SVP_REQUIRE(!img || (warped && image_grad), "svp_gradient: the image term needs warped and image_grad");
    cudaStream_t s = (cudaStream_t)stream;
    const bool mixed = p->precision == SVP_PRECISION_MIXED;
    bool cellwork = terms & (SVP_TERM_JD | SVP_TERM_CURL | SVP_TERM_BARRIER);
    if (cellwork) {
        int rc = pair_locals(p, 1);
        if (rc) return rc;
        const uint8_t *has2;
        if (mixed) {
            if ((rc = grad32(p, u, (terms & SVP_TERM_JD) ? 1. : 0., (terms & SVP_TERM_CURL) ? 1. : 0.,
                             (terms & SVP_TERM_BARRIER) != 0, false, active, &has2, s)))
                return rc;
        } else {
            if ((rc = grad64(p, u, (terms & SVP_TERM_JD) ? 1. : 0., (terms & SVP_TERM_CURL) ? 1. : 0.,
                             (terms & SVP_TERM_BARRIER) != 0, false, active, &has2, s)))
                return rc;
        }
        SVP_LAUNCH_CHECK("cell_grad_kernel");
    }
    GatherSpec g{};
    g.nout = 1;
    g.ci[0] = img ? 1. : 0.;
    g.cp[0] = (terms & SVP_TERM_PROXIMITY) ? 1. : 0.;
    g.c1[0] = cellwork ? 1. : 0.;
    g.out[0] = out;
    if (mixed)
        return run_gather<float>(p, g, cellwork ? (const float *)p->loc1 : nullptr, nullptr, nullptr, u, p->u_ref,
                                 img ? warped : nullptr, img ? image_grad : nullptr, s);
    return run_gather<double>(p, g, cellwork ? p->loc1 : nullptr, nullptr, nullptr, u, p->u_ref, img ? warped : nullptr,
                              img ? image_grad : nullptr, s);
}

extern "C" int svp_outer_gradients_masked(svp_pair *p, const double *u, const double *warped,
                                          const double *image_grad, const uint8_t *active, double *gF, double *gD,
                                          double *gE, void *stream) {
    SVP_REQUIRE(p && u && warped && image_grad && gF && gD && gE, "svp_outer_gradients: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = pair_locals(p, 2);
    if (rc) return rc;
    const bool mixed = p->precision == SVP_PRECISION_MIXED;
    const uint8_t *has2 = nullptr;
    if (mixed) {
        if ((rc = grad32(p, u, 1., 1., true, true, active, &has2, s))) return rc;
    } else {
        if ((rc = grad64(p, u, 1., 1., true, true, active, &has2, s))) return rc;
    }
    SVP_LAUNCH_CHECK("cell_grad_kernel");
    GatherSpec g{};
    g.nout = 3;
    // gF = image + barrier; gD = image; gE = image + proximity + soft + barrier
    g.ci[0] = 1.; g.cp[0] = 0.; g.c1[0] = 0.; g.c2[0] = 1.; g.out[0] = gF;
    g.ci[1] = 1.; g.cp[1] = 0.; g.c1[1] = 0.; g.c2[1] = 0.; g.out[1] = gD;
    g.ci[2] = 1.; g.cp[2] = 1.; g.c1[2] = 1.; g.c2[2] = 0.; g.out[2] = gE;
    if (mixed) return run_gather<float>(p, g, (const float *)p->loc1, (const float *)p->loc2, has2, u, p->u_ref, warped, image_grad, s);
    return run_gather<double>(p, g, p->loc1, p->loc2, has2, u, p->u_ref, warped, image_grad, s);
}

extern "C" int svp_ggn_diagonal_masked(svp_pair *p, const double *u, const double *image_grad,
                                       const uint8_t *active, double *out, void *stream) {
    SVP_REQUIRE(p && u && image_grad && out, "svp_ggn_diagonal: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = pair_locals(p, 1);
    if (rc) return rc;
    if (p->precision == SVP_PRECISION_MIXED) {
        {
            svp::KernelTimer _t("cell_ggn_diag32_kernel", s);
            SVP_LAUNCH(cell_ggn_diag32_kernel<<<cell_blocks(p), CT, 0, s>>>(p->q, u, (float *)p->loc1,
                                                                           active ? nullptr : p->flags));
        }
        {
            svp::KernelTimer _t("cell_ggn_barrier32_kernel", s);
            SVP_LAUNCH(cell_ggn_barrier32_kernel<<<barrier_blocks(p->q), CB, 0, s>>>(
                p->q, u, active ? active : p->flags, (float *)p->loc1));
        }
        SVP_LAUNCH(ggn_node_kernel<float><<<node_blocks(p->q.nfree), 256, 0, s>>>(p->q, (const float *)p->loc1, image_grad, nullptr, out));
    } else {
        {
            svp::KernelTimer _t("cell_ggn_diag_kernel", s);
            SVP_LAUNCH(cell_ggn_diag_kernel<<<slice_blocks(p), CS, 0, s>>>(p->q, u, p->loc1,
                                                                         active ? nullptr : p->flags));
        }
        {
            svp::KernelTimer _t("cell_ggn_barrier_kernel", s);
            SVP_LAUNCH(cell_ggn_barrier_kernel<<<flagged_blocks(p->q), BT, sizeof(double) * 27 * BT, s>>>(
                p->q, u, active ? active : p->flags, p->loc1));
        }
        SVP_LAUNCH(ggn_node_kernel<double><<<node_blocks(p->q.nfree), 256, 0, s>>>(p->q, p->loc1, image_grad, nullptr, out));
    }
    SVP_LAUNCH_CHECK("ggn diagonal");
    return SVP_OK;
}

extern "C" int svp_gradient(svp_pair *p, const double *u, const double *warped, const double *image_grad,
                            int32_t terms, double *out, void *stream) {
    return svp_gradient_masked(p, u, warped, image_grad, terms, nullptr, out, stream);
}
extern "C" int svp_outer_gradients(svp_pair *p, const double *u, const double *warped, const double *image_grad,
                                   double *gF, double *gD, double *gE, void *stream) {
    return svp_outer_gradients_masked(p, u, warped, image_grad, nullptr, gF, gD, gE, stream);
}
extern "C" int svp_ggn_diagonal(svp_pair *p, const double *u, const double *image_grad, double *out,
                                void *stream) {
    return svp_ggn_diagonal_masked(p, u, image_grad, nullptr, out, stream);
}

extern "C" int svp_ggn_hvp(svp_pair *p, const double *u, const double *image_grad, const double *pvec,
                           double *out, void *stream) {
    SVP_REQUIRE(p && u && image_grad && pvec && out, "svp_ggn_hvp: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = pair_locals(p, 2);
    if (rc) return rc;
    // inject p into a node field (zero faces) held in loc2's storage
    double *vv = p->loc2;
    rc = svp_inject(&p->grid, pvec, vv, stream);
    if (rc) return rc;
    { svp::KernelTimer _t("cell_ggn_hvp_kernel", s); SVP_LAUNCH(cell_ggn_hvp_kernel<<<slice_blocks(p), CS, slice_bytes(81), s>>>(p->q, u, vv, p->loc1)); }
    SVP_LAUNCH(ggn_node_kernel<double><<<node_blocks(p->q.nfree), 256, 0, s>>>(p->q, p->loc1, image_grad, vv, out));
    SVP_LAUNCH_CHECK("ggn hvp");
    return SVP_OK;
}

extern "C" int svp_node_min_jd_extended(svp_pair *p, const double *u, double extension_activation, double *node,
                                        int64_t *candidates, void *stream) {
    SVP_REQUIRE(p && u && node, "svp_node_min_jd: null argument");
    SVP_REQUIRE(!(extension_activation < 0.) && extension_activation == extension_activation,
                "svp_node_min_jd: extension activation must be >= 0 (0: no extension)");
    cudaStream_t s = (cudaStream_t)stream;
    const bool ext = extension_activation > 0.;
    if (ext && !p->cand) SVP_CUDA(cudaMalloc((void **)&p->cand, sizeof(long long) * p->q.ncell));
    unsigned long long *ncand = (unsigned long long *)(p->counter + 4);
    if (ext) SVP_CUDA(cudaMemsetAsync(ncand, 0, sizeof(unsigned long long), s));
    { svp::KernelTimer _t("cell_min_jd_kernel", s); SVP_LAUNCH(cell_min_jd_kernel<<<slice_blocks(p), CS, slice_bytes(27), s>>>(p->q, u, p->cellbuf, ext ? extension_activation : 0., ncand, p->cand)); }
    if (ext) {
        svp::KernelTimer _t("jd_extension_kernel", s);
        SVP_LAUNCH(jd_extension_kernel<<<148 * 4, 128, 0, s>>>(p->q, u, ncand, p->cand, p->cellbuf));
    }
    SVP_LAUNCH(node_min_kernel<<<node_blocks(p->q.nnode), 256, 0, s>>>(p->q, p->cellbuf, node));
    SVP_LAUNCH_CHECK("node_min_jd");
    if (candidates) {
        unsigned long long nc = 0;
        if (ext) {
            SVP_CUDA(cudaMemcpyAsync(&nc, ncand, sizeof nc, cudaMemcpyDeviceToHost, s));
            SVP_CUDA(cudaStreamSynchronize(s));
        }
        *candidates = (int64_t)nc;
    }
    return SVP_OK;
}

extern "C" int svp_node_min_jd(svp_pair *p, const double *u, double *node, void *stream) {
    return svp_node_min_jd_extended(p, u, 0., node, nullptr, stream);
}

extern "C" int svp_jd_root(svp_pair *p, const double *u, const double *pvec, double limit, double *root,
                           int64_t *invalid, void *stream) {
    SVP_REQUIRE(p && u && pvec && root && limit > 0, "svp_jd_root: invalid argument");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = pair_locals(p, 2);
    if (rc) return rc;
    double *vv = p->loc2;
    rc = svp_inject(&p->grid, pvec, vv, stream);
    if (rc) return rc;
    long long init[2] = {kKeyPosInf, 0};
    SVP_CUDA(cudaMemcpyAsync(p->counter, init, sizeof init, cudaMemcpyHostToDevice, s));
    { svp::KernelTimer _t("jd_root_kernel", s); SVP_LAUNCH(jd_root_kernel<<<cell_blocks(p), CT, 0, s>>>(p->q, u, vv, limit, p->counter,
                                                 (unsigned long long *)(p->counter + 1))); }
    SVP_LAUNCH_CHECK("jd_root_kernel");
    long long out[2];
    SVP_CUDA(cudaMemcpyAsync(out, p->counter, sizeof out, cudaMemcpyDeviceToHost, s));
    SVP_CUDA(cudaStreamSynchronize(s));
    double sv = key_value(out[0]);
    *root = std::isfinite(sv) ? sv * limit : INFINITY;
    if (invalid) *invalid = out[1];
    return SVP_OK;
}

extern "C" int svp_image_shift(svp_pair *p, const double *image_grad, double factor, double *alpha, void *stream) {
    SVP_REQUIRE(p && image_grad && alpha, "svp_image_shift: null argument");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned nb = node_blocks(p->q.nfree);
    SVP_LAUNCH(shift_kernel<<<nb, 256, 0, s>>>(p->q, image_grad, p->partial));
    SVP_LAUNCH_CHECK("shift kernels");
    ReduceSpec red;
    red.add(p->partial, nb, 1, 0);
    int rc = reduce_results(p, red, s);
    if (rc) return rc;
    const double *tmp = p->host;
    *alpha = factor * ((tmp[0] + tmp[1]) / (double)p->q.nfree) / 3;
    return SVP_OK;
}

extern "C" int svp_pg_scale(svp_pair *p, const double *diag, const double *node_jd, double m, double activation,
                            double floor_, double *scale, int64_t *bad, void *stream) {
    SVP_REQUIRE(p && diag && node_jd && scale && m > 0 && activation > 0, "svp_pg_scale: invalid argument");
    cudaStream_t s = (cudaStream_t)stream;
    SVP_CUDA(cudaMemsetAsync(p->counter, 0, sizeof(long long), s));
    SVP_LAUNCH(pg_scale_kernel<<<node_blocks(p->q.nfree), 256, 0, s>>>(p->q, diag, node_jd, std::sqrt(m), activation, floor_,
                                                            scale, (unsigned long long *)p->counter));
    SVP_LAUNCH_CHECK("pg_scale_kernel");
    long long host = 0;
    SVP_CUDA(cudaMemcpyAsync(&host, p->counter, sizeof host, cudaMemcpyDeviceToHost, s));
    SVP_CUDA(cudaStreamSynchronize(s));
    if (bad) *bad = host;
    return SVP_OK;
}
