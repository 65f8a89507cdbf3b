// Q1 cell geometry on the B200: separable evaluation of grad u at the Gauss27 / closed27 points, its adjoint,
// the localized C2 barrier, and deterministic double-double block reductions.
#pragma once
#include "svp_common.cuh"

namespace svp {

// Constants of one registration pair (passed by value: constant bank, race-free across concurrent pairs).
struct Q1Const {
    long long nx, ny, nz, cx, cy, cz, ncell, nnode;
    long long fx, fy, fz, nfree;   // free (interior) node counts per axis and in total
    double h[3], ih[3];            // spacing and fl(1/h) (cell_q1.py:126 divides +-1 by h)
    double gn[3], gm[3];           // Gauss nodes xi and 1 - xi (cell_q1.py:106)
    double gw[27];                 // Gauss27 weights omega*wx*wy*wz, p = 9 iz + 3 iy + ix (cell_q1.py:115)
    double omega;
    double lam, mu, nu, bw;        // weights; bw = kappa omega / 27 (problem.py:310)
    double act, delta;             // localized barrier activation a and delta
    double x0[3];                  // node axis origins (x, y, z)
    float gnf[3], gmf[3], gwf[27], ihf[3];   // the same rule constants rounded to float (the mixed form's kernels)
    // the curl term of the GGN diagonal does not depend on the state: per vertex a and component r,
    // nu sum_p gw[p] sum_(j != r) D_j(p, a)^2 over the Gauss points (index 3 a + r), float copy for the mixed form
    double ggn_curl[24];
    float ggn_curlf[24];
};

// ------------------------------------------------------------------------------------------- double-double
struct dd {
    double hi, lo;
};
__device__ __forceinline__ dd two_sum(double a, double b) {
    double s = a + b;
    double bb = s - a;
    double e = (a - (s - bb)) + (b - bb);
    return {s, e};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    dd s = two_sum(a.hi, b.hi);
    dd t = two_sum(a.lo, b.lo);
    s.lo += t.hi;
    s = two_sum(s.hi, s.lo);
    s.lo += t.lo;
    return two_sum(s.hi, s.lo);
}
__device__ __forceinline__ dd dd_add_d(dd a, double b) {
    dd s = two_sum(a.hi, b);
    s.lo += a.lo;
    return two_sum(s.hi, s.lo);
}
// exact product as an unevaluated pair (FMA)
__device__ __forceinline__ dd two_prod(double a, double b) {
    double p = a * b;
    return {p, fma(a, b, -p)};
}
__device__ __forceinline__ dd dd_shfl_xor(dd a, int o) {
    return {__shfl_xor_sync(0xFFFFFFFFu, a.hi, o), __shfl_xor_sync(0xFFFFFFFFu, a.lo, o)};
}

// Sums of K double-doubles over a warp, lanes 16, 8, 4, 2, 1 apart.  While a lane holds several values it keeps half of
// them and sends the others to its partner, so 6 values take 8 additions per lane in place of 30 (each is 26 float64
// operations: at one element per thread they are the kernel).  dd_add is symmetric, so every value has the bits of
// adding it in all lanes.  Value `first` is in acc[0] of the one lane that returns true for it.
template <int K>
__device__ __forceinline__ bool warp_reduce_dd(dd (&acc)[K], int &first) {
    const int lane = threadIdx.x & 31;
    int count = K, same = 0;      // values of this lane (`have` at most); lane bits over which the sums are equal
    first = 0;
#pragma unroll
    for (int o = 16, have = K; o; o >>= 1) {
        const int low = (have + 1) / 2;
        if (have > 1) {
            const bool up = lane & o;
#pragma unroll
            for (int k = 0; k < K; k++)
                if (k < low) {
                    const dd upper = k + low < have ? acc[(k + low) % K] : dd{0., 0.};
                    const dd got = dd_shfl_xor(up ? acc[k] : upper, o);
                    acc[k] = dd_add(up ? upper : acc[k], got);
                }
            first += up ? low : 0;
            count = up ? count - low : (count < low ? count : low);
        } else {
            acc[0] = dd_add(acc[0], dd_shfl_xor(acc[0], o));
            same |= o;
        }
        have = low;
    }
    return count > 0 && !(lane & same);
}

// Block reduction of K double-double accumulators, fixed tree order: value k of block b to partial[b][k].
template <int K>
__device__ void block_reduce_dd(dd (&acc)[K], dd *partial) {
    __shared__ dd sh[32][K];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int first;
    if (warp_reduce_dd<K>(acc, first)) sh[warp][first] = acc[0];
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < K; k++) acc[k] = lane < nw ? sh[lane][k] : dd{0., 0.};
        if (warp_reduce_dd<K>(acc, first)) partial[(size_t)blockIdx.x * K + first] = acc[0];
    }
}

// One of K interleaved block sums, added up by a block of 256: thread t takes blocks t, t + 256, ... in order (four
// loads in flight), then a fixed tree, whose last 32 values need no barrier.  Thread 0 returns the sum.
__device__ __forceinline__ dd sum_partials(const dd *__restrict__ partial, long long blocks, int K, int k) {
    __shared__ dd sh[256];
    const int t = threadIdx.x;
    dd acc = {0., 0.};
    for (long long b = t; b < blocks; b += 1024) {
        dd v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = b + 256 * j < blocks ? partial[(b + 256 * j) * K + k] : dd{0., 0.};
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (b + 256 * j < blocks) acc = dd_add(acc, v[j]);
    }
    sh[t] = acc;
    __syncthreads();
    if (t < 128) sh[t] = acc = dd_add(acc, sh[t + 128]);
    __syncthreads();
    if (t < 64) sh[t] = acc = dd_add(acc, sh[t + 64]);
    __syncthreads();
    if (t < 32) {
        acc = dd_add(acc, sh[t + 32]);
#pragma unroll
        for (int o = 16; o; o >>= 1) acc = dd_add(acc, dd_shfl_xor(acc, o));
    }
    return acc;
}

// ------------------------------------------------------------------------------------------- cell geometry
__device__ __forceinline__ long long cell_node0(long long c, const Q1Const &q) {
    long long x0, y0, z0;
    unflatten3(c, q.cx, q.cy, x0, y0, z0);
    return (z0 * q.ny + y0) * q.nx + x0;
}
__device__ __forceinline__ long long vertex_node(long long n0, int a, const Q1Const &q) {
    return n0 + (long long)(a >> 2) * q.ny * q.nx + (long long)((a >> 1) & 1) * q.nx + (a & 1);
}

template <class T>
__device__ __forceinline__ void load_cell(const T *__restrict__ u, long long n0, const Q1Const &q, T v[8][3]) {
#pragma unroll
    for (int a = 0; a < 8; a++) {
        const T *p = u + 3 * vertex_node(n0, a, q);
        v[a][0] = __ldg(p);
        v[a][1] = __ldg(p + 1);
        v[a][2] = __ldg(p + 2);
    }
}

// Edge differences E[j][e][r]: axis j, edge e over the two other vertex bits in increasing order
// (j = 0: e = y + 2z; j = 1: e = x + 2z; j = 2: e = x + 2y).
template <class T>
__device__ __forceinline__ void cell_edges(const T v[8][3], T E[3][4][3]) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
        int lo = e & 1, hi = e >> 1;
        int ax = 2 * lo + 4 * hi, ay = lo + 4 * hi, az = lo + 2 * hi;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            E[0][e][r] = v[ax | 1][r] - v[ax][r];
            E[1][e][r] = v[ay | 2][r] - v[ay][r];
            E[2][e][r] = v[az | 4][r] - v[az][r];
        }
    }
}

// Column j of grad u at one point, straight from the edges: first along the lower-numbered other axis (node s), then
// along the higher (t); n nodes, m = 1 - nodes.
template <int J, class T>
__device__ __forceinline__ void column(const T E[3][4][3], T ms, T ns, T mt, T nt, T ih, T out[3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
        T l0 = ms * E[J][0][r] + ns * E[J][1][r];
        T l1 = ms * E[J][2][r] + ns * E[J][3][r];
        out[r] = (mt * l0 + nt * l1) * ih;
    }
}

// Point coordinates of the two 3-point rules: Gauss (nodes q.gn, 1 - nodes q.gm) or closed (0, 1/2, 1).
template <bool CLOSED>
__device__ __forceinline__ double rule_n(const Q1Const &q, int i) { return CLOSED ? .5 * i : q.gn[i]; }
template <bool CLOSED>
__device__ __forceinline__ double rule_m(const Q1Const &q, int i) { return CLOSED ? 1. - .5 * i : q.gm[i]; }
// the rule's nodes and 1/h in the arithmetic type R (float: the rounded constants, no conversion in the sweeps)
template <bool CLOSED, class R>
__device__ __forceinline__ R node_n(const Q1Const &q, int i) {
    if constexpr (sizeof(R) == 4) return CLOSED ? .5f * (float)i : q.gnf[i];
    else return rule_n<CLOSED>(q, i);
}
template <bool CLOSED, class R>
__device__ __forceinline__ R node_m(const Q1Const &q, int i) {
    if constexpr (sizeof(R) == 4) return CLOSED ? 1.f - .5f * (float)i : q.gmf[i];
    else return rule_m<CLOSED>(q, i);
}
template <class R>
__device__ __forceinline__ R inv_h(const Q1Const &q, int k) {
    if constexpr (sizeof(R) == 4) return q.ihf[k];
    else return q.ih[k];
}

// Visit the 27 points p = 9 iz + 3 iy + ix of a rule with grad u at each, V[r][j].  Column x depends only on
// (iy, iz) and column y only on (ix, iz), so x is evaluated once per (iy, iz) and y once per (ix, iz): 45 column
// evaluations instead of 81, each bitwise the one of column<J> at that point.  Fields: one (sweep) or two
// (sweep2, same points); body(p, ix, iy, iz, V[, V2]).
template <bool CLOSED, class R = double, class Body>
__device__ __forceinline__ void sweep(const R E[3][4][3], const Q1Const &q, Body &&body) {
    const R ih0 = inv_h<R>(q, 0), ih1 = inv_h<R>(q, 1), ih2 = inv_h<R>(q, 2);
#pragma unroll 1
    for (int iz = 0; iz < 3; iz++) {
        const R nz = node_n<CLOSED, R>(q, iz), mz = node_m<CLOSED, R>(q, iz);
        R Y[3][3];
#pragma unroll
        for (int ix = 0; ix < 3; ix++)
            column<1>(E, node_m<CLOSED, R>(q, ix), node_n<CLOSED, R>(q, ix), mz, nz, ih1, Y[ix]);
#pragma unroll 1
        for (int iy = 0; iy < 3; iy++) {
            const R ny = node_n<CLOSED, R>(q, iy), my = node_m<CLOSED, R>(q, iy);
            R X[3];
            column<0>(E, my, ny, mz, nz, ih0, X);
#pragma unroll
            for (int ix = 0; ix < 3; ix++) {
                R Z[3];
                column<2>(E, node_m<CLOSED, R>(q, ix), node_n<CLOSED, R>(q, ix), my, ny, ih2, Z);
                R V[3][3] = {{X[0], Y[ix][0], Z[0]}, {X[1], Y[ix][1], Z[1]}, {X[2], Y[ix][2], Z[2]}};
                body(9 * iz + 3 * iy + ix, ix, iy, iz, V);
            }
        }
    }
}
template <bool CLOSED, class R = double, class Body>
__device__ __forceinline__ void sweep2(const R E[3][4][3], const R E2[3][4][3], const Q1Const &q, Body &&body) {
    const R ih0 = inv_h<R>(q, 0), ih1 = inv_h<R>(q, 1), ih2 = inv_h<R>(q, 2);
#pragma unroll 1
    for (int iz = 0; iz < 3; iz++) {
        const R nz = node_n<CLOSED, R>(q, iz), mz = node_m<CLOSED, R>(q, iz);
#pragma unroll 1
        for (int iy = 0; iy < 3; iy++) {
            const R ny = node_n<CLOSED, R>(q, iy), my = node_m<CLOSED, R>(q, iy);
            R X[3], X2[3];
            column<0>(E, my, ny, mz, nz, ih0, X);
            column<0>(E2, my, ny, mz, nz, ih0, X2);
#pragma unroll 1
            for (int ix = 0; ix < 3; ix++) {
                const R nx = node_n<CLOSED, R>(q, ix), mx = node_m<CLOSED, R>(q, ix);
                R Y[3], Z[3], Y2[3], Z2[3];
                column<1>(E, mx, nx, mz, nz, ih1, Y);
                column<2>(E, mx, nx, my, ny, ih2, Z);
                column<1>(E2, mx, nx, mz, nz, ih1, Y2);
                column<2>(E2, mx, nx, my, ny, ih2, Z2);
                R V[3][3] = {{X[0], Y[0], Z[0]}, {X[1], Y[1], Z[1]}, {X[2], Y[2], Z[2]}};
                R V2[3][3] = {{X2[0], Y2[0], Z2[0]}, {X2[1], Y2[1], Z2[1]}, {X2[2], Y2[2], Z2[2]}};
                body(9 * iz + 3 * iy + ix, ix, iy, iz, V, V2);
            }
        }
    }
}

// Cofactor rows (cross products of cyclic rows of F = I + V) and J = F0 . A0 (geometry.py:11 cofactor, :26 determinant).
template <class T>
__device__ __forceinline__ void cofactor_det(const T V[3][3], T A[3][3], T &J) {
    T F[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) F[r][c] = V[r][c] + (r == c ? T(1) : T(0));
#pragma unroll
    for (int r = 0; r < 3; r++) {
        int j = (r + 1) % 3, k = (r + 2) % 3;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            int l = (c + 1) % 3, mm = (c + 2) % 3;
            A[r][c] = F[j][l] * F[k][mm] - F[j][mm] * F[k][l];
        }
    }
    J = (F[0][0] * A[0][0] + F[0][1] * A[0][1]) + F[0][2] * A[0][2];
}
template <class T>
__device__ __forceinline__ T det_only(const T V[3][3]) {
    T F[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) F[r][c] = V[r][c] + (r == c ? T(1) : T(0));
    T a0 = F[1][1] * F[2][2] - F[1][2] * F[2][1];
    T a1 = F[1][2] * F[2][0] - F[1][0] * F[2][2];
    T a2 = F[1][0] * F[2][1] - F[1][1] * F[2][0];
    return (F[0][0] * a0 + F[0][1] * a1) + F[0][2] * a2;
}
template <class T>
__device__ __forceinline__ void curl_of(const T V[3][3], T C[3]) {
    C[0] = V[2][1] - V[1][2];
    C[1] = V[0][2] - V[2][0];
    C[2] = V[1][0] - V[0][1];
}

// ------------------------------------------------------------------------------------------- localized barrier
// barrier.py:18-36: b = -w r^2 log t, b' and b'' for J < a (zero above); log t via log1p(-r) when r < 1/2.
__device__ __forceinline__ void barrier_eval(double J, double a, double delta, double w, double &b, double &b1,
                                             double &b2) {
    b = b1 = b2 = 0.;
    if (!(J < a)) return;
    double scale = a - delta;
    double t = (J - delta) / scale;
    double r = (a - J) / scale;
    double logt = r < .5 ? log1p(-r) : log(t);
    b = -w * r * r * logt;
    b1 = w * (2 * r * logt - r * r / t) / scale;
    double rt = r / t;
    b2 = w * (-2 * logt + 4 * r / t + rt * rt) / (scale * scale);
}

// The same barrier's value, slope and stable change (energy_comparison.py:14-62) for the float64 kernels that walk many
// points, each with what it needs alone.  The scale a - delta divides: its reciprocal is a constant of the pair, so its
// rounding would be a bias that the sum over the points keeps (2 units of 2^-53 of the sum at a = .5, delta = .001).
struct BarrierRule {
    double a, delta, w, scale;    // activation, delta, weight, a - delta
};
__device__ __forceinline__ BarrierRule barrier_rule(const Q1Const &q) {
    return {q.act, q.delta, q.bw, q.act - q.delta};
}
// log t, t = (J - delta) / (a - delta) = 1 - r
__device__ __forceinline__ double barrier_log(double r, double t) { return r < .5 ? log1p(-r) : log(t); }
__device__ __forceinline__ double barrier_value(double J, const BarrierRule &k) {
    const double r = (k.a - J) / k.scale, t = (J - k.delta) / k.scale;
    return -k.w * r * r * barrier_log(r, t);
}
__device__ __forceinline__ double barrier_slope(double J, const BarrierRule &k) {
    const double r = (k.a - J) / k.scale, t = (J - k.delta) / k.scale;
    return k.w * (2. * r * barrier_log(r, t) - r * r / t) / k.scale;
}
// psi(jb) - psi(ja), unweighted
__device__ __forceinline__ double barrier_change(double ja, double jb, const BarrierRule &k) {
    const double a = ja < k.a ? ja : k.a, b = jb < k.a ? jb : k.a;
    const double ra = (k.a - a) / k.scale, rb = (k.a - b) / k.scale, h = (b - a) / k.scale;
    const double x = (b - a) / (a - k.delta);
    const double ratio = x >= -.5 ? log1p(x) : log((b - k.delta) / (a - k.delta));
    return h * (ra + rb) * barrier_log(ra, (a - k.delta) / k.scale) - rb * rb * ratio;
}

}  // namespace svp
