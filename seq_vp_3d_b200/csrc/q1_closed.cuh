// Exact Q1 cell algebra on the closed27 points (0, 1/2, 1)^3.
//
// On a trilinear cell, column j of grad u is bilinear in the two other coordinates, J = det(I + grad u) is quadratic
// and a curl component linear in each coordinate.  So
//  - the columns at the closed27 points are edge differences and averages of two (90 operations for all 27 points,
//    against 1,350 for the general evaluation at the Gauss points);
//  - J at the closed27 points determines J, and the 27-point Gauss sums of the JD penalty (exact for the fourth
//    powers that (J - Jr)^2 has) equal the integrals of the interpolating quadratics: diagonal sums in the Legendre
//    basis, or the tensor product of the 1D mass matrix [4 2 -1; 2 16 2; -1 2 4] / 30;
//  - the curl penalty is a sum of squares of 18 Hadamard coefficients of edge differences.
// The localized barrier and the node measure are defined on the closed27 points.  Every sum equals the Gauss27 form's
// in exact arithmetic.  J is formed in two ways, each where it is the closer one:
//  - for a residual J - Jr, J - 1 from grad u without adding the identity first: it rounds relative to |grad u| and not
//    to 1.  Against 80-bit sums the JD penalty and its changes are 1.5 to 9 times closer than the Gauss27 form with F =
//    I + grad u (which 27 independent point errors average), at 2 of 11 operations per point;
//  - for J itself, the determinant of F = I + grad u: its products keep a small J's relative accuracy (5e-16 at J =
//    1e-6, where 1 + (J - 1) has 6e-11 and the barrier's slope and curvature go like 1/J and 1/J^2), at 9 operations
//    per point.
// The operations are explicit round-to-nearest intrinsics: each kernel that evaluates a cell gets the same bits.
#pragma once
#include "q1_common.cuh"

namespace svp {

// Columns of grad u on the cell's edges: X[y + 2 z], Y[x + 2 z], Z[x + 2 y], components r.
struct Columns {
    double X[4][3], Y[4][3], Z[4][3];
};

__device__ __forceinline__ double mean2(double a, double b) { return __dmul_rn(.5, __dadd_rn(a, b)); }

// ID: the columns of F = I + grad u, the identity added in one rounding (of F, which a compression makes small, and not
// of grad u).
template <bool ID = false>
__device__ __forceinline__ void vertex_columns(const double (&v)[8][3], const Q1Const &q, Columns &C) {
    auto entry = [](double difference, double ih, bool diagonal) {
        return ID && diagonal ? __fma_rn(difference, ih, 1.) : __dmul_rn(difference, ih);
    };
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int lo = e & 1, hi = e >> 1;
        const int ax = 2 * lo + 4 * hi, ay = lo + 4 * hi, az = lo + 2 * hi;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            C.X[e][r] = entry(__dsub_rn(v[ax | 1][r], v[ax][r]), q.ih[0], r == 0);
            C.Y[e][r] = entry(__dsub_rn(v[ay | 2][r], v[ay][r]), q.ih[1], r == 1);
            C.Z[e][r] = entry(__dsub_rn(v[az | 4][r], v[az][r]), q.ih[2], r == 2);
        }
    }
}
template <bool ID = false>
__device__ __forceinline__ void load_columns(const double *__restrict__ u, long long n0, const Q1Const &q,
                                             Columns &C) {
    double v[8][3];
    load_cell(u, n0, q, v);
    vertex_columns<ID>(v, q, C);
}

// The column values of one plane t (0, 1, 2) of its higher other coordinate: P[s][r], s the lower other coordinate.
__device__ __forceinline__ void column_plane(const double (&E)[4][3], int t, double (&P)[3][3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
        P[0][r] = t == 0 ? E[0][r] : (t == 2 ? E[2][r] : mean2(E[0][r], E[2][r]));
        P[2][r] = t == 0 ? E[1][r] : (t == 2 ? E[3][r] : mean2(E[1][r], E[3][r]));
        P[1][r] = mean2(P[0][r], P[2][r]);
    }
}

// Visits the closed27 points p = 9 iz + 3 iy + ix: body(p, ix, iy, iz, X, Y, Z) with the columns at the point.
template <class Body>
__device__ __forceinline__ void closed_points(const Columns &C, Body &&body) {
    double Z[3][3][3];     // [iy][ix][r]
#pragma unroll
    for (int iy = 0; iy < 3; iy++) column_plane(C.Z, iy, Z[iy]);
#pragma unroll
    for (int iz = 0; iz < 3; iz++) {
        double X[3][3], Y[3][3];
        column_plane(C.X, iz, X);
        column_plane(C.Y, iz, Y);
#pragma unroll
        for (int iy = 0; iy < 3; iy++)
#pragma unroll
            for (int ix = 0; ix < 3; ix++) body(9 * iz + 3 * iy + ix, ix, iy, iz, X[iy], Y[ix], Z[iy][ix]);
    }
}

// J - 1 for the columns of grad u at a point: F = I + (x, y, z), J = X . (Y x Z) = (1 + x0)(1 + k) + x1 c1 + x2 c2
__device__ __forceinline__ double det_minus_one(const double (&x)[3], const double (&y)[3], const double (&z)[3]) {
    const double k = __fma_rn(-y[2], z[1], __fma_rn(y[1], z[2], __dadd_rn(y[1], z[2])));
    const double c1 = __fma_rn(-y[0], z[2], __fma_rn(y[2], z[0], -y[0]));
    const double c2 = __fma_rn(-y[1], z[0], __fma_rn(y[0], z[1], -z[0]));
    return __fma_rn(x[2], c2, __fma_rn(x[1], c1, __fma_rn(x[0], k, __dadd_rn(x[0], k))));
}
// The bound on J - 1 below which J may be below the activation a.  The two forms of J differ by some 20 roundings of
// products of three column entries, less than 2^-30 for entries up to 100.
__device__ __forceinline__ double near_bound(double a) { return __dadd_rn(__dsub_rn(a, 1.), 0x1p-30); }

// Adds the identity: columns of F from those of grad u.
__device__ __forceinline__ void add_identity(Columns &C) {
#pragma unroll
    for (int e = 0; e < 4; e++) {
        C.X[e][0] = __dadd_rn(C.X[e][0], 1.);
        C.Y[e][1] = __dadd_rn(C.Y[e][1], 1.);
        C.Z[e][2] = __dadd_rn(C.Z[e][2], 1.);
    }
}
// J for the columns x, y, z of F at a point, expanded along the first row as det_only
__device__ __forceinline__ double det_columns(const double (&x)[3], const double (&y)[3], const double (&z)[3]) {
    const double c0 = __fma_rn(y[1], z[2], -__dmul_rn(y[2], z[1])), c1 = __fma_rn(z[1], x[2], -__dmul_rn(z[2], x[1])),
                 c2 = __fma_rn(x[1], y[2], -__dmul_rn(x[2], y[1]));
    return __fma_rn(z[0], c2, __fma_rn(y[0], c1, __dmul_rn(x[0], c0)));
}
// every entry finite (the largest exponent seen, on the integer pipe)
__device__ __forceinline__ bool finite_columns(const Columns &C) {
    int top = 0;
#pragma unroll
    for (int e = 0; e < 4; e++)
#pragma unroll
        for (int r = 0; r < 3; r++)
            top = max(max(top, __double2hiint(C.X[e][r]) & 0x7FFFFFFF),
                      max(__double2hiint(C.Y[e][r]) & 0x7FFFFFFF, __double2hiint(C.Z[e][r]) & 0x7FFFFFFF));
    return top < 0x7FF00000;
}
// The general evaluation interpolates all four edges of a column at every point, so that an edge that is not finite
// reaches also the points where its weight is zero (0 times NaN or an infinity).  closed_points leaves it out there: the
// J of those points become NaN here.  Rolled loops on the field in memory, so that the finite cells' registers stay
// (the general evaluation itself in its place left 176 bytes of spills in the trial's barrier kernel).
__device__ __forceinline__ void spread_nonfinite(const double *__restrict__ u, long long n0, const Q1Const &q,
                                                 double *sl, int T) {
#pragma unroll 1
    for (int i = 0; i < 12; i++) {
        const int j = i >> 2, lo = i & 1, hi = (i >> 1) & 1;
        const int a = j == 0 ? 2 * lo + 4 * hi : (j == 1 ? lo + 4 * hi : lo + 2 * hi);
        const double *v0 = u + 3 * vertex_node(n0, a, q), *v1 = u + 3 * vertex_node(n0, a | (1 << j), q);
        if (finite64(v1[0] - v0[0]) && finite64(v1[1] - v0[1]) && finite64(v1[2] - v0[2])) continue;
#pragma unroll 1
        for (int p = 0; p < 27; p++) {
            const int s = j == 0 ? (p / 3) % 3 : p % 3, t = j == 2 ? (p / 3) % 3 : p / 9;
            if (s == 2 - 2 * lo || t == 2 - 2 * hi) sl[p * T] = __longlong_as_double(0x7FF8000000000000LL);
        }
    }
}
// The closed27 J of a cell into sl[p T]; C then holds the columns of F.  False where some column is not finite.
__device__ __forceinline__ bool closed_jacobians(const double *__restrict__ u, long long n0, const Q1Const &q,
                                                 Columns &C, double *sl, int T) {
    load_columns<true>(u, n0, q, C);
    const bool finite = finite_columns(C);
    closed_points(C, [&](int p, int, int, int, const double (&X)[3], const double (&Y)[3], const double (&Z)[3]) {
        sl[p * T] = det_columns(X, Y, Z);
    });
    if (!finite) spread_nonfinite(u, n0, q, sl, T);
    return finite;
}

// ------------------------------------------------------------------------------------------- JD penalty
// Values at (0, 1/2, 1) -> Legendre coefficients of the interpolating quadratic, per axis and in place: (a, b, c) ->
// (a + 4 b + c, c - a, a - 2 b + c), with integral square c0^2 / 36 + c1^2 / 12 + c2^2 / 45.
__device__ __forceinline__ void legendre27(double (&c)[27]) {
#pragma unroll
    for (int axis = 0; axis < 3; axis++) {
        const int st = axis == 0 ? 1 : (axis == 1 ? 3 : 9);
#pragma unroll
        for (int l = 0; l < 9; l++) {
            const int o = axis == 0 ? 3 * l : (axis == 1 ? (l / 3) * 9 + l % 3 : l);
            const double a = c[o], b = c[o + st], d = c[o + 2 * st], e = __dadd_rn(a, d);
            c[o] = __fma_rn(4., b, e);
            c[o + st] = __dsub_rn(d, a);
            c[o + 2 * st] = __fma_rn(-2., b, e);
        }
    }
}
// the ten distinct products of the 1D weights: class of a coefficient by how many of its indices are 1 and 2
__device__ constexpr int legendre_class(int k) {
    const int i[3] = {k % 3, (k / 3) % 3, k / 9};
    int n1 = 0, n2 = 0;
    for (int a = 0; a < 3; a++) {
        n1 += i[a] == 1;
        n2 += i[a] == 2;
    }
    return n2 == 0 ? n1 : (n2 == 1 ? 4 + n1 : (n2 == 2 ? 7 + n1 : 9));
}
__device__ constexpr double legendre_weight(int cls) {
    const int n2 = cls < 4 ? 0 : (cls < 7 ? 1 : (cls < 9 ? 2 : 3));
    const int n1 = cls < 4 ? cls : (cls < 7 ? cls - 4 : (cls < 9 ? cls - 7 : 0));
    double w = 1.;
    for (int k = 0; k < 3 - n1 - n2; k++) w /= 36.;
    for (int k = 0; k < n1; k++) w /= 12.;
    for (int k = 0; k < n2; k++) w /= 45.;
    return w;
}
// sum of the weighted terms f(k), grouped by weight
template <class F>
__device__ __forceinline__ double legendre_sum(F &&f) {
    double acc[10];
#pragma unroll
    for (int i = 0; i < 10; i++) acc[i] = 0.;
#pragma unroll
    for (int k = 0; k < 27; k++) f(k, acc[legendre_class(k)]);
    double s = 0.;
#pragma unroll
    for (int i = 9; i >= 0; i--) s = __fma_rn(legendre_weight(i), acc[i], s);
    return s;
}

// r -> (M x M x M) r with M = [4 2 -1; 2 16 2; -1 2 4] (30 x the 1D mass matrix), per axis and in place
__device__ __forceinline__ void mass27(double (&c)[27]) {
#pragma unroll
    for (int axis = 0; axis < 3; axis++) {
        const int st = axis == 0 ? 1 : (axis == 1 ? 3 : 9);
#pragma unroll
        for (int l = 0; l < 9; l++) {
            const int o = axis == 0 ? 3 * l : (axis == 1 ? (l / 3) * 9 + l % 3 : l);
            const double a = c[o], b = c[o + st], d = c[o + 2 * st], b2 = __dadd_rn(b, b);
            c[o] = __dadd_rn(__fma_rn(4., a, -d), b2);
            c[o + st] = __fma_rn(8., b2, __dmul_rn(2., __dadd_rn(a, d)));
            c[o + 2 * st] = __dadd_rn(__fma_rn(4., d, -a), b2);
        }
    }
}

// ------------------------------------------------------------------------------------------- curl penalty
// A bilinear function's values (a0, a1, a2, a3) at (0,0), (1,0), (0,1), (1,1) -> (4 mean, 2 slope in the first, 2
// slope in the second coordinate, cross difference); the integral square is S^2/16 + (D1^2 + D2^2)/48 + D12^2/144.
struct Bilinear {
    double S, D1, D2, D12;
};
__device__ __forceinline__ Bilinear hadamard(double a0, double a1, double a2, double a3) {
    const double p = __dadd_rn(a0, a1), m = __dsub_rn(a1, a0), P = __dadd_rn(a2, a3), M = __dsub_rn(a3, a2);
    return {__dadd_rn(p, P), __dadd_rn(m, M), __dsub_rn(P, p), __dsub_rn(M, m)};
}
// its adjoint: d/d a_e of S gS + D1 g1 + D2 g2 + D12 g12
__device__ __forceinline__ void hadamard_adjoint(const Bilinear &g, double (&a)[4]) {
    const double p = g.S - g.D2, P = g.S + g.D2, m = g.D1 - g.D12, M = g.D1 + g.D12;
    a[0] = p - m; a[1] = p + m; a[2] = P - M; a[3] = P + M;
}

// The 18 coefficients of curl u over the cell: c[0..2] the means (x4), c[3..11] the slopes (x2), c[12..17] the cross
// differences.  C0 = dy uz - dz uy etc.; each component is a difference of two bilinear functions that share one
// coordinate (x, y, z in turn), so the mean and that slope subtract and the other coefficients stand alone.
__device__ __forceinline__ void curl_coefficients(const Columns &C, double (&c)[18]) {
    const Bilinear A0 = hadamard(C.Y[0][2], C.Y[1][2], C.Y[2][2], C.Y[3][2]);    // dy uz (x, z)
    const Bilinear B0 = hadamard(C.Z[0][1], C.Z[1][1], C.Z[2][1], C.Z[3][1]);    // dz uy (x, y)
    const Bilinear A1 = hadamard(C.Z[0][0], C.Z[1][0], C.Z[2][0], C.Z[3][0]);    // dz ux (x, y)
    const Bilinear B1 = hadamard(C.X[0][2], C.X[1][2], C.X[2][2], C.X[3][2]);    // dx uz (y, z)
    const Bilinear A2 = hadamard(C.X[0][1], C.X[1][1], C.X[2][1], C.X[3][1]);    // dx uy (y, z)
    const Bilinear B2 = hadamard(C.Y[0][0], C.Y[1][0], C.Y[2][0], C.Y[3][0]);    // dy ux (x, z)
    c[0] = __dsub_rn(A0.S, B0.S); c[1] = __dsub_rn(A1.S, B1.S); c[2] = __dsub_rn(A2.S, B2.S);
    c[3] = __dsub_rn(A0.D1, B0.D1); c[4] = __dsub_rn(A1.D2, B1.D1); c[5] = __dsub_rn(A2.D2, B2.D2);
    c[6] = A0.D2; c[7] = B0.D2; c[8] = A1.D1; c[9] = B1.D2; c[10] = A2.D1; c[11] = B2.D1;
    c[12] = A0.D12; c[13] = B0.D12; c[14] = A1.D12; c[15] = B1.D12; c[16] = A2.D12; c[17] = B2.D12;
}
// The same of a - b, from the fields' vertices.  The curl is linear, and the difference of two close states is small and
// formed almost without rounding, so its coefficients round relative to themselves, where the difference of the two
// fields' coefficients carries the rounding of both.
__device__ __forceinline__ void curl_difference(const double (&a)[8][3], const double (&b)[8][3], const Q1Const &q,
                                                double (&c)[18]) {
    double d[8][3];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int r = 0; r < 3; r++) d[i][r] = __dsub_rn(a[i][r], b[i][r]);
    Columns D;
    vertex_columns(d, q, D);
    curl_coefficients(D, c);
}
__device__ constexpr double curl_weight(int k) { return k < 3 ? 1. / 16 : (k < 12 ? 1. / 48 : 1. / 144); }
template <class F>
__device__ __forceinline__ double curl_sum(F &&f) {
    double s[3] = {0., 0., 0.};
#pragma unroll
    for (int k = 0; k < 18; k++) f(k, s[k < 3 ? 0 : (k < 12 ? 1 : 2)]);
    return __fma_rn(curl_weight(0), s[0], __fma_rn(curl_weight(3), s[1], __dmul_rn(curl_weight(12), s[2])));
}
// Adds scale x the curl energy's derivative by the edge columns to G, for residual coefficients c (u minus
// reference); scale = nu omega.
__device__ __forceinline__ void curl_adjoint(const double (&c)[18], double scale, Columns &G) {
    const double wS = scale * curl_weight(0), wD = scale * curl_weight(3), wX = scale * curl_weight(12);
    double a[4];
    const double s0 = wS * c[0], s1 = wS * c[1], s2 = wS * c[2], d0 = wD * c[3], d1 = wD * c[4], d2 = wD * c[5];
    hadamard_adjoint({s0, d0, wD * c[6], wX * c[12]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.Y[e][2] += a[e];
    hadamard_adjoint({-s0, -d0, wD * c[7], wX * c[13]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.Z[e][1] += a[e];
    hadamard_adjoint({s1, wD * c[8], d1, wX * c[14]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.Z[e][0] += a[e];
    hadamard_adjoint({-s1, -d1, wD * c[9], wX * c[15]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.X[e][2] += a[e];
    hadamard_adjoint({s2, wD * c[10], d2, wX * c[16]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.X[e][1] += a[e];
    hadamard_adjoint({-s2, wD * c[11], -d2, wX * c[17]}, a);
#pragma unroll
    for (int e = 0; e < 4; e++) G.Y[e][0] += a[e];
}

// ------------------------------------------------------------------------------------------- adjoint of J
// acc + g (a x b), component-wise fused
__device__ __forceinline__ void cross_add(const double (&a)[3], const double (&b)[3], double (&s)[3]) {
    s[0] = fma(a[1], b[2], fma(-a[2], b[1], s[0]));
    s[1] = fma(a[2], b[0], fma(-a[0], b[2], s[1]));
    s[2] = fma(a[0], b[1], fma(-a[1], b[0], s[2]));
}
// Adjoint of column_plane: adds plane values S[s] at plane t to the edge values.
__device__ __forceinline__ void column_plane_adjoint(const double (&S)[3][3], int t, double (&E)[4][3]) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
        const double a = fma(.5, S[1][r], S[0][r]), b = fma(.5, S[1][r], S[2][r]);
        if (t == 1) {
            E[0][r] = fma(.5, a, E[0][r]);
            E[2][r] = fma(.5, a, E[2][r]);
            E[1][r] = fma(.5, b, E[1][r]);
            E[3][r] = fma(.5, b, E[3][r]);
        } else {
            E[t][r] += a;
            E[t + 1][r] += b;
        }
    }
}
// G = sum_p g(p) dJ_p / d(edge columns) for columns C of F: dJ/dX = Y x Z, dJ/dY = Z x X, dJ/dZ = X x Y at each
// closed27 point.
template <class Weight>
__device__ __forceinline__ void closed_adjoint(const Columns &C, Columns &G, Weight &&g) {
#pragma unroll
    for (int e = 0; e < 4; e++)
#pragma unroll
        for (int r = 0; r < 3; r++) G.X[e][r] = G.Y[e][r] = G.Z[e][r] = 0.;
    double SZ[3][3][3];    // [iy][ix][r]
#pragma unroll
    for (int k = 0; k < 9; k++)
#pragma unroll
        for (int r = 0; r < 3; r++) SZ[k / 3][k % 3][r] = 0.;
#pragma unroll
    for (int iz = 0; iz < 3; iz++) {
        double X[3][3], Y[3][3], SX[3][3], SY[3][3];
        column_plane(C.X, iz, X);
        column_plane(C.Y, iz, Y);
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int r = 0; r < 3; r++) SX[k][r] = SY[k][r] = 0.;
#pragma unroll
        for (int iy = 0; iy < 3; iy++) {
            double Z[3][3];
            column_plane(C.Z, iy, Z);
#pragma unroll
            for (int ix = 0; ix < 3; ix++) {
                const double w = g(9 * iz + 3 * iy + ix);
                const double wY[3] = {w * Y[ix][0], w * Y[ix][1], w * Y[ix][2]};
                const double wX[3] = {w * X[iy][0], w * X[iy][1], w * X[iy][2]};
                cross_add(wY, Z[ix], SX[iy]);
                cross_add(Z[ix], wX, SY[ix]);
                cross_add(X[iy], wY, SZ[iy][ix]);
            }
        }
        column_plane_adjoint(SX, iz, G.X);
        column_plane_adjoint(SY, iz, G.Y);
    }
#pragma unroll
    for (int iy = 0; iy < 3; iy++) column_plane_adjoint(SZ[iy], iy, G.Z);
}
// Edge values -> vertex values: the adjoint of load_columns.
__device__ __forceinline__ void columns_to_vertices(const Columns &G, const Q1Const &q, double (&L)[8][3]) {
#pragma unroll
    for (int a = 0; a < 8; a++)
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const int x = a & 1, y = (a >> 1) & 1, z = a >> 2;
            const double gx = q.ih[0] * G.X[y + 2 * z][r], gy = q.ih[1] * G.Y[x + 2 * z][r],
                         gz = q.ih[2] * G.Z[x + 2 * y][r];
            L[a][r] = ((x ? gx : -gx) + (y ? gy : -gy)) + (z ? gz : -gz);
        }
}

}  // namespace svp
