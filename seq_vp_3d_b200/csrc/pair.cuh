// Internal definition of a registration pair: the device constants of one (grid, images, weights, reference).
#pragma once
#include "q1_common.cuh"

struct svp_pair {
    svp_grid grid;
    svp_weights w;
    svp::Q1Const q;
    int device = 0;
    // one allocation for everything whose size the grid fixes (the arrays below except loc1, loc2, cand): a
    // registration allocates and frees 5 blocks instead of 30
    char *slab = nullptr;
    // images and spline
    double *fixed = nullptr;      // (nz, ny, nx)
    double *coeff = nullptr;      // (nz, ny, nx) not-a-knot cubic coefficients
    double *knots[3] = {nullptr, nullptr, nullptr};  // x, y, z knot vectors (n + 4)
    double *spline_rcp[3] = {nullptr, nullptr, nullptr};  // per span, 6 reciprocal knot differences (n x 6)
    double *u_ref = nullptr;      // (nz, ny, nx, 3) frozen reference displacement
    // workspace
    double *loc1 = nullptr, *loc2 = nullptr;  // (24, ncell) per-cell vertex values (SoA)
    double *cellbuf = nullptr;                // (ncell)
    svp::dd *partial = nullptr;               // block partial sums
    double *host = nullptr;                   // pinned results that kernels write (64 doubles)
    long long *counter = nullptr;             // small device counters (8)
    long long *cand = nullptr;                // candidate cells of the T69/T73 node JD extension (ncell)
    uint8_t *flags = nullptr;                 // (ncell) cells the soft cell kernels hand to the barrier kernels
    // DST-I Poisson metric
    // folded orthonormal DST-I half matrices, x, y, z, zero-padded and in the mma's fragment order (DstFrag)
    double *dst_f64[3] = {nullptr, nullptr, nullptr};
    int dst_n[3] = {0, 0, 0};                               // their transform lengths (free nodes per axis)
    // the same rounded to float32 for the mixed form, as TF32 parts (big cells, small cells)
    unsigned *dst_tf32[3] = {nullptr, nullptr, nullptr};
    int precision = 0;                                      // SVP_PRECISION_PLAIN or SVP_PRECISION_MIXED
    double *dst_tmp = nullptr;                          // 2 * 3 * nfree scratch
    double *den = nullptr;                              // (nz-2, ny-2, nx-2) omega (a + b lambda)
    double den_a = -1, den_b = -1;
    int den_metric = -1;
};

namespace svp {
int pair_locals(svp_pair *p, int n);
// block sums (double-double) of the largest evaluation of a grid
long long pair_partial_count(const Q1Const &q);
// consecutive 256-byte aligned pieces of the slab; with a null base only the size is counted
struct SlabCursor {
    char *base;
    size_t used = 0;
    template <class T>
    void take(T *&ptr, size_t count) {
        if (base) ptr = reinterpret_cast<T *>(base + used);
        used += (sizeof(T) * count + 255) / 256 * 256;
    }
};
void pair_dst_carve(svp_pair *p, SlabCursor &c);
int pair_dst_setup(svp_pair *p, cudaStream_t s);
}  // namespace svp
