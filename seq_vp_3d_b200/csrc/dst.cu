// Dense per-axis transforms of (batch, nz, ny, nx) float64 fields: the orthonormal DST-I of the Q1 Poisson metric
// (jd_curl/three_d/poisson.py:99, scipy dstn type=1 norm='ortho') and the not-a-knot spline prefilter
// (interpolation.py:29).  Each axis pass is a batched GEMM with a small square matrix.
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "pair.cuh"

namespace svp {
namespace {

constexpr int TM = 64, TN = 64, TK = 16;  // output tile 64 x 64, K step 16, 256 threads x (4 x 4) outputs

// C[b][i][w] = sum_j M[i][j] X[b][j][w]  (M: n x n row-major; X rows of length W with stride ldx, batch stride bs)
__global__ void __launch_bounds__(256) gemm_left_kernel(const double *__restrict__ M, int n,
                                                        const double *__restrict__ X, long long W, long long ldx,
                                                        long long bs, double *__restrict__ C) {
    __shared__ double sM[TK][TM + 1];
    __shared__ double sX[TK][TN];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const long long b = blockIdx.z;
    const int i0 = blockIdx.y * TM;
    const long long w0 = (long long)blockIdx.x * TN;
    const double *Xb = X + b * bs;
    double *Cb = C + b * bs;
    double acc[4][4] = {};
    for (int k0 = 0; k0 < n; k0 += TK) {
        for (int e = threadIdx.x; e < TK * TM; e += 256) {
            int kk = e % TK, ii = e / TK;
            int i = i0 + ii, k = k0 + kk;
            sM[kk][ii] = (i < n && k < n) ? M[(long long)i * n + k] : 0.;
        }
        for (int e = threadIdx.x; e < TK * TN; e += 256) {
            int ww = e % TN, kk = e / TN;
            long long w = w0 + ww;
            int k = k0 + kk;
            sX[kk][ww] = (k < n && w < W) ? Xb[(long long)k * ldx + w] : 0.;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            double a[4], x[4];
#pragma unroll
            for (int r = 0; r < 4; r++) a[r] = sM[kk][ty + 16 * r];
#pragma unroll
            for (int c = 0; c < 4; c++) x[c] = sX[kk][tx + 16 * c];
#pragma unroll
            for (int r = 0; r < 4; r++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[r][c] = fma(a[r], x[c], acc[r][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < 4; r++) {
        int i = i0 + ty + 16 * r;
        if (i >= n) continue;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            long long w = w0 + tx + 16 * c;
            if (w < W) Cb[(long long)i * ldx + w] = acc[r][c];
        }
    }
}

// C[r][i] = sum_j X[r][j] M[i][j]  (rows of length n, contiguous; R rows)
__global__ void __launch_bounds__(256) gemm_right_kernel(const double *__restrict__ M, int n,
                                                         const double *__restrict__ X, long long R,
                                                         double *__restrict__ C) {
    __shared__ double sX[TK][TM + 1];
    __shared__ double sM[TK][TN + 1];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const long long r0 = (long long)blockIdx.x * TM;
    const int i0 = blockIdx.y * TN;
    double acc[4][4] = {};
    for (int k0 = 0; k0 < n; k0 += TK) {
        for (int e = threadIdx.x; e < TK * TM; e += 256) {
            int kk = e % TK, rr = e / TK;
            long long r = r0 + rr;
            int k = k0 + kk;
            sX[kk][rr] = (r < R && k < n) ? X[r * n + k] : 0.;
        }
        for (int e = threadIdx.x; e < TK * TN; e += 256) {
            int kk = e % TK, ii = e / TK;
            int i = i0 + ii, k = k0 + kk;
            sM[kk][ii] = (i < n && k < n) ? M[(long long)i * n + k] : 0.;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            double a[4], m[4];
#pragma unroll
            for (int q = 0; q < 4; q++) a[q] = sX[kk][ty + 16 * q];
#pragma unroll
            for (int c = 0; c < 4; c++) m[c] = sM[kk][tx + 16 * c];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[q][c] = fma(a[q], m[c], acc[q][c]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        long long r = r0 + ty + 16 * q;
        if (r >= R) continue;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            int i = i0 + tx + 16 * c;
            if (i < n) C[r * n + i] = acc[q][c];
        }
    }
}

// ------------------------------------------------------------------------------------------- DST-I passes
// The orthonormal DST-I matrix is centro-symmetric along columns: S[i][n-1-k] = (-1)^i S[i][k] (0-indexed).  So
// output rows of one parity need only half the columns, against the folded input u_k = x_k + x_(n-1-k) (even i;
// u_mid = x_mid when n is odd) or v_k = x_k - x_(n-1-k) (odd i): half the FLOPs of the dense product.  The folded
// half matrices are stored per parity, H0 (ceil(n/2) x ceil(n/2)) then H1 (floor(n/2) x floor(n/2)), row-major.
//
// One kernel does a pass along any axis, D = H F with H a half matrix (m16 row tiles) and F the folded field, [k][col].
// A block takes QC columns and up to 8 row tiles of BOTH parities: the raw pair (x_k, x_(n-1-k)) is loaded once, and
// its sum and its difference are staged side by side for the warps of parity 0 and 1.  The half matrices are laid out
// once per grid in the order in which the lanes of an mma read them, so a warp loads its fragments of H with two
// 16-byte loads per tile and 8 k through L1, and only the field goes through shared memory.  The columns of all
// batches are one flattened range: a short x axis leaves no part-filled tile per (batch, z).  The result returns
// through shared memory, so that both parities of a line and QC columns (x pass: whole rows) are stored together and
// the epilogue's operands are read along lines.  Every output is accumulated in k order, so the values do not depend
// on the tiling.
//
// Bound by the FP64 tensor pipe (float64: half busy, the rest is the latency of the field's loads and the phases
// around the products) and by instruction issue (3xTF32).  Blocks of 4 warps, 4 per SM, cover each other's phases
// better than 2 of 8 warps (1278 against 1350 us for the six float64 passes on 224 x 192 x 160, 367 against 377 us for
// the six mixed ones on 119 x 165 x 141).  Against 128 x 64 (x: 64 or 128 x 16 ceil(k0 / 16)) tiles per parity with
// both operands staged through shared memory: six passes 1584 -> 1205 us float64, 672 -> 344 us mixed; the operations
// of the float64 passes (11.4 G fused multiply-adds) take 614 us at 18.6 T/s, the right-hand side, scale and result of
// the mixed ones 29 us.
//
// Float64: mma.sync m16n8k8 f64 (FP64 has no tcgen05 kind on sm_100a; this is B200's FP64 tensor path).  Mixed form:
// float32 operands as 3xTF32 (mma.sync m16n8k8 .tf32, float32 accumulate): each operand x splits into big = tf32(x)
// and small = tf32(x - big); the product sums small*big + big*small + big*big, which keeps float32-level accuracy (the
// small*small term is below float32 rounding).  Fragments of m16n8k8, both types (lane: gid = lane / 4, tig = lane %
// 4): a0 = A[gid][tig], a1 = A[gid + 8][tig], a2 = A[gid][tig + 4], a3 = A[gid + 8][tig + 4]; b0 = B[tig][gid],
// b1 = B[tig + 4][gid]; d0, d1 = D[gid][2 tig + {0, 1}], d2, d3 = D[gid + 8][2 tig + {0, 1}].
__device__ __forceinline__ unsigned tf32_of(float x) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void tf32_split(float x, unsigned &big, unsigned &small) {
    big = tf32_of(x);
    small = tf32_of(x - __uint_as_float(big));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint4 &a, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f64(double (&d)[4], const double2 &a01, const double2 &a23, const double2 &b) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
                 : "d"(a01.x), "d"(a01.y), "d"(a23.x), "d"(a23.y), "d"(b.x), "d"(b.y));
}

// A 16-byte cell holds what one lane needs of an operand for a pair (k, k + 4): both values (float64), or the big and
// small part of each (3xTF32).  H: per parity, tile and 8 k, two cells per lane (float64: a0 a1, a2 a3; 3xTF32: the
// four big parts, the four small parts); F: one cell per (k % 4, column).
constexpr int QK = 16;                                             // K block: two mma steps
constexpr int DT = 128;                                            // threads: parity x two row warps
constexpr int kLines = 8;                                          // lines of the epilogue in flight per thread
template <class TC> constexpr int kNC = sizeof(TC) == 8 ? 2 : 4;   // n8 tiles per warp
template <class TC> constexpr int kQC = 8 * kNC<TC>;               // columns per block

struct DstFrag {
    const uint4 *h[2];       // per parity
    int n, kg[2];            // axis length, rows per parity
    int k8, mt, tiles;       // mma steps along K, m16 tiles per block (<= 8) and blocks along the rows
};
// The rows of parity 0 are split evenly: 16 ceil(k0 / 16) rows leave at most 15 + 16 (tiles - 1) rows of padding.
inline DstFrag frag_geometry(int n) {
    DstFrag F;
    F.h[0] = F.h[1] = nullptr;
    F.n = n;
    F.kg[0] = (n + 1) / 2;
    F.kg[1] = n / 2;
    F.k8 = (F.kg[0] + 7) / 8;
    const int m16 = (F.kg[0] + 15) / 16;
    F.tiles = (m16 + 7) / 8;
    F.mt = (m16 + F.tiles - 1) / F.tiles;
    return F;
}
inline size_t frag_cells(const DstFrag &F) { return (size_t)F.tiles * F.mt * F.k8 * 64; }   // per parity
inline DstFrag frag_of(const void *t, int n) {
    DstFrag F = frag_geometry(n);
    F.h[0] = reinterpret_cast<const uint4 *>(t);
    F.h[1] = F.h[0] + frag_cells(F);
    return F;
}

// h: H0 (k0 x k0) then H1 (k1 x k1), row-major; out: the cells of parity g (src = offset of H_g), zeros outside H_g
template <class TC>
__global__ void frag_kernel(const TC *__restrict__ h, int kg, long long src, long long cells, int k8,
                            uint4 *__restrict__ out) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < cells;
         e += (long long)gridDim.x * blockDim.x) {
        const int lane = (int)(e & 31), half = (int)(e >> 5) & 1, gid = lane >> 2, tig = lane & 3;
        const int step = (int)((e >> 6) % k8), tile = (int)((e >> 6) / k8);
        TC a[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = 16 * tile + gid + 8 * (j & 1), k = 8 * step + tig + 4 * (j >> 1);
            a[j] = (i < kg && k < kg) ? h[src + (long long)i * kg + k] : TC(0);
        }
        if constexpr (sizeof(TC) == 8) {
            reinterpret_cast<double2 *>(out)[e] = half ? make_double2(a[2], a[3]) : make_double2(a[0], a[1]);
        } else {
            unsigned big[4], small[4];
#pragma unroll
            for (int j = 0; j < 4; j++) tf32_split(a[j], big[j], small[j]);
            out[e] = half ? make_uint4(small[0], small[1], small[2], small[3])
                          : make_uint4(big[0], big[1], big[2], big[3]);
        }
    }
}

// Half a cell of a folded value; formed in the input type and rounded once to the pass's type.
template <class TC, class TI>
__device__ __forceinline__ uint2 fold_half(TI v) {
    uint2 h;
    if constexpr (sizeof(TC) == 8) {
        const double d = (double)v;
        h = *reinterpret_cast<const uint2 *>(&d);
    } else {
        tf32_split((float)v, h.x, h.y);
    }
    return h;
}

// Row strides of the returned tile: [line][column] (left passes; a lane writes two columns at once) and
// [row][position] (x pass).
template <class TC> constexpr int kTileCol = kQC<TC> + 4;
inline constexpr __host__ __device__ int tile_row(int mt) { return 32 * mt + 1; }
template <class TC> constexpr int kStep = 4 * (kQC<TC> + 2) + 1;   // cells of one staged mma step, see dst_pass_kernel
template <class TC>
constexpr size_t dst_smem(bool x, int mt) {
    const size_t stage = sizeof(uint4) * 2 * 2 * 2 * kStep<TC>;
    const size_t tile = sizeof(TC) * (x ? (size_t)kQC<TC> * tile_row(mt) : (size_t)32 * mt * kTileCol<TC>);
    return stage > tile ? stage : tile;
}

// address of flattened column col at k = 0 (ncol < 2^32)
__device__ __forceinline__ long long flat_base(long long col, int W, long long bs) {
    const unsigned b = (unsigned)col / (unsigned)W;
    return (long long)b * bs + ((unsigned)col - b * (unsigned)W);
}
__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

// XP (x pass): columns are the R rows of length n, C[r][2i + g] = sum_k fold_g(pre X)[r][k] H_g[i][k], pre an optional
// scale applied first.  Else (y, z): C[b][2i + g][w] = sum_k H_g[i][k] fold_g(X)[b][k][w], rows of length W, stride
// ldx = W, batch stride bs, ncol = batches * W; EPI 1 divides by den[index within the batch] (den is one component's
// array: the z pass's batch stride is its length), EPI 2 multiplies by sign * post[flat].
// MW: m16 tiles per warp, two row warps per parity (the second one has mt - MW).
template <bool XP, bool PRE, int MW, int EPI, class TC, class TI, class TO>
__global__ void __launch_bounds__(DT, 512 / DT) dst_pass_kernel(DstFrag D, const TI *__restrict__ X, long long ncol,
                                                                int W, long long bs, TO *__restrict__ C,
                                                                const double *__restrict__ pre,
                                                                const double *__restrict__ den,
                                                                const double *__restrict__ post, double sign) {
    constexpr bool F64 = sizeof(TC) == 8;
    constexpr int NC = kNC<TC>, QC = kQC<TC>, PC = QC + 2;
    constexpr int NE = QK * QC / DT;   // entries (k, column) of a K block a thread stages
    extern __shared__ __align__(16) unsigned char dsm[];
    // [buffer][parity][step], cell (k % 4, column) at PC (k % 4) + column: the 8 lanes of a 16-byte fragment load (4 k,
    // 2 columns) and the 16 lanes of an x pass's 8-byte store (16 k of a column) fall in distinct banks
    uint4(*sF)[2][2][kStep<TC>] = reinterpret_cast<uint4(*)[2][2][kStep<TC>]>(dsm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
    // both parities' second row warps would share schedulers if they had the same place: they swap
    const int g = warp >> 1, wm = (warp & 1) ^ g;
    const int tile = (int)(blockIdx.x % (unsigned)D.tiles);
    const long long c0 = (long long)(blockIdx.x / (unsigned)D.tiles) * QC;
    const int n = D.n, K = D.kg[0], k1 = D.kg[1], mine = wm ? D.mt - MW : MW;   // MW or MW - 1 tiles
    const bool full = mine == MW;
    const uint4 *H = (g ? D.h[1] : D.h[0]) + (long long)(tile * D.mt + wm * MW) * D.k8 * 64 + lane;
    TC acc[MW][NC][4];
#pragma unroll
    for (int m = 0; m < MW; m++)
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[m][c][e] = TC(0);
    // staging: of a K block's 16 k, y and z passes give a thread one column (lanes along the columns), the x pass one k
    // (16 lanes along a row)
    constexpr int KE = XP ? 0 : DT / QC, CE = XP ? DT / 16 : 0;      // entry e: k + KE e, column + CE e
    const int fk = XP ? (int)threadIdx.x & 15 : (int)threadIdx.x / QC;
    const int fc = XP ? (int)threadIdx.x >> 4 : (int)threadIdx.x % QC;
    const long long ks = XP ? 1 : W;
    const unsigned last = (unsigned)(n - 1) * (unsigned)W;
    const TI *fx = X + (XP ? (c0 + fc) * n : (c0 + fc < ncol ? flat_base(c0 + fc, W, bs) : 0));
    // Float64: the field of the block that will take this one's place (512 / DT per SM) is brought to L2, up to two
    // lines per k, or the rows of the x pass: 1278 -> 1241 us for the six passes above; the 3xTF32 passes, bound by
    // issue, lose by it (367 -> 371 us, 64.6 -> 65.6 ms for a solve on 224 x 192 x 160).
    if (F64) {
        const long long cn = c0 + 148LL * (512 / DT) * QC / D.tiles;
        if (cn + QC <= ncol) {
            if (XP) {
                for (int o = threadIdx.x * 16; o < QC * n; o += DT * 16) {   // 16 doubles to a line
                    prefetch_l2(X + cn * n + o);
                    if (PRE) prefetch_l2(pre + cn * n + o);
                }
            } else {
                const TI *q = X + flat_base(cn + (threadIdx.x & 1) * (QC / 2), W, bs);
                for (int k = threadIdx.x >> 1; k < n; k += DT / 2) prefetch_l2(q + (long long)k * W);
            }
        }
    }
    const double *fp = PRE ? pre + (c0 + fc) * n : nullptr;
    TI xa[NE], xb[NE];
    double pa[PRE ? NE : 1], pb[PRE ? NE : 1];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int k = k0 + fk + KE * e;
            const bool ok = c0 + fc + CE * e < ncol && k < K;
            const long long o = (long long)CE * e * n, a = o + k * ks, b = o + (n - 1 - k) * ks;
            if (XP || EPI) {
                xa[e] = ok ? fx[a] : TI(0);
                xb[e] = ok ? fx[b] : TI(0);
            } else {   // y pass: 32-bit offsets 177 -> 165 us float64, 111 -> 105 mixed; the z passes lose (58 -> 65 us)
                const unsigned at = (unsigned)k * (unsigned)W;
                xa[e] = ok ? fx[at] : TI(0);
                xb[e] = ok ? fx[last - at] : TI(0);
            }
            if (PRE) {
                pa[e] = ok ? fp[a] : 0.;
                pb[e] = ok ? fp[b] : 0.;
            }
        }
    };
    auto stash = [&](int buf, int k0) {
#pragma unroll
        for (int e = 0; e < NE; e++) {
            const int kl = fk + KE * e, k = k0 + kl;
            if (PRE) {
                xa[e] = (TI)(pa[e] * (double)xa[e]);
                xb[e] = (TI)(pb[e] * (double)xb[e]);
            }
            const TI u = k == n - 1 - k ? xa[e] : xa[e] + xb[e];   // the middle of an odd axis has no mirror
            const TI v = k < k1 ? xa[e] - xb[e] : TI(0);
            const int at = 2 * ((kl & 3) * PC + fc + CE * e) + ((kl >> 2) & 1);
            reinterpret_cast<uint2 *>(sF[buf][0][kl >> 3])[at] = fold_half<TC, TI>(u);
            reinterpret_cast<uint2 *>(sF[buf][1][kl >> 3])[at] = fold_half<TC, TI>(v);
        }
    };
    fetch(0);
    stash(0, 0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += QK) {
        const bool more = k0 + QK < K;
        if (more) fetch(k0 + QK);
#pragma unroll
        for (int st = 0; st < 2; st++) {
            const int step = k0 / 8 + st;
            if (step < D.k8) {
                uint4 f[NC];
#pragma unroll
                for (int c = 0; c < NC; c++) f[c] = sF[buf][g][st][tig * PC + 8 * c + gid];
#pragma unroll
                for (int m = 0; m < MW; m++) {
                    if (m < MW - 1 || full) {
                        const uint4 *hm = H + (m * D.k8 + step) * 64;
                        const uint4 h0 = __ldg(hm), h1 = __ldg(hm + 32);
#pragma unroll
                        for (int c = 0; c < NC; c++) {
                            if constexpr (F64) {
                                mma_f64(acc[m][c], *reinterpret_cast<const double2 *>(&h0),
                                        *reinterpret_cast<const double2 *>(&h1),
                                        *reinterpret_cast<const double2 *>(&f[c]));
                            } else if constexpr (XP) {   // field small x H big, field big x H small, big x big
                                mma_tf32(acc[m][c], h0, f[c].y, f[c].w);
                                mma_tf32(acc[m][c], h1, f[c].x, f[c].z);
                                mma_tf32(acc[m][c], h0, f[c].x, f[c].z);
                            } else {                     // H small x field big, H big x field small, big x big
                                mma_tf32(acc[m][c], h1, f[c].x, f[c].z);
                                mma_tf32(acc[m][c], h0, f[c].y, f[c].w);
                                mma_tf32(acc[m][c], h0, f[c].x, f[c].z);
                            }
                        }
                    }
                }
            }
        }
        if (more) stash(buf ^ 1, k0 + QK);
        __syncthreads();
        buf ^= 1;
    }
    // the tile returns through shared memory (the last barrier above also ends the reads of the staged field)
    TC *out = reinterpret_cast<TC *>(dsm);
    const int lines = 32 * D.mt, px = tile_row(D.mt);
#pragma unroll
    for (int m = 0; m < MW; m++) {
        if (m < mine) {
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int line = 2 * (16 * (wm * MW + m) + gid + 8 * (e >> 1)) + g;
                    const int cc = 8 * c + 2 * tig + (e & 1);
                    out[XP ? cc * px + line : line * kTileCol<TC> + cc] = acc[m][c][e];
                }
        }
    }
    __syncthreads();
    const int l0 = tile * lines, left = n - l0 < lines ? n - l0 : lines;
    if (XP) {
        for (int r = warp; r < QC && c0 + r < ncol; r += DT / 32) {
            TO *row = C + (c0 + r) * n + l0;
#pragma unroll 4
            for (int j = lane; j < left; j += 32) row[j] = (TO)out[r * px + j];
        }
    } else {
        constexpr int LC = QC < 32 ? QC : 32, LR = DT / LC;   // threads along a line, lines at a time
        const int l2 = (int)threadIdx.x / LC;
#pragma unroll
        for (int h = 0; h < QC / LC; h++) {
            const int cc = (int)threadIdx.x % LC + LC * h;
            const long long oc = c0 + cc;
            if (oc >= ncol) continue;
            const long long cb = (long long)((unsigned)oc / (unsigned)W) * bs;
            const int w = (int)((unsigned)oc % (unsigned)W);
            // the operands of kLines lines are loaded together, then used: a load and a divide per line in turn would
            // add up their latencies (float64 z passes of the solve above 392 -> 296 us)
            for (int l1 = l2; l1 < left; l1 += LR * kLines) {
                double op[kLines];
#pragma unroll
                for (int j = 0; j < kLines; j++) {
                    const int line = l1 + LR * j;
                    const long long io = (long long)(l0 + line) * W + w;
                    if (EPI) op[j] = line < left ? (EPI == 1 ? den[io] : post[cb + io]) : 1.;
                }
#pragma unroll
                for (int j = 0; j < kLines; j++) {
                    const int line = l1 + LR * j;
                    if (line >= left) break;
                    double v = (double)out[line * kTileCol<TC> + cc];
                    if (EPI == 1) v = v / op[j];
                    if (EPI == 2) v = sign * (op[j] * v);
                    C[cb + (long long)(l0 + line) * W + w] = (TO)v;
                }
            }
        }
    }
}

template <bool XP, bool PRE, int MW, int EPI, class TC, class TI, class TO>
int launch_dst(const DstFrag &F, const TI *in, long long ncol, int W, long long bs, TO *out, const double *pre,
               const double *den, const double *post, double sign, cudaStream_t s) {
    static_assert(dst_smem<TC>(XP, 2 * MW) <= 48 * 1024, "a pass needs no more than the default shared memory");
    const long long blocks = div_up(ncol, kQC<TC>) * F.tiles;
    SVP_REQUIRE(blocks <= 0x7fffffffLL && ncol <= 0xffffffffLL, "dst pass: grid too large");
    SVP_LAUNCH((dst_pass_kernel<XP, PRE, MW, EPI, TC, TI, TO><<<(unsigned)blocks, DT, dst_smem<TC>(XP, F.mt), s>>>(
        F, in, ncol, W, bs, out, pre, den, post, sign)));
    return SVP_OK;
}
template <bool XP, bool PRE, int EPI, class TC, class TI, class TO>
int launch_dst_rows(const DstFrag &F, const TI *in, long long ncol, int W, long long bs, TO *out,
                    const double *pre, const double *den, const double *post, double sign, cudaStream_t s) {
    switch ((F.mt + 1) / 2) {
        case 1: return launch_dst<XP, PRE, 1, EPI, TC, TI, TO>(F, in, ncol, W, bs, out, pre, den, post, sign, s);
        case 2: return launch_dst<XP, PRE, 2, EPI, TC, TI, TO>(F, in, ncol, W, bs, out, pre, den, post, sign, s);
        case 3: return launch_dst<XP, PRE, 3, EPI, TC, TI, TO>(F, in, ncol, W, bs, out, pre, den, post, sign, s);
        default: return launch_dst<XP, PRE, 4, EPI, TC, TI, TO>(F, in, ncol, W, bs, out, pre, den, post, sign, s);
    }
}

__global__ void scale_kernel(const double *__restrict__ x, const double *__restrict__ s, double sign, long long n,
                             double *__restrict__ y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        y[i] = s ? sign * (s[i] * x[i]) : sign * x[i];
}

__global__ void den_kernel(double *__restrict__ den, long long f0, long long f1, long long f2,
                           const double *__restrict__ ex, const double *__restrict__ ey, const double *__restrict__ ez,
                           const double *__restrict__ mx, const double *__restrict__ my, const double *__restrict__ mz,
                           double omega, double a, double b, int metric) {
    long long n = f0 * f1 * f2;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        long long x = i % f0, y = (i / f0) % f1, z = i / (f0 * f1);
        double lam = metric == 1 ? (ex[x] + ey[y]) + ez[z]
                                 : ((ex[x] * my[y]) * mz[z] + (mx[x] * ey[y]) * mz[z]) + (mx[x] * my[y]) * ez[z];
        den[i] = omega * (a + b * lam);
    }
}

}  // namespace

// Apply the n x n matrix M along one axis of `batch` fields of dims (n2, n1, n0) (z, y, x); in and out distinct.
int apply_axis(const double *M, int axis, long long batch, long long n2, long long n1, long long n0,
               const double *in, double *out, cudaStream_t s) {
    if (axis == 0) {
        long long R = batch * n2 * n1;
        dim3 grid((unsigned)div_up(R, TM), (unsigned)div_up(n0, TN));
        { svp::KernelTimer _t("gemm_right_kernel", s); SVP_LAUNCH(gemm_right_kernel<<<grid, 256, 0, s>>>(M, (int)n0, in, R, out)); }
    } else if (axis == 1) {
        dim3 grid((unsigned)div_up(n0, TN), (unsigned)div_up(n1, TM), (unsigned)(batch * n2));
        { svp::KernelTimer _t("gemm_left_kernel", s); SVP_LAUNCH(gemm_left_kernel<<<grid, 256, 0, s>>>(M, (int)n1, in, n0, n0, n1 * n0, out)); }
    } else {
        dim3 grid((unsigned)div_up(n1 * n0, TN), (unsigned)div_up(n2, TM), (unsigned)batch);
        { svp::KernelTimer _t("gemm_left_kernel", s); SVP_LAUNCH(gemm_left_kernel<<<grid, 256, 0, s>>>(M, (int)n2, in, n1 * n0, n1 * n0, n2 * n1 * n0, out)); }
    }
    SVP_LAUNCH_CHECK("axis GEMM");
    return SVP_OK;
}

std::vector<double> dst1_matrix(int n);

// One DST-I pass along `axis` of (3, n2, n1, n0) fields with the folded half matrices; see dst_pass_kernel for pre,
// the epilogues and sign.
template <class TC, class TI, class TO>
static int dst_pass(const svp_pair *p, int axis, const TI *in, TO *out, const double *pre, int epi, double sign,
                    const double *post, cudaStream_t s) {
    const long long n0 = p->q.fx, n1 = p->q.fy, n2 = p->q.fz;
    const DstFrag F = frag_of(sizeof(TC) == 8 ? (const void *)p->dst_f64[axis] : (const void *)p->dst_tf32[axis],
                              p->dst_n[axis]);
    int rc;
    if (axis == 0) {
        SVP_REQUIRE(epi == 0, "dst_pass: x pass has no epilogue");
        const long long R = 3 * n2 * n1;
        svp::KernelTimer _t("dst_right_kernel", s);
        rc = SVP_OK;
        if constexpr (sizeof(TO) == sizeof(TC))   // the x pass returns its own type
            rc = pre ? launch_dst_rows<true, true, 0, TC, TI, TO>(F, in, R, 1, 0, out, pre, nullptr, nullptr, 1., s)
                     : launch_dst_rows<true, false, 0, TC, TI, TO>(F, in, R, 1, 0, out, pre, nullptr, nullptr, 1., s);
    } else {
        SVP_REQUIRE(!pre, "dst_pass: pre-scale only on the x pass");
        SVP_REQUIRE(epi != 1 || axis == 2, "dst_pass: the 1/den epilogue rides in the z pass (batch stride = nfree)");
        const long long W = axis == 1 ? n0 : n1 * n0, bs = axis == 1 ? n1 * n0 : n2 * n1 * n0;
        const long long ncol = (axis == 1 ? 3 * n2 : 3) * W;
        SVP_REQUIRE(p->q.nfree <= 0x7fffffffLL, "dst_pass: more than 2^31 - 1 free nodes");
        svp::KernelTimer _t("dst_left_kernel", s);
        rc = SVP_OK;
        if constexpr (sizeof(TI) == sizeof(TC)) {
            if (epi == 0)
                rc = launch_dst_rows<false, false, 0, TC, TI, TO>(F, in, ncol, (int)W, bs, out, nullptr,
                                                           nullptr, nullptr, 1., s);
            if constexpr (sizeof(TO) == sizeof(TC))
                if (epi == 1)
                    rc = launch_dst_rows<false, false, 1, TC, TI, TO>(F, in, ncol, (int)W, bs, out, nullptr,
                                                               p->den, nullptr, 1., s);
            if constexpr (sizeof(TO) == 8)
                if (epi == 2)
                    rc = launch_dst_rows<false, false, 2, TC, TI, TO>(F, in, ncol, (int)W, bs, out, nullptr,
                                                               nullptr, post, sign, s);
        }
    }
    if (rc) return rc;
    SVP_LAUNCH_CHECK("dst pass");
    return SVP_OK;
}

// Folded half matrices of the orthonormal DST-I (see dst_pass_kernel): H_g[a][k] = S[2a + g][k], k < ceil(n/2) (g = 0) or
// floor(n/2) (g = 1).
std::vector<double> dst1_half(int n) {
    std::vector<double> S = dst1_matrix(n);
    const int k0 = (n + 1) / 2, k1 = n / 2;
    std::vector<double> H((size_t)k0 * k0 + (size_t)k1 * k1);
    for (int a = 0; a < k0; a++)
        for (int k = 0; k < k0; k++) H[(size_t)a * k0 + k] = S[(size_t)(2 * a) * n + k];
    double *H1 = H.data() + (size_t)k0 * k0;
    for (int a = 0; a < k1; a++)
        for (int k = 0; k < k1; k++) H1[(size_t)a * k1 + k] = S[(size_t)(2 * a + 1) * n + k];
    return H;
}

// Orthonormal DST-I matrix S[j][k] = sqrt(2/(n+1)) sin(pi (j+1)(k+1)/(n+1)), evaluated in long double.
std::vector<double> dst1_matrix(int n) {
    std::vector<double> S((size_t)n * n);
    const long double pi = 3.141592653589793238462643383279502884L;
    const long double c = sqrtl(2.0L / (n + 1));
    for (int j = 0; j < n; j++)
        for (int k = 0; k < n; k++) {
            long long m = ((long long)(j + 1) * (k + 1)) % (2LL * (n + 1));
            S[(size_t)j * n + k] = (double)(c * sinl(pi * (long double)m / (long double)(n + 1)));
        }
    return S;
}

// The folded matrices depend only on n; registrations on one grid share them (n^2 long double sines per axis).
static std::vector<double> cached_dst1_half(int n) {
    static std::mutex mu;
    static std::map<int, std::vector<double>> cache;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(n);
        if (it != cache.end()) return it->second;
    }
    std::vector<double> H = dst1_half(n);
    std::lock_guard<std::mutex> lock(mu);
    if (cache.size() >= 32) cache.clear();
    cache.emplace(n, H);
    return H;
}

void pair_dst_carve(svp_pair *p, SlabCursor &c) {
    const long long f[3] = {p->q.fx, p->q.fy, p->q.fz};
    for (int k = 0; k < 3; k++) {
        const size_t cells = 2 * frag_cells(frag_geometry((int)f[k]));
        c.take(p->dst_f64[k], 2 * cells);
        c.take(p->dst_tf32[k], 4 * cells);
    }
    c.take(p->dst_tmp, (size_t)(2 * 3 * p->q.nfree));
    c.take(p->den, (size_t)p->q.nfree);
}

// Fills the fragment cells: the folded half matrices of the three axes, and their values rounded once to float32, go
// up in one copy each and are laid out (and split into TF32 parts with the cvt.rna of the passes) on the device.
int pair_dst_setup(svp_pair *p, cudaStream_t s) {
    const long long f[3] = {p->q.fx, p->q.fy, p->q.fz};
    std::vector<double> all;
    size_t off[3];
    for (int k = 0; k < 3; k++) {
        const std::vector<double> H = cached_dst1_half((int)f[k]);
        off[k] = all.size();
        all.insert(all.end(), H.begin(), H.end());
        p->dst_n[k] = (int)f[k];
    }
    const std::vector<float> all32(all.begin(), all.end());
    double *h = nullptr;
    SVP_CUDA(scratch_alloc((void **)&h, (sizeof(double) + sizeof(float)) * all.size(), s));
    float *h32 = reinterpret_cast<float *>(h + all.size());
    cudaError_t e = cudaMemcpyAsync(h, all.data(), sizeof(double) * all.size(), cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(h32, all32.data(), sizeof(float) * all32.size(), cudaMemcpyHostToDevice, s);
    for (int k = 0; k < 3 && e == cudaSuccess; k++) {
        const DstFrag D = frag_of(p->dst_f64[k], (int)f[k]), T = frag_of(p->dst_tf32[k], (int)f[k]);
        const long long cells = (long long)frag_cells(D);
        for (int g = 0; g < 2; g++) {
            const unsigned nb = blocks_for(cells, 256, 4);
            const long long src = (long long)off[k] + (g ? (long long)D.kg[0] * D.kg[0] : 0);
            frag_kernel<double><<<nb, 256, 0, s>>>(h, D.kg[g], src, cells, D.k8, const_cast<uint4 *>(D.h[g]));
            frag_kernel<float><<<nb, 256, 0, s>>>(h32, D.kg[g], src, cells, T.k8, const_cast<uint4 *>(T.h[g]));
        }
        e = cudaGetLastError();
    }
    const cudaError_t fe = scratch_free(h, s), se = cudaStreamSynchronize(s);   // the host copies must outlive theirs
    if (e != cudaSuccess) return cuda_fail(e, "DST matrices");
    if (fe != cudaSuccess) return cuda_fail(fe, "DST matrices free");
    if (se != cudaSuccess) return cuda_fail(se, "DST matrices");
    return SVP_OK;
}

// poisson.py:16 poisson_spectrum per axis: ell = (2 sin(theta/2)/h)^2, mass = (2 + cos theta)/3,
// theta = pi k/(n-1), k = 1..n-2 (host, double, the reference's expressions).
static int set_denominator(svp_pair *p, double a, double b, int metric, cudaStream_t s) {
    if (p->den_a == a && p->den_b == b && p->den_metric == metric) return SVP_OK;
    const long long nn[3] = {p->q.nx, p->q.ny, p->q.nz};
    std::vector<double> host;
    long long off[7] = {0};
    for (int k = 0; k < 3; k++) off[k + 1] = off[k] + (nn[k] - 2);
    for (int k = 0; k < 3; k++) off[k + 4] = off[k + 3] + (nn[k] - 2);
    host.resize((size_t)off[6]);
    const double pi = 3.141592653589793;
    for (int k = 0; k < 3; k++) {
        long long n = nn[k];
        for (long long i = 1; i < n - 1; i++) {
            double theta = pi * (double)i / (double)(n - 1);
            double e = 2 * sin(theta / 2) / p->q.h[k];
            host[off[k] + i - 1] = e * e;
            host[off[k + 3] + i - 1] = (2 + cos(theta)) / 3;
        }
    }
    double *dev = nullptr;
    SVP_CUDA(scratch_alloc((void **)&dev, sizeof(double) * host.size(), s));
    cudaError_t ce = cudaMemcpyAsync(dev, host.data(), sizeof(double) * host.size(), cudaMemcpyHostToDevice, s);
    if (ce == cudaSuccess)
        SVP_LAUNCH_KEEP(den_kernel<<<blocks_for(p->q.nfree, 256, 8), 256, 0, s>>>(
            p->den, p->q.fx, p->q.fy, p->q.fz, dev + off[0], dev + off[1], dev + off[2], dev + off[3], dev + off[4],
            dev + off[5], p->q.omega, a, b, metric));
    cudaError_t le = cudaGetLastError();
    cudaError_t fe = scratch_free(dev, s);
    if (ce != cudaSuccess) return cuda_fail(ce, "den copy");
    if (le != cudaSuccess) return cuda_fail(le, "den_kernel");
    if (fe != cudaSuccess) return cuda_fail(fe, "den free");
    p->den_a = a;
    p->den_b = b;
    p->den_metric = metric;
    return SVP_OK;
}

}  // namespace svp

using namespace svp;

extern "C" int svp_poisson_apply(svp_pair *p, double a, double b, int32_t metric, const double *scale,
                                 const double *rhs, double sign, double *out, void *stream) {
    SVP_REQUIRE(p && rhs && out, "svp_poisson_apply: null argument");
    SVP_REQUIRE(metric == 0 || metric == 1, "svp_poisson_apply: metric 0 (q1) or 1 (seven_point)");
    SVP_REQUIRE(std::isfinite(a) && a >= 0 && std::isfinite(b) && b > 0, "svp_poisson_apply: a >= 0, b > 0");
    cudaStream_t s = (cudaStream_t)stream;
    int rc = set_denominator(p, a, b, metric, s);
    if (rc) return rc;
    const long long n3 = 3 * p->q.nfree;
    if (p->precision == SVP_PRECISION_MIXED) {
        // the same six passes in float32 (the fold and the epilogues formed in float64, rounded once)
        float *f0 = (float *)p->dst_tmp, *f1 = f0 + n3;
        if ((rc = dst_pass<float>(p, 0, rhs, f0, scale, 0, 1., nullptr, s))) return rc;
        if ((rc = dst_pass<float>(p, 1, f0, f1, nullptr, 0, 1., nullptr, s))) return rc;
        if ((rc = dst_pass<float>(p, 2, f1, f0, nullptr, 1, 1., nullptr, s))) return rc;
        if ((rc = dst_pass<float>(p, 0, f0, f1, nullptr, 0, 1., nullptr, s))) return rc;
        if ((rc = dst_pass<float>(p, 1, f1, f0, nullptr, 0, 1., nullptr, s))) return rc;
        if (scale) return dst_pass<float>(p, 2, f0, out, nullptr, 2, sign, scale, s);
        if ((rc = dst_pass<float>(p, 2, f0, out, nullptr, 0, 1., nullptr, s))) return rc;
        SVP_LAUNCH(scale_kernel<<<blocks_for(n3, 256, 8), 256, 0, s>>>(out, nullptr, sign, n3, out));
        SVP_LAUNCH_CHECK("scale_kernel");
        return SVP_OK;
    }
    double *t0 = p->dst_tmp, *t1 = p->dst_tmp + n3;
    // scale -> DST(x, y, z) -> / den -> DST(x, y, z) -> sign * scale; the elementwise steps ride in the passes
    if ((rc = dst_pass<double>(p, 0, rhs, t0, scale, 0, 1., nullptr, s))) return rc;
    if ((rc = dst_pass<double>(p, 1, t0, t1, nullptr, 0, 1., nullptr, s))) return rc;
    if ((rc = dst_pass<double>(p, 2, t1, t0, nullptr, 1, 1., nullptr, s))) return rc;
    if ((rc = dst_pass<double>(p, 0, t0, t1, nullptr, 0, 1., nullptr, s))) return rc;
    if ((rc = dst_pass<double>(p, 1, t1, t0, nullptr, 0, 1., nullptr, s))) return rc;
    if (scale) return dst_pass<double>(p, 2, t0, out, nullptr, 2, sign, scale, s);
    if ((rc = dst_pass<double>(p, 2, t0, t1, nullptr, 0, 1., nullptr, s))) return rc;
    unsigned eb = blocks_for(n3, 256, 8);
    SVP_LAUNCH(scale_kernel<<<eb, 256, 0, s>>>(t1, nullptr, sign, n3, out));
    SVP_LAUNCH_CHECK("scale_kernel");
    return SVP_OK;
}
