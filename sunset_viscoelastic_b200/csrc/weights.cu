// weights.cu -- LABFM weight construction on the device (labf.F90, svdlib.F90, rbfs.F90).
//
// The weights of a node: its moment matrix
// A = sum_k X(r_k/h) [W(r_k/h) H(r_k/h)]^T (monomials X, Hermite ABFs H, Wendland C2 W),
// factored with the reference's Golub-Kahan-Reinsch SVD, and the factorisation applied to each
// right-hand side.  The SVD is the reference's algorithm with its serial recurrences kept
// serial: threads split only loops whose iterations are independent (columns of a Householder
// update, rows of a Givens rotation), and every dot product is summed by one thread in the
// reference's order.  With -fmad=false each operation then rounds exactly as the
// reference's does, so the factorisation - and the weights - are those of the CPU
// restatement bit for bit.  The weight build takes three kernels (below), the stencil
// adaptation a block a node, and the boundary operators factor on one warp (svd_factor_warp).
//
// The five SVDs of identical matrix copies in labf.F90:157-180 become one factorisation
// applied to five right-hand sides; the filter matrix (labf.F90:258-303) is the same
// matrix whenever h == h_small, the counts agree and the order drops agree, and is then
// not factored again.
#include <algorithm>
#include <cmath>

#include "internal.cuh"

namespace sunset {

namespace {

__host__ __device__ constexpr int nsz(int k) { return (k * k + 3 * k) / 2; }

// (p, q) exponents of unknown m in the reference's degree-graded ordering
// (labf.F90:1815-1920): degree d, p from d down to 0.
__host__ __device__ constexpr int deg_of(int m) {
    int d = 1, base = 0;
    while (m >= base + d + 1) { base += d + 1; d++; }
    return d;
}
__host__ __device__ constexpr int p_of(int m) {
    int d = 1, base = 0;
    while (m >= base + d + 1) { base += d + 1; d++; }
    return d - (m - base);
}
__host__ __device__ constexpr int q_of(int m) { return deg_of(m) - p_of(m); }

__device__ __forceinline__ double fact(int k) {
    double f = 1.0;
    for (int j = 2; j <= k; j++) f *= (double)j;
    return f;
}

// labf.F90:2329-2391 probabilists' Hermite polynomials, in the reference's operation order.
__device__ __forceinline__ double hermite(int n, double z) {
    double z2, z3, z4;
    switch (n) {
    case 0: return 1.0;
    case 1: return z;
    case 2: return z * z - 1.0;
    case 3: return (z * z) * z - 3.0 * z;
    case 4: return ((((z * z) * z) * z) - ((6.0 * z) * z)) + 3.0;
    case 5: z2 = z * z; z3 = z * z2; return ((z2 * z3) - (10.0 * z3)) + (15.0 * z);
    case 6: z2 = z * z; z3 = z * z2; return (((z3 * z3) - ((15.0 * z2) * z2)) + (45.0 * z2)) - 15.0;
    case 7:
        z2 = z * z; z3 = z * z2; z4 = z3 * z;
        return (((z4 * z3) - ((21.0 * z3) * z2)) + (105.0 * z3)) - (105.0 * z);
    case 8:
        z2 = z * z; z4 = z2 * z2;
        return ((((z4 * z4) - ((28.0 * z4) * z2)) + (210.0 * z4)) - (420.0 * z2)) + 105.0;
    case 9:
        z2 = z * z; z3 = z * z2; z4 = z3 * z;
        return (((((z4 * z3) * z2) - ((36.0 * z4) * z3)) + ((378.0 * z3) * z2)) - (1260.0 * z3)) + (945.0 * z);
    case 10:
        z2 = z * z; z4 = z2 * z2;
        return ((((((z4 * z4) * z2) - ((45.0 * z4) * z4)) + ((630.0 * z4) * z2)) - (3150.0 * z4)) + (4725.0 * z2)) - 945.0;
    }
    return 0.0;
}

// x^4 correctly rounded.  The reference evaluates (1-q/2)**4.0 with libm pow; glibc's pow
// returns the correctly rounded power for these arguments, which this reproduces with an
// exact double-double product (Dekker's two-product, built on fma) rounded once.
__device__ __forceinline__ double pow4_cr(double x) {
    double a = x * x;
    double ae = fma(x, x, -a);           // x*x = a + ae exactly
    double b = a * a;                     // (a + ae)^2 = a^2 + 2 a ae + ae^2
    double be = fma(a, a, -b);            // a*a = b + be exactly
    double t = fma(2.0 * a, ae, be);      // small terms
    t = fma(ae, ae, t);
    return b + t;
}

// rbfs.F90:48-57, Wendland C2 (zero at q=0 and q>2).
__device__ __forceinline__ double wab(double qq, double h2) {
    double qq4 = 1.0 - 0.5 * qq;
    qq4 = pow4_cr(qq4);
    double f = 0.0;
    if (qq <= 2.0 && qq > 0.0) f = ((7.0 / ((4.0 * kPi) * h2)) * (2.0 * qq + 1.0)) * qq4;
    return f;
}

__device__ __forceinline__ double nr_hypot(double a, double b) {  // svdlib.F90:308-327
    double absA = fabs(a), absB = fabs(b), t;
    if (absA > absB) {
        t = absB / absA;
        return absA * sqrt(1.0 + t * t);
    }
    if (absB == 0.0) return 0.0;
    t = absA / absB;
    return absB * sqrt(1.0 + t * t);
}

// Shared scalars are written by lane 0 between two warp barriers, so no lane reads a
// half-updated value and every lane sees the new one.
__device__ __forceinline__ void wstore(double *p, double v, int lane) {
    __syncwarp();
    if (lane == 0) *p = v;
    __syncwarp();
}

// svdlib.F90:37-278 on a warp.  U (in: A, out: U) and V are column-major n x n with
// leading dimension ld; W and rv1 are 1-based.  Returns 0 or -1 (no convergence within
// maxits QR sweeps per singular value; the reference's limit is 30).
template <int N>
__device__ int svd_factor_warp(double *U, double *V, double *W, double *rv1, int ld, int lane, int maxits = 30) {
    const int n = N;
#define UM(i, j) U[((j) - 1) * ld + ((i) - 1)]
#define VM(i, j) V[((j) - 1) * ld + ((i) - 1)]
    double anorm = 0.0, c, f, g = 0.0, h, s, scale = 0.0, x, y, z;
    int l = 1, nm;
    for (int i = 1; i <= n; i++) {
        l = i + 1;
        wstore(&rv1[i], scale * g, lane);
        g = 0.0; s = 0.0; scale = 0.0;
        for (int k = i; k <= n; k++) scale = scale + fabs(UM(k, i));
        if (scale != 0.0) {
            __syncwarp();
            for (int k = i + lane; k <= n; k += 32) UM(k, i) = UM(k, i) / scale;
            __syncwarp();
            for (int k = i; k <= n; k++) s = s + UM(k, i) * UM(k, i);
            f = UM(i, i);
            g = -copysign(sqrt(s), f);
            h = f * g - s;
            wstore(&UM(i, i), f - g, lane);
            for (int j = l + lane; j <= n; j += 32) {
                double sj = 0.0;
                for (int k = i; k <= n; k++) sj = sj + UM(k, i) * UM(k, j);
                double fj = sj / h;
                for (int k = i; k <= n; k++) UM(k, j) = UM(k, j) + fj * UM(k, i);
            }
            __syncwarp();
            for (int k = i + lane; k <= n; k += 32) UM(k, i) = scale * UM(k, i);
            __syncwarp();
        }
        wstore(&W[i], scale * g, lane);
        g = 0.0; s = 0.0; scale = 0.0;
        for (int k = l; k <= n; k++) scale = scale + fabs(UM(i, k));
        if (scale != 0.0) {
            __syncwarp();
            for (int k = l + lane; k <= n; k += 32) UM(i, k) = UM(i, k) / scale;
            __syncwarp();
            for (int k = l; k <= n; k++) s = s + UM(i, k) * UM(i, k);
            f = UM(i, l);
            g = -copysign(sqrt(s), f);
            h = f * g - s;
            wstore(&UM(i, l), f - g, lane);
            for (int k = l + lane; k <= n; k += 32) rv1[k] = UM(i, k) / h;
            __syncwarp();
            for (int j = l + lane; j <= n; j += 32) {
                double sj = 0.0;
                for (int k = l; k <= n; k++) sj = sj + UM(j, k) * UM(i, k);
                for (int k = l; k <= n; k++) UM(j, k) = UM(j, k) + sj * rv1[k];
            }
            __syncwarp();
            for (int k = l + lane; k <= n; k += 32) UM(i, k) = scale * UM(i, k);
            __syncwarp();
        }
        double t = fabs(W[i]) + fabs(rv1[i]);
        anorm = (t > anorm) ? t : anorm;
    }
    // right-hand transformations, svdlib.F90:115-141
    for (int i = n; i >= 1; i--) {
        if (i < n) {
            if (g != 0.0) {
                __syncwarp();
                for (int j = l + lane; j <= n; j += 32) VM(j, i) = (UM(i, j) / UM(i, l)) / g;
                __syncwarp();
                for (int j = l + lane; j <= n; j += 32) {
                    double sj = 0.0;
                    for (int k = l; k <= n; k++) sj = sj + UM(i, k) * VM(k, j);
                    for (int k = l; k <= n; k++) VM(k, j) = VM(k, j) + sj * VM(k, i);
                }
                __syncwarp();
            }
            for (int j = l + lane; j <= n; j += 32) { VM(i, j) = 0.0; VM(j, i) = 0.0; }
            __syncwarp();
        }
        wstore(&VM(i, i), 1.0, lane);
        g = rv1[i];
        l = i;
    }
    // left-hand transformations, svdlib.F90:143-171
    for (int i = n; i >= 1; i--) {
        l = i + 1;
        g = W[i];
        __syncwarp();
        for (int j = l + lane; j <= n; j += 32) UM(i, j) = 0.0;
        __syncwarp();
        if (g != 0.0) {
            g = 1.0 / g;
            for (int j = l + lane; j <= n; j += 32) {
                double sj = 0.0;
                for (int k = l; k <= n; k++) sj = sj + UM(k, i) * UM(k, j);
                double fj = (sj / UM(i, i)) * g;
                for (int k = i; k <= n; k++) UM(k, j) = UM(k, j) + fj * UM(k, i);
            }
            __syncwarp();
            for (int j = i + lane; j <= n; j += 32) UM(j, i) = UM(j, i) * g;
            __syncwarp();
        } else {
            for (int j = i + lane; j <= n; j += 32) UM(j, i) = 0.0;
            __syncwarp();
        }
        wstore(&UM(i, i), UM(i, i) + 1.0, lane);
    }
    // diagonalisation, svdlib.F90:173-278
    nm = 1;
    for (int k = n; k >= 1; k--) {
        for (int its = 1; its <= 30; its++) {
            bool to2000 = false;
            for (l = k; l >= 1; l--) {
                nm = l - 1;
                if ((fabs(rv1[l]) + anorm) == anorm) { to2000 = true; break; }
                if ((fabs(W[nm]) + anorm) == anorm) break;
            }
            if (!to2000) {
                c = 0.0; s = 1.0;
                for (int i = l; i <= k; i++) {
                    double r = rv1[i];
                    f = s * r;
                    wstore(&rv1[i], c * r, lane);
                    if ((fabs(f) + anorm) == anorm) break;
                    g = W[i];
                    h = nr_hypot(f, g);
                    wstore(&W[i], h, lane);
                    h = 1.0 / h;
                    c = (g * h);
                    s = -(f * h);
                    for (int j = 1 + lane; j <= n; j += 32) {
                        double yy = UM(j, nm), zz = UM(j, i);
                        UM(j, nm) = (yy * c) + (zz * s);
                        UM(j, i) = -(yy * s) + (zz * c);
                    }
                    __syncwarp();
                }
            }
            z = W[k];
            if (l == k) {
                if (z < 0.0) {
                    wstore(&W[k], -z, lane);
                    for (int j = 1 + lane; j <= n; j += 32) VM(j, k) = -VM(j, k);
                    __syncwarp();
                }
                break;
            }
            if (its >= maxits) return -1;
            x = W[l];
            nm = k - 1;
            y = W[nm];
            g = rv1[nm];
            h = rv1[k];
            f = ((y - z) * (y + z) + (g - h) * (g + h)) / ((2.0 * h) * y);
            g = nr_hypot(f, 1.0);
            f = ((x - z) * (x + z) + h * ((y / (f + copysign(g, f))) - h)) / x;
            c = 1.0; s = 1.0;
            for (int j = l; j <= nm; j++) {
                int i = j + 1;
                g = rv1[i];
                y = W[i];
                h = s * g;
                g = c * g;
                z = nr_hypot(f, h);
                wstore(&rv1[j], z, lane);
                c = f / z;
                s = h / z;
                f = (x * c) + (g * s);
                g = -(x * s) + (g * c);
                h = y * s;
                y = y * c;
                for (int jj = 1 + lane; jj <= n; jj += 32) {
                    double xv = VM(jj, j), zv = VM(jj, i);
                    VM(jj, j) = (xv * c) + (zv * s);
                    VM(jj, i) = -(xv * s) + (zv * c);
                }
                z = nr_hypot(f, h);
                wstore(&W[j], z, lane);
                if (z != 0.0) {
                    z = 1.0 / z;
                    c = f * z;
                    s = h * z;
                }
                f = (c * g) + (s * y);
                x = -(s * g) + (c * y);
                for (int jj = 1 + lane; jj <= n; jj += 32) {
                    double yv = UM(jj, j), zv = UM(jj, i);
                    UM(jj, j) = (yv * c) + (zv * s);
                    UM(jj, i) = -(yv * s) + (zv * c);
                }
                __syncwarp();
            }
            wstore(&rv1[l], 0.0, lane);
            wstore(&rv1[k], f, lane);
            wstore(&W[k], x, lane);
        }
    }
    __syncwarp();
    return 0;
#undef UM
#undef VM
}

// svdlib.F90:279-303: b <- V diag(1/w) U^T b (exactly-zero singular values skipped).
template <int N>
__device__ void svd_apply_warp(const double *U, const double *V, const double *W, double *tmp, double *b, int ld,
                               int lane) {
    __syncwarp();
    for (int j = 1 + lane; j <= N; j += 32) {
        double s = 0.0;
        if (W[j] != 0.0) {
            for (int i = 1; i <= N; i++) s = s + U[(j - 1) * ld + (i - 1)] * b[i - 1];
            s = s / W[j];
        }
        tmp[j] = s;
    }
    __syncwarp();
    for (int j = 1 + lane; j <= N; j += 32) {
        double s = 0.0;
        for (int jj = 1; jj <= N; jj++) s = s + V[(jj - 1) * ld + (j - 1)] * tmp[jj];
        b[j - 1] = s;
    }
    __syncwarp();
}

struct WArgs {
    int npfb, morder, forder;
    double h2;
    const double *px, *py, *h, *hs;
    const int *ntype, *cnt, *cnt_small, *lpt;
    const long long *slice_ptr;
    double *wx, *wy, *wl, *wh;
    int *err;
    int maxits;               // QR sweeps per singular value (<= 0: the reference's 30)
    double *cond_d, *cond_f;  // per node sigma_max / sigma_min of the two moment matrices, or null
};

// 2-norm condition number of a factored matrix, sigma_max / sigma_min over W[1..N]
// (infinite when a singular value is exactly zero).  The reference inverts every nonzero
// sigma however small (svdlib.F90:283-293); the library reports it instead of staying
// silent about a near-singular stencil.
template <int N>
__device__ __forceinline__ double svd_cond(const double *W) {
    double smax = 0.0, smin = INFINITY;
    for (int j = 1; j <= N; j++) {
        const double w = fabs(W[j]);
        smax = w > smax ? w : smax;
        smin = w < smin ? w : smin;
    }
    return smin > 0.0 ? smax / smin : INFINITY;
}

__device__ __forceinline__ long long sell_off(const long long *slice_ptr, int i, int k) {
    return sell_at(slice_ptr[i >> 5], k, i & 31);
}

// ---------------------------------------------------------------------------------------
// The weight build in three kernels over batches of nodes.
//
// One warp doing everything for a node (assembly, SVD, solves) spent nine tenths of its time
// in the QR iteration's scalar recurrence (two hypotenuses, three divisions and a reciprocal a
// rotation, each waiting for the one before) with the node's two matrices parked in shared
// memory, so that six warps a SM filled it: 1.94 s for 1,048,576 nodes at order 8, 26 % of
// the issue slots used.  That recurrence reads only the bidiagonal, never the matrices, so
// it is taken out of the middle:
//   k_moment_bidiag  a block a node: moment matrix (accumulators in registers, a column a
//                    thread), Householder bidiagonalisation and both accumulations;
//   k_bidiag_qr      a thread a node: the QR iteration on the bidiagonal, recording its
//                    rotations;
//   k_weights_apply  a warp a node: the rotations replayed on the rows that the solves read,
//                    the solves and the link weights.
// A rotation acts on each row of U and V by itself, and the right-hand sides are unit vectors
// (or the few entries of the hyperviscous operator), so of U only the four to ten rows that
// meet a nonzero entry are replayed.  Every sum, rotation and solve keeps its order and
// rounding, so the weights stay the reference's bit for bit.
//
// A node whose rotations do not fit its record stops before the sweep that would not fit, and
// the last two kernels run again until every node is done.
//
// 262,144 nodes at order 8: 83 + 7 + 18 ms in the three kernels; 1,048,576: 333 + 30 + 74 (one
// kernel before: 1929), and the call 1943 -> 446-450 ms.
// ---------------------------------------------------------------------------------------
constexpr int kUrows = 10;  // rows of U the solves read: 0, 1, 2, 4 and up to six of the filter's

// Entry c of the hyperviscous right-hand side (labf.F90:325-388): its row, with its value.
__host__ __device__ __forceinline__ int hyp_entry(int order, int c, double *v) {
    const int half = order <= 5 ? 2 : order <= 7 ? 3 : order <= 9 ? 4 : 5;
    if (c > half) return -1;
    double b = 1.0;  // the binomial coefficient of half over c
    for (int k = 1; k <= c; k++) b = b * (double)(half - k + 1) / (double)k;
    *v = (half & 1) ? b : -b;
    const int d = 2 * half;
    return (d * d + d) / 2 - 1 + 2 * c;  // unknowns of degree d start at d (d + 1) / 2 - 1
}

// Order of a node's hyperviscous operator (labf.F90:305-323): reduced next to walls.
__device__ __forceinline__ int filter_order(int forder, int t) {
    int o = forder;
    if (forder >= 7 && (t == 998 || t < 0)) o = 6;
    if (forder >= 5 && t == -1) o = 4;
    return o;
}

// What the three kernels share for one batch.  Arrays of [..][batch] are indexed by the item
// last, so that a thread an item reads them coalesced; a rotation is four doubles (cosine and
// sine on V, then on U) in the item's own record.
struct SvdBatch {
    int n_items, batch, cap;  // items; their capacity; rotations a record holds
    const int *item;          // the node of each item
    int pass;                 // 0: derivative matrix (and the filter where it is the same one), 1: filter
    double *W, *rv1;          // [n + 1][batch], 1-based
    double *anorm;            // [batch]
    int2 *state;              // singular value and sweep to go on from; {0, 0}: done, {-1, 0}: no convergence
    int *nrec;                // record entries of the last k_bidiag_qr; -1: done before it
    double *U, *V;            // [batch][kUrows][n] and [batch][n][n] (column by column)
    double4 *rec;             // [batch][cap]
    int *left;                // items not done yet
};

__host__ __device__ constexpr int bidiag_threads(int order) { return (nsz(order) + 31) / 32 * 32; }
constexpr int kAsmLinks = 16;  // links whose monomials are staged at once
// Doubles of shared memory of moment_bidiag: the matrix (while the moment matrix is assembled, its
// place holds the links' powers, Hermite polynomials and monomials), a staged row, and the
// bidiagonal.
template <int ORDER>
__host__ __device__ constexpr int bidiag_matrix() {
    constexpr int n = nsz(ORDER), mat = n * (n | 1), stage = kAsmLinks * (4 * (ORDER + 1) + 1 + n) + 2;
    return mat > stage ? mat : stage;
}
template <int ORDER>
__host__ __device__ constexpr int bidiag_doubles() { return bidiag_matrix<ORDER>() + (nsz(ORDER) + 2) + 2 * (nsz(ORDER) + 2); }
// Blocks a SM that shared memory leaves room for; the registers are held to them.
__host__ __device__ constexpr int bidiag_blocks(int order) { return order <= 6 ? 24 : order == 8 ? 12 : 6; }

// Whether the filter's moment matrix is the derivative one (labf.F90:258-303).
__device__ __forceinline__ bool same_matrix(const WArgs &a, int i, int t) {
    return a.h[i] == a.hs[i] && a.cnt[i] == a.cnt_small[i] && a.forder == a.morder && t != -2;
}

// Items of the two passes: every node but the boundary nodes, and those whose filter matrix
// is another one.
__global__ void k_weight_items(WArgs a, int *item0, int *item1, int *count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.npfb) return;
    const int t = a.ntype[i];
    if (!(t < 0 || t == 999 || t == 998)) return;  // boundary nodes: labf.F90:505-1039
    item0[atomicAdd(&count[0], 1)] = i;
    if (!same_matrix(a, i, t)) item1[atomicAdd(&count[1], 1)] = i;
}

// A block's moment matrix over links [0, cnt) with length hh (labf.F90:88-148 or 258-303; only the
// first `keep` unknowns, the identity beyond) and svdlib.F90:37-171.  One n x n matrix of
// shared memory (column-major, leading dimension n | 1, at smem) serves in turn for the bidiagonalisation, the
// accumulation of U, of which take_u(U) copies what it wants, and that of V, which it holds on
// return with the bidiagonal W, rv1 (1-based); returns anorm.  M (n x n doubles in memory) gets the
// moment matrix, column by column, and rows (as large) the bidiagonalised one, row by row.
//
// Bound: the shared-memory pipe.  A dependent FP64 operation takes some 25 cycles here, and the sums
// are single chains in the reference's order, so what counts is how many nodes a SM has under way:
// with both matrices in shared memory and the moment matrix's columns in registers they were six at
// order 8 (162 registers, latency-bound), now twelve (262,144 nodes 99 -> 83 ms; order 6,
// twenty-four blocks, 21 -> 17), which keep the LSU data pipe 91 % busy (FP64 37 %; 32,761 nodes
// 10.4 ms).
// Holding a thread's column in registers across a step's two loops, with 16-byte loads of the
// Householder vector, saved instructions and shared-memory traffic but no time at six (103 ms).
template <int ORDER, class TAKEU>
__device__ __forceinline__ double moment_bidiag(const WArgs &a, int i0, int cnt, double hh, int keep, double *smem, double *W,
                                                double *rv1, double *M, double *rows, TAKEU take_u) {
    constexpr int n = nsz(ORDER), ld = n | 1, T = bidiag_threads(ORDER);
    const int tid = threadIdx.x;
    double *U = smem, *V = smem, *pv = smem + bidiag_matrix<ORDER>();
    auto sync = [] {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    };
    {
        // the thread's unknown: exponents and 1 / (p! q!) of its monomial x^p y^q / (p! q!), evaluated
        // as written in labf.F90:1815-1920: x2=x*x, x3=x2*x, ..., then (coef*x^p)*y^q
        const int m = tid < n ? tid : 0;
        const int pm = p_of(m), qm = q_of(m);
        const double den = fact(pm) * fact(qm), inv = 1.0 / den;
        constexpr int P = ORDER + 1, RB = n <= 14 ? n : n <= 44 ? (n + 1) / 2 : 22;  // rows a pass over the links
        double *xp = smem, *yp = xp + kAsmLinks * P, *hx = yp + kAsmLinks * P, *hy = hx + kAsmLinks * P;
        double *ker = hy + kAsmLinks * P, *X = ker + kAsmLinks;
        const double xi = a.px[i0], yi = a.py[i0];
        for (int r0 = 0; r0 < n; r0 += RB) {
            double acc[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) acc[r] = 0.0;
            for (int k0 = 0; k0 < cnt; k0 += kAsmLinks) {
                const int nk = min(kAsmLinks, cnt - k0);
                sync();
                // a thread a link and coordinate
                const int kl = tid & (kAsmLinks - 1), side = tid / kAsmLinks;
                if (side < 2 && kl < nk) {
                    const int p = a.lpt[sell_off(a.slice_ptr, i0, k0 + kl)];
                    const double x = -(xi - a.px[p]), y = -(yi - a.py[p]);
                    if (side == 0) ker[kl] = wab(sqrt(x * x + y * y) / hh, a.h2);
                    const double z = (side ? y : x) / hh;
                    double *zp = side ? yp : xp, *hz = side ? hy : hx;
                    double pz = z;
                    zp[kl] = 1.0;
#pragma unroll
                    for (int d = 1; d <= ORDER; d++) {
                        zp[d * kAsmLinks + kl] = pz;
                        pz = pz * z;
                    }
#pragma unroll
                    for (int d = 0; d <= ORDER; d++) hz[d * kAsmLinks + kl] = hermite(d, z);
                }
                sync();
                if (tid < n)
                    for (int k = 0; k < nk; k++) {
                        const double xv = xp[pm * kAsmLinks + k], yv = yp[qm * kAsmLinks + k];
                        double v;
                        if (den == 1.0) v = pm == 0 ? yv : qm == 0 ? xv : xv * yv;
                        else v = qm == 0 ? inv * xv : pm == 0 ? inv * yv : (inv * xv) * yv;
                        X[k * n + tid] = v;
                    }
                sync();
                for (int k = 0; k < nk; k++) {
                    const double hxv = hx[pm * kAsmLinks + k], hyv = hy[qm * kAsmLinks + k];
                    const double g = (qm == 0 ? hxv : pm == 0 ? hyv : hxv * hyv) * ker[k];
#pragma unroll
                    for (int r = 0; r < RB; r++)  // (a last pass's rows beyond n are not kept)
                        acc[r] = acc[r] + X[k * n + r0 + r] * g;
                }
            }
            if (tid < n) {
#pragma unroll
                for (int r = 0; r < RB; r++)
                    if (r0 + r < n) M[tid * n + r0 + r] = acc[r];
            }
        }
        sync();
        for (int e = tid; e < n * n; e += T) {
            const int c = e / n, r = e - c * n;
            U[c * ld + r] = (c >= keep || r >= keep) ? (r == c ? 1.0 : 0.0) : M[e];
        }
        sync();
    }
#define UM(i, j) U[((j) - 1) * ld + ((i) - 1)]
#define VM(i, j) V[((j) - 1) * ld + ((i) - 1)]
    // svdlib.F90:37-113.  The scalars are computed by every thread alike; the pivot f - g stays in
    // a register until the column (row) is scaled back.
    double anorm = 0.0, g = 0.0, scale = 0.0;
    int l = 1;
    const int me = tid + 1;  // the thread's column, row or entry, 1-based
    for (int i = 1; i <= n; i++) {
        l = i + 1;
        const double ri = scale * g;
        if (tid == 0) rv1[i] = ri;
        g = 0.0;
        double s = 0.0;
        scale = 0.0;
#pragma unroll 4
        for (int k = i; k <= n; k++) scale = scale + fabs(UM(k, i));
        if (scale != 0.0) {
            sync();
            if (me >= i && me <= n) UM(me, i) = UM(me, i) / scale;
            sync();
#pragma unroll 4
            for (int k = i; k <= n; k++) s = s + UM(k, i) * UM(k, i);
            const double f = UM(i, i);
            g = -copysign(sqrt(s), f);
            const double h = f * g - s, piv = f - g;
            if (me >= l && me <= n) {
                double sj = 0.0;
                sj = sj + piv * UM(i, me);
#pragma unroll 4
                for (int k = l; k <= n; k++) sj = sj + UM(k, i) * UM(k, me);
                const double fj = sj / h;
                UM(i, me) = UM(i, me) + fj * piv;
#pragma unroll 4
                for (int k = l; k <= n; k++) UM(k, me) = UM(k, me) + fj * UM(k, i);
            }
            sync();
            if (me >= i && me <= n) UM(me, i) = scale * (me == i ? piv : UM(me, i));
        }
        const double wi = scale * g;
        if (tid == 0) W[i] = wi;
        g = 0.0; s = 0.0; scale = 0.0;
#pragma unroll 4
        for (int k = l; k <= n; k++) scale = scale + fabs(UM(i, k));
        if (scale != 0.0) {
            sync();
            if (me >= l && me <= n) UM(i, me) = UM(i, me) / scale;
            sync();
#pragma unroll 4
            for (int k = l; k <= n; k++) s = s + UM(i, k) * UM(i, k);
            const double f = UM(i, l);
            g = -copysign(sqrt(s), f);
            const double h = f * g - s, piv = f - g;
            if (me >= l && me <= n) rv1[me] = (me == l ? piv : UM(i, me)) / h;
            sync();
            if (me >= l && me <= n) {
                double sj = 0.0;
                sj = sj + UM(me, l) * piv;
#pragma unroll 4
                for (int k = l + 1; k <= n; k++) sj = sj + UM(me, k) * UM(i, k);
#pragma unroll 4
                for (int k = l; k <= n; k++) UM(me, k) = UM(me, k) + sj * rv1[k];
            }
            sync();
            if (me >= l && me <= n) UM(i, me) = scale * (me == l ? piv : UM(i, me));
        }
        sync();
        const double tn = fabs(wi) + fabs(ri);
        anorm = (tn > anorm) ? tn : anorm;
    }
    for (int e = tid; e < n * n; e += T) {
        const int r = e / n, k = e - r * n;
        rows[e] = U[k * ld + r];
    }
    sync();
    // left-hand transformations, svdlib.F90:143-171
    for (int i = n; i >= 1; i--) {
        l = i + 1;
        g = W[i];
        if (me >= l && me <= n) UM(i, me) = 0.0;  // read back by the same thread only
        const double pii = UM(i, i);
        if (g != 0.0) {
            g = 1.0 / g;
            if (me >= l && me <= n) {
                double sj = 0.0;
#pragma unroll 4
                for (int k = l; k <= n; k++) sj = sj + UM(k, i) * UM(k, me);
                const double fj = (sj / pii) * g;
                UM(i, me) = UM(i, me) + fj * pii;
#pragma unroll 4
                for (int k = l; k <= n; k++) UM(k, me) = UM(k, me) + fj * UM(k, i);
            }
            sync();
            if (me >= i && me <= n) UM(me, i) = me == i ? pii * g + 1.0 : UM(me, i) * g;
        } else {
            sync();
            if (me >= i && me <= n) UM(me, i) = me == i ? 0.0 + 1.0 : 0.0;
        }
        sync();
    }
    take_u(U);
    sync();
    // right-hand transformations, svdlib.F90:115-141, on the rows of the bidiagonalised matrix, each
    // fetched an i ahead
    double next = n > 1 && me <= n ? rows[(n - 2) * n + tid] : 0.0;
    g = 0.0;
    for (int i = n; i >= 1; i--) {
        if (i < n) {
            const double u = next;
            if (i > 1 && me <= n) next = rows[(i - 2) * n + tid];
            if (g != 0.0) {
                if (me <= n) pv[me] = u;
                sync();
                if (me >= l && me <= n) VM(me, i) = (u / pv[l]) / g;
                sync();
                if (me >= l && me <= n) {
                    double sj = 0.0;
#pragma unroll 4
                    for (int k = l; k <= n; k++) sj = sj + pv[k] * VM(k, me);
#pragma unroll 4
                    for (int k = l; k <= n; k++) VM(k, me) = VM(k, me) + sj * VM(k, i);
                }
                sync();
            }
            if (me >= l && me <= n) { VM(i, me) = 0.0; VM(me, i) = 0.0; }
        }
        if (tid == 0) VM(i, i) = 1.0;
        sync();
        g = rv1[i];
        l = i;
    }
    return anorm;
#undef UM
#undef VM
}

// One item a block: its matrix and the batch's arrays.  The item's place for V holds the moment
// matrix before, and its record the rows.
template <int ORDER>
__global__ void __launch_bounds__(bidiag_threads(ORDER), bidiag_blocks(ORDER)) k_moment_bidiag(WArgs a, SvdBatch B) {
    constexpr int n = nsz(ORDER), ld = n | 1, T = bidiag_threads(ORDER);
    extern __shared__ double smem[];
    const int it = blockIdx.x, tid = threadIdx.x, me = tid + 1;
    const int i0 = B.item[it], t = a.ntype[i0];
    double *rv1 = smem + bidiag_doubles<ORDER>() - 2 * (n + 2), *W = rv1 + (n + 2);
    // labf.F90:125-148, 305-323: next to walls only the first unknowns are kept
    int keep = n;
    if (B.pass == 0) {
        if (a.morder >= 7 && (t == 998 || t < 0)) keep = min(keep, 27);
        if (a.morder >= 5 && (t == -1 || t == -2)) keep = min(keep, 14);
    } else {
        if (a.forder >= 7 && (t == 998 || t < 0)) keep = min(keep, 27);
        if (a.forder >= 5 && t == -1) keep = min(keep, 14);
    }
    double *V = B.V + (size_t)it * n * n;
    const double anorm = moment_bidiag<ORDER>(
        a, i0, B.pass ? a.cnt[i0] : a.cnt_small[i0], B.pass ? a.h[i0] : a.hs[i0], keep, smem, W, rv1, V,
        reinterpret_cast<double *>(B.rec + (size_t)it * B.cap), [&](const double *U) {  // the rows that the solves read
            const int fo = filter_order(a.forder, t);
            for (int e = tid; e < kUrows * n; e += T) {
                const int r = e / n, c = e % n;
                double dummy;
                int row = r < 3 ? r : 4;
                if (r >= 4) row = hyp_entry(fo, r - 4, &dummy);
                B.U[(size_t)it * kUrows * n + e] = row >= 0 && row < n ? U[c * ld + row] : 0.0;
            }
        });
    for (int e = tid; e < n * n; e += T) V[e] = smem[(e / n) * ld + e % n];
    if (me <= n) {
        B.W[(size_t)me * B.batch + it] = W[me];
        B.rv1[(size_t)me * B.batch + it] = rv1[me];
    }
    if (tid == 0) {
        B.anorm[it] = anorm;
        B.state[it] = make_int2(n, 1);
    }
}

// What a record entry's header says the entries after it are.
enum { kRecSweep = 0, kRecCancel = 1, kRecNegate = 2 };
__device__ __forceinline__ double4 rec_header(int kind, int col, int count) {
    return make_double4(__hiloint2double(kind, col), __hiloint2double(0, count), 0.0, 0.0);
}

constexpr int kQrThreads = 32;

// svdlib.F90:173-278 on the bidiagonal alone, one thread an item.  The item's record gets, for
// each sweep, a header (kind, first column, entries) and the rotations.  Bound: the latency of
// the recurrence (about 700 cycles a rotation; wait stalls lead, FP64 23 % busy), hidden by as many
// items as the batch has (32,761 nodes 0.90 ms).
template <int ORDER>
__global__ void __launch_bounds__(kQrThreads) k_bidiag_qr(SvdBatch B, int maxits) {
    constexpr int n = nsz(ORDER);
    extern __shared__ double smem[];
    const int it = blockIdx.x * kQrThreads + threadIdx.x;
    if (it >= B.n_items) return;
    const int2 st = B.state[it];
    if (st.x <= 0) {
        B.nrec[it] = -1;
        return;
    }
    double *Ws = smem + threadIdx.x, *Rs = Ws + (n + 1) * kQrThreads;
#define WQ(j) Ws[(j) * kQrThreads]
#define RQ(j) Rs[(j) * kQrThreads]
    for (int j = 1; j <= n; j++) {
        WQ(j) = B.W[(size_t)j * B.batch + it];
        RQ(j) = B.rv1[(size_t)j * B.batch + it];
    }
    const double anorm = B.anorm[it];
    double4 *rec = B.rec + (size_t)it * B.cap;
    int pos = 0;
    int2 next = make_int2(0, 0);
    int its0 = st.y;
    for (int k = st.x; k >= 1; k--) {
        bool stop = false;
        for (int its = its0; its <= 30; its++) {
            if (pos + 2 * n + 4 > B.cap) {  // a sweep and a cancellation at most before the next look
                next = make_int2(k, its);
                stop = true;
                break;
            }
            bool to2000 = false;
            int l, nm = 1;
            for (l = k; l >= 1; l--) {
                nm = l - 1;
                if ((fabs(RQ(l)) + anorm) == anorm) { to2000 = true; break; }
                if ((fabs(WQ(nm)) + anorm) == anorm) break;
            }
            if (l < 1) {  // no split found: only a NaN in the bidiagonal gets here
                next = make_int2(-1, 0);
                stop = true;
                break;
            }
            double c, s, f, g, h, x, y, z;
            if (!to2000) {
                const int at = pos++;
                int m = 0;
                c = 0.0; s = 1.0;
                for (int i = l; i <= k; i++) {
                    const double r = RQ(i);
                    f = s * r;
                    RQ(i) = c * r;
                    if ((fabs(f) + anorm) == anorm) break;
                    g = WQ(i);
                    h = nr_hypot(f, g);
                    WQ(i) = h;
                    h = 1.0 / h;
                    c = (g * h);
                    s = -(f * h);
                    rec[pos++] = make_double4(0.0, 0.0, c, s);
                    m++;
                }
                rec[at] = rec_header(kRecCancel, l, m);
            }
            z = WQ(k);
            if (l == k) {
                if (z < 0.0) {
                    WQ(k) = -z;
                    rec[pos++] = rec_header(kRecNegate, k, 0);
                }
                break;
            }
            if (its >= maxits) {
                next = make_int2(-1, 0);
                stop = true;
                break;
            }
            x = WQ(l);
            nm = k - 1;
            y = WQ(nm);
            g = RQ(nm);
            h = RQ(k);
            f = ((y - z) * (y + z) + (g - h) * (g + h)) / ((2.0 * h) * y);
            g = nr_hypot(f, 1.0);
            f = ((x - z) * (x + z) + h * ((y / (f + copysign(g, f))) - h)) / x;
            c = 1.0; s = 1.0;
            rec[pos++] = rec_header(kRecSweep, l, nm - l + 1);
            for (int j = l; j <= nm; j++) {
                const int i = j + 1;
                g = RQ(i);
                y = WQ(i);
                h = s * g;
                g = c * g;
                z = nr_hypot(f, h);
                RQ(j) = z;
                c = f / z;
                s = h / z;
                const double c1 = c, s1 = s;
                f = (x * c) + (g * s);
                g = -(x * s) + (g * c);
                h = y * s;
                y = y * c;
                z = nr_hypot(f, h);
                WQ(j) = z;
                if (z != 0.0) {
                    z = 1.0 / z;
                    c = f * z;
                    s = h * z;
                }
                f = (c * g) + (s * y);
                x = -(s * g) + (c * y);
                rec[pos++] = make_double4(c1, s1, c, s);
            }
            RQ(l) = 0.0;
            RQ(k) = f;
            WQ(k) = x;
        }
        if (stop) break;
        its0 = 1;
    }
    for (int j = 1; j <= n; j++) {
        B.W[(size_t)j * B.batch + it] = WQ(j);
        B.rv1[(size_t)j * B.batch + it] = RQ(j);
    }
    B.state[it] = next;
    B.nrec[it] = pos;
    if (next.x > 0) atomicAdd(B.left, 1);
#undef WQ
#undef RQ
}

constexpr int kApplyWarps = 1;  // items a block of k_weights_apply (one warp each)
template <int ORDER>
__host__ __device__ constexpr int apply_doubles() {
    // rows [n + kUrows][n | 1], two staged halves of 32 record entries, W, one solve, five results
    return ((nsz(ORDER) + kUrows) * (nsz(ORDER) | 1) + 2 * 32 * 4 + (nsz(ORDER) + 2) + 6 * nsz(ORDER) + 3) & ~3;
}

// The recorded rotations replayed on the item's rows (lanes take rows; a sweep's rotation j acts
// on columns j and j + 1, so the second column stays in a register for the next one), then,
// once the item is done, svdlib.F90:279-303 for each right-hand side and the weights of its
// links (labf.F90:157-231, 325-388).  Bound: latency at nine warps a SM, and shared
// memory (12 multiplies and adds and 2 shared loads and stores a rotation and warp: LSU data pipe
// 59 % busy, issue 38 %, FP64 27 %; 32,761 nodes 2.3 ms).
template <int ORDER>
__global__ void __launch_bounds__(kApplyWarps * 32) k_weights_apply(WArgs a, SvdBatch B) {
    constexpr int n = nsz(ORDER), ld = n | 1, rows = n + kUrows, SL = (rows + 31) / 32;
    extern __shared__ __align__(32) double smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int it = blockIdx.x * kApplyWarps + warp;
    if (it >= B.n_items) return;
    const int2 st = B.state[it];
    const int nrec = B.nrec[it];
    if (nrec < 0) return;  // done in an earlier round
    double *stage = smem + (size_t)warp * apply_doubles<ORDER>();  // first, for its alignment
    double *R = stage + 2 * 32 * 4, *W = R + rows * ld, *tmp = W + (n + 2), *bx = tmp + n, *by = bx + n,
           *bxx = by + n, *byy = bxx + n, *bh = byy + n;
    const int i = B.item[it], t = a.ntype[i];
    if (st.x < 0) {
        if (lane == 0) atomicExch(a.err, i + 1);
        return;
    }
    double *Vg = B.V + (size_t)it * n * n, *Ug = B.U + (size_t)it * kUrows * n;
    for (int e = lane; e < n * n; e += 32) R[(e % n) * ld + e / n] = Vg[e];
    for (int e = lane; e < kUrows * n; e += 32) R[(n + e / n) * ld + e % n] = Ug[e];
    const double4 *rec = B.rec + (size_t)it * B.cap;
    double4 pre = lane < nrec ? rec[lane] : make_double4(0, 0, 0, 0);
    int e = 0;
    // entry e of the record: 32 at a time come in ahead of their use
    auto fetch = [&]() -> double4 {
        if ((e & 31) == 0) {
            __syncwarp();
            reinterpret_cast<double4 *>(stage)[(e & 32) + lane] = pre;
            if (e + 32 + lane < nrec) pre = rec[e + 32 + lane];
            __syncwarp();
        }
        const double4 v = reinterpret_cast<const double4 *>(stage)[e & 63];
        e++;
        return v;
    };
    double *row[SL];
    bool isu[SL], live[SL];
#pragma unroll
    for (int q = 0; q < SL; q++) {
        const int r = lane + 32 * q;
        live[q] = r < rows;
        isu[q] = r >= n;
        row[q] = R + (live[q] ? r : 0) * ld;
    }
    __syncwarp();
    while (e < nrec) {
        const double4 hd = fetch();
        const int kind = __double2hiint(hd.x), col = __double2loint(hd.x) - 1, count = __double2loint(hd.y);
        if (kind == kRecSweep) {
            double x[SL];
#pragma unroll
            for (int q = 0; q < SL; q++) x[q] = row[q][col];
            for (int j = 0; j < count; j++) {
                const double4 cs = fetch();
#pragma unroll
                for (int q = 0; q < SL; q++) {
                    const double c = isu[q] ? cs.z : cs.x, s = isu[q] ? cs.w : cs.y;
                    const double z = row[q][col + j + 1];
                    const double xn = (x[q] * c) + (z * s);
                    if (live[q]) row[q][col + j] = xn;
                    x[q] = -(x[q] * s) + (z * c);
                }
            }
#pragma unroll
            for (int q = 0; q < SL; q++)
                if (live[q]) row[q][col + count] = x[q];
        } else if (kind == kRecCancel) {  // columns l - 1 and i of U
            for (int j = 0; j < count; j++) {
                const double4 cs = fetch();
#pragma unroll
                for (int q = 0; q < SL; q++)
                    if (live[q] && isu[q]) {
                        const double y = row[q][col - 1], z = row[q][col + j];
                        row[q][col - 1] = (y * cs.z) + (z * cs.w);
                        row[q][col + j] = -(y * cs.w) + (z * cs.z);
                    }
            }
        } else {
#pragma unroll
            for (int q = 0; q < SL; q++)
                if (live[q] && !isu[q]) row[q][col] = -row[q][col];
        }
    }
    __syncwarp();
    if (st.x > 0) {  // more sweeps to come
        for (int e2 = lane; e2 < n * n; e2 += 32) Vg[e2] = R[(e2 % n) * ld + e2 / n];
        for (int e2 = lane; e2 < kUrows * n; e2 += 32) Ug[e2] = R[(n + e2 / n) * ld + e2 % n];
        return;
    }
    for (int j = lane; j < n; j += 32) W[j + 1] = B.W[(size_t)(j + 1) * B.batch + it];
    __syncwarp();
    const bool same = same_matrix(a, i, t);
    const bool deriv = B.pass == 0, filt = B.pass == 1 || same;
    if (lane == 0) {
        const double cond = svd_cond<n>(W);
        if (deriv && a.cond_d) a.cond_d[i] = cond;
        if (filt && a.cond_f) a.cond_f[i] = cond;
    }
    // b <- V diag(1/w) U^T b; the entries of U^T b are sums over the nonzero entries of b
    auto solve = [&](double *b, int r0, int nr, const double *coef) {
        __syncwarp();
        for (int j = lane; j < n; j += 32) {
            double s = 0.0;
            if (W[j + 1] != 0.0) {
                for (int r = 0; r < nr; r++) s = s + R[(n + r0 + r) * ld + j] * coef[r];
                s = s / W[j + 1];
            }
            tmp[j] = s;
        }
        __syncwarp();
        for (int j = lane; j < n; j += 32) {
            double s = 0.0;
            for (int jj = 0; jj < n; jj++) s = s + R[j * ld + jj] * tmp[jj];
            b[j] = s;
        }
        __syncwarp();
    };
    const double one = 1.0;
    if (deriv) {
        solve(bx, 0, 1, &one);
        solve(by, 1, 1, &one);
        solve(bxx, 2, 1, &one);
        solve(byy, 3, 1, &one);
        for (int m = lane; m < n; m += 32) bxx[m] = bxx[m] + byy[m];  // bvecxx + bvecyy
    }
    if (filt) {
        const int fo = filter_order(a.forder, t);
        double coef[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        int nr = 0;
        while (nr < 6 && hyp_entry(fo, nr, &coef[nr]) >= 0) nr++;
        solve(bh, 4, nr, coef);
    }
    __syncwarp();
    const double hh = deriv ? a.hs[i] : a.h[i];
    const double xi = a.px[i], yi = a.py[i];
    const int cnt = a.cnt[i];
    for (int k = lane; k < cnt; k += 32) {
        const long long o = sell_off(a.slice_ptr, i, k);
        const int p = a.lpt[o];
        const double x = -(xi - a.px[p]), y = -(yi - a.py[p]);
        const double rad = sqrt(x * x + y * y) / hh;
        const double ff1 = wab(rad, a.h2);
        const double xx = x / hh, yy = y / hh;
        double hx[ORDER + 1], hy[ORDER + 1];
#pragma unroll
        for (int d = 0; d <= ORDER; d++) { hx[d] = hermite(d, xx); hy[d] = hermite(d, yy); }
        double sx = 0.0, sy = 0.0, sl = 0.0, sh = 0.0;
#pragma unroll
        for (int m = 0; m < n; m++) {
            const int pm = p_of(m), qm = q_of(m);
            double g = (qm == 0) ? hx[pm] : (pm == 0) ? hy[qm] : hx[pm] * hy[qm];
            g = g * ff1;
            if (deriv) {
                sx = sx + bx[m] * g;
                sy = sy + by[m] * g;
                sl = sl + bxx[m] * g;
            }
            if (filt) sh = sh + bh[m] * g;
        }
        if (deriv) {
            a.wx[o] = sx / hh;
            a.wy[o] = sy / hh;
            a.wl[o] = (sl / hh) / hh;
        }
        if (filt) a.wh[o] = sh;
    }
}

// calc_labf_sums (labf.F90:396-451) and calc_node_volumes (:453-503), one thread per node;
// link k of a slice is read by the 32 threads of a warp at once.
struct SumArgs {
    int npfb;
    double L;
    const double *px, *py, *h, *sp;
    const int *ntype, *cnt, *lpt, *fdpar;
    const long long *slice_ptr;
    double *wx, *wy, *wl, *wh, *gsx, *gsy, *lsum, *hsum, *vol;
};

__global__ void k_labf_sums(SumArgs a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.npfb) return;
    const long long base = a.slice_ptr[i >> 5];
    const int lane = i & 31;
    const int cnt = a.cnt[i];
    double gx = 0.0, gy = 0.0, lp = 0.0, hy = 0.0;
    for (int k = 0; k < cnt; k++) {
        long long o = sell_at(base, k, lane);
        hy = hy + a.wh[o];
        gx = gx + a.wx[o];
        gy = gy + a.wy[o];
        lp = lp + a.wl[o];
    }
    a.gsx[i] = gx / a.L;
    a.gsy[i] = gy / a.L;
    a.lsum[i] = (lp / a.L) / a.L;
    a.hsum[i] = hy;
    for (int k = 0; k < cnt; k++) {
        long long o = sell_at(base, k, lane);
        a.wx[o] = a.wx[o] / a.L;
        a.wy[o] = a.wy[o] / a.L;
        a.wl[o] = (a.wl[o] / a.L) / a.L;
    }
    const int t = a.ntype[i];
    if (t < 0 || t == 999 || t == 998) {
        const double hh = a.h[i], xi = a.px[i], yi = a.py[i];
        double v = 0.0;
        for (int k = 0; k < cnt; k++) {
            int p = a.lpt[sell_at(base, k, lane)];
            double x = -(xi - a.px[p]), y = -(yi - a.py[p]);
            double rad = sqrt(x * x + y * y) / hh;
            double f1 = ((9.0 / kPi) * exp((-9.0 * rad) * rad)) / (hh * hh);
            v = v + f1;
        }
        a.vol[i] = 1.0 / v;
    } else {
        a.vol[i] = a.sp[i] * a.sp[i];
    }
}

// filter_coefficients, labf.F90:1723-1811, with the reduction of the FD rows of walls.
__global__ void k_filter_coeff(SumArgs a) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.npfb) return;
    const long long base = a.slice_ptr[i >> 5];
    const int lane = i & 31;
    const int cnt = a.cnt[i];
    const double xi = a.px[i], yi = a.py[i];
    const int t = a.ntype[i];
    double fc;
    if (t < 0 || t == 999 || t == 998) {
        double lscal = (2.0 * a.h[i]) * sqrt(kPi / (double)cnt);
        double tmp = ((2.0 / 3.0) * kPi) / lscal;
        double lsum = 0.0;
        for (int k = 0; k < cnt; k++) {
            long long o = sell_at(base, k, lane);
            int p = a.lpt[o];
            double x = a.px[p] - xi, y = a.py[p] - yi;
            double fji = 1.0 - cos(tmp * x) * cos(tmp * y);
            lsum = lsum + fji * a.wh[o];
        }
        fc = (2.0 / 3.0) / lsum;
        if (t < 0 && a.ntype[a.fdpar[i]] == 0) {
            const double oosqrt2 = 1.0 / sqrt(2.0);
            if (t == -1) fc = (fc * 0.5) * oosqrt2;
            if (t == -2) fc = fc * 0.5;
            if (t == -3) fc = fc * oosqrt2;
            if (t == -4) fc = fc * oosqrt2;
        }
    } else {
        double tmp = ((2.0 / 3.0) * kPi) / a.sp[i];
        double lsum = 0.0;
        for (int k = 0; k < cnt; k++) {
            long long o = sell_at(base, k, lane);
            int p = a.lpt[o];
            double x = a.px[p] - xi, y = a.py[p] - yi;
            double fji = 1.0 - cos(tmp * sqrt(x * x + y * y));
            lsum = lsum + fji * a.wh[o];
        }
        fc = (1.0 / 3.0) / lsum;
        fc = fc * 0.5;
    }
    double sum = 0.0;
    for (int k = 0; k < cnt; k++) {
        long long o = sell_at(base, k, lane);
        double w = a.wh[o] * fc;
        a.wh[o] = w;
        sum = sum + w;
    }
    a.hsum[i] = sum;
}

// ---------------------------------------------------------------------------------------
// calc_boundary_weights (labf.F90:505-1039): boundary node i0 and its FD rows i1..i4.
// Normal first and second derivatives of i0, i1, i2 are the reference's 5-point finite
// differences; tangential ones come from 6th-order 1-D LABFM on the node's own layer (a
// 6 x 6 moment matrix, factored by the warp SVD above, so bit for bit the restatement's);
// then the wall curvature, the divergence term of rows 1-2 and the rotation of rows 1-2 to
// the x-y frame.  Wall first derivatives stay in the normal-tangent frame: the wall
// equations are written there.
// ---------------------------------------------------------------------------------------
struct BndArgs {
    int npfb, nb, nplink;
    double h3;
    const double *px, *py, *h, *sp, *rnx, *rny;
    const int *ntype, *gpar, *fdpar, *blist, *brow;
    int *cnt, *cnt_small, *lpt, *lidx;
    uint16_t *lloc;
    const long long *slice_ptr;
    const int *slice_w;
    double *wx, *wy, *wl, *wh;
    double *wb2;  // nb x nplink x 2: second derivatives (normal, tangential) of boundary nodes
    int *err;
};

// point p (interior or ghost) -> the interior node whose data it carries
__device__ __forceinline__ int bnd_owner(const BndArgs &a, int p) { return p < a.npfb ? p : a.gpar[p - a.npfb]; }

// rbfs.F90:58-68 (the kernel derivative `fac` of the 1-D operators; it uses the global h3)
__device__ __forceinline__ double fac(double qq, double h3) {
    double qq2 = qq * qq, qq3 = qq * qq2, qq4 = qq * qq3;
    double f = 0.0;
    if (qq <= 2.0 && qq > 0.0)
        f = (7.0 / ((4.0 * kPi) * h3)) * ((((0.625 * qq4) - (3.75 * qq3)) + (7.5 * qq2)) - (5.0 * qq));
    return f;
}

// labf.F90:1041-1048
__device__ __forceinline__ double monomial1d(int m, double z) {
    double z2 = z * z;
    switch (m) {
    case 0: return z;
    case 1: return 0.5 * z2;
    case 2: return ((1.0 / 6.0) * z) * z2;
    case 3: return (z2 * z2) / 24.0;
    case 4: return ((z2 * z2) * z) / 120.0;
    default: return ((z2 * z2) * z2) / 720.0;
    }
}

// labf.F90:1050-1077 (ABF==2)
__device__ __forceinline__ double abf1d(int m, double z, double ff1) {
    if (m == 2) return (ff1 * (1.0 / sqrt(2.0))) * hermite(3, z);
    return ff1 * hermite(m + 1, z);
}

// tangential coordinate (scaled by hh) of point p relative to node i, and its kernel value
__device__ __forceinline__ void tangential(const BndArgs &a, int i, int p, double xt, double yt, double hh,
                                           double &z, double &ff1) {
    double rijx = a.px[i] - a.px[p], rijy = a.py[i] - a.py[p];
    double x = -(rijx * xt + rijy * yt);
    if (i == p) x = 0.0;
    ff1 = fac(fabs(x / hh), a.h3);
    z = x / hh;
}

__device__ __forceinline__ double dot6(const double *b, const double *g) {
    double t = 0.0;
    for (int k = 0; k < 6; k++) t = t + b[k] * g[k];
    return t;
}

constexpr int kBndWarpDoubles = 2 * 6 * 7 + 3 * 8 + 3 * 6;  // U, V, W/rv1/tmp, three right-hand sides

// 1-D moment matrix of node i along (xt, yt) over its links on its own layer, then its
// factorisation; lanes 0..35 each own one matrix entry and sum it over the links in order.
__device__ int bnd_factor_1d(const BndArgs &a, int i, double xt, double yt, double hh, double *U, double *V,
                             double *W, double *rv1, int lane) {
    const long long base = a.slice_ptr[i >> 5];
    const int ti = a.ntype[i], cnt = a.cnt[i];
    for (int e = lane; e < 36; e += 32) {
        const int i1 = e % 6, i2 = e / 6;
        double acc = 0.0;
        for (int k = 0; k < cnt; k++) {
            const int p = a.lpt[sell_at(base, k, i & 31)];
            if (a.ntype[bnd_owner(a, p)] != ti) continue;
            double rijx = a.px[i] - a.px[p], rijy = a.py[i] - a.py[p];
            double x = -(rijx * xt + rijy * yt);
            if (i == p) x = 0.0;
            const double xv = monomial1d(i1, x / hh);
            double z, ff1;
            tangential(a, i, p, xt, yt, hh, z, ff1);
            acc = acc + xv * abf1d(i2, z, ff1);
        }
        U[i2 * 7 + i1] = acc;
    }
    __syncwarp();
    return svd_factor_warp<6>(U, V, W, rv1, 7, lane);
}

// Drop every link of boundary node jj that is neither on its own layer nor one of its FD
// children (labf.F90:541-565), compacting the SELL slots in order; the freed slots become
// padding.
__global__ void k_prune_boundary_links(BndArgs a) {
    const int jj = blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= a.nb) return;
    const int i = a.blist[jj], kk = a.ntype[i], c = a.cnt[i];
    const long long base = a.slice_ptr[i >> 5];
    const int ln = i & 31;
    int w = 0;
    for (int k = 0; k < c; k++) {
        const long long o = sell_at(base, k, ln);
        const int p = a.lpt[o];
        const bool keep = (a.ntype[bnd_owner(a, p)] == kk) || (p < a.npfb && a.fdpar[p] == i);
        if (!keep) continue;
        const long long o2 = sell_at(base, w, ln);
        a.lpt[o2] = p;
        a.lidx[o2] = a.lidx[o];
        a.lloc[o2] = a.lloc[o];
        w++;
    }
    for (int k = w; k < c; k++) {
        const long long o = sell_at(base, k, ln);
        a.lpt[o] = 0;
        a.lidx[o] = 0;
        a.lloc[o] = 0;
    }
    a.cnt[i] = w;
    a.cnt_small[i] = w;
}

// Boundary nodes: normal FD operators (labf.F90:572-612) and tangential 1-D LABFM
// (:688-755).  One warp per boundary node.
__global__ void k_boundary_node_weights(BndArgs a) {
    __shared__ double sm[4][kBndWarpDoubles];
    const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
    const int jj = blockIdx.x * 4 + wrp;
    if (jj >= a.nb) return;
    double *U = sm[wrp], *V = U + 42, *W = V + 42, *rv1 = W + 8, *tmp = rv1 + 8, *bt = tmp + 8, *btt = bt + 6,
           *bh = btt + 6;
    const int i = a.blist[jj];
    const long long base = a.slice_ptr[i >> 5];
    const int ln = i & 31, cnt = a.cnt[i];
    const double dx = a.sp[i], dx2 = dx * dx;
    double *wb = a.wb2 + (size_t)jj * a.nplink * 2;
    for (int k = lane; k < a.slice_w[i >> 5]; k += 32) {
        const long long o = sell_at(base, k, ln);
        a.wx[o] = 0.0; a.wy[o] = 0.0; a.wl[o] = 0.0; a.wh[o] = 0.0;
    }
    for (int k = lane; k < a.nplink; k += 32) { wb[2 * k] = 0.0; wb[2 * k + 1] = 0.0; }
    __syncwarp();
    for (int k = lane; k < cnt; k += 32) {
        const long long o = sell_at(base, k, ln);
        const int p = a.lpt[o];
        if (p >= a.npfb || a.fdpar[p] != i) continue;
        const int t = a.ntype[p];
        if (t == -1) { a.wx[o] = 4.0 / dx; wb[2 * k] = -((104.0 / 12.0) / dx2); }
        if (t == -2) { a.wx[o] = -(3.0 / dx); wb[2 * k] = (114.0 / 12.0) / dx2; }
        if (t == -3) { a.wx[o] = (4.0 / 3.0) / dx; wb[2 * k] = -((56.0 / 12.0) / dx2); }
        if (t == -4) { a.wx[o] = -(0.25 / dx); wb[2 * k] = (11.0 / 12.0) / dx2; }
    }
    const double xt = -a.rny[i], yt = a.rnx[i], hh = a.h[i];
    __syncwarp();
    if (bnd_factor_1d(a, i, xt, yt, hh, U, V, W, rv1, lane)) {
        if (lane == 0) atomicExch(a.err, i + 1);
        return;
    }
    for (int m = lane; m < 6; m += 32) {
        bt[m] = (m == 0) ? 1.0 : 0.0;
        btt[m] = (m == 1) ? 1.0 : 0.0;
        bh[m] = (m == 3) ? -1.0 : 0.0;
    }
    svd_apply_warp<6>(U, V, W, tmp, bt, 7, lane);
    svd_apply_warp<6>(U, V, W, tmp, btt, 7, lane);
    svd_apply_warp<6>(U, V, W, tmp, bh, 7, lane);
    const int ti = a.ntype[i];
    for (int k = lane; k < cnt; k += 32) {
        const long long o = sell_at(base, k, ln);
        const int p = a.lpt[o];
        if (a.ntype[bnd_owner(a, p)] != ti) continue;
        double z, ff1, g[6];
        tangential(a, i, p, xt, yt, hh, z, ff1);
        for (int m = 0; m < 6; m++) g[m] = abf1d(m, z, ff1);
        a.wy[o] = dot6(bt, g) / hh;
        wb[2 * k + 1] = (dot6(btt, g) / hh) / hh;
        a.wh[o] = a.wh[o] + dot6(bh, g);
    }
}

// FD rows 1 and 2: normal FD operators (labf.F90:615-676) and tangential 1-D LABFM on a
// tangent rotated by the tangential gradient of the resolution (:758-955).  One warp per
// (boundary node, row).
__global__ void k_boundary_row_weights(BndArgs a) {
    __shared__ double sm[4][kBndWarpDoubles];
    const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
    const int w = blockIdx.x * 4 + wrp;
    if (w >= 2 * a.nb) return;
    const int jj = w >> 1, row = 1 + (w & 1);
    double *U = sm[wrp], *V = U + 42, *W = V + 42, *rv1 = W + 8, *tmp = rv1 + 8, *bt = tmp + 8, *btt = bt + 6;
    const int i = a.brow[4 * jj + row - 1], par = a.blist[jj];
    const long long base = a.slice_ptr[i >> 5];
    const int ln = i & 31, cnt = a.cnt[i];
    const double dx = a.sp[i], dx2 = dx * dx;
    for (int k = lane; k < a.slice_w[i >> 5]; k += 32) {
        const long long o = sell_at(base, k, ln);
        a.wx[o] = 0.0; a.wy[o] = 0.0; a.wl[o] = 0.0;
    }
    __syncwarp();
    for (int k = lane; k < cnt; k += 32) {
        const long long o = sell_at(base, k, ln);
        const int p = a.lpt[o];
        if (p >= a.npfb) continue;
        const int t = a.ntype[p];
        const bool same = a.fdpar[p] == par;
        if (row == 1) {
            if (p == par) { a.wx[o] = -(0.25 / dx); a.wl[o] = (11.0 / 12.0) / dx2; }
            if (t == -2 && same) { a.wx[o] = 1.5 / dx; a.wl[o] = (6.0 / 12.0) / dx2; }
            if (t == -3 && same) { a.wx[o] = -(0.5 / dx); a.wl[o] = (4.0 / 12.0) / dx2; }
            if (t == -4 && same) { a.wx[o] = (1.0 / 12.0) / dx; a.wl[o] = -((1.0 / 12.0) / dx2); }
        } else {
            if (p == par) { a.wx[o] = (1.0 / 12.0) / dx; a.wl[o] = -((1.0 / 12.0) / dx2); }
            if (t == -1 && same) { a.wx[o] = -((8.0 / 12.0) / dx); a.wl[o] = (16.0 / 12.0) / dx2; }
            if (t == -3 && same) { a.wx[o] = (8.0 / 12.0) / dx; a.wl[o] = (16.0 / 12.0) / dx2; }
            if (t == -4 && same) { a.wx[o] = -((1.0 / 12.0) / dx); a.wl[o] = -((1.0 / 12.0) / dx2); }
        }
    }
    // tangential gradient of the resolution at the boundary node, in the order of its links
    double grads = 0.0;
    {
        const long long pb = a.slice_ptr[par >> 5];
        for (int k = 0; k < a.cnt[par]; k++) {
            const long long o = sell_at(pb, k, par & 31);
            const int p = a.lpt[o];
            grads = grads + (a.sp[bnd_owner(a, p)] - a.sp[par]) * a.wy[o];
        }
    }
    grads = -atan(grads);
    const double xt = cos(grads) * (-a.rny[i]) - sin(grads) * a.rnx[i];
    const double yt = sin(grads) * (-a.rny[i]) + cos(grads) * a.rnx[i];
    const double hh = a.h[i];
    __syncwarp();
    if (bnd_factor_1d(a, i, xt, yt, hh, U, V, W, rv1, lane)) {
        if (lane == 0) atomicExch(a.err, i + 1);
        return;
    }
    for (int m = lane; m < 6; m += 32) {
        bt[m] = (m == 0) ? 1.0 : 0.0;
        btt[m] = (m == 1) ? 1.0 : 0.0;
    }
    svd_apply_warp<6>(U, V, W, tmp, bt, 7, lane);
    svd_apply_warp<6>(U, V, W, tmp, btt, 7, lane);
    const int ti = a.ntype[i];
    const double sec = 1.0 / cos(grads), tn = tan(grads);
    for (int k = lane; k < cnt; k += 32) {
        const long long o = sell_at(base, k, ln);
        const int p = a.lpt[o];
        if (a.ntype[bnd_owner(a, p)] == ti) {
            double z, ff1, g[6];
            tangential(a, i, p, xt, yt, hh, z, ff1);
            for (int m = 0; m < 6; m++) g[m] = abf1d(m, z, ff1);
            a.wy[o] = dot6(bt, g) / hh;
            a.wl[o] = a.wl[o] + (dot6(btt, g) / hh) / hh;
        }
        a.wy[o] = sec * a.wy[o] - tn * a.wx[o];
    }
}

// Wall curvature, outflow sign, divergence term of rows 1-2, wall Laplacian, rows 1-2 to
// the x-y frame (labf.F90:965-1035).  One thread per boundary node.
__global__ void k_boundary_frame(BndArgs a) {
    const int jj = blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= a.nb) return;
    const int i = a.blist[jj], ti = a.ntype[i];
    const long long base = a.slice_ptr[i >> 5];
    const int ln = i & 31;
    double *wb = a.wb2 + (size_t)jj * a.nplink * 2;
    double ooR = 0.0;
    if (ti == 0) {
        double tmp_t = 0.0;
        for (int k = 0; k < a.cnt[i]; k++) {
            const int p = a.lpt[sell_at(base, k, ln)];
            const int q = bnd_owner(a, p);
            if (a.ntype[q] != ti) continue;
            const double tmp_n = ((a.rnx[q] * a.rnx[i] + a.rny[q] * a.rny[i]) + 0.0 * 0.0) - 1.0;
            tmp_t = tmp_t + wb[2 * k + 1] * tmp_n;
        }
        ooR = sqrt(fabs(tmp_t));
    }
    if (ti == 2)
        for (int k = 0; k < a.slice_w[i >> 5]; k++) {
            const long long o = sell_at(base, k, ln);
            a.wx[o] = -a.wx[o];
            a.wy[o] = -a.wy[o];
        }
    for (int row = 1; row <= 2; row++) {
        if (ti != 0) break;
        const int r = a.brow[4 * jj + row - 1];
        const long long rb = a.slice_ptr[r >> 5];
        const double den = row == 1 ? 1.0 + ooR * a.sp[r] : 1.0 + (2.0 * ooR) * a.sp[r];
        for (int k = 0; k < a.slice_w[r >> 5]; k++) {
            const long long o = sell_at(rb, k, r & 31);
            a.wl[o] = a.wl[o] + (a.wx[o] * ooR) / den;
        }
    }
    if (ti == 0)
        for (int k = 0; k < a.cnt[i]; k++) {
            const long long o = sell_at(base, k, ln);
            wb[2 * k] = wb[2 * k] + a.wx[o] * ooR;
            a.wl[o] = wb[2 * k] + wb[2 * k + 1];
        }
    const double xn = a.rnx[i], yn = a.rny[i];
    for (int row = 1; row <= 2; row++) {
        const int r = a.brow[4 * jj + row - 1];
        const long long rb = a.slice_ptr[r >> 5];
        for (int k = 0; k < a.cnt[r]; k++) {
            const long long o = sell_at(rb, k, r & 31);
            const double g1 = a.wx[o], g2 = a.wy[o];
            a.wx[o] = (0.0 + xn * g1) + (-yn) * g2;
            a.wy[o] = (0.0 + yn * g1) + xn * g2;
        }
    }
}

// adapt_stencils + adapt_stencils_main (labf.F90:1079-1721), 2-D, Hermite ABFs.  One warp
// per plain interior node (node_type > 2, not 998).  The length scale shrinks by the
// reference's single-precision factor 0.98 while the Laplacian system's residual stays below
// res_tol / h, no wavenumber q = i pi / (32 s), i = 1..33, is amplified beyond 1.0001 by the
// d/dx, d/dy or Laplacian stencil (nor turned negative by the Laplacian), and at most
// `limit` reductions have been made.  Pass 0 reduces h (h_small with it) over the node's
// list, pass 1 h_small over its small list.  The lists are sorted by distance, so the links
// within 2 h are a prefix of each.  The arithmetic follows the CPU restatement operation for
// operation (the same moment matrix, SVD and sums in the same order); the amplification
// sums run one wavenumber a thread, each over the links in order.  A moment matrix whose SVD
// does not converge ends the node's reduction (the reference stops).
struct AdaptArgs {
    WArgs w;
    double *h, *hs;
    const double *sp;
    double *M;  // a block's moment matrix and its rows
    int *next;  // the next node to take
    int nplink;
    double rf, limit, res_tol[2];
};

// Rows of U that the three solves read: 0, 1, 2 and 4.
constexpr int kAdaptUrows = 4;
template <int ORDER>
__host__ __device__ constexpr int adapt_vectors() {  // the warps' bidiagonals, tmp, bl, bx, by, residual, U's rows
    return (bidiag_threads(ORDER) / 32) * 2 * (nsz(ORDER) + 2) + (5 + kAdaptUrows) * nsz(ORDER) + 8;
}
// The links' coordinates and dot products take the place of V, which is used up by then.
template <int ORDER>
__host__ __device__ inline int adapt_doubles(int nplink) {
    const int mats = bidiag_doubles<ORDER>(), links = 5 * nplink;
    return (mats > links ? mats : links) + adapt_vectors<ORDER>();
}

// Blocks a SM that shared memory leaves room for; the registers are held to them.
__host__ __device__ constexpr int adapt_blocks(int order) { return order <= 6 ? 16 : order == 8 ? 9 : 5; }

// One node a block at a time.  Every length tried takes a factorisation: the block function
// above, then the QR iteration, whose scalars every warp carries along by itself (its own copy
// of the bidiagonal) while each thread turns one row of V, or of the four rows of U that the
// solves read.  One warp a node with all of U, V and the matrix in shared memory held four
// nodes a SM and took 1.5 ms a factorisation at order 8.
template <int ORDER>
__global__ void __launch_bounds__(bidiag_threads(ORDER), adapt_blocks(ORDER)) k_adapt_stencils(AdaptArgs a) {
    constexpr int n = nsz(ORDER), ld = n | 1, T = bidiag_threads(ORDER);
    static_assert(n + kAdaptUrows <= T, "a thread a row");
    extern __shared__ double smem[];
    __shared__ int sh_i, sh_cnt, sh_bad;
    __shared__ double sh_hc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto sync = [] {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    };
    double *V = smem;
    double *rv1 = smem + bidiag_doubles<ORDER>() - 2 * (n + 2), *W = rv1 + (n + 2);
    const int mats = bidiag_doubles<ORDER>(), links = 5 * a.nplink;
    double *vec = smem + (mats > links ? mats : links);
    double *Ws = vec + warp * 2 * (n + 2), *Rs = Ws + (n + 2);  // the warp's bidiagonal
    double *tmp = vec + (T / 32) * 2 * (n + 2), *bl = tmp + n, *bx = bl + n, *by = bx + n, *R = by + n, *Ur = R + n;
    double *lx = smem, *ly = lx + a.nplink, *dl = ly + a.nplink, *dxv = dl + a.nplink, *dyv = dxv + a.nplink;
    double *M = a.M + (size_t)blockIdx.x * 2 * n * n, *rows = M + n * n;
    const WArgs &wa = a.w;
    constexpr double amp_tol = 1.0001;
    constexpr int nk = 32;
    double *row = tid < n ? V + tid : Ur + (tid - n) * n;  // a row of V, or one of U's (0, 1, 2 and 4)
    const int step = tid < n ? ld : 1;
    const bool turns = tid < n + kAdaptUrows, on_u = tid >= n;
    // svdlib.F90:173-278; false where it does not converge (in every thread alike)
    auto qr = [&](double anorm) -> bool {
        for (int j = 1 + lane; j <= n; j += 32) { Ws[j] = W[j]; Rs[j] = rv1[j]; }
        __syncwarp();
        for (int k = n; k >= 1; k--) {
            for (int its = 1; its <= 30; its++) {
                bool to2000 = false;
                int l, nm = 1;
                for (l = k; l >= 1; l--) {
                    nm = l - 1;
                    if ((fabs(Rs[l]) + anorm) == anorm) { to2000 = true; break; }
                    if ((fabs(Ws[nm]) + anorm) == anorm) break;
                }
                if (l < 1) return false;  // only a NaN in the bidiagonal gets here
                double c, s, f, g, h, x, y, z;
                if (!to2000) {
                    c = 0.0; s = 1.0;
                    for (int i = l; i <= k; i++) {
                        const double r = Rs[i];
                        f = s * r;
                        __syncwarp();
                        if (lane == 0) Rs[i] = c * r;
                        if ((fabs(f) + anorm) == anorm) break;
                        g = Ws[i];
                        h = nr_hypot(f, g);
                        __syncwarp();
                        if (lane == 0) Ws[i] = h;
                        h = 1.0 / h;
                        c = (g * h);
                        s = -(f * h);
                        if (turns && on_u) {
                            const double yy = row[(nm - 1) * step], zz = row[(i - 1) * step];
                            row[(nm - 1) * step] = (yy * c) + (zz * s);
                            row[(i - 1) * step] = -(yy * s) + (zz * c);
                        }
                    }
                    __syncwarp();
                }
                z = Ws[k];
                if (l == k) {
                    if (z < 0.0) {
                        __syncwarp();
                        if (lane == 0) Ws[k] = -z;
                        if (turns && !on_u) row[(k - 1) * step] = -row[(k - 1) * step];
                    }
                    __syncwarp();
                    break;
                }
                if (its >= 30) return false;
                x = Ws[l];
                nm = k - 1;
                y = Ws[nm];
                g = Rs[nm];
                h = Rs[k];
                f = ((y - z) * (y + z) + (g - h) * (g + h)) / ((2.0 * h) * y);
                g = nr_hypot(f, 1.0);
                f = ((x - z) * (x + z) + h * ((y / (f + copysign(g, f))) - h)) / x;
                c = 1.0; s = 1.0;
                double xr = turns ? row[(l - 1) * step] : 0.0;  // the row's column j, on its way to column j + 1
                for (int j = l; j <= nm; j++) {
                    const int i = j + 1;
                    // entries j + 1 are read here and not written before the next j; a lane reads
                    // them before lane 0 gets there (the warp runs the scalars in step)
                    g = Rs[i];
                    y = Ws[i];
                    h = s * g;
                    g = c * g;
                    z = nr_hypot(f, h);
                    __syncwarp();
                    if (lane == 0) Rs[j] = z;
                    c = f / z;
                    s = h / z;
                    const double c1 = c, s1 = s;
                    f = (x * c) + (g * s);
                    g = -(x * s) + (g * c);
                    h = y * s;
                    y = y * c;
                    z = nr_hypot(f, h);
                    if (lane == 0) Ws[j] = z;
                    if (z != 0.0) {
                        z = 1.0 / z;
                        c = f * z;
                        s = h * z;
                    }
                    f = (c * g) + (s * y);
                    x = -(s * g) + (c * y);
                    if (turns) {
                        const double cr = on_u ? c : c1, sr = on_u ? s : s1;
                        const double zr = row[(i - 1) * step];
                        row[(j - 1) * step] = (xr * cr) + (zr * sr);
                        xr = -(xr * sr) + (zr * cr);
                    }
                }
                if (turns) row[(k - 1) * step] = xr;
                __syncwarp();
                if (lane == 0) {
                    Rs[l] = 0.0;
                    Rs[k] = f;
                    Ws[k] = x;
                }
                __syncwarp();
            }
        }
        return true;
    };
    for (;;) {
        sync();
        if (tid == 0) sh_i = atomicAdd(a.next, 1);
        sync();
        const int i = sh_i;
        if (i >= wa.npfb) return;
        const int t = wa.ntype[i];
        if (t <= 2 || t == 998) continue;
        const double xi = wa.px[i], yi = wa.py[i], si = a.sp[i];
        int c_all = wa.cnt[i], c_small = wa.cnt_small[i];
        double h_i = a.h[i], hs_i = a.hs[i];
        for (int pass = 0; pass < 2; pass++) {
            const double res_tol = a.res_tol[pass];
            for (int ii = 0;; ii++) {
                const double hh = (pass ? hs_i : h_i) * a.rf;
                const int cur = pass ? c_small : c_all;
                // leading links within hh * ss
                sync();
                if (tid == 0) { sh_cnt = cur; sh_bad = 0; }
                sync();
                for (int k = tid; k < cur; k += T) {
                    const int p = wa.lpt[sell_off(wa.slice_ptr, i, k)];
                    const double rx = xi - wa.px[p], ry = yi - wa.py[p];
                    if (!(sqrt(rx * rx + ry * ry) <= hh * kSs)) {
                        atomicMin(&sh_cnt, k);
                        break;
                    }
                }
                sync();
                const int cnt = sh_cnt;
                const double anorm = moment_bidiag<ORDER>(wa, i, cnt, hh, n, smem, W, rv1, M, rows, [&](const double *U) {
                    for (int e = tid; e < kAdaptUrows * n; e += T) {
                        const int r = e / n;
                        Ur[e] = U[(e - r * n) * ld + (r < 3 ? r : 4)];
                    }
                });
                sync();
                const double thr = res_tol / hh;
                double hc;
                if (!qr(anorm)) {
                    hc = (2.0 * res_tol) / hh;
                } else {
                    sync();  // every row is in place (and the matrix in memory)
                    const double v2 = (1.0 / hh) / hh, v1 = 1.0 / hh;
                    auto solve = [&](double *b, int r0, int r1, double v) {
                        if (tid < n) {
                            double sum = 0.0;
                            const double w = Ws[tid + 1];
                            if (w != 0.0) {
                                sum = sum + Ur[r0 * n + tid] * v;
                                if (r1 >= 0) sum = sum + Ur[r1 * n + tid] * v;
                                sum = sum / w;
                            }
                            tmp[tid] = sum;
                        }
                        sync();
                        if (tid < n) {
                            double sum = 0.0;
#pragma unroll 4
                            for (int jj = 0; jj < n; jj++) sum = sum + V[jj * ld + tid] * tmp[jj];
                            b[tid] = sum;
                        }
                        sync();
                    };
                    solve(bl, 2, 3, v2);  // rows 2 and 4 of U
                    solve(bx, 0, -1, v1);
                    solve(by, 1, -1, v1);
                    // residual of the Laplacian system, rows in parallel, sums in order
                    if (tid < n) {
                        double v = (tid == 2 || tid == 4) ? (-1.0 / hh) / hh : 0.0;
#pragma unroll 4
                        for (int c = 0; c < n; c++) v = v + M[c * n + tid] * bl[c];
                        R[tid] = v;
                    }
                    sync();
                    if (tid == 0) {
                        double q = 0.0;
                        for (int r = 0; r < n; r++) q = q + R[r] * R[r];
                        q = (q * hh) * hh;
                        sh_hc = sqrt(q / (double)n);
                    }
                    sync();
                    hc = sh_hc;
                    if (hc < thr) {
                        // each link's dot products with the three solutions (independent of q)
                        for (int k = tid; k < cnt; k += T) {
                            const int p = wa.lpt[sell_off(wa.slice_ptr, i, k)];
                            const double x = -(xi - wa.px[p]), y = -(yi - wa.py[p]);
                            const double qq = sqrt(x * x + y * y) / hh;
                            const double ff1 = wab(qq, wa.h2);
                            const double xx = x / hh, yy = y / hh;
                            double hx[ORDER + 1], hy[ORDER + 1];
#pragma unroll
                            for (int d = 0; d <= ORDER; d++) { hx[d] = hermite(d, xx); hy[d] = hermite(d, yy); }
                            double sl = 0.0, sx = 0.0, sy = 0.0;
#pragma unroll
                            for (int m = 0; m < n; m++) {
                                const int pm = p_of(m), qm = q_of(m);
                                const double g = ((qm == 0) ? hx[pm] : (pm == 0) ? hy[qm] : hx[pm] * hy[qm]) * ff1;
                                sl = sl + bl[m] * g;
                                sx = sx + bx[m] * g;
                                sy = sy + by[m] * g;
                            }
                            lx[k] = x; ly[k] = y; dl[k] = sl; dxv[k] = sx; dyv[k] = sy;
                        }
                        sync();
                        bool fail = false;
                        for (int i1 = tid + 1; i1 <= nk + 1; i1 += T) {
                            const double q = (((double)i1 * kPi) / si) / (double)nk;
                            double hl = 0.0, hx = 0.0, hy = 0.0;
                            for (int k = 0; k < cnt; k++) {
                                const double x = lx[k], y = ly[k];
                                hl = hl + (0.5 - (0.5 * cos(x * q)) * cos(y * q)) * dl[k];
                                hx = hx + (cos(y * q) * sin(x * q)) * dxv[k];
                                hy = hy + (cos(x * q) * sin(y * q)) * dyv[k];
                            }
                            hl = hl / (q * q);
                            hx = hx / q;
                            hy = hy / q;
                            if (hl > amp_tol || hl < 0.0 || fabs(hx) > amp_tol || fabs(hy) > amp_tol) fail = true;
                        }
                        if (fail) sh_bad = 1;
                        sync();
                        if (sh_bad) hc = (2.0 * res_tol) / hh;
                    }
                }
                if ((double)ii > a.limit) hc = (2.0 * res_tol) / hh;
                if (hc >= thr) break;  // a NaN residual compares false and is accepted, as in the reference
                if (pass == 0) {
                    h_i = hh;
                    hs_i = hh;
                    c_all = cnt;
                    c_small = cnt;
                } else {
                    hs_i = hh;
                    c_small = cnt;
                }
            }
        }
        if (tid == 0) {
            a.h[i] = h_i;
            a.hs[i] = hs_i;
        }
    }
}

// The largest dynamic shared memory a block may opt into on the handle's device (227 KB on B200):
// longer neighbour lists than fit there are refused by the adaptation.
int smem_optin(Handle *H, int *bytes) {
    SUNSET_CUDA(H, cudaDeviceGetAttribute(bytes, cudaDevAttrMaxSharedMemoryPerBlockOptin, H->device));
    return 0;
}

// Record entries an item gets.  The jittered sets take 0.36 n^2 (order 8, at most 0.41) to
// 0.78 n^2 (order 4, at most 0.96); what does not fit takes another round.
template <int ORDER>
constexpr int rec_capacity() { return nsz(ORDER) * nsz(ORDER) / 2 + 5 * nsz(ORDER) + 8; }
// Items a batch takes: enough for k_bidiag_qr's one thread an item to hide its latency (7 warps a
// SM), and 1.9 GB of workspace at order 8.
constexpr int kWeightBatch = 32768;

template <int ORDER>
int weights_batches(Handle *H, const WArgs &a, SvdBatch B, const int *items, int n_items, int pass) {
    constexpr int n = nsz(ORDER);
    cudaStream_t st = H->stream;
    const int maxits = a.maxits > 0 ? a.maxits : 30;
    constexpr size_t smem1 = bidiag_doubles<ORDER>() * sizeof(double);
    constexpr size_t smem2 = 2 * (size_t)(n + 1) * kQrThreads * sizeof(double);
    constexpr size_t smem3 = (size_t)kApplyWarps * apply_doubles<ORDER>() * sizeof(double);
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_moment_bidiag<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem1));
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_bidiag_qr<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2));
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_weights_apply<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem3));
    B.pass = pass;
    for (int b = 0; b < n_items; b += B.batch) {
        B.item = items + b;
        B.n_items = n_items - b < B.batch ? n_items - b : B.batch;
        k_moment_bidiag<ORDER><<<B.n_items, bidiag_threads(ORDER), smem1, st>>>(a, B);
        int left = 1;
        // every round takes each item that is left at least one sweep further
        while (left > 0) {
            SUNSET_CUDA(H, cudaMemsetAsync(B.left, 0, sizeof(int), st));
            k_bidiag_qr<ORDER><<<(B.n_items + kQrThreads - 1) / kQrThreads, kQrThreads, smem2, st>>>(B, maxits);
            k_weights_apply<ORDER><<<(B.n_items + kApplyWarps - 1) / kApplyWarps, kApplyWarps * 32, smem3, st>>>(a, B);
            SUNSET_CUDA(H, cudaGetLastError());
            SUNSET_CUDA(H, cudaMemcpyAsync(&left, B.left, sizeof(int), cudaMemcpyDeviceToHost, st));
            SUNSET_CUDA(H, cudaStreamSynchronize(st));
        }
    }
    return 0;
}

template <int ORDER>
int launch_weights(Handle *H, WArgs &a) {
    constexpr int n = nsz(ORDER);
    cudaStream_t st = H->stream;
    SvdBatch B{};
    B.cap = rec_capacity<ORDER>();
    int *items = nullptr, *count = nullptr;
    char *ws = nullptr;
    if (dalloc(H, &items, 2 * (size_t)a.npfb) || dalloc(H, &count, 4)) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(count, 0, 4 * sizeof(int), st));
    k_weight_items<<<(a.npfb + 255) / 256, 256, 0, st>>>(a, items, items + a.npfb, count);
    int hc[2] = {0, 0};
    SUNSET_CUDA(H, cudaMemcpyAsync(hc, count, sizeof(hc), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    // the workspace, in halves of the batch where memory is short
    B.batch = hc[0] < kWeightBatch ? (hc[0] + 31) / 32 * 32 : kWeightBatch;
    for (; B.batch > 0; B.batch = B.batch / 64 * 32) {
        const size_t per = sizeof(double) * ((size_t)4 * B.cap + (kUrows + n) * n + 2 * (n + 1) + 1) + sizeof(int2) + sizeof(int);
        ws = static_cast<char *>(H->mem.take(per * B.batch));
        if (ws) break;
    }
    if (hc[0] > 0 && !ws) return set_err(H, SUNSET_ERR_NOMEM, "no memory for the weight solves");
    int rc = 0;
    if (ws) {
        char *p = ws;
        auto take = [&](size_t bytes) { char *q = p; p += bytes; return q; };
        const size_t nb = B.batch;
        B.rec = reinterpret_cast<double4 *>(take(nb * B.cap * sizeof(double4)));
        B.V = reinterpret_cast<double *>(take(nb * n * n * sizeof(double)));
        B.U = reinterpret_cast<double *>(take(nb * kUrows * n * sizeof(double)));
        B.W = reinterpret_cast<double *>(take(nb * (n + 1) * sizeof(double)));
        B.rv1 = reinterpret_cast<double *>(take(nb * (n + 1) * sizeof(double)));
        B.anorm = reinterpret_cast<double *>(take(nb * sizeof(double)));
        B.state = reinterpret_cast<int2 *>(take(nb * sizeof(int2)));
        B.nrec = reinterpret_cast<int *>(take(nb * sizeof(int)));
        B.left = count + 2;
        rc = weights_batches<ORDER>(H, a, B, items, hc[0], 0);
        if (!rc && hc[1] > 0) rc = weights_batches<ORDER>(H, a, B, items + a.npfb, hc[1], 1);
        dfree(H, ws);
    }
    dfree(H, items);
    dfree(H, count);
    return rc;
}


}  // namespace

template <int ORDER>
int launch_adapt(Handle *H, AdaptArgs &a) {
    constexpr int n = nsz(ORDER), T = bidiag_threads(ORDER);
    const size_t smem = (size_t)adapt_doubles<ORDER>(a.nplink) * sizeof(double);
    int optin = 0, nsm = 0, per_sm = 0;
    if (int rc = smem_optin(H, &optin)) return rc;
    const int most = optin - 1024;  // the kernel's static part beside it
    if (smem > (size_t)most) return set_err(H, SUNSET_ERR_SCOPE, "neighbour lists too long for the stencil adaptation");
    // the limit is the process's, so it does not follow this handle's lists (setup.cu, build_halos)
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_adapt_stencils<ORDER>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    SUNSET_CUDA(H, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, H->device));
    SUNSET_CUDA(H, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_adapt_stencils<ORDER>, T, smem));
    const int nb = std::max(1, std::min(a.w.npfb, nsm * std::max(1, per_sm)));  // each takes one node after another
    if (dalloc(H, &a.M, (size_t)nb * 2 * n * n) || dalloc(H, &a.next, 1)) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(a.next, 0, sizeof(int), H->stream));
    k_adapt_stencils<ORDER><<<nb, T, smem, H->stream>>>(a);
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    dfree(H, a.M);
    dfree(H, a.next);
    return 0;
}

// The residual tolerance of the adaptation, labf.F90:1126-1139 (Hermite ABFs).
static double adapt_res_tol(int order) {
    const int n = (order * order + 3 * order) / 2;
    const double c = order == 4 ? 1.0e-3 : order == 6 ? 5.0e-3 : order == 8 ? 3.0e-2 : 1.0;
    return ((c * (double)(n * n * n * n)) * 2.220446049250313080847e-16) / (double)order;
}

int adapt_stencils_device(Handle *H) {
    if (H->cfg.forder != H->cfg.morder)
        return set_err(H, SUNSET_ERR_SCOPE, "the device stencil adaptation requires forder == morder");
    AdaptArgs a{};
    a.w = WArgs{H->npfb, H->cfg.morder, H->cfg.forder, H->h2, H->px, H->py, H->h, H->hs, H->ntype, H->cnt,
                H->cnt_small, H->lpt, H->slice_ptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    a.h = H->h;
    a.hs = H->hs;
    a.sp = H->sp;
    a.nplink = H->nplink;
    a.rf = (double)0.98f;                          // reduction_factor = 0.98, a default-real literal
    a.limit = (double)logf(0.6f) / log(a.rf);      // log(0.6) of a default-real literal
    a.res_tol[0] = adapt_res_tol(H->cfg.forder);  // adapt_stencils
    a.res_tol[1] = adapt_res_tol(H->cfg.morder);  // adapt_stencils_main
    int rc;
    switch (H->cfg.morder) {
    case 4: rc = launch_adapt<4>(H, a); break;
    case 6: rc = launch_adapt<6>(H, a); break;
    case 8: rc = launch_adapt<8>(H, a); break;
    case 10: rc = launch_adapt<10>(H, a); break;
    default: return set_err(H, SUNSET_ERR_SCOPE, "order %d", H->cfg.morder);
    }
    if (rc) return rc;
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    return 0;
}

// Condition numbers of the moment matrices the weight build factored: the worst one and the
// number of nodes above the limit (the configured cond_max, else kCondWarn), kept in the
// handle.  With cond_max > 0 such a node is an error; without, it is only counted.
int conditioning_check(Handle *H) {
    const int n = H->npfb;
    std::vector<double> cd(n), cf(n);
    SUNSET_CUDA(H, cudaMemcpyAsync(cd.data(), H->cond_d, n * sizeof(double), cudaMemcpyDeviceToHost, H->stream));
    SUNSET_CUDA(H, cudaMemcpyAsync(cf.data(), H->cond_f, n * sizeof(double), cudaMemcpyDeviceToHost, H->stream));
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    const double lim = H->cfg.cond_max > 0.0 ? H->cfg.cond_max : kCondWarn;
    double worst = 0.0;
    int nill = 0, iworst = -1;
    for (int i = 0; i < n; i++) {
        const double c = cd[i] > cf[i] ? cd[i] : cf[i];
        if (c > lim) nill++;
        if (c > worst || (std::isinf(c) && iworst < 0)) { worst = c; iworst = i; }
    }
    H->cond_worst = worst;
    H->cond_nill = nill;
    H->cond_ok = true;
    if (H->cfg.cond_max > 0.0 && nill > 0)
        return set_err(H, SUNSET_ERR_ILLCOND,
                       "%d nodes have moment matrices with condition number above %g (worst %.3g at reference node %d)",
                       nill, lim, worst, iworst >= 0 ? H->h_perm[iworst] : -1);
    return 0;
}

int labf_weights_device(Handle *H) {
    const int n = H->npfb;
    if (H->cfg.forder != H->cfg.morder)
        return set_err(H, SUNSET_ERR_SCOPE, "the device weight build requires forder == morder");
    if (!H->wx) {
        if (dalloc(H, &H->wx, H->nlinks_sell) || dalloc(H, &H->wy, H->nlinks_sell) ||
            dalloc(H, &H->wl, H->nlinks_sell) || dalloc(H, &H->wh, H->nlinks_sell) || dalloc(H, &H->gsx, n) ||
            dalloc(H, &H->gsy, n) || dalloc(H, &H->lsum, n) || dalloc(H, &H->hsum, n) || dalloc(H, &H->vol, n))
            return SUNSET_ERR_NOMEM;
    }
    cudaStream_t st = H->stream;
    SUNSET_CUDA(H, cudaMemsetAsync(H->wx, 0, H->nlinks_sell * sizeof(double), st));
    SUNSET_CUDA(H, cudaMemsetAsync(H->wy, 0, H->nlinks_sell * sizeof(double), st));
    SUNSET_CUDA(H, cudaMemsetAsync(H->wl, 0, H->nlinks_sell * sizeof(double), st));
    SUNSET_CUDA(H, cudaMemsetAsync(H->wh, 0, H->nlinks_sell * sizeof(double), st));
    int *derr;
    if (dalloc(H, &derr, 1)) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(derr, 0, sizeof(int), st));
    if (!H->cond_d && (dalloc(H, &H->cond_d, n) || dalloc(H, &H->cond_f, n))) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(H->cond_d, 0, n * sizeof(double), st));
    SUNSET_CUDA(H, cudaMemsetAsync(H->cond_f, 0, n * sizeof(double), st));
    WArgs a{n, H->cfg.morder, H->cfg.forder, H->h2, H->px, H->py, H->h, H->hs, H->ntype, H->cnt, H->cnt_small,
            H->lpt, H->slice_ptr, H->wx, H->wy, H->wl, H->wh, derr, H->cfg.svd_max_sweeps, H->cond_d, H->cond_f};
    int rc;
    switch (H->cfg.morder) {
    case 4: rc = launch_weights<4>(H, a); break;
    case 6: rc = launch_weights<6>(H, a); break;
    case 8: rc = launch_weights<8>(H, a); break;
    case 10: rc = launch_weights<10>(H, a); break;
    default: return set_err(H, SUNSET_ERR_ARG, "order must be 4, 6, 8 or 10");
    }
    if (rc) return rc;
    int herr = 0;
    SUNSET_CUDA(H, cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    dfree(H, derr);
    if (herr) return set_err(H, SUNSET_ERR_SVD, "SVD not converging at internal node %d (svdlib.F90:219-222)", herr - 1);
    return conditioning_check(H);
}

int boundary_prune_links(Handle *H);

// calc_boundary_weights (labf.F90:505-1039); the links of the boundary nodes are pruned by
// boundary_prune_links() first.
int boundary_weights_device(Handle *H) {
    if (H->nb == 0) return 0;
    const int nb = H->nb;
    if (!H->wb2 && dalloc(H, &H->wb2, (size_t)nb * H->nplink * 2)) return SUNSET_ERR_NOMEM;
    int *derr;
    if (dalloc(H, &derr, 1)) return SUNSET_ERR_NOMEM;
    cudaStream_t st = H->stream;
    SUNSET_CUDA(H, cudaMemsetAsync(derr, 0, sizeof(int), st));
    BndArgs a{H->npfb, nb, H->nplink, H->h3, H->px, H->py, H->h, H->sp, H->rnx, H->rny, H->ntype, H->gpar,
              H->fdpar, H->blist, H->brow, H->cnt, H->cnt_small, H->lpt, H->lidx, H->lloc, H->slice_ptr,
              H->slice_w, H->wx, H->wy, H->wl, H->wh, H->wb2, derr};
    k_boundary_node_weights<<<(nb + 3) / 4, 128, 0, st>>>(a);
    k_boundary_row_weights<<<(2 * nb + 3) / 4, 128, 0, st>>>(a);
    k_boundary_frame<<<(nb + 127) / 128, 128, 0, st>>>(a);
    SUNSET_CUDA(H, cudaGetLastError());
    int herr = 0;
    SUNSET_CUDA(H, cudaMemcpyAsync(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    dfree(H, derr);
    if (herr) return set_err(H, SUNSET_ERR_SVD, "SVD not converging at boundary node or row %d", herr - 1);
    return 0;
}

int boundary_prune_links(Handle *H) {
    if (H->nb == 0) return 0;
    BndArgs a{H->npfb, H->nb, H->nplink, H->h3, H->px, H->py, H->h, H->sp, H->rnx, H->rny, H->ntype, H->gpar,
              H->fdpar, H->blist, H->brow, H->cnt, H->cnt_small, H->lpt, H->lidx, H->lloc, H->slice_ptr,
              H->slice_w, H->wx, H->wy, H->wl, H->wh, H->wb2, nullptr};
    k_prune_boundary_links<<<(H->nb + 127) / 128, 128, 0, H->stream>>>(a);
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    return 0;
}

// The tangential second-derivative weights of boundary nodes scaled by 1/L^2 and their sums
// over all links (calc_labf_sums, labf.F90:426-446): the transverse Laplacian of the
// conformation tensor on walls (derivatives.F90:306-358).  One thread per boundary node.
__global__ void k_boundary_tangential_sums(int nb, int nplink, double L, const int *blist, const int *cnt,
                                           const double *wb2, double *wbt, double *wbt_sum) {
    const int jj = blockIdx.x * blockDim.x + threadIdx.x;
    if (jj >= nb) return;
    const double *w = wb2 + (size_t)jj * nplink * 2;
    double sum = 0.0;
    for (int k = 0; k < cnt[blist[jj]]; k++) sum = sum + w[2 * k + 1];
    wbt_sum[jj] = (sum / L) / L;
    for (int k = 0; k < nplink; k++) wbt[(size_t)jj * nplink + k] = (w[2 * k + 1] / L) / L;
}

int labf_sums_device(Handle *H) {
    SumArgs a{H->npfb, H->cfg.L_char, H->px, H->py, H->h, H->sp, H->ntype, H->cnt, H->lpt, H->fdpar, H->slice_ptr,
              H->wx, H->wy, H->wl, H->wh, H->gsx, H->gsy, H->lsum, H->hsum, H->vol};
    k_labf_sums<<<(H->npfb + 255) / 256, 256, 0, H->stream>>>(a);
    if (H->nb > 0) {
        if (!H->wbt && (dalloc(H, &H->wbt, (size_t)H->nb * H->nplink) || dalloc(H, &H->wbt_sum, H->nb)))
            return SUNSET_ERR_NOMEM;
        k_boundary_tangential_sums<<<(H->nb + 127) / 128, 128, 0, H->stream>>>(H->nb, H->nplink, H->cfg.L_char, H->blist,
                                                                             H->cnt, H->wb2, H->wbt, H->wbt_sum);
    }
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    return 0;
}

int filter_coefficients_device(Handle *H) {
    SumArgs a{H->npfb, H->cfg.L_char, H->px, H->py, H->h, H->sp, H->ntype, H->cnt, H->lpt, H->fdpar, H->slice_ptr,
              H->wx, H->wy, H->wl, H->wh, H->gsx, H->gsy, H->lsum, H->hsum, H->vol};
    k_filter_coeff<<<(H->npfb + 255) / 256, 256, 0, H->stream>>>(a);
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    return 0;
}

}  // namespace sunset
