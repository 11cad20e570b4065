// setup.cu -- device-resident domain: ghost points, Morton renumbering, cell-list neighbour
// search and per-row distance sort (neighbours.F90, mirror_boundaries.F90).
//
// Compiled with -fmad=false: ghost positions and squared distances are formed with the
// same operations, in the same order, as the reference, so the neighbour sets and the
// distance order match it exactly.
#include <algorithm>

#include <cub/cub.cuh>

#include "internal.cuh"

namespace sunset {

namespace {

// ---------------------------------------------------------------------------------------
// Mirror (ghost) points, mirror_boundaries.F90:34-261.  One pass counts each node's
// mirrors, a scan gives offsets in reference node order, a second pass writes them, so
// the ghost numbering equals the reference's (npfb+1, npfb+2, ... in node order).
// ---------------------------------------------------------------------------------------
struct MirrorArgs {
    const double *x, *y, *h;
    int n;
    double xmin, xmax, ymin, ymax;
    int xL, xU, yL, yU;
};

template <bool WRITE>
__device__ int mirrors_of(const MirrorArgs &a, int i, double *gx, double *gy, int *gpar, int *gvrel) {
    const double xi = a.x[i], yi = a.y[i];
    const double lim = (kSs * a.h[i]) * 2.0;  // ss*h(i)*mlayer_buff
    int m = 0;
    auto emit = [&](int vrel, double xn, double yn) {
        if (WRITE) { gx[m] = xn; gy[m] = yn; gpar[m] = i; gvrel[m] = vrel; }
        m++;
    };
    if (xi <= a.xmin + lim) {
        if (a.xL == 1) emit(1, (xi + a.xmax) - a.xmin, yi);
        else if (a.xL == 2) emit(2, 2.0 * a.xmin - xi, yi);
    }
    if (xi >= a.xmax - lim) {
        if (a.xU == 1) emit(1, (xi - a.xmax) + a.xmin, yi);
        else if (a.xU == 2) emit(2, 2.0 * a.xmax - xi, yi);
    }
    if (yi <= a.ymin + lim) {
        if (a.yL == 1) emit(1, xi, (yi + a.ymax) - a.ymin);
        else if (a.yL == 2) emit(3, xi, 2.0 * a.ymin - yi);
        else if (a.yL == 3) emit(4, xi, 2.0 * a.ymin - yi);
    }
    if (yi >= a.ymax - lim) {
        if (a.yU == 1) emit(1, xi, (yi - a.ymax) + a.ymin);
        else if (a.yU == 2) emit(3, xi, 2.0 * a.ymax - yi);
        else if (a.yU == 3) emit(4, xi, 2.0 * a.ymax - yi);
    }
    const double cx[4] = {a.xmin, a.xmax, a.xmin, a.xmax}, cy[4] = {a.ymin, a.ymin, a.ymax, a.ymax};
    const int bx[4] = {a.xL, a.xU, a.xL, a.xU}, by[4] = {a.yL, a.yL, a.yU, a.yU};
    for (int c = 0; c < 4; c++) {
        double dx = cx[c] - xi, dy = cy[c] - yi, dz = 0.0 - 0.0;
        double cdist = sqrt((dx * dx + dy * dy) + dz * dz);
        if (cdist <= lim && bx[c] != 0 && by[c] != 0) {
            bool right = (c == 1 || c == 3), top = (c == 2 || c == 3);
            double xp = right ? (xi - a.xmax) + a.xmin : (xi + a.xmax) - a.xmin;
            double yp = top ? (yi - a.ymax) + a.ymin : (yi + a.ymax) - a.ymin;
            double xs = right ? 2.0 * a.xmax - xi : 2.0 * a.xmin - xi;
            double ys = top ? 2.0 * a.ymax - yi : 2.0 * a.ymin - yi;
            if (bx[c] == 1 && by[c] == 1) emit(1, xp, yp);
            else if (bx[c] == 2 && by[c] == 1) emit(2, xs, yp);
            else if (bx[c] == 1 && by[c] == 2) emit(3, xp, ys);
            else if (bx[c] == 2 && by[c] == 2) emit(4, xs, ys);
            else emit(-1, xi, yi);  // undefined in the reference (host rejects it)
        }
    }
    return m;
}

__global__ void k_count_mirrors(MirrorArgs a, int *count) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.n) count[i] = mirrors_of<false>(a, i, nullptr, nullptr, nullptr, nullptr);
}

__global__ void k_write_mirrors(MirrorArgs a, const int *offset, double *gx, double *gy, int *gpar_ref,
                                int *gvrel) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    int o = offset[i];
    mirrors_of<true>(a, i, gx + o, gy + o, gpar_ref + o, gvrel + o);
}

__device__ __forceinline__ uint32_t spread16(uint32_t v) {
    v &= 0xffff;
    v = (v | (v << 8)) & 0x00ff00ff;
    v = (v | (v << 4)) & 0x0f0f0f0f;
    v = (v | (v << 2)) & 0x33333333;
    v = (v | (v << 1)) & 0x55555555;
    return v;
}

__global__ void k_morton(const double *x, const double *y, int n, double x0, double y0, double inv_dx,
                         double inv_dy, uint32_t *key, int *val) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double fx = (x[i] - x0) * inv_dx, fy = (y[i] - y0) * inv_dy;
    uint32_t qx = (uint32_t)fmin(fmax(fx, 0.0), 65535.0);
    uint32_t qy = (uint32_t)fmin(fmax(fy, 0.0), 65535.0);
    key[i] = spread16(qx) | (spread16(qy) << 1);
    val[i] = i;
}

__global__ void k_gather_nodes(int n, const int *perm, const double *x, const double *y, const double *h,
                               const double *hs, const double *s, const int *type, double *px, double *py,
                               double *ho, double *hso, double *so, int *to, int *iperm) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int r = perm[i];
    px[i] = x[r]; py[i] = y[r]; ho[i] = h[r]; hso[i] = hs[r]; so[i] = s[r]; to[i] = type[r];
    iperm[r] = i;
}

__global__ void k_place_ghosts(int ng, int npfb, const double *gx, const double *gy, const int *gpar_ref,
                               const int *iperm, double *px, double *py, int *gpar) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ng) return;
    px[npfb + g] = gx[g];
    py[npfb + g] = gy[g];
    gpar[g] = iperm[gpar_ref[g]];
}

// ---------------------------------------------------------------------------------------
// Cell list over all points (interior + ghosts) and the per-node search,
// neighbours.F90:160-270.  The cell side is ss*max(h), so the 3x3 block of cells around
// a node covers its support.
// ---------------------------------------------------------------------------------------
struct Grid {
    double x0, y0, inv;
    int ncx, ncy;
};

__global__ void k_cell_id(const double *px, const double *py, int np, Grid g, int *cid, int *pid) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    int cx = (int)((px[p] - g.x0) * g.inv), cy = (int)((py[p] - g.y0) * g.inv);
    cx = min(max(cx, 0), g.ncx - 1);
    cy = min(max(cy, 0), g.ncy - 1);
    cid[p] = cx + g.ncx * cy;
    pid[p] = p;
}

__global__ void k_cell_bounds(const int *cid_sorted, int np, int *cstart, int *cend) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    int c = cid_sorted[p];
    if (p == 0 || cid_sorted[p - 1] != c) cstart[c] = p;
    if (p == np - 1 || cid_sorted[p + 1] != c) cend[c] = p + 1;
}

// The reference's search grid (cell_generator, neighbours.F90:75-93): square cells of side
// ss*h0 over the domain tripled in each direction.
struct RefGrid {
    double xmint, ymint, unoss;
};

struct SearchArgs {
    const double *px, *py, *h;
    const int *cstart, *cend, *pts;
    Grid g;
    RefGrid rg;
    int npfb;
};

template <bool FILL>
__global__ void k_search(SearchArgs a, int *count, const long long *rowptr, int *opt, double *or2) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.npfb) return;
    const double xi = a.px[i], yi = a.py[i];
    const double hh = a.h[i] * kSs, hs2 = hh * hh;
    int cx = min(max((int)((xi - a.g.x0) * a.g.inv), 0), a.g.ncx - 1);
    int cy = min(max((int)((yi - a.g.y0) * a.g.inv), 0), a.g.ncy - 1);
    // the reference scans only the 3x3 block of its own cells around the node
    // (neighbour_cells, neighbours.F90:95-158), so where a node's ss*h exceeds the cell side
    // ss*h0 (boundary nodes at order 4: hovs_bound > hovs) the points further out are not its
    // neighbours even inside the radius
    const int ci = (int)((xi - a.rg.xmint) * a.rg.unoss), cj = (int)((yi - a.rg.ymint) * a.rg.unoss);
    long long o = FILL ? rowptr[i] : 0;
    int cnt = 0;
    for (int dy = -1; dy <= 1; dy++) {
        int yy = cy + dy;
        if (yy < 0 || yy >= a.g.ncy) continue;
        for (int dx = -1; dx <= 1; dx++) {
            int xx = cx + dx;
            if (xx < 0 || xx >= a.g.ncx) continue;
            int c = xx + a.g.ncx * yy;
            int e = a.cend[c];
            for (int q = a.cstart[c]; q < e; q++) {
                int p = a.pts[q];
                double rx = xi - a.px[p], ry = yi - a.py[p], rz = 0.0 - 0.0;
                double rr2 = (rx * rx + ry * ry) + rz * rz;
                if (rr2 <= hs2) {
                    const int dcx = (int)((a.px[p] - a.rg.xmint) * a.rg.unoss) - ci;
                    const int dcy = (int)((a.py[p] - a.rg.ymint) * a.rg.unoss) - cj;
                    if (dcx < -1 || dcx > 1 || dcy < -1 || dcy > 1) continue;
                    if (FILL) { opt[o + cnt] = p; or2[o + cnt] = rr2; }
                    cnt++;
                }
            }
        }
    }
    if (!FILL) count[i] = cnt;
}

// Reference numbering of a point, used to order links at equal distance deterministically.
__device__ __forceinline__ int ref_point(int p, int npfb, const int *perm) { return p < npfb ? perm[p] : p; }

// Position of the cell (dx, dy) relative to a node's own cell in the reference's scan of the
// neighbouring cells (neighbour_cells, neighbours.F90:95-158): self, E, NE, SE, W, NW, SW, N, S.
__device__ __forceinline__ int scan_position(int dx, int dy) {
    if (dx == 0 && dy == 0) return 0;
    if (dx == 1) return dy == 0 ? 1 : dy == 1 ? 2 : 3;
    if (dx == -1) return dy == 0 ? 4 : dy == 1 ? 5 : 6;
    return dy == 1 ? 7 : 8;
}

constexpr int kMaxRowSort = 1024;  // longest row the reference-order sort accepts
constexpr int kSortWarps = 4;

// order_neighbours (neighbours.F90:272-341), reproducing where links at exactly equal
// distance end up (straight walls, FD rows and their periodic images give such ties): the
// row is first put in the order in which the reference's cell scan finds the links (scan
// position of the link's cell, then point number within a cell, as divide() fills the
// cells), then sorted by squared distance with the reference's quicksort
// (quicksort_neighbours), run with an explicit stack.  ij_count_small counts the links
// inside ss*h_small.
//
// A warp a row, in shared memory: each link's place is the number of nearer links.  Only a row
// with equal distances needs the reference's own order: it goes through the scan order and the
// quicksort, on one lane.  (One thread a row in global memory took 19.6 ms for 262,144 rows of
// 92 links.)
__global__ void __launch_bounds__(kSortWarps * 32) k_sort_rows(int npfb, const long long *rowptr, int width, int *opt,
                                                               const double *or2, const double *hs, const int *perm,
                                                               const double *px, const double *py, RefGrid rg, int *cnt_small,
                                                               int *err) {
    extern __shared__ __align__(16) double ssm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kSortWarps + warp;
    if (i >= npfb) return;
    const long long b = rowptr[i];
    const int n = (int)(rowptr[i + 1] - b);
    if (n > kMaxRowSort) {
        if (lane == 0) atomicExch(err, i + 1);
        return;
    }
    double *r2 = ssm + (size_t)warp * width * 2;
    long long *key = reinterpret_cast<long long *>(r2 + width);
    int *pt = reinterpret_cast<int *>(ssm + (size_t)kSortWarps * width * 2) + (size_t)warp * width;
    const double t = hs[i] * kSs, hs2 = t * t;
    int small = 0;
    for (int k = lane; k < n; k += 32) {
        r2[k] = or2[b + k];
        pt[k] = opt[b + k];
        small += r2[k] <= hs2;
    }
    for (int o = 16; o > 0; o >>= 1) small += __shfl_down_sync(0xffffffffu, small, o);
    if (lane == 0) cnt_small[i] = small;
    __syncwarp();
    bool tie = false;
    for (int k = lane; k < n; k += 32) {
        const double x = r2[k];
        int rank = 0, same = 0;
        for (int j = 0; j < n; j++) {
            const double y = r2[j];
            rank += y < x;
            same += y == x;
        }
        opt[b + rank] = pt[k];  // read in full above; a tie writes the row again
        tie = tie || same != 1;
    }
    if (!__any_sync(0xffffffffu, tie)) return;
    // the reference's order: scan order, then its quicksort
    const int ci = (int)((px[i] - rg.xmint) * rg.unoss), cj = (int)((py[i] - rg.ymint) * rg.unoss);
    for (int k = lane; k < n; k += 32) {
        const int p = pt[k];
        int dx = (int)((px[p] - rg.xmint) * rg.unoss) - ci, dy = (int)((py[p] - rg.ymint) * rg.unoss) - cj;
        // (k_search keeps no link beyond the 3x3 cells; such a link would go last)
        int pos = (dx < -1 || dx > 1 || dy < -1 || dy > 1) ? 9 : scan_position(dx, dy);
        key[k] = ((long long)pos << 32) | (unsigned)ref_point(p, npfb, perm);
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {  // the points' numbers are distinct, so every place is taken once
        const long long x = key[k];
        int rank = 0;
        for (int j = 0; j < n; j++) rank += key[j] < x;
        opt[b + rank] = k;
    }
    __syncwarp();
    // the row in scan order: the keys are no longer needed, their place takes the distances
    double *a = reinterpret_cast<double *>(key);
    for (int k = lane; k < n; k += 32) a[k] = r2[opt[b + k]];
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
        const int q = opt[b + k];
        opt[b + k] = pt[q];
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) pt[k] = opt[b + k];
    __syncwarp();
    if (lane == 0) {
        // quicksort_neighbours on the 1-based range [1, n] of this row
        double *ar = a - 1;
        int *lk = pt - 1;
        int stk[2 * 64];
        int top = 0;
        if (n >= 1) { stk[0] = 1; stk[1] = n; top = 1; }
        while (top > 0) {
            top--;
            const int first = stk[2 * top], last = stk[2 * top + 1];
            const double x = ar[(first + last) / 2];
            int ii = first, jj = last;
            for (;;) {
                while (ar[ii] < x) ii++;
                while (x < ar[jj]) jj--;
                if (ii >= jj) break;
                double td = ar[ii]; ar[ii] = ar[jj]; ar[jj] = td;
                int it = lk[ii]; lk[ii] = lk[jj]; lk[jj] = it;
                ii++;
                jj--;
            }
            if (top + 2 > 64) {  // deeper than any row of kMaxRowSort links needs in practice
                atomicExch(err, i + 1);
                break;
            }
            if (first < ii - 1) { stk[2 * top] = first; stk[2 * top + 1] = ii - 1; top++; }
            if (jj + 1 < last) { stk[2 * top] = jj + 1; stk[2 * top + 1] = last; top++; }
        }
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) opt[b + k] = pt[k];
}

__global__ void k_fill_sell(int npfb, int nslices, const long long *rowptr, const int *opt,
                            const long long *slice_ptr, const int *slice_w, const int *gpar,
                            const int *gvrel, int *lpt, int *lidx, int *mirror_flag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int sl = i >> 5;
    if (sl >= nslices) return;
    int lane = i & 31;
    long long base = slice_ptr[sl];
    int w = slice_w[sl];
    long long b = i < npfb ? rowptr[i] : 0;
    int cnt = i < npfb ? (int)(rowptr[i + 1] - b) : 0;
    for (int k = 0; k < w; k++) {
        long long o = sell_at(base, k, lane);
        if (k < cnt) {
            int p = opt[b + k];
            lpt[o] = p;
            if (p < npfb) {
                lidx[o] = p;
            } else {
                int g = p - npfb;
                int code = gvrel[g] - 1;
                lidx[o] = gpar[g] | (code << 30);
                if (code != 0) *mirror_flag = 1;
            }
        } else {
            lpt[o] = -1;
            lidx[o] = 0;
        }
    }
}

}  // namespace

// ---------------------------------------------------------------------------------------
int build_domain_device(Handle *H, const std::vector<double> &x, const std::vector<double> &y,
                        const std::vector<double> &h, const std::vector<double> &hs,
                        const std::vector<double> &s, const std::vector<int> &type) {
    const int n = H->npfb;
    cudaStream_t st = H->stream;
    double *dx, *dy, *dh, *dhs, *ds;
    int *dt;
    if (dalloc(H, &dx, n) || dalloc(H, &dy, n) || dalloc(H, &dh, n) || dalloc(H, &dhs, n) ||
        dalloc(H, &ds, n) || dalloc(H, &dt, n))
        return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemcpyAsync(dx, x.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(dy, y.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(dh, h.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(dhs, hs.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(ds, s.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(dt, type.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));

    // mirrors
    MirrorArgs ma{dx, dy, dh, n, H->xmin, H->xmax, H->ymin, H->ymax, H->bc[0], H->bc[1], H->bc[2], H->bc[3]};
    int *mcount, *moff;
    if (dalloc(H, &mcount, n + 1) || dalloc(H, &moff, n + 1)) return SUNSET_ERR_NOMEM;
    const int TB = 256;
    k_count_mirrors<<<(n + TB - 1) / TB, TB, 0, st>>>(ma, mcount);
    SUNSET_CUDA(H, cudaMemsetAsync(mcount + n, 0, sizeof(int), st));
    size_t tmpb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmpb, mcount, moff, n + 1, st);
    void *tmp;
    if (dalloc(H, (char **)&tmp, tmpb)) return SUNSET_ERR_NOMEM;
    cub::DeviceScan::ExclusiveSum(tmp, tmpb, mcount, moff, n + 1, st);
    dfree(H, tmp);
    int ng = 0;
    SUNSET_CUDA(H, cudaMemcpyAsync(&ng, moff + n, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    H->nghost = ng;
    H->np = n + ng;
    double *gx, *gy;
    int *gpar_ref;
    if (dalloc(H, &gx, ng) || dalloc(H, &gy, ng) || dalloc(H, &gpar_ref, ng) || dalloc(H, &H->gvrel, ng) ||
        dalloc(H, &H->gpar, ng))
        return SUNSET_ERR_NOMEM;
    k_write_mirrors<<<(n + TB - 1) / TB, TB, 0, st>>>(ma, moff, gx, gy, gpar_ref, H->gvrel);
    {
        std::vector<int> vr(ng);
        SUNSET_CUDA(H, cudaMemcpyAsync(vr.data(), H->gvrel, ng * sizeof(int), cudaMemcpyDeviceToHost, st));
        SUNSET_CUDA(H, cudaStreamSynchronize(st));
        for (int v : vr)
            if (v < 0) return set_err(H, SUNSET_ERR_SCOPE, "corner mirror for this bcond combination is undefined in the reference");
    }

    // Morton renumbering of the interior nodes
    uint32_t *key, *key2;
    int *val, *val2;
    if (dalloc(H, &key, n) || dalloc(H, &key2, n) || dalloc(H, &val, n) || dalloc(H, &val2, n)) return SUNSET_ERR_NOMEM;
    double Lx = H->xmax - H->xmin, Ly = H->ymax - H->ymin;
    k_morton<<<(n + TB - 1) / TB, TB, 0, st>>>(dx, dy, n, H->xmin, H->ymin, 65535.0 / Lx, 65535.0 / Ly, key, val);
    tmpb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmpb, key, key2, val, val2, n, 0, 32, st);
    if (dalloc(H, (char **)&tmp, tmpb)) return SUNSET_ERR_NOMEM;
    cub::DeviceRadixSort::SortPairs(tmp, tmpb, key, key2, val, val2, n, 0, 32, st);
    dfree(H, tmp);
    if (dalloc(H, &H->perm, n) || dalloc(H, &H->iperm, n) || dalloc(H, &H->px, H->np) ||
        dalloc(H, &H->py, H->np) || dalloc(H, &H->h, n) || dalloc(H, &H->hs, n) || dalloc(H, &H->sp, n) ||
        dalloc(H, &H->ntype, n))
        return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemcpyAsync(H->perm, val2, n * sizeof(int), cudaMemcpyDeviceToDevice, st));
    k_gather_nodes<<<(n + TB - 1) / TB, TB, 0, st>>>(n, H->perm, dx, dy, dh, dhs, ds, dt, H->px, H->py, H->h,
                                                     H->hs, H->sp, H->ntype, H->iperm);
    if (ng > 0)
        k_place_ghosts<<<(ng + TB - 1) / TB, TB, 0, st>>>(ng, n, gx, gy, gpar_ref, H->iperm, H->px, H->py, H->gpar);
    SUNSET_CUDA(H, cudaGetLastError());
    H->h_perm.resize(n);
    H->h_iperm.resize(n);
    SUNSET_CUDA(H, cudaMemcpyAsync(H->h_perm.data(), H->perm, n * sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->h_iperm.data(), H->iperm, n * sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    for (void *p : {(void *)dx, (void *)dy, (void *)dh, (void *)dhs, (void *)ds, (void *)dt, (void *)mcount,
                    (void *)moff, (void *)gx, (void *)gy, (void *)gpar_ref, (void *)key, (void *)key2, (void *)val,
                    (void *)val2})
        dfree(H, p);
    return 0;
}

// ---------------------------------------------------------------------------------------
int find_neighbours_device(Handle *H) {
    const int n = H->npfb, np = H->np;
    cudaStream_t st = H->stream;
    const int TB = 256;
    // grid: covers the domain plus the ghost band (ghosts lie within 4 h of an edge)
    double cs = kSs * H->hmax;
    double margin = 2.0 * cs + 4.0 * H->hmax + 1e-12 * (H->xmax - H->xmin);
    Grid g;
    g.x0 = H->xmin - margin;
    g.y0 = H->ymin - margin;
    g.inv = 1.0 / cs;
    g.ncx = (int)((H->xmax - H->xmin + 2 * margin) * g.inv) + 1;
    g.ncy = (int)((H->ymax - H->ymin + 2 * margin) * g.inv) + 1;
    long long ncell = (long long)g.ncx * g.ncy;
    if (ncell > (1LL << 31)) return set_err(H, SUNSET_ERR_SCOPE, "cell grid too large (%lld cells)", ncell);
    int *cid, *cid2, *pid, *pid2, *cstart, *cend;
    if (dalloc(H, &cid, np) || dalloc(H, &cid2, np) || dalloc(H, &pid, np) || dalloc(H, &pid2, np) ||
        dalloc(H, &cstart, ncell) || dalloc(H, &cend, ncell))
        return SUNSET_ERR_NOMEM;
    k_cell_id<<<(np + TB - 1) / TB, TB, 0, st>>>(H->px, H->py, np, g, cid, pid);
    size_t tmpb = 0;
    void *tmp;
    cub::DeviceRadixSort::SortPairs(nullptr, tmpb, cid, cid2, pid, pid2, np, 0, 32, st);
    if (dalloc(H, (char **)&tmp, tmpb)) return SUNSET_ERR_NOMEM;
    cub::DeviceRadixSort::SortPairs(tmp, tmpb, cid, cid2, pid, pid2, np, 0, 32, st);
    dfree(H, tmp);
    SUNSET_CUDA(H, cudaMemsetAsync(cstart, 0, ncell * sizeof(int), st));
    SUNSET_CUDA(H, cudaMemsetAsync(cend, 0, ncell * sizeof(int), st));
    k_cell_bounds<<<(np + TB - 1) / TB, TB, 0, st>>>(cid2, np, cstart, cend);

    const RefGrid rg{H->xmin - (H->xmax - H->xmin), H->ymin - (H->ymax - H->ymin), 1.0 / (1.0 * (kSs * H->h0))};
    SearchArgs sa{H->px, H->py, H->h, cstart, cend, pid2, g, rg, n};
    int *count;
    long long *cnt64, *rowptr;
    if (dalloc(H, &count, n) || dalloc(H, &cnt64, n + 1) || dalloc(H, &rowptr, n + 1)) return SUNSET_ERR_NOMEM;
    k_search<false><<<(n + TB - 1) / TB, TB, 0, st>>>(sa, count, nullptr, nullptr, nullptr);
    std::vector<int> hcount(n);
    SUNSET_CUDA(H, cudaMemcpyAsync(hcount.data(), count, n * sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    std::vector<long long> hrow(n + 1);
    hrow[0] = 0;
    int maxc = 0;
    for (int i = 0; i < n; i++) {
        hrow[i + 1] = hrow[i] + hcount[i];
        maxc = hcount[i] > maxc ? hcount[i] : maxc;
    }
    long long nl = hrow[n];
    SUNSET_CUDA(H, cudaMemcpyAsync(rowptr, hrow.data(), (n + 1) * sizeof(long long), cudaMemcpyHostToDevice, st));
    int *opt;
    double *or2;
    if (dalloc(H, &opt, nl) || dalloc(H, &or2, nl)) return SUNSET_ERR_NOMEM;
    k_search<true><<<(n + TB - 1) / TB, TB, 0, st>>>(sa, nullptr, rowptr, opt, or2);
    if (!H->cnt_small && dalloc(H, &H->cnt_small, n)) return SUNSET_ERR_NOMEM;
    int *serr;
    if (dalloc(H, &serr, 1)) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(serr, 0, sizeof(int), st));
    const int width = std::min(maxc, kMaxRowSort), sort_smem = kSortWarps * width * 20;
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_sort_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, kSortWarps * kMaxRowSort * 20));
    k_sort_rows<<<(n + kSortWarps - 1) / kSortWarps, kSortWarps * 32, sort_smem, st>>>(n, rowptr, width, opt, or2, H->hs, H->perm,
                                                                                     H->px, H->py, rg, H->cnt_small, serr);
    int hserr = 0;
    SUNSET_CUDA(H, cudaMemcpyAsync(&hserr, serr, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    dfree(H, serr);
    if (hserr) return set_err(H, SUNSET_ERR_SCOPE, "neighbour row of node %d too long to sort", hserr - 1);
    std::vector<int> hsmall(n);
    SUNSET_CUDA(H, cudaMemcpyAsync(hsmall.data(), H->cnt_small, n * sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));

    // sliced ELL layout
    H->nslices = (n + kSlice - 1) / kSlice;
    std::vector<long long> sptr(H->nslices + 1);
    std::vector<int> sw(H->nslices), sws(H->nslices);
    sptr[0] = 0;
    for (int sl = 0; sl < H->nslices; sl++) {
        int w = 0, ws = 0;
        for (int i = sl * kSlice; i < n && i < (sl + 1) * kSlice; i++) {
            w = hcount[i] > w ? hcount[i] : w;
            ws = hsmall[i] > ws ? hsmall[i] : ws;
        }
        w = (w + 1) & ~1;  // even widths: links are stored in pairs (sell_at)
        ws = (ws + 1) & ~1;
        sw[sl] = w;
        sws[sl] = ws;
        sptr[sl + 1] = sptr[sl] + (long long)w * kSlice;
    }
    H->nlinks_sell = sptr[H->nslices];
    H->nplink = maxc;
    if (dalloc(H, &H->slice_ptr, H->nslices + 1) || dalloc(H, &H->slice_w, H->nslices) ||
        dalloc(H, &H->slice_ws, H->nslices) || dalloc(H, &H->lpt, H->nlinks_sell) ||
        dalloc(H, &H->lidx, H->nlinks_sell) || (!H->cnt && dalloc(H, &H->cnt, n)))
        return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemcpyAsync(H->slice_ptr, sptr.data(), sptr.size() * sizeof(long long), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->slice_w, sw.data(), sw.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->slice_ws, sws.data(), sws.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->cnt, hcount.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
    int *mflag;
    if (dalloc(H, &mflag, 1)) return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemsetAsync(mflag, 0, sizeof(int), st));
    int nthreads = H->nslices * kSlice;
    k_fill_sell<<<(nthreads + TB - 1) / TB, TB, 0, st>>>(n, H->nslices, rowptr, opt, H->slice_ptr, H->slice_w,
                                                          H->gpar, H->gvrel, H->lpt, H->lidx, mflag);
    int hm = 0;
    SUNSET_CUDA(H, cudaMemcpyAsync(&hm, mflag, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    SUNSET_CUDA(H, cudaGetLastError());
    H->has_mirrors = hm != 0;
    for (void *p : {(void *)cid, (void *)cid2, (void *)pid, (void *)pid2, (void *)cstart, (void *)cend, (void *)count,
                    (void *)cnt64, (void *)rowptr, (void *)opt, (void *)or2, (void *)mflag})
        dfree(H, p);
    return 0;
}

}  // namespace sunset

// ---------------------------------------------------------------------------------------
// Halo lists of the staged stencil kernels.  A thread block owns kTileSlices consecutive
// slices (kTile nodes); its halo is the sorted set of parents its links reach.  The
// kernels load the halo's fields once into shared memory (consecutive halo entries are
// mostly consecutive nodes in Morton order, so these loads coalesce) and every link then
// reads shared memory through a 16-bit position.  Built once per node set.
// ---------------------------------------------------------------------------------------
namespace sunset {

// Boundary framework data in internal order: normals, FD parents, the boundary list in
// the reference's order (setup_domain.F90:314-327 builds it in node order) with each
// boundary node's four FD rows (the reader places them right after their parent), and the
// boundary index of each node.  Inputs are in the reference's node order.
int upload_boundary(Handle *H, const std::vector<double> &nx, const std::vector<double> &ny,
                    const std::vector<int> &fdpar_ref, const std::vector<int> &blist_ref,
                    const std::vector<int> &type) {
    const int n = H->npfb, nb = (int)blist_ref.size();
    const std::vector<int> &perm = H->h_perm, &iperm = H->h_iperm;
    std::vector<double> inx(n), iny(n);
    std::vector<int> ifd(n), ibidx(n, -1), ibl(nb), ibrow(4 * (size_t)(nb ? nb : 1), 0);
    for (int i = 0; i < n; i++) {
        const int r = perm[i];
        inx[i] = nx[r];
        iny[i] = ny[r];
        ifd[i] = fdpar_ref[r] >= 0 ? iperm[fdpar_ref[r]] : -1;
    }
    H->h_btype.resize(nb);
    for (int jj = 0; jj < nb; jj++) {
        const int r = blist_ref[jj];
        ibl[jj] = iperm[r];
        ibidx[iperm[r]] = jj;
        H->h_btype[jj] = type[r];
        for (int j = 1; j <= 4; j++) ibrow[4 * jj + j - 1] = iperm[r + j];
    }
    if (dalloc(H, &H->rnx, n) || dalloc(H, &H->rny, n) || dalloc(H, &H->fdpar, n) || dalloc(H, &H->bidx, n) ||
        dalloc(H, &H->blist, nb ? nb : 1) || dalloc(H, &H->brow, 4 * (size_t)(nb ? nb : 1)))
        return SUNSET_ERR_NOMEM;
    cudaStream_t st = H->stream;
    SUNSET_CUDA(H, cudaMemcpyAsync(H->rnx, inx.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->rny, iny.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->fdpar, ifd.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
    SUNSET_CUDA(H, cudaMemcpyAsync(H->bidx, ibidx.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
    if (nb) {
        SUNSET_CUDA(H, cudaMemcpyAsync(H->blist, ibl.data(), nb * sizeof(int), cudaMemcpyHostToDevice, st));
        SUNSET_CUDA(H, cudaMemcpyAsync(H->brow, ibrow.data(), 4 * (size_t)nb * sizeof(int), cudaMemcpyHostToDevice, st));
    }
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    return 0;
}

namespace {

// The halo of one tile a block: the parents its links reach go into a hash set in shared memory
// (tsize slots, open addressing), which is compacted and sorted.  A tile reaches a few times
// its own nodes (700 of 256 at order 8) over ten thousand links, so nearly every link finds
// its node already there.  count[t] is the halo's size, or -1 where the set overflowed half its
// slots; list[t * tsize / 2 ...] the sorted nodes.
constexpr int kHaloThreads = 256;
__global__ void __launch_bounds__(kHaloThreads) k_tile_halos(int n, int nslices, const long long *slice_ptr, const int *cnt,
                                                             const int *lidx, int tslices, int tsize, int *list, int *count) {
    extern __shared__ int hsm[];
    int *table = hsm, *vals = hsm + tsize;
    __shared__ int num;
    const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = tsize / 2;
    for (int e = tid; e < tsize; e += kHaloThreads) table[e] = -1;
    if (tid == 0) num = 0;
    __syncthreads();
    const int shift = 32 - (31 - __clz(tsize));
    for (int sl = tile * tslices + warp; sl < min(nslices, (tile + 1) * tslices); sl += kHaloThreads / 32) {
        const int i = sl * kSlice + lane;
        const int c = i < n ? cnt[i] : 0;
        const long long base = slice_ptr[sl];
        for (int k = 0; k < c; k++) {
            const int p = lidx[sell_at(base, k, lane)] & kLinkMask;
            unsigned slot = ((unsigned)p * 2654435761u) >> shift;
            // at most half the slots fill before the tile gives up, so a free one is always near
            for (int probe = 0; probe < tsize; probe++) {
                int v = ((volatile int *)table)[slot];
                if (v == p) break;
                if (v < 0) {
                    if (((volatile int *)&num)[0] > half) break;
                    v = atomicCAS(&table[slot], -1, p);
                    if (v == -1) atomicAdd(&num, 1);
                    if (v == -1 || v == p) break;
                }
                slot = (slot + 1) & (tsize - 1);
            }
        }
    }
    __syncthreads();
    const int total = num;
    if (total > half) {
        if (tid == 0) count[tile] = -1;
        return;
    }
    __syncthreads();
    if (tid == 0) num = 0;
    __syncthreads();
    for (int e = tid; e < tsize; e += kHaloThreads) {
        const int v = table[e];
        if (v >= 0) vals[atomicAdd(&num, 1)] = v;
    }
    int np2 = 1;
    while (np2 < total) np2 <<= 1;
    __syncthreads();
    for (int e = total + tid; e < np2; e += kHaloThreads) vals[e] = 0x7fffffff;
    __syncthreads();
    for (int k = 2; k <= np2; k <<= 1)  // bitonic sort; np2 <= half, a power of two
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int e = tid; e < np2; e += kHaloThreads) {
                const int x = e ^ j;
                if (x > e) {
                    const int a = vals[e], b = vals[x];
                    if ((a > b) == ((e & k) == 0)) { vals[e] = b; vals[x] = a; }
                }
            }
            __syncthreads();
        }
    for (int e = tid; e < total; e += kHaloThreads) list[(size_t)tile * half + e] = vals[e];
    if (tid == 0) count[tile] = total;
}

// The tiles' halos into one list, and each link's position in its tile's halo | reflection code
// << 14 (0 in the padding), by binary search in shared memory.
__global__ void __launch_bounds__(kHaloThreads) k_halo_links(int n, int nslices, const long long *slice_ptr, const int *slice_w,
                                                             const int *cnt, const int *lidx, const int *list, int tslices, int half,
                                                             const int *halo_ptr, int *halo, uint16_t *lloc) {
    extern __shared__ int hsm[];
    const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int h0 = halo_ptr[tile], hn = halo_ptr[tile + 1] - h0;
    for (int e = tid; e < hn; e += kHaloThreads) {
        const int v = list[(size_t)tile * half + e];
        hsm[e] = v;
        halo[h0 + e] = v;
    }
    __syncthreads();
    for (int sl = tile * tslices + warp; sl < min(nslices, (tile + 1) * tslices); sl += kHaloThreads / 32) {
        const int i = sl * kSlice + lane;
        const int c = i < n ? cnt[i] : 0;
        const long long base = slice_ptr[sl];
        const int w = slice_w[sl];
        for (int k = 0; k < w; k += 2) {  // a pair of links is one 8-byte load and one 4-byte store
            const long long o = sell_at(base, k, lane);
            const int2 lk = *reinterpret_cast<const int2 *>(lidx + o);
            unsigned out = 0;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                if (k + q >= c) continue;
                const int v = q ? lk.y : lk.x, p = v & kLinkMask;
                int lo = 0, hi = hn;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (hsm[mid] <= p) lo = mid;
                    else hi = mid;
                }
                out |= ((unsigned)lo | (((unsigned)v >> 30) << 14)) << (16 * q);
            }
            *reinterpret_cast<unsigned *>(lloc + o) = out;
        }
    }
}

}  // namespace

// Slices a tile takes; the other warps of its block share the links of the same nodes.  As few
// as leave the set's tiles at most two a SM: a set that fills the device keeps whole tiles, whose
// halo is the smallest a node (FP64 step, microseconds with 8, 4, 2 and 1 slices: 4,096 nodes at
// order 8 100, 71, 58, 50; 16,384 118, 83, 75, 102; 36,864 132, 110, 138, 163; 65,536 178, 227,
// 214, 265; order 4 at 16,384 55, 43, 42, 61).
//
// Shared links are summed in another order.  That is rounding on the periodic sets (3e-16), but
// the sets with boundary nodes can hold a stencil that amplifies it (the cylinder channel: 3e-8
// of the momentum after twenty steps on some seeds), and in mixed precision FP32 sums in
// another order, from other offsets, change the fields by 1e-9 to 3e-8: both keep whole tiles.
// Two ways that keep the order gained too little: a thread a node in smaller blocks with rings
// eight deep (4,096 nodes 96 -> 90), a warp a gathered field (95 -> 86, and 115 -> 156 at 16,384).
static int tile_slices(Handle *H, int nslices, int *ts) {
    SUNSET_CUDA(H, cudaDeviceGetAttribute(&H->nsm, cudaDevAttrMultiProcessorCount, H->device));
    SUNSET_CUDA(H, cudaDeviceGetAttribute(&H->sm_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, H->device));
    *ts = H->cfg.precision == SUNSET_MIXED || H->nb > 0 ? kTileSlices : 1;
    while (*ts < kTileSlices && nslices > 2 * H->nsm * *ts) *ts *= 2;
    return 0;
}

int build_halos(Handle *H) {
    const int n = H->npfb, nsl = H->nslices;
    const long long L = H->nlinks_sell;
    cudaStream_t st = H->stream;
    if (int rc = tile_slices(H, nsl, &H->tslices)) return rc;
    const int ts = H->tslices, nt = (nsl + ts - 1) / ts;
    // the hash set: 4096 slots hold the halos of the orders' own stencils (2048 nodes a tile);
    // where one is larger, 32768, the most a block's shared memory and the 14-bit index take
    int *list = nullptr, *count = nullptr, tsize = 4096, hmax = 0;
    std::vector<int> hptr(nt + 1);
    if (dalloc(H, &count, nt)) return SUNSET_ERR_NOMEM;
    auto set_smem = [](int slots) { return (slots + slots / 2) * (int)sizeof(int); };
    // the limit is the process's, not the handle's: always the larger set's, so that set-ups in
    // other threads never find it too low
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_tile_halos, cudaFuncAttributeMaxDynamicSharedMemorySize, set_smem(2 * (kLocMask + 1))));
    for (;; tsize = 2 * (kLocMask + 1)) {
        const int smem = set_smem(tsize);
        if (dalloc(H, &list, (size_t)nt * (tsize / 2))) return SUNSET_ERR_NOMEM;
        k_tile_halos<<<nt, kHaloThreads, smem, st>>>(n, nsl, H->slice_ptr, H->cnt, H->lidx, ts, tsize, list, count);
        SUNSET_CUDA(H, cudaGetLastError());
        SUNSET_CUDA(H, cudaMemcpyAsync(hptr.data() + 1, count, nt * sizeof(int), cudaMemcpyDeviceToHost, st));
        SUNSET_CUDA(H, cudaStreamSynchronize(st));
        hptr[0] = 0;
        hmax = 0;
        bool over = false;
        for (int t = 0; t < nt; t++) {
            over = over || hptr[t + 1] < 0;
            hmax = std::max(hmax, hptr[t + 1]);
            hptr[t + 1] += hptr[t];
        }
        if (!over) break;
        dfree(H, list);
        if (tsize > kLocMask + 1) {
            dfree(H, count);
            return set_err(H, SUNSET_ERR_SCOPE, "a tile halo of more than %d nodes exceeds the 14-bit local index", kLocMask + 1);
        }
    }
    if (dalloc(H, &H->halo_ptr, nt + 1) || dalloc(H, &H->halo, (size_t)hptr[nt]) || dalloc(H, &H->lloc, L))
        return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemcpyAsync(H->halo_ptr, hptr.data(), hptr.size() * sizeof(int), cudaMemcpyHostToDevice, st));
    const int smem = hmax * (int)sizeof(int);
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_halo_links, cudaFuncAttributeMaxDynamicSharedMemorySize, (kLocMask + 1) * (int)sizeof(int)));
    k_halo_links<<<nt, kHaloThreads, smem, st>>>(n, nsl, H->slice_ptr, H->slice_w, H->cnt, H->lidx, list, ts, tsize / 2,
                                                 H->halo_ptr, H->halo, H->lloc);
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(st));
    dfree(H, list);
    dfree(H, count);
    H->ntiles = nt;
    H->halo_max = hmax;
    return 0;
}

}  // namespace sunset
