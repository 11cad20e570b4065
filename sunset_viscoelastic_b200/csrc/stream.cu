// stream.cu -- the link stream of the time step: bank-aware link order, and the weights the
// stage and filter kernels stream (FP64 copies, or packed fixed-point stage links and FP32
// filter weights for the mixed precision).
//
// The setup, the single-operator entry points and the weight export keep the reference's
// link order (derivatives.F90 sums over ij_link in order).  The time step sums each node's
// links in its own order instead, chosen for the hardware: the stage and filter kernels
// gather the tile halo from shared memory with 8-byte loads, which are served per
// half-warp, one wavefront per bank pair (position mod 16) and distinct position.  In the
// reference order neighbouring lanes often meet in the same bank pair at the same link slot
// (4.9 wavefronts a load on the order-6 set against the ideal 2).  k_deal_links
// re-deals each node's links slot by slot so that the 16 lanes of a half-warp read distinct
// bank pairs wherever a bipartite matching allows it (2.6 on that set).  Only the rounding
// of the sums changes (relative 1e-16 a sum).
//
// Mixed precision: the weight solves stay FP64; the stage kernel streams each link as three
// 32-bit words, one per operator (d/dx, d/dy, Laplacian).  A word is the integer 64 q + b:
// q the weight rounded to a 26-bit integer in units of a power of two per node and operator
// (2^(e-25), e the exponent of the node's largest |w| of that operator), b six bits of the
// link's 16-bit local index (bits 0-5, 6-11 and 12-15 of the index in the x, y and
// Laplacian words).  The stage masks b off and converts 64 q to FP32.  That is 12 bytes a
// link against 26 in FP64 (16-bit index + three doubles), with 25 bits relative to the node's
// largest weight; the stage sums in difference form, sum_k w_k (phi_j - phi_i), so a
// constant field keeps zero derivatives whatever the rounding.  (Converting the whole word,
// index bits included, saves the masks but adds b to 64 q: a perturbation of up to one
// unit of q that is not zero-mean -- the Laplacian word's bits are 0 for halos under 4096
// nodes -- and acts as a small extra Laplacian, 1e-6 of the fields in 100 steps.)
// The filter streams its weight rounded to FP32 with the local index (6 bytes a link).
#include <algorithm>
#include <vector>

#include "internal.cuh"

namespace sunset {

namespace {

struct StreamArgs {
    int npfb, nslices;
    const long long *slice_ptr;
    const int *slice_w;
    const int *src;  // SELL entry -> SELL entry of the reference-order arrays it takes (-1: padding)
    const uint16_t *lloc;
    const double *wx, *wy, *wl, *wh;
    uint16_t *lloc_s;
    double *wx_s, *wy_s, *wl_s, *wh_s;      // FP64 step
    unsigned *pk;                           // mixed step: packed stage links (pk_at)
    float *scx, *scy, *scl;                 // their per-node scales
    unsigned *wf;                           // mixed filter (wf_at)
};

constexpr int kPackBits = 26;  // bits of a packed stage weight (sign included)

// Exponent e with max|w| < 2^e (0 for an all-zero operator row).
__device__ __forceinline__ int pack_exponent(double wmax) {
    int e = 0;
    if (wmax > 0.0) frexp(wmax, &e);
    return e;
}
// A weight as the word 64 q + b: q its kPackBits-bit integer in units of
// 2^(e - kPackBits + 1), b six index bits.
__device__ __forceinline__ unsigned pack_weight(double w, int e, unsigned idx6) {
    const long long lim = (1ll << (kPackBits - 1)) - 1;
    long long q = llrint(ldexp(w, kPackBits - 1 - e));
    q = q > lim ? lim : (q < -lim ? -lim : q);
    return ((unsigned)(int)q << 6) | (idx6 & 63u);
}

// One thread per node: gather its links into the stream order; MX: pack the stage weights
// with the node's scales, round the filter weights to FP32 and sum those.  Padding entries
// keep weight 0 and local index 0.
template <bool MX>
__global__ void k_stream_weights(StreamArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if ((i >> 5) >= a.nslices) return;  // the last slice's lanes without a node get padding: the kernels read it
    const long long base = a.slice_ptr[i >> 5];
    const int lane = i & 31;
    const int w = a.slice_w[i >> 5];
    int ex = 0, ey = 0, el = 0;
    if constexpr (MX) {
        double mx = 0.0, my = 0.0, ml = 0.0;
        for (int k = 0; k < w; k++) {
            const int q = a.src[sell_at(base, k, lane)];
            if (q < 0) continue;
            mx = fmax(mx, fabs(a.wx[q]));
            my = fmax(my, fabs(a.wy[q]));
            ml = fmax(ml, fabs(a.wl[q]));
        }
        ex = pack_exponent(mx);
        ey = pack_exponent(my);
        el = pack_exponent(ml);
        if (i < a.npfb) {
            a.scx[i] = ldexpf(1.0f, ex - (kPackBits - 1) - 6);  // a word's value is 64 q
            a.scy[i] = ldexpf(1.0f, ey - (kPackBits - 1) - 6);
            a.scl[i] = ldexpf(1.0f, el - (kPackBits - 1) - 6);
        }
    }
    // the packed words of a padding slot point at the node itself (its first link in the
    // reference order, distance 0), so even a nonzero weight there would meet phi_i - phi_i
    const unsigned self_loc = a.lloc[sell_at(base, 0, lane)];
    for (int k = 0; k < w; k++) {
        const long long o = sell_at(base, k, lane);
        const int q = a.src[o];
        const unsigned loc = q < 0 ? 0u : a.lloc[q];
        a.lloc_s[o] = (uint16_t)loc;
        if constexpr (MX) {
            const unsigned ploc = q < 0 ? self_loc : loc;
            unsigned *pw = a.pk + pk_at(base, k, lane);
            pw[0] = pack_weight(q < 0 ? 0.0 : a.wx[q], ex, ploc);
            pw[1] = pack_weight(q < 0 ? 0.0 : a.wy[q], ey, ploc >> 6);
            pw[2] = pack_weight(q < 0 ? 0.0 : a.wl[q], el, ploc >> 12);
            unsigned *fw = a.wf + wf_at(base, k >> 1, lane);
            fw[k & 1] = __float_as_uint(q < 0 ? 0.0f : (float)a.wh[q]);
            fw[2] = (k & 1) ? ((fw[2] & 0xffffu) | (loc << 16)) : ((fw[2] & 0xffff0000u) | loc);
        } else {
            a.wx_s[o] = q < 0 ? 0.0 : a.wx[q];
            a.wy_s[o] = q < 0 ? 0.0 : a.wy[q];
            a.wl_s[o] = q < 0 ? 0.0 : a.wl[q];
            a.wh_s[o] = q < 0 ? 0.0 : a.wh[q];
        }
    }
}

// deal_slice_by_bank (bank_deal.cu) on the device, one warp a slice, with the same result: slot
// by slot, the lanes of each group of G are matched to the G bank groups by augmenting paths,
// the most constrained lane first, each lane trying its bank groups in the list order of their
// first remaining link.  src[o]: the SELL entry (in the reference order) whose link goes to
// entry o, or -1 for padding.
//
// A thread plays two parts: lane r of its group (the links it has left, the bank group it takes)
// and bank group t (its owner).  The groups of a warp take the steps of their searches side by
// side: in one step a lane's next bank group is the smallest first link, over the group's
// threads, among the bank groups not tried yet.  A search tries a bank group once, so it ends
// after at most 2 G steps.  Bound: the latency of those steps (a shared load, four shuffles),
// hidden by the slices of the set (issue 65 % active).  1,048,576 nodes at order 8: 36 ms; the
// host's threads took 0.9-2.0 s with their copies both ways.
constexpr unsigned short kNoLink = 0xffff;
constexpr int kDealWarps = 4;
__host__ __device__ inline int deal_smem(int width) { return (width * 32 + 2 * 32 * 16) * (int)sizeof(unsigned short); }

template <int G>
__global__ void __launch_bounds__(kDealWarps * 32) k_deal_links(int n, int nslices, const long long *slice_ptr, const int *slice_w,
                                                                const int *cnt, const int *cnt_small, const uint16_t *pos,
                                                                int width, int *src) {
    extern __shared__ unsigned short dsm[];
    const unsigned all = 0xffffffffu, gmask = (1u << G) - 1u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = blockIdx.x * (blockDim.x >> 5) + warp;
    if (sl >= nslices) return;
    const int t = lane & (G - 1), g0 = lane - t;
    unsigned short *nxt = dsm + (size_t)warp * (deal_smem(width) / sizeof(unsigned short));  // next link of the same bank group
    unsigned short *fr = nxt + width * 32, *fr2 = fr + 32 * 16;  // first link by lane and bank group: current set, other links
    const int i = sl * kSlice + lane;
    const int c = i < n ? cnt[i] : 0, cs = i < n ? min(cnt_small[i], c) : 0;
    const long long base = slice_ptr[sl];
    const int w = slice_w[sl];
    unsigned mask = 0, mask2 = 0;  // bank groups that the lane has links of
    for (int b = 0; b < 16; b++) fr[lane * 16 + b] = fr2[lane * 16 + b] = kNoLink;
    for (int k = c - 1; k >= 0; k--) {
        const int b = pos[sell_at(base, k, lane)] & (G - 1);
        unsigned short *f = (k < cs ? fr : fr2) + lane * 16 + b;
        nxt[k * 32 + lane] = *f;
        *f = (unsigned short)k;
        if (k < cs) mask |= 1u << b;
        else mask2 |= 1u << b;
    }
    for (int k = 0; k < w; k++) {
        if (k == cs && cs < c) {  // the small links are dealt: go on with the others
            for (int b = 0; b < 16; b++) fr[lane * 16 + b] = fr2[lane * 16 + b];
            mask = mask2;
        }
        __syncwarp();
        const bool has = k < c;
        // rank of the lane: fewest bank groups first, then lane order
        const int key = has ? __popc(mask) * 32 + t : 0x10000;
        int rank = 0;
#pragma unroll
        for (int j = 0; j < G; j++) rank += __shfl_sync(all, key, g0 + j) < key;
        if (!has) rank = 99;
        const int nact = __popc((__ballot_sync(all, has) >> g0) & gmask);
        int owner = (t == 0 && nact < G) ? G : -1;  // padding lanes read position 0
        int choice = -1;
        int q = 0, r = -1, depth = 0, sr = 0, sb = 0;
        unsigned seen = 0;
        while (__any_sync(all, q < nact)) {
            const bool run = q < nact;
            const int rq = __ffs((__ballot_sync(all, rank == q) >> g0) & gmask) - 1;
            if (run && r < 0) {
                r = rq;
                seen = 0;
            }
            unsigned v = run ? fr[(g0 + r) * 16 + t] : kNoLink;
            v = (v != kNoLink && !((seen >> t) & 1u)) ? (v << 4 | t) : 0xffffffffu;
#pragma unroll
            for (int o = G / 2; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(all, v, o));
            const bool found = run && v != 0xffffffffu;
            const int b = v & 15;
            const int ob = __shfl_sync(all, owner, g0 + (found ? b : 0));
            const int back = __shfl_sync(all, sr, g0 + (depth > 0 ? depth - 1 : 0));
            const bool won = found && ob < 0;
            if (__any_sync(all, won)) {  // each lane of the path takes the bank group it was trying
                if (won && t == b) owner = r;
                if (won && t == r) choice = b;
                for (int d = depth - 1; __any_sync(all, won && d >= 0); d--) {
                    const int pr = __shfl_sync(all, sr, g0 + (d > 0 ? d : 0)), pb = __shfl_sync(all, sb, g0 + (d > 0 ? d : 0));
                    if (won && d >= 0) {
                        if (t == pb) owner = pr;
                        if (t == pr) choice = pb;
                    }
                }
            }
            if (found) seen |= 1u << b;
            if (won || (run && !found && depth == 0)) {  // matched, or left without a match
                q++;
                r = -1;
                depth = 0;
            } else if (run && !found) {
                depth--;
                r = back;
            } else if (found && ob < G) {  // the owner looks for another bank group
                if (t == depth) {
                    sr = r;
                    sb = b;
                }
                depth++;
                r = ob;
            }
        }
        if (__any_sync(all, has && choice < 0)) {  // unmatched lanes: the least used bank group, in list order
            int used = owner >= 0 ? 1 : 0;
            for (q = 0; __any_sync(all, q < nact); q++) {
                const int rq = __ffs((__ballot_sync(all, rank == q) >> g0) & gmask) - 1;
                const int at = rq > 0 ? rq : 0;
                const bool open = __shfl_sync(all, choice, g0 + at) < 0 && q < nact;
                unsigned v = open ? fr[(g0 + at) * 16 + t] : kNoLink;
                v = v != kNoLink ? ((unsigned)used << 20 | v << 4 | t) : 0xffffffffu;
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(all, v, o));
                if (open && t == at) choice = v & 15;
                if (open && t == (int)(v & 15)) used++;
            }
        }
        __syncwarp();
        int from = -1;
        if (has) {
            const int e = fr[lane * 16 + choice];
            const unsigned short nx = nxt[e * 32 + lane];
            fr[lane * 16 + choice] = nx;
            if (nx == kNoLink) mask &= ~(1u << choice);
            from = (int)sell_at(base, e, lane);
        }
        src[sell_at(base, k, lane)] = from;
    }
}

template <int G>
int launch_deal(Handle *H, int n, int nslices, const long long *slice_ptr, const int *slice_w, const int *cnt,
                const int *cnt_small, const uint16_t *pos, int width, int *src, cudaStream_t st) {
    const int per = deal_smem(width), most = 200 * 1024;
    if (per > most) return set_err(H, SUNSET_ERR_SCOPE, "neighbour lists too long for the link order");
    const int warps = std::max(1, std::min(kDealWarps, (48 * 1024) / per));
    SUNSET_CUDA(H, cudaFuncSetAttribute(k_deal_links<G>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    k_deal_links<G><<<(nslices + warps - 1) / warps, warps * 32, warps * per, st>>>(n, nslices, slice_ptr, slice_w, cnt,
                                                                                   cnt_small, pos, width, src);
    SUNSET_CUDA(H, cudaGetLastError());
    return 0;
}

}  // namespace

// New SELL order of the links for the time step: small links stay in the slots [0, cnt_small)
// and the other links in [cnt_small, cnt), so the stage kernel (small links) and the filter
// (all links) see the same sets as in the reference order.
int deal_links(Handle *H, int group, int n, int nslices, const long long *slice_ptr, const int *slice_w, const int *cnt,
               const int *cnt_small, const uint16_t *pos, int width, int *src) {
    return group == 16 ? launch_deal<16>(H, n, nslices, slice_ptr, slice_w, cnt, cnt_small, pos, width, src, H->stream)
                       : launch_deal<8>(H, n, nslices, slice_ptr, slice_w, cnt, cnt_small, pos, width, src, H->stream);
}

// Called once the FP64 weights, their sums and the filter coefficients exist.
int make_stream_links(Handle *H) {
    const long long L = H->nlinks_sell;
    const int n = H->npfb;
    const bool mx = H->cfg.precision == SUNSET_MIXED;
    if (L >= (1ll << 31)) return set_err(H, SUNSET_ERR_SCOPE, "the link stream supports at most 2^31 link slots");
    if (!H->lloc_s) {
        if (dalloc(H, &H->lloc_s, L)) return SUNSET_ERR_NOMEM;
        if (mx) {
            if (dalloc(H, &H->pk, 3 * L) || dalloc(H, &H->wf, 3 * L / 2) || dalloc(H, &H->scx, n) ||
                dalloc(H, &H->scy, n) || dalloc(H, &H->scl, n))
                return SUNSET_ERR_NOMEM;
        } else {
            if (dalloc(H, &H->wx_s, L) || dalloc(H, &H->wy_s, L) || dalloc(H, &H->wl_s, L) || dalloc(H, &H->wh_s, L))
                return SUNSET_ERR_NOMEM;
        }
    }
    int *d_src = nullptr;
    if (dalloc(H, &d_src, L)) return SUNSET_ERR_NOMEM;
    if (int rc = deal_links(H, 16, n, H->nslices, H->slice_ptr, H->slice_w, H->cnt, H->cnt_small, H->lloc,
                            (H->nplink + 1) & ~1, d_src))
        return rc;
    StreamArgs a{n, H->nslices, H->slice_ptr, H->slice_w, d_src, H->lloc, H->wx, H->wy, H->wl, H->wh, H->lloc_s,
                 H->wx_s, H->wy_s, H->wl_s, H->wh_s, H->pk, H->scx, H->scy, H->scl, H->wf};
    if (mx) k_stream_weights<true><<<(n + 255) / 256, 256, 0, H->stream>>>(a);
    else k_stream_weights<false><<<(n + 255) / 256, 256, 0, H->stream>>>(a);
    SUNSET_CUDA(H, cudaGetLastError());
    SUNSET_CUDA(H, cudaStreamSynchronize(H->stream));
    dfree(H, d_src);
    return 0;
}

}  // namespace sunset

// The device's link order on host arrays in the SELL layout, for the test that compares it with
// deal_slice_by_bank at both group sizes (not part of the interface in include/sunset_gpu.h).
static int check_deal(sunset::Handle *H, int group, int nslices, const long long *slice_ptr, const int *slice_w, const int *cnt,
                      const int *cnt_small, const uint16_t *pos, int width, int *src) {
    using namespace sunset;
    const int n = nslices * kSlice;
    const size_t L = (size_t)slice_ptr[nslices];
    long long *dp;
    int *dw, *dc, *ds, *dsrc;
    uint16_t *dpos;
    if (dalloc(H, &dp, nslices + 1) || dalloc(H, &dw, nslices) || dalloc(H, &dc, n) || dalloc(H, &ds, n) || dalloc(H, &dpos, L) ||
        dalloc(H, &dsrc, L))
        return SUNSET_ERR_NOMEM;
    SUNSET_CUDA(H, cudaMemcpyAsync(dp, slice_ptr, (nslices + 1) * sizeof(long long), cudaMemcpyHostToDevice, H->stream));
    SUNSET_CUDA(H, cudaMemcpyAsync(dw, slice_w, nslices * sizeof(int), cudaMemcpyHostToDevice, H->stream));
    SUNSET_CUDA(H, cudaMemcpyAsync(dc, cnt, n * sizeof(int), cudaMemcpyHostToDevice, H->stream));
    SUNSET_CUDA(H, cudaMemcpyAsync(ds, cnt_small, n * sizeof(int), cudaMemcpyHostToDevice, H->stream));
    SUNSET_CUDA(H, cudaMemcpyAsync(dpos, pos, L * sizeof(uint16_t), cudaMemcpyHostToDevice, H->stream));
    if (int rc = deal_links(H, group, n, nslices, dp, dw, dc, ds, dpos, width, dsrc)) return rc;
    SUNSET_CUDA(H, copy_out(H, src, dsrc, L * sizeof(int)));
    return 0;
}

extern "C" int sunset_check_deal(int group, int nslices, const long long *slice_ptr, const int *slice_w, const int *cnt,
                                 const int *cnt_small, const uint16_t *pos, int width, int *src) {
    if (group != 8 && group != 16) return SUNSET_ERR_ARG;
    sunset::Handle H;
    int rc = SUNSET_ERR_CUDA;
    if (cudaStreamCreateWithFlags(&H.stream, cudaStreamNonBlocking) == cudaSuccess) {
        rc = check_deal(&H, group, nslices, slice_ptr, slice_w, cnt, cnt_small, pos, width, src);
        cudaStreamSynchronize(H.stream);
        cudaStreamDestroy(H.stream);
    }
    H.mem.clear();
    return rc;
}
