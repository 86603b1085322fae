// pixmom.cuh -- box, peaks and exact moment sums of a list of pixels: the
// pixel part of the preanalysis of kept branches (k_deblend.cu) and of the
// robust preanalysis of deblended objects (k_analyse.cu),
// src/cuda/cudaanalyse.cu:1686-2124.
//
// One warp takes a list (one block a long one).  The seven sums are kept in
// double bins (Bin2) per lane and reduced transposed: the lanes halve the set
// of sums they carry with each exchange, so that after three exchanges every
// lane carries one of them (36 shuffles for the 14 bins instead of the 140 of
// a butterfly each), and lanes 0..6 round their sum side by side.  All sums
// are exact, so neither the order nor the split changes a result.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace sx {

constexpr int PM_SUMS = 7;  // cd, sub, cd x, cd y, cd x^2, cd y^2, cd x y

struct PixBox {
    int xmin, xmax, ymin, ymax;
    unsigned pk, cpk;  // f2ord of the largest sub and cd
};

// what the pixel pass hands to the finishing kernel (one thread per object)
struct MomentRaw {
    double mx, my, mx2, my2, mxy;
    float rv, tv, peak, cpeak;
    int dnpix, area2, xmin, xmax, ymin, ymax, ovf;
};

__device__ __forceinline__ PixBox pix_box(const float *cd, const float *sub, const unsigned *pix, int i0, int n,
                                          int step, const FastDiv &wdiv, int w) {
    PixBox b;
    b.xmin = b.ymin = 0x7fffffff;
    b.xmax = b.ymax = -1;
    b.pk = b.cpk = 0u;
    for (int i = i0; i < n; i += step) {
        const unsigned p = __ldg(pix + i);
        const int y = (int)fdiv(p, wdiv), x = (int)p - y * w;
        b.pk = max(b.pk, f2ord(__ldg(sub + p)));
        b.cpk = max(b.cpk, f2ord(__ldg(cd + p)));
        b.xmin = min(b.xmin, x);
        b.xmax = max(b.xmax, x);
        b.ymin = min(b.ymin, y);
        b.ymax = max(b.ymax, y);
    }
    return b;
}

__device__ __forceinline__ void pixbox_warp(PixBox &b) {
    b.xmin = __reduce_min_sync(0xffffffffu, b.xmin);
    b.xmax = __reduce_max_sync(0xffffffffu, b.xmax);
    b.ymin = __reduce_min_sync(0xffffffffu, b.ymin);
    b.ymax = __reduce_max_sync(0xffffffffu, b.ymax);
    b.pk = __reduce_max_sync(0xffffffffu, b.pk);
    b.cpk = __reduce_max_sync(0xffffffffu, b.cpk);
}

// lane l: the warp's total of v[l & 7]
__device__ __forceinline__ double warp_sum8(const double v[8], int lane) {
    double a[4], b[2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double keep = lane & 4 ? v[k + 4] : v[k], give = lane & 4 ? v[k] : v[k + 4];
        a[k] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double keep = lane & 2 ? a[k + 2] : a[k], give = lane & 2 ? a[k] : a[k + 2];
        b[k] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
    }
    const double keep = lane & 1 ? b[1] : b[0], give = lane & 1 ? b[0] : b[1];
    double c = keep + __shfl_xor_sync(0xffffffffu, give, 1);
    c += __shfl_xor_sync(0xffffffffu, c, 8);
    return c + __shfl_xor_sync(0xffffffffu, c, 16);
}

// the sums with XSum, for a term the bins do not hold (out of line: the rare
// path, kept out of the callers' registers); lane k < PM_SUMS gets sum k (FULL:
// a branch's own pixels come in any order)
__device__ __noinline__ void pix_moments_xsum(const float *cd, const float *sub, const unsigned *pix, int i0, int i1,
                                              FastDiv wdiv, int w, int x0, int y0, XSum *out) {
    const int lane = threadIdx.x & 31;
    XSum s[PM_SUMS];
    for (int k = 0; k < PM_SUMS; k++) xs_init(s[k]);
    for (int i = i0 + lane; i < i1; i += 32) {
        const unsigned p = pix[i];
        const int yy = (int)fdiv(p, wdiv), x = (int)p - yy * w - x0, y = yy - y0;
        const float cval = cd[p], val = sub[p];
        xs_add<true>(s[0], cval);
        xs_add<true>(s[1], val);
        xs_add<true>(s[2], cval * x);
        xs_add<true>(s[3], cval * y);
        xs_add<true>(s[4], cval * x * x);
        xs_add<true>(s[5], cval * y * y);
        xs_add<true>(s[6], cval * x * y);
    }
    XSum mine;
    xs_init(mine);
    for (int k = 0; k < PM_SUMS; k++) {
        const XSum t = xs_warp_sum<true>(s[k]);
        if (lane == k) mine = t;
    }
    *out = mine;
}

// One warp over list entries i0 .. i1 - 1, at most DA_WARP_MAX (b: the whole
// list's box; dth: the threshold dn counts above, a2 counts above the middle
// between it and the peak; both per lane).  Lane k < PM_SUMS gets bins t0, t1
// of sum k; false when a term did not fit.
__device__ __forceinline__ bool pix_moments(const float *cd, const float *sub, const unsigned *pix, int i0, int i1,
                                            const FastDiv &wdiv, int w, const PixBox &b, double dth, double &t0,
                                            double &t1, int &dn, int &a2) {
    const int lane = threadIdx.x & 31;
    const float peak = ord2f(b.pk);
    const double dth2 = (dth + peak) / 2.0;
    constexpr int W = 20;  // DA_WARP_MAX = 2^10 terms
    static_assert(DA_WARP_MAX <= 1024, "terms per bin");
    // hints of the bins: the largest values times the box sides
    const int bx = 32 - __clz(b.xmax - b.xmin), by = 32 - __clz(b.ymax - b.ymin);
    const int tc = bs_order(ord2f(b.cpk));
    const unsigned l0 = bin_low(tc, W), l1 = bin_low(bs_order(peak), W), l2 = bin_low(tc + 1 + bx, W),
                   l3 = bin_low(tc + 1 + by, W), l4 = bin_low(tc + 1 + 2 * bx, W), l5 = bin_low(tc + 1 + 2 * by, W),
                   l6 = bin_low(tc + 1 + bx + by, W);
    Bin2 s[PM_SUMS];
#pragma unroll
    for (int k = 0; k < PM_SUMS; k++) bin_init(s[k]);
    bool ok = true;
    for (int i = i0 + lane; i < i1; i += 32) {
        const unsigned p = __ldg(pix + i);
        const int yy = (int)fdiv(p, wdiv), x = (int)p - yy * w - b.xmin, y = yy - b.ymin;
        const float cval = __ldg(cd + p), val = __ldg(sub + p);
        dn += val > dth;
        a2 += val > dth2;
        const float cx = cval * x, cy = cval * y;
        ok &= bin_add(s[0], cval, l0, W);
        ok &= bin_add(s[1], val, l1, W);
        ok &= bin_add(s[2], cx, l2, W);
        ok &= bin_add(s[3], cy, l3, W);
        ok &= bin_add(s[4], cx * x, l4, W);
        ok &= bin_add(s[5], cy * y, l5, W);
        ok &= bin_add(s[6], cx * y, l6, W);
    }
    if (!__all_sync(0xffffffffu, ok)) return false;
    {
        const double v[8] = {s[0].b0, s[1].b0, s[2].b0, s[3].b0, s[4].b0, s[5].b0, s[6].b0, 0.0};
        t0 = warp_sum8(v, lane);
    }
    {
        const double v[8] = {s[0].b1, s[1].b1, s[2].b1, s[3].b1, s[4].b1, s[5].b1, s[6].b1, 0.0};
        t1 = warp_sum8(v, lane);
    }
    return true;
}

// v: lane k < PM_SUMS: sum k
__device__ __forceinline__ void pix_moments_store(double v, int ovf, int dnpix, int area2, const PixBox &b,
                                                  MomentRaw *R) {
    const int lane = threadIdx.x & 31;
    if (lane == 0)
        R->rv = (float)v;
    else if (lane == 1)
        R->tv = (float)v;
    else if (lane < PM_SUMS)
        (&R->mx)[lane - 2] = v;
    else if (lane == PM_SUMS) {
        R->peak = ord2f(b.pk);
        R->cpeak = ord2f(b.cpk);
        R->dnpix = dnpix;
        R->area2 = area2;
        R->ovf = ovf;
    } else if (lane == PM_SUMS + 1) {
        R->xmin = b.xmin;
        R->xmax = b.xmax;
        R->ymin = b.ymin;
        R->ymax = b.ymax;
    }
}

// one warp over a list of n <= DA_WARP_MAX pixels
__device__ __forceinline__ void pix_moments_warp(const float *cd, const float *sub, const unsigned *pix, int n,
                                                 const FastDiv &wdiv, int w, double dth, MomentRaw *R) {
    const int lane = threadIdx.x & 31;
    PixBox b = pix_box(cd, sub, pix, lane, n, 32, wdiv, w);
    pixbox_warp(b);
    double t0, t1, v;
    int dn = 0, a2 = 0, ovf = 0;
    if (pix_moments(cd, sub, pix, 0, n, wdiv, w, b, dth, t0, t1, dn, a2)) {
        v = t0 + t1;
    } else {
        XSum x;
        pix_moments_xsum(cd, sub, pix, 0, n, wdiv, w, b.xmin, b.ymin, &x);
        v = xs_double(x);
        ovf = __any_sync(0xffffffffu, lane < PM_SUMS && x.ovf);
    }
    dn = __reduce_add_sync(0xffffffffu, dn);
    a2 = __reduce_add_sync(0xffffffffu, a2);
    pix_moments_store(v, ovf, dn, a2, b, R);
}

// The sums of a list by one warp where XSum did not hold one of them (R->ovf),
// one pass over the list each, into R; R->ovf: WideSum::bad.  Called by
// the finishing kernels, so that the kernels that sum keep their registers.
__device__ __noinline__ void pix_moments_wide(const float *cd, const float *sub, const unsigned *pix, int n,
                                              FastDiv wdiv, int w, MomentRaw *R) {
    const int lane = threadIdx.x & 31, x0 = R->xmin, y0 = R->ymin;
    double mine = 0.0;
    int bad = 0;
    for (int k = 0; k < PM_SUMS; k++) {
        WideSum s;
        ws_init(s);
        for (int i = lane; i < n; i += 32) {
            const unsigned p = pix[i];
            const int yy = (int)fdiv(p, wdiv), x = (int)p - yy * w - x0, y = yy - y0;
            const float cval = cd[p];
            ws_add(s, k == 0   ? cval
                      : k == 1 ? sub[p]
                      : k == 2 ? cval * x
                      : k == 3 ? cval * y
                      : k == 4 ? cval * x * x
                      : k == 5 ? cval * y * y
                               : cval * x * y);
        }
        s = ws_warp_sum(s);
        bad |= s.bad;
        const double d = ws_double(s);
        if (lane == k) mine = d;
    }
    if (lane == 0)
        R->rv = (float)mine;
    else if (lane == 1)
        R->tv = (float)mine;
    else if (lane < PM_SUMS)
        (&R->mx)[lane - 2] = mine;
    else if (lane == PM_SUMS)
        R->ovf = bad;
}

// a whole block over one list (at most 32 warps)
struct PixBlock {
    PixBox box[32];
    XSum x[32][PM_SUMS];
    int dnpix[32], area2[32];
};

__device__ __forceinline__ void pix_moments_block(const float *cd, const float *sub, const unsigned *pix, int n,
                                                  const FastDiv &wdiv, int w, double dth, PixBlock &sh, MomentRaw *R) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    PixBox b = pix_box(cd, sub, pix, threadIdx.x, n, blockDim.x, wdiv, w);
    pixbox_warp(b);
    if (lane == 0) sh.box[wid] = b;
    __syncthreads();
    b = sh.box[min(lane, nw - 1)];
    pixbox_warp(b);
    XSum x;
    xs_init(x);
    int dn = 0, a2 = 0;
    for (int i0 = wid * DA_WARP_MAX; i0 < n; i0 += nw * DA_WARP_MAX) {
        const int i1 = min(n, i0 + DA_WARP_MAX);
        double t0, t1;
        if (pix_moments(cd, sub, pix, i0, i1, wdiv, w, b, dth, t0, t1, dn, a2)) {
            xs_add_bins<true>(x, t0, t1);
        } else {
            XSum t;
            pix_moments_xsum(cd, sub, pix, i0, i1, wdiv, w, b.xmin, b.ymin, &t);
            xs_merge<true>(x, t);
        }
    }
    dn = __reduce_add_sync(0xffffffffu, dn);
    a2 = __reduce_add_sync(0xffffffffu, a2);
    if (lane < PM_SUMS) sh.x[wid][lane] = x;
    if (lane == 0) {
        sh.dnpix[wid] = dn;
        sh.area2[wid] = a2;
    }
    __syncthreads();
    if (wid == 0) {
        xs_init(x);
        dn = a2 = 0;
        for (int k = 0; k < nw; k++) {
            if (lane < PM_SUMS) xs_merge<true>(x, sh.x[k][lane]);
            dn += sh.dnpix[k];
            a2 += sh.area2[k];
        }
        const int ovf = __any_sync(0xffffffffu, lane < PM_SUMS && x.ovf);
        pix_moments_store(xs_double(x), ovf, dn, a2, b, R);
    }
    __syncthreads();
}

}  // namespace sx
