// k_analyse.cu -- per-object analysis after deblending: the robust
// preanalysis of deblended objects over their final pixels
// (src/cuda/cudaanalyse.cu:1906-2124) and examineiso (:2176-2581).
//
// One warp per object walks the object's pixel list (contiguous, raster
// order), in two kernels: the robust preanalysis, whose moments examineiso
// reads, then examineiso itself.  Sums that feed decisions or integer outputs are exact (XSum);
// the double sums of the position errors and of the FWHM fit are reduced in
// a fixed lane order.
#include "common.cuh"
#include "kernels.cuh"
#include "kron.cuh"
#include "pixmom.cuh"

namespace sx {

constexpr int AN_WARPS = 8;
// four resident CTAs per SM (at most 64 registers, a few spilled): these
// kernels wait on pixel-list loads, and residency hides that better than
// registers saved (analyse stage 1.37 ms at 4 CTAs/SM, 1.45 at 3 with fewer
// spills, 1.65 at 2 with none, one crowded 4096^2 frame when its sums were
// 128-bit; 0.54 ms at 4 now)
constexpr int AN_MINB = 4;

// fixed-order (butterfly) double sum; identical in every lane
__device__ __forceinline__ double warp_sum_d(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// four sums at once, each added in that same order (pairs at distance 16, 8, 4,
// 2, 1): lanes 8k .. 8k + 7 get the sum of v[k]
__device__ __forceinline__ double warp_sum4(const double v[4], int lane) {
    const bool h1 = lane & 16, h2 = lane & 8;
    const double a = (h1 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h1 ? v[0] : v[2], 16);
    const double b = (h1 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h1 ? v[1] : v[3], 16);
    double c = (h2 ? b : a) + __shfl_xor_sync(0xffffffffu, h2 ? a : b, 8);
    for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}

constexpr int EX_TOP = 4;        // largest filtered values a lane keeps
constexpr int EX_TOP_AREA = 16;  // DETECT_MINAREA up to which they are tried first

// k-th smallest (0-based) of the cd values of n pixels, as float bits; the
// values are 0 or positive (object pixels lie at or above the detection
// threshold, which is 0 where the variance is; the filter's sums begin with +0),
// so their bit patterns sort like the values.  Four 8-bit radix passes; in each
// pass the digit that holds rank k is found by a warp scan over 256 bins
// (lane l owns bins 8l..8l+7).
__device__ unsigned warp_select(const unsigned *opix, int n, const float *cd, int k, unsigned *hist) {
    const int lane = threadIdx.x & 31;
    unsigned prefix = 0, mask = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = lane; i < 256; i += 32) hist[i] = 0;
        __syncwarp();
        for (int i = lane; i < n; i += 32) {
            unsigned key = __float_as_uint(__ldg(cd + __ldg(opix + i)));
            if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255], 1u);
        }
        __syncwarp();
        const uint4 h0 = reinterpret_cast<const uint4 *>(hist)[lane * 2];
        const uint4 h1 = reinterpret_cast<const uint4 *>(hist)[lane * 2 + 1];
        const unsigned c[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
        unsigned tot = c[0] + c[1] + c[2] + c[3] + c[4] + c[5] + c[6] + c[7];
        unsigned incl = tot;
        for (int o = 1; o < 32; o <<= 1) {
            unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        unsigned excl = incl - tot;
        unsigned sel = __ballot_sync(0xffffffffu, incl > (unsigned)k);
        int owner = __ffs(sel) - 1;  // k < n, so some lane holds rank k
        unsigned digit = 0, below = excl;
        if (lane == owner) {
            int j = 0;
#pragma unroll
            for (int t = 0; t < 7; t++)
                if (j == t && below + c[t] <= (unsigned)k) {
                    below += c[t];
                    j = t + 1;
                }
            digit = lane * 8 + j;
        }
        digit = __shfl_sync(0xffffffffu, digit, owner);
        below = __shfl_sync(0xffffffffu, below, owner);
        prefix |= digit << shift;
        mask |= 255u << shift;
        k -= (int)below;
        __syncwarp();
    }
    return prefix;
}

// what the pixel pass of examineiso hands to its finishing kernel
struct ExamRaw {
    double err[4];      // sums of err, err x^2, err y^2, err x y (the position errors)
    double fit[5];      // of the FWHM fit: s, sx, sy, sxx, sxy
    double tv, svar;    // flux, variance
    int ovf;
    float opeak, thresh0, mthresh;
    int peakpix, area;
};

struct AnaArgs {
    MomentRaw *raw;     // per-object scratch between the robust kernels
    int *biglist, *counts;  // objects summed by a whole block (list 5)
    ExamRaw *xraw;      // per-object scratch between the two examineiso kernels
    const float *cd, *sub, *back;
    const unsigned *opix;
    unsigned long long *last;   // completion key of every raw object
    ObjBufs O;
    FrameScalars *sc;
    int w, h, nbx, nby, bw, bh, nobj, minarea, clean_flag;
    const int *nobj_dev;  // the object count on the device (nobj is then the capacity), or null
    FastDiv wdiv;
    double gain, satur;
    const float *wvar;  // calibrated variance map, or null
    int wthr;           // analysis threshold follows the local rms
    double afac;        // ANALYSIS_THRESH
    int bp_thick;       // BACKPHOTO_THICK (used when O.dbkg is set)
    KronGeo *geo;       // the photometry's first ellipse and box
};

// Robust preanalysis of a deblended object over its final pixels
// (src/cuda/cudaanalyse.cu:1906-2124); objects of level 0 kept the values of
// the first preanalysis.  One warp per object sums over the pixels (a block
// over those of more than DA_WARP_MAX); the moments, ellipse and area
// correction are finished by k_robust_finish, one thread per object, so that
// the double-precision tail does not run on one lane of a warp.
__global__ void __launch_bounds__(AN_WARPS * 32, 3) k_analyse_robust(AnaArgs A) {
    sx_pdl();
    const int lane = threadIdx.x & 31;
    const int o = blockIdx.x * AN_WARPS + (threadIdx.x >> 5);
    if (o >= sx_count(A.nobj, A.nobj_dev) || A.O.level[o] == 0) return;
    const int n = A.O.n[o];
    if (n > DA_WARP_MAX) {
        if (lane == 0) A.biglist[atomicAdd(A.counts + 5, 1)] = o;
        return;
    }
    pix_moments_warp(A.cd, A.sub, A.opix + A.O.off[o], n, A.wdiv, A.w, A.O.dthr[o], A.raw + o);
}

__global__ void __launch_bounds__(AN_WARPS * 32, 2) k_analyse_robust_big(AnaArgs A) {
    sx_pdl();
    __shared__ PixBlock sh;
    const int nb = A.counts[5];
    for (int i = blockIdx.x; i < nb; i += gridDim.x) {
        const int o = A.biglist[i];
        pix_moments_block(A.cd, A.sub, A.opix + A.O.off[o], A.O.n[o], A.wdiv, A.w, A.O.dthr[o], sh, A.raw + o);
    }
}

__global__ void k_robust_finish(AnaArgs A) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = o < sx_count(A.nobj, A.nobj_dev) && A.O.level[o] != 0;
    const int oo = live ? o : 0;
    MomentRaw R = A.raw[oo];
    int flags = A.O.flags[oo];
    const double dth = A.O.dthr[oo];
    const double mxo = A.O.mx[oo], myo = A.O.my[oo];
    if (warp_each(live && R.ovf, o, [&](int q) {
            pix_moments_wide(A.cd, A.sub, A.opix + A.O.off[q], A.O.n[q], A.wdiv, A.w, A.raw + q);
        }))
        R = A.raw[oo];
    if (!live) return;
    if (R.ovf) atomicOr(&A.sc->status, SX_ST_RANGE);
    const int xmin = R.xmin, ymin = R.ymin, dnpix = R.dnpix, area2 = R.area2;
    if (xmin == 0 || R.xmax == A.w - 1 || ymin == 0 || R.ymax == A.h - 1) flags |= SX_OBJ_TRUNC;
    const float rv = R.rv, peak = R.peak, cpeak = R.cpeak;
    const double dthresh2 = (dth + peak) / 2.0;
    double rvd = rv, mx = R.mx, my = R.my;
    double mx2 = R.mx2, my2 = R.my2, mxy = R.mxy;
    double xm = mx / rvd, ym = my / rvd, xm2, ym2, xym;
    if (flags & SX_OBJ_MERGED) {
        double xn = mxo - xmin, yn = myo - ymin;
        xm2 = mx2 / rvd + xn * xn - 2 * xm * xn;
        ym2 = my2 / rvd + yn * yn - 2 * ym * yn;
        xym = mxy / rvd + xn * yn - xm * yn - xn * ym;
        xm = xn;
        ym = yn;
    } else {
        xm2 = mx2 / rvd - xm * xm;
        ym2 = my2 / rvd - ym * ym;
        xym = mxy / rvd - xm * ym;
    }
    double temp, temp2, theta, pmx2, pmy2, darea, t1t2;
    int singu = 0;
    if ((temp2 = xm2 * ym2 - xym * xym) < 0.00694) {
        xm2 += 0.0833333;
        ym2 += 0.0833333;
        temp2 = xm2 * ym2 - xym * xym;
        singu = 1;
    }
    if ((fabs(temp = xm2 - ym2)) > 0.0)
        theta = atan2(2.0 * xym, temp) / 2.0;
    else
        theta = SX_PI / 4.0;
    temp = sqrt(0.25 * temp * temp + xym * xym);
    pmy2 = pmx2 = 0.5 * (xm2 + ym2);
    pmx2 += temp;
    pmy2 -= temp;
    float a = (float)sqrt(pmx2), b = (float)sqrt(pmy2);
    float abcor;
    darea = (double)area2 - dnpix;
    t1t2 = dth / dthresh2;
    if (t1t2 > 0.0) {
        abcor = (darea < 0.0 ? darea : -1.0) / (2 * SX_PI * log(t1t2 < 1.0 ? t1t2 : 0.99) * a * b);
        if (abcor > 1.0) abcor = 1.0;
    } else
        abcor = 1.0;
    A.O.flags[o] = flags;
    A.O.singu[o] = singu;
    A.O.xmin[o] = xmin;
    A.O.xmax[o] = R.xmax;
    A.O.ymin[o] = ymin;
    A.O.ymax[o] = R.ymax;
    A.O.fdflux[o] = rv;
    A.O.dflux[o] = R.tv;
    A.O.fdpeak[o] = cpeak;
    A.O.dpeak[o] = peak;
    A.O.dnpix[o] = dnpix;
    A.O.mx[o] = xm + xmin;
    A.O.my[o] = ym + ymin;
    A.O.mx2[o] = xm2;
    A.O.my2[o] = ym2;
    A.O.mxy[o] = xym;
    A.O.a[o] = a;
    A.O.b[o] = b;
    A.O.theta[o] = theta * 180.0 / SX_PI;
    A.O.cxx[o] = (float)(ym2 / temp2);
    A.O.cyy[o] = (float)(xm2 / temp2);
    A.O.cxy[o] = (float)(-2 * xym / temp2);
    A.O.abcor[o] = abcor;
}

// an object's flux and variance with XSum (out of line: the rare path)
__device__ __noinline__ void exam_xsum(const AnaArgs &A, const unsigned *pix, int n, double &tv, double &svar,
                                       int &ovf) {
    XSum s, v;
    xs_init(s);
    xs_init(v);
    for (int i = threadIdx.x & 31; i < n; i += 32) {
        const unsigned p = pix[i];
        xs_add(s, A.sub[p]);
        if (A.wvar) xs_add(v, A.wvar[p]);
    }
    s = xs_warp_sum(s);
    v = xs_warp_sum(v);
    tv = xs_double(s);
    svar = xs_double(v);
    ovf = s.ovf | v.ovf;
}

// examineiso (src/cuda/cudaanalyse.cu:2176-2581) and the CLEAN threshold
// mthresh of every object.
__global__ void __launch_bounds__(AN_WARPS * 32, AN_MINB) k_examineiso(AnaArgs A) {
    sx_pdl();
    __shared__ __align__(16) unsigned hist[AN_WARPS][256];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int o = blockIdx.x * AN_WARPS + wid;
    if (o >= sx_count(A.nobj, A.nobj_dev)) return;
    const int n = A.O.n[o], off = A.O.off[o], w = A.w;
    const unsigned *pix = A.opix + off;
    const float dthresh = A.O.dthr[o], thresh = A.O.athr[o], gthresh = A.sc->thresh, backsig = A.sc->backsig;
    const double mxo = A.O.mx[o], myo = A.O.my[o];
    double dbacknoise2 = backsig * backsig;
    unsigned pk = 0u, bc = 0u, bp = 0xffffffffu;
    int area = 0;
    // flux and variance in double bins (hints: the object's peak, the frame's
    // noise), else with XSum
    const bool binned = n <= BIN_MAX_TERMS;
    bool ok = binned;
    const int W = bin_width(min(n, BIN_MAX_TERMS));
    const unsigned low_tv = bin_low(bs_order(A.O.dpeak[o]), W), low_var = bin_low(bs_order(backsig * backsig) + 8, W);
    Bin2 btv, bvar;
    bin_init(btv);
    bin_init(bvar);
    // each lane's largest filtered values, for the CLEAN threshold
    unsigned top[EX_TOP] = {};
    double esum = 0, emx2 = 0, emy2 = 0, emxy = 0;
    // two of a lane's pixels at a time, so that their loads overlap; added in
    // list order
    for (int i0 = lane; i0 < n; i0 += 64) {
        unsigned pp[2];
        float vv[2], cc[2], rr[2];
#pragma unroll
        for (int u = 0; u < 2; u++) pp[u] = i0 + 32 * u < n ? __ldg(pix + i0 + 32 * u) : 0u;
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const bool in = i0 + 32 * u < n;
            vv[u] = in ? __ldg(A.sub + pp[u]) : 0.0f;
            cc[u] = in ? __ldg(A.cd + pp[u]) : 0.0f;
            // with a weight map: the pixel's own analysis threshold and variance
            rr[u] = in && A.wvar ? __ldg(A.wvar + pp[u]) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (i0 + 32 * u >= n) break;
            const unsigned p = pp[u];
            const float pv = vv[u], cdpix = cc[u], pvar = rr[u];
            int iy = (int)fdiv(p, A.wdiv), ix = (int)p - iy * w;
            pk = max(pk, f2ord(pv));
            // first maximum of cd in raster order: max cd, then smallest index
            // (a lane's pixels come in that order); cd is 0 or positive, so its
            // bits sort like its values (a lane's first pixel counts even at 0)
            unsigned key = __float_as_uint(cdpix);
            if (key > bc || bp == 0xffffffffu) {
                bc = key;
                bp = p;
            }
#pragma unroll
            for (int k = 0; k < EX_TOP; k++) {
                const unsigned hi = max(top[k], key);
                key = min(top[k], key);
                top[k] = hi;
            }
            area += pv > sx_pix_thr(A.wthr, A.afac, pvar, gthresh);
            ok &= bin_add(btv, pv, low_tv, W);
            if (A.wvar) ok &= bin_add(bvar, pvar, low_var, W);
            double err = A.wvar ? (double)pvar : dbacknoise2;
            if (A.gain > 0.0 && cdpix > 0.0) err += cdpix / A.gain;
            double x = ix - mxo, y = iy - myo;
            esum += err;
            emx2 += err * x * x;
            emy2 += err * y * y;
            emxy += err * x * y;
        }
    }
    float peak = ord2f(__reduce_max_sync(0xffffffffu, pk));
    const unsigned cmax = __reduce_max_sync(0xffffffffu, bc);
    const unsigned peakpix = __reduce_min_sync(0xffffffffu, bc == cmax ? bp : 0xffffffffu);
    area = __reduce_add_sync(0xffffffffu, area);
    double tv, svar = 0.0;
    int ovf = 0;
    if (__all_sync(0xffffffffu, ok)) {
        const double v[4] = {btv.b0, btv.b1, bvar.b0, bvar.b1};
        const double r = warp_sum4(v, lane);  // lanes 0, 8, 16, 24
        tv = __shfl_sync(0xffffffffu, r, 0) + __shfl_sync(0xffffffffu, r, 8);
        if (A.wvar) svar = __shfl_sync(0xffffffffu, r, 16) + __shfl_sync(0xffffffffu, r, 24);
    } else {
        exam_xsum(A, pix, n, tv, svar, ovf);
    }
    const double errs[4] = {esum, emx2, emy2, emxy};
    const double err = warp_sum4(errs, lane);
    // the minarea-th largest filtered value: the lanes' largest are taken away
    // one by one, each lane offering its next; a lane asked for more than it
    // kept leaves it to the radix select
    float mthresh = 0.0f;
    if (A.clean_flag && n >= A.minarea) {
        unsigned kbits = 0u;
        bool found = A.minarea <= EX_TOP_AREA;
        int left = EX_TOP;
        for (int k = 0; found && k < A.minarea; k++) {
            if (__any_sync(0xffffffffu, left == 0 && n > 32 * EX_TOP)) {
                found = false;
                break;
            }
            kbits = __reduce_max_sync(0xffffffffu, top[0]);
            const unsigned has = __ballot_sync(0xffffffffu, top[0] == kbits);
            if (lane == __ffs(has) - 1) {
#pragma unroll
                for (int q = 0; q < EX_TOP - 1; q++) top[q] = top[q + 1];
                top[EX_TOP - 1] = 0u;
                left--;
            }
        }
        if (!found) kbits = warp_select(pix, n, A.cd, n - A.minarea, hist[wid]);
        mthresh = __uint_as_float(kbits) - dthresh;
    }
    // LOCAL photometry background (src/back.c:568 localback): the annulus mode,
    // subtracted from the flux, threshold, peak and FWHM fit (analyse.c
    // examineiso; the reference's GPU path keeps GLOBAL, dbkg = 0)
    const float dbkg = A.O.dbkg ? A.O.dbkg[o] : 0.0f;
    // isophotal thresholds: lane k < 8 evaluates threshold k, every lane reads all
    float othresh = thresh - dbkg;
    float opeak = peak - dbkg;
    float tk = 0.0f;
    if (opeak > 0.0 && othresh > 0.0 && lane < SX_NISO_)
        tk = othresh * pow((double)opeak / othresh, (double)lane / SX_NISO_);
    float threshs[SX_NISO_];
#pragma unroll
    for (int k = 0; k < SX_NISO_; k++) threshs[k] = __shfl_sync(0xffffffffu, tk, k);
    int iso[SX_NISO_];
#pragma unroll
    for (int k = 0; k < SX_NISO_; k++) iso[k] = 0;
    float thresh0 = opeak / 5.0;
    if (thresh0 < othresh) thresh0 = othresh;
    double s = 0, sx = 0, sy = 0, sxx = 0, sxy = 0;
    double sat = (double)(A.satur - (double)dbkg);
    for (int i = lane; i < n; i += 32) {
        unsigned p = __ldg(pix + i);
        float v = __ldg(A.sub + p);
        bool go = true;
#pragma unroll
        for (int k = 0; k < SX_NISO_; k++) {
            go = go && v > threshs[k];
            iso[k] += go;
        }
        double pv = v - (double)dbkg;
        if (thresh0 > 0.0 && pv > thresh0 && pv < sat) {
            int iy = (int)fdiv(p, A.wdiv), ix = (int)p - iy * w;
            double dx = ix - mxo, dy = iy - myo;
            double lpix = log(pv);
            double inverr2 = pv * pv;
            s += inverr2;
            double d2 = dx * dx + dy * dy;
            sx += d2 * inverr2;
            sxx += d2 * d2 * inverr2;
            sy += lpix * inverr2;
            sxy += lpix * d2 * inverr2;
        }
    }
    int iso_l = 0;  // lane k: iso[k]
#pragma unroll
    for (int k = 0; k < SX_NISO_; k++) {
        const int t = __reduce_add_sync(0xffffffffu, iso[k]);
        if (lane == k) iso_l = t;
    }
    const double fits[4] = {s, sx, sy, sxx};
    const double fit = warp_sum4(fits, lane);
    sxy = warp_sum_d(sxy);
    if (lane < SX_NISO_) A.O.iso[(size_t)o * SX_NISO_ + lane] = iso_l;
    ExamRaw &X = A.xraw[o];
    if ((lane & 7) == 0) {
        X.err[lane >> 3] = err;
        X.fit[lane >> 3] = fit;
    }
    if (lane == 1) {
        X.fit[4] = sxy;
        X.tv = tv;
        X.svar = svar;
    } else if (lane == 2) {
        X.ovf = ovf;
        X.opeak = opeak;
        X.thresh0 = thresh0;
        X.mthresh = mthresh;
        X.peakpix = (int)peakpix;
        X.area = area;
    }
}

// an object's flux and variance by one warp where XSum did not hold one of them
// (ovf), into its state; ovf: WideSum::bad
__device__ __noinline__ void exam_wide(const AnaArgs &A, int o) {
    ExamRaw &X = A.xraw[o];
    const unsigned *pix = A.opix + A.O.off[o];
    const int n = A.O.n[o];
    WideSum s, v;
    ws_init(s);
    ws_init(v);
    for (int i = threadIdx.x & 31; i < n; i += 32) {
        const unsigned p = pix[i];
        ws_add(s, A.sub[p]);
        if (A.wvar) ws_add(v, A.wvar[p]);
    }
    s = ws_warp_sum(s);
    v = ws_warp_sum(v);
    if ((threadIdx.x & 31) == 0) {
        X.tv = ws_double(s);
        X.svar = ws_double(v);
        X.ovf = s.bad | v.bad;
    }
}

// examineiso, per object: position errors, fluxes, FWHM fit, background
// (one thread per object, so that this double-precision tail does not run on
// one lane of a warp)
__global__ void k_examine_finish(const __grid_constant__ AnaArgs A) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = o < sx_count(A.nobj, A.nobj_dev);
    const int oo = live ? o : 0;
    ExamRaw X = A.xraw[oo];
    const int n = A.O.n[oo], w = A.w;
    const double mxo = A.O.mx[oo], myo = A.O.my[oo];
    const float backsig = A.sc->backsig;
    const double var = backsig * backsig;
    const float dbkg = A.O.dbkg ? A.O.dbkg[oo] : 0.0f;
    const int singu = A.O.singu[oo];
    const float fdflux = A.O.fdflux[oo], a = A.O.a[oo], b = A.O.b[oo];
    if (warp_each(live && X.ovf, o, [&](int q) { exam_wide(A, q); })) X = A.xraw[oo];
    if (!live) return;
    double esum = X.err[0], emx2 = X.err[1], emy2 = X.err[2], emxy = X.err[3];
    const double s = X.fit[0], sx = X.fit[1], sy = X.fit[2], sxx = X.fit[3], sxy = X.fit[4];
    const float opeak = X.opeak, thresh0 = X.thresh0, mthresh = X.mthresh;
    const int peakpix = X.peakpix, area = X.area;
    float bkg = back_at(A.back, A.nbx, A.nby, A.bw, A.bh, (int)(mxo + 0.5), (int)(myo + 0.5));
    {
        double flux2 = fdflux * fdflux;
        emx2 /= flux2;
        emy2 /= flux2;
        emxy /= flux2;
        esum *= 0.08333 / flux2;
        if (singu && (emx2 * emy2 - emxy * emxy) < esum * esum) {
            emx2 += esum;
            emy2 += esum;
        }
    }
    double tvd = X.tv;
    if (A.O.dbkg) tvd -= (double)((float)n * dbkg);   // int * float: a float product
    double sigtv = A.wvar ? X.svar : (double)n * var;
    if (A.gain > 0.0 && tvd > 0.0) sigtv += tvd / A.gain;
    float fwhm = 0.0f;
    if (thresh0 > 0.0) {
        double d = s * sxx - sx * sx;
        if (fabs(d) > 0.0) {
            double bb = -(s * sxy - sx * sy) / d, bmax;
            if (bb < (bmax = 1 / (13 * a * b))) bb = bmax;
            fwhm = (float)(1.6651 / sqrt(bb));
            if (fwhm > 0.0) fwhm -= 1 / (4 * fwhm);
        }
    }
    // completion order of the raw object: its last row and the first column on
    // it, over its objects' lists (a list's pixels on its last row come last)
    if (n > 0) {
        const unsigned *pix = A.opix + A.O.off[o];
        const int ymax = (int)fdiv(pix[n - 1], A.wdiv);
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if ((int)pix[mid] >= ymax * w)
                hi = mid;
            else
                lo = mid + 1;
        }
        atomicMax(A.last + A.O.root[o],
                  ((unsigned long long)(unsigned)ymax << 32) | (0xffffffffu - (pix[lo] - (unsigned)ymax * w)));
    }
    // the 6-sigma ellipse and box of the Kron radius (cudaanalyse.cu:318-357)
    kron_geo(A.w, A.h, mxo, myo, a, b, A.O.cxx[o], A.O.cyy[o], A.O.cxy[o], SX_KRON_NSIG, SX_KRON_NSIG * SX_KRON_NSIG,
             A.geo[o]);
    int py = (int)fdiv((unsigned)peakpix, A.wdiv);
    // the mode is added only where it was measured (src/back.c:659)
    A.O.bkg[o] = A.O.dbkg && A.O.lstat[o].nlevels >= 0 ? bkg + dbkg : bkg;
    A.O.peak[o] = opeak;
    A.O.peakx[o] = peakpix - py * w + 1;
    A.O.peaky[o] = py + 1;
    A.O.npix[o] = area;
    A.O.flux[o] = tvd;
    A.O.fluxerr[o] = sigtv;
    A.O.mthresh[o] = mthresh;
    A.O.pmx2[o] = emx2;
    A.O.pmy2[o] = emy2;
    A.O.pmxy[o] = emxy;
    A.O.fwhm[o] = fwhm;
    A.O.fdnpix[o] = n;
    if (X.ovf) atomicOr(&A.sc->status, SX_ST_RANGE);
}

// Object pixel lists, in raster order inside each object: an object's pixels
// are those of its box that the allocation map gives to it, read row by row.
// One warp reads a box of up to OL_WARP_MAX pixels; larger ones are cut into
// bands of rows for whole blocks (a branch that gathers a crowded core's
// outskirts can span the frame), counted first, then written.
constexpr int OL_THREADS = 256;
constexpr int OL_WARP_MAX = 4096;
constexpr int OL_CHUNK = 16384;      // box pixels per band (at least one row)
constexpr int OL_ITEMS = 1 << 17;    // bands per frame; objects beyond are left to their warps

struct ListItem {
    int o, y0, rows, first;  // object, first row, rows, the object's first band
};

// (row, column) of box pixel `start` and its step of `step` pixels
struct BoxWalk {
    int x, y, dx, dy, bw;
    __device__ __forceinline__ BoxWalk(int bw_, int start, int step) {
        bw = bw_;
        y = start / bw;
        x = start - y * bw;
        dy = step / bw;
        dx = step - dy * bw;
    }
    __device__ __forceinline__ void next() {
        x += dx;
        y += dy;
        if (x >= bw) {
            x -= bw;
            y++;
        }
    }
};

struct ListArgs {
    const int *alloc;
    ObjBufs O;
    int w, nobj;
    const int *nobj_dev;
    unsigned *opix;
    ListItem *items;
    int *icount;        // pixels of every band
    int *nitems;        // zero on entry
};

__global__ void __launch_bounds__(OL_THREADS) k_obj_lists(const ListArgs A) {
    sx_pdl();
    const int lane = threadIdx.x & 31, o = (blockIdx.x * OL_THREADS + threadIdx.x) >> 5;
    if (o >= sx_count(A.nobj, A.nobj_dev)) return;
    const int x0 = A.O.xmin[o], y0 = A.O.ymin[o], bw = A.O.xmax[o] - x0 + 1, bh = A.O.ymax[o] - y0 + 1;
    if (bw <= 0 || bh <= 0) return;
    const long long area = (long long)bw * bh;
    if (area > OL_WARP_MAX) {
        const int rows = max(1, OL_CHUNK / bw), nit = (bh + rows - 1) / rows;
        int c0 = 0;
        if (lane == 0) c0 = atomicAdd(A.nitems, nit);
        c0 = __shfl_sync(0xffffffffu, c0, 0);
        const bool fits = c0 >= 0 && c0 <= OL_ITEMS - nit;
        const int cend = c0 < 0 ? c0 : min(c0 + nit, OL_ITEMS);
        for (int c = c0 + lane; c < cend; c += 32) {
            ListItem it;
            it.o = fits ? o : -1;
            it.y0 = y0 + (c - c0) * rows;
            it.rows = min(rows, y0 + bh - it.y0);
            it.first = c0;
            A.items[c] = it;
        }
        if (fits) return;
    }
    unsigned *out = A.opix + A.O.off[o];
    BoxWalk q(bw, lane, 32);
    constexpr int AHEAD = 4;  // rows of 32 box pixels whose loads are in flight
    for (long long i0 = 0; i0 < area; i0 += 32 * AHEAD) {
        int a[AHEAD], p[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            p[k] = (y0 + q.y) * A.w + x0 + q.x;
            a[k] = q.y < bh ? __ldg(A.alloc + p[k]) : -1;
            q.next();
        }
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            const unsigned m = __ballot_sync(0xffffffffu, a[k] == o);
            if (a[k] == o) out[__popc(m & ((1u << lane) - 1u))] = (unsigned)p[k];
            out += __popc(m);
        }
    }
}

__global__ void __launch_bounds__(OL_THREADS) k_obj_list_count(const ListArgs A) {
    sx_pdl();
    __shared__ int s_n;
    const int n = min(*A.nitems, OL_ITEMS);
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        const ListItem it = A.items[c];
        if (it.o < 0) continue;
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        const int x0 = A.O.xmin[it.o], bw = A.O.xmax[it.o] - x0 + 1;
        BoxWalk q(bw, threadIdx.x, OL_THREADS);
        int k = 0;
        for (; q.y < it.rows; q.next()) k += __ldg(A.alloc + (size_t)(it.y0 + q.y) * A.w + x0 + q.x) == it.o;
        k = __reduce_add_sync(0xffffffffu, k);
        if ((threadIdx.x & 31) == 0 && k) atomicAdd(&s_n, k);
        __syncthreads();
        if (threadIdx.x == 0) A.icount[c] = s_n;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(OL_THREADS) k_obj_list_write(const ListArgs A) {
    sx_pdl();
    __shared__ int s_base, s_warp[2][OL_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int n = min(*A.nitems, OL_ITEMS);
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        const ListItem it = A.items[c];
        if (it.o < 0) continue;
        if (threadIdx.x == 0) s_base = A.O.off[it.o];
        __syncthreads();
        int before = 0;
        for (int k = it.first + threadIdx.x; k < c; k += OL_THREADS) before += A.icount[k];
        before = __reduce_add_sync(0xffffffffu, before);
        if (lane == 0 && before) atomicAdd(&s_base, before);
        __syncthreads();
        int base = s_base;
        const int x0 = A.O.xmin[it.o], bw = A.O.xmax[it.o] - x0 + 1, npix = bw * it.rows;
        BoxWalk q(bw, threadIdx.x, OL_THREADS);
        for (int i0 = 0, turn = 0; i0 < npix; i0 += OL_THREADS, turn ^= 1, q.next()) {
            const int p = (it.y0 + q.y) * A.w + x0 + q.x;
            const bool in = q.y < it.rows && __ldg(A.alloc + p) == it.o;
            const unsigned m = __ballot_sync(0xffffffffu, in);
            if (lane == 0) s_warp[turn][wid] = __popc(m);
            __syncthreads();
            int pre = 0, tot = 0;
#pragma unroll
            for (int k = 0; k < OL_THREADS / 32; k++) {
                if (k < wid) pre += s_warp[turn][k];
                tot += s_warp[turn][k];
            }
            if (in) A.opix[base + pre + __popc(m & ((1u << lane) - 1u))] = (unsigned)p;
            base += tot;
        }
        __syncthreads();
    }
}

int launch_obj_lists(const ListArgs &A, cudaStream_t st) {
    if (A.nobj <= 0) return 0;
    const unsigned per = OL_THREADS / 32;
    sx_launch(k_obj_lists, (A.nobj + per - 1) / per, OL_THREADS, 0, st, A);
    sx_launch(k_obj_list_count, dt_grid(A.nobj, 4), OL_THREADS, 0, st, A);
    sx_launch(k_obj_list_write, dt_grid(A.nobj, 4), OL_THREADS, 0, st, A);
    return 3;
}

void launch_analyse(const AnaArgs &A, cudaStream_t st) {
    if (A.nobj <= 0) return;
    const unsigned grid = (A.nobj + AN_WARPS - 1) / AN_WARPS;
    sx_launch(k_analyse_robust, grid, AN_WARPS * 32, 0, st, A);
    sx_launch(k_analyse_robust_big, dt_grid(A.nobj, 2), AN_WARPS * 32, 0, st, A);
    sx_launch(k_robust_finish, (unsigned)((A.nobj + 127) / 128), 128, 0, st, A);
    if (A.O.dbkg) {
        sx_launch(k_local_stat, (unsigned)((A.nobj + GW_WARPS - 1) / GW_WARPS), 32 * GW_WARPS, 0, st, A.sub, A.w,
                  A.h, A.bp_thick, A.O.xmin, A.O.xmax, A.O.ymin, A.O.ymax, A.nobj, A.nobj_dev, A.O.lstat, A.O.dbkg);
        sx_launch(k_local_guess, (unsigned)A.nobj, GUESS_THREADS, 0, st, A.sub, A.w, A.h, A.bp_thick, A.O.xmin,
                  A.O.xmax, A.O.ymin, A.O.ymax, A.nobj, A.nobj_dev, A.O.lstat, A.O.dbkg);
    }
    sx_launch(k_examineiso, grid, AN_WARPS * 32, 0, st, A);
    sx_launch(k_examine_finish, (unsigned)((A.nobj + 127) / 128), 128, 0, st, A);
}

}  // namespace sx
