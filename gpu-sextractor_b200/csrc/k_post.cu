// k_post.cu -- CLEAN, merging of cleaned objects, photometry and FLAGS of
// the surviving objects, catalogue order and output.
//
// Reference: src/clean.c:89-180 (the CLEAN test) and :234-287 (mergeobject);
// src/cuda/cudaclean.cu:120-175 (pairwise form); src/cuda/cudaanalyse.cu:62-98
// (isocor), :104-287 (aperture), :293-592 (Kron/AUTO with OBJ_CROWDED and
// OBJ_APERT_PB), :2874 (OBJ_SATUR); catalogue numbering src/scan.c:148-157.
#include "common.cuh"
#include "kernels.cuh"
#include "kron.cuh"
#include "pixmom.cuh"
#include "sexgpu.h"

namespace sx {

// ---------------------------------------------------------------------------
// CLEAN
// ---------------------------------------------------------------------------
constexpr float CL_CELL = 32.0f;

// per-object CLEAN record, stored in cell order so that a cell's objects are
// contiguous (src/clean.c:105-107 for amp and alpha)
struct CleanObj {
    double mx, my, amp, alpha;
    float a, fdflux, cxx, cyy, cxy, mthresh;
    int idx, pad;
};

__device__ __forceinline__ int clean_cell(double mx, double my, int gx, int gy) {
    int cx = (int)floor(mx / CL_CELL), cy = (int)floor(my / CL_CELL);
    cx = min(max(cx, 0), gx - 1);
    cy = min(max(cy, 0), gy - 1);
    return cy * gx + cx;
}

__global__ void k_clean_count(ObjBufs O, int n, const int *n_dev, int *cellcnt, int gx, int gy) {
    sx_pdl();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sx_count(n, n_dev)) return;
    O.master[i] = 0x7fffffff;
    atomicAdd(&cellcnt[clean_cell(O.mx[i], O.my[i], gx, gy)], 1);
}

__global__ void k_clean_pack(ObjBufs O, int n, const int *n_dev, double beta, const int *cellstart, int *cellcur,
                             CleanObj *packed, int gx, int gy) {
    sx_pdl();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sx_count(n, n_dev)) return;
    CleanObj c;
    double unitarea = SX_PI * O.a[i] * O.b[i];
    c.amp = O.fdflux[i] / (2 * unitarea * O.abcor[i]);
    double q = c.amp / O.dthr[i];
    c.alpha = ((beta == 1.0 ? q : pow(q, 1.0 / beta)) - 1) * unitarea / O.fdnpix[i];
    c.mx = O.mx[i];
    c.my = O.my[i];
    c.a = O.a[i];
    c.fdflux = O.fdflux[i];
    c.cxx = O.cxx[i];
    c.cyy = O.cyy[i];
    c.cxy = O.cxy[i];
    c.mthresh = O.mthresh[i];
    c.idx = i;
    c.pad = 0;
    int cell = clean_cell(c.mx, c.my, gx, gy);
    packed[cellstart[cell] + atomicAdd(&cellcur[cell], 1)] = c;
}

// src/clean.c:108-132 on the pair (p, q) with p.idx < q.idx (the kernel's
// orientation, src/cuda/cudaclean.cu:140-170)
__device__ __forceinline__ void clean_test(const CleanObj &p, const CleanObj &q, double beta, int *master) {
    float dx, dy, rlim;
    double val;
    dx = p.mx - q.mx;
    dy = p.my - q.my;
    rlim = p.a + q.a;
    rlim *= rlim;
    if (!(dx * dx + dy * dy < rlim * SX_CLEAN_ZONE * SX_CLEAN_ZONE)) return;
    if (p.fdflux < q.fdflux) {
        val = 1 + q.alpha * (q.cxx * dx * dx + q.cyy * dy * dy + q.cxy * dx * dy);
        if (val > 1.0 && ((float)(val < 1e10 ? q.amp * (beta == 1.0 ? 1.0 / val : pow(val, -beta)) : 0.0)
                          > p.mthresh))
            atomicMin(&master[p.idx], q.idx);
    } else {
        val = 1 + p.alpha * (p.cxx * dx * dx + p.cyy * dy * dy + p.cxy * dx * dy);
        if (val > 1.0 && ((float)(val < 1e10 ? p.amp * (beta == 1.0 ? 1.0 / val : pow(val, -beta)) : 0.0)
                          > q.mthresh))
            atomicMin(&master[q.idx], p.idx);
    }
}

// every pair closer than CLEAN_ZONE*(a_i+a_j) is tested once, by the object
// of larger a (lower index on ties), which searches 20*a around itself.  The
// objects are packed by cell in row-major cell order, so the cells of one row
// of the search box hold one contiguous range of objects: the lanes of a warp
// stride over that range (coalesced, balanced).  One block of CL_PAIR_WARPS
// warps per object, the warps taking the rows of its search box in turn, so
// that the few objects with large boxes do not leave one warp running long
// after the others.
constexpr int CL_PAIR_WARPS = 4;

__global__ void __launch_bounds__(CL_PAIR_WARPS * 32) k_clean_pairs(const CleanObj *__restrict__ packed, int n,
                                                                    const int *n_dev, double beta,
                                                                    const int *__restrict__ cellstart,
                                                                    int *master, int gx, int gy) {
    sx_pdl();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = blockIdx.x;
    if (k >= sx_count(n, n_dev)) return;
    const CleanObj me = packed[k];
    const double rad = 20.0 * me.a * 1.001 + 2.0;
    int x0 = max((int)floor((me.mx - rad) / CL_CELL), 0), x1 = min((int)floor((me.mx + rad) / CL_CELL), gx - 1);
    int y0 = max((int)floor((me.my - rad) / CL_CELL), 0), y1 = min((int)floor((me.my + rad) / CL_CELL), gy - 1);
    for (int cy = y0 + wid; cy <= y1; cy += CL_PAIR_WARPS) {
        const int t1 = __ldg(cellstart + cy * gx + x1 + 1);
        for (int t = __ldg(cellstart + cy * gx + x0) + lane; t < t1; t += 32) {
            const CleanObj o = packed[t];
            if (o.idx == me.idx) continue;
            if (o.a < me.a || (o.a == me.a && o.idx > me.idx)) {
                if (me.idx < o.idx)
                    clean_test(me, o, beta, master);
                else
                    clean_test(o, me, beta, master);
            }
        }
    }
}

// end of the master chain.  The chain of masters of a victim ends at a survivor
// after fewer than n steps (masters have smaller indices); cap: a smaller
// bound set for a failure test (0: n); running out sets SX_ST_LOOP.  Every
// survivor counts its victims (vcnt, zeroed before).
__global__ void k_clean_chain(ObjBufs O, int n, const int *n_dev, int *vcnt, int *status, int cap) {
    sx_pdl();
    n = sx_count(n, n_dev);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int m = O.master[i];
    if (m == 0x7fffffff) {
        O.fmaster[i] = -1;
        return;
    }
    const int lim = cap > 0 && cap < n ? cap : n;
    int it = 0;
    for (; it < lim && O.master[m] != 0x7fffffff; it++) m = O.master[m];
    if (O.master[m] != 0x7fffffff) atomicOr(status, SX_ST_LOOP);
    O.fmaster[i] = m;
    atomicAdd(vcnt + m, 1);
}

// The victims of every survivor, in index order: put into its range of vlist
// in any order (voff: exclusive sums of vcnt; vfill zeroed before), then each
// to its rank among them in vsort.  A victim compares itself with the others
// of its survivor only, usually a handful.
// The pixels of a victim belong to its survivor in the allocation map (one warp
// per object).
__global__ void k_victim_scatter(ObjBufs O, int n, const int *n_dev, const int *voff, int *vfill, int *vlist,
                                 const unsigned *opix, int *alloc) {
    sx_pdl();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= sx_count(n, n_dev)) return;
    const int m = O.fmaster[i];
    if (m < 0) return;
    if (lane == 0) vlist[voff[m] + atomicAdd(vfill + m, 1)] = i;
    const int off = O.off[i], cnt = O.n[i];
    for (int k = lane; k < cnt; k += 32) alloc[opix[off + k]] = m;
}

__global__ void k_victim_rank(ObjBufs O, int n, const int *n_dev, const int *voff, const int *vcnt, const int *vlist,
                              int *vsort) {
    sx_pdl();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= sx_count(n, n_dev)) return;
    const int m = O.fmaster[i];
    if (m < 0) return;
    const int v0 = voff[m], v1 = v0 + vcnt[m];
    int rank = 0;
    for (int k = v0; k < v1; k++) rank += vlist[k] < i;
    vsort[v0 + rank] = i;
}

// each survivor merges its victims in index order (src/clean.c:234-287)
__global__ void k_clean_merge(ObjBufs O, int n, const int *n_dev, const int *voff, const int *vcnt, const int *vsort) {
    sx_pdl();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= sx_count(n, n_dev)) return;
    const int v0 = voff[m], v1 = v0 + vcnt[m];
    for (int j = v0; j < v1; j++) {
        const int s = vsort[j];
        O.fdnpix[m] += O.fdnpix[s];
        O.dnpix[m] += O.dnpix[s];
        O.fdflux[m] += O.fdflux[s];
        O.dflux[m] += O.dflux[s];
        O.flux[m] += O.flux[s];
        O.fluxerr[m] += O.fluxerr[s];
        if (O.fdpeak[s] > O.fdpeak[m]) {
            O.fdpeak[m] = O.fdpeak[s];
            O.peakx[m] = O.peakx[s];
            O.peaky[m] = O.peaky[s];
        }
        if (O.dpeak[s] > O.dpeak[m]) O.dpeak[m] = O.dpeak[s];
        if (O.peak[s] > O.peak[m]) O.peak[m] = O.peak[s];
        if (O.xmin[s] < O.xmin[m]) O.xmin[m] = O.xmin[s];
        if (O.xmax[s] > O.xmax[m]) O.xmax[m] = O.xmax[s];
        if (O.ymin[s] < O.ymin[m]) O.ymin[m] = O.ymin[s];
        if (O.ymax[s] > O.ymax[m]) O.ymax[m] = O.ymax[s];
        O.flags[m] |= (O.flags[s] & (~(SX_OBJ_MERGED | SX_OBJ_CROWDED)));
    }
}

// ---------------------------------------------------------------------------
// photometry and FLAGS of the survivors
// ---------------------------------------------------------------------------
struct EndRaw;

struct EndArgs {
    EndRaw *raw;    // per-object state between the photometry kernels
    int *surv;      // per object: 1 for a survivor of CLEAN, 0 for a victim (k_end_finish)
    KronGeo *geo;   // per object: the next pass's ellipse and box (pass 1's from k_examine_finish)
    double2 *aper;  // per object and aperture: flux, variance
    const float *sub;
    const int *alloc;
    ObjBufs O;
    FrameScalars *sc;
    int w, h, n, mask_type;
    const int *n_dev;   // the object count on the device (n is then the capacity), or null
    double autoparam0, autoparam1, gain, zp, satur;
    int naper;                          // apertures (>= 1)
    double apertures[SEXGPU_MAXAPER];
    const float *wvar;  // calibrated variance map, or null
    KronBufs K;         // queued Kron boxes
    const sexgpu_nnw *nnw;  // CLASS_STAR network (device), or null
    double seeing, pixscale;
};

// src/cuda/cudaanalyse.cu:104-287 (computeaperflux, one aperture of diameter
// `diameter`).  The lanes of the warp evaluate 32 aperture pixels at a time
// (sub-pixel area, masked value) and put the terms of the three double sums in
// raster order in shared memory; one lane per sum then adds them one by one, so
// the rounding is the sequential loop's.  Lane 1 gets the variance, lane 2 the
// flux.
struct AperTerms {
    double t[3][32];  // area, variance, flux
};

__device__ __forceinline__ double aper_warp(const EndArgs &A, int o, double mx, double my, int &flags, double diameter,
                                            AperTerms &T) {
    const int lane = threadIdx.x & 31, w = A.w, h = A.h;
    const int corrflag = (A.mask_type == 2);
    const float backsig = A.sc->backsig;
    const double var = backsig * backsig;
    const float raper = diameter / 2.0;
    const float raper2 = raper * raper;
    const float rintlim = raper - 0.75;
    const float rintlim2 = (rintlim > 0.0) ? rintlim * rintlim : 0.0;
    const float rextlim2 = (raper + 0.75) * (raper + 0.75);
    const float scalex = 1.0 / SX_APER_OVERSAMP, scaley = scalex;
    const float scale2 = scalex * scaley;
    const float offsetx = 0.5 * (scalex - 1.0), offsety = 0.5 * (scaley - 1.0);
    int xmin = (int)(mx - raper + 0.499999);
    int xmax = (int)(mx + raper + 1.499999);
    int ymin = (int)(my - raper + 0.499999);
    int ymax = (int)(my + raper + 1.499999);
    if (xmin < 0) {
        xmin = 0;
        flags |= SX_OBJ_APERT_PB;
    }
    if (xmax > w) {
        xmax = w;
        flags |= SX_OBJ_APERT_PB;
    }
    if (ymin < 0) {
        ymin = 0;
        flags |= SX_OBJ_APERT_PB;
    }
    if (ymax > h) {
        ymax = h;
        flags |= SX_OBJ_APERT_PB;
    }
    double acc = 0.0;
    const int bw = xmax - xmin, bh = ymax - ymin, nn = bw * bh;
    if (bw <= 0 || bh <= 0) return 0.0;
    int yo = lane / bw, xo = lane - yo * bw;
    const int dyo = 32 / bw, dxo = 32 - dyo * bw;
    for (int base = 0; base < nn; base += 32) {
        bool in = false;
        float locarea = 0.0f;
        double pix = 0.0, pvar = var;
        if (yo < bh) {
            const int x = xmin + xo, y = ymin + yo;
            float dx = x - mx, dy = y - my, r2;
            if ((r2 = dx * dx + dy * dy) < rextlim2) {
                in = true;
                pix = A.sub[(size_t)y * w + x];
                int t = A.alloc[(size_t)y * w + x], x2, y2;
                if (r2 > rintlim2) {
                    dx += offsetx;
                    dy += offsety;
                    float dx2[SX_APER_OVERSAMP];
#pragma unroll
                    for (int k = 0; k < SX_APER_OVERSAMP; k++, dx += scalex) dx2[k] = dx * dx;
#pragma unroll
                    for (int sy = 0; sy < SX_APER_OVERSAMP; sy++, dy += scaley) {
                        const float dy2 = dy * dy;
#pragma unroll
                        for (int k = 0; k < SX_APER_OVERSAMP; k++)
                            if (dx2[k] + dy2 < raper2) locarea += scale2;
                    }
                } else
                    locarea = 1.0;
                // with a weight map: the variance of the pixel actually used,
                // 0 for a pixel replaced by 0 (src/photom.c:128-145)
                if (A.wvar) pvar = A.wvar[(size_t)y * w + x];
                if ((t >= 0 && t != o) || pix <= -SX_BIG) {
                    if (corrflag && (x2 = (int)(2 * mx + 0.49999 - x)) >= 0 && x2 < w &&
                        (y2 = (int)(2 * my + 0.49999 - y)) >= 0 && y2 < h &&
                        ((t = A.alloc[(size_t)y2 * w + x2]) == o || t == -1) &&
                        A.sub[(size_t)y2 * w + x2] > -SX_BIG) {
                        pix = A.sub[(size_t)y2 * w + x2];
                        if (A.wvar) pvar = A.wvar[(size_t)y2 * w + x2];
                    } else {
                        pix = 0.0;
                        if (A.wvar) pvar = 0.0;
                    }
                }
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        __syncwarp();
        if (in) {
            const int k = __popc(m & ((1u << lane) - 1u));
            T.t[0][k] = locarea;
            T.t[1][k] = pvar * locarea;
            T.t[2][k] = locarea * pix;
        }
        __syncwarp();
        if (lane < 3) {
            const int n = __popc(m);
            const double *t = T.t[lane];
#pragma unroll 4
            for (int k = 0; k < n; k++) acc += t[k];
        }
        xo += dxo;
        yo += dyo;
        if (xo >= bw) {
            xo -= bw;
            yo++;
        }
    }
    const double area = __shfl_sync(0xffffffffu, acc, 0);
    if (A.O.dbkg && lane == 2) acc -= area * (double)A.O.dbkg[o];
    return acc;
}

// ---------------------------------------------------------------------------
// AUTO / Kron photometry, src/cuda/cudaanalyse.cu:293-592.  Pass 1 sums
// r*pix and pix over the 6-sigma ellipse (kron radius), pass 2 the flux inside
// kron*ellipse.  Both sums are exact, so a box may be split and walked freely:
// a warp takes the boxes of up to KronBufs::warp_max pixels; larger ones (a
// kron radius that grew over a faint, elongated object can span the frame) are
// queued and cut into work items of whole rows for whole CTAs.  Geometry and
// the tails in double precision are done one thread per object between and
// after the passes.
//
// A warp walks a box in strips of 8 columns, 4 rows at a time: what depends on
// the column alone (dx, and with it two of the ellipse's three terms) is
// computed once a strip, and the strip is cut to the rows the ellipse can
// reach there (a widened root; every pixel is still tested).
// ---------------------------------------------------------------------------
// partial sums of a work item
struct KronPart {
    XSum s0, s1;  // pass 1: r*pix, pix;  pass 2: pix, variance
    int area, areab;
};

// per-object state between the photometry kernels
struct EndRaw {
    double s0, s1;        // the last pass's sums
    int area, areab, ovf;
    float kron;
    int flags, have2;
};

// a warp's sums: sum 0 in the even lanes, sum 1 in the odd ones, as bins or XSum
struct KronLane {
    bool binned;
    double t0, t1;
    XSum x;
};

// a warp's sums over rows y0 .. y1 - 1 and strips c0, c0 + cstep, ... of the
// box; area, areab in every lane.  BIN: in double bins (hints: the object's peak
// and, for r*pix, the ellipse's largest r, for the variances the frame's);
// false when a term did not fit.  XS: with XSum.  WIDE: with WideSum (t0: the
// sum of the lane's parity; x.ovf: WideSum::bad).
enum { KS_BIN, KS_XS, KS_WIDE };

template <int PASS, bool WVAR, int MODE>
__device__ __forceinline__ bool kron_strips(const EndArgs &A, int o, double mx, double my, const KronGeo &g, int y0,
                                            int y1, int c0, int cstep, KronLane &out, int &area_out, int &areab_out) {
    const int lane = threadIdx.x & 31, w = A.w, h = A.h;
    const int cl = lane & 7, rl = lane >> 3;
    const int corrflag = (A.mask_type == 2);
    constexpr bool TWO = PASS == 1 || WVAR, BIN = MODE == KS_BIN;
    const int W = bin_width(min((y1 - y0) * (g.xmax - g.xmin), BIN_MAX_TERMS));
    unsigned low0 = 0u, low1 = 0u;
    Bin2 b0, b1;
    XSum x0, x1;
    WideSum w0, w1;
    if (BIN) {
        const int peak = bs_order(A.O.peak[o]);
        low0 = bin_low(PASS == 1 ? peak + bs_order(sqrtf(g.klim2)) + 1 : peak, W);
        const float bsig = A.sc->backsig;
        low1 = bin_low(WVAR ? bs_order(bsig * bsig) + 8 : peak, W);
        bin_init(b0);
        bin_init(b1);
    } else if (MODE == KS_XS) {
        xs_init(x0);
        xs_init(x1);
    } else {
        ws_init(w0);
        ws_init(w1);
    }
    int area = 0, areab = 0;
    bool ok = true;
    for (int c = c0; g.xmin + 8 * c < g.xmax; c += cstep) {
        const int x = g.xmin + 8 * c + cl;
        const bool col = x < g.xmax;
        const float dx = x - mx;
        const float qa = g.cx2 * dx * dx, qb = g.cxy * dx;
        // rows where cy2 dy^2 + qb dy + qa <= klim2 can hold: the discriminant
        // widened by 1e-4 of its terms (they are off by 1e-6 of them), the
        // ends by 1.5 pixels
        int ylo = 0x7fffffff, yhi = -1;
        if (col) {
            const float t4 = 4.0f * g.cy2, disc = qb * qb - t4 * (qa - g.klim2) +
                                                  1e-4f * (qb * qb + fabsf(t4) * (fabsf(qa) + g.klim2));
            ylo = y0;
            yhi = y1 - 1;
            if (g.cy2 > 0.0f && disc < 0.0f) {
                yhi = -1;
                ylo = 0x7fffffff;
            } else if (g.cy2 > 0.0f && disc < 1e30f) {
                const float r = sqrtf(disc), i2 = 0.5f / g.cy2, fmy = (float)my;
                const float lo = fmy + (-qb - r) * i2 - 1.5f, hi = fmy + (r - qb) * i2 + 1.5f;
                if (lo > (float)ylo) ylo = (int)fminf(lo, 2e9f);
                if (hi < (float)yhi) yhi = (int)fmaxf(hi, -1.0f) + 1;
                yhi = min(yhi, y1 - 1);
            }
        }
        ylo = __reduce_min_sync(0xffffffffu, ylo);
        yhi = __reduce_max_sync(0xffffffffu, yhi);
        constexpr int U = 2;  // groups of 4 rows whose loads are in flight
        for (int yb = ylo; yb <= yhi; yb += 4 * U) {
            bool in[U];
            float r2[U], pixv[U], pvar[U];
            int tv[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int y = yb + 4 * u + rl;
                const float dy = y - my;
                r2[u] = qa + g.cy2 * dy * dy + qb * dy;
                in[u] = col && y <= yhi && r2[u] <= g.klim2;
                pixv[u] = pvar[u] = 0.0f;
                tv[u] = 0;
                if (in[u]) {
                    const size_t at = (size_t)y * w + x;
                    pixv[u] = __ldg(A.sub + at);
                    tv[u] = __ldg(A.alloc + at);
                    if (WVAR) pvar[u] = __ldg(A.wvar + at);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (!in[u]) continue;
                float pix = pixv[u];
                int t = tv[u];
                // (f > (float)-BIG as (double)f > -BIG, see seq_in)
                if (PASS == 1) {
                    if ((t == o || t == -1) & (pix > (float)-SX_BIG)) {
                        area++;
                        const float rp = sqrtf(r2[u]) * pix;
                        if (BIN) {
                            ok &= bin_add(b0, rp, low0, W);
                            ok &= bin_add(b1, pix, low1, W);
                        } else if (MODE == KS_XS) {
                            xs_add(x0, rp);
                            xs_add(x1, pix);
                        } else {
                            ws_add(w0, rp);
                            ws_add(w1, pix);
                        }
                    } else
                        areab++;
                } else {
                    area++;
                    float pv = pvar[u];
                    if ((t >= 0 && t != o) || pix <= (float)-SX_BIG) {
                        areab++;
                        const int y = yb + 4 * u + rl;
                        int x2, y2;
                        if (corrflag && (x2 = (int)(2 * mx + 0.49999 - x)) >= 0 && x2 < w &&
                            (y2 = (int)(2 * my + 0.49999 - y)) >= 0 && y2 < h &&
                            ((t = A.alloc[(size_t)y2 * w + x2]) == -1 || t == o) &&
                            A.sub[(size_t)y2 * w + x2] > (float)-SX_BIG) {
                            pix = A.sub[(size_t)y2 * w + x2];
                            if (WVAR) pv = A.wvar[(size_t)y2 * w + x2];
                        } else {
                            pix = 0.0;
                            pv = 0.0f;
                        }
                    }
                    if (BIN) {
                        ok &= bin_add(b0, pix, low0, W);
                        if (WVAR) ok &= bin_add(b1, pv, low1, W);
                    } else if (MODE == KS_XS) {
                        xs_add(x0, pix);
                        if (WVAR) xs_add(x1, pv);
                    } else {
                        ws_add(w0, pix);
                        if (WVAR) ws_add(w1, pv);
                    }
                }
            }
        }
    }
    if (BIN && !__all_sync(0xffffffffu, ok)) return false;
    if (BIN) {
        // lanes 8k .. 8k + 7: bin 0, 1 of sum 0, then of sum 1; each parity
        // fetches its two
        const double v[4] = {b0.b0, b0.b1, TWO ? b1.b0 : 0.0, TWO ? b1.b1 : 0.0};
        const double r = warp_sum4(v, lane);
        const int src = 16 * (lane & 1);
        out.t0 = __shfl_sync(0xffffffffu, r, src);
        out.t1 = __shfl_sync(0xffffffffu, r, src + 8);
    } else if (MODE == KS_XS) {
        x0 = xs_warp_sum(x0);
        x1 = xs_warp_sum(x1);
        out.x = lane & 1 ? x1 : x0;
    } else {
        w0 = ws_warp_sum(w0);
        w1 = ws_warp_sum(w1);
        out.t0 = ws_double(lane & 1 ? w1 : w0);
        out.x.ovf = w0.bad | w1.bad;
    }
    area_out = __reduce_add_sync(0xffffffffu, area);
    areab_out = __reduce_add_sync(0xffffffffu, areab);
    return true;
}

// the same with XSum, out of line: for terms the bins do not hold
template <int PASS, bool WVAR>
__device__ __noinline__ void kron_strips_xsum(const EndArgs &A, int o, double mx, double my, const KronGeo &g, int y0,
                                              int y1, int c0, int cstep, KronPart *out) {
    KronLane l;
    int area, areab;
    kron_strips<PASS, WVAR, KS_XS>(A, o, mx, my, g, y0, y1, c0, cstep, l, area, areab);
    out->s0 = l.x;
    out->area = area;
    out->areab = areab;
}

template <int PASS, bool WVAR>
__device__ __forceinline__ void kron_warp(const EndArgs &A, int o, double mx, double my, const KronGeo &g, int y0,
                                          int y1, int c0, int cstep, KronLane &l, int &area, int &areab) {
    // at most BIN_MAX_TERMS terms of the warp per bin
    l.binned = (long long)(y1 - y0) * (g.xmax - g.xmin) <= BIN_MAX_TERMS &&
               kron_strips<PASS, WVAR, KS_BIN>(A, o, mx, my, g, y0, y1, c0, cstep, l, area, areab);
    if (l.binned) return;
    KronPart p;
    kron_strips_xsum<PASS, WVAR>(A, o, mx, my, g, y0, y1, c0, cstep, &p);
    l.x = p.s0;
    area = p.area;
    areab = p.areab;
}

// an object's sums (lane 0: sum 0, lane 1: sum 1) into its state
__device__ __forceinline__ void kron_store(const EndArgs &A, int o, const KronLane &l, int area, int areab) {
    const int lane = threadIdx.x & 31;
    const double d = l.binned ? l.t0 + l.t1 : xs_double(l.x);
    const int ovf = __any_sync(0xffffffffu, !l.binned && lane < 2 && l.x.ovf);
    EndRaw &R = A.raw[o];
    if (lane == 0) {
        R.s0 = d;
        R.area = area;
        R.areab = areab;
        R.ovf = ovf;
    } else if (lane == 1)
        R.s1 = d;
}

// an object's sums over its whole box by one warp, where XSum did not hold one of
// them (R.ovf), into its state; R.ovf: WideSum::bad.  Called by the kernels
// that read the sums, so that the passes keep their registers.
template <int PASS, bool WVAR>
__device__ __noinline__ void kron_box_wide(const EndArgs &A, int o) {
    const int lane = threadIdx.x & 31;
    const KronGeo g = A.geo[o];
    KronLane l;
    int area, areab;
    kron_strips<PASS, WVAR, KS_WIDE>(A, o, A.O.mx[o], A.O.my[o], g, g.ymin, g.ymax, 0, 1, l, area, areab);
    EndRaw &R = A.raw[o];
    if (lane == 0) {
        R.s0 = l.t0;
        R.ovf = l.x.ovf;
    } else if (lane == 1)
        R.s1 = l.t0;
}

// Queue object o's pass-`pass` box (one thread).  False when the queue is
// full; its warp then sums the box.
__device__ bool kron_defer(const EndArgs &A, int pass, int o, const KronGeo &g) {
    const int bw = g.xmax - g.xmin, bh = g.ymax - g.ymin;
    const int rows = max(1, KR_CHUNK / bw), nch = (bh + rows - 1) / rows;
    const int k = atomicAdd(&A.sc->kitems[pass], 1), c0 = atomicAdd(&A.sc->kchunks[pass], nch);
    const bool ok = k < A.K.icap && c0 >= 0 && c0 <= A.K.ccap - nch;
    // this box's range of work items: its index, or -1 where it did not fit
    if (c0 >= 0)
        for (int c = c0; c < min(c0 + nch, A.K.ccap); c++) A.K.chunk[pass][c] = ok ? k : -1;
    if (k < A.K.icap) {
        KronItem it;
        it.o = o;
        it.c0 = c0;
        it.nch = ok ? nch : -1;
        it.rows = rows;
        it.done = 0;
        A.K.item[pass][k] = it;
    }
    return ok;
}

// The photometry's beginning, one thread per object: an error so far empties
// the frame (the host reads the status at its end), and the boxes of pass 1
// that are too large for a warp are queued (have2: 1 summed by its warp, 2
// queued, as k_kron_mid sets it for pass 2).
__global__ void k_end_begin(const __grid_constant__ EndArgs A) {
    sx_pdl();
    if (A.sc->status & SX_ST_STOP) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            A.sc->nroots = A.sc->nrootpix = A.sc->nobj = A.sc->nsurv = 0;
        return;
    }
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= sx_count(A.n, A.n_dev) || A.O.fmaster[o] >= 0) return;
    const KronGeo g = A.geo[o];
    A.raw[o].have2 = kron_npix(g) > A.K.warp_max && kron_defer(A, 0, o, g) ? 2 : 1;
}

// A pass over the boxes.  The first KR_BLOCKS blocks take the queued boxes' work
// items in turn, their warps an item's strips; the block that finishes a box's
// last item merges them.  The others take one object a warp: its apertures
// before pass 1, and its box unless it is queued.  A launch of its own for the
// queue began when the longest warp had ended, and cost 4 us where the queue
// was empty; with it and boxes of up to 8192 pixels a warp the photometry of
// 68,000 objects took 0.66 ms, of 3900 0.198, of 780,000 11.5, now 0.62, 0.086
// and 10.5.
constexpr int EO_WARPS = 4;
constexpr int KR_BLOCKS = 4 * 148;

template <int PASS, bool WVAR>
__device__ __forceinline__ void kron_merge(const EndArgs &A, int k, const KronItem &it, int c, KronLane &l, int area,
                                           int areab, KronPart *red, int &s_last) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (l.binned) {
        xs_init(l.x);
        xs_add_bins(l.x, l.t0, l.t1);
    }
    if (lane == 0) {
        red[wid].s0 = l.x;
        red[wid].area = area;
        red[wid].areab = areab;
    } else if (lane == 1)
        red[wid].s1 = l.x;
    __syncthreads();
    KronPart *part = A.K.part[PASS - 1];
    if (threadIdx.x == 0) {
        KronPart r = red[0];
        for (int q = 1; q < EO_WARPS; q++) {
            xs_merge(r.s0, red[q].s0);
            xs_merge(r.s1, red[q].s1);
            r.area += red[q].area;
            r.areab += red[q].areab;
        }
        part[c] = r;
        __threadfence();
        s_last = it.nch == 1 || atomicAdd(&A.K.item[PASS - 1][k].done, 1) == it.nch - 1;
    }
    __syncthreads();
    if (s_last && wid == 0) {
        __threadfence();
        XSum s0, s1;
        xs_init(s0);
        xs_init(s1);
        int a = 0, ab = 0;
        for (int j = lane; j < it.nch; j += 32) {
            const volatile KronPart *q = part + it.c0 + j;
            XSum t;
            t.v = ((__int128)((const volatile long long *)&q->s0.v)[1] << 64) |
                  (unsigned long long)((const volatile long long *)&q->s0.v)[0];
            t.e = q->s0.e;
            t.ovf = q->s0.ovf;
            xs_merge(s0, t);
            t.v = ((__int128)((const volatile long long *)&q->s1.v)[1] << 64) |
                  (unsigned long long)((const volatile long long *)&q->s1.v)[0];
            t.e = q->s1.e;
            t.ovf = q->s1.ovf;
            xs_merge(s1, t);
            a += q->area;
            ab += q->areab;
        }
        s0 = xs_warp_sum(s0);
        s1 = xs_warp_sum(s1);
        a = __reduce_add_sync(0xffffffffu, a);
        ab = __reduce_add_sync(0xffffffffu, ab);
        l.binned = false;
        l.x = lane & 1 ? s1 : s0;
        kron_store(A, it.o, l, a, ab);
    }
    __syncthreads();
}

template <int PASS, bool WVAR>
__global__ void __launch_bounds__(EO_WARPS * 32, 8) k_end_pass(const __grid_constant__ EndArgs A) {
    sx_pdl();
    __shared__ union {
        AperTerms terms[PASS == 1 ? EO_WARPS : 1];
        KronPart red[EO_WARPS];
    } sh;
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool queue = blockIdx.x < KR_BLOCKS;
    const int nc = queue ? min(A.sc->kchunks[PASS - 1], A.K.ccap) : 0;
    int c = blockIdx.x, k = -1, o = (int)(blockIdx.x - KR_BLOCKS) * EO_WARPS + wid;
    if (!queue) {
        if (o >= sx_count(A.n, A.n_dev) || A.O.fmaster[o] >= 0) return;
        if (PASS == 1) {
            int flags = A.O.flags[o];
            const double mx = A.O.mx[o], my = A.O.my[o];
            for (int q = 0; q < A.naper; q++) {
                const double acc = aper_warp(A, o, mx, my, flags, A.apertures[q], sh.terms[wid]);
                if (lane == 1 || lane == 2) (&A.aper[(size_t)o * A.naper + q].x)[2 - lane] = acc;
            }
            if (lane == 0) A.raw[o].flags = flags | A.geo[o].flags;
        }
        if (A.raw[o].have2 != 1) return;
    }
    for (;; c += KR_BLOCKS) {
        KronItem it;
        if (queue) {
            if (c >= nc) return;
            k = A.K.chunk[PASS - 1][c];
            if (k < 0) continue;
            it = A.K.item[PASS - 1][k];
            o = it.o;
        }
        const KronGeo g = A.geo[o];
        const int y0 = queue ? g.ymin + (c - it.c0) * it.rows : g.ymin, y1 = queue ? min(g.ymax, y0 + it.rows) : g.ymax;
        KronLane l;
        int area, areab;
        kron_warp<PASS, WVAR>(A, o, A.O.mx[o], A.O.my[o], g, y0, y1, queue ? wid : 0, queue ? EO_WARPS : 1, l, area,
                              areab);
        if (!queue) {
            kron_store(A, o, l, area, areab);
            return;
        }
        kron_merge<PASS, WVAR>(A, k, it, c, l, area, areab, sh.red, s_last);
    }
}

// kron radius from pass 1 and the pass-2 ellipse and box (cudaanalyse.cu:
// 385-440), one thread per object; no AUTO flux when pass 1 found no pixel
__global__ void k_kron_mid(const __grid_constant__ EndArgs A) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = o < sx_count(A.n, A.n_dev) && A.O.fmaster[o] < 0;
    EndRaw &R = A.raw[live ? o : 0];
    const int areab = R.areab, area = R.area + R.areab;
    double r1 = R.s0, v1 = R.s1;
    int ovf = R.ovf;
    if (warp_each(live && ovf, o, [&](int q) { kron_box_wide<1, false>(A, q); })) {
        r1 = R.s0;
        v1 = R.s1;
        ovf = R.ovf;
    }
    if (!live) return;
    if (ovf) atomicOr(&A.sc->status, SX_ST_RANGE);
    R.kron = 0.0f;
    R.have2 = 0;
    KronGeo g;
    if (!area) return;
    float kron;
    if (r1 > 0.0 && v1 > 0.0) {
        kron = A.autoparam0 * r1 / v1;
        if (kron < A.autoparam1) kron = A.autoparam1;
    } else
        kron = A.autoparam1;
    if ((float)areab / area > SX_CROWD_THRESHOLD) R.flags |= SX_OBJ_CROWDED;
    if (!kron_geo(A.w, A.h, A.O.mx[o], A.O.my[o], A.O.a[o], A.O.b[o], A.O.cxx[o], A.O.cyy[o], A.O.cxy[o], kron,
                  kron * kron, g))
        kron = 0.0;
    R.kron = kron;
    R.flags |= g.flags;
    A.geo[o] = g;
    // 1: summed by its warp, 2: queued
    R.have2 = kron_npix(g) > A.K.warp_max && kron_defer(A, 1, o, g) ? 2 : 1;
}

// catalogue columns of a survivor from its photometry sums: apertures, AUTO,
// ISOCOR and ISO fluxes, magnitudes and errors, FLAGS (one thread per object,
// so that this double-precision tail does not run on one lane of a warp)
__global__ void k_end_finish(const __grid_constant__ EndArgs A) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = o < sx_count(A.n, A.n_dev), victim = live && A.O.fmaster[o] >= 0;
    if (live) A.surv[o] = victim ? 0 : 1;
    const bool mine = live && !victim;
    for (int k = 0; mine && k < A.naper; k++) {
        const double2 ap = A.aper[(size_t)o * A.naper + k];
        const double tv = ap.x;
        double sigtv = ap.y;
        if (A.gain > 0.0 && tv > 0.0) sigtv += tv / A.gain;
        const float f = tv, fe = sqrt(sigtv), mg = tv > 0.0 ? -2.5 * log10(tv) + A.zp : 99.0,
                    me = tv > 0.0 ? 1.086 * sqrt(sigtv) / tv : 99.0;
        // the first aperture fills the catalogue columns; with several, every
        // one goes to O.aper
        if (k == 0) {
            A.O.flux_aper[o] = f;
            A.O.fluxerr_aper[o] = fe;
            A.O.mag_aper[o] = mg;
            A.O.magerr_aper[o] = me;
        }
        if (A.naper > 1) A.O.aper[(size_t)o * A.naper + k] = make_float4(f, fe, mg, me);
    }
    EndRaw R = A.raw[mine ? o : 0];
    if (warp_each(mine && R.have2 && R.ovf, o, [&](int q) {
            if (A.wvar)
                kron_box_wide<2, true>(A, q);
            else
                kron_box_wide<2, false>(A, q);
        }))
        R = A.raw[mine ? o : 0];
    if (!mine) return;
    const bool have2 = R.have2 != 0;
    int flags = R.flags;
    float kron = R.kron;
    const float backsig = A.sc->backsig;
    const double var = backsig * backsig;
    double tv, sigtv;
    if (have2) {
        const int area = R.area, areab = R.areab;
        if ((float)areab > SX_CROWD_THRESHOLD * area) flags |= SX_OBJ_CROWDED;
        tv = R.s0;
        sigtv = A.wvar ? R.s1 : (double)area * var;
        if (A.O.dbkg) tv -= area * (double)A.O.dbkg[o];
        if (A.gain > 0.0 && tv > 0.0) sigtv += tv / A.gain;
        if (R.ovf) atomicOr(&A.sc->status, SX_ST_RANGE);
    } else
        tv = sigtv = 0.0;
    const float flux = A.O.flux[o], fluxerr = A.O.fluxerr[o], dthresh = A.O.dthr[o];
    const int fdnpix = A.O.fdnpix[o];
    float flux_auto = tv, fluxerr_auto = sqrt(sigtv);
    if (tv <= 0.0) kron = 0.0;
    A.O.kron[o] = kron;
    A.O.flux_auto[o] = flux_auto;
    A.O.fluxerr_auto[o] = fluxerr_auto;
    A.O.mag_auto[o] = flux_auto > 0.0 ? -2.5 * log10(flux_auto) + A.zp : 99.0;
    A.O.magerr_auto[o] = flux_auto > 0.0 ? 1.086 * fluxerr_auto / flux_auto : 99.0;
    // isocor, src/cuda/cudaanalyse.cu:62-98
    double ati = (flux > 0.0) ? (fdnpix * dthresh / flux) : 0.0;
    if (ati > 1.0)
        ati = 1.0;
    else if (ati < 0.0)
        ati = 0.0;
    A.O.flux_isocor[o] = flux / (1.0 - 0.196099 * ati - 0.751208 * ati * ati);
    if (flux > 0.0) {
        double dati, sg;
        sg = fluxerr / (flux * flux);
        dati = fdnpix ? ati * sqrt(sg + 1.0 / fdnpix) : 0.0;
        dati = 0.196099 * dati + 0.751208 * 2 * ati * dati;
        A.O.fluxerr_isocor[o] = sqrt(sg + dati * dati) * flux;
    } else
        A.O.fluxerr_isocor[o] = sqrt(fluxerr);
    float fluxerr_iso = sqrt(fluxerr);
    A.O.fluxerr_iso[o] = fluxerr_iso;
    A.O.mag_iso[o] = flux > 0.0 ? -2.5 * log10(flux) + A.zp : 99.0;
    A.O.magerr_iso[o] = flux > 0.0 ? 1.086 * fluxerr_iso / flux : 99.0;
    if (A.O.peak[o] + A.O.bkg[o] >= A.satur) flags |= SX_OBJ_SATUR;
    A.O.flags[o] = flags;
}

// CLASS_STAR, src/cuda/cudaanalyse.cu:2901-2920 with the network response of
// :599-632 (src/neurro.c neurresp): inputs are log10 of the eight isophotal
// areas in seeing units and of FLUX_MAX over the threshold, plus log10 of the
// seeing; every layer applies the logistic function; double arithmetic.
__global__ void k_class_star(ObjBufs O, int n, const int *n_dev, const sexgpu_nnw *__restrict__ net, double fwhm,
                             double pixscale) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= sx_count(n, n_dev) || O.fmaster[o] >= 0) return;
    double fac2 = fwhm / pixscale;
    fac2 *= fac2;
    const float thresh = O.athr[o], peak = O.peak[o];
    double in[SEXGPU_NNW_NEURONS], nx[SEXGPU_NNW_NEURONS];
    const int *iso = O.iso + (size_t)o * SX_NISO_;
    int j = 0;
    in[j] = log10(iso[0] ? iso[0] / fac2 : 0.01);
    in[++j] = thresh > 0.0 ? log10(peak > 0.0 ? peak / thresh : 0.1) : -1.0;
    for (int i = 1; i < SX_NISO_; i++) in[++j] = log10(iso[i] ? iso[i] / fac2 : 0.01);
    in[++j] = log10(fwhm);
    const int last = net->nlayers - 1;
    for (int i = 0; i < net->nn[0]; i++) in[i] = in[i] * net->inscale[i] + net->inbias[i];
    for (int l = 0; l < last; l++) {
        for (int k = 0; k < net->nn[l + 1]; k++) {
            double sum = net->b[l][k];
            for (int i = 0; i < net->nn[l]; i++) sum += net->w[l][i][k] * in[i];
            nx[k] = 1.0 / (1.0 + exp(-sum));
        }
        for (int k = 0; k < net->nn[l + 1]; k++) in[k] = nx[k];
    }
    O.sprob[o] = (float)((in[0] - net->outbias[0]) / net->outscale[0]);
}

void launch_endobject(const EndArgs &E, int nobj, cudaStream_t st, int &launches) {
    const unsigned gw = KR_BLOCKS + (unsigned)((nobj + EO_WARPS - 1) / EO_WARPS),
                   gt = (unsigned)((std::max(nobj, 1) + 127) / 128);
    sx_launch(k_end_begin, gt, 128, 0, st, E);
    launches += 1;
    if (nobj <= 0) return;
    sx_launch(k_end_pass<1, false>, gw, EO_WARPS * 32, 0, st, E);
    sx_launch(k_kron_mid, gt, 128, 0, st, E);
    if (E.wvar)
        sx_launch(k_end_pass<2, true>, gw, EO_WARPS * 32, 0, st, E);
    else
        sx_launch(k_end_pass<2, false>, gw, EO_WARPS * 32, 0, st, E);
    sx_launch(k_end_finish, gt, 128, 0, st, E);
    launches += 4;
    if (E.nnw) {
        sx_launch(k_class_star, (unsigned)((nobj + 127) / 128), 128, 0, st, E.O, nobj, E.n_dev, E.nnw, E.seeing,
                  E.pixscale);
        launches += 1;
    }
}

// ---------------------------------------------------------------------------
// catalogue order and output
// ---------------------------------------------------------------------------
// Completion order: raw objects by the position of the first pixel on their
// last row, the survivors of one raw object in index order.  Raw objects have
// distinct such pixels, and their elements (raster order) come in the same
// order, so the place of a raw object's survivors is a count: those of the
// element tiles before its own, and those of the raw objects of its tile whose
// element is smaller (a linked list of a few).
constexpr int NO_TILE = 1024;  // elements; 3 to 20 raw objects of a crowded frame

struct OrderBufs {
    const int *pos;         // exclusive sums of the survivor flags
    int *tcnt, *thead;      // per tile: survivors (then their exclusive sums), list head + 1 (zeroed before)
    int *next, *elem, *ns;  // per raw object: list, its element, survivors
};

__global__ void k_order_roots(ObjBufs O, RootBufs R, const int *pos2idx, int w, int nroots, const int *nroots_dev,
                              OrderBufs Q) {
    sx_pdl();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= sx_count(nroots, nroots_dev)) return;
    const int K = R.nkept[r], ob = R.objbase[r];
    if (K <= 0) return;
    const int last = ob + K - 1, ns = Q.pos[last] + (O.fmaster[last] < 0) - Q.pos[ob];
    if (ns == 0) return;
    const unsigned long long key = R.last[r];
    const int e = pos2idx[(size_t)(key >> 32) * w + (0xffffffffu - (unsigned)key)], t = e / NO_TILE;
    Q.elem[r] = e;
    Q.ns[r] = ns;
    atomicAdd(Q.tcnt + t, ns);
    Q.next[r] = atomicExch(Q.thead + t, r + 1);
}

// NUMBER of every survivor and the objects in catalogue order (numbering 1:
// index order)
__global__ void k_order_objs(ObjBufs O, RootBufs R, int n, const int *n_dev, int numbering, OrderBufs Q,
                             unsigned *order) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= sx_count(n, n_dev)) return;
    if (O.fmaster[o] >= 0) {
        O.number[o] = 0;
        return;
    }
    int k = Q.pos[o];
    if (numbering == 0) {
        const int r = O.root[o], e = Q.elem[r], t = e / NO_TILE;
        k += Q.tcnt[t] - Q.pos[R.objbase[r]];
        for (int q = Q.thead[t]; q; q = Q.next[q - 1])
            if (Q.elem[q - 1] < e) k += Q.ns[q - 1];
    }
    O.number[o] = k + 1;
    order[k] = (unsigned)o;
}

__global__ void k_write_rows(ObjBufs O, const unsigned *vals, int ns, const int *ns_dev, sexgpu_object *rows) {
    sx_pdl();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= sx_count(ns, ns_dev)) return;
    int o = (int)vals[k];
    // built in a union with 16-byte words so that the row, padding bytes
    // included, is stored as whole words (rows are byte-for-byte reproducible)
    union {
        sexgpu_object o;
        uint4 v[sizeof(sexgpu_object) / 16];
    } u;
    static_assert(sizeof(sexgpu_object) % 16 == 0, "row size");
    for (int i = 0; i < (int)(sizeof(sexgpu_object) / 16); i++) u.v[i] = make_uint4(0, 0, 0, 0);
    sexgpu_object &q = u.o;
    q.number = k + 1;
    q.root = O.root[o];
    q.level = O.level[o];
    q.fdnpix = O.fdnpix[o];
    q.dnpix = O.dnpix[o];
    q.npix = O.npix[o];
    q.xmin = O.xmin[o];
    q.xmax = O.xmax[o];
    q.ymin = O.ymin[o];
    q.ymax = O.ymax[o];
    q.peakx = O.peakx[o];
    q.peaky = O.peaky[o];
    q.flags = O.flags[o];
    for (int i = 0; i < SX_NISO_; i++) q.iso[i] = O.iso[(size_t)o * SX_NISO_ + i];
    q.fdflux = O.fdflux[o];
    q.dflux = O.dflux[o];
    q.flux = O.flux[o];
    q.fluxerr = O.fluxerr[o];
    q.fdpeak = O.fdpeak[o];
    q.dpeak = O.dpeak[o];
    q.peak = O.peak[o];
    q.mx = O.mx[o];
    q.my = O.my[o];
    q.mx2 = O.mx2[o];
    q.my2 = O.my2[o];
    q.mxy = O.mxy[o];
    q.a = O.a[o];
    q.b = O.b[o];
    q.theta = O.theta[o];
    q.abcor = O.abcor[o];
    q.cxx = O.cxx[o];
    q.cyy = O.cyy[o];
    q.cxy = O.cxy[o];
    q.class_star = O.sprob ? O.sprob[o] : 0.0f;
    q.poserr_mx2 = O.pmx2[o];
    q.poserr_my2 = O.pmy2[o];
    q.poserr_mxy = O.pmxy[o];
    q.bkg = O.bkg[o];
    q.thresh = O.dbkg ? O.athr[o] - O.dbkg[o] : O.athr[o];
    q.dthresh = O.dthr[o];
    q.mthresh = O.mthresh[o];
    q.fwhm = O.fwhm[o];
    q.flux_iso = O.flux[o];
    q.fluxerr_iso = O.fluxerr_iso[o];
    q.mag_iso = O.mag_iso[o];
    q.magerr_iso = O.magerr_iso[o];
    q.flux_isocor = O.flux_isocor[o];
    q.fluxerr_isocor = O.fluxerr_isocor[o];
    q.flux_aper = O.flux_aper[o];
    q.fluxerr_aper = O.fluxerr_aper[o];
    q.mag_aper = O.mag_aper[o];
    q.magerr_aper = O.magerr_aper[o];
    q.kronfactor = O.kron[o];
    q.flux_auto = O.flux_auto[o];
    q.fluxerr_auto = O.fluxerr_auto[o];
    q.mag_auto = O.mag_auto[o];
    q.magerr_auto = O.magerr_auto[o];
    q.elong = q.a / q.b;
    q.ellip = 1 - q.b / q.a;
    q.polar = (q.a * q.a - q.b * q.b) / (q.a * q.a + q.b * q.b);
    // whole words: an assignment may store the members only and leave the
    // padding of the destination row as it was
    uint4 *dst = reinterpret_cast<uint4 *>(rows + k);
    for (int i = 0; i < (int)(sizeof(sexgpu_object) / 16); i++) dst[i] = u.v[i];
}

// every aperture of the catalogue rows, in catalogue order (naper per row)
__global__ void k_write_apers(ObjBufs O, const unsigned *order, int ns, int naper, float4 *out) {
    sx_pdl();
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= ns) return;
    const int o = (int)order[r];
    for (int k = 0; k < naper; k++)
        out[(size_t)r * naper + k] = naper > 1 ? O.aper[(size_t)o * naper + k]
                                               : make_float4(O.flux_aper[o], O.fluxerr_aper[o], O.mag_aper[o],
                                                             O.magerr_aper[o]);
}

// segmentation map: NUMBER of the owning object, 0 elsewhere; four pixels a
// thread (both maps are 16-byte aligned buffers of the context)
__global__ void __launch_bounds__(256) k_segmap(const int *alloc, const int *number, int *seg, long long npix) {
    sx_pdl();
    const long long p = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    if (p >= npix) return;
    auto num = [&](int a) { return a >= 0 && a != SX_ALLOC_OTHER ? __ldg(number + a) : 0; };
    if (p + 3 < npix) {
        const int4 a = *reinterpret_cast<const int4 *>(alloc + p);
        *reinterpret_cast<int4 *>(seg + p) = make_int4(num(a.x), num(a.y), num(a.z), num(a.w));
    } else {
        for (long long q = p; q < npix; q++) seg[q] = num(alloc[q]);
    }
}

}  // namespace sx
