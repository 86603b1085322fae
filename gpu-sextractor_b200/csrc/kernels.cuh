// kernels.cuh -- buffers and launchers shared by the stages of libsexgpu.
#pragma once
#include <atomic>
#include "common.cuh"

namespace sx {

struct MeshStat {
    float mean, sigma, lcut, hcut, qzero, qscale;
    int nlevels, npix;
};

struct BackBufs {
    MeshStat *ms;
    float *back, *sigma, *back2, *back3, *sigma3, *dback, *u;
    float *rownode, *rowdnode, *rowu;   // h x nbx each
    int *colk;                          // w
    float *coldx;                       // w
};

// per-root data (index = root id, first-pixel order)
struct RootBufs {
    int *size, *off;                    // pixels, their exclusive sums
    unsigned long long *last;           // completion order: last row << 32 | ~(first column on it), over its objects
    int *nkept, *objbase;
    float *dthresh, *thresh;            // smallest detection / analysis threshold of its pixels
    unsigned *peak;                     // f2ord of its largest filtered value
    int *npk, *nbkt, *nown;             // peaks, buckets, pixels of kept branches (deblending)
};

// deblending scratch (k_deblend.cu).  "Element" is a position in the list of
// all raw objects' pixels (raster order); the arrays "per raw object, from its
// offset" hold one entry per peak, bucket, kept branch or branch pixel, of
// which a raw object has no more than pixels.
struct DebBufs {
    // per element
    int *up;                            // towards its peak, then its peak, then its first representative
    unsigned char *lev;                 // level
    // per peak, at its element
    unsigned long long *rec, *evm;      // join record; levels of the joins it stands for
    int *boff, *pidx;                   // first bucket; index among its raw object's peaks
    int2 *kown;                         // kept branch it stands for: level + 1 (0: none), rank
    int *peaks;                         // every peak of the frame
    // per raw object, from its offset
    int *plist;                         // peaks
    int *bsz, *bmin;                    // buckets: pixels, smallest index,
    unsigned long long *acc;            // flux limbs
    int *olev;                          // kept branches in order: level
    unsigned *ownpix;                   // the branches' own pixels
    int *rest;                          // elements no branch owns
    // the same, for the raw objects whose joins are taken in global memory
    unsigned long long *kept, *g_evm;
    int *krep, *g_b0, *g_par, *g_nson, *g_label, *g_flags, *g_dlist, *g_elist;
    signed char *g_m;
    float *thr;                         // nthresh thresholds per raw object
    int *lists, *counts;                // raw objects by class of peaks (stride nroots); list lengths
    int *biglist;                       // objects whose pixels a whole block sums
};
// raw objects of at most this many peaks: joins taken by one warp, a block of
// 256 threads, a block of 512 (state in shared memory); more: a cluster of
// blocks on global memory
constexpr int DT_WARP_PEAKS = 32;
constexpr int DT_MID_PEAKS = 320;
constexpr int DT_BIG_PEAKS = 1536;
constexpr int DT_NCOUNTS = 8;
// objects of more pixels than this are summed by a block, not a warp
constexpr int DA_WARP_MAX = 1024;

// Persistent grids (deblending joins, subtract/filter tiles) are sized to
// the resident capacity divided by this (set per host thread; 1 by default,
// the batch workers take the "batch_grid_div" parameter of their context:
// measured on the 64-frame batch, whole-GPU grids with 8 workers were the
// fastest).
extern thread_local int sx_grid_div;
inline int sx_share(int grid) { return sx_grid_div > 1 ? (grid + sx_grid_div - 1) / sx_grid_div : grid; }

// A value per device computed on first use (resident grid sizes, device
// attributes), for the current device.  Several host threads (batch workers)
// may ask at once: the slots are atomic, and a value computed twice is
// computed the same way; 0 means "not computed yet".
struct DevCache {
    std::atomic<int> v[64];
    template <class F> int get(F compute) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= 64) return compute(dev);
        int x = v[dev].load(std::memory_order_relaxed);
        if (x == 0) {
            x = compute(dev);
            v[dev].store(x, std::memory_order_relaxed);
        }
        return x;
    }
};

// Kron boxes too large for one warp, summed by whole CTAs (k_post.cu)
constexpr int KR_CHUNK = 4096;     // box pixels per CTA work item (whole rows, at least one)
// Larger boxes than this are queued, unless the caller has set a size: the fewer
// objects there are, the sooner the longest box of a warp is what a pass waits
// for.  Photometry in ms by objects and size (fields of 0.006 sources a pixel up
// to 20,800 objects, of 0.0119 above; 780,000 are a mosaic of its own):
//              1024    2048    6144    8192 pixels
//     3,900   0.088   0.107   0.172   0.170
//     7,100   0.117   0.125   0.201   0.197
//    10,500   0.131   0.153   0.204   0.206
//    20,800   0.195   0.198   0.235   0.255
//    77,900   0.971   0.633   0.656   0.672   (the queue overflows at 1024)
//   116,000   1.305   0.906   0.914   0.924
//   146,000   1.497   1.099   1.113   1.113
//   190,000   1.762   1.414   1.386   1.399
//   780,000   13.7    11.4    10.46   10.5
// Neither line costs much where it lies: 1024 would be as good or better up to some
// 20,000 objects, and 2048 up to some 150,000.
inline int kr_warp_max(int nobj) { return nobj <= 8192 ? 1024 : nobj <= 131072 ? 2048 : 6144; }
// queued boxes and work items per pass: an eighth of the objects and 8 items
// each, at least 8192 boxes (a crowded mosaic queues 2% of its objects; with
// a fixed 8192 its warps were left with boxes of thousands of pixels)
inline int kr_items(int nobj) { return nobj / 8 > 8192 ? nobj / 8 : 8192; }
inline int kr_chunks(int nobj) { return 8 * kr_items(nobj); }

struct KronGeo {
    float cx2, cy2, cxy, klim2;
    int xmin, xmax, ymin, ymax;
    int flags;        // OBJ_APERT_PB where the frame cuts the box
};
struct KronItem {
    int o, c0, nch, rows;  // object, first work item, items (-1: summed by its warp), box rows per item
    int done;              // items finished
};
struct KronPart;
struct KronBufs {
    KronItem *item[2];
    int *chunk[2];     // work item -> queued box
    KronPart *part[2]; // work item -> partial sums
    int icap, ccap, warp_max;
};

// per-object data (index = object id: root order, then (level, label))
struct ObjBufs {
    int *root, *level, *n, *off;
    int *xmin, *xmax, *ymin, *ymax, *dnpix, *flags, *singu;
    float *fdflux, *dflux, *fdpeak, *dpeak, *node_dthresh;
    double *mx, *my, *mx2, *my2, *mxy;
    float *a, *b, *theta, *abcor, *cxx, *cyy, *cxy;
    int *npix, *peakx, *peaky, *iso;    // iso: 8 per object
    float *flux, *fluxerr, *peak, *bkg, *mthresh, *fwhm;
    double *pmx2, *pmy2, *pmxy;
    int *master, *fmaster, *number;
    float *flux_isocor, *fluxerr_isocor, *flux_aper, *fluxerr_aper, *mag_aper, *magerr_aper;
    float *kron, *flux_auto, *fluxerr_auto, *mag_auto, *magerr_auto;
    float *mag_iso, *magerr_iso, *fluxerr_iso;
    int *fdnpix;
    float *dthr, *athr;                 // the raw object's detection / analysis thresholds
    float *sprob;                       // CLASS_STAR
    float *dbkg;                        // LOCAL photometry background per object, or null (GLOBAL)
    MeshStat *lstat;                    // LOCAL annulus statistics
    float4 *aper;                       // every aperture: (flux, error, mag, mag error), naper per object
};

void launch_background(BackBufs &B, const float *img, const FrameParams &P, FrameScalars *d_sc, cudaStream_t st,
                       int &launches);
void launch_weight_mask(const float *img, const float *wmap, int wtype, float *imgm, long long n, cudaStream_t st);
void launch_weight_var(const BackBufs &B, const float *wmap, const FrameParams &P, float *ratio, float *wvar,
                       FrameScalars *d_sc, cudaStream_t st);

// The detection mask of one extraction: row-major mw x mh values on the
// device and on the host (per context, so that contexts extracting at the
// same time with different masks do not share it).
struct ConvMask {
    const float *dev;
    const float *host;
    int mw, mh;
};

void launch_sub_filter(const float *img, float *sub, float *cd, int *lab, int *cnt, const BackBufs &B,
                       const FrameParams &P, FrameScalars *d_sc, const float *d_var, const ConvMask &M,
                       cudaStream_t st, int &launches);

void launch_ccl(int *lab, int *cnt, const FrameParams &P, FrameScalars *d_sc, cudaStream_t st, int &launches);

struct MomentRaw;
// a kept branch's centre and shape, as the gatherup reads them (32 bytes)
struct __align__(16) GatherObj {
    int ix, iy;
    float fx, fy;
    float cxx, cyy, cxy, abcor;
};
// ... and a bound: the distance of a pixel 16 or more away is above lam times the
// square of its offset from (ix, iy) (lam 0: no bound)
struct __align__(16) GatherBound {
    int ix, iy;
    float lam;
    int pad;
};
struct DebArgs {
    const float *cd, *sub;
    const int *pos2idx;
    const unsigned *rpix;       // pixel of every element
    const unsigned *rid;        // raw object of every element
    RootBufs R;
    DebBufs D;
    ObjBufs O;
    MomentRaw *raw;             // per-object scratch of the preanalysis
    GatherObj *gobj;
    GatherBound *gbound;
    FrameScalars *sc;
    int *alloc;                 // W*H object id map (-1 elsewhere)
    unsigned *objkey;           // object of every element (~0: not a branch's own pixel)
    int nroots, nrootpix, nobj; // counts, or the capacities of the launches when the device counts are given
    const int *nroots_dev, *nrootpix_dev, *nobj_dev;
    int w, h, N, debminarea;
    FastDiv wdiv;
    double mincont;
    int loop_cap;               // > 0: cap on join walks and retries (failure tests); 0: the object's size
};

// merge trees and kept branches (R.nkept), then the objects; both return the
// number of kernels launched
int launch_deblend_tree(const DebArgs &A, cudaStream_t st);
int launch_deblend_assign(const DebArgs &A, cudaStream_t st);

}  // namespace sx
