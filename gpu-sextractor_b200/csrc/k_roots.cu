// k_roots.cu -- raw objects ("roots"): connected components of at least
// DETECT_MINAREA pixels, numbered in order of their first pixel, and their
// pixels compacted in raster order of the frame.  (The pixels are not grouped
// by raw object: the deblending works on all of them at once, and only the
// objects it ends with get pixel lists, k_analyse.cu.)
//
// Reference: src/cuda/cudadetection.cu:677-897 (compact_and_sort: sort by
// label, segment counts, minarea prune, consecutive relabel) and :899-1105
// (pre_analyse: fdpeak / fdflux per raw object).
#include "common.cuh"
#include "kernels.cuh"
#include "prim.cuh"

namespace sx {

// Each raw object's thresholds with a weight map: the smallest detection and
// analysis threshold of its pixels.  A threshold is a factor times the root of
// the variance, rounded, and so grows with the variance: the smallest variance
// of the object's pixels gives both.  It is found over the compacted pixels
// (positive floats order like their bits; in the warp first, since neighbouring
// pixels mostly share their raw object, then by an atomic where it would lower
// the value).  Two square roots in double and the labels of every pixel of the
// frame took 2.6 ms of a 16384 x 16384 frame.
__global__ void __launch_bounds__(256) k_root_minvar(const unsigned *__restrict__ erid,
                                                     const unsigned *__restrict__ epix, int n, const int *n_dev,
                                                     const float *__restrict__ wvar, int *__restrict__ rvar) {
    sx_pdl();
    const int j = blockIdx.x * 256 + threadIdx.x;
    n = sx_count(n, n_dev);
    if (blockIdx.x * 256 >= n) return;
    int r = -1, v = 0x7fffffff;
    if (j < n) {
        r = (int)erid[j];
        const float x = __ldg(wvar + epix[j]);
        if (x >= 0.0f) v = __float_as_int(fabsf(x));
    }
    const unsigned grp = __match_any_sync(0xffffffffu, r);
    if (r < 0) return;
    v = __reduce_min_sync(grp, v);
    if ((int)(threadIdx.x & 31) == __ffs(grp) - 1 && v < __ldcg(rvar + r)) atomicMin(rvar + r, v);
}

// the thresholds from those variances (in place of rvar); the fixed-point scale
// of the exact branch sums, sc->e0cd, becomes the exponent of the smallest
__global__ void k_root_thresholds(int nroots, const int *nroots_dev, double dfac, double afac, FrameScalars *sc,
                                  float *rdthr, float *rathr) {
    sx_pdl();
    nroots = sx_count(nroots, nroots_dev);
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    int e = 0x7fffffff;
    if (r < nroots) {
        const int v = reinterpret_cast<const int *>(rdthr)[r];
        float dt = __int_as_float(0x7f7f7f7f), at = dt;  // no usable variance
        if (v < 0x7f7f7f7f) {
            dt = sx_pix_thr(true, dfac, __int_as_float(v), 0.0f);
            at = sx_pix_thr(true, afac, __int_as_float(v), 0.0f);
            e = fexpo(dt);
        }
        rdthr[r] = dt;
        rathr[r] = at;
    }
    e = __reduce_min_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0 && e < *(volatile int *)&sc->e0cd) atomicMin(&sc->e0cd, e);
}

// ---- the raw-object numbering and the kept-pixel compaction as two scans
// whose inputs are computed on the fly (a root: lab[p] == p with at least
// minarea pixels; a kept pixel: its root has at least minarea pixels).  The
// tiles of SCAN_TILE pixels are those of the scan primitive (1024 threads, 4
// consecutive pixels each), so the per-tile counts of k_root_tile_counts and
// the in-tile prefixes of k_root_number / k_root_compact line up.
// The flags of a thread's SCAN_ITEMS (= 4) consecutive pixels from base (a
// multiple of 4), with one 16-byte load of their labels where all four are
// in the frame and the label array is 16-byte aligned.
__device__ __forceinline__ void root_kept_flags4(const int *__restrict__ lab, const int *__restrict__ cnt,
                                                 long long base, long long n, int minarea, int *isroot, int *kept,
                                                 int *l) {
    static_assert(SCAN_ITEMS == 4, "four pixels per thread");
    if (base + 3 < n && ((reinterpret_cast<uintptr_t>(lab) & 15) == 0)) {
        const int4 v = *reinterpret_cast<const int4 *>(lab + base);
        l[0] = v.x;
        l[1] = v.y;
        l[2] = v.z;
        l[3] = v.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) l[k] = base + k < n ? lab[base + k] : -1;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        kept[k] = l[k] >= 0 && cnt[l[k]] >= minarea;
        isroot[k] = kept[k] && l[k] == (int)(base + k);
    }
}

// per tile: number of roots and of kept pixels
__global__ void __launch_bounds__(SCAN_THREADS) k_root_tile_counts(const int *__restrict__ lab,
                                                                  const int *__restrict__ cnt, long long n,
                                                                  int minarea, int *__restrict__ troots,
                                                                  int *__restrict__ tkept) {
    sx_pdl();
    __shared__ int sh[32];
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    int cr = 0, ck = 0, r[SCAN_ITEMS], kp[SCAN_ITEMS], l[SCAN_ITEMS];
    root_kept_flags4(lab, cnt, base, n, minarea, r, kp, l);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        cr += r[k];
        ck += kp[k];
    }
    int tot;
    block_exclusive_scan(cr, sh, tot);
    if (threadIdx.x == 0) troots[blockIdx.x] = tot;
    block_exclusive_scan(ck, sh, tot);
    if (threadIdx.x == 0) tkept[blockIdx.x] = tot;
}

// roots numbered in raster order: rid at the root pixel, and size; their
// thresholds start as the global ones, or (minvar) as the largest variance
__global__ void __launch_bounds__(SCAN_THREADS) k_root_number(const int *__restrict__ lab, const int *__restrict__ cnt,
                                                             long long n, int minarea, const int *__restrict__ toff,
                                                             int *__restrict__ rid, int *__restrict__ rsize,
                                                             const FrameScalars *sc, bool minvar,
                                                             float *__restrict__ rdthr, float *__restrict__ rathr) {
    sx_pdl();
    __shared__ int sh[32];
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    int fr[SCAN_ITEMS], kp[SCAN_ITEMS], l[SCAN_ITEMS], c = 0;
    root_kept_flags4(lab, cnt, base, n, minarea, fr, kp, l);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) c += fr[k];
    const float dthr = minvar ? __int_as_float(0x7f7f7f7f) : sc->dthresh, athr = sc->thresh;
    int tot;
    int id = block_exclusive_scan(c, sh, tot) + toff[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (fr[k]) {
            const long long p = base + k;
            rid[p] = id;
            rsize[id] = cnt[p];
            rdthr[id] = dthr;
            rathr[id] = athr;
            id++;
        }
}

// kept pixels compacted in raster order: their positions, raw objects and the
// pixel -> element map (-1 elsewhere); the allocation map starts as "unassigned
// object pixel" / background
__global__ void __launch_bounds__(SCAN_THREADS) k_root_compact(const int *__restrict__ lab, const int *__restrict__ cnt,
                                                              long long n, int minarea, const int *__restrict__ toff,
                                                              const int *__restrict__ rid, unsigned *__restrict__ erid,
                                                              unsigned *__restrict__ epix, int *__restrict__ alloc,
                                                              int *__restrict__ pos2idx) {
    sx_pdl();
    __shared__ int sh[32];
    const long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
    int fk[SCAN_ITEMS], lb[SCAN_ITEMS], fr[SCAN_ITEMS], c = 0;
    root_kept_flags4(lab, cnt, base, n, minarea, fr, fk, lb);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) c += fk[k];
    int tot;
    int j = block_exclusive_scan(c, sh, tot) + toff[blockIdx.x];
    const bool vec = base + 3 < n && ((reinterpret_cast<uintptr_t>(alloc) | reinterpret_cast<uintptr_t>(pos2idx)) & 15) == 0;
    if (vec) {
        *reinterpret_cast<int4 *>(alloc + base) =
            make_int4(lb[0] >= 0 ? SX_ALLOC_OTHER : -1, lb[1] >= 0 ? SX_ALLOC_OTHER : -1,
                      lb[2] >= 0 ? SX_ALLOC_OTHER : -1, lb[3] >= 0 ? SX_ALLOC_OTHER : -1);
        int e[4], i = j;
#pragma unroll
        for (int k = 0; k < 4; k++) e[k] = fk[k] ? i++ : -1;
        *reinterpret_cast<int4 *>(pos2idx + base) = make_int4(e[0], e[1], e[2], e[3]);
    }
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        const long long p = base + k;
        if (p >= n) break;
        if (!vec) {
            alloc[p] = lb[k] >= 0 ? SX_ALLOC_OTHER : -1;
            pos2idx[p] = fk[k] ? j : -1;
        }
        if (fk[k]) {
            erid[j] = (unsigned)rid[lb[k]];
            epix[j] = (unsigned)p;
            j++;
        }
    }
}

}  // namespace sx
