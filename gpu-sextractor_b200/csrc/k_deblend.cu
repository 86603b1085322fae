// k_deblend.cu -- multi-threshold deblending of every raw object.
//
// Reference: src/cuda/cudadeblend.cu:199-217 (thresholds), :579-727 (one
// global CCL per sub-threshold level with host synchronisation), :1425-1776
// (cut_branch: MINCONT pruning, level by level with count read-backs),
// :1262-1360 (gatherup), src/cuda/cudaanalyse.cu:1686-1903 (preanalysis of the
// kept branches).
//
// The branches of a raw object are the connected components of its pixels at
// or above each threshold.  They form a merge tree, and only the levels at
// which components join matter to the MINCONT cut: between two joins a branch
// just grows.  So there is no sweep over the levels here.  All raw objects of
// the frame are worked on at once, one thread per pixel, whatever their sizes:
//
//  1. every pixel points at the largest of its 8 neighbours and itself
//     (larger filtered value, then smaller pixel index); following the
//     pointers leads to a local maximum, its peak, through pixels of
//     rising value, so at every level a pixel is in its peak's component;
//  2. two neighbours of different peaks join those peaks' components at the
//     lower of the two pixels' levels.  dt_join inserts such an edge into the
//     merge tree: of the two components' representative peaks the junior one
//     is recorded as joining the senior one at that level.  The records only
//     ever rise (atomicMax on level and target), an edge that a higher one
//     displaces is inserted again between what it connected, and so the
//     result does not depend on the order of the insertions;
//  3. a peak that stands for its component over several joins has one bucket
//     per stretch between them; each pixel adds itself (count, smallest
//     index, exact flux in fixed-scale limbs) to the bucket of the
//     representative and stretch it first appears in;
//  4. the joins of each raw object are taken from the highest level down
//     (one warp, one block with shared state, or a cluster of blocks on global
//     memory, by the number of peaks) and give the kept branches;
//  5. each pixel finds its kept branch by walking the joins from its peak;
//     the branches are pre-analysed over their own pixels, and the remaining
//     pixels gathered up.
//
// Raw objects with a single peak (93% of those of at most 64 pixels on a
// crowded frame) skip 2 to 4: they are one branch at level 0.
//
// What bounds it: the gathers of 1 to 3 (8 filtered values and about 10 map
// entries a pixel, L1/L2 hits) and the latency of the join loop in 4.
// Measured (deblend stage, plain form) against the level-by-level union-find
// of one block or warp per raw object that stood here before: 4096 x 4096
// crowded, 7.1 M pixels in 36,000 raw objects, 3.12 -> 1.34 ms; 1023 x 1021,
// 71,000 pixels in 1,400, where the largest object's levels were the time,
// 0.99 -> 0.115 ms; a 4096 x 4096 cluster with one raw object of about 2 M
// pixels, 64 levels, 791 -> 2.7 ms; 16384 x 16384, 108 M pixels, 38 -> 15.9 ms.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.cuh"
#include "pixmom.cuh"

namespace sx {

constexpr int DT_THREADS = 256;
// Fluxes of buckets: sum_k acc[k] * 2^(DT_RADIX k) in units of 2^(e0cd - 23),
// exact under atomics in any order.  A value of exponent e >= e0cd is a 24-bit
// mantissa shifted by e - e0cd <= 100 bits (more sets SX_ST_RANGE), so it falls
// into two neighbouring limbs; the 64-bit words hold the limbs of any frame.
constexpr int DT_LIMBS = 5;
constexpr int DT_RADIX = 27;        // 32 lanes' limbs add up in 32 bits
constexpr unsigned DT_LIMB_MASK = (1u << DT_RADIX) - 1u;

// walk and retry caps: no walk is longer than the raw object; or a smaller
// cap set for a failure test
__device__ __forceinline__ int dt_cap(const DebArgs &A) { return A.loop_cap > 0 ? A.loop_cap : (1 << 28); }

// a walk ran out of its cap: the joins may be incomplete, and nothing below
// relies on them (the frame ends with SX_ST_LOOP)
__device__ __forceinline__ bool dt_failed(const DebArgs &A) { return (A.sc->status & SX_ST_LOOP) != 0; }

// join record of a peak: (level of the join + 1) << 32 | the peak it joins; 0
// for the peak that stands for the whole raw object
__device__ __forceinline__ unsigned long long dt_pack(int level, int to) {
    return ((unsigned long long)(unsigned)(level + 1) << 32) | (unsigned)to;
}

// representative at level s of the component of peak a (read past L1: other
// threads raise the records)
__device__ __forceinline__ int dt_rep(const unsigned long long *rec, int a, int s, int cap, int *status) {
    for (int n = 0; n <= cap; n++) {
        const unsigned long long w = __ldcg(rec + a);
        if ((int)(w >> 32) <= s) return a;
        a = (int)(unsigned)w;
    }
    atomicOr(status, SX_ST_LOOP);
    return a;
}

// the components of peaks a and b join at level s.  Seniority: higher level,
// then smaller index (any strict order gives the same components; this one
// lets noise peaks join their star rather than the other way round).
__device__ __forceinline__ void dt_join(unsigned long long *rec, const unsigned char *lev, int a, int b, int s, int cap,
                                        int *status) {
    for (int n = 0; n <= cap; n++) {
        a = dt_rep(rec, a, s, cap, status);
        b = dt_rep(rec, b, s, cap, status);
        if (a == b) return;
        const int la = lev[a], lb = lev[b];
        const bool a_senior = la > lb || (la == lb && a < b);
        const int jun = a_senior ? b : a, sen = a_senior ? a : b;
        const unsigned long long mine = dt_pack(s, sen), old = atomicMax(rec + jun, mine);
        if (old >= mine) continue;  // joined meanwhile, at s or above: look again
        if (old == 0ull) return;
        // the lower join that was recorded holds between its target and the
        // component that jun is now part of
        a = sen;
        b = (int)(unsigned)old;
        s = (int)(old >> 32) - 1;
    }
    atomicOr(status, SX_ST_LOOP);
}

// ---- 1. peaks
// Neighbours below the raw object's threshold never win the comparison; with
// a weight map a pixel outside the object can, and then only the neighbours
// with a list index count (pixels of two raw objects are never adjacent).
__global__ void __launch_bounds__(DT_THREADS) k_dt_up(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    const bool in = j < sx_count(A.nrootpix, A.nrootpix_dev);
    bool peak = false;
    int r = -1;
    float c = 0.0f;
    if (in) {
        r = (int)A.rid[j];
        const int p = (int)A.rpix[j], y = (int)fdiv((unsigned)p, A.wdiv), x = p - y * A.w;
        c = A.cd[p];
        float best = c;
        int bp = p;
        const bool inner = x > 0 && y > 0 && x < A.w - 1 && y < A.h - 1;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int ddx[8] = {-1, 0, 1, -1, 1, -1, 0, 1}, ddy[8] = {-1, -1, -1, 0, 0, 1, 1, 1};
            const int nx = x + ddx[q], ny = y + ddy[q];
            if (!inner && (nx < 0 || ny < 0 || nx >= A.w || ny >= A.h)) continue;
            const int np = p + ddy[q] * A.w + ddx[q];
            const float v = __ldg(A.cd + np);
            if (v > best || (v == best && np < bp)) {
                best = v;
                bp = np;
            }
        }
        int u = j;
        if (bp != p) {
            u = __ldg(A.pos2idx + bp);
            if (u < 0) {
                best = c;
                bp = p;
                u = j;
#pragma unroll 1
                for (int q = 0; q < 9; q++) {
                    const int nx = x + q % 3 - 1, ny = y + q / 3 - 1;
                    if (q == 4 || nx < 0 || ny < 0 || nx >= A.w || ny >= A.h) continue;
                    const int np = ny * A.w + nx, e = __ldg(A.pos2idx + np);
                    const float v = __ldg(A.cd + np);
                    if (e >= 0 && (v > best || (v == best && np < bp))) {
                        best = v;
                        bp = np;
                        u = e;
                    }
                }
            }
        }
        A.D.up[j] = u;
        peak = u == j;
    }
    // the peaks of a raw object are counted and listed once per warp
    const unsigned pm = __ballot_sync(0xffffffffu, peak);
    if (!pm) return;
    const int lane = threadIdx.x & 31, lead = __ffs(pm) - 1;
    int base = 0;
    if (lane == lead) base = atomicAdd(&A.sc->npeaks, __popc(pm));
    base = __shfl_sync(0xffffffffu, base, lead);
    if (!peak) return;
    A.D.peaks[base + __popc(pm & ((1u << lane) - 1u))] = j;
    A.D.rec[j] = 0ull;
    A.D.evm[j] = 0ull;
    A.D.kown[j] = make_int2(0, 0);
    const unsigned grp = __match_any_sync(pm, r);
    const unsigned top = __reduce_max_sync(grp, f2ord(c));
    const int first = __ffs(grp) - 1;
    int i = 0;
    if (lane == first) {
        atomicMax(A.R.peak + r, top);
        i = atomicAdd(A.R.npk + r, __popc(grp));
    }
    i = __shfl_sync(grp, i, first) + __popc(grp & ((1u << lane) - 1u));
    A.D.plist[A.R.off[r] + i] = j;
    A.D.pidx[j] = i;
}

// Thresholds of every raw object (d0, then N-1 above it, src/cuda/
// cudadeblend.cu:199-217), one thread each; the first of a raw object also
// puts it on the list of its class: one peak (done here), up to 32 peaks (one
// warp), more (blocks).
__global__ void __launch_bounds__(DT_THREADS) k_dt_thresholds(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const long long t = (long long)blockIdx.x * DT_THREADS + threadIdx.x;
    const int r = (int)(t / A.N), i = (int)(t - (long long)r * A.N);
    if (r >= sx_count(A.nroots, A.nroots_dev)) return;
    const float d0 = A.R.dthresh[r], fdpeak = ord2f(A.R.peak[r]);
    float *thr = A.D.thr + (size_t)r * A.N;
    if (i > 0) {
        const double dt0 = d0, dp = fdpeak;
        thr[i] = dt0 * pow(dp / dt0, (double)i / A.N);
        return;
    }
    thr[0] = d0;
    const int off = A.R.off[r];
    // a term the fixed-scale sums cannot hold
    if (fexpo(fdpeak) - A.sc->e0cd > 100) atomicOr(&A.sc->status, SX_ST_RANGE);
    const int B = A.R.npk[r];
    if (B == 1) {
        A.R.nkept[r] = 1;
        A.D.olev[off] = 0;
        return;
    }
    const int k = B <= DT_WARP_PEAKS ? 0 : B <= DT_MID_PEAKS ? 1 : B <= DT_BIG_PEAKS ? 2 : 3;
    A.D.lists[(size_t)k * A.nroots + atomicAdd(A.D.counts + k, 1)] = r;
}

// level of every pixel (the highest threshold it reaches) and its peak
__global__ void __launch_bounds__(DT_THREADS) k_dt_level(const __grid_constant__ DebArgs A) {
    sx_pdl();
    __shared__ unsigned s_lp;
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    const int n = sx_count(A.nrootpix, A.nrootpix_dev);
    if (blockIdx.x * DT_THREADS >= n) return;
    if (threadIdx.x == 0) s_lp = 0u;
    __syncthreads();
    int lo = 0;
    if (j < n) {
        const int r = (int)A.rid[j];
        const float c = A.cd[A.rpix[j]];
        const float *thr = A.D.thr + (size_t)r * A.N;
        int hi = A.N - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (c >= __ldg(thr + mid))
                lo = mid;
            else
                hi = mid - 1;
        }
        A.D.lev[j] = (unsigned char)lo;
        if (A.R.npk[r] > 1) {
            // (a pointer read while its pixel's thread replaces it is one
            // to an ancestor either way)
            int u = A.D.up[j];
            const int cap = dt_cap(A);
            int k = 0;
            for (; k <= cap; k++) {
                const int v = A.D.up[u];
                if (v == u) break;
                u = v;
            }
            if (k > cap) atomicOr(&A.sc->status, SX_ST_LOOP);
            A.D.up[j] = u;
        }
    }
    const unsigned s = __reduce_add_sync(0xffffffffu, (unsigned)lo);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(&s_lp, s);
    __syncthreads();
    if (threadIdx.x == 0 && s_lp) atomicAdd(&A.sc->levpix, (unsigned long long)s_lp);
}

// ---- 2. joins.  An edge belongs to its lower pixel (level, then element): a
// pixel joins the peaks of all its higher neighbours at its own level, each
// different peak once.  (Taking the four backward or forward neighbours each
// at the lower level of the two meant twice as many walks.)
__global__ void __launch_bounds__(DT_THREADS) k_dt_edges(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    if (j >= sx_count(A.nrootpix, A.nrootpix_dev)) return;
    if (A.R.npk[A.rid[j]] <= 1) return;
    const int p = (int)A.rpix[j], y = (int)fdiv((unsigned)p, A.wdiv), x = p - y * A.w;
    const int a = A.D.up[j], l = A.D.lev[j];
    const bool inner = x > 0 && y > 0 && x < A.w - 1 && y < A.h - 1;
    int e[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int ddx[8] = {-1, 0, 1, -1, 1, -1, 0, 1}, ddy[8] = {-1, -1, -1, 0, 0, 1, 1, 1};
        const int nx = x + ddx[q], ny = y + ddy[q];
        e[q] = inner || (nx >= 0 && ny >= 0 && nx < A.w && ny < A.h) ? __ldg(A.pos2idx + p + ddy[q] * A.w + ddx[q]) : -1;
    }
    int b[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        b[q] = a;
        if (e[q] >= 0) {
            const int le = A.D.lev[e[q]];
            if (le > l || (le == l && e[q] > j)) b[q] = A.D.up[e[q]];
        }
    }
    unsigned todo = 0u;
#pragma unroll
    for (int q = 0; q < 8; q++) {
        bool again = b[q] == a;
#pragma unroll
        for (int k = 0; k < q; k++) again |= b[k] == b[q];
        if (!again) todo |= 1u << q;
    }
    // one join of every lane at a time, whichever neighbours they are
    const int cap = dt_cap(A);
    for (; todo; todo &= todo - 1u) {
        const int q = __ffs(todo) - 1;
        int t = b[0];
#pragma unroll
        for (int k = 1; k < 8; k++) t = q == k ? b[k] : t;
        dt_join(A.D.rec, A.D.lev, a, t, l, cap, &A.sc->status);
    }
}

// each join straight to the representative of that level, which gets a bit
// for it
__global__ void __launch_bounds__(DT_THREADS) k_dt_flatten(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    const int n = A.sc->npeaks;
    for (int i = blockIdx.x * DT_THREADS + threadIdx.x; i < n; i += gridDim.x * DT_THREADS) {
        const int d = A.D.peaks[i];
        const unsigned long long w = __ldcg(A.D.rec + d);
        if (w == 0ull) continue;
        const int m = (int)(w >> 32) - 1, q = dt_rep(A.D.rec, (int)(unsigned)w, m, dt_cap(A), &A.sc->status);
        // (a walk through d meanwhile passes the same level either way)
        if (q != (int)(unsigned)w) A.D.rec[d] = dt_pack(m, q);
        atomicOr(A.D.evm + q, 1ull << m);
    }
}

// buckets of every peak: one per stretch between the joins it stands for; a
// raw object of P pixels has at most P of them (peaks are never adjacent, and
// no more joins than peaks)
__global__ void __launch_bounds__(DT_THREADS) k_dt_buckets(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    const int n = A.sc->npeaks;
    for (int i = blockIdx.x * DT_THREADS + threadIdx.x; i < n; i += gridDim.x * DT_THREADS) {
        const int d = A.D.peaks[i], r = (int)A.rid[d];
        if (A.R.npk[r] <= 1) continue;
        const int nb = __popcll(A.D.evm[d]) + 1;
        const int b = A.R.off[r] + atomicAdd(A.R.nbkt + r, nb);
        A.D.boff[d] = b;
        for (int k = b; k < b + nb; k++) {
            A.D.bsz[k] = 0;
            A.D.bmin[k] = 0x7fffffff;
            for (int l = 0; l < DT_LIMBS; l++) A.D.acc[(size_t)k * DT_LIMBS + l] = 0ull;
        }
    }
}

constexpr int DT_FILL_RUNS = 12;

// ---- 3. every pixel into the bucket of the representative and stretch it
// first appears in; lanes of one bucket add up first (taking the buckets of
// the warp in turn: the lanes of each doing so by themselves diverged, 201 us
// instead of 150 for 7.1 M pixels)
__global__ void __launch_bounds__(DT_THREADS) k_dt_fill(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    const int n = sx_count(A.nrootpix, A.nrootpix_dev);
    if (blockIdx.x * DT_THREADS >= n) return;
    int bkt = -1, e = 0;
    unsigned lo = 0u, hi = 0u;
    int sh = 0;
    if (j < n) {
        const int r = (int)A.rid[j];
        if (A.R.npk[r] > 1) {
            const int l = A.D.lev[j];
            const int q = dt_rep(A.D.rec, A.D.up[j], l, dt_cap(A), &A.sc->status);
            A.D.up[j] = q;
            bkt = A.D.boff[q] + __popcll(A.D.evm[q] >> l);
            e = j;
            // (a term of exponent below e0cd cannot occur: every pixel is at
            // or above the smallest threshold; one more than 100 above it
            // has set SX_ST_RANGE)
            const unsigned u = __float_as_uint(A.cd[A.rpix[j]]);
            sh = min(max((int)((u >> 23) & 0xff) - 127 - A.sc->e0cd, 0), 100);
            const unsigned m = (u >> 23) & 0xff ? (u & 0x7fffffu) | 0x800000u : 0u;
            const int k = sh / DT_RADIX;
            const unsigned long long t = (unsigned long long)m << (sh - k * DT_RADIX);
            sh = k;  // first limb
            lo = (unsigned)t & DT_LIMB_MASK;
            hi = (unsigned)(t >> DT_RADIX);
        }
    }
    const int lane = threadIdx.x & 31;
    // many short runs of buckets (a noisy giant): every lane by itself
    const int prev = __shfl_up_sync(0xffffffffu, bkt, 1);
    if (__popc(__ballot_sync(0xffffffffu, lane == 0 || prev != bkt)) > DT_FILL_RUNS) {
        if (bkt >= 0) {
            unsigned long long *acc = A.D.acc + (size_t)bkt * DT_LIMBS + sh;
            atomicAdd(A.D.bsz + bkt, 1);
            atomicMin(A.D.bmin + bkt, e);
            if (lo) atomicAdd(acc, (unsigned long long)lo);
            if (hi) atomicAdd(acc + 1, (unsigned long long)hi);
        }
        return;
    }
    // one bucket (and first limb) of the warp at a time, every lane in step
    for (unsigned left = __ballot_sync(0xffffffffu, bkt >= 0); left;) {
        const int lead = __ffs(left) - 1;
        const int kb = __shfl_sync(0xffffffffu, bkt, lead), ks = __shfl_sync(0xffffffffu, sh, lead);
        const bool mine = bkt == kb && sh == ks;
        const unsigned grp = __ballot_sync(0xffffffffu, mine);
        const unsigned slo = __reduce_add_sync(0xffffffffu, mine ? lo : 0u),
                       shi = __reduce_add_sync(0xffffffffu, mine ? hi : 0u);
        if (lane == lead) {
            // (elements rise with the lane: this one has the smallest)
            unsigned long long *acc = A.D.acc + (size_t)bkt * DT_LIMBS + sh;
            atomicAdd(A.D.bsz + bkt, __popc(grp));
            atomicMin(A.D.bmin + bkt, e);
            if (slo) atomicAdd(acc, (unsigned long long)slo);
            if (shi) atomicAdd(acc + 1, (unsigned long long)shi);
        }
        left &= ~grp;
    }
}

// ---- 4. the cut
// a flux from its limbs, rounded once to double and then to float as every
// exact sum is.  It may have up to 155 bits (values 100 binary orders above the
// threshold, as blank pixels give under a mask with negative taps): above 127
// the two lowest limbs only count as "not zero", far below the last bit kept.
template <class T>
__device__ __forceinline__ float dt_flux(const T *a, int e0) {
    unsigned l[DT_LIMBS];
    unsigned long long c = 0ull;
#pragma unroll
    for (int k = 0; k < DT_LIMBS; k++) {
        c += a[k];
        l[k] = (unsigned)c & DT_LIMB_MASK;
        c >>= DT_RADIX;
    }
    const bool wide = c != 0ull || (l[DT_LIMBS - 1] >> (126 - DT_RADIX * (DT_LIMBS - 1))) != 0u;
    XSum s;
    __int128 v = wide ? (__int128)c : 0;
#pragma unroll
    for (int k = DT_LIMBS - 1; k >= 2; k--) v = (v << DT_RADIX) + l[k];
    if (wide)
        v |= (l[0] | l[1]) != 0u;
    else
        v = (((v << DT_RADIX) + l[1]) << DT_RADIX) + l[0];
    s.v = v;
    s.e = e0 + (wide ? 2 * DT_RADIX : 0);
    s.ovf = 0;
    return xs_float(s);
}

// state of one raw object's joins: in shared memory, or in global memory for
// the largest (volatile: there, other threads of the block change it by
// atomics, which pass L1 by)
struct DtState {
    volatile unsigned long long *acc, *evm;
    volatile int *bsz, *bmin, *b0, *par, *nson, *label, *flags;
    volatile signed char *m;  // level of its join, -1 for the last
};
constexpr int DT_OK = 1, DT_OKC = 2, DT_FLAG = 4;

// peak i stands for a component of level L + 1 that takes part in a join at
// level L: its stretch k is complete, so that bucket goes to its total (its
// first bucket), and the component's label and MINCONT flag at level L + 1 are
// known (:1425-1776)
__device__ __forceinline__ void dt_child(const DtState &S, int i, int k, const float thr, int debminarea, double value0,
                                         int e0) {
    // (every load is issued before the first is used: in global memory each wait
    // is most of a microsecond)
    const int b = S.b0[i], f = S.flags[i];
    int size = S.bsz[b], mn = S.bmin[b];
    unsigned long long v[DT_LIMBS];
#pragma unroll
    for (int l = 0; l < DT_LIMBS; l++) v[l] = S.acc[(size_t)b * DT_LIMBS + l];
    if (k > 0) {
        const int size2 = S.bsz[b + k], mn2 = S.bmin[b + k];
        unsigned long long u[DT_LIMBS];
#pragma unroll
        for (int l = 0; l < DT_LIMBS; l++) u[l] = S.acc[(size_t)(b + k) * DT_LIMBS + l];
        size += size2;
        mn = min(mn, mn2);
        S.bsz[b] = size;
        S.bmin[b] = mn;
#pragma unroll
        for (int l = 0; l < DT_LIMBS; l++)
            if (u[l]) {
                v[l] += u[l];
                S.acc[(size_t)b * DT_LIMBS + l] = v[l];
            }
    }
    bool flag = false;
    if (size >= debminarea) {
        const float lhs = dt_flux(v, e0) - thr * (float)(unsigned)size;
        flag = lhs > value0;
    }
    S.label[i] = mn;
    const int ok = f & DT_OK;
    S.flags[i] = ok | (ok ? DT_OKC : 0) | (flag ? DT_FLAG : 0);
    S.nson[i] = flag;
}

// peak i ends here: what it stood for goes to the peak it joins
__device__ __forceinline__ void dt_merge(const DtState &S, int i) {
    const int q = S.par[i], b = S.b0[i], f = S.flags[i];
    const int bq = S.b0[q], size = S.bsz[b], mn = S.bmin[b];
    unsigned long long v[DT_LIMBS];
#pragma unroll
    for (int l = 0; l < DT_LIMBS; l++) v[l] = S.acc[(size_t)b * DT_LIMBS + l];
    if (f & DT_FLAG) atomicAdd((int *)S.nson + q, 1);
    if (!(f & DT_OK)) atomicAnd((int *)S.flags + q, ~DT_OKC);
    atomicAdd((int *)S.bsz + bq, size);
    atomicMin((int *)S.bmin + bq, mn);
#pragma unroll
    for (int l = 0; l < DT_LIMBS; l++)
        if (v[l]) atomicAdd((unsigned long long *)S.acc + (size_t)bq * DT_LIMBS + l, v[l]);
}

// the same for a whole warp (i < 0: nothing), where most joins of a level go to
// one component: the lanes of the first lane's target add up first (an atomic
// of each on the same few words was most of the time of a raw object of 2 M
// pixels)
__device__ __forceinline__ void dt_merge_warp(const DtState &S, int i) {
    const int lane = threadIdx.x & 31;
    const int q = i >= 0 ? S.par[i] : -1;
    const unsigned all = __ballot_sync(0xffffffffu, i >= 0);
    if (!all) return;
    const int lead = __ffs(all) - 1, q0 = __shfl_sync(0xffffffffu, q, lead);
    const bool mine = q == q0;
    const unsigned grp = __ballot_sync(0xffffffffu, mine);
    if (__popc(grp) >= 4) {
        int b = 0, f = DT_OK, size = 0, mn = 0x7fffffff;
        unsigned long long lim[DT_LIMBS] = {};
        if (mine) {
            b = S.b0[i];
            f = S.flags[i];
            size = S.bsz[b];
            mn = S.bmin[b];
#pragma unroll
            for (int l = 0; l < DT_LIMBS; l++) lim[l] = S.acc[(size_t)b * DT_LIMBS + l];
        }
        size = __reduce_add_sync(0xffffffffu, size);
        mn = __reduce_min_sync(0xffffffffu, mn);
        const int flagged = __popc(__ballot_sync(0xffffffffu, mine && (f & DT_FLAG)));
        const bool split = __any_sync(0xffffffffu, !(f & DT_OK));
        const int bq = S.b0[q0];
#pragma unroll
        for (int l = 0; l < DT_LIMBS; l++) {
            unsigned long long v = lim[l];
            if (!__any_sync(0xffffffffu, v != 0ull)) continue;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == lead) atomicAdd((unsigned long long *)S.acc + (size_t)bq * DT_LIMBS + l, v);
        }
        if (lane == lead) {
            if (flagged) atomicAdd((int *)S.nson + q0, flagged);
            if (split) atomicAnd((int *)S.flags + q0, ~DT_OKC);
            atomicAdd((int *)S.bsz + bq, size);
            atomicMin((int *)S.bmin + bq, mn);
        }
        if (mine) i = -1;
    }
    if (i >= 0) dt_merge(S, i);
}

// is the child i of the join at (peak q) kept as an object of its own
__device__ __forceinline__ bool dt_kept(const DtState &S, int i, int q) {
    return (S.flags[i] & (DT_OK | DT_FLAG)) == (DT_OK | DT_FLAG) && S.nson[q] > 1;
}

// bytes of shared state per peak, and of the whole for a block of C peaks
constexpr int DT_SBYTES = 2 * DT_LIMBS * 8 + 8 + 8 + 2 * 4 + 2 * 4 + 4 * 6 + 4;
__host__ __device__ constexpr size_t dt_smem(int cap) { return (size_t)cap * DT_SBYTES; }

template <int NT>
__device__ __forceinline__ void dt_sync() {
    if (NT == 32)
        __syncwarp();
    else
        __syncthreads();
}

// raw objects of at most cap peaks: NT threads (32: one warp), state in smem
template <int NT>
__device__ __forceinline__ void dt_cut(const DebArgs &A, const int r, unsigned char *smem, const int cap,
                                       unsigned long long *s_all) {
    // s_all: 8 words shared by the NT threads
    const int tid = NT == 32 ? (threadIdx.x & 31) : threadIdx.x;
    const int off = A.R.off[r], B = A.R.npk[r], NB = A.R.nbkt[r];
    const int e0 = A.sc->e0cd;
    const float *thr = A.D.thr + (size_t)r * A.N;
    DtState S;
    unsigned long long *acc = reinterpret_cast<unsigned long long *>(smem);
    unsigned long long *evm = acc + 2 * cap * DT_LIMBS, *keys = evm + cap;
    int *bsz = reinterpret_cast<int *>(keys + cap), *bmin = bsz + 2 * cap, *b0 = bmin + 2 * cap, *par = b0 + cap,
        *nson = par + cap, *label = nson + cap, *flags = label + cap, *kloc = flags + cap;
    signed char *m = reinterpret_cast<signed char *>(kloc + cap);
    S.acc = acc;
    S.evm = evm;
    S.bsz = bsz;
    S.bmin = bmin;
    S.b0 = b0;
    S.par = par;
    S.nson = nson;
    S.label = label;
    S.flags = flags;
    S.m = m;
    if (tid < 8) s_all[tid] = 0ull;  // total flux limbs, levels with joins, kept
    dt_sync<NT>();
    unsigned long long tot[DT_LIMBS], all = 0ull;
    for (int l = 0; l < DT_LIMBS; l++) tot[l] = 0ull;
    for (int k = tid; k < NB; k += NT) {
        bsz[k] = A.D.bsz[off + k];
        bmin[k] = A.D.bmin[off + k];
        for (int l = 0; l < DT_LIMBS; l++) {
            const unsigned long long v = A.D.acc[(size_t)(off + k) * DT_LIMBS + l];
            acc[k * DT_LIMBS + l] = v;
            tot[l] += v;
        }
    }
    for (int i = tid; i < B; i += NT) {
        const int d = A.D.plist[off + i];
        const unsigned long long w = A.D.rec[d], ev = A.D.evm[d];
        evm[i] = ev;
        all |= ev;
        b0[i] = A.D.boff[d] - off;
        m[i] = (signed char)((int)(w >> 32) - 1);
        par[i] = w ? A.D.pidx[(int)(unsigned)w] : -1;
        flags[i] = DT_OK;
        nson[i] = 0;
    }
    for (int o = 16; o > 0; o >>= 1) {
        for (int l = 0; l < DT_LIMBS; l++) tot[l] += __shfl_xor_sync(0xffffffffu, tot[l], o);
        all |= __shfl_xor_sync(0xffffffffu, all, o);
    }
    if ((threadIdx.x & 31) == 0) {
        for (int l = 0; l < DT_LIMBS; l++)
            if (tot[l]) atomicAdd(s_all + l, tot[l]);
        atomicOr(s_all + DT_LIMBS, all);
    }
    dt_sync<NT>();
    const double value0 = (double)dt_flux(s_all, e0) * A.mincont;
    unsigned long long left = s_all[DT_LIMBS];
    int *nk = reinterpret_cast<int *>(s_all + DT_LIMBS + 1);
    while (left) {
        const int L = 63 - __clzll((long long)left);
        left &= ~(1ull << L);
        // (joins at the highest level are between peaks of that level: nothing
        // stands above them)
        const float t = L + 1 < A.N ? thr[L + 1] : 0.0f;
        for (int i = tid; i < B; i += NT) {
            const unsigned long long ev = evm[i];
            if (m[i] == L)
                dt_child(S, i, __popcll(ev), t, A.debminarea, value0, e0);
            else if ((ev >> L) & 1ull)
                dt_child(S, i, __popcll(ev >> L) - 1, t, A.debminarea, value0, e0);
        }
        dt_sync<NT>();
        for (int i = tid; i < B; i += NT)
            if (m[i] == L) dt_merge(S, i);
        dt_sync<NT>();
        for (int i = tid; i < B; i += NT) {
            const bool dead = m[i] == L, ev = !dead && ((evm[i] >> L) & 1ull);
            if (!dead && !ev) continue;
            if (dt_kept(S, i, dead ? par[i] : i)) {
                const int k = atomicAdd(nk, 1);
                keys[k] = ((unsigned long long)(L + 1) << 32) | (unsigned)label[i];
                kloc[k] = i;
            }
            if (ev) {
                const int f = flags[i];
                flags[i] = (f & ~DT_OK) | ((f & DT_OKC) && nson[i] <= 1 ? DT_OK : 0);
            }
        }
        dt_sync<NT>();
    }
    // level 0: the whole object is one branch
    for (int i = tid; i < B; i += NT)
        if (m[i] < 0) {
            if ((flags[i] & DT_OK) && A.R.size[r] >= A.debminarea) {
                const int k = atomicAdd(nk, 1);
                keys[k] = 0ull;
                kloc[k] = i;
            }
        }
    dt_sync<NT>();
    // the kept branches in (level, label) order
    const int K = *nk;
    for (int k = tid; k < K; k += NT) {
        const unsigned long long key = keys[k];
        int rank = 0;
        for (int q = 0; q < K; q++) rank += keys[q] < key;
        const int lv = (int)(key >> 32);
        A.D.olev[off + rank] = lv;
        A.D.kown[A.D.plist[off + kloc[k]]] = make_int2(lv + 1, rank);
    }
    if (tid == 0) A.R.nkept[r] = K;
    dt_sync<NT>();
}

// one warp per raw object of up to DT_WARP_PEAKS peaks
constexpr int DT_CUT_WARPS = 4;
__global__ void __launch_bounds__(DT_CUT_WARPS * 32) k_dt_cut_warp(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    __shared__ __align__(16) unsigned char smem[DT_CUT_WARPS][dt_smem(DT_WARP_PEAKS)];
    __shared__ unsigned long long s_all[DT_CUT_WARPS][8];
    const int wid = threadIdx.x >> 5, n = A.D.counts[0];
    for (int i = blockIdx.x * DT_CUT_WARPS + wid; i < n; i += gridDim.x * DT_CUT_WARPS)
        dt_cut<32>(A, A.D.lists[i], smem[wid], DT_WARP_PEAKS, s_all[wid]);
}

// one block per raw object of up to cap peaks
template <int NT>
__global__ void __launch_bounds__(NT) k_dt_cut_block(const __grid_constant__ DebArgs A, int list, int cap) {
    sx_pdl();
    if (dt_failed(A)) return;
    extern __shared__ __align__(16) unsigned char dt_smem_buf[];
    __shared__ unsigned long long s_all[8];
    const int n = A.D.counts[list];
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
        dt_cut<NT>(A, A.D.lists[(size_t)list * A.nroots + i], dt_smem_buf, cap, s_all);
        __syncthreads();
    }
}

// the largest raw objects: one cluster of blocks each, state in global memory,
// the peaks and their joins listed by level first; the kept branches are
// ranked by k_dt_rank over the whole grid.  A level is three short steps over
// its joins, each ended by a barrier of the cluster, and waits mostly on its
// loads: a raw object of 2 M pixels and 64 levels took 1.2 ms in one block and
// 0.86 so (1.5 before the lanes added up their joins to one component).
constexpr int DT_HUGE_THREADS = 1024;
constexpr int DT_HUGE_BLOCKS = 8;

struct HugeShared {
    unsigned long long tot[DT_LIMBS];
    int dead[65], ev[65];  // joins and the peaks they go to by level: counts, then first places
    int dcur[64], ecur[64], nk;
};

// the warp's peaks (join level m, -1: none; levels ev of the joins it stands
// for) added level by level to nd, ne (shared); with d, e lists, written there
// instead, at the places the counters give (index i)
__device__ __forceinline__ void dt_by_level(int i, int m, unsigned long long ev, int N, int *nd, int *ne, int *dlist,
                                            int *elist) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (int L = 0; L < N - 1; L++) {
        const unsigned dm = __ballot_sync(0xffffffffu, m == L), em = __ballot_sync(0xffffffffu, (int)(ev >> L) & 1);
        if (!(dm | em)) continue;
        int b = 0;
        if (lane == 0 && dm) b = atomicAdd(nd + L, __popc(dm));
        if (lane == 1 && em) b = atomicAdd(ne + L, __popc(em));
        if (!dlist) continue;
        const int bd = __shfl_sync(0xffffffffu, b, 0), be = __shfl_sync(0xffffffffu, b, 1);
        if (m == L) dlist[bd + __popc(dm & below)] = i;
        if ((ev >> L) & 1ull) elist[be + __popc(em & below)] = i;
    }
}

__global__ void __cluster_dims__(DT_HUGE_BLOCKS, 1, 1) __launch_bounds__(DT_HUGE_THREADS)
    k_dt_cut_huge(const __grid_constant__ DebArgs A) {
    sx_pdl();
    namespace cg = cooperative_groups;
    __shared__ HugeShared s_own;
    __shared__ int s_nd[64], s_ne[64];  // this block's counts by level, then its next places
    if (dt_failed(A)) return;  // (the status is settled before this kernel: every block alike)
    const cg::cluster_group cl = cg::this_cluster();
    HugeShared &H = *cl.map_shared_rank(&s_own, 0);  // the cluster's first block's
    const int tid = cl.block_rank() * DT_HUGE_THREADS + threadIdx.x, NT = DT_HUGE_THREADS * DT_HUGE_BLOCKS;
    const int nl = A.D.counts[3];
    for (int it = blockIdx.x / DT_HUGE_BLOCKS; it < nl; it += gridDim.x / DT_HUGE_BLOCKS) {
        const int r = A.D.lists[(size_t)3 * A.nroots + it];
        const int off = A.R.off[r], B = A.R.npk[r], NB = A.R.nbkt[r];
        const int e0 = A.sc->e0cd;
        const float *thr = A.D.thr + (size_t)r * A.N;
        DtState S;
        S.acc = A.D.acc + (size_t)off * DT_LIMBS;
        S.bsz = A.D.bsz + off;
        S.bmin = A.D.bmin + off;
        S.evm = A.D.g_evm + off;
        S.b0 = A.D.g_b0 + off;
        S.par = A.D.g_par + off;
        S.nson = A.D.g_nson + off;
        S.label = A.D.g_label + off;
        S.flags = A.D.g_flags + off;
        S.m = A.D.g_m + off;
        int *dlist = A.D.g_dlist + off, *elist = A.D.g_elist + off;
        if (cl.block_rank() == 0) {
            if (threadIdx.x < DT_LIMBS) s_own.tot[threadIdx.x] = 0ull;
            if (threadIdx.x < 65) s_own.dead[threadIdx.x] = s_own.ev[threadIdx.x] = 0;
            if (threadIdx.x == 0) s_own.nk = 0;
        }
        if (threadIdx.x < 64) s_nd[threadIdx.x] = s_ne[threadIdx.x] = 0;
        cl.sync();
        unsigned long long tot[DT_LIMBS];
        for (int l = 0; l < DT_LIMBS; l++) tot[l] = 0ull;
        for (int k = tid; k < NB; k += NT)
            for (int l = 0; l < DT_LIMBS; l++) tot[l] += S.acc[(size_t)k * DT_LIMBS + l];
        for (int l = 0; l < DT_LIMBS; l++) {
            for (int o = 16; o > 0; o >>= 1) tot[l] += __shfl_xor_sync(0xffffffffu, tot[l], o);
            if ((threadIdx.x & 31) == 0 && tot[l]) atomicAdd(H.tot + l, tot[l]);
        }
        for (int i0 = 0; i0 < B; i0 += NT) {
            const int i = i0 + tid;
            int m = -1;
            unsigned long long ev = 0ull;
            if (i < B) {
                const int d = A.D.plist[off + i];
                const unsigned long long w = A.D.rec[d];
                ev = A.D.evm[d];
                m = (int)(w >> 32) - 1;
                S.evm[i] = ev;
                S.b0[i] = A.D.boff[d] - off;
                S.m[i] = (signed char)m;
                S.par[i] = w ? A.D.pidx[(int)(unsigned)w] : -1;
                S.flags[i] = DT_OK;
                S.nson[i] = 0;
            }
            dt_by_level(i, m, ev, A.N, s_nd, s_ne, nullptr, nullptr);
        }
        __syncthreads();
        if (threadIdx.x < 64) {
            if (s_nd[threadIdx.x]) atomicAdd(H.dead + threadIdx.x, s_nd[threadIdx.x]);
            if (s_ne[threadIdx.x]) atomicAdd(H.ev + threadIdx.x, s_ne[threadIdx.x]);
        }
        cl.sync();
        if (tid == 0) {
            int a = 0, b = 0;
            for (int L = 0; L < 65; L++) {
                const int x = L < 64 ? H.dead[L] : 0, y = L < 64 ? H.ev[L] : 0;
                H.dead[L] = a;
                H.ev[L] = b;
                if (L < 64) {
                    H.dcur[L] = a;
                    H.ecur[L] = b;
                }
                a += x;
                b += y;
            }
        }
        cl.sync();
        if (threadIdx.x < 64) {
            s_nd[threadIdx.x] = atomicAdd(H.dcur + threadIdx.x, s_nd[threadIdx.x]);
            s_ne[threadIdx.x] = atomicAdd(H.ecur + threadIdx.x, s_ne[threadIdx.x]);
        }
        __syncthreads();
        for (int i0 = 0; i0 < B; i0 += NT) {
            const int i = i0 + tid;
            dt_by_level(i, i < B ? S.m[i] : -1, i < B ? S.evm[i] : 0ull, A.N, s_nd, s_ne, dlist, elist);
        }
        if (cl.block_rank() != 0) {
            if (threadIdx.x < DT_LIMBS) s_own.tot[threadIdx.x] = H.tot[threadIdx.x];
            if (threadIdx.x < 65) {
                s_own.dead[threadIdx.x] = H.dead[threadIdx.x];
                s_own.ev[threadIdx.x] = H.ev[threadIdx.x];
            }
        }
        cl.sync();
        const double value0 = (double)dt_flux(s_own.tot, e0) * A.mincont;
        for (int L = A.N - 2; L >= 0; L--) {
            const int d0 = s_own.dead[L], d1 = s_own.dead[L + 1], v0 = s_own.ev[L], v1 = s_own.ev[L + 1];
            if (d0 == d1) continue;
            const float t = thr[L + 1];
            for (int k = d0 + tid; k < d1; k += NT) {
                const int i = __ldcg(dlist + k);
                dt_child(S, i, __popcll(S.evm[i]), t, A.debminarea, value0, e0);
            }
            for (int k = v0 + tid; k < v1; k += NT) {
                const int i = __ldcg(elist + k);
                dt_child(S, i, __popcll(S.evm[i] >> L) - 1, t, A.debminarea, value0, e0);
            }
            cl.sync();
            for (int k0 = d0; k0 < d1; k0 += NT) dt_merge_warp(S, k0 + tid < d1 ? __ldcg(dlist + k0 + tid) : -1);
            cl.sync();
            for (int k = d0 + tid; k < d1; k += NT) {
                const int i = __ldcg(dlist + k);
                if (dt_kept(S, i, S.par[i])) {
                    const int q = atomicAdd(&H.nk, 1);
                    A.D.kept[off + q] = ((unsigned long long)(L + 1) << 32) | (unsigned)S.label[i];
                    A.D.krep[off + q] = A.D.plist[off + i];
                }
            }
            for (int k = v0 + tid; k < v1; k += NT) {
                const int i = __ldcg(elist + k);
                if (dt_kept(S, i, i)) {
                    const int q = atomicAdd(&H.nk, 1);
                    A.D.kept[off + q] = ((unsigned long long)(L + 1) << 32) | (unsigned)S.label[i];
                    A.D.krep[off + q] = A.D.plist[off + i];
                }
                const int f = S.flags[i];
                S.flags[i] = (f & ~DT_OK) | ((f & DT_OKC) && S.nson[i] <= 1 ? DT_OK : 0);
            }
            cl.sync();
        }
        for (int i = tid; i < B; i += NT)
            if (S.m[i] < 0 && (S.flags[i] & DT_OK) && A.R.size[r] >= A.debminarea) {
                const int q = atomicAdd(&H.nk, 1);
                A.D.kept[off + q] = 0ull;
                A.D.krep[off + q] = A.D.plist[off + i];
            }
        cl.sync();
        if (tid == 0) A.R.nkept[r] = H.nk;
        cl.sync();
    }
    cl.sync();  // (no block leaves while another may still read its shared memory)
}

// kept branches of the largest raw objects in (level, label) order: the
// whole grid counts, one thread per branch (a cluster's raw object of 2 M
// pixels keeps thousands)
__global__ void __launch_bounds__(DT_THREADS) k_dt_rank(const __grid_constant__ DebArgs A) {
    sx_pdl();
    if (dt_failed(A)) return;
    const int nl = A.D.counts[3];
    for (int it = 0; it < nl; it++) {
        const int r = A.D.lists[(size_t)3 * A.nroots + it], off = A.R.off[r], K = A.R.nkept[r];
        const unsigned long long *kept = A.D.kept + off;
        for (int k = blockIdx.x * DT_THREADS + threadIdx.x; k < K; k += gridDim.x * DT_THREADS) {
            const unsigned long long key = kept[k];
            int rank = 0;
#pragma unroll 8
            for (int q = 0; q < K; q++) rank += kept[q] < key;
            const int lv = (int)(key >> 32);
            A.D.olev[off + rank] = lv;
            A.D.kown[A.D.krep[off + k]] = make_int2(lv + 1, rank);
        }
    }
}

// DEBLEND_NTHRESH 1: no level above the detection threshold
__global__ void __launch_bounds__(DT_THREADS) k_dt_whole(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int r = blockIdx.x * DT_THREADS + threadIdx.x;
    if (r >= sx_count(A.nroots, A.nroots_dev)) return;
    A.R.nkept[r] = 1;
    A.D.olev[A.R.off[r]] = 0;
}

// ---------------------------------------------------------------------------
// 5. ownership of the kept branches, preanalysis, gatherup
// ---------------------------------------------------------------------------
// objects of every raw object, one warp each.  O.n counts the pixels (all of
// them where the raw object is one branch at level 0), O.off is the place of
// the branch's own pixels and O.npix the fill of that list until later stages
// set them.
__global__ void __launch_bounds__(DT_THREADS) k_da_objects(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int lane = threadIdx.x & 31, r = (blockIdx.x * DT_THREADS + threadIdx.x) >> 5;
    if (r >= sx_count(A.nroots, A.nroots_dev)) return;
    const int K = A.R.nkept[r], ob = A.R.objbase[r], off = A.R.off[r], P = A.R.size[r];
    for (int i = lane; i < K; i += 32) {
        const int o = ob + i, lv = A.D.olev[off + i];
        const bool whole = K == 1 && lv == 0;
        A.O.root[o] = r;
        A.O.level[o] = lv;
        A.O.node_dthresh[o] = A.D.thr[(size_t)r * A.N + lv];
        A.O.dthr[o] = A.R.dthresh[r];
        A.O.athr[o] = A.R.thresh[r];
        A.O.n[o] = whole ? P : 0;
        A.O.off[o] = off;
        A.O.npix[o] = 0;
    }
}

__device__ __forceinline__ bool da_whole(const DebArgs &A, int r, int K) {
    return K == 1 && A.D.olev[A.R.off[r]] == 0;
}

// Owner of each pixel: its component at level L is the representative of its
// chain of joins that covers L (a peak covers the levels above its join, down
// from where the previous one of the chain joined it); a kept branch (L,
// peak) owns the pixel when the peak covers L on the chain.
__global__ void __launch_bounds__(DT_THREADS) k_da_own(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    const int n = sx_count(A.nrootpix, A.nrootpix_dev);
    if (blockIdx.x * DT_THREADS >= n) return;
    __shared__ int s_wcnt[DT_THREADS / 32], s_base;
    int count = -1;
    bool rest = false;
    if (j < n) {
        const int r = (int)A.rid[j], K = A.R.nkept[r], ob = A.R.objbase[r];
        int o = -1;
        if (da_whole(A, r, K)) {
            o = ob;
        } else {
            int x = A.D.up[j], hi = A.D.lev[j];
            const int cap = dt_cap(A);
            int k = 0;
            for (; k <= cap; k++) {
                const int2 ko = A.D.kown[x];
                const unsigned long long w = A.D.rec[x];
                const int lo = (int)(w >> 32) - 1;
                if (ko.x > 0 && ko.x - 1 > lo && ko.x - 1 <= hi) {
                    o = ob + ko.y;
                    break;
                }
                if (lo < 0) break;
                hi = lo;
                x = (int)(unsigned)w;
            }
            if (k > cap) atomicOr(&A.sc->status, SX_ST_LOOP);
            count = o;
        }
        A.objkey[j] = (unsigned)o;
        if (o >= 0) A.alloc[A.rpix[j]] = o;
        rest = o < 0;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned grp = __match_any_sync(0xffffffffu, count);
    if (count >= 0 && lane == __ffs(grp) - 1) atomicAdd(A.O.n + count, __popc(grp));
    // the pixels no branch owns, listed for the gatherup (one atomic a block)
    const unsigned rm = __ballot_sync(0xffffffffu, rest);
    if (lane == 0) s_wcnt[wid] = __popc(rm);
    __syncthreads();
    int before = 0, tot = 0;
#pragma unroll
    for (int k = 0; k < DT_THREADS / 32; k++) {
        if (k < wid) before += s_wcnt[k];
        tot += s_wcnt[k];
    }
    if (threadIdx.x == 0 && tot) s_base = atomicAdd(A.D.counts + 7, tot);
    __syncthreads();
    if (rest) A.D.rest[s_base + before + __popc(rm & ((1u << lane) - 1u))] = j;
}

// lists of the branches' own pixels, inside their raw object's range (in any
// order: every sum over them is exact)
__global__ void __launch_bounds__(DT_THREADS) k_da_starts(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int o = blockIdx.x * DT_THREADS + threadIdx.x;
    if (o >= sx_count(A.nobj, A.nobj_dev)) return;
    const int r = A.O.root[o], n = A.O.n[o];
    if (!da_whole(A, r, A.R.nkept[r])) A.O.off[o] = A.R.off[r] + atomicAdd(A.R.nown + r, n);
}

__global__ void __launch_bounds__(DT_THREADS) k_da_scatter(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int j = blockIdx.x * DT_THREADS + threadIdx.x;
    const int n = sx_count(A.nrootpix, A.nrootpix_dev);
    if (blockIdx.x * DT_THREADS >= n) return;
    const int o = j < n ? (int)A.objkey[j] : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, o);
    if (o < 0) return;
    const int lane = threadIdx.x & 31, lead = __ffs(grp) - 1;
    int b = 0;
    if (lane == lead) b = A.O.off[o] + atomicAdd(A.O.npix + o, __popc(grp));
    b = __shfl_sync(grp, b, lead);
    A.D.ownpix[b + __popc(grp & ((1u << lane) - 1u))] = A.rpix[j];
}

// preanalysis of each kept branch over its own pixels (cudaanalyse.cu:
// 1686-1903): one warp per branch, one block for those of more than
// DA_WARP_MAX pixels; the ellipse is finished by k_da_finish, one thread per
// object
__global__ void __launch_bounds__(DT_THREADS, 3) k_da_moments(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int o = (blockIdx.x * DT_THREADS + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (o >= sx_count(A.nobj, A.nobj_dev)) return;
    const int n = A.O.n[o];
    if (n > DA_WARP_MAX) {
        if (lane == 0) A.D.biglist[atomicAdd(A.D.counts + 4, 1)] = o;
        return;
    }
    pix_moments_warp(A.cd, A.sub, A.D.ownpix + A.O.off[o], n, A.wdiv, A.w, A.O.node_dthresh[o], A.raw + o);
}

__global__ void __launch_bounds__(DT_THREADS, 2) k_da_moments_big(const __grid_constant__ DebArgs A) {
    sx_pdl();
    __shared__ PixBlock sh;
    const int nb = A.D.counts[4];
    for (int i = blockIdx.x; i < nb; i += gridDim.x) {
        const int o = A.D.biglist[i];
        pix_moments_block(A.cd, A.sub, A.D.ownpix + A.O.off[o], A.O.n[o], A.wdiv, A.w, A.O.node_dthresh[o], sh, A.raw + o);
    }
}

__global__ void k_da_finish(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = o < sx_count(A.nobj, A.nobj_dev);
    const int oo = live ? o : 0;
    MomentRaw R = A.raw[oo];
    const int L = A.O.level[oo];
    const double dthresh = A.O.node_dthresh[oo];
    if (warp_each(live && R.ovf, o, [&](int q) {
            pix_moments_wide(A.cd, A.sub, A.D.ownpix + A.O.off[q], A.O.n[q], A.wdiv, A.w, A.raw + q);
        }))
        R = A.raw[oo];
    if (!live) return;
    if (R.ovf) atomicOr(&A.sc->status, SX_ST_RANGE);
    const int xmin = R.xmin, xmax = R.xmax, ymin = R.ymin, ymax = R.ymax;
    int flag = 0;
    if (L > 0) flag |= SX_OBJ_MERGED;
    if (xmin == 0 || xmax == A.w - 1 || ymin == 0 || ymax == A.h - 1) flag |= SX_OBJ_TRUNC;
    const float rv = R.rv, peak = R.peak;
    const double rvd = rv, mx = R.mx, my = R.my, mx2 = R.mx2, my2 = R.my2, mxy = R.mxy;
    const double dthresh2 = (dthresh + peak) / 2.0;
    const double xm = mx / rvd, ym = my / rvd;
    double xm2 = mx2 / rvd - xm * xm, ym2 = my2 / rvd - ym * ym, xym = mxy / rvd - xm * ym;
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
    const float fa = (float)sqrt(pmx2), fb = (float)sqrt(pmy2);
    float abcor;
    darea = (double)R.area2 - R.dnpix;
    t1t2 = dthresh / dthresh2;
    if (t1t2 > 0.0) {
        abcor = (darea < 0.0 ? darea : -1.0) / (2 * SX_PI * log(t1t2 < 1.0 ? t1t2 : 0.99) * fa * fb);
        if (abcor > 1.0) abcor = 1.0;
    } else
        abcor = 1.0;
    A.O.xmin[o] = xmin;
    A.O.xmax[o] = xmax;
    A.O.ymin[o] = ymin;
    A.O.ymax[o] = ymax;
    A.O.flags[o] = flag;
    A.O.singu[o] = singu;
    A.O.dnpix[o] = R.dnpix;
    A.O.fdflux[o] = rv;
    A.O.dflux[o] = R.tv;
    A.O.fdpeak[o] = R.cpeak;
    A.O.dpeak[o] = peak;
    A.O.mx[o] = xm + xmin;
    A.O.my[o] = ym + ymin;
    A.O.mx2[o] = xm2;
    A.O.my2[o] = ym2;
    A.O.mxy[o] = xym;
    A.O.a[o] = fa;
    A.O.b[o] = fb;
    A.O.theta[o] = theta * 180.0 / SX_PI;
    A.O.cxx[o] = (float)(ym2 / temp2);
    A.O.cyy[o] = (float)(xm2 / temp2);
    A.O.cxy[o] = (float)(-2 * xym / temp2);
    A.O.abcor[o] = abcor;
    // the gatherup's copy: the centre as whole pixels and a float remainder
    GatherObj G;
    const double cx = xm + xmin, cy = ym + ymin;
    G.ix = (int)floor(cx);
    G.iy = (int)floor(cy);
    G.fx = (float)(cx - G.ix);
    G.fy = (float)(cy - G.iy);
    G.cxx = (float)(ym2 / temp2);
    G.cyy = (float)(xm2 / temp2);
    G.cxy = (float)(-2 * xym / temp2);
    G.abcor = abcor;
    // the form is at least its smaller eigenvalue times |offset|^2; in single
    // precision it is off by less than 1e-5 of the coefficients' sum times that,
    // and the offset from whole pixels is at least 0.91 of its length beyond 16
    const double qa = G.cxx, qb = G.cyy, qc = G.cxy;
    const double lam = 0.5 * (qa + qb - sqrt((qa - qb) * (qa - qb) + qc * qc)) - 1e-5 * (fabs(qa) + fabs(qb) + fabs(qc));
    GatherBound Bd;
    Bd.ix = G.ix;
    Bd.iy = G.iy;
    Bd.lam = lam > 0.0 && abcor > 0.0f ? (float)(0.4 * lam / abcor) : 0.0f;
    Bd.pad = 0;
    A.gobj[o] = G;
    A.gbound[o] = Bd;
}

// gatherup (cudadeblend.cu:1262-1360): every other pixel to the nearest kept
// branch in the elliptical metric, the first in order on ties.  The metric
// takes its offsets in double and ends in a double division; a branch whose
// single-precision distance is clearly above the smallest so far is passed
// over without them.  The offset from whole pixels and remainder is off by
// less than 2^-23 of 1 + |offset|, so the quadratic form, of terms that add up
// to T, by less than 2e-6 (T + the coefficients' sum).  In a raw object of many
// branches most are far away: a bound by the offset alone passes those over
// first: deblending of a cluster with one raw object of 2 M pixels 2.80 -> 2.51
// ms, the same from 8, 16, 32 or 64 branches on; of a crowded field 1.360, 1.352,
// 1.340 and 1.341 ms, 1.341 without.
constexpr int GATHER_MANY = 32;  // branches

__global__ void __launch_bounds__(DT_THREADS) k_da_gather(const __grid_constant__ DebArgs A) {
    sx_pdl();
    const int n = A.D.counts[7], nround = (n + 31) & ~31;
    for (int i0 = blockIdx.x * DT_THREADS + threadIdx.x; i0 < nround; i0 += gridDim.x * DT_THREADS) {
        int o = -1, x = 0, y = 0;
        if (i0 < n) {
            const int j = A.D.rest[i0];
            const int r = (int)A.rid[j], K = A.R.nkept[r], ob = A.R.objbase[r];
            const int p = (int)A.rpix[j];
            y = (int)fdiv((unsigned)p, A.wdiv);
            x = p - y * A.w;
            int iclst = 0;
            float distmin = 1e+31f;
            for (int i = 0; i < K; i++) {
                const int q = ob + i;
                if (K >= GATHER_MANY) {
                    const int4 g2 = __ldg(reinterpret_cast<const int4 *>(A.gbound + q));
                    const float ux = (float)(x - g2.x), uy = (float)(y - g2.y), d2 = ux * ux + uy * uy;
                    const float t = __int_as_float(g2.z) * d2;
                    if (d2 > 256.0f && t > 1e-30f && t > distmin) continue;
                }
                const int4 g0 = __ldg(reinterpret_cast<const int4 *>(A.gobj + q));
                const float4 g1 = __ldg(reinterpret_cast<const float4 *>(A.gobj + q) + 1);
                const float abc = g1.w;
                {
                    const float ux = (float)(x - g0.x) - __int_as_float(g0.z), uy = (float)(y - g0.y) - __int_as_float(g0.w);
                    const float qx = g1.x * ux * ux, qy = g1.y * uy * uy, qc = g1.z * ux * uy;
                    const float f = qx + qy + qc - 2e-6f * (fabsf(qx) + fabsf(qy) + fabsf(qc) + fabsf(g1.x) + fabsf(g1.y) +
                                                            fabsf(g1.z) * (1.0f + fabsf(ux) + fabsf(uy)));
                    if (f > 1e-30f && abc > 0.0f && 0.499999f * f > distmin * abc) continue;
                }
                const float dx = x - __ldg(A.O.mx + q), dy = y - __ldg(A.O.my + q);
                const float dist = 0.5 * (g1.x * dx * dx + g1.y * dy * dy + g1.z * dx * dy) / abc;
                if (dist < distmin) {
                    distmin = dist;
                    iclst = i;
                }
            }
            o = ob + iclst;
            A.alloc[p] = o;
        }
        // the objects grow by them: their pixel counts and boxes
        const unsigned grp = __match_any_sync(0xffffffffu, o);
        if (o < 0) continue;
        const int x0 = __reduce_min_sync(grp, x), x1 = __reduce_max_sync(grp, x);
        const int y0 = __reduce_min_sync(grp, y), y1 = __reduce_max_sync(grp, y);
        if ((int)(threadIdx.x & 31) == __ffs(grp) - 1) {
            atomicAdd(A.O.n + o, __popc(grp));
            if (x0 < A.O.xmin[o]) atomicMin(A.O.xmin + o, x0);
            if (x1 > A.O.xmax[o]) atomicMax(A.O.xmax + o, x1);
            if (y0 < A.O.ymin[o]) atomicMin(A.O.ymin + o, y0);
            if (y1 > A.O.ymax[o]) atomicMax(A.O.ymax + o, y1);
        }
    }
}

// resident blocks of a grid-stride kernel over a device-side count, at most n
static unsigned dt_grid(long long n, int per_sm) {
    static DevCache nsm;
    const int sms = nsm.get([](int dev) {
        int k = 148;
        cudaDeviceGetAttribute(&k, cudaDevAttrMultiProcessorCount, dev);
        return k > 0 ? k : 148;
    });
    return (unsigned)std::max(1ll, std::min(n, (long long)sx_share(sms * per_sm)));
}

int launch_deblend_tree(const DebArgs &A, cudaStream_t st) {
    if (A.nroots <= 0 || A.nrootpix <= 0) return 0;
    static DevCache smem_set;
    smem_set.get([](int) {
        cudaFuncSetAttribute(k_dt_cut_block<512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)dt_smem(DT_BIG_PEAKS));
        return 1;
    });
    const unsigned gp = (unsigned)((A.nrootpix + DT_THREADS - 1) / DT_THREADS);
    const unsigned gt = (unsigned)(((long long)A.nroots * A.N + DT_THREADS - 1) / DT_THREADS);
    const unsigned gk = dt_grid((A.nrootpix / 2 + DT_THREADS) / DT_THREADS, 8);
    sx_launch(k_dt_up, gp, DT_THREADS, 0, st, A);
    sx_launch(k_dt_thresholds, gt, DT_THREADS, 0, st, A);
    sx_launch(k_dt_level, gp, DT_THREADS, 0, st, A);
    if (A.N < 2) {  // one level: every raw object is one branch
        sx_launch(k_dt_whole, (A.nroots + DT_THREADS - 1) / DT_THREADS, DT_THREADS, 0, st, A);
        return 4;
    }
    sx_launch(k_dt_edges, gp, DT_THREADS, 0, st, A);
    sx_launch(k_dt_flatten, gk, DT_THREADS, 0, st, A);
    sx_launch(k_dt_buckets, gk, DT_THREADS, 0, st, A);
    sx_launch(k_dt_fill, gp, DT_THREADS, 0, st, A);
    sx_launch(k_dt_cut_warp, dt_grid((A.nroots + DT_CUT_WARPS - 1) / DT_CUT_WARPS, 8), DT_CUT_WARPS * 32, 0, st, A);
    sx_launch(k_dt_cut_block<256>, dt_grid(A.nroots, 4), 256, dt_smem(DT_MID_PEAKS), st, A, 1, DT_MID_PEAKS);
    sx_launch(k_dt_cut_block<512>, dt_grid(A.nroots, 1), 512, dt_smem(DT_BIG_PEAKS), st, A, 2, DT_BIG_PEAKS);
    sx_launch(k_dt_cut_huge, (unsigned)std::min((long long)A.nroots, 8ll) * DT_HUGE_BLOCKS, DT_HUGE_THREADS, 0, st,
              A);
    sx_launch(k_dt_rank, dt_grid(A.nrootpix / DT_THREADS + 1, 4), DT_THREADS, 0, st, A);
    return 12;
}

int launch_deblend_assign(const DebArgs &A, cudaStream_t st) {
    if (A.nroots <= 0 || A.nrootpix <= 0) return 0;
    const unsigned gp = (unsigned)((A.nrootpix + DT_THREADS - 1) / DT_THREADS);
    const unsigned go = (unsigned)((std::max(A.nobj, 1) + DT_THREADS - 1) / DT_THREADS);
    const unsigned gw = (unsigned)((std::max(A.nobj, 1) + DT_THREADS / 32 - 1) / (DT_THREADS / 32));
    sx_launch(k_da_objects, (A.nroots + DT_THREADS / 32 - 1) / (DT_THREADS / 32), DT_THREADS, 0, st, A);
    sx_launch(k_da_own, gp, DT_THREADS, 0, st, A);
    sx_launch(k_da_starts, go, DT_THREADS, 0, st, A);
    sx_launch(k_da_scatter, gp, DT_THREADS, 0, st, A);
    sx_launch(k_da_moments, gw, DT_THREADS, 0, st, A);
    sx_launch(k_da_moments_big, dt_grid(A.nobj, 2), DT_THREADS, 0, st, A);
    sx_launch(k_da_finish, go, DT_THREADS, 0, st, A);
    sx_launch(k_da_gather, dt_grid(gp, 8), DT_THREADS, 0, st, A);
    return 8;
}

}  // namespace sx
