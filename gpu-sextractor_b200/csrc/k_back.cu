// k_back.cu -- background estimation (reference: src/back.c makeback,
// backstat, backhisto, backguess, filterback, makebackspline, subbackline and
// the CUDA driver src/cuda/cudaback.cu:1212).
//
// Results are bit-identical to the reference's CPU functions:
//  * the per-mesh mean/sigma are the reference's sequential double sums with
//    its roundings, composed from stretches of the sequence (seq_sums);
//  * histogram sums are exact integers, so they are reduced in parallel;
//  * the two-pointer median walk of backguess is replaced by a binary search
//    on the merge path of the two cumulative sums, which lands on the same
//    split;
//  * spline and interpolation arithmetic is float, in the reference's order.
#include "common.cuh"
#include "kernels.cuh"

namespace sx {

// ---------------------------------------------------------------------------
// The two sequential double sums of backstat (src/back.c:214-279), sum of
// the pixels and sum of their squares in pixel order, by one warp.
//
// A sequential sum is a chain of roundings, but in the one binade [2^k,
// 2^(k+1)) that the partial sum stays in for long it can be cut into pieces:
// there S + t is rounded to a multiple of q = 2^(k-52), and how depends on t
// and on whether S / q is even or odd (ties), on nothing else of S.  So each
// lane adds its stretch of the sequence to 2^k and, in a second chain, to
// 2^k + q; the two increments and final parities describe what the stretch
// does to any sum of that binade.  A scan over the lanes composes them in
// order.  Where the sum reaches 2^(k+1) in a lane's stretch, that stretch is
// added pixel by pixel and the lanes after it start again in the new binade:
// a handful of times, since the sum has to double each time.  The squares of
// floats are exact in double, so fma(p, p, s) is s + p * p rounded once.
//
// The sum of the pixels themselves is exact whatever the order when the sum
// of the magnitudes is below 2^53 units of the smallest exponent present
// (checked; pixel by pixel otherwise).
//
// One lane per mesh adding pixel by pixel took 33 cycles a pixel and pass:
// 138 us for the 64 x 64 meshes of any frame, 0.55 ms for 128 x 128.  Composed
// and followed by the mode in the same warp, the background stage went from
// 0.165 to 0.083 ms (160 x 160), 0.375 to 0.249 (4096 x 4096, 64 x 64
// meshes), 0.67 to 0.215 (128 x 128), 4.6 to 4.1 (16384 x 16384); it is bound
// by issue there (about 45 warp instructions per 32 pixels and pass).
// ---------------------------------------------------------------------------
constexpr int SEQ_G = 16;                          // pixels of a lane's stretch
constexpr int SEQ_CHUNK = 32 * SEQ_G;              // pixels taken at a time
constexpr int SEQ_PITCH = SEQ_G + 4;               // staged stretches: 16-byte reads on distinct banks
constexpr int SEQ_STAGE = 32 * SEQ_PITCH;          // floats of a staged chunk

// asynchronous copies into shared memory, and the wait for all but the newest
// N groups of this lane's
__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct SeqSums {
    double sum, sq;
    int n;
    bool exact;     // the sum of the pixels is the sequential one
    unsigned amin;  // smallest nonzero magnitude's bits - 1 (0xffffffff: none)
};

// the test of a pixel: pass 0 valid (above -BIG), pass 1 inside the cuts
// (and, for an annulus, valid).  It is made on the float: a float compares
// with the float cuts as its double does, and f > (float)-BIG as (double)f >
// -BIG (the float nearest -1e30 lies below it, the next one up above it).
template <int PASS, bool VALID>
__device__ __forceinline__ bool seq_in(float f, float lcut, float hcut) {
    if (PASS == 0) return f > (float)-SX_BIG;
    return (!VALID || f > (float)-SX_BIG) && f <= hcut && f >= lcut;
}

// LOAD: fetch<G, STRETCH>(dst) starts the copies of the sequence's next 32 G
// pixels (NaN beyond the end) to dst, as they come or into their lanes'
// stretches, as one group.  Each chunk is on its way while the one before it is
// taken (with a chunk loaded, stored and taken in turn, DRAM and L2 latency were
// a tenth of the background stage of a frame of few meshes: 0.199 ms for 128 x 128
// meshes of 4096 x 4096 pixels, 0.176 so).  stage: 2 SEQ_STAGE floats of
// this warp, 16-byte aligned.  amin: for pass 1, what pass 0 found (its pixels
// are among them).
template <int PASS, bool VALID, class LOAD>
__device__ __forceinline__ SeqSums seq_sums(LOAD load, int n, float lcut, float hcut, unsigned amin, float *stage) {
    const int lane = threadIdx.x & 31;
    double S = 0.0, m = 0.0;
    int cnt = 0;
    load.template fetch<SEQ_G, true>(stage);
    const float *cur = stage;
    for (int c0 = 0; c0 < n; c0 += SEQ_CHUNK) {
        if (c0 + SEQ_CHUNK < n) {
            load.template fetch<SEQ_G, true>(cur == stage ? stage + SEQ_STAGE : stage);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncwarp();
        const float4 *mine = reinterpret_cast<const float4 *>(cur + lane * SEQ_PITCH);
        double d[SEQ_G];
#pragma unroll
        for (int g = 0; g < SEQ_G / 4; g++) {
            const float4 f4 = mine[g];
            const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool in = seq_in<PASS, VALID>(f[k], lcut, hcut);
                const float v = in ? f[k] : 0.0f;
                cnt += in;
                if (PASS == 0) amin = min(amin, (__float_as_uint(v) & 0x7fffffffu) - 1u);
                d[4 * g + k] = (double)v;
                m += d[4 * g + k];
            }
        }
        for (int first = 0; first < 32;) {
            // S in [2^k, 2 * 2^k)
            const long long bits = __double_as_longlong(S);
            const double lo = __longlong_as_double(bits & 0x7ff0000000000000ll),
                         lo1 = __longlong_as_double((bits & 0x7ff0000000000000ll) | 1ll), hi = lo + lo;
            int stop = first;  // the lane whose stretch is added pixel by pixel
            if (S > 1e-290 && hi < 1e300) {
                double s0 = lo, s1 = lo1;
                if (lane >= first) {
#pragma unroll
                    for (int g = 0; g < SEQ_G; g++) {
                        s0 = fma(d[g], d[g], s0);
                        s1 = fma(d[g], d[g], s1);
                    }
                }
                // the parity each lane's stretch begins with: parity in ->
                // parity out of a stretch is one of two constants, or keeps
                // or flips it; so the last constant below the lane (or the
                // sum's own parity), flipped as often as lanes after it flip
                const unsigned b0 = __ballot_sync(0xffffffffu, (int)(__double_as_longlong(s0) & 1ll)),
                               b1 = __ballot_sync(0xffffffffu, (int)(__double_as_longlong(s1) & 1ll));
                const unsigned below = (1u << lane) - 1u, flips = b0 & ~b1, consts = ~(b0 ^ b1) & below;
                const int c = 31 - __clz(consts);  // -1: none
                const unsigned since = c < 0 ? below : below & ~((2u << c) - 1u);
                const unsigned par = ((c < 0 ? (unsigned)(bits & 1ll) : b0 >> c) + __popc(flips & since)) & 1u;
                // (a stretch that leaves the binade takes the sum with it)
                const double se = par ? s1 : s0;
                double f = s0 < hi && s1 < hi ? se - (par ? lo1 : lo) : hi;
                // inclusive scan (multiples of 2^(k-52) below 2^(k+1): exact)
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double e = __shfl_up_sync(0xffffffffu, f, o);
                    if (lane >= o) f += e;
                }
                const double after = S + f;
                const unsigned bal = __ballot_sync(0xffffffffu, !(after < hi));
                stop = bal ? __ffs(bal) - 1 : 32;
                if (stop > 0) S = __shfl_sync(0xffffffffu, after, stop - 1);
            }
            if (stop < 32) {
                const float *st = cur + stop * SEQ_PITCH;
#pragma unroll
                for (int g = 0; g < SEQ_G; g++) {
                    const double x = seq_in<PASS, VALID>(st[g], lcut, hcut) ? (double)st[g] : 0.0;
                    S = fma(x, x, S);
                }
            }
            first = stop + 1;
        }
        __syncwarp();  // (every lane has read this chunk: its place takes the next but one)
        cur = cur == stage ? stage + SEQ_STAGE : stage;
    }
    SeqSums r;
    r.sq = S;
    r.n = (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
    for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
    r.sum = m;
    r.amin = PASS == 0 ? __reduce_min_sync(0xffffffffu, amin) : amin;
    // every partial sum is a multiple of 2^(e - 23), e the smallest exponent,
    // and at most the sum of the magnitudes, itself at most sqrt(n S); exact
    // in any order when that is below 2^53 units
    const int e = (int)((r.amin + 1u) >> 23) - 127;
    r.exact = r.amin == 0xffffffffu || (e > -127 && sqrt((double)r.n * S) < scalbn(1.0, e - 23 + 52));
    return r;
}

// the sum of the pixels one by one, for data whose sums round
template <int PASS, bool VALID, class LOAD>
__device__ __noinline__ double seq_sum_slow(LOAD load, int n, float lcut, float hcut, float *stage) {
    double m = 0.0;
    for (int c0 = 0; c0 < n; c0 += SEQ_CHUNK) {
        load.template fetch<SEQ_G, true>(stage);
        cp_wait<0>();
        __syncwarp();
        for (int l = 0; l < 32; l++)
#pragma unroll
            for (int k = 0; k < SEQ_G; k++) {
                const float f = stage[l * SEQ_PITCH + k];
                m += seq_in<PASS, VALID>(f, lcut, hcut) ? (double)f : 0.0;
            }
        __syncwarp();
    }
    return m;
}

// backstat of one sequence of pixels by one warp (all lanes get the result).
// minpix: valid pixels below which the mesh is bad (mean = sigma = -BIG)
template <bool VALID, class LOAD>
__device__ __forceinline__ void seq_stat(const LOAD &load, int n, float minpix, float *stage, MeshStat &o, int &nvalid) {
    const double step = sqrt(2 / SX_PI) * SX_QUANTIF_NSIGMA / SX_QUANTIF_AMIN;
    o.mean = o.sigma = o.lcut = o.hcut = o.qzero = o.qscale = 0.f;
    o.nlevels = o.npix = 0;
    SeqSums a = seq_sums<0, VALID>(load, n, 0.0f, 0.0f, 0xffffffffu, stage);
    nvalid = a.n;
    if ((float)a.n < minpix) {
        o.mean = o.sigma = -SX_BIG;
        return;
    }
    if (!a.exact) a.sum = seq_sum_slow<0, VALID>(load, n, 0.0f, 0.0f, stage);
    double sig, mean = a.sum, sigma = a.sq;
    mean /= (double)a.n;
    sigma = (sig = sigma / a.n - mean * mean) > 0.0 ? sqrt(sig) : 0.0;
    const float lcut = o.lcut = (float)(mean - 2.0 * sigma);
    const float hcut = o.hcut = (float)(mean + 2.0 * sigma);
    a = seq_sums<1, VALID>(load, n, lcut, hcut, a.amin, stage);
    if (!a.exact) a.sum = seq_sum_slow<1, VALID>(load, n, lcut, hcut, stage);
    mean = a.sum;
    sigma = a.sq;
    o.npix = a.n;
    mean /= (double)a.n;
    sig = sigma / a.n - mean * mean;
    sigma = sig > 0.0 ? sqrt(sig) : 0.0;
    o.mean = mean;
    o.sigma = sigma;
    if ((o.nlevels = (int)(step * a.n + 1)) > SX_QUANTIF_NMAXLEVELS) o.nlevels = SX_QUANTIF_NMAXLEVELS;
    o.qscale = sigma > 0.0 ? 2 * SX_QUANTIF_NSIGMA * sigma / o.nlevels : 1.0;
    o.qzero = mean - SX_QUANTIF_NSIGMA * sigma;
}

// place of pixel i of a fetch
template <bool STRETCH>
__device__ __forceinline__ int seq_slot(int i) {
    return STRETCH ? (i / SEQ_G) * SEQ_PITCH + i % SEQ_G : i;
}

// the pixels of a mw x mh mesh in row-major order: lane l copies words l,
// l + 32, ... of a fetch, of four pixels (VEC: frame and mesh
// width multiples of 4, frame 16-byte aligned) or one
template <bool VEC>
struct MeshLoad {
    static constexpr int V = VEC ? 4 : 1;
    static constexpr bool REGS = VEC;  // the histogram's pixels go through registers
    const float *origin;
    int off, left, col, mw, step, wrap, dcol;
    __device__ __forceinline__ MeshLoad(const float *origin_, int w, int mw_, int mh) {
        const int lane = threadIdx.x & 31;
        origin = origin_;
        mw = mw_;
        const int drow = 32 * V / mw, row = V * lane / mw;
        dcol = 32 * V - drow * mw;
        col = V * lane - row * mw;
        off = row * w + col;
        step = drow * w + dcol;
        wrap = w - mw;
        left = mw * mh - V * lane;
    }
    __device__ __forceinline__ void next() {
        left -= 32 * V;
        col += dcol;
        off += step;
        if (col >= mw) {
            col -= mw;
            off += wrap;
        }
    }
    template <int G, bool STRETCH>
    __device__ __forceinline__ void fetch(float *dst) {
        dst += seq_slot<STRETCH>(V * (threadIdx.x & 31));
        const bool whole = VEC && left > 32 * V * (G / V - 1);
#pragma unroll
        for (int g = 0; g < G / V; g++) {
            float *to = dst + seq_slot<STRETCH>(32 * V * g);
            if (whole || left > 0) {
                if (VEC)
                    cp_async16(to, origin + off);
                else
                    cp_async4(to, origin + off);
            } else {
                // beyond the mesh: NaN, which every test rejects as it does a NaN pixel
                for (int k = 0; k < V; k++) to[k] = __int_as_float(0x7fffffff);
            }
            next();
        }
        cp_commit();
    }
    // the same into registers (VEC)
    template <int G>
    __device__ __forceinline__ void take(float (&v)[G]) {
        const float nan = __int_as_float(0x7fffffff);
#pragma unroll
        for (int g = 0; g < G / 4; g++) {
            const float4 f = left > 0 ? __ldg(reinterpret_cast<const float4 *>(origin + off))
                                      : make_float4(nan, nan, nan, nan);
            v[4 * g] = f.x;
            v[4 * g + 1] = f.y;
            v[4 * g + 2] = f.z;
            v[4 * g + 3] = f.w;
            next();
        }
    }
};

__device__ __forceinline__ void mesh_geometry(int m, int w, int h, int bw, int bh, int nbx, int nby, int &x0, int &y0,
                                              int &mw, int &mh) {
    const int mx = m % nbx, my = m / nbx;
    x0 = mx * bw;
    y0 = my * bh;
    mw = (mx == nbx - 1 && w % bw) ? w % bw : bw;
    mh = (my == nby - 1 && h % bh) ? h % bh : bh;
}

// the frame's scalars as it begins (by the first kernel that every frame runs)
__device__ __forceinline__ void init_scalars(FrameScalars *sc) {
    FrameScalars z;
    memset(&z, 0, sizeof(z));
    z.sigfac = 1.0f;
    *sc = z;
}

// backstat of every mesh, one warp each (meshes whose histogram takes a block)
template <bool VEC>
__global__ void __launch_bounds__(32) k_mesh_stat(const float *__restrict__ img, int w, int h, int bw, int bh, int nbx,
                                                  int nby, MeshStat *__restrict__ ms, FrameScalars *sc) {
    sx_pdl();
    if (blockIdx.x == 0 && threadIdx.x == 0) init_scalars(sc);
    __shared__ __align__(16) float stage[2 * SEQ_STAGE];
    const int m = blockIdx.x;
    int x0, y0, mw, mh, nv;
    mesh_geometry(m, w, h, bw, bh, nbx, nby, x0, y0, mw, mh);
    MeshStat o;
    seq_stat<false>(MeshLoad<VEC>(img + (size_t)y0 * w + x0, w, mw, mh), mw * mh,
                    (float)(mw * mh * SX_BACK_MINGOODFRAC), stage, o, nv);
    if (threadIdx.x == 0) ms[m] = o;
}

constexpr int GUESS_THREADS = 256;

// src/back.c:297-339 (backhisto) + :347-432 (backguess), one CTA per mesh
// src/back.c:347-432 (backguess) on a histogram already in shared memory,
// for the whole CTA: the prefix sums, the clipping iteration with exact
// integer moments and the median split, the mode; thread 0 writes the mode
// and sigma to *back_out, *sig_out.
__device__ void guess_from_hist(int *hist, int *pfx, const MeshStat &bm, float *back_out, float *sig_out) {
    __shared__ long long red[3][GUESS_THREADS / 32];
    __shared__ int sh_lcut, sh_hcut, sh_go;
    const int nlevels = bm.nlevels;
    // exclusive prefix of the histogram: 17 consecutive bins per thread
    {
        constexpr int PER = (SX_QUANTIF_NMAXLEVELS + 2 + GUESS_THREADS - 1) / GUESS_THREADS;
        __shared__ int wsum[32];
        int base = threadIdx.x * PER, loc = 0;
        for (int k = 0; k < PER; k++)
            if (base + k < SX_QUANTIF_NMAXLEVELS + 2) loc += hist[base + k];
        int tot;
        int run = block_exclusive_scan(loc, wsum, tot);
        for (int k = 0; k < PER; k++)
            if (base + k < SX_QUANTIF_NMAXLEVELS + 2) {
                pfx[base + k] = run;
                run += hist[base + k];
            }
    }
    __syncthreads();

    int nlevelsm1 = nlevels - 1;
    double sig_ = 10.0 * nlevelsm1, sig1 = 1.0, mea = bm.mean, med = bm.mean;
    if (threadIdx.x == 0) {
        sh_lcut = 0;
        sh_hcut = nlevelsm1;
    }
    for (int n = 100;;) {
        if (threadIdx.x == 0) sh_go = (n-- && (sig_ >= 0.1) && (fabs(sig_ / sig1 - 1.0) > SX_EPS));
        __syncthreads();
        if (!sh_go) break;
        int lcut = sh_lcut, hcut = sh_hcut;
        // exact integer sums over [lcut, hcut]
        long long s0 = 0, s1 = 0, s2 = 0;
        for (int i = lcut + threadIdx.x; i <= hcut; i += GUESS_THREADS) {
            long long pv = hist[i];
            s0 += pv;
            s1 += pv * i;
            s2 += pv * i * (long long)i;
        }
        for (int o = 16; o > 0; o >>= 1) {
            s0 += __shfl_down_sync(0xffffffffu, s0, o);
            s1 += __shfl_down_sync(0xffffffffu, s1, o);
            s2 += __shfl_down_sync(0xffffffffu, s2, o);
        }
        if ((threadIdx.x & 31) == 0) {
            red[0][threadIdx.x >> 5] = s0;
            red[1][threadIdx.x >> 5] = s1;
            red[2][threadIdx.x >> 5] = s2;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            long long sum = 0, t1 = 0, t2 = 0;
            for (int k = 0; k < GUESS_THREADS / 32; k++) {
                sum += red[0][k];
                t1 += red[1][k];
                t2 += red[2][k];
            }
            // split of the two-pointer walk: smallest a with NOT(A(a) < B(nn-1-a))
            int nn = hcut - lcut + 1, lo = 0, hi = nn;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                int A = pfx[lcut + mid] - pfx[lcut];
                int B = pfx[hcut + 1] - pfx[hcut + 1 - (nn - 1 - mid)];
                if (A < B)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            int il = lcut + lo, ih = il - 1;
            unsigned long lowsum = (unsigned long)(pfx[il] - pfx[lcut]);
            unsigned long highsum = (unsigned long)(pfx[hcut + 1] - pfx[il]);
            double ftemp;
            sig1 = sig_;
            sig_ = (double)t2;
            mea = (double)t1;
            long hl = hist[il], hh = ih >= 0 ? hist[ih] : 0;
            med = ih >= 0 ? ((double)ih + 0.5 + ((double)highsum - lowsum) / (2.0 * (hl > hh ? hl : hh))) : 0.0;
            if (sum) {
                mea /= (double)sum;
                sig_ = sig_ / sum - mea * mea;
            }
            sig_ = sig_ > 0.0 ? sqrt(sig_) : 0.0;
            sh_lcut = (ftemp = med - 3.0 * sig_) > 0.0 ? (int)(ftemp > 0.0 ? ftemp + 0.5 : ftemp - 0.5) : 0;
            sh_hcut = (ftemp = med + 3.0 * sig_) < nlevelsm1 ? (int)(ftemp > 0.0 ? ftemp + 0.5 : ftemp - 0.5)
                                                               : nlevelsm1;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        float mean;
        // src/back.c:408: the C library abs(int) applied to the double sig
        if (abs((int)sig_) > 0.0) {
            if (fabs((mea - med) / sig_) < 0.3)
                mean = bm.qzero + (2.5 * med - 1.5 * mea) * bm.qscale;
            else
                mean = bm.qzero + med * bm.qscale;
        } else
            mean = bm.qzero + mea * bm.qscale;
        *back_out = mean;
        *sig_out = sig_ * bm.qscale;
    }
}

__global__ void __launch_bounds__(GUESS_THREADS) k_mesh_guess(const float *__restrict__ img, int w, int h, int bw,
                                                                int bh, int nbx, int nby,
                                                                const MeshStat *__restrict__ ms,
                                                                float *__restrict__ back, float *__restrict__ sig) {
    sx_pdl();
    __shared__ int hist[SX_QUANTIF_NMAXLEVELS + 2];
    __shared__ int pfx[SX_QUANTIF_NMAXLEVELS + 2];   // pfx[i] = sum_{k<i} hist[k]
    int m = blockIdx.x;
    int mx = m % nbx, my = m / nbx;
    MeshStat bm = ms[m];
    if (bm.mean <= -SX_BIG) {
        if (threadIdx.x == 0) back[m] = sig[m] = -SX_BIG;
        return;
    }
    int x0 = mx * bw, y0 = my * bh;
    int mw = (mx == nbx - 1 && w % bw) ? w % bw : bw;
    int mh = (my == nby - 1 && h % bh) ? h % bh : bh;
    for (int i = threadIdx.x; i < SX_QUANTIF_NMAXLEVELS + 2; i += GUESS_THREADS) hist[i] = 0;
    __syncthreads();
    int nlevels = bm.nlevels;
    float qscale = bm.qscale;
    float cste = 0.499999 - bm.qzero / qscale;
    // one warp per mesh row, lanes along the row (no index division)
    for (int r = threadIdx.x >> 5; r < mh; r += GUESS_THREADS / 32) {
        const float *row = img + (size_t)(y0 + r) * w + x0;
        for (int x = threadIdx.x & 31; x < mw; x += 32) {
            float b = __ldg(row + x) / qscale + cste;
            if (b != b) continue;  // NaN: the host conversion yields INT_MIN
            int bin = (int)b;
            if (bin >= 0 && bin < nlevels) atomicAdd(&hist[bin], 1);
        }
    }
    __syncthreads();
    guess_from_hist(hist, pfx, bm, back + m, sig + m);
}

// ---------------------------------------------------------------------------
// backhisto + backguess with one warp per mesh (or annulus), for fewer than
// 65536 pixels (no bin count reaches 2^16).  The histogram is kept as 16-bit
// counts, two per word, and summarised per chunk of 32 bins: the counts
// below each chunk (cp) and each chunk's first and second moments (c1, c2).
// A clipping iteration then reads the two partial chunks at the ends of its
// cut range and the chunk sums between them, and finds the median split from
// the chunk prefix and one chunk's scan, instead of walking the cut range.
// The integer sums, the split and the double arithmetic are those of
// guess_from_hist, so the mode and sigma are the same bits.
constexpr int GW_WARPS = 4;                        // meshes (warps) per CTA
constexpr int GW_CH = (SX_QUANTIF_NMAXLEVELS + 2 + 31) / 32;  // 32-bin chunks
constexpr int GW_WORDS = GW_CH * 16;              // 16-bit counts of GW_CH * 32 bins

struct __align__(16) GuessWarpSmem {
    unsigned hw[GW_WORDS];  // bin b: bits 16 (b & 1) .. of word b >> 1
    long long c2[GW_CH];    // sum over the chunk of bin^2 * count
    int c1[GW_CH];          // sum over the chunk of bin * count (< 2^28)
    int cp[GW_CH + 1];      // counts of the bins below chunk c
};

__device__ __forceinline__ int gw_hist(const GuessWarpSmem &S, int b) {
    return (int)((S.hw[b >> 1] >> ((b & 1) << 4)) & 0xffffu);
}

// counts of the bins below bin i (0 <= i <= 32 GW_CH), whole warp
__device__ __forceinline__ int gw_pfx(const GuessWarpSmem &S, int i, int lane) {
    const int c = i >> 5, r = i & 31;
    const int v = lane < r ? gw_hist(S, 32 * c + lane) : 0;
    return S.cp[c] + (int)__reduce_add_sync(0xffffffffu, (unsigned)v);
}

// one pixel into the histogram
__device__ __forceinline__ void gw_count(GuessWarpSmem &S, float v, float qscale, float cste, int nlevels) {
    const float b = v / qscale + cste;
    if (b != b) return;  // NaN: the host conversion yields INT_MIN
    const int bin = (int)b;
    if (bin >= 0 && bin < nlevels) atomicAdd(&S.hw[bin >> 1], 1u << ((bin & 1) << 4));
}

// backguess on the warp's histogram; every lane gets the mode and sigma
__device__ __forceinline__ void gw_guess(GuessWarpSmem &S, const MeshStat &bm, float &mode, float &sg) {
    const int lane = threadIdx.x & 31, nlevels = bm.nlevels;
    // chunk sums: lane owns chunks lane, lane + 32, ...; words read in an
    // order rotated by the lane (at most two lanes on a bank)
    int carry = 0;
    for (int c0 = 0; c0 < GW_CH; c0 += 32) {
        const int c = c0 + lane;
        int s0 = 0, k1 = 0, k2 = 0;
        if (c < GW_CH) {
#pragma unroll 4
            for (int t = 0; t < 16; t++) {
                const int tw = (t + lane) & 15;
                const unsigned wv = S.hw[16 * c + tw];
                const int n0 = (int)(wv & 0xffffu), n1 = (int)(wv >> 16), k = 2 * tw;
                s0 += n0 + n1;
                k1 += k * n0 + (k + 1) * n1;
                k2 += k * k * n0 + (k + 1) * (k + 1) * n1;
            }
            S.c1[c] = 32 * c * s0 + k1;
            S.c2[c] = (long long)(32 * c) * (32 * c) * s0 + (long long)(64 * c) * k1 + k2;
        }
        int inc = s0;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (c < GW_CH) S.cp[c] = carry + inc - s0;
        carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) S.cp[GW_CH] = carry;
    __syncwarp();

    // src/back.c:347-432, every lane computing the same values
    const int nlevelsm1 = nlevels - 1;
    double sig_ = 10.0 * nlevelsm1, sig1 = 1.0, mea = bm.mean, med = bm.mean;
    int lcut = 0, hcut = nlevelsm1;
    for (int n = 100;;) {
        if (!(n-- && (sig_ >= 0.1) && (fabs(sig_ / sig1 - 1.0) > SX_EPS))) break;
        const int nn = hcut - lcut + 1;
        // exact integer sums over [lcut, hcut]
        long long sum = 0, t1 = 0, t2 = 0;
        int il = lcut;
        const int base = gw_pfx(S, lcut, lane);
        if (nn > 0) {
            const int cl = lcut >> 5, ch = hcut >> 5;
            int p0 = 0, p1 = 0;
            long long p2 = 0;
            {
                const int b = 32 * cl + lane;
                if (b >= lcut && b <= hcut) {
                    const int v = gw_hist(S, b);
                    p0 += v;
                    p1 += b * v;
                    p2 += (long long)b * b * v;
                }
            }
            if (ch != cl) {
                const int b = 32 * ch + lane;
                if (b <= hcut) {
                    const int v = gw_hist(S, b);
                    p0 += v;
                    p1 += b * v;
                    p2 += (long long)b * b * v;
                }
            }
            for (int c = cl + 1 + lane; c < ch; c += 32) {
                p0 += S.cp[c + 1] - S.cp[c];
                p1 += S.c1[c];
                p2 += S.c2[c];
            }
            sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)p0);
            t1 = (int)__reduce_add_sync(0xffffffffu, (unsigned)p1);
            for (int o = 16; o > 0; o >>= 1) p2 += __shfl_xor_sync(0xffffffffu, p2, o);
            t2 = p2;
            // split of the two-pointer walk: the smallest bin i >= lcut with
            // pfx(i) + pfx(i + 1) >= sum + 2 pfx(lcut) (bin hcut qualifies);
            // first the chunk whose last bin qualifies, then the bin in it
            const int T = (int)sum + 2 * base;
            int cstar = ch;
            for (int c0 = cl; c0 <= ch; c0 += 32) {
                const int c = c0 + lane;
                const bool ok = c <= ch && 2 * S.cp[c + 1] - gw_hist(S, 32 * c + 31) >= T;
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                if (bal) {
                    cstar = c0 + __ffs(bal) - 1;
                    break;
                }
            }
            const int hk = gw_hist(S, 32 * cstar + lane);
            int inc = hk;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            const int pk = S.cp[cstar] + inc - hk;  // pfx(32 cstar + lane)
            const unsigned bal = __ballot_sync(0xffffffffu, 2 * pk + hk >= T);
            il = max(32 * cstar + (bal ? __ffs(bal) - 1 : 31), lcut);
        }
        const int ih = il - 1;
        const int pil = gw_pfx(S, il, lane), phc = gw_pfx(S, hcut + 1, lane);
        const unsigned long lowsum = (unsigned long)(pil - base);
        const unsigned long highsum = (unsigned long)(phc - pil);
        sig1 = sig_;
        sig_ = (double)t2;
        mea = (double)t1;
        const long hl = gw_hist(S, il), hh = ih >= 0 ? gw_hist(S, ih) : 0;
        med = ih >= 0 ? ((double)ih + 0.5 + ((double)highsum - lowsum) / (2.0 * (hl > hh ? hl : hh))) : 0.0;
        if (sum) {
            mea /= (double)sum;
            sig_ = sig_ / sum - mea * mea;
        }
        sig_ = sig_ > 0.0 ? sqrt(sig_) : 0.0;
        double ftemp;
        lcut = (ftemp = med - 3.0 * sig_) > 0.0 ? (int)(ftemp > 0.0 ? ftemp + 0.5 : ftemp - 0.5) : 0;
        hcut = (ftemp = med + 3.0 * sig_) < nlevelsm1 ? (int)(ftemp > 0.0 ? ftemp + 0.5 : ftemp - 0.5) : nlevelsm1;
    }
    // src/back.c:408: the C library abs(int) applied to the double sig
    if (abs((int)sig_) > 0.0) {
        if (fabs((mea - med) / sig_) < 0.3)
            mode = bm.qzero + (2.5 * med - 1.5 * mea) * bm.qscale;
        else
            mode = bm.qzero + med * bm.qscale;
    } else
        mode = bm.qzero + mea * bm.qscale;
    sg = sig_ * bm.qscale;
}

// The histogram of the n pixels of a sequence and its mode, by one warp, the
// next pixels on their way while these are counted: in registers, or through
// two buffers in the place of the chunk sums, which are not in use yet.
constexpr int GW_FETCH = 8;  // pixels of a lane at a time
static_assert(sizeof(GuessWarpSmem) - sizeof(unsigned) * GW_WORDS >= 2 * 32 * GW_FETCH * sizeof(float) &&
                  sizeof(unsigned) * GW_WORDS >= 2 * SEQ_STAGE * sizeof(float) && GW_WORDS % 4 == 0,
              "staged pixels fit the histogram's memory");

template <bool VALID, class LOAD>
__device__ __forceinline__ void gw_mode(LOAD load, int n, GuessWarpSmem &S, const MeshStat &bm, float &mode, float &sg) {
    const int lane = threadIdx.x & 31;
    const int nlevels = bm.nlevels;
    const float qscale = bm.qscale;
    const float cste = 0.499999 - bm.qzero / qscale;
    if constexpr (LOAD::REGS) {
        float v[SEQ_G], nv[SEQ_G];
        load.take(nv);
        for (int i = lane; i < GW_WORDS; i += 32) S.hw[i] = 0u;
        __syncwarp();
        for (int k0 = 0; k0 < n; k0 += SEQ_CHUNK) {
#pragma unroll
            for (int g = 0; g < SEQ_G; g++) v[g] = nv[g];
            load.take(nv);
#pragma unroll
            for (int g = 0; g < SEQ_G; g++)
                if (!VALID || v[g] > (float)-SX_BIG) gw_count(S, v[g], qscale, cste, nlevels);
        }
        __syncwarp();
    } else {
        float *const stage = reinterpret_cast<float *>(S.hw + GW_WORDS), *cur = stage;
        load.template fetch<GW_FETCH, false>(stage);
        for (int i = lane; i < GW_WORDS; i += 32) S.hw[i] = 0u;
        for (int k0 = 0; k0 < n; k0 += 32 * GW_FETCH) {
            float *const other = cur == stage ? stage + 32 * GW_FETCH : stage;
            if (k0 + 32 * GW_FETCH < n) {
                load.template fetch<GW_FETCH, false>(other);
                cp_wait<1>();
            } else {
                cp_wait<0>();
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < GW_FETCH; g++) {
                const float v = cur[lane + 32 * g];
                if (!VALID || v > (float)-SX_BIG) gw_count(S, v, qscale, cste, nlevels);
            }
            __syncwarp();
            cur = other;
        }
    }
    gw_guess(S, bm, mode, sg);
}

// backstat, backhisto and backguess of every mesh, one warp each
template <bool VEC>
__global__ void __launch_bounds__(32 * GW_WARPS) k_mesh_mode(const float *__restrict__ img, int w, int h, int bw, int bh,
                                                             int nbx, int nby, float *__restrict__ back,
                                                             float *__restrict__ sig, FrameScalars *sc) {
    sx_pdl();
    if (blockIdx.x == 0 && threadIdx.x == 0) init_scalars(sc);
    __shared__ GuessWarpSmem smem[GW_WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int m = blockIdx.x * GW_WARPS + wid;
    if (m >= nbx * nby) return;  // whole warp
    int x0, y0, mw, mh, nv;
    mesh_geometry(m, w, h, bw, bh, nbx, nby, x0, y0, mw, mh);
    const MeshLoad<VEC> load(img + (size_t)y0 * w + x0, w, mw, mh);
    MeshStat bm;
    // (the histogram's words hold the staged stretches first)
    seq_stat<false>(load, mw * mh, (float)(mw * mh * SX_BACK_MINGOODFRAC), reinterpret_cast<float *>(smem[wid].hw), bm,
                    nv);
    float mode = -SX_BIG, sg = -SX_BIG;
    if (bm.mean > -SX_BIG) {
        __syncwarp();
        gw_mode<false>(load, mw * mh, smem[wid], bm, mode, sg);
    }
    if (lane == 0) {
        back[m] = mode;
        sig[m] = sg;
    }
}

// ---------------------------------------------------------------------------
// BACKPHOTO_TYPE LOCAL, src/back.c:568-660 (localback): the mode of the
// background-subtracted pixels in a rectangular annulus, BACKPHOTO_THICK
// wide, around the object's box widened by a quarter of its size.  The
// reference collects the annulus pixels (per row the left and right strips,
// then the rows above the box, then the rows below) and runs backstat (two
// sequential double passes in that order), the histogram and backguess.
// ---------------------------------------------------------------------------
struct LocalBox {
    int ok, ixmin, ixmax, iymin, iymax, bxmin, bxmax, bymin, bymax;
};

__device__ __forceinline__ LocalBox local_box(int xmin, int xmax, int ymin, int ymax, int w, int h, int pbs) {
    LocalBox B;
    const int oxsize = xmax - xmin + 1, oysize = ymax - ymin + 1;
    const int bxnml = oxsize < w / 2 ? oxsize / 4 : (w - oxsize) / 4;
    const int bynml = oysize < h / 2 ? oysize / 4 : (h - oysize) / 4;
    B.ixmin = xmin - bxnml;
    B.ixmax = xmax + 1 + bxnml;
    B.iymin = ymin - bynml;
    B.iymax = ymax + 1 + bynml;
    B.bxmin = B.ixmin - pbs;
    B.bxmax = B.ixmax + pbs;
    B.bymin = B.iymin - pbs;
    B.bymax = B.iymax + pbs;
    B.ok = B.bymin >= 0 && B.bymax < h && B.bxmin >= 0 && B.bxmax < w;
    return B;
}

__device__ __forceinline__ int local_npix(const LocalBox &B, int pbs) {
    return (B.bymax - B.bymin) * 2 * pbs + ((B.iymin - B.bymin) + (B.bymax - B.iymax)) * (B.ixmax - B.ixmin);
}

// The annulus pixels lane, lane + 32, ... in the reference's collection order:
// three rectangles, the first (both strips) with a gap in its rows.  One copy
// after the other in a short loop: with sixteen at a time, each with its
// divisions, in three places, the warps waited for instructions more than half
// the time and the annuli of a 2501 x 1999 frame took 0.68 ms, now 0.56; the largest annuli, one
// warp each, last longest.
struct LocalLoad {
    static constexpr bool REGS = false;
    const float *sub;
    int w, n, i, reg, W, end, col, off, dcol, step, split, gap;  // split: first column beyond the gap
    LocalBox B;
    int pbs;
    __device__ __forceinline__ LocalLoad(const float *sub_, int w_, const LocalBox &B_, int pbs_)
        : sub(sub_), w(w_), i(threadIdx.x & 31), B(B_), pbs(pbs_) {
        n = local_npix(B, pbs);
        enter(0);
    }
    // to this lane's place in rectangle r
    __device__ __forceinline__ void enter(int r) {
        const int ns = (B.bymax - B.bymin) * 2 * pbs, iw = B.ixmax - B.ixmin, nt = (B.iymin - B.bymin) * iw;
        reg = r;
        W = max(r ? iw : 2 * pbs, 1);
        end = r == 0 ? ns : r == 1 ? ns + nt : n;
        split = r ? 0x7fffffff : pbs;
        gap = B.ixmax - pbs - B.bxmin;
        const int k = i - (r == 0 ? 0 : r == 1 ? ns : ns + nt), row = k / W, drow = 32 / W;
        col = k - row * W;
        off = ((r < 2 ? B.bymin : B.iymax) + row) * w + (r ? B.ixmin : B.bxmin);
        dcol = 32 - drow * W;
        step = drow * w;
    }
    template <int G, bool STRETCH>
    __device__ __forceinline__ void fetch(float *dst) {
        dst += seq_slot<STRETCH>(threadIdx.x & 31);
#pragma unroll 1
        for (int g = 0; g < G; g++, dst += seq_slot<STRETCH>(32)) {
            if (i < n) {
                while (i >= end) enter(reg + 1);
                cp_async4(dst, sub + off + col + (col >= split ? gap : 0));
            } else {
                *dst = __int_as_float(0x7fffffff);
            }
            i += 32;
            col += dcol;
            off += step;
            if (col >= W) {
                col -= W;
                off += w;
            }
        }
        cp_commit();
    }
};

// one warp per object: backstat over the valid annulus pixels (one mesh of
// one column) and, for annuli of fewer than 65536 pixels, the mode; nlevels =
// -1 marks "no local background" (annulus outside the frame, or no valid
// pixel)
__global__ void __launch_bounds__(32 * GW_WARPS) k_local_stat(const float *__restrict__ sub, int w, int h, int pbs,
                                                              const int *__restrict__ xmin,
                                                              const int *__restrict__ xmax,
                                                              const int *__restrict__ ymin,
                                                              const int *__restrict__ ymax, int n, const int *n_dev,
                                                              MeshStat *__restrict__ ls, float *__restrict__ dbkg) {
    sx_pdl();
    __shared__ GuessWarpSmem smem[GW_WARPS];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int o = blockIdx.x * GW_WARPS + wid;
    if (o >= sx_count(n, n_dev)) return;
    MeshStat s;
    s.mean = s.sigma = s.lcut = s.hcut = s.qzero = s.qscale = 0.f;
    s.nlevels = -1;
    s.npix = 0;
    float mode = 0.0f;
    const LocalBox B = local_box(xmin[o], xmax[o], ymin[o], ymax[o], w, h, pbs);
    if (B.ok) {
        const LocalLoad load(sub, w, B, pbs);
        MeshStat t;
        int nv;
        seq_stat<true>(load, load.n, 1.0f, reinterpret_cast<float *>(smem[wid].hw), t, nv);
        if (nv) {
            s = t;
            float sg;
            __syncwarp();
            if (load.n < 65536) gw_mode<true>(load, load.n, smem[wid], s, mode, sg);
        }
    }
    if (lane == 0) {
        ls[o] = s;
        dbkg[o] = mode;
    }
}

// annuli of 65536 pixels or more, one CTA per object: the histogram (integer
// counts, any order) and backguess
__global__ void __launch_bounds__(GUESS_THREADS) k_local_guess(const float *__restrict__ sub, int w, int h, int pbs,
                                                                 const int *__restrict__ xmin,
                                                                 const int *__restrict__ xmax,
                                                                 const int *__restrict__ ymin,
                                                                 const int *__restrict__ ymax, int n,
                                                                 const int *n_dev,
                                                                 const MeshStat *__restrict__ ls, float *dbkg) {
    sx_pdl();
    __shared__ int hist[SX_QUANTIF_NMAXLEVELS + 2];
    __shared__ int pfx[SX_QUANTIF_NMAXLEVELS + 2];
    const int o = blockIdx.x;
    if (o >= sx_count(n, n_dev)) return;
    const MeshStat bm = ls[o];
    if (bm.nlevels < 0) return;
    const LocalBox B = local_box(xmin[o], xmax[o], ymin[o], ymax[o], w, h, pbs);
    if (local_npix(B, pbs) < 65536) return;
    for (int i = threadIdx.x; i < SX_QUANTIF_NMAXLEVELS + 2; i += GUESS_THREADS) hist[i] = 0;
    __syncthreads();
    const int nlevels = bm.nlevels;
    const float qscale = bm.qscale, cste = 0.499999 - bm.qzero / qscale;
    auto bin_of = [&](float p) {
        if (!(p > -SX_BIG)) return;
        const float b = p / qscale + cste;
        if (b != b) return;
        const int bin = (int)b;
        if (bin >= 0 && bin < nlevels) atomicAdd(&hist[bin], 1);
    };
    const int sw = 2 * pbs, rows = B.bymax - B.bymin, iw = B.ixmax - B.ixmin;
    for (int i = threadIdx.x; i < rows * sw; i += GUESS_THREADS) {
        const int r = i / sw, c = i - r * sw;
        bin_of(sub[(size_t)(B.bymin + r) * w + (c < pbs ? B.bxmin + c : B.ixmax + c - pbs)]);
    }
    const int nt = B.iymin - B.bymin, nb2 = B.bymax - B.iymax;
    for (int i = threadIdx.x; i < (nt + nb2) * iw; i += GUESS_THREADS) {
        const int r = i / iw, c = i - r * iw;
        const int y = r < nt ? B.bymin + r : B.iymax + (r - nt);
        bin_of(sub[(size_t)y * w + B.ixmin + c]);
    }
    __syncthreads();
    float sg;
    guess_from_hist(hist, pfx, bm, dbkg + o, &sg);
}

// src/back.c:455-480: bad meshes take the mean of the nearest valid meshes.
// Writes back2 (all meshes) and fixes sigma in place for bad meshes.
__global__ void k_mesh_badfill(const float *__restrict__ back, float *__restrict__ sigma, float *__restrict__ back2,
                               int nx, int ny) {
    sx_pdl();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx * ny) return;
    float b = back[i];
    back2[i] = b;
    if (b > -SX_BIG) return;
    int px = i % nx, py = i / nx;
    float d2min = SX_BIG, val = 0.f, sval = 0.f, d2;
    int nmin = 0;
    for (int j = 0, y = 0; y < ny; y++)
        for (int x = 0; x < nx; x++, j++)
            if (back[j] > -SX_BIG) {
                d2 = (float)(x - px) * (x - px) + (y - py) * (y - py);
                if (d2 < d2min) {
                    val = back[j];
                    sval = sigma[j];
                    nmin = 1;
                    d2min = d2;
                } else if (d2 == d2min) {
                    val += back[j];
                    sval += sigma[j];
                    nmin++;
                }
            }
    back2[i] = nmin ? val / nmin : 0.0;
    sigma[i] = nmin ? sval / nmin : 1.0;
}

__device__ __forceinline__ float median_small(float *v, int n) {
    for (int i = 1; i < n; i++) {
        float t = v[i];
        int j = i - 1;
        while (j >= 0 && v[j] > t) {
            v[j + 1] = v[j];
            j--;
        }
        v[j + 1] = t;
    }
    return n & 1 ? v[n / 2] : (float)((v[n / 2 - 1] + v[n / 2]) / 2.0);
}

// src/back.c:482-533: median filter of the mesh maps (window shrunk at edges)
__global__ void k_mesh_median(const float *__restrict__ back, const float *__restrict__ sigma,
                              float *__restrict__ back3, float *__restrict__ sigma3, int nx, int ny, int npx,
                              int npy, float fthresh) {
    sx_pdl();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nx * ny) return;
    int px = i % nx, py = i / nx;
    int npx2 = nx - px - 1, npy2 = ny - py - 1;
    if (npx2 > npx) npx2 = npx;
    if (npx2 > px) npx2 = px;
    if (npy2 > npy) npy2 = npy;
    if (npy2 > py) npy2 = py;
    float bm[121], sm[121];
    int n = 0;
    for (int dy = -npy2; dy <= npy2; dy++)
        for (int dx = -npx2; dx <= npx2; dx++) {
            int j = (py + dy) * nx + px + dx;
            bm[n] = back[j];
            sm[n++] = sigma[j];
        }
    float med = median_small(bm, n);
    if (fabs(med - back[i]) >= fthresh) {
        back3[i] = med;
        sigma3[i] = median_small(sm, n);
    } else {
        back3[i] = back[i];
        sigma3[i] = sigma[i];
    }
}

// k-th smallest (0-based) of n floats (orderable keys), single CTA radix select
__device__ unsigned select_kth(const float *v, int n, int k, unsigned lowkey, unsigned *hist) {
    unsigned prefix = 0, mask = 0;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        // (mesh values are close together: most of a warp on one bin, which it
        // counts once; whole warps, 256 for a lane without a value)
        for (int i0 = 0; i0 < n; i0 += blockDim.x) {
            const int i = i0 + threadIdx.x;
            unsigned d = 256u;
            if (i < n) {
                const unsigned key = f2ord(v[i]);
                if (key >= lowkey && (key & mask) == prefix) d = (key >> shift) & 255u;
            }
            const unsigned same = __match_any_sync(0xffffffffu, d);
            if (d < 256u && (int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&hist[d], (unsigned)__popc(same));
        }
        __syncthreads();
        __shared__ unsigned s_digit, s_k;
        if (threadIdx.x < 32) {
            // the digit holding rank k: lane l owns bins 8l..8l+7, a warp scan
            // of the lane totals finds the owner, the owner its bin
            const int lane = threadIdx.x;
            unsigned c[8], tot = 0;
#pragma unroll
            for (int t = 0; t < 8; t++) tot += (c[t] = hist[lane * 8 + t]);
            unsigned incl = tot;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const unsigned sel = __ballot_sync(0xffffffffu, incl > (unsigned)k);
            const int owner = sel ? __ffs(sel) - 1 : 31;
            if (lane == owner) {
                unsigned below = incl - tot, d = lane * 8;
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if (d == (unsigned)(lane * 8 + t) && below + c[t] <= (unsigned)k && t < 7) {
                        below += c[t];
                        d++;
                    }
                s_digit = d;
                s_k = k - below;
            }
        }
        __syncthreads();
        prefix |= s_digit << shift;
        mask |= 255u << shift;
        k = s_k;
        __syncthreads();
    }
    return prefix;
}

// median of the n values with key >= lowkey out of v[0..m), by one CTA: the
// element of rank n / 2, or for even n the mean with the one below it (the
// next rank is the same value again or the smallest above it)
__device__ float median_of(const float *v, int m, int n, unsigned lowkey, unsigned *hist) {
    __shared__ unsigned s_le, s_above;
    const int k = n & 1 ? n / 2 : n / 2 - 1;
    const unsigned ka = select_kth(v, m, k, lowkey, hist);
    if (n & 1) return ord2f(ka);
    if (threadIdx.x == 0) {
        s_le = 0u;
        s_above = 0xffffffffu;
    }
    __syncthreads();
    unsigned le = 0, above = 0xffffffffu;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const unsigned key = f2ord(v[i]);
        if (key < lowkey) continue;
        if (key <= ka)
            le++;
        else
            above = min(above, key);
    }
    le = __reduce_add_sync(0xffffffffu, le);
    above = __reduce_min_sync(0xffffffffu, above);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_le, le);
        atomicMin(&s_above, above);
    }
    __syncthreads();
    const float a = ord2f(ka), b = s_le > (unsigned)k + 1u ? a : ord2f(s_above);
    __syncthreads();
    return (float)((a + b) / 2.0);
}

// global medians of the filtered maps (src/back.c:536-557), one CTA (which 0)
// for the background and one (1) for the rms and the thresholds that follow
// from it
struct MedianArgs {
    const float *back3, *sigma3;
    int nb, back_type, thresh_type;
    float back_value;
    double dthr, athr;
    FrameScalars *sc;  // null: no medians
};

__device__ __noinline__ void back_medians(const MedianArgs &M, int which) {
    const float *back3 = M.back3, *sigma3 = M.sigma3;
    const int nb = M.nb;
    FrameScalars *sc = M.sc;
    __shared__ unsigned hist[256];
    __shared__ unsigned s_npos;
    if (which == 0) {
        const float med = median_of(back3, nb, nb, 0u, hist);
        if (threadIdx.x == 0) sc->backmean = M.back_type == 1 ? M.back_value : med;
        return;
    }
    float backsig = median_of(sigma3, nb, nb, 0u, hist);
    if (backsig <= 0.0) {
        // median of the strictly positive sigmas, else 1.0
        if (threadIdx.x == 0) s_npos = 0;
        __syncthreads();
        unsigned c = 0;
        for (int i = threadIdx.x; i < nb; i += blockDim.x) c += sigma3[i] > 0.0f;
        atomicAdd(&s_npos, c);
        __syncthreads();
        const int npos = (int)s_npos;
        const unsigned low = f2ord(__uint_as_float(1u));  // smallest positive float
        if (npos > 0 && npos < nb)
            backsig = median_of(sigma3, nb, npos, low, hist);
        else
            backsig = 1.0;
    }
    if (threadIdx.x == 0) {
        sc->backsig = backsig;
        if (M.thresh_type == 1) {
            sc->dthresh = (float)M.dthr;
            sc->thresh = (float)M.athr;
        } else {
            sc->dthresh = (float)(M.dthr * backsig);
            sc->thresh = (float)(M.athr * backsig);
        }
        sc->e0cd = fexpo(sc->dthresh);
    }
}

// ... by themselves, for maps of more meshes than MED_BESIDE or whose rows take
// k_row_nodes_long
__global__ void __launch_bounds__(1024) k_back_medians(const __grid_constant__ MedianArgs M) {
    sx_pdl();
    back_medians(M, blockIdx.x);
}

// Splines.  The forward recurrences of src/back.c divide by values that do not
// depend on the data, and end in (float) / 6.0, a double division rounded to
// float.  A float divided by 6 never lies near the middle of two floats (6 m
// would need 25 bits or more for a midpoint m, and a float is at least 2^-28
// of it away), or is that middle exactly, so the float division gives the same
// value and is a third of the latency.
//
// One thread walks a line; what it reads again on the way back is kept in
// shared memory (the walks waited about 600 cycles a step on their own stores:
// 40 us and 37 us under ncu for the 64 x 64 meshes of a 4096 x 4096 frame, 28
// and 13 so).
constexpr int SPL_MAX = 768;   // longest line kept there; longer ones use the global arrays

// src/back.c:739-773 (makebackspline), one thread per mesh column; u: scratch
// of the columns longer than SPL_MAX
__global__ void __launch_bounds__(32) k_back_spline(const float *__restrict__ map, float *__restrict__ dmap,
                                                    float *__restrict__ u, int nbx, int nby) {
    sx_pdl();
    extern __shared__ float spl[];
    const int x = blockIdx.x * 32 + threadIdx.x;
    if (x >= nbx) return;
    if (nby <= 1) {
        dmap[x] = 0.0;
        return;
    }
    const bool in_smem = nby <= SPL_MAX;
    float *ux = in_smem ? spl + threadIdx.x : u + (size_t)x * nby;
    float *dx = in_smem ? spl + (size_t)32 * nby + threadIdx.x : dmap + x;
    const int us = in_smem ? 32 : 1, ds = in_smem ? 32 : nbx;
    float temp, dprev = 0.0f, uprev = 0.0f;
    dmap[x] = 0.0;
    float m0 = map[x], m1 = map[nbx + x];
#pragma unroll 8
    for (int y = 1; y < nby - 1; y++) {
        const float m2 = map[(size_t)(y + 1) * nbx + x];
        temp = -1 / (dprev + 4);
        dx[(size_t)y * ds] = dprev = temp;
        temp *= uprev - 6 * (m2 + m0 - 2 * m1);
        ux[(size_t)y * us] = uprev = temp;
        m0 = m1;
        m1 = m2;
    }
    dmap[(size_t)(nby - 1) * nbx + x] = 0.0;
    float dnext = 0.0f;
#pragma unroll 4
    for (int y = nby - 2; y >= 1; y--)
        dmap[(size_t)y * nbx + x] = dnext = (dx[(size_t)y * ds] * dnext + ux[(size_t)y * us]) / 6.0f;
}

// src/back.c:938-1040 (backrmsline): the rms map of every pixel from the
// row nodes of the sigma map, the same x interpolation as the background
// square: write rms * rms (the variance of WEIGHT_TYPE BACKGROUND)
__global__ void k_rms_map(const float *__restrict__ node, const float *__restrict__ dnode, const int *__restrict__ colk,
                          const float *__restrict__ coldx, int nbx, int w, long long n, float *__restrict__ out,
                          int square) {
    sx_pdl();
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int y = (int)(p / w), x = (int)(p - (long long)y * w);
    const float *nd = node + (size_t)y * nbx, *dnd = dnode + (size_t)y * nbx;
    float v;
    if (nbx <= 1) {
        v = nd[0];
    } else {
        const int k = colk[x];
        const float dx = coldx[x], cdx = 1 - dx;
        v = (float)(cdx * (nd[k] + (cdx * cdx - 1) * dnd[k]) + dx * (nd[k + 1] + (dx * dx - 1) * dnd[k + 1]));
    }
    out[p] = square ? v * v : v;
}

// src/back.c:790-862: y-interpolated nodes of every image row and their
// x-direction second derivatives; one block takes SPL_ROWS rows, all its
// threads the nodes, then one thread per row the recurrence.  The medians of
// the maps, which nothing here reads, are two more blocks in front where they
// do not last longer than the rows: with 4096 meshes the background stage took
// 0.238 ms with a launch of their own and 0.235 so, with 16384 2.87 and 2.93.
constexpr int SPL_ROWS = 32;
constexpr int SPL_THREADS = 256;
constexpr int MED_BESIDE = 4096;  // meshes

struct RowNode {
    const float *blo, *bhi, *dblo, *dbhi;
    float dy, cdy, dy3, cdy3;
    __device__ __forceinline__ RowNode(const float *back, const float *dback, int nbx, int nby, int backh, int y) {
        int yl;
        dy = (float)y / backh - 0.5;
        dy -= (yl = (int)dy);
        if (yl < 0) {
            yl = 0;
            dy -= 1.0;
        } else if (yl >= nby - 1) {
            yl = nby < 2 ? 0 : nby - 2;
            dy += 1.0;
        }
        cdy = 1 - dy;
        dy3 = (dy * dy * dy - dy);
        cdy3 = (cdy * cdy * cdy - cdy);
        blo = back + (size_t)nbx * yl;
        bhi = blo + nbx;
        dblo = dback + (size_t)nbx * yl;
        dbhi = dblo + nbx;
    }
    __device__ __forceinline__ float at(int x) const {
        return cdy * __ldg(blo + x) + dy * __ldg(bhi + x) + cdy3 * __ldg(dblo + x) + dy3 * __ldg(dbhi + x);
    }
};

__global__ void __launch_bounds__(SPL_THREADS) k_row_nodes(const float *__restrict__ back,
                                                           const float *__restrict__ dback, int nbx, int nby,
                                                           int backh, int h, float *__restrict__ node,
                                                           float *__restrict__ dnode,
                                                           const __grid_constant__ MedianArgs M) {
    sx_pdl();
    int block = blockIdx.x;
    if (M.sc) {
        if (block < 2) {
            back_medians(M, block);
            return;
        }
        block -= 2;
    }
    extern __shared__ float spl[];  // SPL_ROWS x (nbx | 1) nodes, as many u, the d of every column
    const int y0 = block * SPL_ROWS, rows = min(SPL_ROWS, h - y0), pitch = nbx | 1;
    float *su = spl + SPL_ROWS * pitch, *sd = su + SPL_ROWS * pitch;
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < rows; r += SPL_THREADS / 32) {
        const size_t at = (size_t)(y0 + r) * nbx;
        if (nby > 1) {
            const RowNode N(back, dback, nbx, nby, backh, y0 + r);
            for (int x = lane; x < nbx; x += 32) node[at + x] = spl[r * pitch + x] = N.at(x);
        } else {
            for (int x = lane; x < nbx; x += 32) {
                node[at + x] = __ldg(back + x);
                dnode[at + x] = __ldg(dback + x);
            }
        }
    }
    if (nby <= 1) return;
    __syncthreads();
    const bool walks = threadIdx.x < rows;
    float *u = su + threadIdx.x * pitch;
    if (walks) {
        const float *n = spl + threadIdx.x * pitch;
        float temp, dprev = 0.0f, uprev = 0.0f;
        // (every row's d is the same: the first row's is kept)
#pragma unroll 4
        for (int x = 1; x < nbx - 1; x++) {
            temp = -1 / (dprev + 4);
            dprev = temp;
            if (threadIdx.x == 0) sd[x] = temp;
            temp *= uprev - 6 * (n[x + 1] + n[x - 1] - 2 * n[x]);
            u[x] = uprev = temp;
        }
        u[0] = u[nbx - 1] = 0.0;
    }
    __syncthreads();
    if (walks) {
        float dnext = 0.0f;
#pragma unroll 4
        for (int x = nbx - 2; x >= 1; x--) u[x] = dnext = (sd[x] * dnext + u[x]) / 6.0f;
    }
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < rows; r += SPL_THREADS / 32)
        for (int x = lane; x < nbx; x += 32) dnode[(size_t)(y0 + r) * nbx + x] = su[r * pitch + x];
}

// the same for rows of more than SPL_MAX nodes, one thread per row, what it
// reads again in global memory (u: h x nbx)
__global__ void k_row_nodes_long(const float *__restrict__ back, const float *__restrict__ dback, int nbx, int nby,
                                 int backh, int h, float *__restrict__ node, float *__restrict__ dnode,
                                 float *__restrict__ u) {
    sx_pdl();
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    if (y >= h) return;
    float *nd = node + (size_t)y * nbx, *dnd = dnode + (size_t)y * nbx, *uu = u + (size_t)y * nbx;
    if (nby <= 1) {
        for (int x = 0; x < nbx; x++) {
            nd[x] = back[x];
            dnd[x] = dback[x];
        }
        return;
    }
    const RowNode N(back, dback, nbx, nby, backh, y);
    for (int x = 0; x < nbx; x++) nd[x] = N.at(x);
    float temp, dprev = 0.0f, uprev = 0.0f, nm = N.at(0), n0 = N.at(1);
    dnd[0] = uu[0] = 0.0;
    for (int x = 1; x < nbx - 1; x++) {
        const float np = N.at(x + 1);
        temp = -1 / (dprev + 4);
        dnd[x] = dprev = temp;
        temp *= uprev - 6 * (np + nm - 2 * n0);
        uu[x] = uprev = temp;
        nm = n0;
        n0 = np;
    }
    dnd[nbx - 1] = 0.0;
    float dnext = 0.0f;
    for (int x = nbx - 2; x >= 1; x--) dnd[x] = dnext = (dnd[x] * dnext + uu[x]) / 6.0f;
}

// the splines of a mesh map along y (dmap), then the nodes of every image row
// and their second derivatives along x; u: max(nbx * nby, h * nbx) floats; M:
// the medians to take beside (M.sc null: none).  Returns the launches.
int launch_map_nodes(const float *map, float *dmap, float *u, int nbx, int nby, int bh, int h, float *node,
                     float *dnode, float *rowu, const MedianArgs &M, cudaStream_t st) {
    static DevCache attr;
    attr.get([](int) {
        cudaFuncSetAttribute(k_back_spline, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * SPL_MAX * 4);
        cudaFuncSetAttribute(k_row_nodes, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             ((2 * SPL_ROWS + 1) * (SPL_MAX + 1)) * 4);
        return 1;
    });
    const size_t sb = nby <= SPL_MAX ? (size_t)64 * nby * 4 : 0;
    sx_launch(k_back_spline, (nbx + 31) / 32, 32, sb, st, map, dmap, u, nbx, nby);
    MedianArgs beside = M;
    if (nbx > SPL_MAX || M.nb > MED_BESIDE) beside.sc = nullptr;
    if (M.sc && !beside.sc) sx_launch(k_back_medians, 2, 1024, 0, st, M);
    if (nbx <= SPL_MAX)
        sx_launch(k_row_nodes, (h + SPL_ROWS - 1) / SPL_ROWS + (beside.sc ? 2 : 0), SPL_THREADS,
                  (size_t)(2 * SPL_ROWS + 1) * (nbx | 1) * 4, st, map, dmap, nbx, nby, bh, h, node, dnode, beside);
    else
        sx_launch(k_row_nodes_long, (h + 127) / 128, 128, 0, st, map, dmap, nbx, nby, bh, h, node, dnode, rowu);
    return M.sc && !beside.sc ? 3 : 2;
}

// ---------------------------------------------------------------------------
// weight maps: blank the unusable pixels, then (after the background) the
// scale factor sigfac and the calibrated variance map
// ---------------------------------------------------------------------------
// Maps are read and written once: four pixels (16 bytes) at a time where the
// arrays are aligned, two such words in flight per thread.  One pixel a thread,
// these passes over a 16384 x 16384 frame took 1.18 (mask) and 0.75 ms
// (variance); the bytes take 0.49 and 0.33.
constexpr int WM_PIX = 2048;  // pixels per block of 256 threads

template <class F>
__device__ __forceinline__ void map_words(long long n, bool vec, F f) {
    const long long base = (long long)blockIdx.x * WM_PIX;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const long long p = base + u * 1024 + threadIdx.x * 4;
        if (vec && p + 3 < n)
            f(p, true);
        else
            for (int k = 0; k < 4; k++)
                if (p + k < n) f(p + k, false);
    }
}

__global__ void __launch_bounds__(256) k_weight_mask(const float *__restrict__ img, const float *__restrict__ wmap,
                                                     int wtype, float *__restrict__ imgm, long long n) {
    sx_pdl();
    const bool vec = ((reinterpret_cast<uintptr_t>(img) | reinterpret_cast<uintptr_t>(wmap) |
                       reinterpret_cast<uintptr_t>(imgm)) & 15) == 0;
    auto one = [&](float v, float w) { return sx_rel_var(w, wtype) < 1e30f ? v : -1e30f; };
    map_words(n, vec, [&](long long p, bool four) {
        if (four) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(img + p)),
                         w = __ldg(reinterpret_cast<const float4 *>(wmap + p));
            *reinterpret_cast<float4 *>(imgm + p) =
                make_float4(one(v.x, w.x), one(v.y, w.y), one(v.z, w.z), one(v.w, w.w));
        } else {
            imgm[p] = one(__ldg(img + p), __ldg(wmap + p));
        }
    });
}

// One warp per mesh: exact mean of the relative variance over its usable
// pixels; ratio = mesh rms / sqrt(mean) for a usable mesh, -1 otherwise.  The
// map's pixels come as in the background statistics, the next ones on their way
// while these are added, in two double bins under a hint from the mesh's first
// pixels; a mesh with more pixels than bins hold, or a term outside them, is
// added (again) with XSum.  With XSum alone and four loads in flight, 16384 x
// 16384 pixels took 0.72 ms, now 0.28.  Maps without 16-byte rows (VEC false) are
// added with XSum as before: copied four bytes at a time the background stage of
// 2501 x 1999 pixels took 0.262 ms instead of 0.250.
constexpr int WR_WARPS = 4;

template <bool VEC>
__global__ void __launch_bounds__(32 * WR_WARPS) k_weight_ratio(const float *__restrict__ wmap, int wtype, int w, int h,
                                                                int bw, int bh, int nbx, int nby,
                                                                const float *__restrict__ sigma,
                                                                float *__restrict__ ratio) {
    sx_pdl();
    __shared__ __align__(16) float stage[VEC ? WR_WARPS : 1][2][VEC ? SEQ_CHUNK : 4];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int m = blockIdx.x * WR_WARPS + wid;
    if (m >= nbx * nby) return;
    int x0, y0, mw, mh;
    mesh_geometry(m, w, h, bw, bh, nbx, nby, x0, y0, mw, mh);
    const int np = mw * mh;
    const float *origin = wmap + (size_t)y0 * w + x0;
    Bin2 bins;
    bin_init(bins);
    bool ok = VEC && np <= BIN_MAX_TERMS;
    int n = 0;
    if (VEC && ok) {
        const int W = bin_width(np);
        const float r0 = lane < mw ? sx_rel_var(__ldg(origin + lane), wtype) : 0.0f;
        const unsigned seen = __reduce_max_sync(0xffffffffu, r0 > 0.0f && r0 < 1e30f ? __float_as_uint(r0) : 0u);
        const unsigned low = bin_low(bs_order(__uint_as_float(seen)) + 6, W);
        MeshLoad<VEC> load(origin, w, mw, mh);
        load.template fetch<SEQ_G, false>(stage[wid][0]);
        for (int k0 = 0, b = 0; k0 < np; k0 += SEQ_CHUNK, b ^= 1) {
            if (k0 + SEQ_CHUNK < np) {
                load.template fetch<SEQ_G, false>(stage[wid][b ^ 1]);
                cp_wait<1>();
            } else {
                cp_wait<0>();
            }
            __syncwarp();
#pragma unroll
            for (int g = 0; g < SEQ_G; g++) {
                const float r = sx_rel_var(stage[wid][b][lane + 32 * g], wtype);  // (NaN beyond the mesh: unusable)
                if (r < 1e30f) {
                    ok &= bin_add(bins, r, low, W);
                    n++;
                }
            }
            __syncwarp();
        }
    }
    double vsum;
    if (__all_sync(0xffffffffu, ok)) {
        for (int o = 16; o > 0; o >>= 1) {
            bins.b0 += __shfl_xor_sync(0xffffffffu, bins.b0, o);
            bins.b1 += __shfl_xor_sync(0xffffffffu, bins.b1, o);
        }
        vsum = bins.b0 + bins.b1;
    } else {
        XSum sv;
        xs_init(sv);
        n = 0;
        for (int y = 0; y < mh; y++) {
            const float *row = origin + (size_t)y * w;
            for (int x = lane; x < mw; x += 32) {
                const float r = sx_rel_var(__ldg(row + x), wtype);
                if (r < 1e30f) {
                    xs_add(sv, r);
                    n++;
                }
            }
        }
        vsum = xs_double(xs_warp_sum(sv));
    }
    n = (int)__reduce_add_sync(0xffffffffu, (unsigned)n);
    if (lane) return;
    float rt = -1.0f;
    if (!((float)n < (float)(mw * mh * SX_BACK_MINGOODFRAC))) {
        const double vmean = vsum / n;
        const float sm = sigma[m];
        if (vmean > 0.0 && sm > 0.0f) rt = (float)(sm / sqrt(vmean));
    }
    ratio[m] = rt;
}

// sigfac: median of the usable meshes' ratios (hmedian, src/misc.c:30), 1 if none
__global__ void k_weight_sigfac(const float *__restrict__ ratio, int nb, FrameScalars *sc) {
    sx_pdl();
    __shared__ unsigned hist[256];
    __shared__ unsigned s_npos;
    if (threadIdx.x == 0) s_npos = 0;
    __syncthreads();
    unsigned c = 0;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) c += ratio[i] > 0.0f;
    atomicAdd(&s_npos, c);
    __syncthreads();
    const int npos = (int)s_npos;
    const unsigned low = f2ord(__uint_as_float(1u));  // smallest positive float
    float f = 1.0f;
    if (npos) f = median_of(ratio, nb, npos, low, hist);
    if (threadIdx.x == 0) sc->sigfac = f;
}

__global__ void __launch_bounds__(256) k_weight_var(const float *__restrict__ wmap, int wtype, const FrameScalars *sc,
                                                    float *__restrict__ wvar, long long n) {
    sx_pdl();
    const float sigfac = sc->sigfac, sigfac2 = sigfac * sigfac;
    const bool vec = ((reinterpret_cast<uintptr_t>(wmap) | reinterpret_cast<uintptr_t>(wvar)) & 15) == 0;
    map_words(n, vec, [&](long long p, bool four) {
        if (four) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(wmap + p));
            *reinterpret_cast<float4 *>(wvar + p) =
                make_float4(sx_calib_var(v.x, wtype, sigfac2), sx_calib_var(v.y, wtype, sigfac2),
                            sx_calib_var(v.z, wtype, sigfac2), sx_calib_var(v.w, wtype, sigfac2));
        } else {
            wvar[p] = sx_calib_var(__ldg(wmap + p), wtype, sigfac2);
        }
    });
}

void launch_weight_mask(const float *img, const float *wmap, int wtype, float *imgm, long long n, cudaStream_t st) {
    if (n > 0) sx_launch(k_weight_mask, (unsigned)((n + WM_PIX - 1) / WM_PIX), 256, 0, st, img, wmap, wtype, imgm, n);
}

// after launch_background: sigfac from the filtered mesh rms map, then the
// calibrated variance of every pixel
void launch_weight_var(const BackBufs &B, const float *wmap, const FrameParams &P, float *ratio, float *wvar,
                       FrameScalars *d_sc, cudaStream_t st) {
    const int nb = P.nbx * P.nby;
    const long long n = (long long)P.w * P.h;
    if (P.wtype != 2) {
        const bool vec = P.w % 4 == 0 && P.bw % 4 == 0 && ((uintptr_t)wmap & 15) == 0;
        sx_launch(vec ? k_weight_ratio<true> : k_weight_ratio<false>, (nb + WR_WARPS - 1) / WR_WARPS, 32 * WR_WARPS,
                  0, st, wmap, P.wtype, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.sigma3, ratio);
        sx_launch(k_weight_sigfac, 1, 1024, 0, st, ratio, nb, d_sc);
    }
    sx_launch(k_weight_var, (unsigned)((n + WM_PIX - 1) / WM_PIX), 256, 0, st, wmap, P.wtype, d_sc, wvar, n);
}

void launch_background(BackBufs &B, const float *img, const FrameParams &P, FrameScalars *d_sc,
                       cudaStream_t st, int &launches) {
    int nb = P.nbx * P.nby;
    // 16-byte loads where every mesh row begins on and is a multiple of 16 bytes
    const bool vec = P.w % 4 == 0 && P.bw % 4 == 0 && ((uintptr_t)img & 15) == 0;
    if ((long long)P.bw * P.bh < 65536) {
        const unsigned g = (unsigned)((nb + GW_WARPS - 1) / GW_WARPS);
        if (vec)
            sx_launch(k_mesh_mode<true>, g, 32 * GW_WARPS, 0, st, img, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.back,
                      B.sigma, d_sc);
        else
            sx_launch(k_mesh_mode<false>, g, 32 * GW_WARPS, 0, st, img, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.back,
                      B.sigma, d_sc);
    } else {
        if (vec)
            sx_launch(k_mesh_stat<true>, nb, 32, 0, st, img, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.ms, d_sc);
        else
            sx_launch(k_mesh_stat<false>, nb, 32, 0, st, img, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.ms, d_sc);
        sx_launch(k_mesh_guess, nb, GUESS_THREADS, 0, st, img, P.w, P.h, P.bw, P.bh, P.nbx, P.nby, B.ms, B.back,
                  B.sigma);
        launches += 1;
    }
    sx_launch(k_mesh_badfill, (nb + 127) / 128, 128, 0, st, B.back, B.sigma, B.back2, P.nbx, P.nby);
    sx_launch(k_mesh_median, (nb + 127) / 128, 128, 0, st, B.back2, B.sigma, B.back3, B.sigma3, P.nbx, P.nby, P.nfx /
              2, P.nfy / 2, P.fthresh);
    MedianArgs M;
    M.back3 = B.back3;
    M.sigma3 = B.sigma3;
    M.nb = nb;
    M.back_type = P.back_type;
    M.thresh_type = P.thresh_type;
    M.back_value = P.back_value;
    M.dthr = P.detect_thresh;
    M.athr = P.analysis_thresh;
    M.sc = d_sc;
    launches += 3 + launch_map_nodes(B.back3, B.dback, B.u, P.nbx, P.nby, P.bh, P.h, B.rownode, B.rowdnode, B.rowu, M,
                                     st);
}

}  // namespace sx
