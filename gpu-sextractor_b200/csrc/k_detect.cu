// k_detect.cu -- background subtraction fused with the detection filter and
// the threshold, then 8-connected component labelling.
//
// Reference: src/back.c:863-899 (subbackline, x interpolation),
// src/filter.c:39-95 (convolve), src/cuda/cudadetection.cu:36-276
// (threshold + CCL).  The CCL here is a union-find over the label image
// (tile-local union in shared memory, then unions across tile borders with
// atomicMin, then path flattening); every component ends labelled with its
// smallest linear pixel index, the label the reference's iterative
// propagation converges to.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "common.cuh"
#include "kernels.cuh"

namespace sx {

// mask taps of the size-specialised kernels, passed by value (constant bank)
struct ConvTaps {
    float m[121];
};

// background at (x, y) from the per-row node splines (src/back.c:863-899)
__device__ __forceinline__ float bkg_at(int x, int y, const BackBufs &B, int nbx, int back_type, float backmean) {
    if (back_type == 1) return backmean;
    const float *nd = B.rownode + (size_t)y * nbx;
    if (nbx <= 1) return nd[0];
    const float *dnd = B.rowdnode + (size_t)y * nbx;
    int k = B.colk[x];
    float dx = B.coldx[x];
    float cdx = 1 - dx;
    return (float)(cdx * (nd[k] + (cdx * cdx - 1) * dnd[k]) + dx * (nd[k + 1] + (dx * dx - 1) * dnd[k + 1]));
}

// The background map of every pixel, the values src/back.c:790-936
// (subbackline) writes into backline and subtracts: the BACKGROUND check
// image (src/readimage.c:114); backmean everywhere for an absolute background.
__global__ void k_back_map(BackBufs B, int nbx, int back_type, const FrameScalars *sc, int w, long long n,
                           float *__restrict__ out) {
    sx_pdl();
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int y = (int)(p / w), x = (int)(p - (long long)y * w);
    out[p] = bkg_at(x, y, B, nbx, back_type, sc->backmean);
}

// ---------------------------------------------------------------------------
// Background subtraction, detection filter, threshold and tile-local labels in
// one pass over the frame.
//
// Bound by issue slots (a 7x7 mask is 98 separately rounded multiplies and adds
// a pixel against 16 bytes), so the rest of the work is kept to few
// instructions: 64 x 32 output tiles on persistent CTAs, the next tile (halo
// included) in flight into a second buffer while this one is computed.  A
// thread subtracts the background from quads of one column position, whose
// spline constants stay in its registers for all the tile's rows, then filters
// 4 columns x 2 rows from 16-byte shared-memory words and writes 16-byte words;
// tiles without foreground skip the labelling.  With one column of 8 rows a
// thread, one pixel a store and lanes 18 to 31 idle over the background,
// 4096 x 4096 pixels with a 7x7 mask took 233 us and 336 warp instructions per
// 32 pixels, now 133 us and 193 (98 of them the mask's); a crowded field under
// a 5x5 mask 304, now 169 us; a weighted 16384 x 16384 frame 5.9, now 3.4 ms.
// Multiplies and adds of register pairs save a quarter of the instructions but
// no time (138 us: the pairs go through the pipe at half the rate).
//
// Frames whose rows are not a multiple of 16 bytes, or that do not start on a
// 16-byte boundary, cannot be brought in by TMA: for those (TMA = false) the
// tile comes by 4-byte asynchronous copies and the results go out a pixel at a
// time.  Under a kernel of their own, labelled in a pass of its own, a frame of
// 1023 x 1023 took 35 us here and 34 us for its components, now 17 and 18.
// ---------------------------------------------------------------------------
constexpr int ST_TW = 64, ST_TH = 32, ST_THREADS = 256;
constexpr int ST_MAXBH = ST_TH + 2 * 15;      // masks up to 31x31
constexpr unsigned ST_WAIT_LIMIT = 1u << 24;  // polls of the load barrier
constexpr int ST_QR = 2;                      // output rows of a thread's quads (16 quads x 16 row pairs)
constexpr int SP_NK = 16;                     // staged spline nodes per row (segments touching a tile + 1)

struct SpArgs {
    const float *img;
    float *sub, *cd;
    int *lab, *cnt;  // cnt: set to 0 at every tile component's label pixel, or null
    BackBufs B;
    int w, h, nbx, back_type, mw, mh, rxa, wthr, tilesx, ntiles;
    double dfac;
    const float *mask, *wvar;
    FrameScalars *sc;
};

__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Convolution of one quad of output columns in rows r0, r0 + 1 from the shared
// tile.  Each input row is read once and added into the output rows it serves;
// an output receives its terms in mask row-major order (mask rows in increasing
// order, columns left to right), as convolve() adds them.
template <int MW, int MH>
__device__ __forceinline__ void conv_quad(const ConvTaps &taps, const float *__restrict__ tile, int bw, int quad,
                                          int r0, float (&acc)[ST_QR][4]) {
    constexpr int RXA = ((MW / 2) + 3) & ~3, OFF = RXA - MW / 2, NQ = (OFF + MW + 2) / 4 + 1;
#pragma unroll
    for (int k = 0; k < ST_QR; k++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[k][c] = 0.0f;
#pragma unroll
    for (int R = 0; R < ST_QR + MH - 1; R++) {
        float v[4 * NQ];
        const float4 *row = reinterpret_cast<const float4 *>(tile + (r0 + R) * bw) + quad;
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const float4 f = row[q];
            v[4 * q] = f.x;
            v[4 * q + 1] = f.y;
            v[4 * q + 2] = f.z;
            v[4 * q + 3] = f.w;
        }
#pragma unroll
        for (int k = 0; k < ST_QR; k++) {
            const int j = R - k;
            if (j >= 0 && j < MH) {
#pragma unroll
                for (int i = 0; i < MW; i++)
#pragma unroll
                    for (int c = 0; c < 4; c++) acc[k][c] += taps.m[j * MW + i] * v[OFF + i + c];
            }
        }
    }
}

// any mask size (runtime loops, same order); c0: tile column of the first tap
__device__ __forceinline__ void conv_quad_any(const float *__restrict__ mask, const float *__restrict__ tile, int bw,
                                              int c0, int r0, int mw, int mh, float (&acc)[ST_QR][4]) {
#pragma unroll
    for (int k = 0; k < ST_QR; k++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[k][c] = 0.0f;
    for (int j = 0; j < mh; j++) {
        const float *t0 = tile + (r0 + j) * bw + c0;
        for (int i = 0; i < mw; i++) {
            const float m = __ldg(mask + j * mw + i);
#pragma unroll
            for (int k = 0; k < ST_QR; k++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[k][c] += m * t0[k * bw + i + c];
        }
    }
}

__device__ __forceinline__ void sp_issue(const CUtensorMap *tmap, float *buf, unsigned bar, int x, int y,
                                         unsigned bytes) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(smem_u32(buf)),
        "l"(tmap), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// the tile at (x, y) by 4-byte asynchronous copies, a warp per row; zero outside
// the frame (a copy of no bytes fills its destination with zeros)
__device__ __forceinline__ void sp_copy(const SpArgs &A, float *buf, int x, int y, int bw, int bh) {
    const int lane = threadIdx.x & 31;
    for (int ty = threadIdx.x >> 5; ty < bh; ty += ST_THREADS / 32) {
        const int gy = y + ty;
        const bool rin = gy >= 0 && gy < A.h;
        const float *row = A.img + (size_t)(rin ? gy : 0) * A.w;
        for (int tx = lane; tx < bw; tx += 32) {
            const int gx = x + tx;
            const bool in = rin && gx >= 0 && gx < A.w;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(buf + ty * bw + tx)),
                         "l"(row + (in ? gx : 0)), "r"(in ? 4 : 0)
                         : "memory");
        }
    }
}

__device__ __forceinline__ bool sp_wait(unsigned bar, unsigned parity) {
    unsigned done = 0;
    for (unsigned it = 0; it < ST_WAIT_LIMIT && !done; it++)
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
    return done != 0;
}

// acc >= the pixel's threshold, the float nearest to fac * sqrt(var) in double:
// an approximate threshold (its error below 5e-7 of it) decides unless acc is
// within 1e-5 of it, so that the double-precision root is rarely taken
__device__ __forceinline__ bool above_pix_thr(float acc, bool wthr, double fac, float var, float global) {
    if (!wthr) return acc >= global;
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(var));
    const float t = (float)fac * r;
    if (t > 1e-30f && t < 1e30f) {
        if (acc > t * 1.00001f) return true;
        if (acc < t * 0.99999f) return false;
    }
    return acc >= sx_pix_thr(true, fac, var, global);
}

// ---- union-find in shared memory (tile-local components)
__device__ __forceinline__ int sfind(const int *L, int a) {
    while (L[a] != a) a = L[a];
    return a;
}

__device__ __forceinline__ void sunion(int *L, int a, int b) {
    for (int it = 0; it < 4096; it++) {
        a = sfind(L, a);
        b = sfind(L, b);
        if (a == b) return;
        if (a < b) {
            int t = a;
            a = b;
            b = t;
        }
        int old = atomicMin(&L[a], b);
        if (old == a) return;
        a = old;
    }
}

// runs of foreground bits in a 64-pixel row mask
__device__ __forceinline__ int run_start64(unsigned long long starts, int b) {  // start of the run holding bit b
    return 63 - __clzll((long long)(starts & (~0ull >> (63 - b))));
}
__device__ __forceinline__ int run_end64(unsigned long long m, int b) {  // last bit of the run holding bit b
    const unsigned long long r = ~(m >> b);
    return r ? b + __ffsll((long long)r) - 2 : 63;
}

template <int MW, int MH, bool WEIGHTED, bool TMA>
__global__ void __launch_bounds__(ST_THREADS, 4) k_sub_filter(const __grid_constant__ CUtensorMap tmap,
                                                           const __grid_constant__ SpArgs A,
                                                           const __grid_constant__ ConvTaps taps) {
    sx_pdl();
    extern __shared__ __align__(128) float sp_smem[];
    __shared__ __align__(8) unsigned long long bars[2];
    __shared__ float2 s_nd[ST_MAXBH][SP_NK + 1];   // spline nodes (value, second derivative) of the tile's rows
    __shared__ unsigned long long s_row[ST_TH];    // the tile rows' foreground
    __shared__ int s_L[ST_TH * ST_TW];             // tile-local union-find, set at the runs' first pixels
    const int mw = MW > 0 ? MW : A.mw, mh = MH > 0 ? MH : A.mh;
    const int rx = mw / 2, ry = mh / 2, rxa = MW > 0 ? ((MW / 2) + 3) & ~3 : A.rxa;
    const int bw = ST_TW + 2 * rxa, bh = ST_TH + 2 * ry;
    const int tsz = (bw * bh + 31) & ~31;  // floats per tile buffer (128-byte multiple)
    float *const buf0 = sp_smem, *const buf1 = sp_smem + tsz;
    const int tid = threadIdx.x, lane = tid & 31;
    const int w = A.w, h = A.h;
    const unsigned bar0 = smem_u32(&bars[0]), bar1 = smem_u32(&bars[1]);
    const unsigned tbytes = (unsigned)(bw * bh * 4);
    if (TMA) {
        if (tid == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar1), "r"(1));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }
    auto load = [&](int t, int b) {  // tile t into buffer b
        const int x = (t % A.tilesx) * ST_TW - rxa, y = (t / A.tilesx) * ST_TH - ry;
        if (TMA) {
            if (tid == 0 && t < A.ntiles) sp_issue(&tmap, b ? buf1 : buf0, b ? bar1 : bar0, x, y, tbytes);
        } else {
            if (t < A.ntiles) sp_copy(A, b ? buf1 : buf0, x, y, bw, bh);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    };
    int t = blockIdx.x;
    load(t, 0);
    const float backmean = A.sc->backmean, dthresh = A.sc->dthresh;
    const bool spline = A.back_type != 1 && A.nbx > 1;
    // the background's part: one quad of the tile's columns, every rpp-th row
    const int nq = bw / 4, rpp = ST_THREADS / nq, brow = tid / nq, bq = tid - brow * nq;
    const bool bcol = brow < rpp, binner = 4 * bq >= rxa && 4 * bq < rxa + ST_TW;
    // the filter's part: one quad of the output columns in two rows
    const int qc = tid & 15, r0 = (tid >> 4) * ST_QR;
    int nabove = 0;
    bool failed = false;
    for (int it = 0; t < A.ntiles; it++, t += gridDim.x) {
        const int cur = it & 1;
        float *const tile = cur ? buf1 : buf0;
        const int x0 = (t % A.tilesx) * ST_TW, y0 = (t / A.tilesx) * ST_TH;
        // next tile into the other buffer (free: its last reads came before
        // this iteration's predecessor's barrier after the filter)
        load(t + gridDim.x, cur ^ 1);
        // while the load is in flight, the spline nodes of this tile's rows and
        // the column constants of this thread's quad
        const int gxa = x0 - rxa, qx = gxa + 4 * bq;
        const int nin = bcol && qx >= 0 ? min(max(w - qx, 0), 4) : 0;  // its columns in the frame
        int kmin = 0, k0 = 0;
        bool staged = true, step[4];
        float cdx[4], cb[4], cx[4], cdd[4];
        if (spline) {
            kmin = __ldg(A.B.colk + max(gxa, 0));
            const int nk = __ldg(A.B.colk + min(gxa + bw, w) - 1) - kmin + 2;
            staged = nk <= SP_NK;
            if (staged)
                for (int j = tid & 3; j < nk; j += 4)
                    for (int ty = tid >> 2; ty < bh; ty += ST_THREADS / 4) {
                        const int gy = y0 - ry + ty;
                        const size_t o = (size_t)gy * A.nbx + min(kmin + j, A.nbx - 1);
                        if (gy >= 0 && gy < h) s_nd[ty][j] = make_float2(__ldg(A.B.rownode + o), __ldg(A.B.rowdnode + o));
                    }
            int kp = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int x = min(max(qx + q, 0), w - 1);
                const float dx = __ldg(A.B.coldx + x);
                const int k = __ldg(A.B.colk + x) - kmin;
                if (q == 0) k0 = k;
                step[q] = q > 0 && k != kp;  // the next segment begins here
                kp = k;
                cx[q] = dx;
                cdx[q] = 1 - dx;
                cb[q] = cdx[q] * cdx[q] - 1;
                cdd[q] = dx * dx - 1;
            }
        }
        if (TMA) {
            // every thread polls; the outcome is made uniform before anyone acts on it
            if (!__syncthreads_and(sp_wait(cur ? bar1 : bar0, (unsigned)((it >> 1) & 1)))) {
                failed = true;
                break;
            }
        } else {
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
        }
        // subtract the background in place; outside the frame the loads left 0
        if (nin > 0)
            for (int ty = brow; ty < bh; ty += rpp) {
                const int gy = y0 - ry + ty;
                if (gy < 0 || gy >= h) continue;
                float4 *tp = reinterpret_cast<float4 *>(tile + ty * bw) + bq;
                float4 v4 = *tp;
                float v[4] = {v4.x, v4.y, v4.z, v4.w}, b[4];
                if (!spline) {
                    b[0] = A.back_type == 1 ? backmean : __ldg(A.B.rownode + (size_t)gy * A.nbx);
                    b[1] = b[2] = b[3] = b[0];
                } else if (staged) {
                    const float2 *nd = s_nd[ty] + k0;
                    float2 lo = nd[0], hi = nd[1];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (step[q]) {
                            nd++;
                            lo = hi;
                            hi = nd[1];
                        }
                        b[q] = cdx[q] * (lo.x + cb[q] * lo.y) + cx[q] * (hi.x + cdd[q] * hi.y);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        b[q] = bkg_at(min(qx + q, w - 1), gy, A.B, A.nbx, A.back_type, backmean);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) v[q] = TMA || q < nin ? sx_unblank(v[q]) - b[q] : 0.0f;
                v4 = make_float4(v[0], v[1], v[2], v[3]);
                *tp = v4;
                if (binner && ty >= ry && ty < ry + ST_TH) {
                    float *out = A.sub + (size_t)gy * w + qx;
                    if (TMA) {
                        *reinterpret_cast<float4 *>(out) = v4;
                    } else {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            if (q < nin) out[q] = v[q];
                    }
                }
            }
        __syncthreads();
        // convolution and threshold
        float acc[ST_QR][4];
        if constexpr (MW > 0)
            conv_quad<MW, MH>(taps, tile, bw, qc, r0, acc);
        else
            conv_quad_any(A.mask, tile, bw, 4 * qc + rxa - rx, r0, mw, mh, acc);
        const int gx = x0 + 4 * qc, ncol = min(max(w - gx, 0), 4);
        unsigned nib[ST_QR];  // bit c of nib[k]: pixel (gx + c, r0 + k) at or above its threshold
#pragma unroll
        for (int k = 0; k < ST_QR; k++) {
            const int gy = y0 + r0 + k;
            nib[k] = 0u;
            if (gy < h && ncol > 0) {
                const size_t p = (size_t)gy * w + gx;
                float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                if (TMA) {
                    *reinterpret_cast<float4 *>(A.cd + p) = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
                    if (WEIGHTED) {
                        const float4 f = __ldg(reinterpret_cast<const float4 *>(A.wvar + p));
                        v[0] = f.x;
                        v[1] = f.y;
                        v[2] = f.z;
                        v[3] = f.w;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (c < ncol) {
                            A.cd[p + c] = acc[k][c];
                            if (WEIGHTED) v[c] = __ldg(A.wvar + p + c);
                        }
                }
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    bool fg;
                    if (WEIGHTED)
                        fg = (v[c] < 1e30f) && above_pix_thr(acc[k][c], A.wthr, A.dfac, v[c], dthresh);
                    else
                        fg = acc[k][c] >= dthresh;
                    if (TMA || c < ncol) nib[k] |= (unsigned)fg << c;
                }
                nabove += __popc(nib[k]);
            }
        }
        // Components within the tile (the first step of the CCL, done here
        // while the tile's foreground is on chip): each tile row's foreground
        // as 64 bits, gathered from the 16 lanes of the row; the pixels of a
        // horizontal run have the run's first pixel as their tile label; a run
        // joins the runs of the row above that touch it or its diagonal ends.
        // Every link goes to a smaller tile index, so a tile component ends at
        // its smallest pixel, which is written as the label of each of its
        // pixels (global index).
        unsigned long long m[ST_QR];
        const bool wany = __any_sync(0xffffffffu, (nib[0] | nib[1]) != 0u);
#pragma unroll
        for (int k = 0; k < ST_QR; k++) {
            m[k] = 0ull;
            if (wany) {
                unsigned a = nib[k] << (4 * (lane & 7));
                a |= __shfl_xor_sync(0xffffffffu, a, 1);
                a |= __shfl_xor_sync(0xffffffffu, a, 2);
                a |= __shfl_xor_sync(0xffffffffu, a, 4);
                const unsigned o = __shfl_xor_sync(0xffffffffu, a, 8);
                m[k] = lane & 8 ? ((unsigned long long)a << 32) | o : ((unsigned long long)o << 32) | a;
                const unsigned long long st = m[k] & ~(m[k] << 1);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int b = 4 * qc + c, i = (r0 + k) * ST_TW + b;
                    if ((st >> b) & 1ull) s_L[i] = i;
                }
            }
            if (qc == 0) s_row[r0 + k] = m[k];
        }
        const bool any = __syncthreads_or(wany);
        if (any) {
#pragma unroll
            for (int k = 0; k < ST_QR; k++) {
                const int ty = r0 + k;
                const unsigned long long mk = m[k], st = mk & ~(mk << 1);
                unsigned mine = ty > 0 ? (unsigned)(st >> (4 * qc)) & 15u : 0u;
                if (!mine) continue;
                const unsigned long long mp = k ? m[0] : s_row[ty - 1], sp = mp & ~(mp << 1);
                while (mine) {
                    const int b = 4 * qc + __ffs(mine) - 1;
                    mine &= mine - 1;
                    const int e = run_end64(mk, b);
                    const int s1 = b > 0 ? b - 1 : 0, e1 = e < 63 ? e + 1 : 63;
                    const unsigned long long dil =
                        (e1 == 63 ? ~0ull : ((2ull << e1) - 1ull)) & ~((1ull << s1) - 1ull);
                    unsigned long long ov = mp & dil;
                    while (ov) {
                        const int o = __ffsll((long long)ov) - 1;
                        sunion(s_L, ty * ST_TW + b, (ty - 1) * ST_TW + run_start64(sp, o));
                        const int eo = run_end64(mp, o);
                        ov = eo >= 63 ? 0ull : ov & ~((2ull << eo) - 1ull);
                    }
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < ST_QR; k++) {
            const int gy = y0 + r0 + k;
            if (gy >= h || ncol == 0) continue;
            int l[4] = {-1, -1, -1, -1};
            if (nib[k]) {
                const unsigned long long st = m[k] & ~(m[k] << 1);
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    if (!((nib[k] >> c) & 1u)) continue;
                    if (c > 0 && ((nib[k] >> (c - 1)) & 1u)) {
                        l[c] = l[c - 1];
                    } else {
                        const int r = sfind(s_L, (r0 + k) * ST_TW + run_start64(st, 4 * qc + c));
                        l[c] = (y0 + r / ST_TW) * w + x0 + r % ST_TW;
                        if (A.cnt && l[c] == gy * w + gx + c) A.cnt[l[c]] = 0;
                    }
                }
            }
            int *out = A.lab + (size_t)gy * w + gx;
            if (TMA) {
                *reinterpret_cast<int4 *>(out) = make_int4(l[0], l[1], l[2], l[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++)
                    if (c < ncol) out[c] = l[c];
            }
        }
    }
    if (TMA && failed) {
        // A load did not complete in time: report it, and give the copies
        // still in flight one more bounded wait before the CTA exits.  A copy
        // that outlasts that wait too may still write into shared memory after
        // the CTA has gone, so this status (SEXGPU_ERR_LOAD) tells the caller
        // to destroy the context rather than use it again.
        if (tid == 0) {
            atomicOr(&A.sc->status, SX_ST_LOAD);
            sp_wait(bar0, 0);
            sp_wait(bar0, 1);
            sp_wait(bar1, 0);
            sp_wait(bar1, 1);
        }
        return;
    }
    nabove = __reduce_add_sync(0xffffffffu, nabove);
    if (lane == 0 && nabove) atomicAdd(&A.sc->npix_above, nabove);
}

// a 2D float tensor map of the frame with the tile box of this mask, or false
static bool make_frame_tmap(CUtensorMap *m, const float *img, int w, int h, int rxa, int ry) {
    // the driver's encoder, looked up once (a function-local static is
    // initialised once even when host threads arrive together)
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        cudaDriverEntryPointQueryResult q;
        void *fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (PFN_cuTensorMapEncodeTiled_v12000)fn;
        cudaGetLastError();
        return nullptr;
    }();
    if (!encode || ((uintptr_t)img & 15) || (w % 4) != 0) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)w, (cuuint64_t)h};
    const cuuint64_t strides[1] = {(cuuint64_t)w * 4};
    const cuuint32_t box[2] = {(cuuint32_t)(ST_TW + 2 * rxa), (cuuint32_t)(ST_TH + 2 * ry)};
    const cuuint32_t estr[2] = {1, 1};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void *)img, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// (smem << 8) | resident CTAs of each instance, per device
template <int MW, int MH, bool WEIGHTED, bool TMA>
static void sp_launch(const CUtensorMap &tmap, const SpArgs &A, const ConvTaps &taps, size_t smem, cudaStream_t st) {
    static DevCache nsm_cache;
    const int nsm = nsm_cache.get([](int dev) {
        int n = 148;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 148;
    });
    auto kern = k_sub_filter<MW, MH, WEIGHTED, TMA>;
    static std::atomic<long long> cached[64];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<long long> &slot = cached[dev >= 0 && dev < 64 ? dev : 0];
    const long long c = slot.load(std::memory_order_relaxed);
    int per = (int)(c & 255);
    if ((c >> 8) != (long long)smem) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        per = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, ST_THREADS, smem);
        per = std::min(std::max(per, 1), 255);
        slot.store(((long long)smem << 8) | per, std::memory_order_relaxed);
    }
    const int grid = std::max(1, std::min(A.ntiles, sx_share(nsm * per)));
    sx_launch(kern, grid, ST_THREADS, smem, st, tmap, A, taps);
}

template <bool WEIGHTED, bool TMA>
static void sp_launch_mask(const CUtensorMap &tmap, const SpArgs &A, const ConvTaps &taps, size_t smem,
                           cudaStream_t st) {
    const int m = A.mw == A.mh ? A.mw : 0;
    switch (m) {
        case 1: sp_launch<1, 1, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        case 3: sp_launch<3, 3, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        case 5: sp_launch<5, 5, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        case 7: sp_launch<7, 7, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        case 9: sp_launch<9, 9, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        case 11: sp_launch<11, 11, WEIGHTED, TMA>(tmap, A, taps, smem, st); break;
        default: sp_launch<0, 0, WEIGHTED, TMA>(tmap, A, taps, smem, st);
    }
}

// Subtracted and filtered frame, and as labels the components within each
// ST_TW x ST_TH tile; cnt (or null) is zeroed at the labels' pixels.
void launch_sub_filter(const float *img, float *sub, float *cd, int *lab, int *cnt, const BackBufs &B,
                       const FrameParams &P, FrameScalars *d_sc, const float *d_var, const ConvMask &M,
                       cudaStream_t st, int &launches) {
    const int mw = M.mw, mh = M.mh;
    const int rxa = ((mw / 2) + 3) & ~3;  // halo width rounded up to 16 bytes
    SpArgs A;
    A.img = img;
    A.sub = sub;
    A.cd = cd;
    A.lab = lab;
    A.cnt = cnt;
    A.B = B;
    A.w = P.w;
    A.h = P.h;
    A.nbx = P.nbx;
    A.back_type = P.back_type;
    A.mw = mw;
    A.mh = mh;
    A.rxa = rxa;
    A.wthr = P.wthr;
    A.tilesx = (P.w + ST_TW - 1) / ST_TW;
    A.ntiles = A.tilesx * ((P.h + ST_TH - 1) / ST_TH);
    A.dfac = P.detect_thresh;
    A.mask = M.dev;
    A.wvar = d_var;
    A.sc = d_sc;
    ConvTaps taps;
    memset(&taps, 0, sizeof(taps));
    if (mw * mh <= 121) memcpy(taps.m, M.host, sizeof(float) * mw * mh);
    const int bw = ST_TW + 2 * rxa, bh = ST_TH + 2 * (mh / 2);
    const size_t smem = 2 * sizeof(float) * (size_t)((bw * bh + 31) & ~31);
    CUtensorMap tmap;
    memset(&tmap, 0, sizeof(tmap));
    const bool tma = make_frame_tmap(&tmap, img, P.w, P.h, rxa, mh / 2);
    if (d_var)
        tma ? sp_launch_mask<true, true>(tmap, A, taps, smem, st) : sp_launch_mask<true, false>(tmap, A, taps, smem, st);
    else
        tma ? sp_launch_mask<false, true>(tmap, A, taps, smem, st)
            : sp_launch_mask<false, false>(tmap, A, taps, smem, st);
    launches += 1;
}

// ---------------------------------------------------------------------------
// union-find CCL
// ---------------------------------------------------------------------------
// walk to the root; a walk longer than cap steps sets SX_ST_LOOP and stops
__device__ __forceinline__ int gfind(const int *L, int a, int cap, int *status) {
    for (int n = 0; n <= cap; n++) {
        int p = L[a];
        if (p == a) return a;
        a = p;
    }
    atomicOr(status, SX_ST_LOOP);
    return a;
}

// walk and link caps: the built-in ones, or a smaller cap set for a test
__device__ __forceinline__ int ccl_walk_cap(int loop_cap) { return loop_cap > 0 ? loop_cap : (1 << 28); }
__device__ __forceinline__ int ccl_link_cap(int loop_cap) { return loop_cap > 0 ? loop_cap : (1 << 20); }

__device__ __forceinline__ void gunion(int *L, int a, int b, int *status, int loop_cap) {
    const int wcap = ccl_walk_cap(loop_cap), lcap = ccl_link_cap(loop_cap);
    for (int it = 0; it < lcap; it++) {
        a = gfind(L, a, wcap, status);
        b = gfind(L, b, wcap, status);
        if (a == b) return;
        if (a < b) {
            int t = a;
            a = b;
            b = t;
        }
        int old = atomicMin(&L[a], b);
        if (old == a) return;
        a = old;
    }
    atomicOr(status, SX_ST_LOOP);
}

// unions across tile borders (TW x TH tiles): pixels on the first row or
// first/last column of a tile look at their backward neighbours in other
// tiles, those on the last column at the NE one (row y - 1 of the next tile)
template <int TW, int TH>
__global__ void k_ccl_border(int *__restrict__ lab, int w, int h, int *status, int loop_cap) {
    sx_pdl();
    const int tilesx = (w + TW - 1) / TW, tile = blockIdx.x, k = threadIdx.x;  // k < TW + 2 (TH - 1)
    const int tx0 = (tile % tilesx) * TW, ty0 = (tile / tilesx) * TH;
    const bool east = k >= TW + TH - 1;
    const int x = k < TW ? tx0 + k : east ? tx0 + TW - 1 : tx0, y = k < TW ? ty0 : ty0 + 1 + (k - TW) % (TH - 1);
    if (x >= w || y >= h) return;
    const int p = y * w + x;
    if (lab[p] < 0) return;
    if (east) {
        if (x < w - 1 && lab[p - w + 1] >= 0) gunion(lab, p, p - w + 1, status, loop_cap);
        return;
    }
    // W neighbour (other tile when x is the tile's first column)
    if (x == tx0 && x > 0 && lab[p - 1] >= 0) gunion(lab, p, p - 1, status, loop_cap);
    if (y > 0) {
        // NW: other tile when x or y is on the tile's first column/row
        if (x > 0 && (x == tx0 || y == ty0) && lab[p - w - 1] >= 0) gunion(lab, p, p - w - 1, status, loop_cap);
        if (y == ty0 && lab[p - w] >= 0) gunion(lab, p, p - w, status, loop_cap);
        if (x < w - 1 && y == ty0 && lab[p - w + 1] >= 0) gunion(lab, p, p - w + 1, status, loop_cap);
    }
}

// every pixel to its root, and the component sizes: lanes of a warp holding
// the same root add once to cnt (zeroed before).  Four consecutive pixels a
// thread, their labels read and written as one 16-byte word where all four
// are in the frame: each entry written is -1 (background, which nothing else
// writes) or the pixel's root, so a concurrent walk through it still reads an
// ancestor (the walks only read).
__global__ void k_ccl_flatten(int *__restrict__ lab, long long n, int *__restrict__ cnt, int *status, int loop_cap) {
    sx_pdl();
    const long long base = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    const bool vec = base + 3 < n && (reinterpret_cast<uintptr_t>(lab) & 15) == 0;
    int l[4], r[4];
    if (vec) {
        const int4 v = *reinterpret_cast<const int4 *>(lab + base);
        l[0] = v.x;
        l[1] = v.y;
        l[2] = v.z;
        l[3] = v.w;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) l[k] = base + k < n ? lab[base + k] : -1;
    }
    bool changed = false;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        r[k] = l[k] >= 0 ? gfind(lab, (int)(base + k), ccl_walk_cap(loop_cap), status) : -1;
        changed |= r[k] != l[k];
    }
    if (changed) {
        if (vec) {
            *reinterpret_cast<int4 *>(lab + base) = make_int4(r[0], r[1], r[2], r[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (r[k] != l[k]) lab[base + k] = r[k];
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned same = __match_any_sync(0xffffffffu, r[k]);
        if (r[k] >= 0 && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&cnt[r[k]], __popc(same));
    }
}

// cnt: w*h ints, zeroed at the components' labels; receives the size of every component at its root
// lab: the tile-local components of k_sub_filter's tiles
void launch_ccl(int *lab, int *cnt, const FrameParams &P, FrameScalars *d_sc, cudaStream_t st, int &launches) {
    int *status = &d_sc->status;
    const int ntiles = ((P.w + ST_TW - 1) / ST_TW) * ((P.h + ST_TH - 1) / ST_TH);
    sx_launch(k_ccl_border<ST_TW, ST_TH>, ntiles, ST_TW + 2 * (ST_TH - 1), 0, st, lab, P.w, P.h, status, P.loop_cap);
    launches += 2;
    long long n = (long long)P.w * P.h;
    sx_launch(k_ccl_flatten, (unsigned)((n + 1023) / 1024), 256, 0, st, lab, n, cnt, status, P.loop_cap);
}

}  // namespace sx
