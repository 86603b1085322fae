// common.cuh -- shared device helpers for libsexgpu (sm_100a).
//
// Compiled with -fmad=false: every floating-point expression below evaluates
// with separately rounded IEEE operations in the order written, the same
// arithmetic the reference's host C code performs.
#pragma once

#include <cstdint>
#include <utility>
#include <cuda_runtime.h>

// ---------------------------------------------------------------------------
// Launches.  A frame is 70 short kernels in one stream, most of them a few
// microseconds on small frames, each depending on the one before.  They are
// launched with programmatic stream serialization: the next kernel's blocks are
// set up while the current one drains, and wait for its end (sx_pdl, the first
// statement of every kernel) before they touch anything.  The order of all
// memory operations is that of the plain launches.  160 x 160 frame 0.64 ->
// 0.53 ms, 1024 x 1024 through a captured graph 0.84 -> 0.74, 4096 x 4096 4.22
// -> 4.10.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sx_pdl() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
inline void sx_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

#define SX_BIG 1e+30
// blank (NaN) input pixels read as -BIG, like the FITS reader's blank value
__device__ __forceinline__ float sx_unblank(float v) { return v != v ? -1e+30f : v; }
#define SX_PI 3.1415926535898
#define SX_EPS (1e-4)
#define SX_BACK_MINGOODFRAC 0.5
#define SX_QUANTIF_NSIGMA 5
#define SX_QUANTIF_NMAXLEVELS 4096
#define SX_QUANTIF_AMIN 4
#define SX_MAXDEBAREA 3
#define SX_CLEAN_ZONE 10.0
#define SX_APER_OVERSAMP 5
#define SX_KRON_NSIG (3 * 2.0)
#define SX_CROWD_THRESHOLD 0.1
#define SX_MAXCONV 31
#define SX_NISO_ 8

// object flags, src/cuda/cudatypes.h:30-37
#define SX_OBJ_CROWDED 0x0001
#define SX_OBJ_MERGED 0x0002
#define SX_OBJ_SATUR 0x0004
#define SX_OBJ_TRUNC 0x0008
#define SX_OBJ_APERT_PB 0x0010

// device status word bits
#define SX_ST_RANGE 1
#define SX_ST_LOOP 2
#define SX_ST_CAPACITY 4  // a count beyond the capacity a captured pipeline was sized for
#define SX_ST_LOAD 8     // a tile load of the subtract/filter pipeline did not complete in time
#define SX_ST_THRESH 16   // zero or negative detection or analysis threshold
#define SX_ST_STOP (SX_ST_RANGE | SX_ST_LOOP | SX_ST_CAPACITY | SX_ST_LOAD | SX_ST_THRESH)

// A count known on the device only: *n_dev, at most the capacity n the launch
// was sized for; n itself when n_dev is null (the count known on the host).
__device__ __forceinline__ int sx_count(int n, const int *n_dev) { return n_dev ? min(n, max(*n_dev, 0)) : n; }

#define SX_ALLOC_OTHER 0x7fffffff

// ---------------------------------------------------------------------------
// Exact, order-free sums of float terms.
//
// The value v * 2^(e-23) is exact; e is the smallest binary exponent of the
// non-zero terms seen so far.  Adding a smaller-exponent term shifts v left
// (exactly).  Any order of adds and merges gives the same exact value, which
// is rounded once when read; denormal terms count as zero.  A term or a partial
// sum that does not fit when it is brought to the smallest exponent raises ovf.
// Whether one does depends on the order, so the kernel that reads the sum then
// takes it again as a WideSum.  (Terms that fit one by one may still add up to
// more than 127 bits: with FULL, for terms in no fixed order, that raises ovf
// too.)
// ---------------------------------------------------------------------------
#define XS_EMPTY 1000

struct XSum {
    __int128 v;
    int e;
    int ovf;
};

__device__ __forceinline__ void xs_init(XSum &s) {
    s.v = 0;
    s.e = XS_EMPTY;
    s.ovf = 0;
}

__device__ __forceinline__ int xs_bits(__int128 v) {
    unsigned __int128 m = v < 0 ? (unsigned __int128)(-v) : (unsigned __int128)v;
    unsigned long long hi = (unsigned long long)(m >> 64), lo = (unsigned long long)m;
    if (hi) return 128 - __clzll(hi);
    if (lo) return 64 - __clzll(lo);
    return 0;
}

// |v| at or above 2^126: two of them could wrap
__device__ __forceinline__ bool xs_full(__int128 v) {
    const unsigned long long hi = (unsigned long long)((unsigned __int128)v >> 64);
    return (hi ^ (hi << 1)) >> 63;
}

__device__ __forceinline__ void xs_rescale(XSum &s, int e) {
    if (e >= s.e) return;
    if (s.v != 0) {
        int sh = s.e - e;
        if (sh > 125 || xs_bits(s.v) + sh > 125) {
            s.ovf = 1;
            s.v = 0;
        } else {
            s.v = (__int128)((unsigned __int128)s.v << sh);
        }
    }
    s.e = e;
}

template <bool FULL = false>
__device__ __forceinline__ void xs_add(XSum &s, float f) {
    unsigned int u = __float_as_uint(f);
    int ef = (int)((u >> 23) & 0xff);
    if (ef == 0) return;
    ef -= 127;
    if (ef < s.e) xs_rescale(s, ef);
    int sh = ef - s.e;
    if (sh > 100) {
        s.ovf = 1;
        return;
    }
    unsigned int m = (u & 0x7fffffu) | 0x800000u;
    __int128 t = (__int128)((unsigned __int128)m << sh);
    if (u >> 31)
        s.v -= t;
    else
        s.v += t;
    if (FULL && xs_full(s.v)) s.ovf = 1;
}

template <bool FULL = false>
__device__ __forceinline__ void xs_merge(XSum &s, XSum b) {
    if (b.ovf) s.ovf = 1;
    if (b.e == XS_EMPTY) return;
    if (s.e == XS_EMPTY) {
        s.v = b.v;
        s.e = b.e;
        return;
    }
    if (b.e < s.e)
        xs_rescale(s, b.e);
    else if (s.e < b.e)
        xs_rescale(b, s.e);
    if (b.ovf) s.ovf = 1;
    s.v += b.v;
    if (FULL && xs_full(s.v)) s.ovf = 1;
}

// exact value -> nearest double (ties to even)
__device__ __forceinline__ double xs_double(const XSum &s) {
    if (s.v == 0 || s.e == XS_EMPTY) return 0.0;
    bool neg = s.v < 0;
    unsigned __int128 mag = neg ? (unsigned __int128)(-s.v) : (unsigned __int128)s.v;
    unsigned long long hi = (unsigned long long)(mag >> 64), lo = (unsigned long long)mag;
    double d;
    int sc;
    if (!hi) {
        d = __ull2double_rn(lo);
        sc = 0;
    } else {
        int k = 127 - __clzll(hi);  // msb position
        int drop = k - 63;
        unsigned long long top = (unsigned long long)(mag >> drop);
        unsigned __int128 rem = mag & ((((unsigned __int128)1) << drop) - 1);
        if (rem) top |= 1ull;
        d = __ull2double_rn(top);
        sc = drop;
    }
    d = scalbn(d, sc + s.e - 23);
    return neg ? -d : d;
}

__device__ __forceinline__ float xs_float(const XSum &s) { return (float)xs_double(s); }

__device__ __forceinline__ XSum xs_shfl_down(const XSum &s, int off) {
    XSum r;
    unsigned long long lo = (unsigned long long)s.v, hi = (unsigned long long)(s.v >> 64);
    lo = __shfl_down_sync(0xffffffffu, lo, off);
    hi = __shfl_down_sync(0xffffffffu, hi, off);
    r.v = (__int128)(((unsigned __int128)hi << 64) | lo);
    r.e = __shfl_down_sync(0xffffffffu, s.e, off);
    r.ovf = __shfl_down_sync(0xffffffffu, s.ovf, off);
    return r;
}

// full-warp reduction by a merge tree; the result is valid in lane 0
template <bool FULL>
__device__ __noinline__ XSum xs_warp_reduce_tree(XSum s) {
    for (int off = 16; off > 0; off >>= 1) xs_merge<FULL>(s, xs_shfl_down(s, off));
    return s;
}

// Full-warp exact sum, valid in every lane.  Every lane's value is brought to
// the warp's smallest exponent; when each then fits in 122 bits the 32 of them
// add in an int128 without overflow (a butterfly of plain integer adds).
// Otherwise the merge tree above decides, with its range check.  The exact
// value, and so every rounding of it, is the same either way.
template <bool FULL = false>
__device__ __forceinline__ XSum xs_warp_sum(XSum s) {
    int emin = s.e;
    for (int o = 16; o > 0; o >>= 1) emin = min(emin, __shfl_xor_sync(0xffffffffu, emin, o));
    int ovf = __any_sync(0xffffffffu, s.ovf);
    XSum r;
    r.e = emin;
    r.ovf = ovf;
    r.v = 0;
    if (emin == XS_EMPTY) return r;
    bool fits = true;
    __int128 v = 0;
    if (s.e != XS_EMPTY && s.v != 0) {
        int sh = s.e - emin;
        if (sh > 122 || xs_bits(s.v) + sh > 122)
            fits = false;
        else
            v = (__int128)((unsigned __int128)s.v << sh);
    }
    if (__all_sync(0xffffffffu, fits)) {
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long lo = (unsigned long long)v, hi = (unsigned long long)(v >> 64);
            lo = __shfl_xor_sync(0xffffffffu, lo, o);
            hi = __shfl_xor_sync(0xffffffffu, hi, o);
            v += (__int128)(((unsigned __int128)hi << 64) | lo);
        }
        r.v = v;
        if (FULL) r.ovf |= xs_full(v);
        return r;
    }
    s = xs_warp_reduce_tree<FULL>(s);
    unsigned long long lo = (unsigned long long)s.v, hi = (unsigned long long)(s.v >> 64);
    lo = __shfl_sync(0xffffffffu, lo, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    r.v = (__int128)(((unsigned __int128)hi << 64) | lo);
    r.e = __shfl_sync(0xffffffffu, s.e, 0);
    r.ovf = __shfl_sync(0xffffffffu, s.ovf, 0);
    return r;
}

// ---------------------------------------------------------------------------
// Exact sums of float terms, binned form: two double bins of W binary orders
// each, the upper one ending at the order `top` (a hint, for instance the order
// of the largest term expected).  A term of order e in (top - W, top] goes to
// the upper bin, one in (top - 2W, top - W] to the lower: it is a multiple of
// 2^(e - 23), so up to 2^t such terms (of one bin, over every lane that adds
// them up) sum below 2^53 units when W + 23 + t <= 53, and every double
// addition in the bin is exact.  The total is b0 + b1 rounded once, one double
// addition.  A nonzero term outside the bins (a subnormal one included, which
// xs_add counts as zero) makes bin_add return false; the caller then takes the
// sum again with XSum.  The hint only decides which terms fit: a wrong one costs
// a second pass, never a different result.
// ---------------------------------------------------------------------------
constexpr int BIN_MAX_BITS = 14;                  // at most 2^14 terms per sum
constexpr int BIN_MAX_TERMS = 1 << BIN_MAX_BITS;

struct Bin2 {
    double b0, b1;
};

__device__ __forceinline__ void bin_init(Bin2 &s) { s.b0 = s.b1 = 0.0; }

// width of the bins for up to n <= BIN_MAX_TERMS terms
__device__ __forceinline__ int bin_width(int n) { return 30 - (32 - __clz(max(n - 1, 1))); }

// magnitude bits of the smallest term of the lower bin, for the hint `top`;
// with a hint so small that the lower bin would reach the subnormals, no term
// fits
__device__ __forceinline__ unsigned bin_low(int top, int W) {
    const int e = top + 128 - 2 * W;
    return e > 0 ? (unsigned)min(e, 255 - 2 * W) << 23 : 0x80000000u;
}

__device__ __forceinline__ bool bin_add(Bin2 &s, float f, unsigned low, int W) {
    const unsigned ua = __float_as_uint(f) & 0x7fffffffu, r = ua - low;
    const double d = (double)f;
    // (predicated additions: neither a branch nor an addition of 0.0 a bin)
    asm("{ .reg .pred p; setp.ge.s32 p, %2, %3; @p add.rn.f64 %0, %0, %4; @!p add.rn.f64 %1, %1, %4; }"
        : "+d"(s.b0), "+d"(s.b1)
        : "r"((int)r), "r"(W << 23), "d"(d));
    return r < (unsigned)(2 * W) << 23 || ua == 0u;
}

// order of a float for the hint: exponent field - 127 (-127 for 0)
__device__ __forceinline__ int bs_order(float f) { return (int)((__float_as_uint(f) >> 23) & 0xff) - 127; }

// s += d exactly, for a double d that is a multiple of a power of two no
// smaller than 2^-1074 (every bin sum is)
template <bool FULL = false>
__device__ __forceinline__ void xs_add_double(XSum &s, double d) {
    if (d == 0.0) return;
    const unsigned long long u = (unsigned long long)__double_as_longlong(d);
    const int ed = (int)((u >> 52) & 0x7ff);
    unsigned long long m = u & 0xfffffffffffffull;
    if (ed) m |= 1ull << 52;
    const int tz = __ffsll((long long)m) - 1;
    m >>= tz;
    // d = m * 2^(te - 23) in the units of xs_add
    const int te = (ed ? ed : 1) - 1075 + tz + 23;
    if (te < s.e) xs_rescale(s, te);
    const int sh = te - s.e;
    if (sh + (64 - __clzll(m)) > 125) {
        s.ovf = 1;
        return;
    }
    const __int128 t = (__int128)((unsigned __int128)m << sh);
    if (u >> 63)
        s.v -= t;
    else
        s.v += t;
    if (FULL && xs_full(s.v)) s.ovf = 1;
}

template <bool FULL = false>
__device__ __forceinline__ void xs_add_bins(XSum &s, double b0, double b1) {
    xs_add_double<FULL>(s, b1);
    xs_add_double<FULL>(s, b0);
}

// ---------------------------------------------------------------------------
// Exact sums in any order, for the few that XSum does not hold: 320-bit integers
// in units of 2^-149, which hold 2^31 terms of any finite size; denormal terms
// count as zero, as in xs_add.  bad: a term is not finite, or the terms span
// more than WS_SPAN binary orders, which XSum holds in no order (one of its
// mantissas shifted by more than 101 bits needs more than 125).
// ---------------------------------------------------------------------------
constexpr unsigned WS_SPAN = 101;
constexpr int WS_WORDS = 5;

struct WideSum {
    unsigned long long w[WS_WORDS];
    unsigned lo, hi;  // smallest and largest exponent field of a term
    int bad;          // (of a warp's total)
};

__device__ __forceinline__ void ws_init(WideSum &s) {
#pragma unroll
    for (int k = 0; k < WS_WORDS; k++) s.w[k] = 0ull;
    s.lo = 255u;
    s.hi = 0u;
    s.bad = 0;
}

// w += t, or -= t as adding ~t and 1
__device__ __forceinline__ void ws_add_words(WideSum &s, const unsigned long long (&t)[WS_WORDS], bool neg) {
    unsigned long long carry = neg;
#pragma unroll
    for (int k = 0; k < WS_WORDS; k++) {
        const unsigned long long a = s.w[k] + carry, b = a + (neg ? ~t[k] : t[k]);
        carry = (unsigned long long)(a < carry) | (unsigned long long)(b < a);
        s.w[k] = b;
    }
}

__device__ __forceinline__ void ws_add(WideSum &s, float f) {
    const unsigned u = __float_as_uint(f), ef = (u >> 23) & 0xff;
    if (ef == 0u) return;
    s.lo = min(s.lo, ef);
    s.hi = max(s.hi, ef);
    if (ef == 255u) return;
    const unsigned sh = ef - 1u, o = sh & 63u;
    const int q = (int)(sh >> 6);
    const unsigned long long m = (u & 0x7fffffu) | 0x800000u, lo = m << o, hi = o > 40u ? m >> (64u - o) : 0ull;
    unsigned long long t[WS_WORDS];
#pragma unroll
    for (int k = 0; k < WS_WORDS; k++) t[k] = k == q ? lo : k == q + 1 ? hi : 0ull;
    ws_add_words(s, t, (u >> 31) != 0u);
}

// the warp's total, in every lane
__device__ __forceinline__ WideSum ws_warp_sum(WideSum s) {
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long t[WS_WORDS];
#pragma unroll
        for (int k = 0; k < WS_WORDS; k++) t[k] = __shfl_xor_sync(0xffffffffu, s.w[k], o);
        ws_add_words(s, t, false);
    }
    s.lo = __reduce_min_sync(0xffffffffu, s.lo);
    s.hi = __reduce_max_sync(0xffffffffu, s.hi);
    s.bad = s.hi == 255u || (s.hi > s.lo && s.hi - s.lo > WS_SPAN);
    return s;
}

// exact value -> nearest double (ties to even)
__device__ __forceinline__ double ws_double(WideSum s) {
    const bool neg = s.w[WS_WORDS - 1] >> 63;
    if (neg) {
        WideSum z;
        ws_init(z);
        ws_add_words(z, s.w, true);
        s = z;
    }
    // the top word that is not zero, the one below it, and the others
    int q = -1;
#pragma unroll
    for (int k = 0; k < WS_WORDS; k++)
        if (s.w[k] != 0ull) q = k;
    if (q < 0) return 0.0;
    unsigned long long top = 0ull, next = 0ull, rest = 0ull;
#pragma unroll
    for (int k = 0; k < WS_WORDS; k++) {
        top = k == q ? s.w[k] : top;
        next = k == q - 1 ? s.w[k] : next;
        rest |= k < q - 1 ? s.w[k] : 0ull;
    }
    const int lead = __clzll((long long)top);
    unsigned long long v = lead ? top << lead | next >> (64 - lead) : top;
    if ((next << lead | rest) != 0ull) v |= 1ull;
    const double d = scalbn(__ull2double_rn(v), 64 * q - lead - 149);
    return neg ? -d : d;
}

// f(o) by the whole warp, for the o of each lane with need set, one after the
// other (every lane of the warp calls this); false if there was none.  Callers
// have loaded what else they need before: the vote waits for need.
template <class F>
__device__ __forceinline__ bool warp_each(bool need, int o, F f) {
    unsigned m = __ballot_sync(0xffffffffu, need);
    if (!m) return false;
    for (; m; m &= m - 1u) {
        f(__shfl_sync(0xffffffffu, o, __ffs(m) - 1));
        __syncwarp();
    }
    return true;
}

// orderable integer image of a float (monotone for all finite floats)
__device__ __forceinline__ unsigned int f2ord(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned int o) {
    unsigned int u = (o & 0x80000000u) ? (o & 0x7fffffffu) : ~o;
    return __uint_as_float(u);
}

// Division of a pixel index by the frame width without the integer divide:
// q = floor(p * m / 2^64) with m = ceil(2^64 / d) is exact whenever
// p * d < 2^64, which holds for any 32-bit p and d.  d == 1 is m == 0.
struct FastDiv {
    unsigned long long m;
    unsigned d;
};
inline FastDiv make_fastdiv(unsigned d) {
    FastDiv f;
    f.d = d;
    f.m = d > 1 ? (~0ull) / d + 1 : 0ull;
    return f;
}
__device__ __forceinline__ unsigned fdiv(unsigned p, const FastDiv &f) {
    return f.m ? (unsigned)__umul64hi((unsigned long long)p, f.m) : p;
}

__device__ __forceinline__ int fexpo(float v) { return (int)((__float_as_uint(v) >> 23) & 0xff) - 127; }

// bilinear background at (x, y), src/back.c:685-731
__device__ __forceinline__ float back_at(const float *b, int nx, int ny, int backw, int backh, int x, int y) {
    int xl, yl, pos;
    double dx, dy, cdx;
    float b0, b1, b2, b3;
    dx = (double)x / backw - 0.5;
    dy = (double)y / backh - 0.5;
    dx -= (xl = (int)dx);
    dy -= (yl = (int)dy);
    if (xl < 0) {
        xl = 0;
        dx -= 1.0;
    } else if (xl >= nx - 1) {
        xl = nx < 2 ? 0 : nx - 2;
        dx += 1.0;
    }
    if (yl < 0) {
        yl = 0;
        dy -= 1.0;
    } else if (yl >= ny - 1) {
        yl = ny < 2 ? 0 : ny - 2;
        dy += 1.0;
    }
    pos = yl * nx + xl;
    cdx = 1 - dx;
    b += pos;
    b0 = *b;
    b1 = nx < 2 ? b0 : *(++b);
    b2 = ny < 2 ? *b : *(b += nx);
    b3 = nx < 2 ? *b : *(--b);
    return (float)((1 - dy) * (cdx * b0 + dx * b1) + dy * (dx * b2 + cdx * b3));
}

// ---------------------------------------------------------------------------
// Device-side parameters of one extraction
// ---------------------------------------------------------------------------
struct FrameParams {
    int w, h;
    int bw, bh, nbx, nby;           // meshes
    int nfx, nfy;                   // mesh filter window
    float fthresh;                  // BACK_FILTTHRESH
    int back_type;
    float back_value;
    int thresh_type;
    double detect_thresh, analysis_thresh;
    int conv_w, conv_h, filter_flag;
    int minarea, debminarea, nthresh;
    double mincont;
    int clean_flag;
    double clean_param;
    double satur_level, gain, mag_zeropoint, aperture;
    int naper;                      // PHOT_APERTURES diameters (>= 1); aperture = apertures[0]
    double apertures[SEXGPU_MAXAPER];
    double autoparam0, autoparam1;
    int mask_type, numbering;
    int wtype;                      // weight map: 0 none, 1 MAP_VAR, 2 MAP_RMS, 3 MAP_WEIGHT
    int wthr;                       // thresholds follow the local rms (weight map, relative thresholds)
    double seeing, pixscale;        // SEEING_FWHM, PIXEL_SCALE (CLASS_STAR)
    int bp_local, bp_thick;         // BACKPHOTO_TYPE LOCAL, BACKPHOTO_THICK
    int loop_cap;                   // > 0: cap on union-find walks and retries (failure tests); 0: built-in caps
};

// scalars computed on the device during one extraction
struct FrameScalars {
    float backmean, backsig, dthresh, thresh;
    float sigfac;                   // weight-map scale factor (1 without a map)
    int e0cd;                       // exponent of dthresh (all object cd >= dthresh)
    int status;                     // SX_ST_* bits
    int npix_above;
    int nroots;
    int nrootpix;
    int nobj;                       // objects after deblending
    int nsurv;                      // after CLEAN
    int kitems[2], kchunks[2];      // queued Kron boxes and their work items (pass 1, 2)
    int npeaks;                     // peaks of all raw objects (deblending)
    unsigned long long levpix;      // sum of the deblending level of every raw-object pixel
};

// ---------------------------------------------------------------------------
// Weight maps (restated after the SExtractor manual and src/weight.c:91-125;
// the reference has no weighted path).  Relative variance of a weight value:
// MAP_VAR v, MAP_RMS v^2, MAP_WEIGHT 1/v; calibrated variance: MAP_VAR
// v*sigfac^2, MAP_RMS v^2, MAP_WEIGHT sigfac^2/v.  NaN, a variance or rms at
// or above BIG and a weight at or below 0 are unusable (BIG).
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ float sx_rel_var(float v, int wtype) {
    float r;
    if (wtype == 1)
        r = v;
    else if (wtype == 2)
        r = v < 1e30f ? v * v : 1e30f;
    else
        r = v > 0.0f ? 1.0f / v : 1e30f;
    return r < 1e30f ? r : 1e30f;
}

__host__ __device__ __forceinline__ float sx_calib_var(float v, int wtype, float sigfac2) {
    float r;
    if (wtype == 1)
        r = v < 1e30f ? v * sigfac2 : 1e30f;
    else if (wtype == 2)
        r = v < 1e30f ? v * v : 1e30f;
    else
        r = v > 0.0f ? sigfac2 / v : 1e30f;
    return r < 1e30f ? r : 1e30f;
}

// detection / analysis threshold at a pixel of calibrated variance var
__device__ __forceinline__ float sx_pix_thr(bool wthr, double fac, float var, float global) {
    return wthr ? (float)(fac * sqrt((double)var)) : global;
}

