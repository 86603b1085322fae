// prim.cu -- device-wide exclusive scan, written for this library (no
// CUB/Thrust/CUDPP).  It replaces the CUDPP cudppScan / cudppCompact calls of
// the reference (src/cuda/cudadetection.cu:720-1072, cudadeblend.cu:792-1901);
// its cudppRadixSort calls have no counterpart: what they ordered is placed
// by counts instead (k_roots.cu, k_analyse.cu, k_post.cu).
#include "prim.cuh"

namespace sx {

constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// block-wide exclusive scan of one int per thread; returns the block total
__device__ __forceinline__ int block_exclusive_scan(int v, int *sh_warp, int &total) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int s = lane < nw ? sh_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) sh_warp[lane] = s;
    }
    __syncthreads();
    int base = wid ? sh_warp[wid - 1] : 0;
    total = sh_warp[nw - 1];
    __syncthreads();
    return base + x - v;
}

// The element count of a scan: n, or, when the count is only known on
// the device (a launch sized before the count exists, as in a captured graph),
// the smaller of n and *n_dev.
__device__ __forceinline__ int dev_count(int n, const int *n_dev) { return n_dev ? min(n, max(*n_dev, 0)) : n; }

__global__ void k_tile_sums(const int *__restrict__ in, int n, int *__restrict__ sums, const int *n_dev) {
    sx_pdl();
    __shared__ int sh[32];
    n = dev_count(n, n_dev);
    long long base = (long long)blockIdx.x * SCAN_TILE;
    int acc = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        long long i = base + (long long)threadIdx.x * SCAN_ITEMS + k;
        if (i < n) acc += in[i];
    }
    int tot;
    block_exclusive_scan(acc, sh, tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_tile_scan(const int *__restrict__ in, int *__restrict__ out, int n,
                            const int *__restrict__ offs, int *total, const int *n_dev) {
    sx_pdl();
    __shared__ int sh[32];
    n = dev_count(n, n_dev);
    long long base = (long long)blockIdx.x * SCAN_TILE;
    int v[SCAN_ITEMS], acc = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        long long i = base + (long long)threadIdx.x * SCAN_ITEMS + k;
        v[k] = i < n ? in[i] : 0;
        acc += v[k];
    }
    int tot;
    int pre = block_exclusive_scan(acc, sh, tot) + (offs ? offs[blockIdx.x] : 0);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        long long i = base + (long long)threadIdx.x * SCAN_ITEMS + k;
        if (i < n) out[i] = pre;
        pre += v[k];
    }
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *total = pre;
}

// One block over the whole array, SCAN_ONE_TILE elements a turn, with a second
// array of the same length for a second block.
constexpr int SCAN_ONE_ITEMS = 16;
constexpr int SCAN_ONE_TILE = SCAN_THREADS * SCAN_ONE_ITEMS;
// longest array scanned by one block: 64 Ki elements in four turns take about
// as long as the three launches of the tiled form (9 us), shorter ones less
constexpr int SCAN_ONE_MAX = 4 * SCAN_ONE_TILE;

struct ScanArray {
    const int *in;
    int *out, *total;
};

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_one(const ScanArray A, const ScanArray B, int n, const int *n_dev) {
    sx_pdl();
    __shared__ int sh[32];
    const ScanArray S = blockIdx.x ? B : A;
    n = dev_count(n, n_dev);
    int carry = 0;
    // 16-byte words where the arrays are aligned (a thread's elements are
    // consecutive: one at a time, a warp's loads touched 32 lines each)
    const bool vec = ((reinterpret_cast<uintptr_t>(S.in) | reinterpret_cast<uintptr_t>(S.out)) & 15) == 0;
    for (int t0 = 0; t0 < n; t0 += SCAN_ONE_TILE) {
        const int base = t0 + threadIdx.x * SCAN_ONE_ITEMS;
        const bool whole = vec && base + SCAN_ONE_ITEMS <= n;
        int v[SCAN_ONE_ITEMS], acc = 0;
        if (whole) {
#pragma unroll
            for (int k = 0; k < SCAN_ONE_ITEMS; k += 4) {
                const int4 q = *reinterpret_cast<const int4 *>(S.in + base + k);
                v[k] = q.x;
                v[k + 1] = q.y;
                v[k + 2] = q.z;
                v[k + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < SCAN_ONE_ITEMS; k++) v[k] = base + k < n ? S.in[base + k] : 0;
        }
#pragma unroll
        for (int k = 0; k < SCAN_ONE_ITEMS; k++) acc += v[k];
        int tot;
        int pre = block_exclusive_scan(acc, sh, tot) + carry;
        carry += tot;
        if (whole) {
#pragma unroll
            for (int k = 0; k < SCAN_ONE_ITEMS; k += 4) {
                int4 q;
                q.x = pre;
                q.y = q.x + v[k];
                q.z = q.y + v[k + 1];
                q.w = q.z + v[k + 2];
                pre = q.w + v[k + 3];
                *reinterpret_cast<int4 *>(S.out + base + k) = q;
            }
        } else {
#pragma unroll
            for (int k = 0; k < SCAN_ONE_ITEMS; k++) {
                if (base + k < n) S.out[base + k] = pre;
                pre += v[k];
            }
        }
    }
    if (S.total && threadIdx.x == 0) *S.total = carry;
}

size_t scan_temp_ints(long long n) {
    size_t t = 0;
    while (n > SCAN_ONE_MAX) {
        n = (n + SCAN_TILE - 1) / SCAN_TILE;
        t += 2 * n + 2;
    }
    return t + 2;
}

// out[i] = sum_{j<i} in[j]; *total (device, may be NULL) = sum of all.
// in and out may alias.  tmp: scan_temp_ints(n) ints.  n_dev (device, may
// be NULL): the count, at most n, when only the device knows it; the launch
// is sized for n.  Returns the number of kernels launched.
int exclusive_scan(const int *in, int *out, long long n, int *total, int *tmp, cudaStream_t st, const int *n_dev) {
    if (n <= 0) {
        if (total) cudaMemsetAsync(total, 0, sizeof(int), st);
        return 0;
    }
    if (n <= SCAN_ONE_MAX) {
        const ScanArray A{in, out, total};
        sx_launch(k_scan_one, 1, SCAN_THREADS, 0, st, A, A, (int)n, n_dev);
        return 1;
    }
    const int nt = (int)((n + SCAN_TILE - 1) / SCAN_TILE);
    int *sums = tmp, *offs = tmp + nt;
    sx_launch(k_tile_sums, nt, SCAN_THREADS, 0, st, in, (int)n, sums, n_dev);
    const int k = exclusive_scan(sums, offs, nt, nullptr, tmp + 2 * nt + 2, st, nullptr);
    sx_launch(k_tile_scan, nt, SCAN_THREADS, 0, st, in, out, (int)n, offs, total, n_dev);
    return 2 + k;
}

// two scans of arrays of the same length (one launch where one block each
// does it)
int exclusive_scan2(const int *in0, int *out0, int *total0, const int *in1, int *out1, int *total1, long long n,
                    int *tmp, cudaStream_t st) {
    if (n > 0 && n <= SCAN_ONE_MAX) {
        sx_launch(k_scan_one, 2, SCAN_THREADS, 0, st, ScanArray{in0, out0, total0}, ScanArray{in1, out1, total1},
                  (int)n, nullptr);
        return 1;
    }
    return exclusive_scan(in0, out0, n, total0, tmp, st, nullptr) + exclusive_scan(in1, out1, n, total1, tmp, st, nullptr);
}

}  // namespace sx
